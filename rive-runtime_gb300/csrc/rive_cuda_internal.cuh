// Internal definitions shared by the sm_103a kernels of the flush backend.
//
// Record layouts are the reference's GPU records (renderer/include/rive/
// renderer/gpu.hpp): TessVertexSpan (291-376), GradientSpan (248-271),
// PathData (1593-1619), PaintData (1627-1653), PaintAuxData (1660-1691),
// ContourData (1698-1716), FlushUniforms (1466-1537). Flag values are those of
// renderer/src/shaders/constants.glsl.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace rivecuda
{
constexpr int kTessTextureWidth = 2048;
constexpr int kTessTextureWidthLog2 = 11;
constexpr int kGradTextureWidth = 512;
constexpr int kPatchSegmentSpan = 8;   // kMidpointFanPatchSegmentSpan
constexpr int kPatchVertexCount = 42;  // kMidpointFanPatchVertexCount
constexpr int kPatchIndexCount = 72;   // kMidpointFanPatchIndexCount
constexpr int kPatchTriangleCount = 24;
// Outer-curve patches (interior triangulation; gpu.hpp:591-646).
constexpr int kOuterPatchSegmentSpan = 17;   // OuterCubicPatchSegmentSpanPlusJoin
constexpr int kOuterPatchVertexCount = 153;  // kOuterCurvePatchVertexCount
constexpr int kOuterPatchTriangleCount = 83; // kOuterCurvePatchIndexCount / 3
// Center-AA midpoint-fan patches (feathered fills; gpu.hpp:591-646): both AA
// ramps of an 8-segment span, the 9-vertex fan and the midpoint vertex.
constexpr int kCenterPatchVertexCount = 8 * 8 + 8 + 2;           // 74
constexpr int kCenterPatchTriangleCount = (8 * 12 + 7 * 3 + 3) / 3; // 40
// gpu::DrawType values (gpu.hpp:657-668).
constexpr uint32_t DRAW_MIDPOINT_FAN_PATCHES = 0u;
constexpr uint32_t DRAW_MIDPOINT_FAN_CENTER_AA_PATCHES = 1u;
constexpr uint32_t DRAW_OUTER_CURVE_PATCHES = 2u;
constexpr uint32_t DRAW_INTERIOR_TRIANGULATION = 3u;
constexpr uint32_t DRAW_FEATHER_ATLAS_BLIT = 4u;
constexpr uint32_t DRAW_IMAGE_MESH = 6u;

constexpr float kPi = 3.14159265359f;
constexpr float k2Pi = 6.28318530718f;
constexpr float kAARadius = .5f;

constexpr uint32_t GRAD_SPAN_FLAG_LEFT_BORDER = 0x80000000u;
constexpr uint32_t GRAD_SPAN_FLAG_RIGHT_BORDER = 0x40000000u;
constexpr uint32_t GRAD_SPAN_FLAG_COMPLEX_BORDER = 0x20000000u;
constexpr uint32_t GRAD_SPAN_FLAGS_MASK = 0xe0000000u;

constexpr uint32_t RETROFIT_TRI_STRIP_CONTOUR_FLAG = 1u << 31;
constexpr uint32_t CULL_EXCESS_TESSELLATION_SEGMENTS_CONTOUR_FLAG = 1u << 29;
constexpr uint32_t JOIN_TYPE_MASK = 7u << 26;
constexpr uint32_t MITER_CLIP_JOIN_CONTOUR_FLAG = 5u << 26;
constexpr uint32_t MITER_REVERT_JOIN_CONTOUR_FLAG = 4u << 26;
constexpr uint32_t ROUND_JOIN_CONTOUR_FLAG = 2u << 26;
constexpr uint32_t FEATHER_JOIN_CONTOUR_FLAG = 1u << 26;
constexpr uint32_t EMULATED_STROKE_CAP_CONTOUR_FLAG = 1u << 25;
constexpr uint32_t NEGATE_PATH_FILL_COVERAGE_FLAG = 1u << 24;
constexpr uint32_t MIRRORED_CONTOUR_CONTOUR_FLAG = 1u << 23;
constexpr uint32_t JOIN_TANGENT_0_CONTOUR_FLAG = 1u << 22;
constexpr uint32_t JOIN_TANGENT_INNER_CONTOUR_FLAG = 1u << 21;
constexpr uint32_t LEFT_JOIN_CONTOUR_FLAG = 1u << 20;
constexpr uint32_t RIGHT_JOIN_CONTOUR_FLAG = 1u << 19;
constexpr uint32_t CONTOUR_ID_MASK = 0xffffu;

constexpr int STROKE_VERTEX = 0;
constexpr int FAN_VERTEX = 1;
constexpr int FAN_MIDPOINT_VERTEX = 2;

constexpr uint32_t CLIP_UPDATE_PAINT_TYPE = 0u;
constexpr uint32_t SOLID_COLOR_PAINT_TYPE = 1u;
constexpr uint32_t LINEAR_GRADIENT_PAINT_TYPE = 2u;
constexpr uint32_t RADIAL_GRADIENT_PAINT_TYPE = 3u;
constexpr uint32_t PAINT_FLAG_EVEN_ODD_FILL = 0x200u;

constexpr uint32_t MAX_DENORM_F16 = 1023u;
constexpr float EPSILON_FP16_NON_DENORM = 6.2e-5f;

// gpu::ShaderFeatures (gpu.hpp:840-856).
constexpr uint32_t SF_CLIPPING = 1u << 0;
constexpr uint32_t SF_CLIP_RECT = 1u << 1;
constexpr uint32_t SF_ADVANCED_BLEND = 1u << 2;
constexpr uint32_t SF_FEATHER = 1u << 3;
constexpr uint32_t SF_EVEN_ODD = 1u << 4;
constexpr uint32_t SF_NESTED_CLIPPING = 1u << 5;
constexpr uint32_t SF_HSL_BLEND_MODES = 1u << 6;
constexpr uint32_t SF_DITHER = 1u << 7;
constexpr uint32_t SF_MODULATED_IMAGE = 1u << 8;
// gpu::ShaderMiscFlags::clockwiseFill (gpu.hpp:917), the one misc flag a
// rasterOrdering draw batch carries. It travels with each triangle's shader
// features in bit 15, which ShaderFeatures leaves free.
constexpr uint32_t MISC_CLOCKWISE_FILL = 1u << 1;
// Feathering (constants.glsl:19-43, draw_path_common.glsl:7-13).
constexpr int kGaussianTableSize = 512;
constexpr float kGaussianStddevs = 3.f;
constexpr float kFeatherCoverageBias = -2.f;
constexpr float kFeatherCoverageThreshold = -1.5f;
constexpr float kFeatherXCoordBias = .25f;
constexpr float kHorizontalCotangentThreshold = 1e3f;
constexpr float kHorizontalCotangentValue = 1e6f;
constexpr float kFeatherJoinHelperVertexCount = 3.f;
// The inverse feather table for tessellation softening (kernels_tess.cu).
cudaError_t upload_inverse_feather_lut(const float table[kGaussianTableSize]);
void build_inverse_feather_table(float out[kGaussianTableSize]);
// The tessellation pass's device functions on n host items (kernels_tess.cu;
// rive_cuda_eval_tessellation_math).
cudaError_t run_tess_math(int fn, const float* in, float* out, size_t n);
// Uploads the feather table to a device once (kernels_raster.cu).
cudaError_t ensure_feather_lut(int device);
void feather_table_f16(uint16_t out[kGaussianTableSize]);
constexpr uint32_t FEATURE_CLOCKWISE_FILL = 1u << 15;
// A featherAtlasBlit triangle (main scenes): its coverage is the feather
// atlas sampled at the pixel, its coverage planes carry atlas coordinates.
constexpr uint32_t FEATURE_ATLAS_BLIT = 1u << 12;
// An atlas fill triangle that faced away (the atlas fill pipeline culls
// nothing): turned clockwise, its coverage is subtracted.
constexpr uint32_t FEATURE_ATLAS_NEGATE = 1u << 11;
// An image-mesh triangle: its colour is the batch's image at the texture
// coordinates of the pixel (planes in the feather-plane slots), blended at
// once, triangle by triangle.
constexpr uint32_t FEATURE_IMAGE_MESH = 1u << 10;
// Set by the raster as it stages a triangle: its path resolves without a clip,
// clip rect, advanced blend mode or image, from a solid colour or a gradient.
constexpr uint32_t FEATURE_SIMPLE = 1u << 9;
// The same bit of a triangle record: its tiles need the raster's extended variant
// (an image mesh, an atlas blit, a feathered draw, or an image paint).
constexpr uint32_t FEATURE_EXTENDED = 1u << 9;
// Two more bits of a triangle record's feature half-word, set only when the
// batch draws interior tiles as winding records: a fan triangle whose tiles
// are counted after its path's winding grid is complete, and the record of a
// patch's winding slot (one per midpoint-fan patch, after its 24 triangles).
constexpr uint32_t FEATURE_FAN_DEFERRED = 1u << 14;
constexpr uint32_t FEATURE_WINDING_SLOT = 1u << 13;
// A bin entry's value with this bit set names a winding slot, not a triangle.
constexpr uint32_t BIN_WINDING_ENTRY = 1u << 31;
// tileCounts value of a deferred fan triangle until its tiles are counted.
constexpr uint32_t kDeferredCount = 0xffffffffu;

// Per path of a batch, for drawing interior tiles as winding records: the
// path's tile box (clipped to the canvas), its place in the grid pool (one
// int32 winding and one edge byte per tile of the box), and the slot that
// carries its winding entries.
struct PathGrid
{
    int tx0, ty0, tx1, ty1; // tiles [tx0, tx1) x [ty0, ty1)
    uint32_t offset;        // first cell in the pool
    uint32_t flags;         // PATH_GRID_* bits
    uint32_t anchor;        // winding slot of the path's first patch
    uint32_t entries;       // winding entries (interior tiles with a nonzero winding)
    float length;           // pixels of control polygon (bounds the contour's length)
};
constexpr uint32_t PATH_GRID_ELIGIBLE = 1u; // a fill whose interior tiles may be winding records
constexpr uint32_t PATH_GRID_UNSAFE = 2u;   // a patch was discarded or non-finite: no winding records
constexpr uint32_t PATH_GRID_PLACED = 4u;   // the grid fits the pool (offset valid)
// Pixels of margin around a tile's pixel centres within which a contour edge
// or midpoint makes the tile an edge tile: an AA ramp lies within 1 px
// (max norm) of its contour edge, plus snapping and float rounding.
constexpr float kWindingEdgeMargin = 2.f;
// A path gets a winding grid only when its contour cannot mark more than
// this share of its box's tiles as edge tiles (a contour of length L crosses
// at most about 1.5 L / T tiles of size T, margins included): scribbles whose
// contour passes through nearly every tile keep their plain fans.
constexpr float kWindingMaxEdgeShare = .75f;

// Raster tiles: 16x16 by default; 8x8 and 32x32 are the autotuner's other
// choices (rive_cuda_set_raster_config).
constexpr int kTileSize = 16;
constexpr int kTileLog2 = 4;
// 32x32 tiles: staged records, block bits, per-warp triangle lists and coverage
// planes.
constexpr int kRaster32SmemBytes = 1024 * 80 + 32 * 32 * 4 + 32 * 1024 * 2 + 32 * 32 * 32 + 512;

// Device error word bits (read by rive_cuda_sync).
constexpr uint32_t ERR_BAD_TESS_INDEX = 1u << 0;
constexpr uint32_t ERR_BAD_CONTOUR = 1u << 1;
constexpr uint32_t ERR_BAD_PATH = 1u << 2;
constexpr uint32_t ERR_RESERVED_8 = 1u << 3; // no longer raised (feathers are drawn)
constexpr uint32_t ERR_COORD_RANGE = 1u << 4;
constexpr uint32_t ERR_BIN_OVERFLOW = 1u << 5;
constexpr uint32_t ERR_BAD_MESH_INDEX = 1u << 6;

// One set-up triangle, ready for the tile raster (96 bytes). Edge k is
// E_k(p) = A_k * (p.x - ax_k) + B_k * (p.y - ay_k), positive inside. Each edge
// is anchored at its canonical endpoint (the same vertex for the two triangles
// that share the edge), so shared edges evaluate to bitwise-negated values and
// the fill is watertight. Coverage components are planes anchored at edge 0's
// anchor: cov(p) = c + gx * (p.x - ax_0) + gy * (p.y - ay_0). The record also
// carries the path's PaintData words, so the raster never reads them from
// global memory, and the pixel bounding box for sub-tile rejection.
struct __align__(16) TriRecord
{
    float4 e0;   // ax, ay, A, B
    float4 e1;
    float4 e2;
    float4 cov0; // covx: c, gx, gy; covy: c
    float4 cov1; // covy: gx, gy; paint.x, paint.y (as float bits)
    uint4 meta;  // pathAndFeatures, x0 | x1 << 16, y0 | y1 << 16, key | scene << 16
};
static_assert(sizeof(TriRecord) == 96, "TriRecord layout");

// An image texture in device memory: RGBA8 premultiplied texels of every mip
// level, level l at texel offset off[l] with size max(w >> l, 1) x
// max(h >> l, 1); `sampler` is the ImageSampler key it is drawn with
// (include/rive/shapes/paint/image_sampler.hpp: wrapX + 3 wrapY + 9 filter).
constexpr int kMaxMipLevels = 16;
struct ImageTex
{
    const uchar4* texels;
    uint32_t width, height, levels, sampler;
    uint32_t off[kMaxMipLevels];
};
constexpr uint32_t PAINT_FLAG_HAS_IMAGE = 0x800u;
constexpr uint32_t kNoImage = 0xffffffffu;

// The mesh of an imageMesh draw batch: its render buffers (float2 positions,
// float2 texture coordinates, uint16 triangle list), the vertices both
// vertex buffers hold, its ImageDrawInstance and its image slot.
struct MeshDesc
{
    const float2* positions;
    const float2* uvs;
    const uint16_t* indices;
    uint32_t vertexCount, indexCount;
    uint32_t imageDraw, image;
    uint32_t pad;
};
constexpr uint32_t kNoMesh = 0xffffffffu;

struct FlushParams
{
    // Record buffers at the frame's element 0.
    const uint4* paths;      // PathData as 4 x uint4
    const uint2* paints;     // PaintData
    const float4* paintAux;  // PaintAuxData as 8 x float4
    const uint4* contours;   // ContourData
    const uint4* gradSpans;  // GradientSpan
    const uint4* tessSpans;  // TessVertexSpan as 4 x uint4
    uint32_t firstPath, firstPaint, firstPaintAux, firstContour;
    uint32_t firstGradSpan, gradSpanCount;
    uint32_t firstTessSpan, tessSpanCount;
    uint32_t pathCount, contourCount;
    uint32_t gradDataHeight, tessDataHeight;
    uint32_t gradTextureHeight; // rows the normalised gradient coordinate spans
    uint32_t width, height;
    uint32_t pathIDGranularity;
    float ditherScale, ditherBias;
    uint32_t wireframe;
    uint32_t loadClear;
    uint32_t clearColorPremulRGBA; // packed RGBA8, R in the low byte
    // Intermediate textures.
    uint4* tess;    // 2048 x tessDataHeight
    uchar4* grad;   // 512 x gradDataHeight
    uint32_t* error;
    uint32_t* fb;   // render target, RGBA8, width x height
    uint32_t tilesX;
    const uint32_t* triangleVertices; // TriangleVertex records (3 words each)
    uint32_t triangleVertexCount;
    // This flush's FlushUniforms record (device); scene_uniforms_kernel copies
    // pathIDGranularity and the dither terms from it before any other pass.
    const uint8_t* uniforms;
    // The flush's feather atlas: atlasW x atlasH fp16 texels, row-major. A
    // main scene samples it for its featherAtlasBlit draws; the flush's atlas
    // scene (atlasMode = 1: width x height = the atlas content, no target)
    // renders it.
    uint16_t* atlas;
    uint32_t atlasW, atlasH;
    uint32_t atlasMode;
    // Images: the batch's image table, and per path of this flush the slot of
    // the image its paint modulates (kNoImage: none), written by the set-up.
    const ImageTex* images;
    uint32_t* pathImage;
    // Image meshes: the flush's ImageDrawInstance records (4 x float4 each:
    // view matrix, clip-rect inverse matrix, translates, then opacity, clip
    // ID, blend mode, z index as words), and FlushUniforms::mipMapLODBias
    // (copied by scene_uniforms_kernel).
    const float4* imageDraws;
    uint32_t imageDrawCount;
    float mipLodBias;
};

// One DrawBatch of one flush in a set-up work list: its first element (patch
// instance, or triangle vertex for interior triangulation), its shader
// features and where its triangle slots start.
struct PatchSegment
{
    uint32_t scene, baseElement, features, slotBase;
    // Pixel rectangle the segment's triangles are clipped to, as
    // left | top << 16 and right | bottom << 16: an atlas batch's scissor, or
    // everything (0, 0xffffffff) for the draw batches of a main scene.
    uint32_t scissorLT, scissorRB;
    // The draw batch's image: a slot of the batch's image table, or kNoImage.
    uint32_t image;
    // An imageMesh batch's entry in the batch's mesh table, or kNoMesh.
    uint32_t mesh;
};

// Lanes that tessellate one span where spans are few (latency counts), and the
// most spans a warp takes where they are many (kernels_tess.cu). A 1080x1920 UI
// screen of 4.6 k spans 11 us with lanes, 14 packed; 4, 8 and 16 800x600 screens, 10, 16
// and 36 k spans, 18, 22 and 41 with lanes, 15, 15 and 19 packed, whose colour ramps
// then need a launch (4 screens' whole call 112 us with lanes, 114 packed; 8: 157 and
// 147); 16 recorded frames, 33 k, 43 and 35; 64 UI screens, 139 k, 138 and 35.
constexpr int kTessLanes = 16;
constexpr int kTessPacked = 16;
constexpr uint32_t kTessPackedSpans = 16384;
// Spans a warp takes in the packed tessellation, as a power of two: 8, or 16 where
// eight spans' vertices (half their texels) would not give every lane two and there
// are warps enough (64 UI screens, 10 texels a span, 36 us with 16 and 43 with 8;
// strokes, 16 texels, 77 and 73; 16 recorded frames, 33 k spans of 13 texels, 41 and 35).
inline int tess_spans_log2(uint32_t spans, uint64_t texels)
{
    return spans >= 1u << 16 && texels < (uint64_t)spans * 12 ? 4 : 3;
}

// Triangles with large tile boxes. One warp tests a triangle's tiles 32 at a
// time; a canvas-wide triangle of a backdrop has 8,000 to 65,000 of them, and a
// patch of such triangles keeps its warp busy for hundreds of microseconds while
// the rest of the GPU is idle. Large boxes are therefore set aside and cut into up
// to kWideStrips strips of at least kWideStripTiles tiles, a warp each. With and
// without: set-up and binner of a 1080x1920 UI screen 18 + 24 us, 49 + 146; of 16
// recorded frames 175 + 71, 419 + 846 (the call alone 2.37 and 3.39 ms). The line of
// large batches lies where the two extra passes stop costing those whose many such
// triangles fill the GPU anyway: 20 plain canvases 8.56, 8.17 and 8.15 ms with it
// at 256, 512 and 1024 tiles, 8.15 ms without.
constexpr int kWideTiles = 1024;
// The line of a batch of `slots` triangles, where some scene has more than kWideTiles
// tiles: lower for small frames, which wait for their longest warp (1080x1080
// recorded feathered frame, 109 k slots: scan and binner 21, 21, 21 and 29 us at 128,
// 256, 512 and 1024 tiles, the call alone 133, 133, 134 and 145; a 1080x1920 UI screen
// the same at all four; 16 recorded frames, 1.8 M slots, 161, 94, 71 and 68, so not
// theirs).
inline uint32_t wide_tiles(uint32_t slots) { return slots <= 1u << 18 ? 256 : kWideTiles; }
constexpr int kWideStrips = 64;
constexpr int kWideStripTiles = 128;
constexpr uint32_t kWideCapacity = 16384; // triangles kept; more are walked in place

// Plain midpoint-fan set-up: up to kFanWarpEach patches (about a wave of warps)
// a warp each, above that three a warp; 128-thread CTAs.
constexpr uint32_t kFanWarpEach = 8192;

// Set-up work lists: midpoint-fan patches, outer-curve patches, interior
// triangles, center-AA midpoint-fan patches (items: instances, instances,
// triangles, instances).
constexpr int kSetupLists = 4;

// The work of a batch of independent logical flushes ("scenes"); a single
// flush is a batch of one. Every kernel maps its global work index to a scene
// through the prefix arrays (base[0] = 0, base[count] = total).
struct BatchTables
{
    const FlushParams* scenes;       // [sceneCount]
    const uint32_t* gradSpanBase;    // [sceneCount + 1]
    const uint32_t* tessSpanBase;    // [sceneCount + 1]
    const uint32_t* tileBase;        // [sceneCount + 1]
    const uint2* sceneTiles;         // [sceneCount]: (tileBase, tilesX)
    // Per set-up list: segments [segCount] and the prefix of their items
    // [segCount + 1].
    const PatchSegment* segments[kSetupLists];
    const uint32_t* segBase[kSetupLists];
    uint32_t segCount[kSetupLists];
    uint32_t totalItems[kSetupLists];
    uint32_t sceneCount;
    uint32_t totalGradSpans, totalTessSpans, totalTiles;
    // Tiles [0, mainTiles) belong to the flushes' targets, the rest to their
    // feather atlases (scenes after the main ones).
    uint32_t mainTiles;
    int tileLog2; // raster tile size of this batch (3, 4 or 5)
    // Per triangle slot, when the batch holds feathered fills or image
    // meshes: the planes of the feather coverage's third and fourth
    // components (cotTheta, y0), or of a mesh triangle's texture coordinates
    // (u, v), as (z0, dz/dx, dz/dy, w0), (dw/dx, dw/dy, anchor x, anchor y).
    float4* featherPlanes;
    // Image meshes of the batch (PatchSegment::mesh indexes it).
    const MeshDesc* meshes;
    // Triangles whose tile box holds more than wideTiles tiles: wide[0] of
    // them (at most wideCap are kept), slots from wide[1] on, and per kept
    // triangle the entries of each of its kWideStrips strips. Null: none is set
    // aside (no scene has more than kWideTiles tiles, or winding records).
    uint32_t* wide;
    uint32_t* wideStrips;
    uint32_t wideCap, wideTiles;
    // Interior tiles as winding records (null grids: off). Midpoint-fan
    // patches then take fanSlotStride = 25 slots (24 triangles and the
    // winding slot), otherwise 24.
    uint32_t fanSlotStride;
    const uint32_t* pathBase;  // [sceneCount + 1]: first path of each scene
    PathGrid* grids;           // [pathBase[sceneCount]]
    int32_t* gridWinding;      // pool: per cell, deltas, then the winding
    uint8_t* gridEdge;         // pool: per cell, nonzero for an edge tile
    uint32_t gridCapacity;     // cells in the pool
    uint32_t* gridCounters;    // [0] cells asked for, [1] winding entries
};

// The binner's view of BatchTables::wide and how many of its first CTAs write
// those triangles' pairs (0: no list).
struct WideScatter
{
    const uint32_t* list = nullptr;
    const uint32_t* strips = nullptr;
    uint32_t cap = 0;
    uint32_t blocks = 0;
    uint32_t perWarp = 32; // slots a warp takes of the others (bin_slots_per_warp)
};

// A small frame's binner waits for its longest warp, one with a backdrop's large
// triangles one after another: 8 slots a warp, not 32. Scan and binner at 4, 8, 16
// and 32: 1080x1080 recorded feathered frame, 109 k slots, 21, 21, 23 and 25 us; 240x180
// widget 18, 19, 21 and 21; 1080x1920 UI screen, 150 k, 26, 24, 27 and 28. Frames of
// more slots have other warps to run meanwhile: 16 recorded frames, 1.8 M, 113, 83, 72
// and 70; full-feature 1021x767, 8.4 M, 392, 242, 173 and 141.
inline uint32_t bin_slots_per_warp(uint32_t slots) { return slots <= 1u << 18 ? 8 : 32; }

struct TileHead;
// The binner's view of the main tiles that need the raster's extended variant
// (heads null: the whole batch takes one variant). Binning a triangle with
// FEATURE_EXTENDED to a tile sets kExtendedTile in the tile's head.
struct ExtendedTiles
{
    TileHead* heads = nullptr;
    uint32_t tiles = 0; // the main tiles, atlas tiles follow
};
constexpr uint32_t kExtendedTile = 1u << 31; // in TileHead::scene
// Batches are split from this many main tiles on: two launches are slower where a
// raster is short (4,624 tiles of a feathered frame 40 us, 44 split) or most of its tiles
// are extended (19,293 tiles: 647 and 656 us). 15,645 tiles, feathers on some: 312 and
// 301; 16 recorded frames, the whole call 2,026 and 1,995.
constexpr uint32_t kSplitTiles = 8192;

// CTAs (256 threads) of the two wide-triangle passes: two per SM's worth, a
// strip for every warp of 38 triangles.
constexpr uint32_t kWideBlocks = 304;

// A raster tile: its sorted bin entries [first, end), its scene, and its place
// there (tx | ty << 16), so a raster CTA starts from one 16-byte load instead of
// a binary search over the scenes and a division.
struct __align__(16) TileHead
{
    uint32_t first, end, scene, at;
};

// What flush_start_kernel prepares (kernels_small.cu): the flushes' uniforms, and
// the buffers that start at zero (gradVectors in 16-byte units; wide and error
// may be null).
struct FlushStart
{
    FlushParams* scenes;
    uint32_t sceneCount;
    uint32_t* wide;
    uint32_t* error;
    uint4* grad;
    uint32_t gradVectors;
    TileHead* ranges;
    uint32_t tiles;
    const uint32_t* tileBase; // BatchTables
    const uint2* sceneTiles;
};
// The scan and the sort of small frames, one cluster each (kernels_small.cu).
// small_passes_init finds the device's largest cluster for them (once per
// device, before any stream capture); the scan takes up to kSmallScanSlots slots,
// the sort up to small_sort_capacity entries.
constexpr uint32_t kSmallScanSlots = 1u << 18;
cudaError_t small_passes_init(int device, uint32_t* largest);
uint32_t small_sort_capacity(uint32_t largest);
cudaError_t launch_small_scan(uint32_t largest, uint32_t slots, const uint32_t* counts,
                              uint32_t* offsets, uint32_t* hostTotal, cudaStream_t stream,
                              bool overlap);
cudaError_t launch_small_sort(uint32_t largest, uint32_t entries, const uint32_t* entryTotal,
                              bool guarded, int keyBits, const uint16_t* keys, const uint32_t* vals,
                              uint32_t* sortedVals, TileHead* ranges, cudaStream_t stream,
                              bool overlap);

// Batches the raster grid orders its tiles for (tile_order_kernel).
constexpr uint32_t kOrderMinTiles = 512;
constexpr uint32_t kOrderTiles = 16384;

// The start of every kernel of a flush's chain, before it reads anything another
// one wrote: waits until the kernel before this one is complete (griddepcontrol;
// nothing in a launch without the attribute of chain_launch). Returns 0, opaque:
// added to the index that every load depends on, it keeps loads behind the wait
// also where the compiler takes their memory for constant.
__device__ __forceinline__ uint32_t chain_wait()
{
    uint32_t zero;
    asm volatile("griddepcontrol.wait;\n\t"
                 "mov.u32 %0, 0;"
                 : "=r"(zero)::"memory");
    return zero;
}
// Lets the next kernel of the chain start its CTAs once all of this one have
// started. Not in the kernels before a raster, whose CTAs would take every SM
// from other streams only to wait.
__device__ __forceinline__ void chain_next()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launches a kernel of a flush's chain. With `overlap` (the stream's last
// operation is a kernel that starts with chain_wait) its CTAs take their places
// while that one runs out; a small flush is eight kernels of a few microseconds,
// and a launch after a complete kernel adds one or two to each. With and without,
// other contexts' calls in the gaps: 240x180 widget 41 and 48 us, 1080x1080 recorded
// feathered frame 68 and 82; alone 73 and 90, 133 and 153, 1080x1920 UI screen 158 and
// 173 (81 and 77 among others). The host does it for frames of up to kSmallScanSlots:
// above, 64 UI screens, 4.1 M slots, lose 1% by it, a full-feature 1021x767 frame, 8.4
// M, gains 1%. At *priority unless that is null.
template <typename... P, typename... A>
cudaError_t chain_launch(void (*kernel)(P...), uint32_t ctas, int threads, size_t smem,
                         cudaStream_t stream, bool overlap, const int* priority, const A&... args)
{
    cudaLaunchAttribute attrs[2] = {};
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(ctas);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    c.attrs = attrs;
    if (overlap)
    {
        attrs[c.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attrs[c.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (priority)
    {
        attrs[c.numAttrs].id = cudaLaunchAttributePriority;
        attrs[c.numAttrs++].val.priority = *priority;
    }
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// Index j with base[j] <= i < base[j + 1] (empty ranges skipped), n >= 1.
__device__ __forceinline__ uint32_t find_range(const uint32_t* __restrict__ base, uint32_t n,
                                               uint32_t i)
{
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1)
    {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(base + mid) <= i)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}
} // namespace rivecuda
