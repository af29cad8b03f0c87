// gs_kernels.h -- launch arguments of the training-step kernels (host and
// device share these plain structs; nothing here is part of the C ABI).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "gs_common.cuh"

namespace gs {

// The projection's rectangle adds go to one of GRID_COPIES copies of the
// difference grid (by splat index), summed when the counts are read: every
// splat of a tile adds to the same four corner cells, and spreading those
// atomics over copies shortens the queues on the busiest cells.  Integer
// sums: the counts do not depend on the split.
constexpr uint32_t GRID_COPIES = 4;

// First kernel of a pass (k_step_begin).
struct StepBeginArgs {
  const uint32_t* ring;    // pinned host memory: `slots` parameter records `stride` words apart
  uint32_t slots, stride;
  uint32_t words;          // words of the record that the pass needs
  uint32_t* seq;           // passes run so far: this one takes slot seq % slots
  uint32_t* params;        // device copy of the record
  uint32_t* nItems;        // presort items of the pass, set to `items`
  uint32_t items;
  uint32_t* clear[3];      // word ranges set to zero
  uint32_t count[3];
  uint32_t sms;            // of the device
};

struct ProjectArgs {
  const float* params;     // n * 16
  const float* sh;         // n * 3K (channel-major) or null
  uint32_t n;
  int V;
  const DevCam* cams;      // V views
  float eCut, aMin, radClamp;
  int tile;
  RenderRec* recs;         // V * n
  uint32_t* pkeys;         // V * n presort keys: depth bits (all ones when culled)
  uint32_t* pvals;         // V * n presort values: slot = view * n + splat
  uint2* rect;             // V * n
  int32_t* diffGrid;       // GRID_COPIES copies of: per view (tilesX+1)*(tilesY+1), cleared before
  const uint32_t* gridBase;  // V offsets into a copy
  uint32_t gridCells;      // cells of one copy (all views)
  float4* cullRecs;        // V * n cull parameters (p, q, kA, 0) for the raster, or null: it has block bits
  uint4* itemSrc;          // V * n * 2: per visible slot (rect, mean, cull parameters, slot) for the expansion
};

struct TileRangeArgs {
  int V;
  const DevCam* cams;
  int32_t* diffGrid;
  const uint32_t* gridBase;
  uint32_t gridCells;
  uint32_t* tileCnt;       // per global tile: the reference's tileCnt
  uint8_t* dropped;        // per global tile: dropped by the entry budget
  uint2* ranges;           // per global tile: [start, end) in the sorted entries, or null: not wanted
  uint32_t* viewDrops;     // per view: number of dropped tiles
  uint32_t* viewTotal;     // per view: kept entries
  uint32_t* stats;         // stats[3] += dropped tiles
  uint64_t entriesCap;     // per-view entry budget (ENTCAP)
  uint32_t* totalEntries;  // out: kept entries over the batch
  uint32_t* buckets;       // out: tiles per bucket (tile_bucket), zero before
};

constexpr uint32_t EXPAND_BLOCK = 256;  // presorted items per block of k_expand

// Entry expansion of the presorted (view, depth, id) items (k_expand).
struct ExpandArgs {
  uint32_t n;
  int V;
  const DevCam* cams;
  const uint32_t* sortedSlots;  // presorted (view, depth, id) order
  const uint4* itemSrc;         // V * n * 2 by slot: (rect, mean, cull parameters, slot) from the projection
  uint4* itemRecs;              // V * n * 2: the same per presorted item
  const uint32_t* liveItems;    // presorted items kept (the culled ones left the presort)
  const uint8_t* dropped;
  const uint32_t* viewDrops;
  float eCut, aMin;
  int tile;
  int cull;                     // 1: keep only entries tileLive() accepts
  int masks;                    // 1 (tile 16): entry values carry the 8x8 block bits
  uint32_t* counts;             // entries per presorted item (count pass -> key pass)
  uint32_t* partials;           // entries per block of EXPAND_BLOCK items; scanned between the passes
  uint32_t* keys;               // global tile id per entry
  uint32_t* vals;               // entry value: splat id (and block bits)
  uint64_t capacity;
  uint32_t* status;
};

struct RadixHistArgs {
  const void* keys;        // uint32_t or uint64_t
  const uint32_t* nItems;
  uint32_t* hist;           // passes * 256
  int passes;
  uint32_t* epoch;
  uint32_t* nKept;          // non-null: all-ones keys are dropped (not counted); kept keys are counted here
};

#ifndef GS_SORT_ITEMS
#define GS_SORT_ITEMS 16  // keys per thread of a onesweep block (256 threads)
#endif
constexpr int SORT_BLOCK_ENTRIES = 256 * GS_SORT_ITEMS;  // entries one onesweep block ranks
constexpr uint32_t RS_SMALL = 256u * 1024u;              // up to here blocks of a quarter of that
// look-back words (per digit) that sorts of up to N entries use
constexpr uint64_t sort_status_blocks(uint64_t N) {
  const uint64_t big = (N + SORT_BLOCK_ENTRIES - 1) / SORT_BLOCK_ENTRIES;
  const uint64_t few = (N < RS_SMALL ? N : RS_SMALL), small = (few + SORT_BLOCK_ENTRIES / 4 - 1) / (SORT_BLOCK_ENTRIES / 4);
  return big > small ? big : small;
}

struct OnesweepArgs {
  const void* keysIn;
  const uint32_t* valsIn;
  void* keysOut;            // null: do not write keys (last pass)
  uint32_t* valsOut;
  const uint32_t* nItems;
  const uint32_t* hist;
  uint32_t* tileCounter;    // per pass
  uint64_t* status;         // look-back words, one per (block, digit)
  uint32_t* statusWord;     // error bits
  const uint32_t* epoch;
  int pass;
  uint32_t spinLimit;       // look-back spins before the block gives up and flags a timeout
  int smallBlocks;          // 1: few entries are sorted in blocks of a quarter of the size
  int dropAllOnes;          // all-ones keys leave the sort (output compacted to the kept keys);
                            // selects the kernel instantiation that drops them
};

struct RadixSortArgs {
  void* keys[2];            // ping-pong key buffers of keyBytes-wide keys
  int keyBytes;             // 4 or 8
  uint32_t* vals[2];
  const uint32_t* nItems;
  uint32_t* hist;
  uint32_t* tileCounter;
  uint64_t* status;
  uint32_t* statusWord;
  uint32_t* epoch;
  int passes;
  bool keepKeys;
  unsigned histGrid, sweepGrid;
  uint32_t* nKept;          // non-null (32-bit keys): all-ones keys are dropped in the first pass and the
                            // kept count lands here (zero before the call); later passes sort only those
  uint32_t orPasses;        // 32-bit keys, bit p: pass p ranks its digits with the OR form (digits spread
                            // across a warp: tile ids, the low bytes of depths)
};

// Entry values.  With block masks on (16-pixel tiles, at most 2^28 splats) a
// value is the splat id in the low ID_BITS bits and, above it, one bit per 8x8
// block of the tile (row-major): set when the splat may reach the block.
constexpr uint32_t ID_BITS = 28;
constexpr uint32_t ID_MASK = (1u << ID_BITS) - 1u;

constexpr int RW_WARPS = 4;                    // warps per block of k_raster_warp
// composited entries a warp caches (k_raster_warp): in an allocation of its own,
// and at most, where the memory is there anyway
constexpr uint32_t RASTER_CACHE_ENTRIES = 256, RASTER_CACHE_MAX = 1024;

// Work-order bucket of a tile: 32 empty, 0 longest.
__device__ __forceinline__ uint32_t tile_bucket(uint2 r) { return (uint32_t)__clz((int)(r.y - r.x)); }

struct RasterArgs {
  const DevCam* cams;
  int V;
  uint32_t n;
  const RenderRec* recs;   // V * n
  const float4* cullRecs;  // V * n warp-block cull parameters
  const uint32_t* ids;     // sorted entry values: splat ids under idMask, block bits above it
  uint32_t idMask;         // ID_MASK with block masks, else all ones
  const uint2* ranges;     // per global tile
  uint32_t totalTiles;
  const uint32_t* workOrder;  // null: item order
  uint32_t* workCounter;      // null: one item per block (blockIdx.x)
  float eCut, aMin;
  float4* outImg;          // per batch pixel (RGB, 1 - T)
  float* finalT;
  uint32_t* endIdx;
  const uint32_t* targets;
  int32_t* gradP;          // V * n * GP_STRIDE
  uint32_t* stats;
  int32_t* gradCam;
  float* tStore;           // stored-state variant: T before each entry, per pixel
  // k_raster_warp's exponential cache: cacheWarps slices of cacheCap + 2 entries, and one more
  uint32_t cacheCap, cacheWarps;
  float2* cacheG;          // per entry 32 lanes x 2 pixels
  uint32_t* cacheId;       // per entry the splat id
};

struct AdamHP {
  float lr[16];
  float b1, b2, eps, bc1, bc2, minLS, maxLS, maxLogit, reg, shLr;
};

// floats per (view, splat) chain result: 14 parameter gradients, gated
// colour gradient (3), view direction (3)
constexpr int VIEWGRAD_STRIDE = 20;

struct ChainArgs {
  uint32_t n;
  int V;
  const DevCam* cams;
  float* params;
  float* sh;
  int32_t* gradP;
  const uint2* rect;
  float* viewGrad;         // V * n * VIEWGRAD_STRIDE: per-(view, splat) chain results
  uint32_t* visList;       // V * n: per view, indices of the visible splats
  uint32_t* visCount;      // V counters, cleared before the step
  uint32_t chainStrips;    // strips of 128 list items per chain block (set by the launcher)
  uint32_t sms;            // of the device
  float anisoReg;
  int32_t* gradCam;
  float* gradF;            // optional readout (n * 16)
  float* shGrad;           // optional readout (n * 3K)
  int doAdam;
  const AdamHP* hp;        // device-resident (updated every step)
  float* m;
  float* v;
  float* shM;
  float* shV;
};

// refine: one spawned splat of the plan the host draws (trainer.js:713-752)
struct RefineSpawn {
  uint32_t pos;    // position in the donor list, or in the sorted big-donor list when split
  uint32_t split;  // 1: split a big donor, 0: clone a donor
  double g[3];     // the three gauss() jitters of the position
};

struct RefineApplyArgs {
  const RefineSpawn* plan;
  uint32_t count;          // moved + grown
  uint32_t moved;          // the first `moved` spawns relocate dead splats
  uint32_t n;              // splat count before growth
  const uint32_t* deadList;
  const uint32_t* donorList;
  const uint32_t* bigSorted;   // donors by mean log-scale, descending (stable)
  const uint32_t* splitSeq;    // per splat: sequence number of its split, or ~0
  float* params;
  float* m;
  float* v;
  float* sh;
  float* shM;
  float* shV;
  int shr;                 // 3K
};

// launchers
void launch_step_begin(const StepBeginArgs& a, cudaStream_t s);
void launch_project(const ProjectArgs& a, int deg, cudaStream_t s);
void launch_tile_ranges(const TileRangeArgs& a, uint32_t totalTiles, cudaStream_t s);
void launch_expand(const ExpandArgs& a, bool keys, cudaStream_t s);
void launch_ranges_from_keys(const uint32_t* keys, const uint32_t* nItems, uint32_t totalTiles, uint2* ranges,
                             uint32_t* buckets, cudaStream_t s);
void launch_scan_blocks(uint32_t* partials, const uint32_t* nItems, uint32_t perBlock, uint32_t* total, cudaStream_t s);
uint32_t scan_partials_needed(uint64_t N);
void launch_exclusive_scan(const uint32_t* in, uint64_t N, uint32_t* out, uint32_t* partials, uint32_t* total,
                           cudaStream_t s);
int onesweep_grid(int device);
// RGBA8 packing of one camera's float RGB target (host memory) into out,
// staged through scratch (3 floats per pixel) on stream s.
int pack_targets_device(const float* rgbHost, uint64_t np, float* scratch, uint32_t* out, cudaStream_t s);
int export_ply_records(const float* params, const float* sh, uint32_t n, uint32_t K, int bake, double f,
                       const double* camPosHost, uint32_t ncams, double* dCam, float* dOut, void* outHost,
                       cudaStream_t s);
int debug_lookback_timeout(int device, uint32_t spinLimit, uint32_t* statusOut, double* msOut);
void launch_radix_sort(const RadixSortArgs& a, cudaStream_t s);
void launch_raster(const RasterArgs& a, bool train, int tile, unsigned grid, cudaStream_t s);
unsigned raster_grid(uint32_t items, int sms, int perSm);
void launch_raster_stored(const RasterArgs& a, int tile, int batchDepth, unsigned grid, cudaStream_t s);
int raster_blocks_per_sm(int tile, bool train);
void launch_work_place(const uint2* ranges, uint32_t totalTiles, const uint32_t* counts, uint32_t* cursors,
                       uint32_t* order, cudaStream_t s);
void launch_chain_adam(const ChainArgs& a, int deg, cudaStream_t s);
void launch_refine_classify(const float* params, uint32_t n, uint32_t* deadFlag, uint32_t* donorFlag,
                            cudaStream_t s);
void launch_refine_compact(const float* params, uint32_t n, const uint32_t* deadFlag, const uint32_t* deadOff,
                           const uint32_t* donorFlag, const uint32_t* donorOff, uint32_t* deadList,
                           uint32_t* donorList, uint64_t* donorKeys, uint32_t* donorVals, cudaStream_t s);
void launch_refine_apply(const RefineApplyArgs& a, uint32_t* splitSeq, cudaStream_t s);
void launch_donor_opacity(const float* params, const uint32_t* donorList, uint32_t nDonors, float* out,
                          cudaStream_t s);
void launch_max_u32(const uint32_t* x, uint32_t count, uint32_t* out, cudaStream_t s);

}  // namespace gs
