// LBVH over terminal boxes: Morton keys, radix sort, and the tree (Karras's
// topology and node numbers, with the boxes) joined bottom up, in one kernel per
// tile of leaves (k_tree) and one per group of tiles (k_join).
//
// Restates ContextSensitivity::GPU::BVHConstructor::construct
// (include/pga/core/GPUBVHConstructor.cuh:44-331) for the terminal records of
// a derivation, with three changes:
//  * key = morton30 << 34 | path >> 30: equal Morton codes are ordered by the
//    derivation-path hash (ties on those 34 bits resolved on the full hash)
//    instead of the emission index, which depends on queue order;
//  * the Karras codes are morton30 << 32 | sorted position, as the reference's
//    `(code << 32) | j` with j replaced by that deterministic position;
//  * AABBs start from -FLT_MAX instead of FLT_MIN (AABB.cuh:20) and the two
//    climbers that meet at a node are ordered by an acquire-release exchange.
// The reference sorts with thrust::sort (GPUBVHConstructor.cuh:311-312); here
// the sort is this file's own radix sort (see k_sort_pass).
#include <cuda_runtime.h>

#include <cfloat>
#include <algorithm>
#include <mutex>
#include <string>

#include "engine_host.h"

namespace pga {

constexpr int kLbvhThreads = 256;

// spread / morton30 (GPUBVHConstructor.cuh:44-64).
__device__ __forceinline__ uint32_t spread(uint32_t v) {
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

// The kernels of a small build (kSmallSort) are launched with programmatic
// stream serialization: a kernel's blocks may be placed while the last ones of
// the kernel before are still running, so its launch and whatever it does
// ahead of await_previous (shared memory only) hide behind them.  Every thread
// passes await_previous before it touches global memory, which makes the whole
// chain's stores visible, as with ordinary launches.  20,011 leaves: 66 -> 55
// us.  Large builds lose by it (3.0M leaves 386 -> 418 us): the waiting blocks
// take the places of blocks with work.
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void await_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// A buffer that an earlier kernel of the chain writes, as the pointer to read
// it through after the wait: opaque to the compiler, so that no load through it
// moves ahead of the wait or becomes a read-only (non-coherent) one, which the
// buffer is not while the waiting kernel already runs.
template <typename T>
__device__ __forceinline__ const T* written(const T* p) {
  asm volatile("" : "+l"(p) : : "memory");
  return p;
}

struct Bounds {
  float mn[3];
  float sz[3];
};

// Leaf AABB: corners of the terminal box (8) or quad (4), as
// BoundingVolumeConstructor<AABB>::construct (BoundingVolumeConstructor.cuh:22-76)
// with the scale folded into the terminal matrix.  Rounding is monotone, so the
// smallest corner sum is the sum with every term negative and the largest the
// one with every term positive; where those are finite so is every corner, and
// the eight corners need not be formed.
// (One row of the box at a time and by value: a box passed by pointer would
// live in local memory for the leaves that never come here, too.)
__device__ __noinline__ float2 leaf_aabb_corners(float4 r, bool quad) {
  float mn = FLT_MAX, mx = -FLT_MAX;
  for (int cz = 0; cz < (quad ? 1 : 2); cz++)
    for (int cy = 0; cy < 2; cy++)
      for (int cx = 0; cx < 2; cx++) {
        const float x = cx ? 0.5f : -0.5f, y = cy ? 0.5f : -0.5f, z = quad ? 0.0f : (cz ? 0.5f : -0.5f);
        const float v = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(r.x, x), __fmul_rn(r.y, y)), __fmul_rn(r.z, z)), r.w);
        mn = fminf(mn, v);
        mx = fmaxf(mx, v);
      }
  return make_float2(mn, mx);
}
// One axis of the box, from the matrix's row.
__device__ __forceinline__ void leaf_extent(const float4& r, bool quad, float& mn, float& mx) {
  const float hx = fabsf(__fmul_rn(r.x, 0.5f)), hy = fabsf(__fmul_rn(r.y, 0.5f));
  const float hz = fabsf(__fmul_rn(r.z, quad ? 0.0f : 0.5f));
  const float h = __fadd_rn(__fadd_rn(hx, hy), hz);
  mn = __fsub_rn(r.w, h);
  mx = __fadd_rn(r.w, h);
  if (!(fabsf(mn) < FLT_MAX && fabsf(mx) < FLT_MAX)) {
    const float2 c = leaf_aabb_corners(r, quad);
    mn = c.x;
    mx = c.y;
  }
}
__device__ __forceinline__ void leaf_aabb(const float4 r[3], bool quad, float mn[3], float mx[3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) leaf_extent(r[k], quad, mn[k], mx[k]);
}

// Leaf count of a build: the host value `n`, or, when the count lives on the
// device (dN != nullptr), min(*dN, n) with `n` the capacity the launches and
// the sort were sized for.
__device__ __forceinline__ unsigned long long leaf_count(const unsigned long long* dN, unsigned long long n) {
  return dN ? min(*dN, n) : n;
}

// The radix sort orders the leaves by Morton code (30 bits) and, below it, by
// the path hash's top 10 bits: four passes of 10-bit digits.  The first takes
// its digit from the hash (an array of its own, read by that pass only); after
// it a leaf is its code and its terminal index, 8 bytes a pass each way.  The
// full keys (Morton code << 34 | path hash >> 30) are formed by the tree
// kernel, which gathers the records anyway.
constexpr int kRadixBits = 10;
constexpr uint32_t kBins = 1u << kRadixBits;
constexpr int kSortPasses = 4;
constexpr int kHashShift = 54;  // path >> kHashShift: the hash digit
static_assert(30 == (kSortPasses - 1) * kRadixBits && 64 - kHashShift == kRadixBits, "the passes cover code and hash");

__device__ __forceinline__ uint32_t code_digit(uint32_t code, int q) {  // pass q = 1 .. 3
  return (code >> ((q - 1) * kRadixBits)) & (kBins - 1u);
}

// Histogram of one digit of a warp's 32 keys into shared memory: one add for
// the whole warp when every lane has the same digit (the Morton code's high
// digits, for neighbouring terminals), else one add per lane.
__device__ __forceinline__ void hist_add(uint32_t* h, uint32_t d, bool valid) {
  const uint32_t d0 = __shfl_sync(0xFFFFFFFFu, d, 0);
  const unsigned same = __ballot_sync(0xFFFFFFFFu, valid && d == d0);
  if (same == 0xFFFFFFFFu) {
    if ((threadIdx.x & 31u) == 0) atomicAdd(h + d0, 32u);
  } else if (valid) {
    atomicAdd(h + d, 1u);
  }
}
__device__ __forceinline__ void hist_leaf(uint32_t* sh, uint32_t code, uint32_t hash, bool valid) {
  hist_add(sh, hash, valid);
#pragma unroll
  for (int q = 1; q < kSortPasses; q++) hist_add(sh + q * kBins, code_digit(code, q), valid);
}

// generateMortonCodes (GPUBVHConstructor.cuh:66-86) on terminal centres, and
// the hash digits.  The sort's values start as the terminal index, which its
// first pass generates, so none are written here.
// With a device count, the entries in [count, capacity) are padding: all ones,
// after every real one in the stable radix sort.
// HIST: also counts the digits, for the small builds' sort (the large ones
// count them pass by pass).
constexpr int kHistThreads = 512;
template <bool HIST>
__global__ void __launch_bounds__(HIST ? kHistThreads : kLbvhThreads)
    k_morton(const PgaTerminal* __restrict__ t, unsigned long long cap, const unsigned long long* __restrict__ dN,
             Bounds b, uint32_t* __restrict__ codes, uint16_t* __restrict__ hashes, uint32_t* __restrict__ hist) {
  __shared__ uint32_t sh[HIST ? kSortPasses * kBins : 1];
  allow_next();
  if (HIST) {
    for (uint32_t k = threadIdx.x; k < kSortPasses * kBins; k += kHistThreads) sh[k] = 0u;
    __syncthreads();
  }
  const unsigned long long n = leaf_count(dN, cap);
  const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t code = ~0u, hash = kBins - 1u;
  if (i < n) {
    const float c[3] = {__ldg(&t[i].m[3]), __ldg(&t[i].m[7]), __ldg(&t[i].m[11])};
    hash = __ldg(reinterpret_cast<const uint32_t*>(&t[i].path) + 1) >> (kHashShift - 32);
    code = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      float nc = __fdiv_rn(__fsub_rn(c[k], b.mn[k]), b.sz[k]);
      code |= spread(__float2uint_rz(__fmul_rn(nc, 1023.0f))) << k;
    }
  }
  if (i < cap) {
    codes[i] = code;
    hashes[i] = (uint16_t)hash;
  }
  if (HIST) {
    hist_leaf(sh, code, hash, i < cap);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < kSortPasses * kBins; k += kHistThreads)
      if (sh[k] != 0u) atomicAdd(hist + k, sh[k]);
  }
}

// One pass of the radix sort, stable: entries [0, n) ordered by their digit.
// FIRST: the digit is the hash and the value the index; else the digit is
// code >> shift.
// A block takes a tile of 512 x ITEMS entries.  Its warps rank their entries by
// digit in input order (warp-private 16-bit histograms) and the tile goes to
// shared memory in digit order; thread t owns bins 2t and 2t + 1.  Entries then go out in
// contiguous runs per digit, to the digit's start (a scan of the pass's digit
// counts, made with the tile's own) plus the digit's count in the earlier
// tiles.  Where that count comes from is the difference between two forms:
//
// * Up to kSmallSort leaves (or capacity, where the count is on the device), that
//   is while every tile has a block of its own on the chip at once:
//   one launch a pass ("onesweep", Adinets & Merrill 2022).  A block takes the
//   next tile from an atomic counter, so a tile's predecessors were taken by
//   blocks that started earlier, publishes its bins' counts as one 64-bit word
//   (each half carries the flag) and looks back over the earlier tiles' words
//   until one carries an inclusive prefix.  A wait gives up after spinLimit
//   polls, raising PGA_ERR_TIMEOUT in *err (the order is then unspecified).
//   ITEMS = 4: few serial ranking rounds, a pass takes as long as one tile.
//   Lanes sharing a digit are found through a mask per digit in which each sets
//   its bit (20,011 leaves: 5.9 us a pass, 6.9 with ballots).
// * Larger builds: k_sort_count and k_sort_scan before the pass (COUNTED).
//   With hundreds of tiles in flight the look-back takes eight steps of 16
//   words and 0.7 us each, most of a tile's instructions; a count reads 4 bytes
//   an entry, which mostly hit L2, and its scan 4 KB a tile.  City of 5.9M
//   leaves: four passes took 281 us with the look-back and the histograms that
//   it needs, 224 with the counts.  Lanes sharing a digit are found with a
//   ballot per digit bit: the masks' atomics collide where many neighbours
//   share one (19M leaves of the mixed batch: 152 us a pass, ballots 141).
//
// Whole builds at either side of kSmallSort (records spread over the bounds; the
// city's are within 5%), the first form and the second: 100,000 leaves 71 and 135
// us, 300,000 106 and 149, 600,000 142 and 164; 650,000 153 and 166, 800,000 176
// and 172, 1,000,000 202 and 182.  The two cross near 750,000, past the line.
constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSmallItems = 4, kLargeItems = 16;
constexpr unsigned long long kSmallSort = 304ull * kSortThreads * kSmallItems;  // two blocks on each of 152 SMs
constexpr uint32_t kHistStride = kBins + 16;  // u16 per warp histogram (padded: the warps' rows start in other banks)
constexpr uint32_t kFlagAggregate = 1u << 30, kFlagPrefix = 2u << 30, kCountMask = (1u << 30) - 1u;
constexpr int kLookback = 16;  // predecessor words loaded at once by a look-back step
static_assert(kBins == 2 * kSortThreads, "each thread owns two bins");
// The tile's entries, and before them the warps' digit masks in their place.
__host__ __device__ constexpr size_t sort_entry_bytes(int items) {
  const size_t entries = (size_t)kSortThreads * items * 8;
  const size_t masks = items == kSmallItems ? (size_t)kSortWarps * kBins * 4 : 0;
  return entries > masks ? entries : masks;
}
constexpr size_t sort_pass_smem(int items) {
  return sort_entry_bytes(items) + (size_t)kSortWarps * kHistStride * 2 + (size_t)kBins * 8;
}

__device__ __forceinline__ void st_relaxed64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long pair_word(uint32_t flag, uint32_t c0, uint32_t c1) {
  return ((unsigned long long)(flag | c1) << 32) | (flag | c0);
}

// The counted form.  Group g of kSortGroups blocks counts a contiguous run of
// tiles: rows[tile][bin] gets the bin's count in the group's earlier tiles,
// groups[g][bin] the group's total.
constexpr uint32_t kSortGroups = 304;  // two blocks on each of 152 SMs
template <bool FIRST>
__global__ void __launch_bounds__(kSortThreads) k_sort_count(const uint32_t* codes, const uint16_t* hashes,
                                                             unsigned long long n, uint32_t shift, uint32_t tiles,
                                                             uint32_t perGroup, uint32_t* rows, uint32_t* groups) {
  constexpr uint32_t kTileItems = kSortThreads * kLargeItems;
  __shared__ uint32_t sh[kBins];
  const uint32_t first = blockIdx.x * perGroup, last = min(tiles, first + perGroup);
  uint2* bins = reinterpret_cast<uint2*>(sh) + threadIdx.x;
  uint2 run = make_uint2(0u, 0u);
  *bins = run;
  __syncthreads();
  for (uint32_t tile = first; tile < last; tile++) {
    const unsigned long long base = (unsigned long long)tile * kTileItems;
    const uint32_t count = (uint32_t)min((unsigned long long)kTileItems, n - base);
    uint32_t d[kLargeItems];
#pragma unroll
    for (int k = 0; k < kLargeItems / 4; k++) {
      const uint32_t x = (k * kSortThreads + threadIdx.x) * 4u;
      if (x + 4 <= count) {
        if (FIRST) {
          const ushort4 h = *reinterpret_cast<const ushort4*>(hashes + base + x);
          d[k * 4 + 0] = h.x; d[k * 4 + 1] = h.y; d[k * 4 + 2] = h.z; d[k * 4 + 3] = h.w;
        } else {
          const uint4 c = *reinterpret_cast<const uint4*>(codes + base + x);
          d[k * 4 + 0] = c.x; d[k * 4 + 1] = c.y; d[k * 4 + 2] = c.z; d[k * 4 + 3] = c.w;
        }
      } else {
#pragma unroll
        for (int u = 0; u < 4; u++)
          d[k * 4 + u] = x + u < count ? (FIRST ? (uint32_t)hashes[base + x + u] : codes[base + x + u]) : 0u;
      }
    }
#pragma unroll
    for (int k = 0; k < kLargeItems; k++) {
      const bool valid = ((k / 4) * kSortThreads + threadIdx.x) * 4u + (k & 3) < count;
      hist_add(sh, FIRST ? d[k] : (d[k] >> shift) & (kBins - 1u), valid);
    }
    __syncthreads();
    const uint2 c = *bins;
    *bins = make_uint2(0u, 0u);
    reinterpret_cast<uint2*>(rows + (size_t)tile * kBins)[threadIdx.x] = run;
    run.x += c.x;
    run.y += c.y;
    __syncthreads();
  }
  reinterpret_cast<uint2*>(groups + (size_t)blockIdx.x * kBins)[threadIdx.x] = run;
}

// groups[g][bin] becomes the bin's count in the groups before g, totals[bin]
// its count in all.  A block of 32 x 32 threads per 32 bins: lane = bin, each
// warp a run of ten groups.
__global__ void __launch_bounds__(1024) k_sort_scan(uint32_t* groups, uint32_t* totals) {
  constexpr uint32_t kPer = (kSortGroups + 31) / 32;
  __shared__ uint32_t sSum[32][33];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t* col = groups + blockIdx.x * 32u + lane;
  uint32_t v[kPer], sum = 0;
#pragma unroll
  for (uint32_t k = 0; k < kPer; k++) {
    const uint32_t g = warp * kPer + k;
    v[k] = g < kSortGroups ? col[(size_t)g * kBins] : 0u;
  }
#pragma unroll
  for (uint32_t k = 0; k < kPer; k++) sum += v[k];
  sSum[warp][lane] = sum;
  __syncthreads();
  uint32_t before = 0;
  for (uint32_t w = 0; w < warp; w++) before += sSum[w][lane];
#pragma unroll
  for (uint32_t k = 0; k < kPer; k++) {
    const uint32_t g = warp * kPer + k;
    if (g < kSortGroups) col[(size_t)g * kBins] = before;
    before += v[k];
  }
  if (warp == 31) totals[blockIdx.x * 32u + lane] = before;
}

struct SortPass {
  const uint32_t* codesIn;
  const uint16_t* hashes;
  const uint32_t* valsIn;
  uint32_t* codesOut;
  uint32_t* valsOut;
  unsigned long long n;
  uint32_t shift;
  const uint32_t* hist;  // the pass's digit counts
  // the look-back's words and the tiles' counter
  unsigned long long* status;
  uint32_t* tileCounter;
  int* err;
  uint32_t spinLimit;
  // COUNTED: the rows of k_sort_count and the groups of k_sort_scan (perGroup tiles each)
  const uint32_t* rows;
  const uint32_t* groups;
  uint32_t perGroup;
};

// One tile; FULL: all of its entries exist (every tile but the last).
template <int ITEMS, bool FIRST, bool COUNTED, bool FULL>
__device__ __forceinline__ void sort_tile(const SortPass& a, uint32_t tile, uint32_t count, uint2 all) {
  constexpr uint32_t kTileItems = kSortThreads * ITEMS;
  constexpr bool kMasks = !COUNTED;
  static_assert(kTileItems <= 1u << 16, "ranks and tile-local indexes of 16 bits");
  extern __shared__ __align__(16) unsigned char smem_sort[];
  uint32_t* sCodes = reinterpret_cast<uint32_t*>(smem_sort);
  uint32_t* sVals = sCodes + kTileItems;  // FIRST: digit << 16 | index in the tile
  uint16_t* sHist = reinterpret_cast<uint16_t*>(smem_sort + sort_entry_bytes(ITEMS));
  uint32_t* sStart = reinterpret_cast<uint32_t*>(sHist + kSortWarps * kHistStride);
  int32_t* sDst = reinterpret_cast<int32_t*>(sStart + kBins);
  __shared__ unsigned long long sWarpSum[kSortWarps];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint16_t* mine = sHist + warp * kHistStride;
  uint32_t* match = sCodes + warp * kBins;  // while the warps rank: per digit the lanes that have it
  const unsigned long long tileBase = (unsigned long long)tile * kTileItems;
  const uint32_t* codesIn = a.codesIn + tileBase;
  const uint32_t shift = a.shift;
  const uint32_t local = warp * (32u * ITEMS) + lane;  // + 32 k: this thread's entries in the tile
  unsigned lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  uint32_t code[ITEMS];
  uint32_t digit[ITEMS];  // FIRST only; then digit << 16 | rank
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const uint32_t x = local + 32u * k;
    code[k] = FULL || x < count ? __ldcs(codesIn + x) : 0u;
    digit[k] = FIRST && (FULL || x < count) ? (uint32_t)__ldcs(a.hashes + tileBase + x) : 0u;
  }
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const bool valid = FULL || local + 32u * k < count;
    const uint32_t d = FIRST ? digit[k] : (code[k] >> shift) & (kBins - 1u);
    unsigned peers;  // the lanes with the same digit
    if (kMasks) {    // each sets its bit in the digit's mask
      if (valid) atomicOr(match + d, 1u << lane);
      __syncwarp();
      peers = valid ? match[d] : 1u << lane;
      __syncwarp();
    } else {  // one ballot per digit bit
      peers = FULL ? 0xFFFFFFFFu : __ballot_sync(0xFFFFFFFFu, valid);
      if (!valid) peers = ~peers;
#pragma unroll
      for (int bit = 0; bit < kRadixBits; bit++) {
        const unsigned on = __ballot_sync(0xFFFFFFFFu, (d >> bit) & 1u);
        peers &= ((d >> bit) & 1u) ? on : ~on;
      }
    }
    const int leader = 31 - __clz((int)peers);
    uint32_t old = 0;
    if ((int)lane == leader && valid) {
      old = mine[d];
      mine[d] = (uint16_t)(old + __popc(peers));
      if (kMasks) match[d] = 0u;
    }
    old = __shfl_sync(0xFFFFFFFFu, old, leader);
    digit[k] = (d << 16) | (old + __popc(peers & lt));
    __syncwarp();  // the leader's stores, before the next turn's accesses to the same words by other lanes
  }
  __syncthreads();
  // Thread t owns bins 2t and 2t + 1: the warps' exclusive prefixes in place,
  // the tile's count of each bin, published for the later tiles.
  uint32_t tot[2] = {0u, 0u};
#pragma unroll
  for (int w = 0; w < kSortWarps; w++) {
    uint32_t* h = reinterpret_cast<uint32_t*>(sHist + w * kHistStride) + threadIdx.x;
    const uint32_t c = *h;
    *h = tot[0] | (tot[1] << 16);
    tot[0] += c & 0xFFFFu;
    tot[1] += c >> 16;
  }
  unsigned long long* st = a.status + (size_t)tile * (kBins / 2) + threadIdx.x;
  if (!COUNTED) st_relaxed64(st, pair_word(tile == 0 ? kFlagPrefix : kFlagAggregate, tot[0], tot[1]));
  // Exclusive scans over the bins: the tile's bin starts (low half) and the
  // whole input's (high half).
  uint32_t base0, base1;
  {
    const unsigned long long v = ((unsigned long long)(all.x + all.y) << 32) | (tot[0] + tot[1]);
    unsigned long long x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, x, d);
      if (lane >= (uint32_t)d) x += y;
    }
    if (lane == 31) sWarpSum[warp] = x;
    __syncthreads();
    unsigned long long before = x - v;
    for (uint32_t w = 0; w < warp; w++) before += sWarpSum[w];
    sStart[2u * threadIdx.x] = (uint32_t)before;
    sStart[2u * threadIdx.x + 1] = (uint32_t)before + tot[0];
    base0 = (uint32_t)(before >> 32);
    base1 = base0 + all.x;
  }
  __syncthreads();
  // Both bins' counts over the earlier tiles: counted before, or (below) by
  // decoupled look-back.
  uint32_t prefix0 = 0, prefix1 = 0;
  if (COUNTED) {
    const uint2 r = reinterpret_cast<const uint2*>(a.rows + (size_t)tile * kBins)[threadIdx.x];
    const uint2 g = reinterpret_cast<const uint2*>(a.groups + (size_t)(tile / a.perGroup) * kBins)[threadIdx.x];
    prefix0 = r.x + g.x;
    prefix1 = r.y + g.y;
  }
  // The tile in digit order in shared memory (before the look-back: it needs
  // only the tile's own counts).
  uint32_t val[ITEMS];
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const uint32_t x = local + 32u * k;
    if (FIRST) val[k] = (digit[k] & 0xFFFF0000u) | x;
    else val[k] = FULL || x < count ? __ldcs(a.valsIn + tileBase + x) : 0u;
  }
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    if (FULL || local + 32u * k < count) {
      const uint32_t d = digit[k] >> 16;
      const uint32_t pos = sStart[d] + mine[d] + (digit[k] & 0xFFFFu);
      sCodes[pos] = code[k];
      sVals[pos] = val[k];
    }
  }
  // The look-back.  The words of kLookback predecessors are loaded at once
  // (independent loads), then summed nearest first up to the first inclusive
  // prefix; a word not yet published stops the sum there and is polled again.
  if (!COUNTED && tile > 0) {
    long long p = (long long)tile - 1;
    uint32_t spins = 0;
    while (p >= 0) {
      unsigned long long w[kLookback];
#pragma unroll
      for (int k = 0; k < kLookback; k++)
        w[k] = p - k >= 0 ? ld_relaxed64(a.status + (size_t)(p - k) * (kBins / 2) + threadIdx.x)
                          : pair_word(kFlagPrefix, 0u, 0u);
      int used = 0;
      bool done = false, stalled = false;
#pragma unroll
      for (int k = 0; k < kLookback; k++) {
        if (done || stalled) continue;
        const uint32_t lo = (uint32_t)w[k], hi = (uint32_t)(w[k] >> 32);
        if ((lo >> 30) == 0u) {
          stalled = true;
          continue;
        }
        prefix0 += lo & kCountMask;
        prefix1 += hi & kCountMask;
        used++;
        if ((lo & kFlagPrefix) != 0u) done = true;
      }
      if (done) break;
      p -= used;
      if (stalled) {
        if (++spins > a.spinLimit) {
          atomicCAS(a.err, 0, (int)PGA_ERR_TIMEOUT);
          break;
        }
        __nanosleep(32);
      }
    }
    st_relaxed64(st, pair_word(kFlagPrefix, prefix0 + tot[0], prefix1 + tot[1]));
  }
  sDst[2u * threadIdx.x] = (int32_t)(base0 + prefix0 - sStart[2u * threadIdx.x]);
  sDst[2u * threadIdx.x + 1] = (int32_t)(base1 + prefix1 - sStart[2u * threadIdx.x + 1]);
  __syncthreads();
  // Out: consecutive positions of one digit go to consecutive places.
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const uint32_t p = threadIdx.x + (uint32_t)k * kSortThreads;
    if (!FULL && p >= count) break;
    const uint32_t c = sCodes[p], v = sVals[p];
    const uint32_t d = FIRST ? v >> 16 : (c >> shift) & (kBins - 1u);
    const uint32_t o = (uint32_t)sDst[d] + p;
    if (!COUNTED && o >= a.n) continue;  // only after a look-back that gave up
    a.codesOut[o] = c;
    a.valsOut[o] = FIRST ? (uint32_t)tileBase + (v & 0xFFFFu) : v;
  }
}

template <int ITEMS, bool FIRST, bool COUNTED>
__global__ void __launch_bounds__(kSortThreads, 2) k_sort_pass(SortPass a) {
  constexpr uint32_t kTileItems = kSortThreads * ITEMS;
  extern __shared__ __align__(16) unsigned char smem_sort[];
  __shared__ uint32_t sTile;
  if (!COUNTED) allow_next();
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint16_t* mine = reinterpret_cast<uint16_t*>(smem_sort + sort_entry_bytes(ITEMS)) + warp * kHistStride;
  for (uint32_t k = lane; k < kBins / 8; k += 32) reinterpret_cast<uint4*>(mine)[k] = make_uint4(0u, 0u, 0u, 0u);
  if (!COUNTED) {
    uint32_t* match = reinterpret_cast<uint32_t*>(smem_sort) + warp * kBins;
    for (uint32_t k = lane; k < kBins / 4; k += 32) reinterpret_cast<uint4*>(match)[k] = make_uint4(0u, 0u, 0u, 0u);
  }
  if (!COUNTED) {
    await_previous();
    a.codesIn = written(a.codesIn);
    a.hashes = written(a.hashes);
    a.valsIn = written(a.valsIn);
    a.hist = written(a.hist);
  }
  const uint2 all = reinterpret_cast<const uint2*>(a.hist)[threadIdx.x];  // this thread's bins, whole input
  if (!COUNTED) {
    if (threadIdx.x == 0) sTile = atomicAdd(a.tileCounter, 1u);
    __syncthreads();
  } else {
    __syncwarp();  // the warp's histogram is clear
  }
  const uint32_t tile = COUNTED ? blockIdx.x : sTile;
  const uint32_t count =
      (uint32_t)min((unsigned long long)kTileItems, a.n - (unsigned long long)tile * kTileItems);
  if (count == kTileItems) sort_tile<ITEMS, FIRST, COUNTED, true>(a, tile, count, all);
  else sort_tile<ITEMS, FIRST, COUNTED, false>(a, tile, count, all);
}

__device__ __forceinline__ uint64_t term_path(const PgaTerminal* t, uint32_t i) {
  const uint2 v = __ldg(reinterpret_cast<const uint2*>(&t[i].path));
  return ((uint64_t)v.y << 32) | v.x;
}

// ------------------------------------------------------------------ the tree
//
// buildRadixTree and propagateBVH (GPUBVHConstructor.cuh:88-261) in one
// bottom-up kernel and the k_join after it.  A block takes kTile consecutive sorted leaves, puts the
// leaves of equal sorted bits in their final order, gathers the leaves'
// records and joins neighbouring subtrees in shared memory: subtree [l, r] is
// joined across its boundary with the longer common prefix (the agglomerative
// construction of Apetrei, 2014), the second of the two climbers that reach a
// boundary goes on.  A joined node has the index Karras gives it: its right
// end when it is a left child, its left end otherwise.  Subtrees whose parent
// reaches past the tile stay open (one for every node that crosses the tile's
// ends: about a dozen, at most kMaxOpen) and are left to k_join, which joins
// those of kGroup tiles at a time, then of kGroup groups, up to the root.
//
// This replaces four kernels (tie ranks, Karras's searches, and a refit in
// two).  They were bound by latency: dependent probes per node, and climbs to
// the root through counters at GPU scope; and they moved each leaf's box
// through memory three times and each node's links twice.  Here a leaf costs
// its key, value and record read once (76 bytes) and the results written once
// (52 bytes).  Measured with k_join: 51 -> 21 us at 20,011 leaves, 251 -> 148
// us at 3.0M, 421 -> 287 us for the city's 5.9M, of which 110 us are the bytes
// at the copy rate and the rest the climb (93 us) and its barriers.  Tile of
// 256: a climb in it is eight to fifteen steps, and six blocks of it fit on an
// SM (five 276 us, eight, with spills, 321 us on the city; six 264), so that
// the gathers and climbs of different tiles overlap.  Groups of 32: two levels
// of joining for a million leaves, three for 268M.

constexpr uint32_t kTile = kLbvhThreads;  // leaves per block
constexpr uint32_t kGroup = 32;           // tiles, then groups, joined by the last to finish
constexpr uint32_t kHalo = 32;            // keys either side of a tile that its tie runs may reach into
// A tile's open subtrees hang off the two paths from its end leaves up to the
// tile's topmost crossing node, at most one on each level of a path; the
// codes have 30 Morton and 30 position bits.
constexpr uint32_t kMaxOpen = 128;
constexpr uint32_t kJoin = 512;  // open subtrees joined at once

struct __align__(16) OpenTree {
  float box[6];
  uint32_t left;  // first leaf (the next open subtree's is this one's end)
  int32_t delta;  // common prefix of the codes at left - 1 and left; -1 at the first leaf
};
static_assert(sizeof(OpenTree) == 32, "two 16-byte words");

struct TreeArgs {
  const uint32_t* codes;  // Morton codes, sorted (and below them by the hash digit)
  const uint32_t* vals;
  const PgaTerminal* t;
  unsigned long long cap;
  const unsigned long long* dN;
  int32_t* nodes;
  uint32_t* leafParents;
  float* aabbs;
  uint32_t* leafTerminal;
  unsigned long long* outKeys;
  OpenTree* open;       // kMaxOpen per tile
  uint32_t* openCount;  // per tile
  uint32_t* joins;      // arrivals per group, level after level (zero before the launch)
};

// Common prefix of the codes at positions j - 1 and j: Morton code, then
// position (`(code << 32) | j`, GPUBVHConstructor.cuh:85).
__device__ __forceinline__ int boundary_delta(uint32_t c0, uint32_t c1, uint32_t j) {
  const uint32_t x = c0 ^ c1;
  return x != 0u ? __clz(x) : 32 + __clz((j - 1u) ^ j);
}

__device__ __forceinline__ void load_box(const float* p, float mn[3], float mx[3]) {
  const float2* q = reinterpret_cast<const float2*>(p);
  const float2 a = q[0], b = q[1], c = q[2];
  mn[0] = a.x; mn[1] = a.y; mn[2] = b.x; mx[0] = b.y; mx[1] = c.x; mx[2] = c.y;
}
__device__ __forceinline__ void store_box(float* p, const float mn[3], const float mx[3]) {
  float2* o = reinterpret_cast<float2*>(p);
  o[0] = make_float2(mn[0], mn[1]);
  o[1] = make_float2(mn[2], mx[0]);
  o[2] = make_float2(mx[1], mx[2]);
}

// A tile's forest in shared memory: leaves in order, delta[e] the common
// prefix at leaf e's left boundary (delta[count]: at the tile's right end).
struct Forest {
  float* box;      // per leaf; an open subtree's box ends up at its first leaf
  float* nodeBox;  // per joined node, at its right end (left child) or left end
  uint32_t* flag;  // per boundary (e, e + 1): the far end + 1 of a climber that waits for its sibling
  const signed char* delta;
  uint32_t* open;  // bit per leaf: an open subtree starts here
};

// Climbs with subtree [l, r] (box mn, mx) for at most `steps` joins.  Returns
// true when it made them all and can go on from the [l, r] it leaves, false
// when it is done: its sibling's climber goes on, its parent reaches past the
// forest, or it made the root.  links: parent, left, right of the node with
// index base + e; leafUp: the parent of leaf base + e.
__device__ __forceinline__ bool climb(const Forest& f, int& l, int& r, float mn[3], float mx[3],
                                      int steps, int count, uint32_t base, int32_t* links, uint32_t* leafUp) {
  for (int step = 0; step < steps; step++) {
    const bool up = f.delta[r + 1] > f.delta[l];  // [l, r] is its parent's left child
    const int s = up ? r : l - 1;                 // the parent joins at boundary (s, s + 1)
    if (s < 0 || s + 1 >= count) {
      store_box(f.box + l * 6, mn, mx);
      atomicOr(f.open + (l >> 5), 1u << (l & 31));
      return false;
    }
    uint32_t old;
    asm volatile("atom.acq_rel.cta.shared::cta.exch.b32 %0, [%1], %2;"
                 : "=r"(old)
                 : "r"((uint32_t)__cvta_generic_to_shared(f.flag + s)), "r"((uint32_t)(up ? l : r) + 1u)
                 : "memory");
    if (old == 0u) return false;  // the sibling's climber goes on
    f.flag[s] = 0u;
    const int far = (int)old - 1;
    const int sib = up ? s + 1 : s;
    float smn[3], smx[3];
    load_box((far == sib ? f.box : f.nodeBox) + sib * 6, smn, smx);
    const bool leftOne = (up ? l : far) == s, rightOne = (up ? far : r) == s + 1;  // single entries
    l = up ? l : far;
    r = up ? far : r;
    // the union in (left, right) order
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const float lmn = up ? mn[k] : smn[k], rmn = up ? smn[k] : mn[k];
      const float lmx = up ? mx[k] : smx[k], rmx = up ? smx[k] : mx[k];
      mn[k] = fminf(lmn, rmn);
      mx[k] = fmaxf(lmx, rmx);
    }
    const int dl = f.delta[l], dr = f.delta[r + 1];
    const int at = dr > dl ? r : l;
    store_box(f.nodeBox + at * 6, mn, mx);
    const int32_t gs = (int32_t)base + s, id = (int32_t)base + at;
    links[at * 3 + 1] = leftOne ? gs : -gs;
    links[at * 3 + 2] = rightOne ? gs + 1 : -(gs + 1);
    *(leftOne ? reinterpret_cast<int32_t*>(leafUp) + s : links + s * 3) = id;
    *(rightOne ? reinterpret_cast<int32_t*>(leafUp) + s + 1 : links + (s + 1) * 3) = id;
    if (dl < 0 && dr < 0) {
      links[0] = -1;
      return false;
    }
  }
  return true;
}

// After the climbs: a climber still waiting at boundary (s, s + 1) has a
// sibling that stayed open, so its subtree ([far, s], or [s + 1, far]) is open
// too.  The whole block, between barriers.
__device__ __forceinline__ void open_waiting(const Forest& f, int count) {
  for (int s = (int)threadIdx.x; s + 1 < count; s += (int)kTile) {
    const uint32_t w = f.flag[s];
    if (w == 0u) continue;
    const int far = (int)w - 1;
    const int l = far <= s ? far : s + 1;
    if (far != (far <= s ? s : s + 1)) {  // a joined node: its box to its first entry
      float mn[3], mx[3];
      load_box(f.nodeBox + (far <= s ? s : s + 1) * 6, mn, mx);
      store_box(f.box + l * 6, mn, mx);
    }
    atomicOr(f.open + (l >> 5), 1u << (l & 31));
  }
}

// Rank of entry e among the open subtrees (bits below e) and their number.
__device__ __forceinline__ uint32_t open_rank(const uint32_t* open, int e) {
  uint32_t n = __popc(open[e >> 5] & ((1u << (e & 31)) - 1u));
  for (int w = 0; w < (e >> 5); w++) n += __popc(open[w]);
  return n;
}

// The terminal index at sorted position i (bounded by the leaf count, should a
// look-back wait of the sort have given up and left old contents).
__device__ __forceinline__ uint32_t leaf_value(const TreeArgs& a, unsigned long long i, unsigned long long n) {
  return min(*(a.vals + i), (uint32_t)n - 1u);
}

// The leaves' final order.  The radix sort orders the Morton code and the path
// hash's top 10 bits only and leaves runs of equal ones in input order; inside
// a run the order is by the full path hash, then by terminal index: what a
// full 64-bit sort with a path tie fix gives.  Most runs are short: a tile's
// threads see the tile's paths and those of kHalo leaves either side in shared
// memory (window position q is leaf base - kHalo + q), and each member of a
// run counts the members before it.  A run that reaches past the window is
// ordered by the whole block (tie_select).
struct TieWindow {
  uint64_t path[kTile + 2 * kHalo];
  uint32_t val[kTile + 2 * kHalo];
};
constexpr int kWindowWords = (int)(kTile + 2 * kHalo) / 32;

// The run around window position q: its first and last position.  eq holds a
// bit per position: equal to the left neighbour (bit 0 of the window clear
// unless the run goes on to the left of it).
__device__ __forceinline__ void tie_run(const uint32_t* eq, int q, int& s, int& e) {
  int w = q >> 5;
  uint32_t m = ~eq[w] & (0xFFFFFFFFu >> (31 - (q & 31)));
  while (m == 0u && w > 0) m = ~eq[--w];
  s = m != 0u ? w * 32 + 31 - __clz(m) : 0;
  w = (q + 1) >> 5;
  if (w >= kWindowWords) {
    e = q;
    return;
  }
  m = ~eq[w] & (0xFFFFFFFFu << ((q + 1) & 31));
  while (m == 0u && w + 1 < kWindowWords) m = ~eq[++w];
  e = m != 0u ? w * 32 + __ffs(m) - 2 : kWindowWords * 32 - 1;
}

// What the sort ordered at position i: Morton code, then hash digit.
__device__ __forceinline__ uint64_t tie_key(const TreeArgs& a, unsigned long long n, unsigned long long i) {
  return ((uint64_t)*(a.codes + i) << kRadixBits) | (term_path(a.t, leaf_value(a, i, n)) >> kHashShift);
}

// Whether the leaf at position i has code c and hash digit h; its value and
// path when the code agrees.
__device__ __forceinline__ bool tie_leaf(const TreeArgs& a, unsigned long long n, unsigned long long i, uint32_t c,
                                         uint32_t h, uint32_t& val, uint64_t& path) {
  if (*(a.codes + i) != c) return false;
  val = leaf_value(a, i, n);
  path = term_path(a.t, val);
  return (uint32_t)(path >> kHashShift) == h;
}

// (path, value) number `rank` in order among those of sorted positions
// [lo, hi): a radix select by the whole block, 8 bits a round from the top
// (digits: 256 words of shared memory).
__device__ __noinline__ void tie_select(const TreeArgs& a, unsigned long long n, unsigned long long lo, unsigned long long hi,
                                        unsigned long long rank, uint32_t* digits, uint64_t& path, uint32_t& val) {
  __shared__ uint32_t sDigit, sBefore;
  uint64_t p = 0;
  uint32_t v = 0;
  for (int round = 0; round < 12; round++) {
    for (uint32_t k = threadIdx.x; k < 256u; k += kTile) digits[k] = 0u;
    __syncthreads();
    const int shift = round < 8 ? 56 - 8 * round : 24 - 8 * (round - 8);
    for (unsigned long long i = lo + threadIdx.x; i < hi; i += kTile) {
      const uint32_t vi = leaf_value(a, i, n);
      const uint64_t pi = term_path(a.t, vi);
      if (round < 8) {
        if (round == 0 || (pi >> (shift + 8)) == (p >> (shift + 8))) atomicAdd(digits + ((pi >> shift) & 255u), 1u);
      } else if (pi == p && (round == 8 || (vi >> (shift + 8)) == (v >> (shift + 8)))) {
        atomicAdd(digits + ((vi >> shift) & 255u), 1u);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t before = 0, d = 0;
      while (d < 255u && before + digits[d] <= rank) before += digits[d++];
      sDigit = d;
      sBefore = before;
    }
    __syncthreads();
    rank -= sBefore;
    if (round < 8) p |= (uint64_t)sDigit << shift;
    else v |= sDigit << shift;
  }
  path = p;
  val = v;
}

__device__ __forceinline__ void gather_leaf(const PgaTerminal* t, uint32_t v, float mn[3], float mx[3],
                                            uint64_t& path) {
  const float4* p = reinterpret_cast<const float4*>(t + v);
  const float4 r[3] = {__ldg(p + 0), __ldg(p + 1), __ldg(p + 2)};
  const uint4 meta = __ldg(reinterpret_cast<const uint4*>(p + 3));
  leaf_aabb(r, (meta.x >> 31) != 0, mn, mx);
  path = ((uint64_t)meta.w << 32) | meta.z;
}

__global__ void __launch_bounds__(kTile, 6) k_tree(TreeArgs a) {
  constexpr unsigned kAll = 0xFFFFFFFFu;
  __shared__ __align__(16) float sBox[kTile * 6];
  // the joined nodes' boxes; before the climb, the window and the final paths
  __shared__ __align__(16) float sNodeBox[kTile * 6];
  __shared__ int32_t links[kTile * 3];
  __shared__ uint32_t leafUp[kTile];
  __shared__ uint32_t fVal[kTile];
  __shared__ uint32_t sFlag[kTile];
  __shared__ uint32_t sQueue[kTile / 2 + kTile / 4];
  __shared__ signed char sDelta[kTile + 2];
  __shared__ uint32_t sOpen[kTile / 32];
  __shared__ uint32_t sEq[kWindowWords];
  __shared__ int sLong;  // bit 0 / 1: the run at the tile's left / right end reaches past the window
  __shared__ uint32_t sCount, sQueued[2];
  TieWindow& win = *reinterpret_cast<TieWindow*>(sNodeBox);
  uint64_t* fPath = reinterpret_cast<uint64_t*>(sNodeBox + sizeof(TieWindow) / 4);
  static_assert(sizeof(TieWindow) + kTile * 8 <= kTile * 24, "window and paths in the node boxes' place");
  allow_next();
  await_previous();
  a.codes = written(a.codes);
  a.vals = written(a.vals);
  const unsigned long long n = leaf_count(a.dN, a.cap);
  const unsigned long long base = (unsigned long long)blockIdx.x * kTile;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const unsigned long long k = base + tid;
  if (k >= n && k < a.cap) a.outKeys[k] = ~0ull;  // padding past a device count
  // a single leaf has a key and no tree (out->keys held the sort's hash digits until here)
  if (n == 1 && k == 0) a.outKeys[0] = ((unsigned long long)*a.codes << 34) | (term_path(a.t, 0) >> 30);
  if (n < 2 || base >= n) return;
  const uint32_t cnt = (uint32_t)min((unsigned long long)kTile, n - base);
  const bool valid = tid < cnt;

  uint32_t code = 0, before = ~0u;  // this leaf's and its left neighbour's
  uint32_t val = 0;
  uint64_t path = 0;
  float mn[3], mx[3];
  if (valid) {
    code = *(a.codes + k);
    val = leaf_value(a, k, n);
    int d = -1;
    if (k > 0) {
      before = *(a.codes + k - 1);
      d = boundary_delta(before, code, (uint32_t)k);
    }
    sDelta[tid] = (signed char)d;
    win.val[kHalo + tid] = val;
    fVal[tid] = val;
  }
  // The warp's 32 records, eight at a time: four lanes fetch a record's four 16
  // bytes, so that a load touches 8 lines and not 32; three of them make an
  // axis of the box each, the fourth has the path.  (A lane per record kept the
  // L1 at 70% of its throughput with line look-ups: 5.9M leaves of the city 263
  // us, 240 this way; 19M of the mixed batch 932 and 850; 3.0M records 130 and
  // 117.)
  {
    const uint32_t part = lane & 3u;
    float4 row[4];
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) {
      const uint32_t v = __shfl_sync(kAll, val, (int)(q * 8 + (lane >> 2)));
      row[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (warp * 32 + q * 8 + (lane >> 2) < cnt) row[q] = __ldg(reinterpret_cast<const float4*>(a.t + v) + part);
    }
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) {
      const uint32_t e = warp * 32 + q * 8 + (lane >> 2);
      const bool quad = (__shfl_sync(kAll, __float_as_uint(row[q].x), (int)(lane | 3u)) >> 31) != 0;
      if (e >= cnt) continue;
      if (part < 3) {
        leaf_extent(row[q], quad, sBox[e * 6 + part], sBox[e * 6 + 3 + part]);
      } else {
        const uint64_t p = ((uint64_t)__float_as_uint(row[q].w) << 32) | __float_as_uint(row[q].z);
        win.path[kHalo + e] = p;
        fPath[e] = p;
      }
    }
    __syncwarp();
    if (valid) path = fPath[tid];
  }
  bool sameEnd = false;
  if (tid == cnt - 1) {  // the tile's right end
    int d = -1;
    if (k + 1 < n) {
      const uint32_t after = *(a.codes + k + 1);
      d = boundary_delta(code, after, (uint32_t)(k + 1));
      sameEnd = after == code;  // then cnt == kTile
    }
    sDelta[cnt] = (signed char)d;
  }
  if (tid < kTile / 32) sOpen[tid] = 0u;
  if (tid == 0) {
    sEq[0] = 0u;
    sLong = 0;
    sQueued[0] = sQueued[1] = 0u;
  }
  if (tid == cnt - 1) sEq[kWindowWords - 1] = 0u;
  const bool same = valid && k > 0 && before == code;
  if (__syncthreads_or(same || sameEnd)) {
    if (valid) load_box(sBox + tid * 6, mn, mx);
    // Equal to the left neighbour?  (The first leaf's and the right end's
    // neighbours are in other tiles.)
    bool eq = same;
    if (same) {
      const uint64_t other = tid > 0 ? win.path[kHalo + tid - 1] : term_path(a.t, leaf_value(a, k - 1, n));
      eq = (other >> kHashShift) == (path >> kHashShift);
    }
    const unsigned eqs = __ballot_sync(kAll, eq);
    if (lane == 0) sEq[1 + warp] = eqs;
    if (sameEnd && (term_path(a.t, leaf_value(a, k + 1, n)) >> kHashShift) == (path >> kHashShift))
      sEq[kWindowWords - 1] = 1u;
    __syncthreads();
    // the halo leaves that belong to the runs at the tile's ends
    bool halo = false;
    int hq = 0;
    uint64_t hPath = 0;
    if (warp == 0 && (sEq[1] & 1u)) {
      const uint32_t c = __shfl_sync(kAll, code, 0);
      const uint32_t h = (uint32_t)(win.path[kHalo] >> kHashShift);
      const long long i = (long long)base - kHalo + lane;
      const bool in = i >= 0 && tie_leaf(a, n, (unsigned long long)max(i, 0ll), c, h, val, hPath);
      const int have = __clz((int)~__ballot_sync(kAll, in));  // consecutive ones from lane 31 down
      halo = (int)lane >= 32 - have;
      hq = (int)lane;
      if (lane == 0) {
        uint32_t v;
        uint64_t p;
        const bool more = have == 32 && base > kHalo && tie_leaf(a, n, base - kHalo - 1, c, h, v, p);
        sEq[0] = (have >= 2 ? kAll << (33 - have) : 0u) | (more ? 1u : 0u);
        if (more) atomicOr(&sLong, 1);
      }
    } else if (warp == 1 && (sEq[kWindowWords - 1] & 1u)) {
      const uint32_t c = *(a.codes + base + kTile - 1);
      const uint32_t h = (uint32_t)(win.path[kHalo + kTile - 1] >> kHashShift);
      const unsigned long long i = base + kTile + lane;
      const bool in = i < n && tie_leaf(a, n, min(i, n - 1), c, h, val, hPath);
      const unsigned m = __ballot_sync(kAll, in);
      const int have = m == kAll ? 32 : __ffs((int)~m) - 1;
      halo = (int)lane < have;
      hq = (int)(kHalo + kTile + lane);
      if (lane == 0) {
        const unsigned long long past = base + kTile + kHalo;
        uint32_t v;
        uint64_t p;
        const bool more = have == 32 && past < n && tie_leaf(a, n, past, c, h, v, p);
        sEq[kWindowWords - 1] = have == 32 ? kAll : (1u << have) - 1u;
        if (more) atomicOr(&sLong, 2);
      }
    }
    if (halo) {
      win.path[hq] = hPath;
      win.val[hq] = val;
    }
    __syncthreads();
    const int isLong = sLong;
    // this thread's leaf, then (two warps) its halo key
    for (int turn = 0; turn < 2; turn++) {
      const int q = turn == 0 ? (int)(kHalo + tid) : hq;
      if (turn == 0 ? !valid : !halo) continue;
      const bool left = (sEq[q >> 5] >> (q & 31)) & 1u;
      const bool right = q + 1 < kWindowWords * 32 && ((sEq[(q + 1) >> 5] >> ((q + 1) & 31)) & 1u);
      if (!left && !right) continue;
      int s, e;
      tie_run(sEq, q, s, e);
      if ((isLong & 1) && s < (int)kHalo) continue;
      if ((isLong & 2) && e >= (int)(kHalo + kTile)) continue;
      const uint64_t p = win.path[q];
      const uint32_t v = win.val[q];
      int pos = s - (int)kHalo;
      for (int x = s; x <= e; x++) {
        const uint64_t px = win.path[x];
        pos += (px < p || (px == p && win.val[x] < v)) ? 1 : 0;
      }
      if (pos < 0 || pos >= (int)cnt) continue;  // a neighbouring tile's leaf
      if (turn == 1) {
        uint64_t again;
        gather_leaf(a.t, v, mn, mx, again);
      }
      store_box(sBox + pos * 6, mn, mx);
      fPath[pos] = p;
      fVal[pos] = v;
    }
    // runs that reach past the window: the members whose places are in this tile
    for (int side = 0; side < 2; side++) {
      if (!(isLong & (1 << side))) continue;
      __shared__ unsigned long long sRun[2];
      __syncthreads();
      const unsigned long long end = side == 0 ? base : base + cnt - 1;
      if (tid == 0) {
        const uint64_t top = tie_key(a, n, end);
        unsigned long long lo = 0, hi = end;  // first position with this code and hash digit
        while (lo < hi) {
          const unsigned long long mid = (lo + hi) >> 1;
          if (tie_key(a, n, mid) < top) lo = mid + 1;
          else hi = mid;
        }
        sRun[0] = lo;
        lo = end + 1;
        hi = n;  // first position past them
        while (lo < hi) {
          const unsigned long long mid = (lo + hi) >> 1;
          if (tie_key(a, n, mid) <= top) lo = mid + 1;
          else hi = mid;
        }
        sRun[1] = lo;
        sCount = 0u;
      }
      __syncthreads();
      const unsigned long long lo = sRun[0], hi = sRun[1];
      const unsigned long long first = max(lo, base), last = min(hi, base + cnt) - 1;
      uint64_t p0, p1;
      uint32_t v0, v1;
      tie_select(a, n, lo, hi, first - lo, sFlag, p0, v0);
      tie_select(a, n, lo, hi, last - lo, sFlag, p1, v1);
      for (unsigned long long i = lo + tid; i < hi; i += kTile) {
        const uint32_t v = leaf_value(a, i, n);
        const uint64_t p = term_path(a.t, v);
        if (p < p0 || (p == p0 && v < v0) || p > p1 || (p == p1 && v > v1)) continue;
        const uint32_t at = atomicAdd(&sCount, 1u);
        if (at > last - first) continue;  // never: the selects bound the members by their ranks
        win.path[at] = p;
        win.val[at] = v;
      }
      __syncthreads();
      const int m = (int)min((unsigned long long)sCount, last - first + 1);
      if ((int)tid < m) {
        const uint64_t p = win.path[tid];
        const uint32_t v = win.val[tid];
        uint32_t pos = (uint32_t)(first - base);  // at most first - base + m - 1 after the loop
        for (int x = 0; x < m; x++) pos += (win.path[x] < p || (win.path[x] == p && win.val[x] < v)) ? 1u : 0u;
        uint64_t again;
        gather_leaf(a.t, v, mn, mx, again);
        store_box(sBox + pos * 6, mn, mx);
        fPath[pos] = p;
        fVal[pos] = v;
      }
      __syncthreads();
      if (isLong == 3 && hi >= base + cnt) break;  // one run over the whole tile
    }
    __syncthreads();
  }
  const Forest f{sBox, sNodeBox, sFlag, sDelta, sOpen};
  if (valid) {
    a.leafTerminal[k] = fVal[tid];
    a.outKeys[k] = ((unsigned long long)code << 34) | (fPath[tid] >> 30);
    load_box(sBox + tid * 6, mn, mx);
  }
  __syncthreads();  // the node boxes take the window's place
  // First the leaves that are each other's sibling: joined by the left one's
  // thread.  Any other leaf waits at its boundary or, at the tile's ends, stays
  // open; no two climbers meet in this step, so it needs no exchange.
  int l = (int)tid, r = (int)tid;
  bool on = false;
  if (valid) {
    const bool up = sDelta[tid + 1] > sDelta[tid];
    const bool inside = tid + 1 < cnt;
    const bool nextDown = inside && !(sDelta[tid + 2] > sDelta[tid + 1]);
    uint32_t wait = 0;  // at boundary (tid, tid + 1)
    if (inside && up && !nextDown) wait = tid + 1;
    if (inside && !up && nextDown) wait = tid + 2;
    sFlag[tid] = wait;
    if ((up && !inside) || (!up && tid == 0)) atomicOr(&sOpen[tid >> 5], 1u << lane);
    on = up && nextDown;
  }
  if (on) {
    float smn[3], smx[3];
    load_box(sBox + (tid + 1) * 6, smn, smx);
#pragma unroll
    for (int q = 0; q < 3; q++) {
      mn[q] = fminf(mn[q], smn[q]);
      mx[q] = fmaxf(mx[q], smx[q]);
    }
    const int dl = sDelta[tid], dr = sDelta[tid + 2];
    const int at = (int)tid + (dr > dl ? 1 : 0);
    store_box(sNodeBox + at * 6, mn, mx);
    links[at * 3 + 1] = (int32_t)k;
    links[at * 3 + 2] = (int32_t)k + 1;
    leafUp[tid] = leafUp[tid + 1] = (uint32_t)base + (uint32_t)at;
    if (dl < 0 && dr < 0) {  // two leaves in all
      links[0] = -1;
      on = false;
    }
  }
  // Then the climb, in rounds: every join ends one of two climbers, so the
  // lanes left are few and far apart; they are packed into the first warps
  // before they go on.
  for (int round = 0; round < 2; round++) {
    const unsigned going = __ballot_sync(kAll, on);
    uint32_t at = 0;
    if (lane == 0 && going) at = atomicAdd(&sQueued[round], (uint32_t)__popc(going));
    at = __shfl_sync(kAll, at, 0) + __popc(going & ((1u << lane) - 1u));
    uint32_t* queue = sQueue + (round == 0 ? 0 : kTile / 2);  // subtrees of two leaves or more, then of four
    if (on) queue[at] = (uint32_t)l | ((uint32_t)(round == 0 ? l + 1 : r) << 16);
    __syncthreads();
    on = tid < sQueued[round];
    if (on) {
      const uint32_t w = queue[tid];
      l = (int)(w & 0xFFFFu);
      r = (int)(w >> 16);
      load_box(sNodeBox + (sDelta[r + 1] > sDelta[l] ? r : l) * 6, mn, mx);
      on = climb(f, l, r, mn, mx, round == 0 ? 2 : (int)cnt, (int)cnt, (uint32_t)base, links, leafUp);
    }
  }
  __syncthreads();
  open_waiting(f, (int)cnt);
  // Out, coalesced.  Open subtrees' parents and the nodes that cross the
  // tile's ends have no value yet: what goes out for them is written again by
  // the join that makes them, after this tile has arrived.
  const uint32_t inner = (uint32_t)min((unsigned long long)cnt, n - 1 - base);
  if (valid) a.leafParents[k] = leafUp[tid];
  for (uint32_t w = tid; w < inner * 3; w += kTile) a.nodes[base * 3 + w] = links[w];
  {
    float2* dst = reinterpret_cast<float2*>(a.aabbs + base * 6);
    const float2* src = reinterpret_cast<const float2*>(sNodeBox);
    for (uint32_t w = tid; w < inner * 3; w += kTile) dst[w] = src[w];
  }
  if (n <= kTile) return;
  __syncthreads();
  // The open subtrees, in leaf order, for k_join.
  const unsigned long long slot = blockIdx.x;
  if (valid && ((sOpen[tid >> 5] >> lane) & 1u)) {
    const uint32_t at = open_rank(sOpen, (int)tid);
    load_box(sBox + tid * 6, mn, mx);
    if (at < kMaxOpen) {
      float4* o = reinterpret_cast<float4*>(a.open + slot * kMaxOpen + at);
      o[0] = make_float4(mn[0], mn[1], mn[2], mx[0]);
      o[1] = make_float4(mx[1], mx[2], __uint_as_float((uint32_t)k), __int_as_float(sDelta[tid]));
    }
  }
  if (tid == 0) {
    uint32_t m = 0;
    for (uint32_t w = 0; w < kTile / 32; w++) m += __popc(sOpen[w]);
    a.openCount[slot] = min(m, kMaxOpen);
  }
}

// Joins the open subtrees of kGroup tiles a block, publishes what is still
// open, and the last of kGroup blocks to do so goes on with their group.  A
// kernel of its own: in k_tree's blocks the fence and the arrival held a
// tile's place on its SM for a quarter of its time (city of 5.9M leaves: 98 of
// 363 us).
//
// Open subtrees of neighbouring tiles join one after another, so a climb
// through them is 30 dependent steps long (city: 64 us, 20,011 leaves: 20 us
// for its two levels).  Here every join of a group is found on its own: the
// node at boundary c (before entry c) spans the entries up to the nearest
// smaller prefix on either side, found by descending a table of range minima,
// and its box comes from prefix and suffix boxes of 32-entry runs: 47 and 14 us.
constexpr int kJoinLevels = 10;             // range minima of 2^k boundaries, k < kJoinLevels

__device__ __forceinline__ void grow_box(float mn[3], float mx[3], const float* p) {
  float a[3], b[3];
  load_box(p, a, b);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    mn[k] = fminf(mn[k], a[k]);
    mx[k] = fmaxf(mx[k], b[k]);
  }
}

__global__ void __launch_bounds__(kTile) k_join(TreeArgs a) {
  constexpr unsigned kAll = 0xFFFFFFFFu;
  constexpr uint32_t kPer = kJoin / kTile;  // boundaries per thread
  __shared__ __align__(16) float sBox[kJoin * 6];
  __shared__ __align__(16) float sBefore[kJoin * 6];  // from the run's first entry to this one
  __shared__ __align__(16) float sAfter[kJoin * 6];   // from this entry to the run's last
  __shared__ uint32_t sLeft[kJoin + 1];
  __shared__ signed char sMin[kJoinLevels][kJoin + 1];  // [0]: the prefix at each entry's left boundary
  __shared__ uint32_t sClosed[kJoin / 32];              // bit c: the node at boundary c lies in the group
  __shared__ uint32_t sOpen[kJoin / 32];                // bit e: an open subtree starts at entry e
  __shared__ uint32_t sAt[kGroup];
  __shared__ uint32_t sCount, sTaken, sLast;
  signed char* delta = sMin[0];
  await_previous();
  a.codes = written(a.codes);
  a.open = const_cast<OpenTree*>(written(a.open));
  a.openCount = const_cast<uint32_t*>(written(a.openCount));
  const unsigned long long n = leaf_count(a.dN, a.cap);
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (n <= (unsigned long long)blockIdx.x * kGroup * kTile || n <= kTile) return;
  unsigned long long items = (n + kTile - 1) / kTile;  // tiles, then groups of the level being joined
  unsigned long long g = blockIdx.x, stride = 1;       // the group, and the tiles per item of this level
  uint32_t* joins = a.joins;
  for (;;) {
    const unsigned long long first = g * kGroup;
    const uint32_t size = (uint32_t)min((unsigned long long)kGroup, items - first);
    // The group's open subtrees, as many slots at a time as fit (always
    // several: what stays open of those joined so far is at most kMaxOpen).
    uint32_t carry = 0, next = 0;
    bool whole = false;
    while (!whole) {
      if (warp == 0) {
        const uint32_t j = next + lane;
        const uint32_t c = j < size ? __ldcg(a.openCount + (first + j) * stride) : 0u;
        uint32_t x = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t y = __shfl_up_sync(kAll, x, d);
          if (lane >= (uint32_t)d) x += y;
        }
        const unsigned fits = __ballot_sync(kAll, j < size && carry + x <= kJoin);  // a prefix of the lanes
        const uint32_t take = __popc(fits);
        sAt[lane] = carry + x - c;  // where slot j's entries go
        if (lane == take - 1u) sCount = carry + x;
        if (lane == 0) sTaken = take;
      }
      if (tid < kJoin / 32) sClosed[tid] = sOpen[tid] = 0u;
      __syncthreads();
      const uint32_t take = sTaken, count = sCount;
      // slots four at a time per warp, eight lanes to a slot
      for (uint32_t j = warp * 4 + (lane >> 3); j < take; j += kTile / 8) {
        const unsigned long long at = (first + next + j) * stride;
        const uint32_t to = sAt[j], c = (j + 1 < take ? sAt[j + 1] : count) - to;
        for (uint32_t x = lane & 7u; x < c; x += 8) {
          const float4* o = reinterpret_cast<const float4*>(a.open + at * kMaxOpen + x);
          const float4 p = __ldcg(o), q = __ldcg(o + 1);
          float* b = sBox + (to + x) * 6;
          b[0] = p.x; b[1] = p.y; b[2] = p.z; b[3] = p.w; b[4] = q.x; b[5] = q.y;
          sLeft[to + x] = __float_as_uint(q.z);
          delta[to + x] = (signed char)__float_as_int(q.w);
        }
      }
      next += take;
      whole = next >= size;
      if (tid == 0) {
        const unsigned long long end = min(n, (first + next) * stride * kTile);
        sLeft[count] = (uint32_t)end;
        delta[count] = (signed char)(end < n ? boundary_delta(*(a.codes + end - 1), *(a.codes + end), (uint32_t)end)
                                             : -1);
      }
      __syncthreads();
      // prefix and suffix boxes of the runs (a warp per run)
      for (uint32_t run = warp; run * 32 < count; run += kTile / 32) {
        const uint32_t e = run * 32 + lane;
        float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        if (e < count) load_box(sBox + e * 6, mn, mx);
        float pn[3] = {mn[0], mn[1], mn[2]}, px[3] = {mx[0], mx[1], mx[2]};
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
          for (int k = 0; k < 3; k++) {
            const float un = __shfl_up_sync(kAll, pn[k], d), ux = __shfl_up_sync(kAll, px[k], d);
            const float dn = __shfl_down_sync(kAll, mn[k], d), dx = __shfl_down_sync(kAll, mx[k], d);
            // (a lane past the end gets its own value back)
            pn[k] = fminf(un, pn[k]);
            px[k] = fmaxf(ux, px[k]);
            mn[k] = fminf(mn[k], dn);
            mx[k] = fmaxf(mx[k], dx);
          }
        }
        if (e < count) {
          store_box(sBefore + e * 6, pn, px);
          store_box(sAfter + e * 6, mn, mx);
        }
      }
      // range minima: sMin[k][c] over boundaries [c, c + 2^k)
#pragma unroll
      for (int k = 1; k < kJoinLevels; k++) {
        const int half = 1 << (k - 1);
        for (int c = (int)tid; c + 2 * half <= (int)count + 1; c += (int)kTile)
          sMin[k][c] = min(sMin[k - 1][c], sMin[k - 1][c + half]);
        __syncthreads();
      }
      float mn[kPer][3], mx[kPer][3];
      int from[kPer], to[kPer];  // the entries of the node at boundary c; from < 0: it reaches past the group
#pragma unroll
      for (uint32_t u = 0; u < kPer; u++) {
        const int c = (int)(u * kTile + tid);
        from[u] = -1;
        to[u] = -1;
        if (c == 0 || c >= (int)count) continue;
        const int v = delta[c];
        int p = c, q = c + 1;  // [p, c) and [c + 1, q) hold no smaller prefix
#pragma unroll
        for (int k = kJoinLevels - 1; k >= 0; k--) {
          const int w = 1 << k;
          if (p >= w && sMin[k][p - w] >= v) p -= w;
          if (q + w <= (int)count + 1 && sMin[k][q] >= v) q += w;
        }
        if (p == 0 || q > (int)count) continue;
        const int l = p - 1, r = q - 1;
        from[u] = l;
        to[u] = r;
        atomicOr(&sClosed[c >> 5], 1u << (c & 31));
        load_box(sAfter + l * 6, mn[u], mx[u]);
        if ((l >> 5) == (r >> 5)) {
          load_box(sBox + l * 6, mn[u], mx[u]);
          for (int x = l + 1; x <= r; x++) grow_box(mn[u], mx[u], sBox + x * 6);
        } else {
          for (int x = (l >> 5) + 1; x < (r >> 5); x++) grow_box(mn[u], mx[u], sAfter + x * 32 * 6);
          grow_box(mn[u], mx[u], sBefore + r * 6);
        }
        const bool left = delta[r + 1] > delta[l];  // a left child: its index is its right end
        const int32_t gl = (int32_t)sLeft[l], gr = (int32_t)sLeft[r + 1] - 1, gs = (int32_t)sLeft[c] - 1;
        const int32_t id = left ? gr : gl;
        a.nodes[(size_t)id * 3 + 1] = gl == gs ? gs : -gs;
        a.nodes[(size_t)id * 3 + 2] = gs + 1 == gr ? gr : -(gs + 1);
        *(gl == gs ? reinterpret_cast<int32_t*>(a.leafParents) + gs : a.nodes + (size_t)gs * 3) = id;
        *(gs + 1 == gr ? reinterpret_cast<int32_t*>(a.leafParents) + gr : a.nodes + (size_t)(gs + 1) * 3) = id;
        store_box(a.aabbs + (size_t)id * 6, mn[u], mx[u]);
        if (delta[l] < 0 && delta[r + 1] < 0) a.nodes[0] = -1;
      }
      __syncthreads();
      // A subtree (an entry, or a node made here) is open when its parent, at
      // the boundary of its larger prefix, is not in the group.
#pragma unroll
      for (uint32_t u = 0; u < kPer; u++) {
        const int e = (int)(u * kTile + tid);
        if (e < (int)count) {
          const int c = delta[e + 1] > delta[e] ? e + 1 : e;
          if (c >= (int)count || !((sClosed[c >> 5] >> (c & 31)) & 1u)) atomicOr(&sOpen[e >> 5], 1u << (e & 31));
        }
        if (from[u] >= 0) {
          const int l = from[u], r = to[u];
          const int c = delta[r + 1] > delta[l] ? r + 1 : l;
          const bool root = delta[l] < 0 && delta[r + 1] < 0;
          if (!root && (c >= (int)count || !((sClosed[c >> 5] >> (c & 31)) & 1u))) {
            store_box(sBox + l * 6, mn[u], mx[u]);
            atomicOr(&sOpen[l >> 5], 1u << (l & 31));
          }
        }
      }
      __syncthreads();
      // The subtrees still open, in order: to the front of the forest for the
      // next slots, or out to the group's place (its first tile's).
      uint32_t keepAt[kPer], keepLeft[kPer];
      int keepDelta[kPer];
#pragma unroll
      for (uint32_t u = 0; u < kPer; u++) {
        const uint32_t x = u * kTile + tid;
        keepAt[u] = kJoin;
        if (x < count && ((sOpen[x >> 5] >> (x & 31u)) & 1u)) {
          keepAt[u] = open_rank(sOpen, (int)x);
          keepLeft[u] = sLeft[x];
          keepDelta[u] = delta[x];
          load_box(sBox + x * 6, mn[u], mx[u]);
        }
      }
      carry = 0;
      for (uint32_t w = 0; w < kJoin / 32; w++) carry += __popc(sOpen[w]);
      carry = min(carry, kMaxOpen);
      __syncthreads();
#pragma unroll
      for (uint32_t u = 0; u < kPer; u++) {
        if (keepAt[u] >= kMaxOpen) continue;
        if (whole) {
          float4* o = reinterpret_cast<float4*>(a.open + first * stride * kMaxOpen + keepAt[u]);
          __stcg(o, make_float4(mn[u][0], mn[u][1], mn[u][2], mx[u][0]));
          __stcg(o + 1, make_float4(mx[u][1], mx[u][2], __uint_as_float(keepLeft[u]), __int_as_float(keepDelta[u])));
        } else {
          sLeft[keepAt[u]] = keepLeft[u];
          delta[keepAt[u]] = (signed char)keepDelta[u];
          store_box(sBox + keepAt[u] * 6, mn[u], mx[u]);
        }
      }
      __syncthreads();
    }
    const unsigned long long groups = (items + kGroup - 1) / kGroup;
    if (groups == 1) return;
    if (tid == 0) __stcg(a.openCount + first * stride, carry);
    items = groups;
    stride *= kGroup;
    const uint32_t peers = (uint32_t)min((unsigned long long)kGroup, items - g / kGroup * kGroup);
    __syncthreads();
    if (tid == 0) {
      __threadfence();  // the block's stores, ordered before it by the barrier, before its arrival
      sLast = atomicAdd(joins + g / kGroup, 1u) == peers - 1u ? 1u : 0u;
      __threadfence();
    }
    __syncthreads();
    if (!sLast) return;
    g /= kGroup;
    joins += (items + kGroup - 1) / kGroup;
  }
}

}  // namespace pga

using namespace pga;

// Sort scratch: the passes' digit counts and tile counters, the tree's arrival
// counters, and the look-back words (all of it zeroed by one memset) or the
// rows and groups of a counted pass (then only the arrival counters are).
static unsigned long long sort_tiles(unsigned long long n) {
  const unsigned long long tile = (unsigned long long)kSortThreads * (n <= kSmallSort ? kSmallItems : kLargeItems);
  return (n + tile - 1) / tile;
}
static unsigned long long tree_tiles(unsigned long long n) { return (n + kTile - 1) / kTile; }
static unsigned long long tree_joins(unsigned long long n) {
  unsigned long long sum = 0;
  for (unsigned long long items = tree_tiles(n); items > 1;) {
    items = (items + kGroup - 1) / kGroup;
    sum += items;
  }
  return (sum + 1) & ~1ull;  // the look-back words after them are 8 bytes wide
}

static size_t sort_words(unsigned long long n) {
  // small builds: the look-back words of each pass; large ones: the tiles' rows and the groups of one
  return (size_t)(kSortPasses * kBins + 64 + tree_joins(n) +
                  (n <= kSmallSort ? kSortPasses * sort_tiles(n) : sort_tiles(n) + kSortGroups) * kBins);
}

extern "C" size_t pga_lbvh_temp_bytes(uint64_t n) {
  n = n ? n : 1;
  // a smaller build may have more, smaller tiles
  return std::max(sort_words(n), sort_words(std::min<unsigned long long>(n, kSmallSort))) * sizeof(uint32_t);
}

// The tiles' open subtrees, then their counts.
extern "C" size_t pga_lbvh_open_bytes(uint64_t n) {
  return (size_t)tree_tiles(n ? n : 1) * (kMaxOpen * sizeof(OpenTree) + sizeof(uint32_t));
}

namespace pga {

// Scratch of one build: keys, two value arrays, the tiles' open subtrees, the
// radix sort's scratch, and the word a sort wait that gives up raises
// PGA_ERR_TIMEOUT in.
struct LbvhScratch {
  unsigned long long* keysA;
  uint32_t* valsA;
  uint32_t* valsB;
  void* open;
  void* sortTemp;
  size_t sortTempBytes;
  int* err;
};

// Polls of a look-back wait before it gives up (each followed by a 32 ns sleep).
constexpr uint32_t kSortSpinLimit = 1u << 22;

// Launches a kernel of a build behind the one before it; early: with its blocks
// placed ahead of that one's end (see await_previous).
template <typename... Params, typename... Args>
static cudaError_t launch_behind(bool early, void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem,
                                 cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

struct SortBuffers {
  uint32_t *codesA, *codesB;
  const uint16_t* hashes;
  uint32_t *valsA, *valsB;
  uint32_t* hist;      // digit counts of the passes
  uint32_t* counters;  // tile counters (small)
  uint32_t* words;     // look-back words of the passes (small), or rows and groups of one (large)
  int* err;
};

// Pass q of the sort: from the A arrays to the B arrays and back in turn.
template <bool SMALL, bool FIRST>
static PgaStatus launch_sort_pass(int q, unsigned long long n, const SortBuffers& b, cudaStream_t s) {
  constexpr int kItems = SMALL ? kSmallItems : kLargeItems;
  constexpr size_t smem = sort_pass_smem(kItems);
  const auto kernel = k_sort_pass<kItems, FIRST, !SMALL>;
  const unsigned tiles = (unsigned)sort_tiles(n);
  const uint32_t shift = FIRST ? 0u : (uint32_t)((q - 1) * kRadixBits);
  const bool even = q % 2 == 0;
  const uint32_t* cIn = even ? b.codesA : b.codesB;
  uint32_t* cOut = even ? b.codesB : b.codesA;
  const uint32_t* vIn = even ? b.valsA : b.valsB;
  uint32_t* vOut = even ? b.valsB : b.valsA;
  uint32_t* hist = b.hist + q * kBins;
  uint32_t* rows = b.words;
  uint32_t* groups = rows + (size_t)tiles * kBins;
  const uint32_t perGroup = (tiles + kSortGroups - 1) / kSortGroups;
  if (!SMALL) {
    k_sort_count<FIRST><<<kSortGroups, kSortThreads, 0, s>>>(cIn, b.hashes, n, shift, tiles, perGroup, rows, groups);
    PGA_CUDA_TRY(cudaGetLastError());
    k_sort_scan<<<kBins / 32, 1024, 0, s>>>(groups, hist);
    PGA_CUDA_TRY(cudaGetLastError());
  }
  PGA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const SortPass a{cIn, b.hashes, vIn, cOut, vOut, n, shift, hist,
                   reinterpret_cast<unsigned long long*>(b.words) + (SMALL ? (size_t)q * tiles * (kBins / 2) : 0),
                   b.counters + q, b.err, kSortSpinLimit, rows, groups, perGroup};
  PGA_CUDA_TRY(launch_behind(SMALL, +kernel, tiles, kSortThreads, smem, s, a));
  return PGA_OK;
}

template <bool SMALL>
static PgaStatus launch_sort(unsigned long long n, const SortBuffers& b, cudaStream_t s) {
  PgaStatus st = launch_sort_pass<SMALL, true>(0, n, b, s);
  for (int q = 1; q < kSortPasses && st == PGA_OK; q++) st = launch_sort_pass<SMALL, false>(q, n, b, s);
  static_assert(kSortPasses % 2 == 0, "an even number of passes ends in the A arrays");
  return st;
}

// The launches of a build over `cap` leaves, or over min(*dN, cap) when dN is
// a device count (then `cap` sizes the grids and the sort): Morton codes and
// digit histograms, four sort passes (codes and values ping-pong and end in
// the A arrays) and the tree.  The codes' two arrays share keysA; the hash
// digits lie in out->keys until the tree writes the final keys there.
static PgaStatus launch_lbvh(const PgaTerminal* t, unsigned long long cap, const unsigned long long* dN,
                             const PgaBounds* bounds, const PgaLbvh* out, const LbvhScratch& w, cudaStream_t s) {
  Bounds b;
  for (int k = 0; k < 3; k++) {
    b.mn[k] = bounds->min[k];
    b.sz[k] = bounds->max[k] - bounds->min[k];
  }
  if (sort_words(cap) * sizeof(uint32_t) > w.sortTempBytes) {
    set_error("LBVH: sort scratch too small for " + std::to_string(cap) + " keys");
    return PGA_ERR_INVALID_ARGUMENT;
  }
  uint32_t* hist = static_cast<uint32_t*>(w.sortTemp);
  uint32_t* counters = hist + kSortPasses * kBins;
  uint32_t* joins = counters + 64;
  const bool small = cap <= kSmallSort;
  uint32_t* words = joins + tree_joins(cap);
  // large builds read none of hist, counters and words before writing them
  uint32_t* clear = small ? hist : joins;
  const size_t clearWords = small ? sort_words(cap) : tree_joins(cap);
  PGA_CUDA_TRY(cudaMemsetAsync(clear, 0, clearWords * sizeof(uint32_t), s));
  uint32_t* codesA = reinterpret_cast<uint32_t*>(w.keysA);
  uint16_t* hashes = reinterpret_cast<uint16_t*>(out->keys);
  const SortBuffers sort{codesA, codesA + ((cap + 3) & ~3ull), hashes, w.valsA, w.valsB, hist, counters, words, w.err};
  const unsigned blocks = (unsigned)((cap + kLbvhThreads - 1) / kLbvhThreads);
  PgaStatus st;
  if (small) {
    k_morton<true><<<(unsigned)((cap + kHistThreads - 1) / kHistThreads), kHistThreads, 0, s>>>(t, cap, dN, b, codesA,
                                                                                              hashes, hist);
    PGA_CUDA_TRY(cudaGetLastError());
    st = launch_sort<true>(cap, sort, s);
  } else {
    k_morton<false><<<blocks, kLbvhThreads, 0, s>>>(t, cap, dN, b, codesA, hashes, hist);
    PGA_CUDA_TRY(cudaGetLastError());
    st = launch_sort<false>(cap, sort, s);
  }
  if (st != PGA_OK) return st;
  OpenTree* open = static_cast<OpenTree*>(w.open);
  const TreeArgs a{codesA, w.valsA, t, cap, dN, out->nodes, out->leafParents, out->aabbs, out->leafTerminal,
                   (unsigned long long*)out->keys, open,
                   reinterpret_cast<uint32_t*>(open + (size_t)blocks * kMaxOpen), joins};
  PGA_CUDA_TRY(launch_behind(small, k_tree, blocks, kTile, 0, s, a));
  if (blocks > 1) PGA_CUDA_TRY(launch_behind(small, k_join, (blocks + kGroup - 1) / (unsigned)kGroup, kTile, 0, s, a));
  return PGA_OK;
}

static LbvhScratch engine_scratch(PgaEngine* e) {
  return LbvhScratch{e->dKeysA, e->dValsA, e->dValsB, e->dOpenTrees, e->dSortTemp, e->sortTempBytes,
                     &e->dState->status};
}

static bool lbvh_out_ok(const PgaLbvh* out) {
  return out && out->nodes && out->leafParents && out->aabbs && out->leafTerminal && out->keys;
}

}  // namespace pga

extern "C" PgaStatus pga_lbvh_build(PgaEngine* e, const PgaTerminal* dTerminals, uint64_t n, const PgaBounds* bounds,
                                    const PgaLbvh* out, void* stream) {
  if (!e || !dTerminals || !bounds || !lbvh_out_ok(out)) {
    set_error("pga_lbvh_build: null argument");
    return PGA_ERR_INVALID_ARGUMENT;
  }
  if (n < 2 || n > e->cfg.maxTerminals || n >= (1ull << 30)) {
    set_error("pga_lbvh_build: need 2 <= n <= maxTerminals (and < 2^30)");
    return PGA_ERR_INVALID_ARGUMENT;
  }
  return launch_lbvh(dTerminals, n, nullptr, bounds, out, engine_scratch(e), (cudaStream_t)stream);
}

extern "C" PgaStatus pga_lbvh_build_counted(PgaEngine* e, const PgaTerminal* dTerminals, const uint64_t* dCount,
                                            uint64_t capacity, const PgaBounds* bounds, const PgaLbvh* out,
                                            void* stream) {
  if (!e || !dTerminals || !dCount || !bounds || !lbvh_out_ok(out)) {
    set_error("pga_lbvh_build_counted: null argument");
    return PGA_ERR_INVALID_ARGUMENT;
  }
  if (capacity < 2 || capacity > e->cfg.maxTerminals || capacity >= (1ull << 30)) {
    set_error("pga_lbvh_build_counted: need 2 <= capacity <= maxTerminals (and < 2^30)");
    return PGA_ERR_INVALID_ARGUMENT;
  }
  return launch_lbvh(dTerminals, capacity, (const unsigned long long*)dCount, bounds, out, engine_scratch(e),
                     (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// pga_lbvh_build_static: the same LBVH build with every piece of scratch taken
// from one fixed device array of this file instead of an engine's buffers.
//
// Some callers cannot allocate device memory when they build a hierarchy: a
// host process whose device-memory budget was handed out in full at start-up,
// a plug-in running inside an application that owns the allocator, or code
// that must not hit the driver's allocator inside a latency-critical loop.
// They pass only their inputs and outputs; the scratch lives in
// g_lbvhStaticScratch, which every GPU that loads this library holds until
// the process exits.
//
// The array's name denotes a host-side stand-in in host code, not a device
// address, so the device address is looked up once per device with
// cudaGetSymbolAddress (with that device current) on the first call made on
// it.  Under CUDA's lazy module loading the array itself is committed on the
// device only when this file's module first loads there -- at that lookup at
// the latest -- so a caller that hands out its device budget at start-up
// makes one call on each device first: a call with n = 0 (pointers may be
// null) does only this set-up.  Make it before any stream capture too.  The
// address is cached per device ordinal for the life of the process: the
// library assumes that each device's primary context lives as long as the
// process (after cudaDeviceReset the cached address is stale).  All calls
// share the array and it keeps the last call's contents: the counters that
// must start at zero are cleared on every call, and calls that overlap
// on the GPU (on different streams, or from different threads) race on it.

namespace pga {

constexpr size_t kStaticScratchBytes = 6u << 20;  // 6 MiB
static __device__ __align__(256) unsigned char g_lbvhStaticScratch[kStaticScratchBytes];

static std::mutex g_staticMutex;
static void* g_staticAddr[64];  // device address of g_lbvhStaticScratch per device ordinal

static size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace pga

extern "C" PgaStatus pga_lbvh_build_static(const PgaTerminal* dTerminals, uint64_t n, const PgaBounds* bounds,
                                           const PgaLbvh* out, void* stream) {
  if (n != 0 && (!dTerminals || !bounds || !lbvh_out_ok(out))) {
    set_error("pga_lbvh_build_static: null argument");
    return PGA_ERR_INVALID_ARGUMENT;
  }
  if (n == 1 || n > PGA_LBVH_STATIC_MAX_LEAVES) {
    set_error("pga_lbvh_build_static: n must be 0 (set-up only) or in [2, " +
              std::to_string(PGA_LBVH_STATIC_MAX_LEAVES) +
              "] (the fixed scratch holds at most that many leaves); use pga_lbvh_build for larger sets");
    return PGA_ERR_INVALID_ARGUMENT;
  }
  int dev = 0;
  PGA_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    set_error("pga_lbvh_build_static: device ordinal out of range");
    return PGA_ERR_INVALID_ARGUMENT;
  }
  unsigned char* base = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_staticMutex);
    if (!g_staticAddr[dev]) {
      void* p = nullptr;
      cudaError_t err = cudaGetSymbolAddress(&p, g_lbvhStaticScratch);
      if (err != cudaSuccess) return cuda_status(err, "pga_lbvh_build_static: cudaGetSymbolAddress");
      g_staticAddr[dev] = p;
    }
    base = static_cast<unsigned char*>(g_staticAddr[dev]);
  }
  if (n == 0) return PGA_OK;  // set-up only
  // Carve the scratch: keys, two value arrays, the tiles' open subtrees, sort temp.
  size_t temp = pga_lbvh_temp_bytes(n);
  size_t off = 0;
  unsigned long long* keysA = reinterpret_cast<unsigned long long*>(base + off);
  off += align256(n * sizeof(unsigned long long));
  uint32_t* valsA = reinterpret_cast<uint32_t*>(base + off);
  off += align256(n * sizeof(uint32_t));
  uint32_t* valsB = reinterpret_cast<uint32_t*>(base + off);
  off += align256(n * sizeof(uint32_t));
  void* open = base + off;
  off += align256(pga_lbvh_open_bytes(n));
  void* sortTemp = base + off;
  off += align256(temp);
  int* err = reinterpret_cast<int*>(base + off);  // a sort wait that gives up marks it (unreported)
  off += 256;
  if (off > kStaticScratchBytes) {
    set_error("pga_lbvh_build_static: fixed scratch too small for the radix sort of " + std::to_string(n) + " keys");
    return PGA_ERR_INVALID_ARGUMENT;
  }
  const LbvhScratch w{keysA, valsA, valsB, open, sortTemp, temp, err};
  return launch_lbvh(dTerminals, n, nullptr, bounds, out, w, (cudaStream_t)stream);
}
