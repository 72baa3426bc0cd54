// Onesweep-style stable LSD radix sort of (key, uint32 value) pairs, 8-bit digits.
//
// Replaces cub::DeviceRadixSort::SortPairs (lib/builder/LBVH_CUDA.cu:185-193) and
// SortPairsDescending (lib/builder/Bittner13CUDA.cu:674-680). Design (Adinets & Merrill 2022):
//   1. one read of all keys builds the digit histograms of every pass;
//   2. per pass, one kernel: each CTA makes the digits' global offsets from the pass's histogram (a tiny
//      scan launch does for the large tiles) and takes tile indices from an atomic counter until none is left
//      (so the tiles it looks back on are already running). It ranks a tile's keys stably (per item, the lanes holding the same digit are
//      found with 9 ballots and a warp-private counter per digit is advanced by one shared-memory
//      atomic of the lowest such lane; the atomics of all items are issued before any result is
//      used), publishes per-digit counts, resolves its exclusive prefix by decoupled look-back (kLook
//      predecessors per round trip, bounded spin), stages the tile in shared memory in digit order and
//      writes it out in runs, so each digit's run is a contiguous store.
// A status word holds a flag and a count together and nothing else is read through it, so it is
// published and polled with relaxed gpu-scope accesses (no fences); the next pass reads the keys
// this pass wrote only after the kernel boundary.
#include <atomic>

#include "common.cuh"
#include "sort.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

namespace bvhgb {

namespace {

constexpr int kThreads = 512;  // histogram blocks; the onesweep tile shape is a template parameter
constexpr int kMinTile = 2048;  // smallest tile: the status arrays are sized for it
constexpr int kRadix = 256;
constexpr int kBins = kRadix + 1;  // + a bin for padding keys of the last tile
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagInc = 2u << 30;
constexpr uint32_t kFlagMask = 3u << 30;
constexpr uint32_t kValMask = (1u << 30) - 1u;
// Predecessors read per look-back round trip. The tiles of a wave start together, so a tile k
// places behind the last finished one needs about k / kLook round trips.
constexpr int kLook = 16;
// Polls of an unpublished predecessor before a tile gives up and raises kErrTimeout (the tile then
// scatters with the partial prefix it has: positions below the true ones, so every write stays in
// bounds). Adjustable for tests of that path (bvhgb_sort_set_spin_limit).
__constant__ uint32_t g_lookback_spin_limit = kSpinLimit;

// The last digit may be narrower than 8 bits when (endBit - beginBit) is not a multiple of 8.
__host__ __device__ __forceinline__ uint32_t digit_mask(uint32_t shift, uint32_t endBit) {
  const uint32_t w = endBit - shift;
  return w >= 8 ? 0xFFu : ((1u << w) - 1u);
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

struct Layout {
  size_t hist, counters, err, status, altKeys, altVals, total;
  uint32_t passes, tiles;
};

Layout make_layout(uint32_t n, uint32_t keyBytes, uint32_t beginBit, uint32_t endBit, uint32_t tile = kMinTile) {
  Layout L{};
  L.passes = (endBit > beginBit) ? (endBit - beginBit + 7) / 8 : 0;
  L.tiles = n ? (uint32_t)((n + tile - 1) / tile) : 0;
  size_t off = 0;
  L.hist = off;     off = align256(off + sizeof(uint32_t) * kRadix * (L.passes ? L.passes : 1));
  L.counters = off; off = align256(off + sizeof(uint32_t) * (L.passes ? L.passes : 1));
  L.err = off;      off = align256(off + sizeof(uint32_t));
  L.status = off;   off = align256(off + sizeof(uint32_t) * kRadix * (size_t)L.tiles * (L.passes ? L.passes : 1));
  L.altKeys = off;  off = align256(off + (size_t)keyBytes * n);
  L.altVals = off;  off = align256(off + sizeof(uint32_t) * (size_t)n);
  L.total = off;
  return L;
}

// A kernel given this word does nothing where it is set (null: it always works).
__device__ __forceinline__ bool skipped(const uint32_t *word) { return word && __ldcg(word) != 0u; }

template <typename K>
__device__ __forceinline__ void histogram_all(const K *keys, uint32_t n, uint32_t beginBit, uint32_t endBit,
                                              uint32_t passes, uint32_t *hist, uint32_t *sh) {  // sh: passes * 256 words
  for (uint32_t i = threadIdx.x; i < passes * kRadix; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    K k = __ldcg(keys + i);
    for (uint32_t p = 0; p < passes; ++p) {
      const uint32_t sh0 = beginBit + 8 * p;
      uint32_t d = (uint32_t)(k >> sh0) & digit_mask(sh0, endBit);
      atomicAdd(&sh[p * kRadix + d], 1u);
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < passes * kRadix; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

template <typename K>
__global__ void __launch_bounds__(kThreads) histogram_kernel(const K *__restrict__ keys, uint32_t n,
                                                             uint32_t beginBit, uint32_t endBit, uint32_t passes,
                                                             uint32_t *__restrict__ hist, MortonCells cells) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cells.words; i += gridDim.x * blockDim.x)
    if (__ldg(cells.count + i) >= heavy_cell(n)) *cells.heavy = 1u;
  extern __shared__ uint32_t histSm[];
  histogram_all(keys, n, beginBit, endBit, passes, hist, histSm);
}

// Exclusive scan of each pass's 256 counts, in place. One CTA per pass. For the tile shapes whose CTAs do not
// scan their pass's counts themselves: the large ones, which have no registers to spare for it (a pass of
// 4.19M pairs 39 us, 41 so; the launch saved is worth 2 us of a small sort).
__global__ void __launch_bounds__(kRadix) scan_kernel(uint32_t *hist, const uint32_t *skip) {
  if (skipped(skip)) return;
  __shared__ uint32_t s[kRadix];
  uint32_t *h = hist + blockIdx.x * kRadix;
  uint32_t v = h[threadIdx.x];
  s[threadIdx.x] = v;
  __syncthreads();
  for (int off = 1; off < kRadix; off <<= 1) {
    uint32_t t = threadIdx.x >= (unsigned)off ? s[threadIdx.x - off] : 0u;
    __syncthreads();
    s[threadIdx.x] += t;
    __syncthreads();
  }
  h[threadIdx.x] = s[threadIdx.x] - v;
}

template <int THREADS>
constexpr bool kScans = THREADS == 256;  // the CTAs scan their pass's counts themselves

template <int ITEMS>  // CTAs per SM of a tile shape
constexpr int kSortCtas = ITEMS <= 8 ? 3 : 2;

template <typename K, int THREADS, int ITEMS>
struct OnesweepSmem {
  static constexpr int kWarps = THREADS / 32;
  static constexpr int kTile = THREADS * ITEMS;
  uint32_t warpHist[kWarps][kBins];
  uint32_t tileStart[kRadix];
  uint32_t globalBase[kRadix];
  uint32_t digitBase[kScans<THREADS> ? kRadix : 1], digitTot[kRadix / 32];  // keys of lower digits in the same 32, and of each 32
  uint32_t scanTot[kRadix / 32];
  uint32_t tileIdx;
  // The tile in digit order; its values beside the keys or, where two CTAs would not fit then, in their
  // place once the keys are written.
  static constexpr bool kSplit = sizeof(K) == 8 && THREADS == 512;
  K keys[kTile];
  uint32_t valsOwn[kSplit ? 1 : kTile];
  __device__ __forceinline__ uint32_t *vals() { return kSplit ? reinterpret_cast<uint32_t *>(keys) : valsOwn; }
};

// CTAs take tiles from the counter until none is left. Bound: a tile's phases (load, rank, look back,
// stage, write) are a chain of latencies with barriers between them, so a second CTA per SM is what
// fills them: 64 registers per thread (ranks kept as 16-bit pairs, values read when the keys are out
// of the way) and one staging buffer for keys and then values (82 KB for 8,192 64-bit keys). A pass of
// 4.19M / 33.5M pairs of 64-bit keys in tiles of 8,192: 45 / 310 us (39.5 for 4.19M in tiles of 7,168); with one CTA per SM and 124 registers 49 / 336;
// with the look-back before the staging 50 / 298, in the lower warps while the upper ones stage 48 /
// 374; 32 predecessors per round trip 46 / 334; digits matched by match.any 58 / 397.
// FRESH: the pairs and offsets were written in this launch (the loads go past L1); otherwise by an earlier
// one (33.5M 64-bit pairs, a pass: read-only loads 310 us, past L1 336).
template <bool FRESH, typename T>
__device__ __forceinline__ T load_once(const T *p) {
  return FRESH ? __ldcg(p) : __ldg(p);
}

template <typename K, int THREADS, int ITEMS, bool FRESH>
__device__ __forceinline__ void onesweep_tiles(OnesweepSmem<K, THREADS, ITEMS> &sm, const K *keysIn, K *keysOut,
                                               const uint32_t *valsIn, uint32_t *valsOut, uint32_t n, uint32_t tiles,
                                               uint32_t shift, uint32_t mask, const uint32_t *hist,
                                               uint32_t *tileCounter, uint32_t *status, uint32_t *err) {
  using Smem = OnesweepSmem<K, THREADS, ITEMS>;
  constexpr int kWarps = Smem::kWarps, kTile = Smem::kTile;
  constexpr bool kSplit = Smem::kSplit, kLate = THREADS == 512;
  static_assert(THREADS >= kRadix, "one thread per digit in the look-back");
  constexpr int kGroup = ITEMS % 4 == 0 ? 4 : 2;  // items ranked together
  static_assert(ITEMS % 2 == 0 && kTile <= 65536, "ranks as 16-bit pairs");
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t ltMask = (1u << lane) - 1u;
  if (threadIdx.x == 0) sm.tileIdx = atomicAdd(tileCounter, 1u);
  if (kScans<THREADS> && threadIdx.x < kRadix) {  // where each digit's keys begin, from the pass's histogram
    const uint32_t v = load_once<FRESH>(hist + threadIdx.x);
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= (uint32_t)o) incl += y;
    }
    sm.digitBase[threadIdx.x] = incl - v;
    if (lane == 31) sm.digitTot[warp] = incl;
  }
  for (;;) {
    for (uint32_t i = lane; i < kBins; i += 32) sm.warpHist[warp][i] = 0;
    __syncthreads();
    const uint32_t tile = sm.tileIdx;
    if (tile >= tiles) return;
    const uint64_t base = (uint64_t)tile * kTile;
    const uint32_t valid = (uint32_t)min((uint64_t)kTile, (uint64_t)n - base);
    const uint32_t t0 = warp * (ITEMS * 32) + lane;  // warp-striped: item j of the thread is key t0 + 32 j

    K key[ITEMS];
    uint32_t val[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      key[j] = t0 + 32 * j < valid ? load_once<FRESH>(keysIn + base + t0 + 32 * j) : (K)0;
      if (!kSplit) val[j] = t0 + 32 * j < valid ? load_once<FRESH>(valsIn + base + t0 + 32 * j) : 0u;
    }
    // Stable rank within the warp: items in order, lanes in order. Peers of an item are the lanes
    // with the same digit (8 ballots, and one for the padding bin in the last tile); the lowest of
    // them advances the warp's counter for that digit by their number. The atomics of a group of items are
    // issued, in item order (__syncwarp orders them), before their results are used.
    uint32_t rank[ITEMS / 2];
#pragma unroll
    for (int j0 = 0; j0 < ITEMS; j0 += kGroup) {
      uint32_t old[kGroup], peers[kGroup];
#pragma unroll
      for (int q = 0; q < kGroup; ++q) {
        const int j = j0 + q;
        const bool in = t0 + 32 * j < valid;
        const uint32_t d = in ? (uint32_t)(key[j] >> shift) & mask : (uint32_t)kRadix;
        uint32_t p = 0xFFFFFFFFu;
        if (valid != (uint32_t)kTile) {
          const uint32_t bal = __ballot_sync(0xFFFFFFFFu, in);
          p = in ? bal : ~bal;
        }
#pragma unroll
        for (int bit = 0; bit < 8; ++bit) {
          const bool on = (d >> bit) & 1u;
          const uint32_t bal = __ballot_sync(0xFFFFFFFFu, on);
          p &= on ? bal : ~bal;
        }
        peers[q] = p;
        old[q] = 0;
        if ((p & ltMask) == 0) old[q] = atomicAdd(&sm.warpHist[warp][d], (uint32_t)__popc(p));
        __syncwarp();
      }
#pragma unroll
      for (int q = 0; q < kGroup; q += 2) {
        const uint32_t a = __shfl_sync(0xFFFFFFFFu, old[q], __ffs(peers[q]) - 1) + __popc(peers[q] & ltMask);
        const uint32_t b = __shfl_sync(0xFFFFFFFFu, old[q + 1], __ffs(peers[q + 1]) - 1) + __popc(peers[q + 1] & ltMask);
        rank[(j0 + q) / 2] = a | (b << 16);
      }
    }
    __syncthreads();

    // Per digit (one thread each): the tile's count, published; its place in the tile (a warp scan per
    // 32 digits) and from it every warp's. Staging needs no more, so for the large tile the
    // look-back comes after it: the predecessors' counts arrive meanwhile and the keys' registers are
    // free for it. The smaller tiles look back at once (65,536 30-bit pairs in tiles of 2,048: 51 us
    // against 58; 4.19M in tiles of 8,192: 213 against 191).
    auto look_back = [&](uint32_t d, uint32_t count) {
      uint32_t excl = 0;
      if (tile > 0) {
        int64_t pred = (int64_t)tile - 1;
        bool done = false;
        while (!done) {
          uint32_t v[kLook];
#pragma unroll
          for (int q = 0; q < kLook; ++q) v[q] = pred - q >= 0 ? ld_relaxed(status + (size_t)(pred - q) * kRadix + d) : kFlagInc;
#pragma unroll
          for (int q = 0; q < kLook; ++q) {
            if (done) break;
            if (pred - q < 0) {
              done = true;
              break;
            }
            const uint32_t *ps = status + (size_t)(pred - q) * kRadix + d;
            uint32_t spins = 0;
            while ((v[q] & kFlagMask) == 0u) {
              if (++spins > g_lookback_spin_limit) {
                atomicOr(err, kErrTimeout);
                break;
              }
              __nanosleep(32);
              v[q] = ld_relaxed(ps);
            }
            if ((v[q] & kFlagMask) == 0u) {
              done = true;
              break;
            }
            excl += v[q] & kValMask;
            if (v[q] & kFlagInc) done = true;
          }
          pred -= kLook;
        }
        st_relaxed(status + (size_t)tile * kRadix + d, kFlagInc | (excl + count));
      }
      if (kScans<THREADS>) {
        excl += sm.digitBase[d];
#pragma unroll
        for (uint32_t w = 0; w < kRadix / 32; ++w) excl += w < d / 32 ? sm.digitTot[w] : 0u;
        sm.globalBase[d] = excl;
      } else {
        sm.globalBase[d] = load_once<FRESH>(hist + d) + excl;
      }
    };
    uint32_t count = 0, incl = 0;
    if (threadIdx.x < kRadix) {
      const uint32_t d = threadIdx.x;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) count += sm.warpHist[w][d];
      st_relaxed(status + (size_t)tile * kRadix + d, (tile == 0 ? kFlagInc : kFlagAgg) | count);
      incl = count;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
      }
      if (lane == 31) sm.scanTot[warp] = incl;
      if (!kLate) look_back(d, count);
    }
    __syncthreads();
    if (threadIdx.x < kRadix) {
      const uint32_t d = threadIdx.x;
      uint32_t at = incl - count;
      for (uint32_t w = 0; w < warp; ++w) at += sm.scanTot[w];
      sm.tileStart[d] = at;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const uint32_t c = sm.warpHist[w][d];
        sm.warpHist[w][d] = at;
        at += c;
      }
    }
    __syncthreads();
    // Stage the tile's keys in digit order; a rank becomes the place in the tile.
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      if (t0 + 32 * j < valid) {
        const uint32_t d = (uint32_t)(key[j] >> shift) & mask;
        const uint32_t pos = sm.warpHist[warp][d] + ((rank[j / 2] >> (16 * (j & 1))) & 0xFFFFu);
        sm.keys[pos] = key[j];
        if (!kSplit) sm.valsOwn[pos] = val[j];
        if (kSplit) rank[j / 2] = j & 1 ? (rank[j / 2] & 0xFFFFu) | (pos << 16) : (rank[j / 2] & 0xFFFF0000u) | pos;
      }
    }
    if (kLate && threadIdx.x < kRadix) look_back(threadIdx.x, count);
    // The next tile (every thread has read this one's index), if there are more tiles than CTAs. Tiles
    // are taken in order and a CTA's tile waits for lower ones only, so the lowest unfinished tile is
    // always being worked on.
    const bool more = gridDim.x < tiles;
    if (more && threadIdx.x == THREADS - 1) sm.tileIdx = atomicAdd(tileCounter, 1u);
    if (kSplit) {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) val[j] = t0 + 32 * j < valid ? load_once<FRESH>(valsIn + base + t0 + 32 * j) : 0u;
    }
    __syncthreads();
    uint32_t dst[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const uint32_t i = j * THREADS + threadIdx.x;
      dst[j] = n;
      if (i < valid) {
        const K k = sm.keys[i];
        const uint32_t d = (uint32_t)(k >> shift) & mask;
        dst[j] = sm.globalBase[d] + (i - sm.tileStart[d]);
        // Always true for a consistent sort; after a look-back timeout (err set) a later pass reads a
        // permuted, partly stale key array whose digits no longer match the histogram, and this keeps
        // its writes inside the arrays.
        if (dst[j] < n) {
          keysOut[dst[j]] = k;
          if (!kSplit) valsOut[dst[j]] = sm.valsOwn[i];
        }
      }
    }
    if (kSplit) {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if (t0 + 32 * j < valid) sm.vals()[(rank[j / 2] >> (16 * (j & 1))) & 0xFFFFu] = val[j];
      __syncthreads();
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if (dst[j] < n) valsOut[dst[j]] = sm.vals()[j * THREADS + threadIdx.x];
    }
    if (!more) return;
  }
}

template <typename K, int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS, kSortCtas<ITEMS>) onesweep_kernel(
    const K *__restrict__ keysIn, K *__restrict__ keysOut, const uint32_t *__restrict__ valsIn,
    uint32_t *__restrict__ valsOut, uint32_t n, uint32_t tiles, uint32_t shift, uint32_t mask,
    const uint32_t *__restrict__ hist, uint32_t *tileCounter, uint32_t *status, uint32_t *err,
    const uint32_t *skip) {
  if (skipped(skip)) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  onesweep_tiles<K, THREADS, ITEMS, false>(*reinterpret_cast<OnesweepSmem<K, THREADS, ITEMS> *>(smraw), keysIn, keysOut, valsIn,
                                    valsOut, n, tiles, shift, mask, hist, tileCounter, status, err);
}

// The passes over bits [beginBit, endBit) between the out and alternate arrays, the last one into the out
// arrays (outLast) or into the alternate ones.
template <typename K, int THREADS, int ITEMS>
int onesweep_passes(const Layout &L, const K *keysIn, K *keysOut, const uint32_t *valsIn, uint32_t *valsOut, K *altK,
                    uint32_t *altV, uint32_t *hist, uint32_t *counters, uint32_t *status, uint32_t *err, uint32_t n,
                    uint32_t beginBit, uint32_t endBit, cudaStream_t s, bool outLast, const uint32_t *skip) {
  const size_t smem = sizeof(OnesweepSmem<K, THREADS, ITEMS>);
  const uint32_t grid = min(L.tiles, (uint32_t)(sm_count() * kSortCtas<ITEMS>));
  const K *srcK = keysIn;
  const uint32_t *srcV = valsIn;
  for (uint32_t p = 0; p < L.passes; ++p) {
    const bool toOut = (((L.passes - 1 - p) % 2) == 0) == outLast;
    K *dstK = toOut ? keysOut : altK;
    uint32_t *dstV = toOut ? valsOut : altV;
    const uint32_t shift = beginBit + 8 * p;
    onesweep_kernel<K, THREADS, ITEMS><<<grid, THREADS, smem, s>>>(
        srcK, dstK, srcV, dstV, n, L.tiles, shift, digit_mask(shift, endBit), hist + p * kRadix, counters + p,
        status + (size_t)p * L.tiles * kRadix, err, skip);
    BVHGB_LAUNCH_CHECK("radix onesweep");
    srcK = dstK;
    srcV = dstV;
  }
  return BVHGB_OK;
}

// Histogram and passes; hist, counters, err and status start at zero.
template <typename K>
int sort_passes(const Layout &L, uint32_t tileKeys, const K *keysIn, K *keysOut, const uint32_t *valsIn,
                uint32_t *valsOut, K *altK, uint32_t *altV, uint32_t *hist, uint32_t *counters, uint32_t *status,
                uint32_t *err, uint32_t n, uint32_t beginBit, uint32_t endBit, cudaStream_t s, bool outLast,
                const MortonCells &cells = {}) {
  const uint32_t hgrid = min(ceil_div(n, kThreads * 8), (uint32_t)sm_count() * 4);
  histogram_kernel<K><<<hgrid, kThreads, sizeof(uint32_t) * kRadix * L.passes, s>>>(keysIn, n, beginBit, endBit,
                                                                                    L.passes, hist, cells);
  BVHGB_LAUNCH_CHECK("radix histogram");
  if (tileKeys > 4096) {  // the shapes of 512 threads
    scan_kernel<<<L.passes, kRadix, 0, s>>>(hist, cells.heavy);
    BVHGB_LAUNCH_CHECK("radix scan");
  }
  switch (tileKeys) {
    case 2048:
      return onesweep_passes<K, 256, 8>(L, keysIn, keysOut, valsIn, valsOut, altK, altV, hist, counters, status, err, n,
                                        beginBit, endBit, s, outLast, cells.heavy);
    case 4096:
      return onesweep_passes<K, 256, 16>(L, keysIn, keysOut, valsIn, valsOut, altK, altV, hist, counters, status, err,
                                         n, beginBit, endBit, s, outLast, cells.heavy);
    case 6144:
      return onesweep_passes<K, 512, 12>(L, keysIn, keysOut, valsIn, valsOut, altK, altV, hist, counters, status, err,
                                         n, beginBit, endBit, s, outLast, cells.heavy);
    case 7168:
      return onesweep_passes<K, 512, 14>(L, keysIn, keysOut, valsIn, valsOut, altK, altV, hist, counters, status, err,
                                         n, beginBit, endBit, s, outLast, cells.heavy);
    default:
      return onesweep_passes<K, 512, 16>(L, keysIn, keysOut, valsIn, valsOut, altK, altV, hist, counters, status, err,
                                         n, beginBit, endBit, s, outLast, cells.heavy);
  }
}

std::atomic<uint32_t> g_default_tile{BVHGB_SORT_TILE_AUTO};

// Keys per CTA of a sort that is given none: the process-wide setting or, where that leaves the choice
// (BVHGB_SORT_TILE_AUTO), by the number of pairs. Small sorts fill few CTAs at the large tiles (63-bit keys,
// 2,048 / 4,096 / 8,192: 262,144 pairs 81 / 88 / 104 us, 524,288 100 / 91 / 109). From there to 8M pairs
// the tile is the one whose SMs are done first: w tiles an SM take about (w + ceil(w)) / 2 times a tile's
// time, which grows with its items and, for 16 of them, the registers they spill. 63-bit keys, tiles of
// 4,096 / 6,144 / 7,168 / 8,192: 1M 122 / 124 / 114 / 121 us, 1.5M 154 / 137 / 142 / 154, 2.49M 190 / 191 /
// 199 / 175, 4.19M 297 / 266 / 249 / 272, 8.39M 546 / 479 / 466 / 474. Beyond, where the arrays do not fit
// L2, the longer runs of the largest tile count: 12M 895 / 768 / 757 / 720, 33.5M 2,424 / 2,067 / 1,983 / 1,852.
uint32_t auto_tile(uint32_t n) {
  const uint32_t given = g_default_tile.load(std::memory_order_relaxed);
  if (given != BVHGB_SORT_TILE_AUTO) return given;
  if (n <= (1u << 18)) return (uint32_t)kMinTile;
  if (n > (1u << 23)) return kSortTileDefault;
  constexpr uint32_t shapes[4][2] = {{4096, 12}, {6144, 16}, {7168, 18}, {8192, 22}};  // keys, a tile's time
  uint32_t best = 0;
  float least = 0.0f;
  for (const auto &t : shapes) {
    const float w = (float)ceil_div(n, t[0]) / (float)sm_count(), cost = (w + std::ceil(w)) * (float)t[1];
    if (best == 0 || cost < least) {
      best = t[0];
      least = cost;
    }
  }
  return best;
}

// ---- a few keys ------------------------------------------------------------------------------------
//
// Up to kRankSort pairs: a pair's place is the number of pairs that come before it, which kRankParts threads
// count, one launch. Bound: a launch and a block's read of all keys; the histogram and four or eight passes are a
// chain of launches. 32-bit / 64-bit keys, passes and this: 500 pairs 20.2 / 38.6 and 2.3 / 2.6 us, 2,048
// 21.6 / 42.0 and 3.3 / 4.1, 4,096 28.0 / 48.9 and 7.3 / 9.5 (with four threads a pair 36 / 42).
constexpr uint32_t kRankSort = 4096;
constexpr uint32_t kRankThreads = 256, kRankParts = 16;

template <typename K>
__global__ void __launch_bounds__((int)kRankThreads) rank_sort_kernel(const K *__restrict__ keysIn, K *__restrict__ keysOut,
                                                                 const uint32_t *__restrict__ valsIn,
                                                                 uint32_t *__restrict__ valsOut, uint32_t n,
                                                                 uint32_t beginBit, K mask, uint32_t *err) {
  constexpr uint32_t kVec = 16 / sizeof(K);  // keys in a load
  __shared__ __align__(16) K digits[kRankSort];
  constexpr uint32_t kStep = kRankParts * kVec;
  const uint32_t part = threadIdx.x % kRankParts, e = (blockIdx.x * kRankThreads + threadIdx.x) / kRankParts;
  if (blockIdx.x == 0 && threadIdx.x == 0) *err = 0u;
  // Padding comes after every pair: no digit is higher, and its place is.
  const uint32_t padded = (n + kStep - 1) / kStep * kStep;  // at most kRankSort
  for (uint32_t j = threadIdx.x; j < padded; j += kRankThreads) digits[j] = j < n ? (__ldg(keysIn + j) >> beginBit) & mask : ~(K)0;
  __syncthreads();
  const bool live = e < n;
  const K mine = live ? digits[e] : (K)0;
  uint32_t before = 0;
#pragma unroll 4
  for (uint32_t j0 = part * kVec; j0 < padded; j0 += kStep) {
    K k[kVec];
    *reinterpret_cast<uint4 *>(k) = *reinterpret_cast<const uint4 *>(digits + j0);
#pragma unroll
    for (uint32_t q = 0; q < kVec; ++q) before += k[q] < mine || (k[q] == mine && j0 + q < e) ? 1u : 0u;
  }
#pragma unroll
  for (uint32_t o = 1; o < kRankParts; o <<= 1) before += __shfl_xor_sync(0xFFFFFFFFu, before, o);
  if (!live || part != 0) return;
  keysOut[before] = __ldg(keysIn + e);
  valsOut[before] = __ldg(valsIn + e);
}

// In and out arrays that share memory: the counting sort's blocks read all keys while others write, and one tile of
// the largest shape reads everything before it writes where several small ones would not.
bool shares_memory(const void *in, const void *out, size_t inBytes, size_t outBytes) {
  const auto a = reinterpret_cast<uintptr_t>(in), b = reinterpret_cast<uintptr_t>(out);
  return a < b + outBytes && b < a + inBytes;
}

template <typename K>
int sort_impl(void *temp, uint32_t tileKeys, const K *keysIn, K *keysOut, const uint32_t *valsIn, uint32_t *valsOut,
              uint32_t n, uint32_t beginBit, uint32_t endBit, cudaStream_t s) {
  const size_t keyBytes = sizeof(K) * (size_t)n, valBytes = 4 * (size_t)n;
  const bool shared = shares_memory(keysIn, keysOut, keyBytes, keyBytes) || shares_memory(keysIn, valsOut, keyBytes, valBytes) ||
                      shares_memory(valsIn, keysOut, valBytes, keyBytes) || shares_memory(valsIn, valsOut, valBytes, valBytes);
  if (tileKeys == 0) tileKeys = shared ? kSortTileDefault : auto_tile(n);
  const Layout L = make_layout(n, sizeof(K), beginBit, endBit, tileKeys);
  const Layout Lmax = make_layout(n, sizeof(K), beginBit, endBit, kMinTile);  // the temp space's layout
  char *t = static_cast<char *>(temp);
  uint32_t *hist = reinterpret_cast<uint32_t *>(t + Lmax.hist);
  uint32_t *counters = reinterpret_cast<uint32_t *>(t + Lmax.counters);
  uint32_t *err = reinterpret_cast<uint32_t *>(t + Lmax.err);
  uint32_t *status = reinterpret_cast<uint32_t *>(t + Lmax.status);
  K *altK = reinterpret_cast<K *>(t + Lmax.altKeys);
  uint32_t *altV = reinterpret_cast<uint32_t *>(t + Lmax.altVals);
  if (n == 0) return BVHGB_OK;
  if (L.passes == 0) {
    BVHGB_CUDA_TRY(cudaMemcpyAsync(keysOut, keysIn, sizeof(K) * n, cudaMemcpyDeviceToDevice, s));
    BVHGB_CUDA_TRY(cudaMemcpyAsync(valsOut, valsIn, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s));
    return BVHGB_OK;
  }
  if (tileKeys == (uint32_t)kMinTile && n <= kRankSort && !shared) {
    const K mask = endBit - beginBit >= 8 * sizeof(K) ? ~(K)0 : ((K)1 << (endBit - beginBit)) - 1;
    rank_sort_kernel<K><<<ceil_div(n, kRankThreads / kRankParts), kRankThreads, 0, s>>>(keysIn, keysOut, valsIn, valsOut, n,
                                                                              beginBit, mask, err);
    BVHGB_LAUNCH_CHECK("rank sort");
    return BVHGB_OK;
  }
  // hist, counters, err and the status words this tile size uses start at zero
  const size_t zeroed = Lmax.status + sizeof(uint32_t) * kRadix * (size_t)L.tiles * L.passes;
  BVHGB_CUDA_TRY(cudaMemsetAsync(t, 0, zeroed, s));
  int st = sort_prepare();
  if (st) return st;
  return sort_passes<K>(L, tileKeys, keysIn, keysOut, valsIn, valsOut, altK, altV, hist, counters, status, err, n,
                        beginBit, endBit, s, true);
}

// ---- 63-bit Morton keys -----------------------------------------------------------------------------
//
// sort_morton: the stable order of 63-bit keys from passes over their upper 32 or 40 bits only and one
// kernel that puts the groups with equal upper bits in order: a group's members stand in their
// original order, so a member's place is the number of members with a lower key, or an equal one and
// an earlier position, and every member counts that for itself. A mesh leaves few triangles in one
// cell of the upper bits; a group of more than kMaxGroup raises the gate, and the full eight-pass
// sort, whose launch otherwise returns at once, makes the order instead. Measured, launched one after the
// other (65,536 keys / 262,144 / 1M / 4.19M / 33.5M): 55 / 65 / 96 / 225 / 1,822 us; eight passes over tiles of 8,192 keys,
// one per SM, as the sort was before this: 120 / 129 / 150 / 442 / 2,855.
//
// Where a cell is that full (a detailed object in a large scene), the passes over the upper bits would be
// for nothing, so the kernel that makes the keys samples its cells (MortonCells) and a full one sends all keys to
// the full sort at once. With a quarter of the triangles in one cell, before / sampled / the eight passes as
// they were: 65,536 keys 182 / 110 / 127 us, 1M 317 / 180 / 154, 4.19M 687 / 435 / 445, 16.8M 2,647 / 1,531 / 1,471.
constexpr int kGroupTile = 1024;  // keys per block, 256 threads
constexpr int kMaxGroup = 256;

__global__ void __launch_bounds__(256) order_groups_kernel(const uint64_t *__restrict__ keys,
                                                           const uint32_t *__restrict__ vals, uint32_t n,
                                                           uint32_t beginBit, uint64_t *__restrict__ keysOut,
                                                           uint32_t *__restrict__ valsOut, uint32_t *gate,
                                                           const uint32_t *skip) {
  if (skipped(skip)) return;
  constexpr int kSpan = kGroupTile + kMaxGroup;
  __shared__ uint64_t key[kSpan + 1];  // [e + 1]: the tile's keys and the halo behind it; [0]: the key before the tile
  const uint32_t base = blockIdx.x * kGroupTile;
  const int valid = (int)min((uint32_t)kSpan, n - base);
  const bool first = base == 0;
  for (int e = (int)threadIdx.x - 1; e < valid; e += 256)
    if (e >= 0 || !first) key[e + 1] = __ldg(keys + base + e);
  __syncthreads();
  const uint64_t last = key[min(kGroupTile, valid)] >> beginBit;  // the tile's last group, which the halo may go on with
  for (int e = threadIdx.x; e < valid; e += 256) {
    const uint64_t mine = key[e + 1], u = mine >> beginBit;
    if (e >= kGroupTile && u != last) break;  // sorted: no later one either
    int lo = e, hi = e + 1;
    while (lo > 0 && key[lo] >> beginBit == u && e - lo <= kMaxGroup) --lo;
    if (lo == 0 && !first && key[0] >> beginBit == u && e <= kMaxGroup) continue;  // an earlier tile's group, which orders it
    while (hi < valid && hi - lo <= kMaxGroup && key[hi + 1] >> beginBit == u) ++hi;  // the halo is as long as a group may be
    if (hi - lo > kMaxGroup) {
      *gate = 1u;
      continue;
    }
    int at = lo;
    for (int j = lo; j < hi; ++j) at += key[j + 1] < mine || (key[j + 1] == mine && j < e) ? 1 : 0;
    keysOut[base + at] = mine;
    valsOut[base + at] = __ldg(vals + base + e);
  }
}

// The full sort of 63-bit keys behind the gate: every step in one cooperative launch, which returns at
// once where the gate is closed (a chain of ten launches that did so took 22 us of a 4.19M build, this
// one 2.5). The blocks, all resident, meet at bounded barriers between the steps.
struct FullSort {
  const uint64_t *keysIn;
  const uint32_t *valsIn;
  uint64_t *keysOut, *altK;
  uint32_t *valsOut, *altV, *words, *hist, *counters, *status, *err, *barrier;
  uint32_t n, tiles, passes, zeroed;  // words[0, zeroed) are cleared, but for the error and barrier words
  uint32_t *gate, *heavy;  // both 0 between sorts
  uint32_t *route;         // receives what they were
};

__device__ __forceinline__ bool grid_barrier(const FullSort &f, uint32_t target) {
  int ok = 1;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(f.barrier, 1u);
    for (uint32_t spins = 0; ld_relaxed(f.barrier) < target; ++spins) {
      if (spins > kSpinLimit) {
        atomicOr(f.err, kErrTimeout);
        ok = 0;
        break;
      }
      __nanosleep(32);
    }
    __threadfence();
  }
  return __syncthreads_and(ok) != 0;
}

template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS, kSortCtas<ITEMS>) full_sort_kernel(const __grid_constant__ FullSort f) {
  const bool gate = __ldcg(f.gate) != 0u, heavy = skipped(f.heavy);
  if (blockIdx.x == 0 && threadIdx.x == 0) *f.route = heavy ? 2u : gate ? 1u : 0u;
  if (!gate && !heavy) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  auto &sm = *reinterpret_cast<OnesweepSmem<uint64_t, THREADS, ITEMS> *>(smraw);
  uint32_t *sh = reinterpret_cast<uint32_t *>(smraw);
  static_assert(sizeof(sm) >= 8 * kRadix * sizeof(uint32_t), "room for the histograms of eight passes");
  uint32_t met = 0;
  for (uint32_t i = blockIdx.x * THREADS + threadIdx.x; i < f.zeroed; i += gridDim.x * THREADS)
    if (f.words + i != f.err && f.words + i != f.barrier) f.words[i] = 0u;
  if (!grid_barrier(f, met += gridDim.x)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {  // every block has read them: closed for the next sort
    *f.gate = 0u;
    if (f.heavy) *f.heavy = 0u;
  }
  histogram_all(f.keysIn, f.n, 0u, 63u, f.passes, f.hist, sh);
  if constexpr (!kScans<THREADS>) {
    if (!grid_barrier(f, met += gridDim.x)) return;
    // Exclusive scans, a pass per block (or more): one warp, eight digits a lane.
    for (uint32_t p = blockIdx.x; p < f.passes && threadIdx.x < 32u; p += gridDim.x) {
      uint32_t v[kRadix / 32], sum = 0;
#pragma unroll
      for (int q = 0; q < kRadix / 32; ++q) sum += v[q] = __ldcg(f.hist + p * kRadix + threadIdx.x * (kRadix / 32) + q);
      uint32_t at = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, at, o);
        if (threadIdx.x >= (uint32_t)o) at += y;
      }
      at -= sum;
#pragma unroll
      for (int q = 0; q < kRadix / 32; ++q) {
        f.hist[p * kRadix + threadIdx.x * (kRadix / 32) + q] = at;
        at += v[q];
      }
    }
  }
  const uint64_t *srcK = f.keysIn;
  const uint32_t *srcV = f.valsIn;
  for (uint32_t p = 0; p < f.passes; ++p) {
    if (!grid_barrier(f, met += gridDim.x)) return;
    const bool toOut = (f.passes - 1 - p) % 2 == 0;
    uint64_t *dstK = toOut ? f.keysOut : f.altK;
    uint32_t *dstV = toOut ? f.valsOut : f.altV;
    onesweep_tiles<uint64_t, THREADS, ITEMS, true>(sm, srcK, dstK, srcV, dstV, f.n, f.tiles, 8 * p, digit_mask(8 * p, 63u),
                                             f.hist + p * kRadix, f.counters + p,
                                             f.status + (size_t)p * f.tiles * kRadix, f.err);
    srcK = dstK;
    srcV = dstV;
  }
}

template <int THREADS, int ITEMS>
int launch_full_sort(const FullSort &f, cudaStream_t s) {
  int perSm = 0;
  const size_t smem = sizeof(OnesweepSmem<uint64_t, THREADS, ITEMS>);
  BVHGB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, full_sort_kernel<THREADS, ITEMS>, THREADS, smem));
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(std::min(f.tiles, (uint32_t)(perSm * sm_count())));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  BVHGB_CUDA_TRY(cudaLaunchKernelEx(&cfg, full_sort_kernel<THREADS, ITEMS>, f));
  BVHGB_LAUNCH_CHECK("full sort");
  return BVHGB_OK;
}

template <typename K, int THREADS, int ITEMS>
cudaError_t set_smem_attr() {
  return cudaFuncSetAttribute(onesweep_kernel<K, THREADS, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)sizeof(OnesweepSmem<K, THREADS, ITEMS>));
}

}  // namespace

int sort_prepare() {
  // Opt in to more than 48 KB of dynamic shared memory. The attribute belongs to the context, so it
  // is set once per context (another device, or the context after a device reset, sets it again);
  // the first call on a context must come before any stream capture. Thread-safe.
  static std::mutex m;
  static std::vector<uint64_t> done;
  const uint64_t ctx = context_id();
  std::lock_guard<std::mutex> lock(m);
  if (ctx != 0 && std::find(done.begin(), done.end(), ctx) != done.end()) return BVHGB_OK;
  BVHGB_CUDA_TRY((set_smem_attr<uint32_t, 256, 8>()));
  BVHGB_CUDA_TRY((set_smem_attr<uint32_t, 256, 16>()));
  BVHGB_CUDA_TRY((set_smem_attr<uint32_t, 512, 12>()));
  BVHGB_CUDA_TRY((set_smem_attr<uint32_t, 512, 14>()));
  BVHGB_CUDA_TRY((set_smem_attr<uint32_t, 512, 16>()));
  BVHGB_CUDA_TRY((set_smem_attr<uint64_t, 256, 8>()));
  BVHGB_CUDA_TRY((set_smem_attr<uint64_t, 256, 16>()));
  BVHGB_CUDA_TRY((set_smem_attr<uint64_t, 512, 12>()));
  BVHGB_CUDA_TRY((set_smem_attr<uint64_t, 512, 14>()));
  BVHGB_CUDA_TRY((set_smem_attr<uint64_t, 512, 16>()));
  BVHGB_CUDA_TRY(cudaFuncSetAttribute(full_sort_kernel<256, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(OnesweepSmem<uint64_t, 256, 8>)));
  BVHGB_CUDA_TRY(cudaFuncSetAttribute(full_sort_kernel<512, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(OnesweepSmem<uint64_t, 512, 16>)));
  if (ctx != 0) done.push_back(ctx);
  return BVHGB_OK;
}

int sort_set_spin_limit(uint32_t limit, uint32_t *previous) {
  uint32_t old = 0;
  BVHGB_CUDA_TRY(cudaMemcpyFromSymbol(&old, g_lookback_spin_limit, sizeof(old)));
  const uint32_t v = limit == 0xFFFFFFFFu ? kSpinLimit : limit;
  BVHGB_CUDA_TRY(cudaMemcpyToSymbol(g_lookback_spin_limit, &v, sizeof(v)));
  if (previous) *previous = old;
  return BVHGB_OK;
}

bool sort_tile_valid(uint32_t tileKeys) { return tileKeys == 2048 || tileKeys == 4096 || tileKeys == 8192; }

size_t sort_temp_bytes(uint32_t n, uint32_t keyBytes, uint32_t beginBit, uint32_t endBit) {
  return make_layout(n, keyBytes, beginBit, endBit).total;
}

uint32_t *sort_error_word(void *temp, uint32_t n, uint32_t keyBytes, uint32_t beginBit, uint32_t endBit) {
  Layout L = make_layout(n, keyBytes, beginBit, endBit);
  return reinterpret_cast<uint32_t *>(static_cast<char *>(temp) + L.err);
}

int sort_morton(void *temp, const uint64_t *keysIn, uint64_t *keysOut, const uint32_t *valsIn, uint32_t *valsOut,
                uint32_t n, uint32_t *gate, uint32_t *route, const MortonCells &cells, cudaStream_t s) {
  int st = sort_prepare();
  if (st) return st;
  if (n == 0) return BVHGB_OK;
  if (n <= kRankSort) return sort_impl<uint64_t>(temp, 0, keysIn, keysOut, valsIn, valsOut, n, 0, 63, s);
  const uint32_t beginBit = morton_cell_bit(n);
  const uint32_t tileKeys = auto_tile(n);
  const Layout L = make_layout(n, 8, beginBit, 63, tileKeys);
  const Layout Lmax = make_layout(n, 8, 0, 63, kMinTile);  // the temp space's layout
  char *t = static_cast<char *>(temp);
  uint32_t *hist = reinterpret_cast<uint32_t *>(t + Lmax.hist);
  uint32_t *counters = reinterpret_cast<uint32_t *>(t + Lmax.counters);
  uint32_t *err = reinterpret_cast<uint32_t *>(t + Lmax.err);
  uint32_t *status = reinterpret_cast<uint32_t *>(t + Lmax.status);
  uint64_t *altK = reinterpret_cast<uint64_t *>(t + Lmax.altKeys);
  uint32_t *altV = reinterpret_cast<uint32_t *>(t + Lmax.altVals);
  BVHGB_CUDA_TRY(cudaMemsetAsync(t, 0, Lmax.status + sizeof(uint32_t) * kRadix * (size_t)L.tiles * L.passes, s));
  st = sort_passes<uint64_t>(L, tileKeys, keysIn, keysOut, valsIn, valsOut, altK, altV, hist, counters, status, err, n,
                             beginBit, 63, s, false, cells);
  if (st) return st;
  order_groups_kernel<<<ceil_div(n, kGroupTile), 256, 0, s>>>(altK, altV, n, beginBit, keysOut, valsOut, gate,
                                                                    cells.heavy);
  BVHGB_LAUNCH_CHECK("order groups");
  // The full sort, in small tiles or in large ones.
  const bool small = tileKeys == (uint32_t)kMinTile;
  const Layout F = make_layout(n, 8, 0, 63, small ? kMinTile : 8192);
  const FullSort f{keysIn, valsIn, keysOut, altK, valsOut, altV, reinterpret_cast<uint32_t *>(t), hist, counters, status,
                   err, err + 1, n, F.tiles, F.passes,
                   (uint32_t)(Lmax.status / 4 + kRadix * (size_t)F.tiles * F.passes), gate, cells.heavy, route};
  return small ? launch_full_sort<256, 8>(f, s) : launch_full_sort<512, 16>(f, s);
}

void *sort_alternate(void *temp, uint32_t n, uint32_t keyBytes, uint32_t beginBit, uint32_t endBit) {
  return static_cast<char *>(temp) + make_layout(n, keyBytes, beginBit, endBit).altKeys;
}

int sort_pairs(void *temp, const void *keysIn, void *keysOut, const uint32_t *valsIn, uint32_t *valsOut, uint32_t n,
               uint32_t keyBytes, uint32_t beginBit, uint32_t endBit, cudaStream_t s, uint32_t tileKeys) {
  if (keyBytes == 4)
    return sort_impl<uint32_t>(temp, tileKeys, static_cast<const uint32_t *>(keysIn), static_cast<uint32_t *>(keysOut),
                               valsIn, valsOut, n, beginBit, endBit, s);
  return sort_impl<uint64_t>(temp, tileKeys, static_cast<const uint64_t *>(keysIn), static_cast<uint64_t *>(keysOut),
                             valsIn, valsOut, n, beginBit, endBit, s);
}


// ---- stable selection of the k smallest keys ------------------------------------------------------
//
// The first k pairs of a stable ascending sort of (keys, vals), without sorting all n: a radix
// selection finds the k-th smallest key T (three histogram passes over 11, 11 and 10 bits, each
// counting only the keys that match the digits found so far), a stable compaction keeps the keys
// below T and, of those equal to T, the first ones in index order up to k in all, and the k kept
// pairs are sorted. The compaction keeps index order, so the stable sort of the kept pairs is the
// prefix of the stable sort of all pairs.
namespace {

constexpr uint32_t kSelBins = 2048;
constexpr uint32_t kSelTile = 4096;        // keys per compaction tile (256 threads x 16)
__host__ __device__ constexpr uint32_t sel_shift(int pass) { return pass == 0 ? 21u : pass == 1 ? 10u : 0u; }
__host__ __device__ constexpr uint32_t sel_bits(int pass) { return pass == 2 ? 10u : 11u; }

struct SelState {
  uint32_t prefix;  // the digits of T found so far
  uint32_t below;   // keys below every key with that prefix
};

struct SelLayout {
  size_t state, hist, tileLt, tileEq, keys, vals, keysOut, sortTemp, total;
  uint32_t tiles;
};

SelLayout make_sel_layout(uint32_t n, uint32_t k) {
  SelLayout L{};
  auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
  L.tiles = ceil_div(max(n, 1u), kSelTile);
  size_t o = 0;
  L.state = o; o = up(o + sizeof(SelState));
  L.hist = o; o = up(o + 4ull * kSelBins);
  L.tileLt = o; o = up(o + 4ull * L.tiles);
  L.tileEq = o; o = up(o + 4ull * L.tiles);
  L.keys = o; o = up(o + 4ull * k);
  L.vals = o; o = up(o + 4ull * k);
  L.keysOut = o; o = up(o + 4ull * k);
  L.sortTemp = o; o = up(o + sort_temp_bytes(k, 4, 0, 32));
  L.total = o;
  return L;
}

// Histogram of digit 'pass' of the keys whose higher digits equal the prefix found so far (the lanes
// of a warp with the same bin add together; the block's counts go out once).
__global__ void __launch_bounds__(512) select_hist_kernel(const uint32_t *__restrict__ keys, uint32_t n,
                                                          const SelState *__restrict__ st, uint32_t *__restrict__ hist,
                                                          int pass, bool vec) {
  __shared__ uint32_t sh[kSelBins];
  for (uint32_t b = threadIdx.x; b < kSelBins; b += blockDim.x) sh[b] = 0;
  __syncthreads();
  const uint32_t shift = sel_shift(pass), mask = (1u << sel_bits(pass)) - 1u, hi = shift + sel_bits(pass);
  const uint32_t prefix = pass ? st->prefix : 0u;
  const uint32_t lane = threadIdx.x & 31u;
  // Four keys per thread and trip (one 16-byte load when the keys are 16-byte aligned).
  for (size_t base = (size_t)blockIdx.x * blockDim.x * 4; base < n; base += (size_t)gridDim.x * blockDim.x * 4) {
    const size_t i0 = base + 4 * (size_t)threadIdx.x;  // warp-uniform loop
    uint32_t k4[4];
    if (vec && i0 + 4 <= n) {
      const uint4 q = __ldg(reinterpret_cast<const uint4 *>(keys + i0));
      k4[0] = q.x;
      k4[1] = q.y;
      k4[2] = q.z;
      k4[3] = q.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) k4[j] = i0 + j < n ? __ldg(keys + i0 + j) : 0u;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t bin = 0xFFFFFFFFu;
      if (i0 + j < n && (pass == 0 || (k4[j] >> hi) == prefix)) bin = (k4[j] >> shift) & mask;
      if (__ballot_sync(0xFFFFFFFFu, bin != 0xFFFFFFFFu) == 0u) continue;  // after the first pass, most warps
      const uint32_t peers = __match_any_sync(0xFFFFFFFFu, bin);
      if (bin != 0xFFFFFFFFu && (peers & ((1u << lane) - 1u)) == 0u) atomicAdd(&sh[bin], (uint32_t)__popc(peers));
    }
  }
  __syncthreads();
  for (uint32_t b = threadIdx.x; b < kSelBins; b += blockDim.x)
    if (sh[b]) atomicAdd(&hist[b], sh[b]);
}

// Block-wide exclusive sum (blocks of up to 1024 threads); *total receives the sum.
__device__ __forceinline__ uint32_t block_exclusive_sum(uint32_t v, uint32_t *warpSums, uint32_t &total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = (blockDim.x + 31u) >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= (uint32_t)o) inc += t;
  }
  if (lane == 31u) warpSums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < warps ? warpSums[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, wi, o);
      if (lane >= (uint32_t)o) wi += t;
    }
    warpSums[lane] = wi - w;
    if (lane == 31u) warpSums[32] = wi;
  }
  __syncthreads();
  total = warpSums[32];
  const uint32_t r = warpSums[warp] + inc - v;
  __syncthreads();  // warpSums may be reused
  return r;
}

// The bin of digit 'pass' that holds the k-th smallest key: the prefix and the count below it
// advance; the histogram is cleared for the next pass. One block of 1024 threads, 2 bins each.
__global__ void __launch_bounds__(1024) select_find_kernel(SelState *st, uint32_t *hist, uint32_t k, int pass) {
  __shared__ uint32_t warpSums[33];
  const uint32_t b0 = 2u * threadIdx.x;
  const uint32_t h0 = hist[b0], h1 = hist[b0 + 1];
  const uint32_t below = pass ? st->below : 0u, prefix = pass ? st->prefix : 0u;
  uint32_t total;
  const uint32_t ex = block_exclusive_sum(h0 + h1, warpSums, total);
  const uint32_t need = k - below;  // rank (from 1) of the wanted key among those with the prefix
  int bin = -1;
  uint32_t exb = 0;
  if (ex < need && need <= ex + h0) {
    bin = (int)b0;
    exb = ex;
  } else if (ex + h0 < need && need <= ex + h0 + h1) {
    bin = (int)b0 + 1;
    exb = ex + h0;
  }
  __syncthreads();  // every thread has read the state
  if (bin >= 0) {
    st->prefix = (prefix << sel_bits(pass)) | (uint32_t)bin;
    st->below = below + exb;
  }
  hist[b0] = 0u;
  hist[b0 + 1] = 0u;
}

// Per tile: keys below T and keys equal to T.
__global__ void __launch_bounds__(256) select_count_kernel(const uint32_t *__restrict__ keys, uint32_t n,
                                                           const SelState *__restrict__ st, uint32_t *__restrict__ tileLt,
                                                           uint32_t *__restrict__ tileEq) {
  __shared__ uint32_t warpSums[33];
  const uint32_t T = st->prefix;
  const size_t base = (size_t)blockIdx.x * kSelTile;
  uint32_t lt = 0, eq = 0;
  for (uint32_t j = threadIdx.x; j < kSelTile; j += blockDim.x) {
    const size_t i = base + j;
    if (i < n) {
      const uint32_t key = __ldg(keys + i);
      lt += key < T ? 1u : 0u;
      eq += key == T ? 1u : 0u;
    }
  }
  uint32_t totLt, totEq;
  block_exclusive_sum(lt, warpSums, totLt);
  block_exclusive_sum(eq, warpSums, totEq);
  if (threadIdx.x == 0) {
    tileLt[blockIdx.x] = totLt;
    tileEq[blockIdx.x] = totEq;
  }
}

// Exclusive prefix of both tile counts, in place (one block, any number of tiles).
__global__ void __launch_bounds__(1024) select_scan_kernel(uint32_t *tileLt, uint32_t *tileEq, uint32_t tiles) {
  __shared__ uint32_t warpSums[33];
  uint32_t carryLt = 0, carryEq = 0;
  for (uint32_t c = 0; c < tiles; c += blockDim.x) {
    const uint32_t t = c + threadIdx.x;
    const uint32_t lt = t < tiles ? tileLt[t] : 0u, eq = t < tiles ? tileEq[t] : 0u;
    uint32_t sumLt, sumEq;
    const uint32_t exLt = block_exclusive_sum(lt, warpSums, sumLt);
    const uint32_t exEq = block_exclusive_sum(eq, warpSums, sumEq);
    if (t < tiles) {
      tileLt[t] = carryLt + exLt;
      tileEq[t] = carryEq + exEq;
    }
    carryLt += sumLt;
    carryEq += sumEq;
  }
}

// The kept pairs in index order: key < T, or key == T among the first (k - below) such keys. Each
// thread walks 16 consecutive keys; a key's place is (keys below T before it) + min(keys equal to
// T before it, k - below).
__global__ void __launch_bounds__(256) select_scatter_kernel(const uint32_t *__restrict__ keys,
                                                             const uint32_t *__restrict__ vals, uint32_t n, uint32_t k,
                                                             const SelState *__restrict__ st,
                                                             const uint32_t *__restrict__ offLt,
                                                             const uint32_t *__restrict__ offEq,
                                                             uint32_t *__restrict__ outKeys,
                                                             uint32_t *__restrict__ outVals, bool vec) {
  __shared__ uint32_t warpSums[33];
  constexpr uint32_t kPer = kSelTile / 256;
  const uint32_t T = st->prefix, need = k - st->below;
  const size_t first = (size_t)blockIdx.x * kSelTile + (size_t)threadIdx.x * kPer;
  uint32_t key[kPer];
  if (vec && first + kPer <= n) {  // 16-byte loads: keys 16-byte aligned, first a multiple of 16 keys
#pragma unroll
    for (uint32_t j = 0; j < kPer; j += 4) {
      const uint4 q = __ldg(reinterpret_cast<const uint4 *>(keys + first + j));
      key[j] = q.x;
      key[j + 1] = q.y;
      key[j + 2] = q.z;
      key[j + 3] = q.w;
    }
  } else {
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) key[j] = first + j < n ? __ldg(keys + first + j) : 0xFFFFFFFFu;
  }
  uint32_t lt = 0, eq = 0;
#pragma unroll
  for (uint32_t j = 0; j < kPer; ++j) {
    const bool live = first + j < n;
    lt += live && key[j] < T ? 1u : 0u;
    eq += live && key[j] == T ? 1u : 0u;
  }
  uint32_t totLt, totEq;
  uint32_t ltBefore = offLt[blockIdx.x] + block_exclusive_sum(lt, warpSums, totLt);
  uint32_t eqBefore = offEq[blockIdx.x] + block_exclusive_sum(eq, warpSums, totEq);
#pragma unroll
  for (uint32_t j = 0; j < kPer; ++j) {
    if (first + j >= n) break;
    if (key[j] < T) {
      const uint32_t pos = ltBefore + min(eqBefore, need);
      if (pos < k) {  // always, unless the keys changed between the passes
        outKeys[pos] = key[j];
        outVals[pos] = __ldg(vals + first + j);
      }
      ++ltBefore;
    } else if (key[j] == T) {
      const uint32_t pos = ltBefore + eqBefore;
      if (eqBefore < need && pos < k) {
        outKeys[pos] = key[j];
        outVals[pos] = __ldg(vals + first + j);
      }
      ++eqBefore;
    }
  }
}

}  // namespace

size_t select_temp_bytes(uint32_t n, uint32_t k) { return make_sel_layout(n, min(k, n)).total; }

int select_smallest(void *temp, const uint32_t *keys, const uint32_t *vals, uint32_t n, uint32_t k, uint32_t *valsOut,
                    cudaStream_t s, uint32_t tileKeys) {
  k = min(k, n);
  if (k == 0) return BVHGB_OK;
  const SelLayout L = make_sel_layout(n, k);
  char *t = static_cast<char *>(temp);
  SelState *st = reinterpret_cast<SelState *>(t + L.state);
  uint32_t *hist = reinterpret_cast<uint32_t *>(t + L.hist);
  uint32_t *tileLt = reinterpret_cast<uint32_t *>(t + L.tileLt);
  uint32_t *tileEq = reinterpret_cast<uint32_t *>(t + L.tileEq);
  uint32_t *ck = reinterpret_cast<uint32_t *>(t + L.keys);
  uint32_t *cv = reinterpret_cast<uint32_t *>(t + L.vals);
  uint32_t *ko = reinterpret_cast<uint32_t *>(t + L.keysOut);
  if (k == n) return sort_pairs(t + L.sortTemp, keys, ko, vals, valsOut, n, 4, 0, 32, s, tileKeys);
  BVHGB_CUDA_TRY(cudaMemsetAsync(hist, 0, 4ull * kSelBins, s));
  const bool vec = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0u;
  const uint32_t hgrid = min(ceil_div(n, 512u * 4u), (uint32_t)sm_count() * 4);
  for (int pass = 0; pass < 3; ++pass) {
    select_hist_kernel<<<hgrid, 512, 0, s>>>(keys, n, st, hist, pass, vec);
    BVHGB_LAUNCH_CHECK("select histogram");
    select_find_kernel<<<1, kSelBins / 2, 0, s>>>(st, hist, k, pass);
    BVHGB_LAUNCH_CHECK("select find");
  }
  select_count_kernel<<<L.tiles, 256, 0, s>>>(keys, n, st, tileLt, tileEq);
  BVHGB_LAUNCH_CHECK("select count");
  select_scan_kernel<<<1, 1024, 0, s>>>(tileLt, tileEq, L.tiles);
  BVHGB_LAUNCH_CHECK("select scan");
  select_scatter_kernel<<<L.tiles, 256, 0, s>>>(keys, vals, n, k, st, tileLt, tileEq, ck, cv, vec);
  BVHGB_LAUNCH_CHECK("select scatter");
  return sort_pairs(t + L.sortTemp, ck, ko, cv, valsOut, k, 4, 0, 32, s, tileKeys);
}

// ---- the selection over many segments --------------------------------------------------------------
//
// select_smallest's steps, a block per tile of one segment, thresholds and counts per segment. The
// first histogram (of the upper 11 bits) comes from the kernel that makes the keys. Bound: reading the
// keys four times (20M keys in 256 segments: histograms 40 us each, counts 20, scatter 38; the stable
// sort of all of them by segment and key took 1,130).
namespace {

__global__ void __launch_bounds__(kSegThreads) seg_hist_kernel(SegSelect q, const uint32_t *__restrict__ keys,
                                                               uint32_t *__restrict__ hist, int pass) {
  __shared__ uint32_t sh[kSegBins];
  const SegTile t = q.tile[blockIdx.x];
  const uint32_t row = q.row[t.seg];
  if (row == kNone) return;
  for (uint32_t b = threadIdx.x; b < kSegBins; b += kSegThreads) sh[b] = 0;
  __syncthreads();
  const uint32_t shift = sel_shift(pass), mask = (1u << sel_bits(pass)) - 1u, hi = shift + sel_bits(pass);
  const uint32_t prefix = q.state[row].x;
  for (uint32_t base = 0; base < t.len; base += kSegThreads) {
    const uint32_t j = base + threadIdx.x;
    uint32_t bin = 0xFFFFFFFFu;
    if (j < t.len) {
      const uint32_t key = __ldg(keys + t.start + j);
      if ((key >> hi) == prefix) bin = (key >> shift) & mask;
    }
    if (__ballot_sync(0xFFFFFFFFu, bin != 0xFFFFFFFFu) != 0u) count_bin(sh, bin);  // most warps have none
  }
  __syncthreads();
  for (uint32_t b = threadIdx.x; b < kSegBins; b += kSegThreads)
    if (sh[b]) atomicAdd(&hist[(size_t)row * kSegBins + b], sh[b]);
}

__global__ void __launch_bounds__(kSegBins / 2) seg_find_kernel(SegSelect q, uint32_t *__restrict__ hist, int pass) {
  __shared__ uint32_t warpSums[33];
  const uint32_t row = blockIdx.x, b0 = 2u * threadIdx.x;
  uint32_t *h = hist + (size_t)row * kSegBins;
  const uint32_t h0 = h[b0], h1 = h[b0 + 1];
  const uint2 st = pass ? q.state[row] : make_uint2(0u, 0u);
  uint32_t total;
  const uint32_t ex = block_exclusive_sum(h0 + h1, warpSums, total);  // its barriers: every thread has read the state
  const uint32_t need = q.keep[q.rowSeg[row]] - st.y;  // rank (from 1) of the wanted key among those with the prefix
  if (ex < need && need <= ex + h0) q.state[row] = make_uint2((st.x << sel_bits(pass)) | b0, st.y + ex);
  else if (ex + h0 < need && need <= ex + h0 + h1) q.state[row] = make_uint2((st.x << sel_bits(pass)) | (b0 + 1u), st.y + ex + h0);
  h[b0] = h[b0 + 1] = 0u;
}

__global__ void __launch_bounds__(kSegThreads) seg_count_kernel(SegSelect q, const uint32_t *__restrict__ keys) {
  __shared__ uint32_t warpSums[33];
  const SegTile t = q.tile[blockIdx.x];
  const uint32_t row = q.row[t.seg];
  if (row == kNone) {
    if (threadIdx.x == 0) q.count[blockIdx.x] = make_uint2(t.len, 0u);
    return;
  }
  const uint32_t T = q.state[row].x;
  uint32_t c = 0;  // at T: upper half (a tile has at most kSegTile of either)
  for (uint32_t j = threadIdx.x; j < t.len; j += kSegThreads) {
    const uint32_t key = __ldg(keys + t.start + j);
    c += (key < T ? 1u : 0u) + (key == T ? 1u << 16 : 0u);
  }
  uint32_t total;
  block_exclusive_sum(c, warpSums, total);
  if (threadIdx.x == 0) q.count[blockIdx.x] = make_uint2(total & 0xFFFFu, total >> 16);
}

// Exclusive prefixes of a segment's tile counts, in place, one block per segment.
__global__ void __launch_bounds__(256) seg_scan_kernel(SegSelect q) {
  __shared__ uint32_t warpSums[33];
  const uint32_t first = q.tileOff[blockIdx.x], last = q.tileOff[blockIdx.x + 1];
  uint2 carry = make_uint2(0u, 0u);
  for (uint32_t c = first; c < last; c += 256u) {
    const uint32_t i = c + threadIdx.x;
    const uint2 v = i < last ? q.count[i] : make_uint2(0u, 0u);
    uint32_t sumLt, sumEq;
    const uint32_t lt = block_exclusive_sum(v.x, warpSums, sumLt), eq = block_exclusive_sum(v.y, warpSums, sumEq);
    if (i < last) q.count[i] = make_uint2(carry.x + lt, carry.y + eq);
    carry.x += sumLt;
    carry.y += sumEq;
  }
}

__global__ void __launch_bounds__(kSegThreads) seg_scatter_kernel(SegSelect q, const uint32_t *__restrict__ keys,
                                                                  uint64_t *__restrict__ outKeys,
                                                                  uint32_t *__restrict__ outVals) {
  __shared__ uint32_t warpSums[33];
  constexpr uint32_t kPer = kSegTile / kSegThreads;
  const SegTile t = q.tile[blockIdx.x];
  const uint32_t row = q.row[t.seg], keep = q.keep[t.seg], out = q.outOff[t.seg];
  const uint64_t high = (uint64_t)t.seg << 32;
  uint2 before = q.count[blockIdx.x];
  if (row == kNone) {
    for (uint32_t j = threadIdx.x; j < t.len; j += kSegThreads) {
      outKeys[out + before.x + j] = high | __ldg(keys + t.start + j);
      outVals[out + before.x + j] = t.local + j;
    }
    return;
  }
  const uint2 st = q.state[row];
  const uint32_t T = st.x, need = keep - st.y;
  // A warp takes 32 consecutive keys at a time, a thread's 16 are 32 apart: a lane's place among the
  // warp's keys comes from ballots.
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, ltMask = (1u << lane) - 1u;
  const uint32_t j0 = warp * 32u * kPer + lane;
  uint32_t key[kPer], c = 0;
#pragma unroll
  for (uint32_t j = 0; j < kPer; ++j) {
    const bool live = j0 + 32u * j < t.len;
    key[j] = live ? __ldg(keys + t.start + j0 + 32u * j) : 0xFFFFFFFFu;
    c += (live && key[j] < T ? 1u : 0u) + (live && key[j] == T ? 1u << 16 : 0u);
  }
  // The counts before this warp: lane 0's place in the block's order of (warp, lane).
  uint32_t total;
  const uint32_t ex = block_exclusive_sum(c, warpSums, total);
  const uint32_t warpEx = __shfl_sync(0xFFFFFFFFu, ex, 0);
  before.x += warpEx & 0xFFFFu;
  before.y += warpEx >> 16;
#pragma unroll
  for (uint32_t j = 0; j < kPer; ++j) {
    const bool live = j0 + 32u * j < t.len;
    const bool lt = live && key[j] < T, eq = live && key[j] == T;
    const uint32_t lts = __ballot_sync(0xFFFFFFFFu, lt), eqs = __ballot_sync(0xFFFFFFFFu, eq);
    const uint32_t myLt = before.x + __popc(lts & ltMask), myEq = before.y + __popc(eqs & ltMask);
    if (lt || (eq && myEq < need)) {
      const uint32_t pos = myLt + min(myEq, need);
      if (pos < keep) {  // always, unless the keys changed between the passes
        outKeys[out + pos] = high | key[j];
        outVals[out + pos] = t.local + j0 + 32u * j;
      }
    }
    before.x += __popc(lts);
    before.y += __popc(eqs);
  }
}

}  // namespace

int select_segments(const SegSelect &q, const uint32_t *keys, uint32_t *hist, uint64_t *outKeys, uint32_t *outVals,
                    cudaStream_t s) {
  static_assert(kSegBins == 1u << sel_bits(0) && kSegTile < 1u << 16, "one digit per row, counts in 16 bits");
  if (q.rows) {
    for (int pass = 0; pass < 3; ++pass) {
      if (pass) {
        seg_hist_kernel<<<q.tiles, kSegThreads, 0, s>>>(q, keys, hist, pass);
        BVHGB_LAUNCH_CHECK("segment histogram");
      }
      seg_find_kernel<<<q.rows, kSegBins / 2, 0, s>>>(q, hist, pass);
      BVHGB_LAUNCH_CHECK("segment find");
    }
  }
  seg_count_kernel<<<q.tiles, kSegThreads, 0, s>>>(q, keys);
  BVHGB_LAUNCH_CHECK("segment count");
  seg_scan_kernel<<<q.segs, 256, 0, s>>>(q);
  BVHGB_LAUNCH_CHECK("segment scan");
  seg_scatter_kernel<<<q.tiles, kSegThreads, 0, s>>>(q, keys, outKeys, outVals);
  BVHGB_LAUNCH_CHECK("segment scatter");
  return BVHGB_OK;
}

}  // namespace bvhgb

extern "C" BVHGB_API int bvhgb_radix_sort_pairs(void *temp, size_t *tempBytes, const void *keysIn, void *keysOut,
                                                const uint32_t *valsIn, uint32_t *valsOut, uint32_t n,
                                                uint32_t keyBytes, uint32_t beginBit, uint32_t endBit,
                                                bvhgb_stream stream) {
  if (!tempBytes || (keyBytes != 4 && keyBytes != 8) || beginBit > endBit || endBit > 8 * keyBytes)
    return BVHGB_INVALID_ARGUMENT;
  if (n >= (1u << 30)) return BVHGB_TOO_LARGE;
  size_t need = bvhgb::sort_temp_bytes(n, keyBytes, beginBit, endBit);
  if (!temp) {
    *tempBytes = need;
    return BVHGB_OK;
  }
  if (*tempBytes < need || (n && (!keysIn || !keysOut || !valsIn || !valsOut))) return BVHGB_INVALID_ARGUMENT;
  return bvhgb::sort_pairs(temp, keysIn, keysOut, valsIn, valsOut, n, keyBytes, beginBit, endBit,
                           bvhgb::as_stream(stream));
}

extern "C" BVHGB_API int bvhgb_select_smallest_pairs(void *temp, size_t *tempBytes, const uint32_t *keys,
                                                     const uint32_t *vals, uint32_t *valsOut, uint32_t n, uint32_t k,
                                                     bvhgb_stream stream) {
  if (!tempBytes || k > n) return BVHGB_INVALID_ARGUMENT;
  if (n >= (1u << 30)) return BVHGB_TOO_LARGE;
  const size_t need = bvhgb::select_temp_bytes(n, k);
  if (!temp) {
    *tempBytes = need;
    return BVHGB_OK;
  }
  if (*tempBytes < need || (k && (!keys || !vals || !valsOut))) return BVHGB_INVALID_ARGUMENT;
  return bvhgb::select_smallest(temp, keys, vals, n, k, valsOut, bvhgb::as_stream(stream));
}

extern "C" BVHGB_API int bvhgb_sort_set_default_tile(uint32_t tileKeys, uint32_t *previous) {
  if (tileKeys != 0 && tileKeys != BVHGB_SORT_TILE_AUTO && !bvhgb::sort_tile_valid(tileKeys)) return BVHGB_INVALID_ARGUMENT;
  const uint32_t old = tileKeys ? bvhgb::g_default_tile.exchange(tileKeys) : bvhgb::g_default_tile.load();
  if (previous) *previous = old;
  return BVHGB_OK;
}

extern "C" BVHGB_API int bvhgb_sort_set_spin_limit(uint32_t limit, uint32_t *previous) {
  return bvhgb::sort_set_spin_limit(limit, previous);
}
