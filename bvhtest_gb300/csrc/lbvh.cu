// LBVH build: scene box, Morton codes, onesweep sort, and topology + refit block by block.
//
// Reference: lib/builder/LBVH_CUDA.cu. Kernel plan (HBM-bound, no tensor cores):
//   lbvh_bounds  : per-triangle box (+-FLT_EPSILON) reduced into the scene box, whose initial value
//                  is the origin box (LBVH_CUDA.cu:60-119). Reads faces + vertices once.
//   lbvh_morton  : re-reads the triangle, centroid -> 30- or 63-bit Morton key + index
//                  (LBVH_CUDA.cu:132-183); also resets the build's exchange slots and, when the
//                  workspace has them, writes each triangle's box as a 32-byte record in face order
//                  (the build then gathers one sector per leaf instead of a face and three vertices).
//   sort         : sort.cu (replaces cub::DeviceRadixSort, LBVH_CUDA.cu:185-193).
//   lbvh_build   : a block makes the inner nodes among its 256 sorted leaves in shared memory and lists
//                  the roots of its subtrees (treelet_build).
//   lbvh_join    : a block makes the nodes over 16 neighbouring lists of roots in the same way, launch by
//                  launch up to the tree's root.
//   lbvh_roots   : climbs from the lists that could not be joined (Apetrei 2014 style): at each step a
//                  climb picks the parent from the two neighbouring key deltas, meets its sibling through
//                  one acq_rel exchange on the split's slot, and the second to arrive merges the boxes
//                  and writes the parent.
//   lbvh_small   : all of it in one launch for up to 1,024 triangles.
//                  All give the nodes the Karras index the reference assigns (kGenLeafNodes +
//                  kBuildTree + kFixAABBTree, LBVH_CUDA.cu:273-374).
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "lbvh_device.cuh"
#include "sort.cuh"

struct bvhgb_lbvh_workspace {
  uint32_t maxFaces = 0;
  bvhgb_lbvh_config cfg{};
  uint32_t keyBytes = 4;
  uint32_t *scene = nullptr;  // 6 order-mapped floats, error word, (free), sort gate, heavy-cell flag, sort route
  bool sceneReady = false;    // they have been written
  bool sorted = false;        // the sort's error word has been
  void *keys = nullptr;
  void *keysSorted = nullptr;
  uint32_t *vals = nullptr;
  uint32_t *valsSorted = nullptr;
  uint32_t *slots = nullptr;
  float4 *triBoxes = nullptr;  // 2 x float4 per face (mn.xyz mx.x | mx.yz 0 0); null: gather the triangle
  bool slotsArmed = false;  // slots hold kNone (set by the Morton kernel)
  // Sampled counts of the Morton cells, 2^cellBits (63-bit keys; null: none). The Morton phase adds to them; the
  // kernel of the scene box clears them, and the Morton phase itself where that has not run since (in the same
  // capture, if any: 0 is none).
  uint32_t *cells = nullptr;
  uint32_t cellBits = 0;
  bool cellsClear = false;
  unsigned long long cellsClearIn = 0;
  void *sortTemp = nullptr;
  size_t sortTempBytes = 0;
};

namespace bvhgb {
namespace {

constexpr int kBoundsThreads = 256;
constexpr int kMortonThreads = 256;

constexpr uint32_t kSceneWords = 11;

__global__ void lbvh_init_kernel(uint32_t *scene) {
  if (threadIdx.x < 6) scene[threadIdx.x] = f2ord(0.0f);  // origin box [(0,0,0),(0,0,0)]
  else if (threadIdx.x < kSceneWords) scene[threadIdx.x] = 0;
}

__global__ void __launch_bounds__(kBoundsThreads) lbvh_bounds_kernel(const float *__restrict__ vert,
                                                                     const uint32_t *__restrict__ faces, uint32_t n,
                                                                     uint32_t *scene, uint32_t *__restrict__ cells,
                                                                     uint32_t cellWords) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cellWords; i += gridDim.x * blockDim.x) cells[i] = 0u;
  // Starting the local box at the origin is the same as merging the reduction's initial value.
  float mn[3] = {0.0f, 0.0f, 0.0f}, mx[3] = {0.0f, 0.0f, 0.0f};
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    Box b;
    tri_box(vert, faces, (uint32_t)i, b, nullptr);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      mn[k] = fminf(mn[k], b.mn[k]);
      mx[k] = fmaxf(mx[k], b.mx[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn[k] = fminf(mn[k], __shfl_xor_sync(0xFFFFFFFFu, mn[k], o));
      mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xFFFFFFFFu, mx[k], o));
    }
  }
  __shared__ float red[kBoundsThreads / 32][6];
  const uint32_t warp = threadIdx.x >> 5;
  if (lane_id() == 0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) { red[warp][k] = mn[k]; red[warp][3 + k] = mx[k]; }
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    float v = red[0][threadIdx.x];
    for (int w = 1; w < kBoundsThreads / 32; ++w)
      v = threadIdx.x < 3 ? fminf(v, red[w][threadIdx.x]) : fmaxf(v, red[w][threadIdx.x]);
    if (threadIdx.x < 3) atomicMin(&scene[threadIdx.x], f2ord(v));
    else atomicMax(&scene[threadIdx.x], f2ord(v));
  }
}

template <int BITS>
__global__ void __launch_bounds__(kMortonThreads) lbvh_morton_kernel(const float *__restrict__ vert,
                                                                     const uint32_t *__restrict__ faces, uint32_t n,
                                                                     uint32_t *__restrict__ scene, void *keysOut,
                                                                     uint32_t *__restrict__ vals,
                                                                     uint32_t *__restrict__ slots,
                                                                     float4 *__restrict__ boxes,
                                                                     uint32_t *__restrict__ cells, uint32_t cellBits) {
  float off[3], sc[3];
  morton_params(scene, off, sc);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    Box b;
    float c[3];
    tri_box(vert, faces, (uint32_t)i, b, c);
    if (BITS == 30) static_cast<uint32_t *>(keysOut)[i] = (uint32_t)morton_key<30>(c, off, sc);
    else {
      const uint64_t key = morton_key<63>(c, off, sc);
      static_cast<uint64_t *>(keysOut)[i] = key;
      if (cells && i % cell_sample(n) == 0) {
        const uint64_t h = (key >> morton_cell_bit(n)) * 0x9E3779B97F4A7C15ull;
        atomicAdd(cells + (h >> (64u - cellBits)), 1u);  // nobody waits for it
      }
    }
    vals[i] = (uint32_t)i;
    if (i + 1 < n) slots[i] = kNone;
    if (boxes) {
      boxes[2 * i] = make_float4(b.mn[0], b.mn[1], b.mn[2], b.mx[0]);
      boxes[2 * i + 1] = make_float4(b.mx[1], b.mx[2], 0.0f, 0.0f);
    }
  }
}

// ---- tree of a block of leaves ----------------------------------------------------------------------
//
// A block takes T consecutive sorted leaves, one per thread, and makes every inner node whose range
// lies among them, all at once: thread t finds the range [l, r] of the node that splits between
// leaves t and t + 1 (the leaves that share as long a prefix with it as its two neighbours do: a
// binary search in the block's keys, or a mask of the index in refCompat mode), its Karras index and
// its children, and takes its box from two overlapping windows of 2^j leaves (W_j[l] and
// W_j[r - 2^j + 1]); the windows double level by level, in the order the queries need them. The
// records are staged in shared memory and written in 16-byte words, neighbours together. What is
// left, the roots of the block's subtrees (about 2 log2 T of them, at most kTreeletRoots), goes to a
// list in leaf order for the joining launches below.
//
// Why: with one climb per leaf every inner node cost an acquire-release exchange, a sibling's box
// from L2 and three scattered stores in one dependent chain (4.19M leaves: 413 us at 24% of DRAM
// throughput; 33.5M: 3,050 us); here all but one node in seventeen costs none of them.
// Measured, block of 256 / 512 / 1,024 leaves: 182 / 209 / 295 us (33.5M, 256: 1,407 us), bound by
// shared memory's wavefronts (83%; DRAM 50%).
//
// Windows overlap, so a box is a plain minimum and maximum over its leaves. The climb's merge differs
// from that only where a coordinate is NaN (its result then depends on the order): a block with a NaN
// among its boxes merges the children's boxes node by node, in rounds.
constexpr int kTreelet = 256;
// Between two neighbouring roots of a block the delta is a strict prefix minimum of the block's deltas
// or a strict suffix minimum, and a delta is at most 96.
constexpr int kTreeletRoots = 193;

// Two buffers of T boxes, a component per array: neighbours' loads share a wavefront.
template <int T>
struct BoxPair {
  float v[2][6][T];
  __device__ __forceinline__ Box get(int buf, int i) const {
    Box x;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      x.mn[k] = v[buf][k][i];
      x.mx[k] = v[buf][3 + k][i];
    }
    return x;
  }
  __device__ __forceinline__ void put(int buf, int i, const Box &x) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      v[buf][k][i] = x.mn[k];
      v[buf][3 + k][i] = x.mx[k];
    }
  }
};

__device__ __forceinline__ bool has_nan(const Box &b) {
  bool nan = false;
#pragma unroll
  for (int k = 0; k < 3; ++k) nan = nan || isnan(b.mn[k]) || isnan(b.mx[k]);
  return nan;
}

template <int T, typename K>
struct TreeletSmem {
  union {
    BoxPair<T> box;          // window boxes, ping-pong
    float4 record[3 * T];    // node records on their way out
  };
  K key[T + 2];              // leaf B0 + i at [i + 1]
  uint32_t parInner[T], parLeaf[T];  // parent | is-left << 31 (an index has 31 bits); kNone: not in this block
  uint8_t gap[T + 1];        // delta of the leaves B0 + i - 1 and B0 + i
  uint8_t made[T];           // inner record i of the block is one of its own
  uint32_t starts[T / 32];   // bit i: a root of the block's subtrees starts at leaf B0 + i
};

// Boxes of ranges from windows of 1, 2, 4 ... boxes: thread t's range [l, r] (if it has one; cnt boxes, T
// threads) comes from the two windows of 2^j boxes that cover it. Buffer 0 holds the boxes, w thread t's own.
template <int T>
__device__ __forceinline__ void window_boxes(BoxPair<T> &box, int &top, int cnt, bool has, int l, int r, Box w, Box &nb) {
  const int t = (int)threadIdx.x;
  const int level = has ? 31 - __clz(r - l + 1) : -1;
  // The highest level any thread needs (block-uniform).
  if (t == 0) top = 0;
  __syncthreads();
  const int warpTop = __reduce_max_sync(0xFFFFFFFFu, level);
  if ((t & 31) == 0 && warpTop > 0) atomicMax(&top, warpTop);
  __syncthreads();
  const int levels = top;
  for (int j = 0; j < levels; ++j) {  // w: window W_j[t]
    const int half = 1 << j;
    const float(*cur)[T] = box.v[j & 1];
    float(*nxt)[T] = box.v[(j + 1) & 1];
    if (t + half < cnt) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        w.mn[k] = fminf(w.mn[k], cur[k][t + half]);
        w.mx[k] = fmaxf(w.mx[k], cur[3 + k][t + half]);
      }
    }
    if (t < cnt) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        nxt[k][t] = w.mn[k];
        nxt[3 + k][t] = w.mx[k];
      }
    }
    __syncthreads();
    if (level == j + 1) {
      const int e = r - 2 * half + 1;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        nb.mn[k] = fminf(nxt[k][l], nxt[k][e]);
        nb.mx[k] = fmaxf(nxt[3 + k][l], nxt[3 + k][e]);
      }
    }
  }
}

// Set bits below bit 'at' of a mask of W words.
template <int W>
__device__ __forceinline__ uint32_t ones_before(const uint32_t *mask, int at) {
  uint32_t p = __popc(mask[at >> 5] & ((1u << (at & 31)) - 1u));
#pragma unroll
  for (int w = 0; w < W; ++w) p += w < (at >> 5) ? __popc(mask[w]) : 0;
  return p;
}

// The block's leaves are B0 .. B0 + cnt - 1; every thread of the T calls it. key, box: the thread's leaf's
// (t < cnt). keys: the tree's sorted keys, read for the neighbouring blocks' leaves only (karras mode).
template <int MODE, int T, typename K>
__device__ __forceinline__ void treelet_build(TreeletSmem<T, K> &sm, uint32_t B0, uint32_t n, uint32_t face, const Box &box,
                                              K key, const K *__restrict__ keys, bvhgb_node *nodes,
                                              uint2 *__restrict__ roots, uint32_t *rootCount) {
  __shared__ int top;
  constexpr int kBits = 8 * (int)sizeof(K);
  const int t = (int)threadIdx.x;
  const int cnt = (int)min((uint32_t)T, n - B0);
  const bool live = t < cnt;
  const uint32_t i = B0 + (uint32_t)t;
  if (MODE == BVHGB_TOPO_KARRAS) {
    if (live) sm.key[t + 1] = key;
    if (t == 0 && B0 > 0) sm.key[0] = __ldg(keys + B0 - 1);
    if (t == 0 && B0 + cnt < n) sm.key[cnt + 1] = __ldg(keys + B0 + cnt);
  }
  sm.parInner[t] = sm.parLeaf[t] = kNone;
  sm.made[t] = 0;
  bool nan = false;
  if (live) {
    sm.box.put(0, t, box);
    nan = has_nan(box);
  }
  const bool ordered = __syncthreads_or(nan) != 0;
  // Deltas of the gaps around the block's leaves: gap g (local) at [g + 1], between leaves g and g + 1.
  auto pair_delta = [&](int a) {  // leaves a and a + 1 (local), both in the tree
    if (MODE == BVHGB_TOPO_REFCOMPAT) return __clz((int)((B0 + a) ^ (B0 + a + 1)));
    const K x = sm.key[a + 1] ^ sm.key[a + 2];
    if (x != 0) return sizeof(K) == 8 ? __clzll((long long)x) : __clz((int)x);
    return kBits + __clz((int)((B0 + a) ^ (B0 + a + 1)));
  };
  if (live && B0 + t + 1 < n) sm.gap[t + 1] = (uint8_t)pair_delta(t);
  if (t == 0 && B0 > 0) sm.gap[0] = (uint8_t)pair_delta(-1);
  __syncthreads();
  // The node of gap t: its range, if that lies in the block.
  int l = t, r = t;
  bool local = live && t + 1 < cnt;
  if (local) {
    const int d = sm.gap[t + 1];
    r = t + 1;
    if (MODE == BVHGB_TOPO_REFCOMPAT) {
      const uint32_t mask = (2u << (31 - d)) - 1u;  // the range is the aligned block of that size (31 - d < 31)
      const uint32_t gl = i & ~mask, gr = min(i | mask, n - 1u);
      local = gl >= B0 && gr < B0 + (uint32_t)cnt;
      l = (int)(gl - B0);
      r = (int)(gr - B0);
    } else {
      const K mine = sm.key[t + 1];
      const K bound = d < kBits ? (K)1 << (kBits - d) : (K)1;
      auto same = [&](int c) {  // leaf c shares d bits with this gap's leaves (c may be a halo leaf)
        if ((K)(sm.key[c + 1] ^ mine) >= bound) return false;
        return d < kBits || __clz((int)((B0 + c) ^ i)) >= d - kBits;
      };
#pragma unroll
      for (int step = T / 2; step > 0; step >>= 1) {
        if (l - step >= 0 && same(l - step)) l -= step;
        if (r + step < cnt && same(r + step)) r += step;
      }
      if (l == 0 && B0 > 0 && same(-1)) local = false;
      if (r == cnt - 1 && B0 + cnt < n && same(cnt)) local = false;
    }
  }
  const bool root = local && B0 + l == 0 && B0 + r == n - 1;
  bool right = false;  // the node is its parent's left child: the parent splits at r
  int slot = 0;        // its Karras index, less B0
  if (local) {
    right = B0 + l == 0 ? true : B0 + r == n - 1 ? false : sm.gap[r + 1] > sm.gap[l];
    slot = root ? 0 : right ? r : l;
    sm.made[slot] = 1;
    const uint32_t parent = B0 + (uint32_t)slot;
    if (l == t) sm.parLeaf[t] = parent | 0x80000000u;
    else sm.parInner[t] = parent | 0x80000000u;
    if (t + 1 == r) sm.parLeaf[t + 1] = parent;
    else sm.parInner[t + 1] = parent;
  }
  Box nb = box;
  if (ordered) {
    // Node by node: inner boxes in the second buffer, made[slot] = 2 once the box is there. A round makes the nodes
    // whose children are there; one that makes none is the last (all are made, or the keys are in no order, which the
    // sort has reported: their nodes wait for children that nobody makes).
    bool done = !local;
    __syncthreads();
    for (;;) {
      const bool now = !done && (l == t || sm.made[t] == 2) && (t + 1 == r || sm.made[t + 1] == 2);
      if (!__syncthreads_or(now)) break;  // every thread has read the marks
      if (now) {
        nb = sm.box.get(l == t ? 0 : 1, t);
        const Box other = sm.box.get(t + 1 == r ? 0 : 1, t + 1);
        merge_into(nb, other);
        sm.box.put(1, slot, nb);
        sm.made[slot] = 2;
        done = true;
      }
      __syncthreads();
    }
  }
  window_boxes<T>(sm.box, top, cnt, local && !ordered, l, r, box, nb);
  __syncthreads();  // the windows make room for the records
  auto stage = [&](int at, const Box &b, uint32_t par, uint32_t left, uint32_t rightLink, uint32_t leaf, uint32_t level) {
    const uint32_t isLeft = par == kNone ? 0u : par >> 31, parent = par == kNone ? kNone : par & 0x7FFFFFFFu;
    sm.record[3 * at] = make_float4(b.mn[0], b.mn[1], b.mn[2], b.mx[0]);
    sm.record[3 * at + 1] = make_float4(b.mx[1], b.mx[2], __uint_as_float(parent), __uint_as_float(left));
    sm.record[3 * at + 2] = make_float4(__uint_as_float(rightLink), __uint_as_float(leaf | (isLeft << 16)),
                                        __uint_as_float(level), surface_area(b));
  };
  if (local)
    stage(slot, nb, root ? 0u : sm.parInner[slot], l == t ? n - 1 + i : i, t + 1 == r ? n + i : i + 1, 0u, 0u);
  __syncthreads();
  float4 *out = reinterpret_cast<float4 *>(nodes + B0);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int q = c * T + t;
    if (q < 3 * cnt && sm.made[q / 3]) out[q] = sm.record[q];
  }
  __syncthreads();
  if (live) stage(t, box, n == 1 ? 0u : sm.parLeaf[t], face, 1u, 1u, 255u);
  __syncthreads();
  out = reinterpret_cast<float4 *>(nodes + (size_t)n - 1 + B0);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int q = c * T + t;
    if (q < 3 * cnt) out[q] = sm.record[q];
  }
  // The roots of the block's subtrees: (l, r | is-left << 31).
  const bool innerRoot = local && !root && sm.parInner[slot] == kNone;
  const bool leafRoot = live && n > 1 && sm.parLeaf[t] == kNone;
  if (roots == nullptr) return;  // one block made the whole tree
  // In the order of the leaves: a root's place is the number of roots that start before it.
  if (t < T / 32) sm.starts[t] = 0;
  __syncthreads();
  if (innerRoot) atomicOr(&sm.starts[l >> 5], 1u << (l & 31));
  if (leafRoot) atomicOr(&sm.starts[t >> 5], 1u << (t & 31));
  __syncthreads();
  uint2 *list = roots + (size_t)(B0 / T) * kTreeletRoots;
  if (innerRoot) {
    const uint32_t p = ones_before<T / 32>(sm.starts, l);
    if (p < (uint32_t)kTreeletRoots) list[p] = make_uint2(B0 + l, (B0 + r) | (right ? 0x80000000u : 0u));
  }
  if (leafRoot) {
    const bool leafRight = i == 0 ? true : i == n - 1 ? false : sm.gap[t + 1] > sm.gap[t];
    const uint32_t p = ones_before<T / 32>(sm.starts, t);
    if (p < (uint32_t)kTreeletRoots) list[p] = make_uint2(i, i | (leafRight ? 0x80000000u : 0u));
  }
  if (t == 0) rootCount[B0 / T] = min(ones_before<T / 32>(sm.starts, T - 1) + (sm.starts[T / 32 - 1] >> 31), (uint32_t)kTreeletRoots);
}

// ---- the subtrees of several blocks joined ------------------------------------------------------------
//
// The roots of kJoinBlocks neighbouring blocks' subtrees, in leaf order, are to the nodes above them
// what the leaves are to a block's: a block takes them one per thread (at most kJoin; 15 a block on
// average) and makes every node whose range lies among them in the same way. A root's place in a
// comparison is taken by its last leaf, whose bits within the range are every leaf's. The roots of what
// it made replace the first of the lists it read, and the next launch joins kJoinBlocks of those, until
// one block makes the tree's root. A list whose roots do not fit one block, or that holds a NaN (whose
// box depends on the order of the merges), stays as it is, as do the wider ones: a last launch climbs
// from its roots through the global exchange slots.
//
// Why: a climb pays an L2 exchange, a sibling's box and a fence a level, 3.7 us, and its upper levels
// are one chain; a joining launch makes about five levels in 7 us. Measured, 4.19M leaves: climbs from
// every block's roots 79 us, one joining launch and climbs from what it leaves 23 + 60, joined to the
// root 45 + 2 (33.5M: 357, 128 + 77, 169 + 3). Climbs from within the joining block cost more than they
// save (93 us; 424): a block lives as long as its longest climb.
constexpr int kJoin = 512, kJoinBlocks = 16;

template <typename K>
struct JoinSmem {
  BoxPair<kJoin> box;
  K key[kJoin + 2];          // of root c's last leaf at [c + 1]; its neighbours outside at both ends
  uint32_t last[kJoin + 2];  // that leaf
  uint8_t gap[kJoin + 1];    // delta of the leaves between the roots c - 1 and c
  uint8_t below[2][kJoin];   // the root (0) or the inner node numbered c (1) has its parent here
  uint32_t before[kJoinBlocks + 1];
  uint32_t starts[kJoin / 32];
};

template <int MODE, typename K>
__global__ void __launch_bounds__(kJoin) lbvh_join_kernel(uint2 *roots, const uint32_t *__restrict__ count,
                                                          uint32_t *__restrict__ joined, uint32_t lists, size_t pitch,
                                                          uint32_t n, const K *__restrict__ keys, bvhgb_node *nodes) {
  __shared__ JoinSmem<K> sm;
  __shared__ int top;
  constexpr int kBits = 8 * (int)sizeof(K);
  const int t = (int)threadIdx.x;
  const uint32_t b0 = blockIdx.x * kJoinBlocks, own = min((uint32_t)kJoinBlocks, lists - b0);
  if (t < 32) {
    uint32_t c = (uint32_t)t < own ? min(__ldg(count + b0 + t), (uint32_t)kJoin + 1u) : 0u;  // kNone: does not fit either
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, c, o);
      if (t >= o) c += x;
    }
    if (t < kJoinBlocks) sm.before[t + 1] = c;
    if (t == 0) sm.before[0] = 0;
  }
  sm.below[0][t] = sm.below[1][t] = 0;
  __syncthreads();
  const int m = (int)sm.before[kJoinBlocks];
  auto root_at = [&](int c) {
    int b = 0;
#pragma unroll
    for (int step = kJoinBlocks / 2; step > 0; step >>= 1)
      if ((uint32_t)c >= sm.before[b + step]) b += step;
    return __ldcg(roots + (b0 + b) * pitch + ((uint32_t)c - sm.before[b]));
  };
  if (m > kJoin) {
    if (t == 0) joined[blockIdx.x] = kNone;
    return;
  }
  const bool live = t < m;
  uint2 e = make_uint2(0u, 0u);
  Box box = {};
  bool nan = false;
  if (live) {
    e = root_at(t);
    const uint32_t l = e.x, r = e.y & 0x7FFFFFFFu;
    box = load_box_cg(nodes + (l == r ? n - 1 + l : (e.y >> 31) != 0u ? r : l));
    sm.last[t + 1] = r;
    if (t == 0) sm.last[0] = l - 1;
    if (t == m - 1) sm.last[m + 1] = r + 1;
    if (MODE == BVHGB_TOPO_KARRAS) {
      sm.key[t + 1] = __ldg(keys + r);
      if (t == 0 && l > 0) sm.key[0] = __ldg(keys + l - 1);
      if (t == m - 1 && r + 1 < n) sm.key[m + 1] = __ldg(keys + r + 1);
    }
    if (r + 1 < n) sm.gap[t + 1] = (uint8_t)delta<MODE, K>(keys, r, r + 1);
    if (t == 0 && l > 0) sm.gap[0] = (uint8_t)delta<MODE, K>(keys, l - 1, l);
    sm.box.put(0, t, box);
    nan = has_nan(box);
  }
  if (__syncthreads_or(nan)) {
    if (t == 0) joined[blockIdx.x] = kNone;
    return;
  }
  // The node that splits between the roots t and t + 1: its range, if that lies among the block's.
  int l = t, r = t;
  bool local = live && t + 1 < m;
  if (local) {
    const int d = sm.gap[t + 1];
    const uint32_t i = sm.last[t + 1];
    r = t + 1;
    const uint32_t mask = MODE == BVHGB_TOPO_REFCOMPAT ? (2u << (31 - d)) - 1u : 0u;
    const K mine = MODE == BVHGB_TOPO_KARRAS ? sm.key[t + 1] : (K)0;
    const K bound = d < kBits ? (K)1 << (kBits - d) : (K)1;
    auto same = [&](int c) {  // root c lies in the node's range
      if (MODE == BVHGB_TOPO_REFCOMPAT) return ((sm.last[c + 1] ^ i) & ~mask) == 0u;
      if ((K)(sm.key[c + 1] ^ mine) >= bound) return false;
      return d < kBits || __clz((int)(sm.last[c + 1] ^ i)) >= d - kBits;
    };
#pragma unroll
    for (int step = kJoin / 2; step > 0; step >>= 1) {
      if (l - step >= 0 && same(l - step)) l -= step;
      if (r + step < m && same(r + step)) r += step;
    }
    if (l == 0 && sm.last[0] != kNone && same(-1)) local = false;
    if (r == m - 1 && sm.last[m + 1] < n && same(m)) local = false;
  }
  const uint32_t L = local ? sm.last[l] + 1u : 0u, R = local ? sm.last[r + 1] : 0u;
  const bool root = local && L == 0 && R == n - 1;
  bool right = false;
  int slot = 0;  // the root whose first or last leaf numbers the node
  if (local) {
    right = L == 0 ? true : R == n - 1 ? false : sm.gap[r + 1] > sm.gap[l];
    slot = root ? 0 : right ? r : l;
    sm.below[l == t ? 0 : 1][t] = 1;
    sm.below[t + 1 == r ? 0 : 1][t + 1] = 1;
  }
  Box nb = box;
  window_boxes<kJoin>(sm.box, top, m, local, l, r, box, nb);
  const uint32_t index = root ? 0u : right ? R : L, split = local ? sm.last[t + 1] : 0u;
  const uint32_t a = L == split ? n - 1 + split : split, b = split + 1 == R ? n + split : split + 1;
  if (local) store_record(nodes + index, nb, root ? 0u : kNone, a, b, 0u, 0u, 0u);
  __syncthreads();  // every record before its parent's links
  if (local) {
    set_parent(nodes + a, index, 1);
    set_parent(nodes + b, index, 0);
  }
  // What is left goes, in leaf order, to the start of the lists this block has read.
  if (t < kJoin / 32) sm.starts[t] = 0;
  __syncthreads();
  const bool rest = live && !sm.below[0][t], innerRest = local && !root && !sm.below[1][slot];
  if (rest) atomicOr(&sm.starts[t >> 5], 1u << (t & 31));
  if (innerRest) atomicOr(&sm.starts[l >> 5], 1u << (l & 31));
  __syncthreads();
  uint2 *list = roots + b0 * pitch;
  if (rest) list[ones_before<kJoin / 32>(sm.starts, t)] = e;
  if (innerRest) list[ones_before<kJoin / 32>(sm.starts, l)] = make_uint2(L, R | (right ? 0x80000000u : 0u));
  if (t == 0) joined[blockIdx.x] = ones_before<kJoin / 32>(sm.starts, kJoin - 1) + (sm.starts[kJoin / 32 - 1] >> 31);
}

// Climbs from the lists that were not joined: a warp looks after kJoinBlocks of the blocks' lists, and
// after the joined list that starts with them if no wider one holds its roots. counts: the blocks', then
// every joining launch's.
constexpr int kClimbThreads = 128;
template <int MODE, typename K>
__global__ void __launch_bounds__(kClimbThreads) lbvh_roots_kernel(const uint2 *__restrict__ roots,
                                                                   const uint32_t *__restrict__ counts,
                                                                   uint32_t blocks, uint32_t n,
                                                                   const K *__restrict__ keys, bvhgb_node *nodes,
                                                                   uint32_t *slots, uint32_t *err) {
  const uint32_t q = (blockIdx.x * kClimbThreads + threadIdx.x) >> 5;
  if (q * kJoinBlocks >= blocks) return;
  // The widest joined list over this warp's blocks; it starts with those of warp 'first'.
  const uint32_t *level = counts + blocks;
  uint32_t lists = (blocks + kJoinBlocks - 1) / kJoinBlocks, span = 1, first = q, joined = kNone;
  for (;;) {
    const uint32_t c = __ldg(level + q / span);
    if (c == kNone) break;
    joined = c;
    first = q / span * span;
    if (lists == 1) break;
    level += lists;
    lists = (lists + kJoinBlocks - 1) / kJoinBlocks;
    span *= kJoinBlocks;
  }
  if (joined != kNone && first != q) return;
  const uint32_t b0 = q * kJoinBlocks;
  for (uint32_t b = b0; b < (joined != kNone ? b0 + 1 : min(b0 + kJoinBlocks, blocks)); ++b) {
    const uint32_t m = min(joined != kNone ? joined : __ldg(counts + b), (uint32_t)kJoin);
    for (uint32_t c = lane_id(); c < m; c += 32u) {
      const uint2 e = __ldg(roots + (size_t)b * kTreeletRoots + c);
      const uint32_t l = e.x, r = e.y & 0x7FFFFFFFu;
      const bool right = (e.y >> 31) != 0u;
      const uint32_t node = l == r ? n - 1 + l : right ? r : l;
      lbvh_climb_from<MODE, K>(l, r, right, load_box_cg(nodes + node), n, keys, nodes, slots, err);
    }
  }
}

template <int MODE, typename K>
__global__ void __launch_bounds__(kTreelet) lbvh_build_kernel(const float *__restrict__ vert,
                                                              const uint32_t *__restrict__ faces,
                                                              const K *__restrict__ keys,
                                                              const uint32_t *__restrict__ idx, uint32_t n,
                                                              const float4 *__restrict__ boxes, bvhgb_node *nodes,
                                                              uint2 *__restrict__ roots, uint32_t *rootCount) {
  __shared__ TreeletSmem<kTreelet, K> sm;
  const uint32_t B0 = blockIdx.x * kTreelet, i = B0 + threadIdx.x;
  uint32_t face = 0;
  K key = 0;
  Box box = {};
  if (i < n) {
    face = __ldg(idx + i);
    if (MODE == BVHGB_TOPO_KARRAS) key = __ldg(keys + i);
    if (boxes) {
      const float4 a = __ldg(boxes + 2 * (size_t)face), c = __ldg(boxes + 2 * (size_t)face + 1);
      box.mn[0] = a.x; box.mn[1] = a.y; box.mn[2] = a.z;
      box.mx[0] = a.w; box.mx[1] = c.x; box.mx[2] = c.y;
    } else {
      tri_box(vert, faces, face, box, nullptr);
    }
  }
  treelet_build<MODE, kTreelet, K>(sm, B0, n, face, box, key, keys, nodes, roots, rootCount);
}

// ---- small meshes in one launch -------------------------------------------------------------------
//
// Up to kSmallMesh triangles one block does it all, one triangle per thread: scene box, Morton key, a
// bitonic sort of (key, face) in registers (shuffles below a stride of 32, shared memory above) and
// the whole tree as one treelet. It leaves in the workspace what the phases would (scene box, keys,
// order, box records). Bound: the latency of that chain, 16 us with the launch for 1,000 triangles; twelve
// launches of a few microseconds each took 59 us.
constexpr int kSmallMesh = 1024;

template <typename K>
struct SmallSmem {
  TreeletSmem<kSmallMesh, K> tree;  // its boxes' place serves the sort first
  uint32_t scene[6];
  float red[kSmallMesh / 32][6];
};

template <int MODE, typename K>
__global__ void __launch_bounds__(kSmallMesh) lbvh_small_kernel(const float *__restrict__ vert,
                                                                const uint32_t *__restrict__ faces, uint32_t n,
                                                                uint32_t *__restrict__ scene,
                                                                uint32_t *__restrict__ sortErr, K *__restrict__ keys,
                                                                uint32_t *__restrict__ vals, K *__restrict__ keysSorted,
                                                                uint32_t *__restrict__ valsSorted,
                                                                float4 *__restrict__ boxes, bvhgb_node *nodes) {
  extern __shared__ __align__(16) unsigned char smraw[];
  SmallSmem<K> &sm = *reinterpret_cast<SmallSmem<K> *>(smraw);
  const uint32_t t = threadIdx.x, warp = t >> 5;
  const bool live = t < n;
  Box box = {};
  float c[3] = {0.0f, 0.0f, 0.0f};
  if (live) tri_box(vert, faces, t, box, c);
  // Scene box, from the origin box (lbvh_bounds_kernel).
  float v[6];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    v[k] = live ? fminf(0.0f, box.mn[k]) : 0.0f;
    v[3 + k] = live ? fmaxf(0.0f, box.mx[k]) : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v[k] = fminf(v[k], __shfl_xor_sync(0xFFFFFFFFu, v[k], o));
      v[3 + k] = fmaxf(v[3 + k], __shfl_xor_sync(0xFFFFFFFFu, v[3 + k], o));
    }
  }
  if (lane_id() < 6) sm.red[warp][lane_id()] = lane_id() == 0 ? v[0] : lane_id() == 1 ? v[1] : lane_id() == 2 ? v[2]
                                             : lane_id() == 3 ? v[3] : lane_id() == 4 ? v[4] : v[5];
  __syncthreads();
  if (warp < 6) {
    float m = sm.red[lane_id()][warp];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float x = __shfl_xor_sync(0xFFFFFFFFu, m, o);
      m = warp < 3 ? fminf(m, x) : fmaxf(m, x);
    }
    if (lane_id() == 0) scene[warp] = sm.scene[warp] = f2ord(m);
  }
  if (t >= 6 && t < kSceneWords) scene[t] = 0;
  if (t == 6) *sortErr = 0;  // which may be a larger mesh's
  __syncthreads();
  K key = ~(K)0;
  uint32_t face = t;  // a padding thread's pair sorts behind every triangle's
  if (live) {
    float off[3], sc[3];
    morton_params(sm.scene, off, sc);
    key = (K)morton_key<sizeof(K) == 8 ? 63 : 30>(c, off, sc);
    keys[t] = key;
    vals[t] = t;
    if (boxes) {
      boxes[2 * t] = make_float4(box.mn[0], box.mn[1], box.mn[2], box.mx[0]);
      boxes[2 * t + 1] = make_float4(box.mx[1], box.mx[2], 0.0f, 0.0f);
    }
  }
  // Bitonic sort by (key, face): the stable order.
  struct Pair {
    K key;
    uint32_t face;
  };
  Pair *pair = reinterpret_cast<Pair *>(&sm.tree.box);
  static_assert(2 * sizeof(Pair) * kSmallMesh <= sizeof(sm.tree.box), "two pair buffers");
  int flip = 0;
  for (uint32_t size = 2; size <= (uint32_t)kSmallMesh; size <<= 1) {
    for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
      K ok;
      uint32_t of;
      if (stride >= 32) {
        pair[flip * kSmallMesh + t] = Pair{key, face};
        __syncthreads();
        const Pair o = pair[flip * kSmallMesh + (t ^ stride)];
        ok = o.key;
        of = o.face;
        flip ^= 1;  // the next exchange writes the other buffer: no second barrier
      } else {
        ok = __shfl_xor_sync(0xFFFFFFFFu, key, stride);
        of = __shfl_xor_sync(0xFFFFFFFFu, face, stride);
      }
      const bool up = (t & size) == 0, low = (t & stride) == 0;
      const bool less = ok < key || (ok == key && of < face);  // the other pair comes first
      if (less == (up == low)) {
        key = ok;
        face = of;
      }
    }
  }
  // The leaf's box: the sorted face's, through shared memory.
  __syncthreads();
  sm.tree.box.put(0, t, box);
  __syncthreads();
  if (live) {
    keysSorted[t] = key;
    valsSorted[t] = face;
    box = sm.tree.box.get(0, face);
  }
  __syncthreads();
  treelet_build<MODE, kSmallMesh, K>(sm.tree, 0u, n, face, box, key, nullptr, nodes, nullptr, nullptr);
}

template <int MODE, typename K>
int launch_small(bvhgb_lbvh_workspace *ws, const float *vert, const uint32_t *faces, uint32_t n, bvhgb_node *nodes,
                 cudaStream_t s) {
  ws->slotsArmed = false;
  ws->sceneReady = ws->sorted = true;
  lbvh_small_kernel<MODE, K><<<1, kSmallMesh, sizeof(SmallSmem<K>), s>>>(
      vert, faces, n, ws->scene, sort_error_word(ws->sortTemp, ws->maxFaces, ws->keyBytes, 0, ws->cfg.mortonBits),
      static_cast<K *>(ws->keys), ws->vals, static_cast<K *>(ws->keysSorted), ws->valsSorted,
      ws->triBoxes, nodes);
  BVHGB_LAUNCH_CHECK("lbvh small");
  return BVHGB_OK;
}

template <int MODE, typename K>
cudaError_t set_small_attr() {
  return cudaFuncSetAttribute(lbvh_small_kernel<MODE, K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)sizeof(SmallSmem<K>));
}

// Opts in to the small kernel's shared memory, once per context (as sort_prepare).
int small_prepare() {
  static std::mutex m;
  static std::vector<uint64_t> done;
  const uint64_t ctx = context_id();
  std::lock_guard<std::mutex> lock(m);
  if (ctx != 0 && std::find(done.begin(), done.end(), ctx) != done.end()) return BVHGB_OK;
  BVHGB_CUDA_TRY((set_small_attr<BVHGB_TOPO_REFCOMPAT, uint32_t>()));
  BVHGB_CUDA_TRY((set_small_attr<BVHGB_TOPO_REFCOMPAT, uint64_t>()));
  BVHGB_CUDA_TRY((set_small_attr<BVHGB_TOPO_KARRAS, uint32_t>()));
  BVHGB_CUDA_TRY((set_small_attr<BVHGB_TOPO_KARRAS, uint64_t>()));
  if (ctx != 0) done.push_back(ctx);
  return BVHGB_OK;
}

template <int MODE, typename K>
int launch_build(bvhgb_lbvh_workspace *ws, const float *vert, const uint32_t *faces, uint32_t n, bvhgb_node *nodes,
                 cudaStream_t s) {
  // The exchange slots are re-armed by the Morton kernel; a second build from the same sorted keys
  // re-arms them here.
  if (!ws->slotsArmed) BVHGB_CUDA_TRY(cudaMemsetAsync(ws->slots, 0xFF, 4ull * n, s));
  ws->slotsArmed = false;
  // The lists of roots take the place of the sort's alternate buffers, which nothing reads after the
  // sort. 8 n bytes hold them: 193 places of 8 bytes per 256 leaves, and the counts at the end
  // (4 (b + b / 15 + 8) bytes for b blocks at most).
  const uint32_t blocks = ceil_div(n, kTreelet);
  static_assert(8 * (kTreelet - kTreeletRoots) >= 2 * 4 * 2 + 4 * 8, "room for the counts beside the roots");
  char *lists = static_cast<char *>(sort_alternate(ws->sortTemp, n, ws->keyBytes, 0, ws->cfg.mortonBits));
  uint2 *roots = blocks > 1 ? reinterpret_cast<uint2 *>(lists) : nullptr;
  uint32_t words = blocks;  // counts: the blocks', then every joining launch's
  for (uint32_t m = blocks; m > 1;) words += m = ceil_div(m, kJoinBlocks);
  uint32_t *counts = reinterpret_cast<uint32_t *>(lists + 8ull * n) - words;
  const K *keys = static_cast<const K *>(ws->keysSorted);
  lbvh_build_kernel<MODE, K><<<blocks, kTreelet, 0, s>>>(
      vert, faces, keys, ws->valsSorted, n, ws->triBoxes, nodes, roots, counts);
  BVHGB_LAUNCH_CHECK("lbvh build");
  if (blocks == 1) return BVHGB_OK;  // one block makes the whole tree
  size_t pitch = kTreeletRoots;
  uint32_t *in = counts;
  for (uint32_t m = blocks; m > 1; pitch *= kJoinBlocks) {
    const uint32_t joins = ceil_div(m, kJoinBlocks);
    lbvh_join_kernel<MODE, K><<<joins, kJoin, 0, s>>>(roots, in, in + m, m, pitch, n, keys, nodes);
    BVHGB_LAUNCH_CHECK("lbvh join");
    in += m;
    m = joins;
  }
  lbvh_roots_kernel<MODE, K><<<ceil_div(ceil_div(blocks, kJoinBlocks), kClimbThreads / 32), kClimbThreads, 0, s>>>(
      roots, counts, blocks, n, keys, nodes, ws->slots, ws->scene + 6);
  BVHGB_LAUNCH_CHECK("lbvh roots");
  return BVHGB_OK;
}

// The scene words hold nothing until a build's first phase writes all of them, on its stream; a call that comes
// before any such phase clears them there.
int scene_ready(bvhgb_lbvh_workspace *ws, cudaStream_t s) {
  if (!ws->sceneReady) BVHGB_CUDA_TRY(cudaMemsetAsync(ws->scene, 0, 4 * kSceneWords, s));
  ws->sceneReady = true;
  return BVHGB_OK;
}

int check_ws(const bvhgb_lbvh_workspace *ws, uint32_t n) {
  if (!ws) return BVHGB_INVALID_ARGUMENT;
  if (n > ws->maxFaces) return BVHGB_TOO_LARGE;
  return BVHGB_OK;
}

}  // namespace
}  // namespace bvhgb

using namespace bvhgb;

extern "C" BVHGB_API int bvhgb_lbvh_create(uint32_t maxFaces, const bvhgb_lbvh_config *cfg, bvhgb_lbvh_workspace **out) {
  if (!out) return BVHGB_INVALID_ARGUMENT;
  *out = nullptr;
  bvhgb_lbvh_config c = cfg ? *cfg : bvhgb_lbvh_config{30u, BVHGB_TOPO_REFCOMPAT};
  if ((c.mortonBits != 30 && c.mortonBits != 63) || c.topology > BVHGB_TOPO_KARRAS) return BVHGB_INVALID_ARGUMENT;
  if (maxFaces >= (1u << 30)) return BVHGB_TOO_LARGE;
  int pst = sort_prepare();
  if (!pst) pst = small_prepare();
  if (pst) return pst;
  auto *ws = new bvhgb_lbvh_workspace();
  ws->maxFaces = maxFaces;
  ws->cfg = c;
  ws->keyBytes = c.mortonBits == 30 ? 4u : 8u;
  const size_t m = maxFaces ? maxFaces : 1;
  ws->sortTempBytes = sort_temp_bytes(maxFaces, ws->keyBytes, 0, c.mortonBits);
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = dev_malloc(&ws->scene, 256);
  if (e == cudaSuccess) e = dev_malloc(&ws->keys, ws->keyBytes * m);
  if (e == cudaSuccess) e = dev_malloc(&ws->keysSorted, ws->keyBytes * m);
  if (e == cudaSuccess) e = dev_malloc(&ws->vals, 4 * m);
  if (e == cudaSuccess) e = dev_malloc(&ws->valsSorted, 4 * m);
  if (e == cudaSuccess) e = dev_malloc(&ws->slots, 4 * m);
  if (e == cudaSuccess) e = dev_malloc(&ws->triBoxes, 32 * m);
  if (e == cudaSuccess) e = dev_malloc(&ws->sortTemp, ws->sortTempBytes ? ws->sortTempBytes : 256);
  if (ws->keyBytes == 8) {  // two places a sample
    for (ws->cellBits = 10; ws->cellBits < 22 && (1u << ws->cellBits) < maxFaces / (cell_sample(maxFaces) / 2);) ++ws->cellBits;
    if (e == cudaSuccess) e = dev_malloc(&ws->cells, 4ull << ws->cellBits);
  }
  if (e != cudaSuccess) {
    set_last_error("bvhgb_lbvh_create", e);
    bvhgb_lbvh_destroy(ws);
    return e == cudaErrorMemoryAllocation ? BVHGB_OUT_OF_MEMORY : BVHGB_CUDA_ERROR;
  }
  *out = ws;
  return BVHGB_OK;
}

extern "C" BVHGB_API int bvhgb_lbvh_destroy(bvhgb_lbvh_workspace *ws) {
  if (!ws) return BVHGB_OK;
  cudaFree(ws->scene);
  cudaFree(ws->keys);
  cudaFree(ws->keysSorted);
  cudaFree(ws->vals);
  cudaFree(ws->valsSorted);
  cudaFree(ws->slots);
  cudaFree(ws->triBoxes);
  cudaFree(ws->cells);
  cudaFree(ws->sortTemp);
  delete ws;
  return BVHGB_OK;
}

extern "C" BVHGB_API int bvhgb_lbvh_init_tri_data(bvhgb_lbvh_workspace *ws, const float *vert, const uint32_t *faces,
                                                  uint32_t n, bvhgb_stream stream) {
  int st = check_ws(ws, n);
  if (st) return st;
  cudaStream_t s = as_stream(stream);
  lbvh_init_kernel<<<1, 32, 0, s>>>(ws->scene);
  BVHGB_LAUNCH_CHECK("lbvh init");
  ws->sceneReady = true;
  if (n == 0) return BVHGB_OK;
  if (!vert || !faces) return BVHGB_INVALID_ARGUMENT;
  uint32_t grid = min(ceil_div(n, kBoundsThreads * 4), (uint32_t)sm_count() * 8);
  lbvh_bounds_kernel<<<grid, kBoundsThreads, 0, s>>>(vert, faces, n, ws->scene, ws->cells,
                                                     ws->cells ? 1u << ws->cellBits : 0u);
  BVHGB_LAUNCH_CHECK("lbvh bounds");
  ws->cellsClear = true;
  ws->cellsClearIn = capture_of(s);
  return BVHGB_OK;
}

extern "C" BVHGB_API int bvhgb_lbvh_calc_morton(bvhgb_lbvh_workspace *ws, const float *vert, const uint32_t *faces,
                                                uint32_t n, bvhgb_stream stream) {
  int st = check_ws(ws, n);
  if (st) return st;
  if (n == 0) return BVHGB_OK;
  if (!vert || !faces) return BVHGB_INVALID_ARGUMENT;
  cudaStream_t s = as_stream(stream);
  if ((st = scene_ready(ws, s))) return st;
  uint32_t grid = ceil_div(n, kMortonThreads * 2);
  if (ws->cells) {
    if (!ws->cellsClear || ws->cellsClearIn != capture_of(s))
      BVHGB_CUDA_TRY(cudaMemsetAsync(ws->cells, 0, 4ull << ws->cellBits, s));
    ws->cellsClear = false;
  }
  if (ws->cfg.mortonBits == 30)
    lbvh_morton_kernel<30><<<grid, kMortonThreads, 0, s>>>(vert, faces, n, ws->scene, ws->keys, ws->vals, ws->slots,
                                                           ws->triBoxes, nullptr, 0u);
  else
    lbvh_morton_kernel<63><<<grid, kMortonThreads, 0, s>>>(vert, faces, n, ws->scene, ws->keys, ws->vals, ws->slots,
                                                           ws->triBoxes, ws->cells, ws->cellBits);
  BVHGB_LAUNCH_CHECK("lbvh morton");
  ws->slotsArmed = true;
  return BVHGB_OK;
}

extern "C" BVHGB_API int bvhgb_lbvh_sort(bvhgb_lbvh_workspace *ws, uint32_t n, bvhgb_stream stream) {
  int st = check_ws(ws, n);
  if (st) return st;
  if ((st = scene_ready(ws, as_stream(stream)))) return st;
  ws->sorted = ws->sorted || n != 0;
  if (ws->keyBytes == 8) {
    return sort_morton(ws->sortTemp, static_cast<const uint64_t *>(ws->keys), static_cast<uint64_t *>(ws->keysSorted),
                       ws->vals, ws->valsSorted, n, ws->scene + 8, ws->scene + 10,
                       MortonCells{ws->cells, ws->cells ? 1u << ws->cellBits : 0u, ws->cells ? ws->scene + 9 : nullptr}, as_stream(stream));
  }
  return sort_pairs(ws->sortTemp, ws->keys, ws->keysSorted, ws->vals, ws->valsSorted, n, ws->keyBytes, 0,
                    ws->cfg.mortonBits, as_stream(stream));
}

extern "C" BVHGB_API int bvhgb_lbvh_build_tree(bvhgb_lbvh_workspace *ws, const float *vert, const uint32_t *faces,
                                               uint32_t n, bvhgb_node *nodes, bvhgb_stream stream) {
  int st = check_ws(ws, n);
  if (st) return st;
  if (n == 0) return BVHGB_OK;
  if (!vert || !faces || !nodes) return BVHGB_INVALID_ARGUMENT;
  cudaStream_t s = as_stream(stream);
  const bool wide = ws->keyBytes == 8;
  if (ws->cfg.topology == BVHGB_TOPO_REFCOMPAT)
    return wide ? launch_build<BVHGB_TOPO_REFCOMPAT, uint64_t>(ws, vert, faces, n, nodes, s)
                : launch_build<BVHGB_TOPO_REFCOMPAT, uint32_t>(ws, vert, faces, n, nodes, s);
  return wide ? launch_build<BVHGB_TOPO_KARRAS, uint64_t>(ws, vert, faces, n, nodes, s)
              : launch_build<BVHGB_TOPO_KARRAS, uint32_t>(ws, vert, faces, n, nodes, s);
}

extern "C" BVHGB_API int bvhgb_lbvh_build(bvhgb_lbvh_workspace *ws, const float *vert, const uint32_t *faces,
                                          uint32_t n, bvhgb_node *nodes, bvhgb_stream stream) {
  int st = check_ws(ws, n);
  if (st) return st;
  if (n == 0) return BVHGB_OK;
  if (!vert || !faces || !nodes) return BVHGB_INVALID_ARGUMENT;
  if (n <= (uint32_t)kSmallMesh) {
    if ((st = small_prepare())) return st;
    cudaStream_t s = as_stream(stream);
    const bool wide = ws->keyBytes == 8;
    if (ws->cfg.topology == BVHGB_TOPO_REFCOMPAT)
      return wide ? launch_small<BVHGB_TOPO_REFCOMPAT, uint64_t>(ws, vert, faces, n, nodes, s)
                  : launch_small<BVHGB_TOPO_REFCOMPAT, uint32_t>(ws, vert, faces, n, nodes, s);
    return wide ? launch_small<BVHGB_TOPO_KARRAS, uint64_t>(ws, vert, faces, n, nodes, s)
                : launch_small<BVHGB_TOPO_KARRAS, uint32_t>(ws, vert, faces, n, nodes, s);
  }
  if ((st = bvhgb_lbvh_init_tri_data(ws, vert, faces, n, stream))) return st;
  if ((st = bvhgb_lbvh_calc_morton(ws, vert, faces, n, stream))) return st;
  if ((st = bvhgb_lbvh_sort(ws, n, stream))) return st;
  return bvhgb_lbvh_build_tree(ws, vert, faces, n, nodes, stream);
}

extern "C" BVHGB_API int bvhgb_lbvh_read_scene_box(bvhgb_lbvh_workspace *ws, bvhgb_aabb *scene, bvhgb_stream stream) {
  if (!ws || !scene) return BVHGB_INVALID_ARGUMENT;
  uint32_t h[6];
  cudaStream_t s = as_stream(stream);
  int st = scene_ready(ws, s);
  if (st) return st;
  BVHGB_CUDA_TRY(cudaMemcpyAsync(h, ws->scene, sizeof(h), cudaMemcpyDeviceToHost, s));
  BVHGB_CUDA_TRY(cudaStreamSynchronize(s));
  float f[6];
  for (int k = 0; k < 6; ++k) {
    uint32_t u = h[k];
    uint32_t bits = (u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u;
    std::memcpy(&f[k], &bits, 4);
  }
  scene->minMax[0] = {f[0], f[1], f[2]};
  scene->minMax[1] = {f[3], f[4], f[5]};
  return BVHGB_OK;
}

extern "C" BVHGB_API int bvhgb_lbvh_set_scene_box(bvhgb_lbvh_workspace *ws, const bvhgb_aabb *scene,
                                                  bvhgb_stream stream) {
  if (!ws || !scene) return BVHGB_INVALID_ARGUMENT;
  // The order-preserving integer image of each float, as the bounds kernel's atomics keep it.
  const float f[6] = {scene->minMax[0].x, scene->minMax[0].y, scene->minMax[0].z,
                      scene->minMax[1].x, scene->minMax[1].y, scene->minMax[1].z};
  uint32_t h[6];
  for (int k = 0; k < 6; ++k) {
    uint32_t u;
    std::memcpy(&u, &f[k], 4);
    h[k] = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  }
  cudaStream_t s = as_stream(stream);
  int st = scene_ready(ws, s);
  if (st) return st;
  BVHGB_CUDA_TRY(cudaMemcpyAsync(ws->scene, h, sizeof(h), cudaMemcpyHostToDevice, s));
  // The copy reads pageable host memory, so it is staged before the call returns.
  return BVHGB_OK;
}

extern "C" BVHGB_API int bvhgb_lbvh_read_keys(bvhgb_lbvh_workspace *ws, int sorted, void *keys_host, uint32_t *idx_host,
                                              uint32_t n, bvhgb_stream stream) {
  int st = check_ws(ws, n);
  if (st) return st;
  cudaStream_t s = as_stream(stream);
  if (keys_host)
    BVHGB_CUDA_TRY(cudaMemcpyAsync(keys_host, sorted ? ws->keysSorted : ws->keys, (size_t)ws->keyBytes * n,
                                   cudaMemcpyDeviceToHost, s));
  if (idx_host)
    BVHGB_CUDA_TRY(cudaMemcpyAsync(idx_host, sorted ? ws->valsSorted : ws->vals, 4ull * n, cudaMemcpyDeviceToHost, s));
  BVHGB_CUDA_TRY(cudaStreamSynchronize(s));
  return BVHGB_OK;
}

extern "C" BVHGB_API int bvhgb_lbvh_read_errors(bvhgb_lbvh_workspace *ws, uint32_t *flags, bvhgb_stream stream) {
  if (!ws || !flags) return BVHGB_INVALID_ARGUMENT;
  uint32_t a = 0, b = 0;
  cudaStream_t s = as_stream(stream);
  int st = scene_ready(ws, s);
  if (st) return st;
  BVHGB_CUDA_TRY(cudaMemcpyAsync(&a, ws->scene + 6, 4, cudaMemcpyDeviceToHost, s));
  const uint32_t *se = sort_error_word(ws->sortTemp, ws->maxFaces, ws->keyBytes, 0, ws->cfg.mortonBits);
  if (ws->sorted) BVHGB_CUDA_TRY(cudaMemcpyAsync(&b, se, 4, cudaMemcpyDeviceToHost, s));
  BVHGB_CUDA_TRY(cudaStreamSynchronize(s));
  *flags = a | b;
  return BVHGB_OK;
}

extern "C" BVHGB_API int bvhgb_lbvh_read_sort_route(bvhgb_lbvh_workspace *ws, uint32_t *route, bvhgb_stream stream) {
  if (!ws || !route) return BVHGB_INVALID_ARGUMENT;
  cudaStream_t s = as_stream(stream);
  int st = scene_ready(ws, s);
  if (st) return st;
  BVHGB_CUDA_TRY(cudaMemcpyAsync(route, ws->scene + 10, 4, cudaMemcpyDeviceToHost, s));
  BVHGB_CUDA_TRY(cudaStreamSynchronize(s));
  return BVHGB_OK;
}

// ---- allocation-free build -------------------------------------------------------------------
//
// Some callers cannot allocate device memory while they build: a per-frame rebuild inside a render
// or simulation loop (cudaMalloc synchronises the whole device and stalls the frame), host
// applications whose device memory is owned by their own pool and that forbid driver allocations,
// and code that must not fail for lack of memory once started. For them the build below takes its
// working memory from one array in this file, sized for BVHGB_STATIC_MAX_FACES triangles and
// reserved on every GPU that loads the library until the process exits.
namespace bvhgb {
namespace {

constexpr size_t kStaticScratchBytes = 12ull << 20;  // covers keys, values, slots and sort scratch
__device__ __align__(256) unsigned char g_lbvh_static_scratch[kStaticScratchBytes];

struct StaticBase {
  uint64_t context;  // context_id() of the context the address belongs to
  unsigned char *base;
};
std::mutex g_static_mutex;
std::vector<StaticBase> g_static_base;

size_t round256(size_t x) { return (x + 255) & ~size_t(255); }

// Device address of the array in the current context, looked up once per context: every device
// has its own copy, and a device reset (cudaDeviceReset, bvhgb_reset_device) makes a new context
// whose copy may sit elsewhere, so an address is never reused across contexts.
int static_scratch(unsigned char **out) {
  const uint64_t ctx = context_id();
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (ctx != 0) {
    for (const StaticBase &b : g_static_base)
      if (b.context == ctx) {
        *out = b.base;
        return BVHGB_OK;
      }
  }
  void *p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_lbvh_static_scratch);
  if (e != cudaSuccess) {
    set_last_error("cudaGetSymbolAddress(g_lbvh_static_scratch)", e);
    return BVHGB_CUDA_ERROR;
  }
  if (ctx != 0) g_static_base.push_back({ctx, static_cast<unsigned char *>(p)});
  *out = static_cast<unsigned char *>(p);
  return BVHGB_OK;
}

// The working memory of one build carved out of the array for the largest size: the same layout
// for a build and for the read-back of its error bits.
int static_workspace(const bvhgb_lbvh_config &c, bvhgb_lbvh_workspace &ws) {
  unsigned char *base = nullptr;
  int st = static_scratch(&base);
  if (st) return st;
  ws.maxFaces = BVHGB_STATIC_MAX_FACES;
  ws.cfg = c;
  ws.keyBytes = c.mortonBits == 30 ? 4u : 8u;
  const size_t m = BVHGB_STATIC_MAX_FACES;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    unsigned char *p = base + off;
    off += round256(bytes);
    return p;
  };
  ws.scene = reinterpret_cast<uint32_t *>(take(256));
  ws.sceneReady = ws.sorted = true;  // the array starts as zeros
  ws.keys = take(ws.keyBytes * m);
  ws.keysSorted = take(ws.keyBytes * m);
  ws.vals = reinterpret_cast<uint32_t *>(take(4 * m));
  ws.valsSorted = reinterpret_cast<uint32_t *>(take(4 * m));
  ws.slots = reinterpret_cast<uint32_t *>(take(4 * m));
  ws.sortTempBytes = sort_temp_bytes(BVHGB_STATIC_MAX_FACES, ws.keyBytes, 0, c.mortonBits);
  ws.sortTemp = take(ws.sortTempBytes);
  if (off > kStaticScratchBytes) return BVHGB_GENERIC_ERROR;  // the array is sized for the worst case
  return BVHGB_OK;
}

bool static_cfg_valid(const bvhgb_lbvh_config &c) {
  return (c.mortonBits == 30 || c.mortonBits == 63) && c.topology <= BVHGB_TOPO_KARRAS;
}

}  // namespace
}  // namespace bvhgb

extern "C" BVHGB_API int bvhgb_lbvh_build_static(const float *vert, const uint32_t *faces, uint32_t numFaces,
                                                 const bvhgb_lbvh_config *cfg, bvhgb_node *nodes,
                                                 bvhgb_stream stream) {
  const bvhgb_lbvh_config c = cfg ? *cfg : bvhgb_lbvh_config{30u, BVHGB_TOPO_REFCOMPAT};
  if (!static_cfg_valid(c)) return BVHGB_INVALID_ARGUMENT;
  if (numFaces > BVHGB_STATIC_MAX_FACES) return BVHGB_TOO_LARGE;
  if (numFaces == 0) return BVHGB_OK;
  if (!vert || !faces || !nodes) return BVHGB_INVALID_ARGUMENT;
  bvhgb_lbvh_workspace ws;
  int st = static_workspace(c, ws);
  if (st) return st;
  st = sort_prepare();  // a function attribute, not an allocation
  if (st) return st;
  // The same phases as bvhgb_lbvh_build; every scratch word that must start at a known value is
  // written by the phase that uses it (scene box init kernel, which also clears the build's error
  // word and the sort's gate; slot reset in the Morton kernel; the sort's memset of its counters and error
  // word), so the previous call's contents do not matter.
  if ((st = bvhgb_lbvh_init_tri_data(&ws, vert, faces, numFaces, stream))) return st;
  if ((st = bvhgb_lbvh_calc_morton(&ws, vert, faces, numFaces, stream))) return st;
  if ((st = bvhgb_lbvh_sort(&ws, numFaces, stream))) return st;
  return bvhgb_lbvh_build_tree(&ws, vert, faces, numFaces, nodes, stream);
}

extern "C" BVHGB_API int bvhgb_lbvh_static_read_errors(const bvhgb_lbvh_config *cfg, uint32_t *flags,
                                                       bvhgb_stream stream) {
  const bvhgb_lbvh_config c = cfg ? *cfg : bvhgb_lbvh_config{30u, BVHGB_TOPO_REFCOMPAT};
  if (!flags || !static_cfg_valid(c)) return BVHGB_INVALID_ARGUMENT;
  bvhgb_lbvh_workspace ws;
  int st = static_workspace(c, ws);
  if (st) return st;
  return bvhgb_lbvh_read_errors(&ws, flags, stream);
}

