// Device side of the parallel Bittner13 optimizer (lib/builder/Bittner13CUDA.cu,
// lib/base/BVHPatch.hpp), shared by the single-tree kernels (bittner.cu) and the batched ones
// (batch.cu): node views, the 10-slot patch, both reinsertion searches, removal / reinsertion,
// and the per-item steps of a chunk.
#pragma once

#include "common.cuh"

namespace bvhgb {
namespace {

constexpr int NSLOT = 10;
enum : uint32_t {
  P_GRAND_PARENT = 0, P_1ST_ROOT = 1, P_1ST_BEST = 2, P_NODE = 3, P_1ST_INSERT = 4,
  P_2ND_ROOT = 5, P_2ND_BEST = 6, P_2ND_INSERT = 7, P_SIBLING = 8, P_PARENT = 9
};
enum StatIdx { S_ITEMS = 0, S_APPLIED = 1, S_CONFLICT = 2, S_INVALID = 3, S_OVERFLOW = 4, S_VISITS = 5, S_COUNT = 6 };

struct SearchCounters {
  uint32_t overflow;  // queue pushes dropped at capacity
  uint32_t visits;    // nodes evaluated by the branch and bound
};

struct NodeP {
  uint32_t parent, left, right;
  uint16_t isLeafFlag, isLeft;
};

struct HeapItem {
  uint32_t node;
  float cost;
};

struct alignas(16) PatchOut {  // what the apply kernel needs
  NodeP nd[NSLOT];
  uint32_t idx[NSLOT];  // then two words of padding: both arrays are read in 16-byte words
};
static_assert(sizeof(NodeP) == 16 && sizeof(PatchOut) == 208, "16-byte words");

// Read-only view of the tree during the patch kernel (nothing writes the tree in that launch).
__device__ __forceinline__ NodeP tree_node(const bvhgb_node *t, uint32_t x) {
  const float4 *p = reinterpret_cast<const float4 *>(t + x);
  const float4 b = __ldg(p + 1), c = __ldg(p + 2);
  NodeP r;
  r.parent = __float_as_uint(b.z);
  r.left = __float_as_uint(b.w);
  r.right = __float_as_uint(c.x);
  const uint32_t fl = __float_as_uint(c.y);
  r.isLeafFlag = (uint16_t)(fl & 0xFFFFu);
  r.isLeft = (uint16_t)(fl >> 16);
  return r;
}
__device__ __forceinline__ Box tree_box(const bvhgb_node *t, uint32_t x) {
  const float4 *p = reinterpret_cast<const float4 *>(t + x);
  const float4 a = __ldg(p), b = __ldg(p + 1);
  Box r;
  r.mn[0] = a.x; r.mn[1] = a.y; r.mn[2] = a.z;
  r.mx[0] = a.w; r.mx[1] = b.x; r.mx[2] = b.y;
  return r;
}
// Links and box of a node, loaded together.
struct NodeRec {
  NodeP n;
  Box b;
};
__device__ __forceinline__ NodeRec tree_rec(const bvhgb_node *t, uint32_t x) {
  const float4 *p = reinterpret_cast<const float4 *>(t + x);
  const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
  NodeRec r;
  r.b.mn[0] = a.x; r.b.mn[1] = a.y; r.b.mn[2] = a.z;
  r.b.mx[0] = a.w; r.b.mx[1] = b.x; r.b.mx[2] = b.y;
  r.n.parent = __float_as_uint(b.z);
  r.n.left = __float_as_uint(b.w);
  r.n.right = __float_as_uint(c.x);
  const uint32_t fl = __float_as_uint(c.y);
  r.n.isLeafFlag = (uint16_t)(fl & 0xFFFFu);
  r.n.isLeft = (uint16_t)(fl >> 16);
  return r;
}
__device__ __forceinline__ float tree_sa(const bvhgb_node *t, uint32_t x) { return __ldg(&t[x].surfaceArea); }

// The storage of a BVHPatch: its node slots and patched boxes. Every lane of a warp that runs one
// item holds the same patch, so the warp kernels keep one copy per warp in shared memory (a copy
// per lane would not fit L1); the thread-per-item kernel keeps its own.
struct PatchData {
  NodeP nd[NSLOT];
  uint32_t idx[NSLOT];
  uint32_t apath[4];
  Box abox[4];
};

// BVHPatch (BVHPatch.hpp:87-335), ENABLE_AABB_PATH = 0.
struct Patch {
  PatchData *d;
  const bvhgb_node *t;
  uint32_t root;
  uint32_t numNodes;
  mutable bool bad;  // an index outside the node array was met (corrupted input); item is dropped

  __device__ uint32_t chk(uint32_t x) const {
    if (x < numNodes) return x;
    bad = true;
    return root;
  }

  __device__ void clear() {
#pragma unroll
    for (int i = 0; i < NSLOT; ++i) d->idx[i] = kNone;
#pragma unroll
    for (int i = 0; i < 4; ++i) d->apath[i] = kNone;
  }
  __device__ uint32_t index_subset(uint32_t x) const {
    if (d->idx[0] == x) return 0;
    if (d->idx[1] == kNone) return kNone;
    if (d->idx[1] == x) return 1;
    if (d->idx[2] == x) return 2;
    if (d->idx[3] == x) return 3;
    return kNone;
  }
  // The first slot of x; every slot is read before the first compare (no chain of loads and exits).
  __device__ __forceinline__ uint32_t index(uint32_t x) const {
    uint32_t v[NSLOT];
#pragma unroll
    for (int i = 0; i < NSLOT; ++i) v[i] = d->idx[i];
    uint32_t r = kNone;
#pragma unroll
    for (int i = NSLOT - 1; i >= 0; --i)
      if (v[i] == x) r = (uint32_t)i;
    return r;
  }
  __device__ NodeP get(uint32_t x) const {
    uint32_t i = index(x);
    return i == kNone ? tree_node(t, chk(x)) : d->nd[i];
  }
  __device__ NodeP get_subset(uint32_t x) const {
    uint32_t i = index_subset(x);
    return i == kNone ? tree_node(t, chk(x)) : d->nd[i];
  }
  __device__ uint32_t patch_node(uint32_t x, uint32_t slot) {
    d->idx[slot] = x;
    d->nd[slot] = tree_node(t, chk(x));
    return slot;
  }
  __device__ uint32_t move(uint32_t from, uint32_t to) {
    d->idx[to] = d->idx[from];
    d->idx[from] = kNone;
    d->nd[to] = d->nd[from];
    return to;
  }
  // get_subset(x) and get_aabb(x) given the tree's 48-byte record of x (a, m, c: its three float4).
  __device__ void subset_aabb_from(uint32_t x, const float4 &a, const float4 &m, const float4 &c, NodeP &n,
                                   Box &b) const {
    const uint32_t i = index_subset(x);
    if (i != kNone) {
      n = d->nd[i];
    } else {
      n.parent = __float_as_uint(m.z);
      n.left = __float_as_uint(m.w);
      n.right = __float_as_uint(c.x);
      const uint32_t fl = __float_as_uint(c.y);
      n.isLeafFlag = (uint16_t)(fl & 0xFFFFu);
      n.isLeft = (uint16_t)(fl >> 16);
    }
    for (int k = 0; k < 4; ++k) {
      if (d->apath[k] == x) {
        b = d->abox[k];
        return;
      }
    }
    b.mn[0] = a.x; b.mn[1] = a.y; b.mn[2] = a.z;
    b.mx[0] = a.w; b.mx[1] = m.x; b.mx[2] = m.y;
  }
  __device__ Box get_aabb(uint32_t x) const {
    for (int i = 0; i < 4; ++i)
      if (d->apath[i] == x) return d->abox[i];
    return tree_box(t, chk(x));
  }
  // patchAABBFrom (BVHPatch.hpp:293-316)
  __device__ void patch_aabb_from(uint32_t x, uint32_t pidx) {
    uint32_t ni = x;
    NodeP n = get_subset(ni);
    Box b = get_aabb(n.left);
    bool lastLeft = true;
    for (uint32_t i = 0; i < 2; ++i) {
      uint32_t sib = lastLeft ? n.right : n.left;
      Box sb = get_aabb(sib);
      merge_into(b, sb);
      d->abox[pidx * 2 + i] = b;
      d->apath[pidx * 2 + i] = ni;
      lastLeft = n.isLeft != 0;
      if (ni == root) break;
      ni = n.parent;
      n = get_subset(ni);
    }
  }
};

// Heap with the hole-based sift of the standard library heap algorithms (CUDAHeap.hpp:33-112);
// "less(a, b)" is a.cost > b.cost, so h[0] holds the smallest induced cost.
__device__ __forceinline__ bool hless(const HeapItem &a, const HeapItem &b) { return a.cost > b.cost; }

// Two-level storage: the first kHeapShared entries of each search live in shared memory,
// interleaved across the warp's lanes (entry i of lane l at i * 32 + l, conflict-free when lanes
// touch the same depth); deeper entries spill to the item's global region. The index space and
// the capacity are unchanged, so the pop order is exactly that of a flat array.
constexpr int kSearchThreads = 32;
constexpr int kHeapShared = 128;

struct Heap {
  HeapItem *sm;  // this lane's entry 0 in shared memory (stride kSearchThreads)
  HeapItem *gm;  // this item's global region (cap entries)
  __device__ __forceinline__ HeapItem &at(long i) const { return i < kHeapShared ? sm[i * kSearchThreads] : gm[i]; }
};

__device__ __forceinline__ void sift_up(const Heap &h, long hole, long top, HeapItem v) {
  long parent = (hole - 1) / 2;
  while (hole > top && hless(h.at(parent), v)) {
    h.at(hole) = h.at(parent);
    hole = parent;
    parent = (hole - 1) / 2;
  }
  h.at(hole) = v;
}
__device__ __forceinline__ void heap_push(const Heap &h, long lenAfter) { sift_up(h, lenAfter - 1, 0, h.at(lenAfter - 1)); }
__device__ __forceinline__ void heap_pop(const Heap &h, long len) {
  if (len <= 1) return;
  const long last = len - 1;
  const HeapItem v = h.at(last);
  h.at(last) = h.at(0);
  const long n = last;
  long hole = 0, second = 0;
  while (second < (n - 1) / 2) {
    second = 2 * (second + 1);
    if (hless(h.at(second), h.at(second - 1))) second--;
    h.at(hole) = h.at(second);
    hole = second;
  }
  if ((n & 1) == 0 && second == (n - 2) / 2) {
    second = 2 * (second + 1);
    h.at(hole) = h.at(second - 1);
    hole = second - 1;
  }
  sift_up(h, hole, 0, v);
}

// Starts fetching a node's 48-byte record into L2 while the search keeps working.
__device__ __forceinline__ void prefetch_node(const bvhgb_node *t, uint32_t x) {
  const char *p = reinterpret_cast<const char *>(t + x);
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p + 32));
}

// findNode1 (Bittner13CUDA.cu:141-191).
__device__ uint32_t find_node(const Patch &p, uint32_t n, const Heap &pq, uint32_t cap, SearchCounters &ctr) {
  float best_cost = __int_as_float(0x7f800000);
  uint32_t best = 0;
  const Box nbox = tree_box(p.t, p.chk(n));
  const float sarea = tree_sa(p.t, p.chk(n));
  long size = 1;
  pq.at(0).node = p.root;
  pq.at(0).cost = 0.0f;
  // A tree pops each node at most once; the bound only matters for corrupted input.
  for (uint32_t it = 0; size > 0; ++it) {
    if (it > p.numNodes) {
      p.bad = true;
      break;
    }
    const HeapItem cur = pq.at(0);
    if (fadd(cur.cost, sarea) >= best_cost) break;
    heap_pop(pq, size);
    size--;
    ctr.visits++;
    const NodeP cn = p.get_subset(cur.node);
    Box b = p.get_aabb(cur.node);
    float induced = fmul(-1.0f, surface_area(b));
    merge_into(b, nbox);
    const float direct = surface_area(b);
    const float total = fadd(cur.cost, direct);
    if (total < best_cost) {
      best_cost = total;
      best = cur.node;
    }
    induced = fadd(induced, total);
    if (fadd(induced, sarea) < best_cost && !cn.isLeafFlag) {
      if ((uint32_t)size + 2 <= cap) {
        if (cn.left < p.numNodes) prefetch_node(p.t, cn.left);
        if (cn.right < p.numNodes) prefetch_node(p.t, cn.right);
        pq.at(size).node = cn.left;
        pq.at(size).cost = induced;
        pq.at(size + 1).node = cn.right;
        pq.at(size + 1).cost = induced;
        heap_push(pq, size + 1);
        heap_push(pq, size + 2);
        size += 2;
      } else {
        ctr.overflow++;
      }
    }
  }
  return best;
}

// findNode2 (Bittner13CUDA.cu:194-264), the approximate search of altFindNode: kAltQueue (cost,
// node) slots, empty = +inf. Each step pops the first slot of smallest cost; an expanded node's
// left child takes the popped slot and its right child the slot the previous scan found to hold
// the largest cost (the first empty one while there is one, else the worst entry, which is lost);
// a scan in which no cost exceeds 0 keeps the previous max slot. One thread per item; the slots
// live in registers (the scans are unrolled, the two writes select by index).
constexpr uint32_t kAltQueue = 16;  // CUDA_ALT_QUEUE_SIZE (Bittner13CUDA.hpp:30)

__device__ uint32_t find_node2(const Patch &p, uint32_t n, SearchCounters &ctr) {
  const float kInf = __int_as_float(0x7f800000);
  float best_cost = kInf;
  uint32_t best = 0;
  const Box nbox = tree_box(p.t, p.chk(n));
  const float sarea = tree_sa(p.t, p.chk(n));
  float co[kAltQueue];
  uint32_t nl[kAltQueue];
#pragma unroll
  for (uint32_t i = 0; i < kAltQueue; ++i) {
    co[i] = kInf;
    nl[i] = 0;
  }
  uint32_t mnI = 0, mxI = 1;
  float mn = 0.0f;
  nl[0] = p.root;
  co[0] = 0.0f;
  for (uint32_t it = 0; mn < kInf; ++it) {
    if (it > p.numNodes) {  // only a corrupted tree gets here
      p.bad = true;
      break;
    }
    uint32_t cur = 0;
    float cc = 0.0f;
#pragma unroll
    for (uint32_t i = 0; i < kAltQueue; ++i)
      if (i == mnI) {
        cur = nl[i];
        cc = co[i];
        co[i] = kInf;
      }
    if (fadd(cc, sarea) >= best_cost) break;
    ctr.visits++;
    const NodeP cn = p.get_subset(cur);
    Box b = p.get_aabb(cur);
    float induced = fmul(-1.0f, surface_area(b));
    merge_into(b, nbox);
    const float direct = surface_area(b);
    const float total = fadd(cc, direct);
    if (total < best_cost) {
      best_cost = total;
      best = cur;
    }
    induced = fadd(induced, total);
    if (fadd(induced, sarea) < best_cost && !cn.isLeafFlag) {
#pragma unroll
      for (uint32_t i = 0; i < kAltQueue; ++i) {
        if (i == mnI) {
          nl[i] = cn.left;
          co[i] = induced;
        }
        if (i == mxI) {  // after the left child: the same slot takes the right one
          nl[i] = cn.right;
          co[i] = induced;
        }
      }
    }
    mn = kInf;
    float mx = 0.0f;
#pragma unroll
    for (uint32_t i = 0; i < kAltQueue; ++i) {
      if (co[i] < mn) {
        mn = co[i];
        mnI = i;
      }
      if (co[i] > mx) {
        mx = co[i];
        mxI = i;
      }
    }
  }
  return best;
}

// removeNode (Bittner13CUDA.cu:267-305) with patchAABBFrom(grand parent) written out. Every record is
// loaded once and as soon as its index is known, all loads of a step before the first use of one:
// node, parent, then grand parent and sibling, then the boxes around the grand parent are four
// dependent round trips (slot by slot they were eight).
__device__ __forceinline__ bool remove_node(Patch &p, uint32_t x, uint32_t ins[2], uint32_t un[2], uint32_t &g_out) {
  NodeP nx = tree_node(p.t, p.chk(x));
  if (nx.isLeafFlag || x == p.root) return false;
  const uint32_t l = nx.left, r = nx.right, pi = nx.parent;
  const NodeP np = tree_node(p.t, p.chk(pi));
  const float sl = tree_sa(p.t, p.chk(l)), sr = tree_sa(p.t, p.chk(r));
  if (pi == p.root) return false;
  const uint32_t s = nx.isLeft == 0 ? np.left : np.right, gi = np.parent;
  NodeRec rs = tree_rec(p.t, p.chk(s));
  NodeP ng = tree_node(p.t, p.chk(gi));
  const uint32_t other = np.isLeft ? ng.right : ng.left;  // the grand parent's other child
  const uint32_t ggi = gi == p.root ? gi : ng.parent;  // what the root's link holds is not looked at
  const Box ob = tree_box(p.t, p.chk(other));
  const NodeP ngg = tree_node(p.t, p.chk(ggi));
  if (np.isLeft) ng.left = s;
  else ng.right = s;
  rs.n.isLeft = np.isLeft ? 1 : 0;
  rs.n.parent = gi;
  Box b = np.isLeft ? rs.b : ob;  // the left child's box merged with the right's
  merge_into(b, np.isLeft ? ob : rs.b);
  p.d->idx[P_NODE] = x;
  p.d->nd[P_NODE] = nx;
  p.d->idx[P_SIBLING] = s;
  p.d->nd[P_SIBLING] = rs.n;
  p.d->idx[P_PARENT] = pi;
  p.d->nd[P_PARENT] = np;
  p.d->idx[P_GRAND_PARENT] = gi;
  p.d->nd[P_GRAND_PARENT] = ng;
  p.d->apath[0] = gi;
  p.d->abox[0] = b;
  if (gi != p.root) {
    merge_into(b, tree_box(p.t, p.chk(ng.isLeft ? ngg.right : ngg.left)));
    p.d->apath[1] = ggi;
    p.d->abox[1] = b;
  }
  if (sl > sr) { ins[0] = l; ins[1] = r; }
  else { ins[0] = r; ins[1] = l; }
  un[0] = x;
  un[1] = pi;
  g_out = gi;
  return true;
}

// ---- batched best-first search: one warp per item -------------------------------------------
//
// The frontier (up to 128 entries, unordered) lives in registers, 4 slots per lane, entry
// e = slot * 32 + lane. Each round the warp evaluates every entry, reduces the best total and
// gathers the children of the expanded entries into the warp's shared buffer, which becomes the
// next frontier. Only when more than 128 children arrive are the 128 lowest in (cost, node) order
// selected (a radix selection by warp sums) and kept, the rest counted as overflow. The best
// position (ties: the earliest round, then the entry first in (cost, node) order) is kept per lane
// and resolved after the last round. oracle/bittner.c (gpu_find_node_batched) restates the same
// rounds.
// Bound: the dependent chain of a round (a record's L2 round trip, the evaluation, the reduction,
// the gather); a search takes 16 to 18 rounds of 6 to 14 entries. With the patch's keys in
// registers, the best per lane, no bound test per entry, records loaded side by side and one copy
// of the search's code for both reinsertions a chunk's launch went from 29.6 to 18 us on 65,536
// triangles (41 items) and from 51.7 to 35 us on 4.19M (2,621 items).
constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr int kFrontier = 4;  // slots per lane (128 entries)
constexpr uint32_t kFrontierCap = 32u * kFrontier;

// The k-th smallest (1 <= k <= number of flagged entries) of the 32-bit keys of the slots flagged
// in 'in' (bit s: this lane's slot s), S slots per lane: a most-significant-first radix selection
// over 2-bit digits, one warp sum per digit, starting below the bits that all flagged keys share.
template <int S>
__device__ __forceinline__ uint32_t warp_select_kth(const uint32_t (&key)[S], uint32_t in, uint32_t k) {
  uint32_t lo = 0xFFFFFFFFu, hi = 0u;
#pragma unroll
  for (int s = 0; s < S; ++s)
    if ((in >> s) & 1u) {
      lo = min(lo, key[s]);
      hi = max(hi, key[s]);
    }
  lo = __reduce_min_sync(kFull, lo);
  hi = __reduce_max_sync(kFull, hi);
  if (lo == hi) return lo;
  const int top = 31 - __clz(lo ^ hi);
  uint32_t res = lo & ~((2u << top) - 1u);  // 2u << 31 wraps to 0: no common bits
  uint32_t alive = in;
  int bit = top;
  // two bits per step: the counts of the digits 00, 01 and 10 (at most 1,023 each) travel packed
  // 10 bits apart in one warp sum
  for (; bit >= 1; bit -= 2) {
    uint32_t hi1 = 0, lo1 = 0;  // this lane's slots whose key has bit / bit - 1 set
#pragma unroll
    for (int s = 0; s < S; ++s) {
      hi1 |= ((key[s] >> bit) & 1u) << s;
      lo1 |= ((key[s] >> (bit - 1)) & 1u) << s;
    }
    const uint32_t m00 = alive & ~hi1 & ~lo1, m01 = alive & ~hi1 & lo1, m10 = alive & hi1 & ~lo1;
    const uint32_t c = __reduce_add_sync(kFull, (uint32_t)__popc(m00) | ((uint32_t)__popc(m01) << 10) |
                                                    ((uint32_t)__popc(m10) << 20));
    const uint32_t c00 = c & 1023u, c01 = (c >> 10) & 1023u, c10 = c >> 20;
    if (k <= c00) {
      alive = m00;
    } else if (k <= c00 + c01) {
      k -= c00;
      alive = m01;
      res |= 1u << (bit - 1);
    } else if (k <= c00 + c01 + c10) {
      k -= c00 + c01;
      alive = m10;
      res |= 1u << bit;
    } else {
      k -= c00 + c01 + c10;
      alive &= hi1 & lo1;
      res |= 3u << (bit - 1);
    }
  }
  if (bit == 0) {
    uint32_t ones = 0;
#pragma unroll
    for (int s = 0; s < S; ++s) ones |= (key[s] & 1u) << s;
    const uint32_t zeros = __reduce_add_sync(kFull, (uint32_t)__popc(alive & ~ones));
    if (k > zeros) res |= 1u;
  }
  return res;
}

constexpr int kWarpItemsPerBlock = 4;

// Per-warp buffer of a round's expanded entries (up to 128: the induced cost and the left child, the
// induced cost and the right child), read back as up to 256 children of 8 bytes.
__device__ __forceinline__ uint4 *child_buffer() {
  __shared__ uint4 buf[kWarpItemsPerBlock][kFrontierCap];
  return buf[(threadIdx.x >> 5) & (kWarpItemsPerBlock - 1)];
}

// The warp's smallest value (a NaN counts only where all are), one instruction in every round's dependent
// chain instead of six around an integer minimum: a chunk's search 17.3 -> 16.8 us on 65,536 triangles,
// 33.6 -> 33.0 on 4.19M.
__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// The patch as the search looks it up, one copy of the keys in every lane's registers: the nodes of
// get_subset (slot 1 empty: only slot 0 is looked at) and of the patched boxes. A search meets a
// patched node in a few rounds only, so an entry costs eight compares and the shared-memory patch
// is read behind one rarely taken branch.
struct PatchKeys {
  uint32_t node[4], box[4];
  __device__ __forceinline__ explicit PatchKeys(const PatchData *d) {
    const bool more = d->idx[1] != kNone;
    node[0] = d->idx[0];
#pragma unroll
    for (int k = 1; k < 4; ++k) node[k] = more ? d->idx[k] : kNone;
#pragma unroll
    for (int k = 0; k < 4; ++k) box[k] = d->apath[k];
  }
  __device__ __forceinline__ bool patched(uint32_t x) const {
    bool hit = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) hit |= x == node[k] || x == box[k];
    return hit;
  }
};

// One batched search. The frontier's entry e = slot * 32 + lane of slots 1 to 3 is live when e < m, slot
// 0's entries are the lanes of 'live'; the per-lane best is the lane's first entry of its smallest
// total, the lowest (cost, node) within a round.
struct BatchedSearch {
  float fc[kFrontier];
  uint32_t fn[kFrontier];
  uint32_t m;         // entries in the frontier (every one is within the bound)
  uint32_t live;      // lanes that hold one in slot 0 (the lowest min(m, 32), or after a narrow round any)
  uint32_t src;       // the lane of slot 0's (lane / 2)-th entry, for a narrow round
  uint32_t round;
  float4 rec[3];      // the tree record of slot 0's entry
  float bestCost;     // warp-uniform
  float myCost, myEntry;
  uint32_t myRound, myNode;
};

// The record of entry x (of the root where x is no node: the entry is flagged when it is evaluated).
__device__ __forceinline__ void load_entry(const Patch &p, uint32_t x, float4 (&rec)[3]) {
  const float4 *q = reinterpret_cast<const float4 *>(p.t + (x < p.numNodes ? x : p.root));
  rec[0] = __ldg(q);
  rec[1] = __ldg(q + 1);
  rec[2] = __ldg(q + 2);
}

// One round over S slots (32 S >= m): evaluates every entry, updates the bound and makes the
// children of the expanded entries the next frontier. The bound only changes here and an entry's
// two children share its induced cost, so every child passes the bound when its round comes: no
// entry is tested against it again. Which entry reached the best total is resolved once, after the
// last round (find_node_batched): a round needs the minimum itself only.
template <int S>
__device__ __forceinline__ void batched_round(const Patch &p, const PatchKeys &keys, BatchedSearch &st, const Box &nbox,
                                              float sarea, uint4 *buf, SearchCounters &ctr) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t ltMask = (1u << lane) - 1u;
  const float kInf = __int_as_float(0x7f800000);
  ctr.visits += st.m;
  float induced[S] = {};
  uint32_t left[S] = {}, right[S] = {};
  uint32_t inner = 0;  // bit s: this lane's slot s holds an inner node
  float roundCost = kInf, roundEntry = kInf;
  uint32_t roundNode = kNone;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    // other lanes compute on what they hold
    const bool live = s == 0 ? (st.live >> lane) & 1u : (uint32_t)s * 32u + lane < st.m;
    const uint32_t x = st.fn[s];
    float4 q[3];
    if (s == 0) {
      q[0] = st.rec[0]; q[1] = st.rec[1]; q[2] = st.rec[2];
    } else {
      if (!live) continue;
      load_entry(p, x, q);
    }
    if (live && x >= p.numNodes) p.bad = true;
    Box b;
    b.mn[0] = q[0].x; b.mn[1] = q[0].y; b.mn[2] = q[0].z;
    b.mx[0] = q[0].w; b.mx[1] = q[1].x; b.mx[2] = q[1].y;
    left[s] = __float_as_uint(q[1].w);
    right[s] = __float_as_uint(q[2].x);
    bool leaf = (__float_as_uint(q[2].y) & 0xFFFFu) != 0u;
    if (live && keys.patched(x)) {
      NodeP n;
      p.subset_aabb_from(x, q[0], q[1], q[2], n, b);
      left[s] = n.left;
      right[s] = n.right;
      leaf = n.isLeafFlag != 0;
    }
    const float ind = fmul(-1.0f, surface_area(b));
    merge_into(b, nbox);
    const float total = fadd(st.fc[s], surface_area(b));
    induced[s] = fadd(ind, total);
    inner |= (live && !leaf ? 1u : 0u) << s;
    if (S == 1) {
      roundCost = live ? total : kInf;
      roundEntry = st.fc[s];
      roundNode = x;
    } else if (live && (total < roundCost || (total == roundCost && (st.fc[s] < roundEntry ||
                                                                 (st.fc[s] == roundEntry && x < roundNode))))) {
      roundCost = total;
      roundEntry = st.fc[s];
      roundNode = x;
    }
  }
  const float kmin = warp_min(roundCost);
  if (kmin < st.bestCost) st.bestCost = kmin;
  if (roundCost < st.myCost) {
    st.myCost = roundCost;
    st.myEntry = roundEntry;
    st.myNode = roundNode;
    st.myRound = st.round;
  }
  // Children of the expanded entries: the k-th expanded entry (slot-major, then lane) writes
  // children 2k and 2k + 1 to the warp's buffer.
  // Rounds of one slot use the buffer's first two quarters in turn, so a round's writes never meet
  // the previous round's reads; wider rounds wait for those reads.
  if (S > 1) __syncwarp();
  else buf += (st.round & 1u) * 32u;
  uint32_t m = 0;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const bool kids = ((inner >> s) & 1u) && fadd(induced[s], sarea) < st.bestCost;
    const uint32_t kmask = __ballot_sync(kFull, kids);
    const uint32_t mk = 2u * __popc(kmask);
    if (kids)
      buf[m / 2 + __popc(kmask & ltMask)] =
          make_uint4(__float_as_uint(induced[s]), left[s], __float_as_uint(induced[s]), right[s]);
    if (m + mk > 32u && kids) {  // children past slot 0: warm their records in L2
      if (left[s] < p.numNodes) prefetch_node(p.t, left[s]);
      if (right[s] < p.numNodes) prefetch_node(p.t, right[s]);
    }
    m += mk;
  }
  __syncwarp();
  const uint2 *child = reinterpret_cast<const uint2 *>(buf);
  st.src = lane >> 1;
  st.live = m >= 32u ? 0xFFFFFFFFu : (1u << m) - 1u;
  if (S <= 2 || m <= kFrontierCap) {
    st.m = m;
    if (lane < m) {  // slot 0 first: its records are on their way while the other slots are read
      const uint2 v = child[lane];
      st.fc[0] = __uint_as_float(v.x);
      st.fn[0] = v.y;
      load_entry(p, v.y, st.rec);
    }
    if (m > 32u) {
#pragma unroll
      for (int s = 1; s < kFrontier; ++s) {
        const uint32_t e = (uint32_t)s * 32u + lane;
        if (e < m) {
          const uint2 v = child[e];
          st.fc[s] = __uint_as_float(v.x);
          st.fn[s] = v.y;
        }
      }
    }
  } else {
    // Overflow: keep the 128 lowest children in (cost, node) order. The frontier is unordered, so
    // only that set matters: select the 128th smallest cost, then, among the children at that cost
    // (siblings share their parent's), the lowest nodes up to 128 entries; the kept entries are
    // compacted to the front of the buffer.
    uint32_t key[2 * kFrontier], nd[2 * kFrontier];
    uint32_t in = 0;  // bit s: slot s holds a child
#pragma unroll
    for (int s = 0; s < 2 * kFrontier; ++s) {
      const uint32_t e = (uint32_t)s * 32u + lane;
      const uint2 v = e < m ? child[e] : make_uint2(0u, kNone);
      in |= (e < m ? 1u : 0u) << s;
      key[s] = f2ord(__uint_as_float(v.x));
      nd[s] = v.y;
    }
    __syncwarp();
    const uint32_t tc = warp_select_kth<2 * kFrontier>(key, in, kFrontierCap);
    uint32_t below = 0, tie = 0;
#pragma unroll
    for (int s = 0; s < 2 * kFrontier; ++s) {
      below += __popc(__ballot_sync(kFull, ((in >> s) & 1u) && key[s] < tc));
      tie |= (((in >> s) & 1u) && key[s] == tc ? 1u : 0u) << s;
    }
    uint32_t ties = 0;
#pragma unroll
    for (int s = 0; s < 2 * kFrontier; ++s) ties += __popc(__ballot_sync(kFull, (tie >> s) & 1u));
    const uint32_t need = kFrontierCap - below;  // 1 <= need <= ties
    uint32_t tn = 0xFFFFFFFFu;                    // largest node kept at cost tc
    if (need < ties) {
      if (need == 1u) {
        uint32_t nl = 0xFFFFFFFFu;
#pragma unroll
        for (int s = 0; s < 2 * kFrontier; ++s)
          if ((tie >> s) & 1u) nl = min(nl, nd[s]);
        tn = __reduce_min_sync(kFull, nl);
      } else {
        tn = warp_select_kth<2 * kFrontier>(nd, tie, need);
      }
    }
    uint32_t pos = 0;
    uint2 *kept = reinterpret_cast<uint2 *>(buf);
#pragma unroll
    for (int s = 0; s < 2 * kFrontier; ++s) {
      const bool keep = ((in >> s) & 1u) && (key[s] < tc || (((tie >> s) & 1u) && nd[s] <= tn));
      const uint32_t km = __ballot_sync(kFull, keep);
      if (keep) kept[pos + __popc(km & ltMask)] = make_uint2(__float_as_uint(ord2f(key[s])), nd[s]);
      pos += __popc(km);
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < kFrontier; ++s) {
      const uint2 v = child[(uint32_t)s * 32u + lane];
      st.fc[s] = __uint_as_float(v.x);
      st.fn[s] = v.y;
    }
    load_entry(p, st.fn[0], st.rec);
    ctr.overflow += m - kFrontierCap;
    st.m = kFrontierCap;
  }
  // A one-slot round may follow and write either quarter before every lane has read this one.
  if (S > 1) __syncwarp();
}

// A read-only load that is issued where it stands.
__device__ __forceinline__ float4 ldg_now(const float4 *p) {
  float4 v;
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// One round over at most 16 entries, which may stand in any lanes (st.live), and their at most 32
// children, one per lane. The children's records are fetched as soon as the entries' links are known,
// while the entries are evaluated and the round's bound is found: a round then takes little more
// than a record's round trip. Records of children that are not expanded are fetched for nothing,
// about as many as of those that are. The survivors stay in their lanes; src tells the next round
// where they are. The loads are volatile: they must not sink below the evaluation. A chunk's launch
// went from 18.0 to 17.3 us on 65,536 triangles and from 35.0 to 33.6 us on 4.19M.
__device__ __forceinline__ void narrow_round(const Patch &p, const PatchKeys &keys, BatchedSearch &st, const Box &nbox,
                                             float sarea, uint4 *buf, SearchCounters &ctr) {
  const uint32_t lane = threadIdx.x & 31u;
  const bool live = (st.live >> lane) & 1u;
  ctr.visits += st.m;
  const uint32_t x = st.fn[0];
  if (live && x >= p.numNodes) p.bad = true;
  Box b;
  b.mn[0] = st.rec[0].x; b.mn[1] = st.rec[0].y; b.mn[2] = st.rec[0].z;
  b.mx[0] = st.rec[0].w; b.mx[1] = st.rec[1].x; b.mx[2] = st.rec[1].y;
  uint32_t left = __float_as_uint(st.rec[1].w), right = __float_as_uint(st.rec[2].x);
  bool leaf = (__float_as_uint(st.rec[2].y) & 0xFFFFu) != 0u;
  if (live && keys.patched(x)) {
    NodeP n;
    p.subset_aabb_from(x, st.rec[0], st.rec[1], st.rec[2], n, b);
    left = n.left;
    right = n.right;
    leaf = n.isLeafFlag != 0;
  }
  // the children, and their records
  const uint32_t inner = __ballot_sync(kFull, live && !leaf);
  const uint32_t cl = __shfl_sync(kFull, left, st.src), cr = __shfl_sync(kFull, right, st.src);
  const uint32_t child = lane & 1u ? cr : cl;
  const bool have = lane < 2u * st.m && ((inner >> st.src) & 1u);
  {
    const float4 *q = reinterpret_cast<const float4 *>(p.t + (have && child < p.numNodes ? child : p.root));
    st.rec[0] = ldg_now(q);
    st.rec[1] = ldg_now(q + 1);
    st.rec[2] = ldg_now(q + 2);
  }
  // the entries
  const float ind = fmul(-1.0f, surface_area(b));
  merge_into(b, nbox);
  const float total = fadd(st.fc[0], surface_area(b));
  const float induced = fadd(ind, total);
  const float cost = live ? total : __int_as_float(0x7f800000);
  const float kmin = warp_min(cost);
  if (kmin < st.bestCost) st.bestCost = kmin;
  if (cost < st.myCost) {
    st.myCost = cost;
    st.myEntry = st.fc[0];
    st.myNode = x;
    st.myRound = st.round;
  }
  const uint32_t kids = __ballot_sync(kFull, live && !leaf && fadd(induced, sarea) < st.bestCost);
  st.fc[0] = __shfl_sync(kFull, induced, st.src);
  st.fn[0] = child;
  const bool stays = have && ((kids >> st.src) & 1u);
  st.live = __ballot_sync(kFull, stays);
  st.m = __popc(st.live);
  // two tables in turn: a round's writes never meet the previous round's reads
  uint32_t *lanes = reinterpret_cast<uint32_t *>(buf + kFrontierCap / 2) + (st.round & 1u) * 32u;
  if (stays) lanes[__popc(st.live & ((1u << lane) - 1u))] = lane;
  __syncwarp();
  st.src = (lane >> 1) < st.m ? lanes[lane >> 1] : 0u;
}

// findNode1's cost model in batched rounds (every lane of the warp calls it with the same patch).
__device__ __forceinline__ uint32_t find_node_batched(const Patch &p, uint32_t n, SearchCounters &ctr) {
  const uint32_t lane = threadIdx.x & 31u;
  __syncwarp();  // the warp's patch writes are visible to every lane
  const float kInf = __int_as_float(0x7f800000);
  const Box nbox = tree_box(p.t, p.chk(n));
  const float sarea = tree_sa(p.t, p.chk(n));
  const PatchKeys keys(p.d);
  BatchedSearch st;
#pragma unroll
  for (int s = 0; s < kFrontier; ++s) {
    st.fc[s] = 0.0f;
    st.fn[s] = p.root;
  }
  load_entry(p, p.root, st.rec);
  st.m = sarea < kInf ? 1u : 0u;  // the root's bound: 0 + sarea against no best yet
  st.live = st.m;
  st.src = 0;
  st.bestCost = kInf;
  st.myCost = st.myEntry = kInf;
  st.myNode = 0;
  st.myRound = 0xFFFFFFFFu;
  uint4 *buf = child_buffer();
  for (st.round = 0; st.m != 0u; ++st.round) {
    if (st.round > p.numNodes) {  // bounded: every round evaluates at least one node
      p.bad = true;
      break;
    }
    if (st.m <= 16u) narrow_round(p, keys, st, nbox, sarea, buf, ctr);
    else if (st.m <= 32u) batched_round<1>(p, keys, st, nbox, sarea, buf, ctr);
    else if (st.m <= 64u) batched_round<2>(p, keys, st, nbox, sarea, buf, ctr);
    else batched_round<kFrontier>(p, keys, st, nbox, sarea, buf, ctr);
  }
  // The first round that reached the best total, and its lowest (cost, node).
  const uint32_t cost = f2ord(st.myCost);
  uint32_t tied = __ballot_sync(kFull, cost == __reduce_min_sync(kFull, cost));
  if (__popc(tied) > 1) {
    const bool in0 = (tied >> lane) & 1u;
    const uint32_t r = __reduce_min_sync(kFull, in0 ? st.myRound : 0xFFFFFFFFu);
    const bool in1 = in0 && st.myRound == r;
    const uint32_t c = __reduce_min_sync(kFull, in1 ? f2ord(st.myEntry) : 0xFFFFFFFFu);
    const bool in2 = in1 && f2ord(st.myEntry) == c;
    const uint32_t node = __reduce_min_sync(kFull, in2 ? st.myNode : 0xFFFFFFFFu);
    tied = __ballot_sync(kFull, in2 && st.myNode == node);
  }
  const uint32_t best = __shfl_sync(kFull, st.myNode, __ffs(tied) - 1);
  __syncwarp();  // every lane is done reading the patch before it changes again
  p.bad = __any_sync(kFull, p.bad);
  return best;
}

// reinsert (Bittner13CUDA.cu:308-358).
// MODE: BVHGB_SEARCH_BATCHED (warp-cooperative), BVHGB_SEARCH_HEAP (findNode1) or
// BVHGB_SEARCH_ALT (findNode2).
template <int MODE>
__device__ __forceinline__ bool reinsert(Patch &p, uint32_t x, uint32_t unused, bool update, const Heap &pq,
                                         uint32_t cap, SearchCounters &ctr) {
  const uint32_t best = MODE == BVHGB_SEARCH_BATCHED ? find_node_batched(p, x, ctr)
                        : MODE == BVHGB_SEARCH_ALT   ? find_node2(p, x, ctr)
                                                     : find_node(p, x, pq, cap, ctr);
  if (best == p.root) return false;
  const NodeP nx = tree_node(p.t, p.chk(x)), nb = tree_node(p.t, p.chk(best));
  const uint32_t bpi = p.index(best);
  uint32_t sb = update ? P_1ST_BEST : P_2ND_BEST;
  const uint32_t sx = update ? P_1ST_INSERT : P_2ND_INSERT;
  const uint32_t su = update ? P_NODE : P_PARENT;
  if (bpi == kNone) {
    p.d->idx[sb] = best;
    p.d->nd[sb] = nb;
  } else if (bpi == P_GRAND_PARENT) {
    sb = P_GRAND_PARENT;
  } else {
    p.move(bpi, sb);
  }
  p.d->idx[sx] = x;
  p.d->nd[sx] = nx;
  const uint32_t ri = p.d->nd[sb].parent;
  const uint32_t rpi = p.index(ri);
  const uint32_t sr = rpi == kNone ? p.patch_node(ri, update ? P_1ST_ROOT : P_2ND_ROOT)
                                   : p.move(rpi, update ? P_1ST_ROOT : P_2ND_ROOT);
  if (p.d->nd[sb].isLeft) {
    p.d->nd[sr].left = unused;
    p.d->nd[su].isLeft = 1;
  } else {
    p.d->nd[sr].right = unused;
    p.d->nd[su].isLeft = 0;
  }
  p.d->nd[su].parent = ri;
  p.d->nd[su].left = best;
  p.d->nd[su].right = x;
  p.d->nd[sb].parent = unused;
  p.d->nd[sb].isLeft = 1;
  p.d->nd[sx].parent = unused;
  p.d->nd[sx].isLeft = 0;
  if (update) p.patch_aabb_from(unused, 1);
  return true;
}

// Both reinsertions of a removed node on a whole warp: one copy of the search's code for the two
// (a launch starts with cold instruction caches).
__device__ __forceinline__ bool reinsert_both(Patch &p, const uint32_t ins[2], const uint32_t un[2], SearchCounters &ctr) {
  const Heap unused{nullptr, nullptr};
#pragma unroll 1
  for (int k = 0; k < 2; ++k)
    if (!reinsert<BVHGB_SEARCH_BATCHED>(p, k ? ins[1] : ins[0], k ? un[1] : un[0], k == 0, unused, 0, ctr)) return false;
  return true;
}

// ---- per-item steps shared by the single-tree and the batched kernels ---------------------------
// (t, root, numNodes) describe one tree; owner / counter point at that tree's entries; rank is the
// item's position in its tree's chunk (lower rank wins a conflict).

// The patch storage of this warp (blocks of kWarpItemsPerBlock warps).
__device__ __forceinline__ PatchData *warp_patch_data() {
  __shared__ PatchData pd[kWarpItemsPerBlock];
  return &pd[(threadIdx.x >> 5) & (kWarpItemsPerBlock - 1)];
}

// kRemoveAndReinsert for one item on a whole warp (batched search); lane 0 publishes.
__device__ __forceinline__ void warp_patch_item(const bvhgb_node *__restrict__ t, uint32_t root, uint32_t numNodes,
                                                uint32_t node, bool ok, uint32_t rank, PatchOut *__restrict__ out,
                                                uint32_t *__restrict__ valid, uint32_t *__restrict__ toFix3,
                                                uint32_t *__restrict__ owner, unsigned long long *__restrict__ stats,
                                                uint32_t *__restrict__ err) {
  const uint32_t lane = threadIdx.x & 31u;
  Patch p;
  p.d = warp_patch_data();
  p.t = t;
  p.root = root;
  p.numNodes = numNodes;
  p.bad = false;
  p.clear();
  SearchCounters ctr = {0u, 0u};
  uint32_t ins[2], un[2], g = kNone;
  ok = ok && remove_node(p, node, ins, un, g);
  ok = ok && reinsert_both(p, ins, un, ctr);
  p.bad = __any_sync(kFull, p.bad);
  if (p.bad) ok = false;
  __syncwarp();
  if (lane < NSLOT) {  // a lane per slot
    const uint32_t y = ok ? p.d->idx[lane] : kNone;
    out->idx[lane] = y;
    out->nd[lane] = p.d->nd[lane];
    if (y != kNone) atomicMin(&owner[y], rank);
  }
  if (lane != 0) return;
  if (p.bad) atomicOr(err, kErrBadIndex);
  *valid = ok ? 1u : 0u;
  toFix3[0] = ok ? g : kNone;
  toFix3[1] = ok ? un[0] : kNone;
  toFix3[2] = ok ? un[1] : kNone;
  if (!ok) atomicAdd(&stats[S_INVALID], 1ull);
  if (ctr.overflow) atomicAdd(&stats[S_OVERFLOW], (unsigned long long)ctr.overflow);
  atomicAdd(&stats[S_VISITS], (unsigned long long)ctr.visits);
  atomicAdd(&stats[S_ITEMS], 1ull);
}

// kCheckConflicts + kApplyPatches for one item.
__device__ __forceinline__ void apply_item(bvhgb_node *t, const PatchOut &in, uint32_t *__restrict__ valid,
                                           uint32_t *__restrict__ toFix3, const uint32_t *__restrict__ owner,
                                           uint32_t rank, unsigned long long *__restrict__ stats) {
  if (!*valid) return;
  bool win = true;
#pragma unroll
  for (int s = 0; s < NSLOT; ++s) {
    const uint32_t x = in.idx[s];
    if (x != kNone && owner[x] != rank) win = false;
  }
  if (!win) {
    *valid = 0;
    toFix3[0] = toFix3[1] = toFix3[2] = kNone;
    atomicAdd(&stats[S_CONFLICT], 1ull);
    return;
  }
#pragma unroll
  for (int s = 0; s < NSLOT; ++s) {
    const uint32_t x = in.idx[s];
    if (x == kNone) continue;
    const NodeP n = in.nd[s];
    t[x].parent = n.parent;
    t[x].left = n.left;
    t[x].right = n.right;
    t[x].isLeft = n.isLeft;
  }
  atomicAdd(&stats[S_APPLIED], 1ull);
}

// Apply and count in one launch, three climbs per item. The count climbs the new tree while the
// winners' patches are still being written: a node that a winning item patched takes its new parent
// from that item's patch record, every other node keeps its parent (its record is not written in
// this launch). A node y is patched by a winner iff its owner o (the lowest rank that claimed it;
// the claims are final before this launch) wins, i.e. owns every node of its own patch: a higher
// rank that also claimed y does not own y, so it cannot win. The claims are released later, by
// the refit launch.
struct PatchIdx {
  uint32_t v[NSLOT];
};
__device__ __forceinline__ PatchIdx patch_idx(const PatchOut &in) {
  const uint4 *q = reinterpret_cast<const uint4 *>(in.idx);
  const uint4 a = __ldg(q), b = __ldg(q + 1);
  const uint2 c = __ldg(reinterpret_cast<const uint2 *>(q + 2));
  return {{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y}};
}
__device__ __forceinline__ bool item_wins(const PatchIdx &in, const uint32_t *__restrict__ owner, uint32_t rank) {
  uint32_t o[NSLOT];  // all loads before the first compare
#pragma unroll
  for (int s = 0; s < NSLOT; ++s) o[s] = in.v[s] != kNone ? __ldg(owner + in.v[s]) : rank;
  bool win = true;
#pragma unroll
  for (int s = 0; s < NSLOT; ++s) win = win && o[s] == rank;
  return win;
}

// Parent and left link of y in the tree being patched, given y's owner o and its links before the
// patch. (A node's patched links are read from the patch of the winner that owns it.)
__device__ __forceinline__ uint2 new_links(const PatchOut *__restrict__ in, const uint32_t *__restrict__ owner,
                                           uint32_t y, uint32_t o, uint2 links) {
  if (o == kNone) return links;
  const PatchIdx idx = patch_idx(in[o]);
  if (!item_wins(idx, owner, o)) return links;
  uint32_t s = kNone;
#pragma unroll
  for (int k = NSLOT - 1; k >= 0; --k)
    if (idx.v[k] == y) s = (uint32_t)k;
  if (s == kNone) return links;
  return make_uint2(in[o].nd[s].parent, in[o].nd[s].left);
}

// The arrivals a node's refit waits for are marked in its counter word: one bit per child that lies on
// a dirty path and one for a node that starts a path. Marks are set without reading them back (an
// atomic or whose result nobody waits for), so a level of a climb is one load round trip: owner,
// links and the marks set so far go out together. A climb that finds marks leaves the rest of the
// way to the climb that set the first one; two that find none go on both, and set the same bits.
// (With counts, a level was one atomic round trip: a chunk's launch took 7.8 us on 65,536 triangles
// and 11.2 us on 4.19M, with marks 7.0 and 10.0; the refit of the latter went from 17.6 to 16.3.)
constexpr uint32_t kMarkLeft = 1u, kMarkRight = 2u, kMarkStart = 4u, kMarks = 7u;

__device__ __forceinline__ uint2 ld_links(const bvhgb_node *t, uint32_t x) {  // parent, left
  return __ldcg(reinterpret_cast<const uint2 *>(reinterpret_cast<const char *>(t + x) + 24));
}

// Climb j of item k: all three decide the item's outcome (the owner array is final; valid[k], the
// patch kernel's decision, is only read here, so the three climbs see the same value); climb 0
// writes the patch and the statistics, climb j marks the item's j-th dirty path (kFixTree3_1) in
// the new tree.
__device__ __forceinline__ void apply_count_path(bvhgb_node *t, uint32_t root, uint32_t numNodes,
                                                 const PatchOut *__restrict__ in, uint32_t k, uint32_t j,
                                                 const uint32_t *__restrict__ valid, uint32_t *__restrict__ toFix,
                                                 const uint32_t *__restrict__ owner, uint32_t *__restrict__ counter,
                                                 unsigned long long *__restrict__ stats, uint32_t *__restrict__ err) {
  const uint32_t isValid = __ldg(valid + k);
  uint32_t x = toFix[3 * k + j];
  const PatchOut &me = in[k];
  const PatchIdx idx = patch_idx(me);
  if (!isValid) return;  // refused by removeNode or the search: it claimed nothing
  if (!item_wins(idx, owner, k)) {
    toFix[3 * k + j] = kNone;  // the refit skips a lost item's paths
    if (j == 0) atomicAdd(&stats[S_CONFLICT], 1ull);
    return;
  }
  if (j == 0) {
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) {
      const uint32_t y = idx.v[s];
      if (y == kNone) continue;
      const NodeP n = me.nd[s];
      t[y].parent = n.parent;
      t[y].left = n.left;
      t[y].right = n.right;
      t[y].isLeft = n.isLeft;
    }
    atomicAdd(&stats[S_APPLIED], 1ull);
  }
  if (x == kNone) return;
  uint32_t from = kNone;
  for (uint32_t steps = 0;; ++steps) {
    if (x >= numNodes || steps > numNodes) {
      atomicOr(err, kErrBadIndex);
      break;
    }
    const uint32_t o = __ldg(owner + x), marks = __ldcg(&counter[x]);
    uint2 links = ld_links(t, x);  // discarded if a winner rewrites them in this launch
    links = new_links(in, owner, x, o, links);
    atomicOr(&counter[x], from == kNone ? kMarkStart : links.y == from ? kMarkLeft : kMarkRight);
    if (marks != 0u || x == root) break;
    from = x;
    x = links.x;
  }
}

// Release a third of an item's claims (after the launch that counted with them).
__device__ __forceinline__ void release_claims(const PatchOut &in, uint32_t j, uint32_t *__restrict__ owner) {
  for (uint32_t s = j; s < (uint32_t)NSLOT; s += 3) {
    const uint32_t y = in.idx[s];
    if (y != kNone) owner[y] = kNone;
  }
}

// Release a third of an item's claims and mark one dirty path (kFixTree3_1), links final.
__device__ __forceinline__ void count_path(const bvhgb_node *__restrict__ t, uint32_t root, uint32_t numNodes,
                                          const PatchOut &in, uint32_t j, uint32_t x, uint32_t *__restrict__ owner,
                                          uint32_t *__restrict__ counter, uint32_t *__restrict__ err) {
  release_claims(in, j, owner);
  if (x == kNone) return;
  uint32_t from = kNone;
  for (uint32_t steps = 0;; ++steps) {
    if (x >= numNodes || steps > numNodes) {
      atomicOr(err, kErrBadIndex);
      break;
    }
    const uint32_t marks = __ldcg(&counter[x]);
    const uint2 links = ld_links(t, x);
    atomicOr(&counter[x], from == kNone ? kMarkStart : links.y == from ? kMarkLeft : kMarkRight);
    if (marks != 0u || x == root) break;
    from = x;
    x = links.x;
  }
}

// ---- dirty-path refit (kFixTree3_2) ------------------------------------------------------------
// The last path to arrive at a node recomputes its box. A node's counter word (set by the count pass)
// holds the arrivals to expect as marks: a dirty left or right child, a path that starts here (grand
// parent or reused node: its children were relinked, so it is always recomputed). Each arrival sets
// its own arrival bit (the mark shifted by 8) and, for the child it comes from (side 0 left, 1
// right), bit 16 + side if it rewrote that child's box in this launch and bit 18 + side if the child
// changed (rewritten, or a start node, which may have moved under a new parent). The arrival that
// completes the marks is the last.
//
// Every counter update is relaxed: a rewritten box does not travel through the node record, whose
// visibility would need a release by the writer and an acquire by the reader (fences that cost
// several L2 round trips each), but through a mail slot of three 64-bit words per child that
// carries its own validity. A path that may not be the last at a node posts its child's new box
// there before its update; the last arrival finds the posting side in the counter bits and reads
// the slot until all three words differ from the empty pattern (each 64-bit word is written and
// read whole), then empties it again; a path that posted and turned out last empties its own. A
// child whose box was not rewritten in this launch is read from its record, loaded speculatively
// together with the counter update. (Two coordinates of a box that both hold the bit pattern
// 0xFFFFFFFF would read as empty: the wait then ends at its limit with kErrTimeout.)
//
// Links do not change in this launch and a node's box is written only by its last arrival, so the
// climb reads one level ahead: while it handles node x it loads the parent's record and counter. A
// node whose word already shows this path as the only arrival left needs no update at all.
constexpr unsigned long long kMailEmpty = 0xFFFFFFFFFFFFFFFFull;

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  return (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32);
}

__device__ __forceinline__ void mail_post(unsigned long long *mail, uint32_t child, const Box &b) {
  unsigned long long *m = mail + 3ull * child;
  __stcg(m, pack2(b.mn[0], b.mn[1]));
  __stcg(m + 1, pack2(b.mn[2], b.mx[0]));
  __stcg(m + 2, pack2(b.mx[1], b.mx[2]));
}

__device__ __forceinline__ void mail_clear(unsigned long long *mail, uint32_t child) {
  unsigned long long *m = mail + 3ull * child;
  __stcg(m, kMailEmpty);
  __stcg(m + 1, kMailEmpty);
  __stcg(m + 2, kMailEmpty);
}

// Takes the box posted for 'child' (bounded wait per word) and empties the slot.
__device__ __forceinline__ Box mail_take(unsigned long long *mail, uint32_t child, uint32_t *__restrict__ err) {
  unsigned long long *m = mail + 3ull * child;
  unsigned long long w[3] = {__ldcg(m), __ldcg(m + 1), __ldcg(m + 2)};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    for (uint32_t spins = 0; w[q] == kMailEmpty; ++spins) {
      if (spins > kSpinLimit) {
        atomicOr(err, kErrTimeout);
        break;
      }
      __nanosleep(32);
      w[q] = __ldcg(m + q);
    }
  }
  mail_clear(mail, child);
  Box b;
  b.mn[0] = __uint_as_float((uint32_t)w[0]); b.mn[1] = __uint_as_float((uint32_t)(w[0] >> 32));
  b.mn[2] = __uint_as_float((uint32_t)w[1]); b.mx[0] = __uint_as_float((uint32_t)(w[1] >> 32));
  b.mx[1] = __uint_as_float((uint32_t)w[2]); b.mx[2] = __uint_as_float((uint32_t)(w[2] >> 32));
  return b;
}

__device__ __forceinline__ void refit_path(bvhgb_node *t, uint32_t root, uint32_t numNodes, uint32_t x,
                                          uint32_t *__restrict__ counter, unsigned long long *__restrict__ mail,
                                          uint32_t *__restrict__ err) {
  if (x == kNone) return;
  if (x >= numNodes) {
    atomicOr(err, kErrBadIndex);
    return;
  }
  const float4 *q = reinterpret_cast<const float4 *>(t + x);
  float4 w0 = __ldcg(q), w1 = __ldcg(q + 1), w2 = __ldcg(q + 2);  // [mn.xyz mx.x] [mx.yz parent left] [right flags . sa]
  uint32_t cnt = __ldcg(&counter[x]);
  uint32_t from = kNone;  // child the path came from, whose box is 'cur'
  Box cur;
  bool written = false;   // cur was rewritten in this launch
  bool changed = true;    // the start node's children were relinked
  for (uint32_t steps = 0;; ++steps) {
    const uint32_t parent = __float_as_uint(w1.z), l = __float_as_uint(w1.w), r = __float_as_uint(w2.x);
    if ((__float_as_uint(w2.y) & 0xFFFFu) || l >= numNodes || r >= numNodes || steps > numNodes ||
        (from != kNone && from != l && from != r)) {
      if (!(__float_as_uint(w2.y) & 0xFFFFu)) atomicOr(err, kErrBadIndex);
      return;
    }
    const bool top = x == root;
    if (!top && parent >= numNodes) {
      atomicOr(err, kErrBadIndex);
      return;
    }
    const uint32_t side = from == r ? 1u : 0u;  // meaningful only when from != kNone
    // this level's child boxes from their records (valid unless rewritten in this launch) and the
    // next level's record and counter
    Box lb = from == l ? cur : load_box_cg(t + l);
    Box rb = from == r ? cur : load_box_cg(t + r);
    float4 n0 = w0, n1 = w1, n2 = w2;
    uint32_t ncnt = 0u;
    if (!top) {
      const float4 *pq = reinterpret_cast<const float4 *>(t + parent);
      n0 = __ldcg(pq);
      n1 = __ldcg(pq + 1);
      n2 = __ldcg(pq + 2);
      ncnt = __ldcg(&counter[parent]);
    }
    uint32_t old = cnt;
    const uint32_t mark = from == kNone ? kMarkStart : side ? kMarkRight : kMarkLeft;
    if ((cnt & kMarks & ~(cnt >> 8)) != mark) {  // other arrivals are still expected here
      const bool post = from != kNone && written;
      if (post) mail_post(mail, from, cur);
      uint32_t add = mark << 8;
      if (from != kNone) add |= (written ? (1u << (16 + side)) : 0u) | (changed ? (1u << (18 + side)) : 0u);
      old = atomicOr(&counter[x], add);
      if ((old & kMarks & ~(old >> 8)) != mark) return;  // not the last arrival
      if (post) mail_clear(mail, from);   // posted for nobody
    }
    if (from != l && ((old >> 16) & 1u)) lb = mail_take(mail, l, err);
    if (from != r && ((old >> 17) & 1u)) rb = mail_take(mail, r, err);
    counter[x] = 0u;
    const bool start = (old & kMarkStart) != 0u;  // x started a path (this one or an earlier arrival)
    const bool anyChanged = changed || start || ((old >> 18) & 3u) != 0u;
    Box b;
    b.mn[0] = w0.x; b.mn[1] = w0.y; b.mn[2] = w0.z;
    b.mx[0] = w0.w; b.mx[1] = w1.x; b.mx[2] = w1.y;
    bool upChanged = false;
    if (anyChanged) {
      merge_into(lb, rb);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        upChanged |= __float_as_uint(lb.mn[k]) != __float_as_uint(b.mn[k]) ||
                     __float_as_uint(lb.mx[k]) != __float_as_uint(b.mx[k]);
      if (upChanged) {
        float4 *p = reinterpret_cast<float4 *>(t + x);
        p[0] = make_float4(lb.mn[0], lb.mn[1], lb.mn[2], lb.mx[0]);
        p[1] = make_float4(lb.mx[1], lb.mx[2], w1.z, w1.w);
        t[x].surfaceArea = surface_area(lb);
        b = lb;
      }
    }
    if (top) return;
    // A start node may have moved (a reused node now hangs under a new parent), so its parent
    // cannot compare against the old box: it always counts as changed.
    written = upChanged;
    changed = upChanged || start;
    from = x;
    cur = b;
    x = parent;
    w0 = n0;
    w1 = n1;
    w2 = n2;
    cnt = ncnt;
  }
}

// kCalcCost for one inner node (0 for a leaf).
__device__ __forceinline__ float inefficiency(const bvhgb_node *__restrict__ t, uint32_t x) {
  const float4 *p = reinterpret_cast<const float4 *>(t + x);
  const float4 b = __ldg(p + 1), c = __ldg(p + 2);
  if ((__float_as_uint(c.y) & 0xFFFFu) != 0) return 0.0f;
  const float sa = c.w;
  const float l = __ldg(&t[__float_as_uint(b.w)].surfaceArea);
  const float r = __ldg(&t[__float_as_uint(c.x)].surfaceArea);
  const float num = fmul(fmul(fmul(sa, sa), sa), 2.0f);
  const float den = fmul(fadd(l, r), l < r ? l : r);
  return fdiv(num, den);
}

}  // namespace
}  // namespace bvhgb
