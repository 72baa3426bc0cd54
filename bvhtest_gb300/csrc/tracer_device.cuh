// Device side of the closest-hit tracer (lib/tracer/CUDAKernels.cu:66-223, restated with a
// watertight triangle test and a short stack), shared by the single-tree kernels (tracer.cu) and
// the batched ones (batch.cu). Errors are OR-ed into the word the caller passes.
#pragma once

#include "common.cuh"

namespace bvhgb {
namespace {

constexpr int kStack = 96;
constexpr float kFarScale = 1.0000004f;   // 1 + 2 * gamma(3), gamma(n) = n u / (1 - n u), u = 2^-24
constexpr float kBestSlack = 1.0000153f;  // relative slack on the best t when culling boxes

struct RayPre {
  float o[3], d[3], inv[3];
  float sx, sy, sz;
  int kx, ky, kz;
};

__device__ __forceinline__ void setup_ray(RayPre &r) {
#pragma unroll
  for (int k = 0; k < 3; ++k) r.inv[k] = fdiv(1.0f, r.d[k]);
  float ax = fabsf(r.d[0]), ay = fabsf(r.d[1]), az = fabsf(r.d[2]);
  int kz = (ax >= ay) ? (ax >= az ? 0 : 2) : (ay >= az ? 1 : 2);
  int kx = kz + 1 == 3 ? 0 : kz + 1;
  int ky = kx + 1 == 3 ? 0 : kx + 1;
  float dz = kz == 0 ? r.d[0] : (kz == 1 ? r.d[1] : r.d[2]);
  if (dz < 0.0f) { int t = kx; kx = ky; ky = t; }
  r.kx = kx; r.ky = ky; r.kz = kz;
  float dx = kx == 0 ? r.d[0] : (kx == 1 ? r.d[1] : r.d[2]);
  float dy = ky == 0 ? r.d[0] : (ky == 1 ? r.d[1] : r.d[2]);
  r.sx = fdiv(dx, dz);
  r.sy = fdiv(dy, dz);
  r.sz = fdiv(1.0f, dz);
}

__device__ __forceinline__ float pick(const float *v, int k) { return k == 0 ? v[0] : (k == 1 ? v[1] : v[2]); }

// Watertight ray/triangle test; every operation rounds once (matches the oracle bit for bit). The
// vertices come with their components in the ray's order (kx, ky, kz), which is how they are loaded:
// nothing is selected here.
__device__ __forceinline__ bool ray_tri(const RayPre &r, const float *v0, const float *v1, const float *v2, float tmin,
                                        float tmax, bool cull, float &tout) {
  const float ox = pick(r.o, r.kx), oy = pick(r.o, r.ky), oz = pick(r.o, r.kz);
  const float Akz = fsub(v0[2], oz), Bkz = fsub(v1[2], oz), Ckz = fsub(v2[2], oz);
  const float Ax = fsub(fsub(v0[0], ox), fmul(r.sx, Akz)), Ay = fsub(fsub(v0[1], oy), fmul(r.sy, Akz));
  const float Bx = fsub(fsub(v1[0], ox), fmul(r.sx, Bkz)), By = fsub(fsub(v1[1], oy), fmul(r.sy, Bkz));
  const float Cx = fsub(fsub(v2[0], ox), fmul(r.sx, Ckz)), Cy = fsub(fsub(v2[1], oy), fmul(r.sy, Ckz));
  float U = fsub(fmul(Cx, By), fmul(Cy, Bx));
  float V = fsub(fmul(Ax, Cy), fmul(Ay, Cx));
  float W = fsub(fmul(Bx, Ay), fmul(By, Ax));
  if (U == 0.0f || V == 0.0f || W == 0.0f) {
    U = (float)__dsub_rn(__dmul_rn((double)Cx, (double)By), __dmul_rn((double)Cy, (double)Bx));
    V = (float)__dsub_rn(__dmul_rn((double)Ax, (double)Cy), __dmul_rn((double)Ay, (double)Cx));
    W = (float)__dsub_rn(__dmul_rn((double)Bx, (double)Ay), __dmul_rn((double)By, (double)Ax));
  }
  if (cull) {
    if (U < 0.0f || V < 0.0f || W < 0.0f) return false;
  } else {
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
  }
  const float det = fadd(fadd(U, V), W);
  if (det == 0.0f) return false;
  const float Az = fmul(r.sz, Akz), Bz = fmul(r.sz, Bkz), Cz = fmul(r.sz, Ckz);
  const float T = fadd(fadd(fmul(U, Az), fmul(V, Bz)), fmul(W, Cz));
  const float t = fdiv(T, det);
  if (!(t > tmin) || !(t <= tmax)) return false;
  tout = t;
  return true;
}

// Robust slab test; sign-selected planes make 0 * inf NaNs drop out of the min/max. The six plane
// distances are three packed subtractions and products over the box's words as they are loaded; the
// far distances are scaled once, after their minimum (rounding is monotonic, so the minimum of the
// scaled distances is the scaled minimum). 18 instructions instead of 27.
__device__ __forceinline__ bool box_hit(const RayPre &r, float4 a, float4 b, float tmin, float tmax, float &tn) {
  const float2 p = mul2(add2(make_float2(a.x, a.y), make_float2(-r.o[0], -r.o[1])), make_float2(r.inv[0], r.inv[1]));
  const float2 q = mul2(add2(make_float2(a.z, a.w), make_float2(-r.o[2], -r.o[0])), make_float2(r.inv[2], r.inv[0]));
  const float2 w = mul2(add2(make_float2(b.x, b.y), make_float2(-r.o[1], -r.o[2])), make_float2(r.inv[1], r.inv[2]));
  const bool nx = __float_as_int(r.inv[0]) < 0, ny = __float_as_int(r.inv[1]) < 0, nz = __float_as_int(r.inv[2]) < 0;
  const float t0 = fmaxf(fmaxf(fmaxf(nx ? q.y : p.x, ny ? w.x : p.y), nz ? w.y : q.x), tmin);
  const float tf = fminf(fminf(nx ? p.x : q.y, ny ? p.y : w.x), nz ? q.x : w.y);
  const float t1 = fminf(fmul(tf, kFarScale), tmax);
  tn = t0;
  return t0 <= t1;
}

struct Hit {
  uint32_t prim;
  float t;
};

__device__ __forceinline__ void load_tri(const float *__restrict__ vert, const uint32_t *__restrict__ faces, uint32_t f,
                                         float *v0, float *v1, float *v2) {
  const uint32_t a = __ldg(faces + 3 * (size_t)f), b = __ldg(faces + 3 * (size_t)f + 1), c = __ldg(faces + 3 * (size_t)f + 2);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    v0[k] = __ldg(vert + 3 * (size_t)a + k);
    v1[k] = __ldg(vert + 3 * (size_t)b + k);
    v2[k] = __ldg(vert + 3 * (size_t)c + k);
  }
}

// The same triangle with every vertex's components in the ray's order.
__device__ __forceinline__ void load_tri_permuted(const RayPre &r, const float *__restrict__ vert,
                                                  const uint32_t *__restrict__ faces, uint32_t f, float *v0, float *v1,
                                                  float *v2) {
  const uint32_t a = __ldg(faces + 3 * (size_t)f), b = __ldg(faces + 3 * (size_t)f + 1), c = __ldg(faces + 3 * (size_t)f + 2);
  const int k[3] = {r.kx, r.ky, r.kz};
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    v0[j] = __ldg(vert + 3 * (size_t)a + k[j]);
    v1[j] = __ldg(vert + 3 * (size_t)b + k[j]);
    v2[j] = __ldg(vert + 3 * (size_t)c + k[j]);
  }
}

__device__ __forceinline__ void test_leaf(const RayPre &r, const float *__restrict__ vert,
                                          const uint32_t *__restrict__ faces, uint32_t first, uint32_t count,
                                          float tmin, float tmax, bool cull, Hit &h) {
  for (uint32_t f = first; f < first + count; ++f) {
    float v0[3], v1[3], v2[3], t;
    load_tri_permuted(r, vert, faces, f, v0, v1, v2);
    if (ray_tri(r, v0, v1, v2, tmin, tmax, cull, t)) {
      if (h.prim == kNone || t < h.t || (t == h.t && f < h.prim)) {
        h.t = t;
        h.prim = f;
      }
    }
  }
}

// Closest hit through the 48-byte node array. Returns the number of inner nodes visited. A stack entry
// holds the far child's links, which were loaded with its box: taking it off needs no load.
__device__ __forceinline__ uint32_t traverse(const RayPre &r, const bvhgb_node *__restrict__ nodes, uint32_t numNodes,
                                             uint32_t root, const float *__restrict__ vert,
                                             const uint32_t *__restrict__ faces, float tmin, float tmax, bool cull,
                                             Hit &h, uint32_t *err) {
  uint4 stack[kStack];  // left, right, leaf, entry distance
  int sp = 0;
  uint32_t visits = 0;
  h.prim = kNone;
  h.t = tmax;
  float lim = tmax;
  float4 a, b, c;
  load_node(nodes, root, a, b, c);
  float tn;
  if (!box_hit(r, a, b, tmin, tmax, tn)) return 0;
  uint32_t left = __float_as_uint(b.w), right = __float_as_uint(c.x);
  bool leaf = (__float_as_uint(c.y) & 0xFFFFu) != 0;
  for (;;) {
    bool go = false;
    if (leaf) {
      test_leaf(r, vert, faces, left, right, tmin, tmax, cull, h);
      if (h.prim != kNone) lim = fmul(h.t, kBestSlack);
    } else {
      // A tree visits each node at most once; the bound turns a cyclic (corrupted) input into an error.
      if (++visits > numNodes) {
        atomicOr(err, kErrBadIndex);
        break;
      }
      if (left >= numNodes || right >= numNodes) {
        atomicOr(err, kErrBadIndex);
      } else {
        float4 la, lb, lc, ra, rb, rc;
        load_node(nodes, left, la, lb, lc);
        load_node(nodes, right, ra, rb, rc);
        float tl, tr;
        const bool hl = box_hit(r, la, lb, tmin, lim, tl);
        const bool hr = box_hit(r, ra, rb, tmin, lim, tr);
        const bool lfirst = hl && (!hr || tl <= tr);
        if (hl && hr) {
          if (sp < kStack)
            stack[sp++] = lfirst ? make_uint4(__float_as_uint(rb.w), __float_as_uint(rc.x), __float_as_uint(rc.y), __float_as_uint(tr))
                                 : make_uint4(__float_as_uint(lb.w), __float_as_uint(lc.x), __float_as_uint(lc.y), __float_as_uint(tl));
          else
            atomicOr(err, kErrStackOverflow);
        }
        go = hl || hr;
        if (go) {
          left = __float_as_uint(lfirst ? lb.w : rb.w);
          right = __float_as_uint(lfirst ? lc.x : rc.x);
          leaf = (__float_as_uint(lfirst ? lc.y : rc.y) & 0xFFFFu) != 0;
        }
      }
    }
    // Pop the next subtree whose entry distance can still beat the best hit.
    while (!go && sp > 0) {
      const uint4 e = stack[--sp];
      go = __uint_as_float(e.w) <= lim;
      left = e.x;
      right = e.y;
      leaf = (e.z & 0xFFFFu) != 0;
    }
    if (!go) break;
  }
  return visits;
}


// ---- traversal records --------------------------------------------------------------------------
// Traversal record of an inner node: both children's boxes and references in 64 bytes (one aligned
// pair of sectors), so a visit loads one record instead of the children's two 48-byte nodes, and a
// leaf child's faces are known without loading the leaf. ref = the node id of an inner child, the
// first face of a leaf child; count = 0 for an inner child, the leaf's face count. Built from the
// drop-in node array before a trace (the boxes are copied bit for bit, so hits do not change).
struct __align__(64) TravNode {
  float4 q0;  // left mn.xyz, left mx.x
  float4 q1;  // left mx.y mx.z, right mn.x mn.y
  float4 q2;  // right mn.z, right mx.xyz
  uint4 q3;   // left ref, right ref, left count, right count
};


__device__ __forceinline__ void build_trav(const bvhgb_node *__restrict__ nodes, uint32_t numNodes, uint32_t x,
                                           TravNode *__restrict__ out, uint32_t *err) {
  const float4 *p = reinterpret_cast<const float4 *>(nodes + x);
  const float4 b = __ldg(p + 1), c = __ldg(p + 2);
  if (__float_as_uint(c.y) & 0xFFFFu) return;  // leaves have no record
  const uint32_t l = __float_as_uint(b.w), r = __float_as_uint(c.x);
  TravNode t;
  if (l >= numNodes || r >= numNodes) {  // no child can be hit: an empty box on both sides
    atomicOr(err, kErrBadIndex);
    const float inf = __int_as_float(0x7f800000);
    t.q0 = make_float4(inf, inf, inf, -inf);
    t.q1 = make_float4(-inf, -inf, inf, inf);
    t.q2 = make_float4(inf, -inf, -inf, -inf);
    t.q3 = make_uint4(0u, 0u, 0u, 0u);
  } else {
    const float4 *pl = reinterpret_cast<const float4 *>(nodes + l);
    const float4 *pr = reinterpret_cast<const float4 *>(nodes + r);
    const float4 la = __ldg(pl), lb = __ldg(pl + 1), lc = __ldg(pl + 2);
    const float4 ra = __ldg(pr), rb = __ldg(pr + 1), rc = __ldg(pr + 2);
    const bool lleaf = (__float_as_uint(lc.y) & 0xFFFFu) != 0, rleaf = (__float_as_uint(rc.y) & 0xFFFFu) != 0;
    t.q0 = la;
    t.q1 = make_float4(lb.x, lb.y, ra.x, ra.y);
    t.q2 = make_float4(ra.z, ra.w, rb.x, rb.y);
    t.q3 = make_uint4(lleaf ? __float_as_uint(lb.w) : l, rleaf ? __float_as_uint(rb.w) : r,
                      lleaf ? __float_as_uint(lc.x) : 0u, rleaf ? __float_as_uint(rc.x) : 0u);
  }
  out[x] = t;
}

// Closest hit through the traversal records (same hits as traverse(): the boxes and triangle tests
// are the same and the closest-hit rule does not depend on the order of the tests). A leaf child
// is tested as soon as its box is hit, so the stack holds inner nodes only. Returns the number of
// inner nodes visited.
__device__ __forceinline__ uint32_t traverse_records(const RayPre &r, const bvhgb_node *__restrict__ nodes,
                                                     const TravNode *__restrict__ trav, uint32_t numNodes,
                                                     uint32_t root, const float *__restrict__ vert,
                                                     const uint32_t *__restrict__ faces, float tmin, float tmax,
                                                     bool cull, Hit &h, uint32_t *err) {
  uint2 stack[kStack];
  int sp = 0;
  uint32_t visits = 0;
  h.prim = kNone;
  h.t = tmax;
  float4 a, b, c;
  load_node(nodes, root, a, b, c);
  float tn;
  if (!box_hit(r, a, b, tmin, tmax, tn)) return 0;
  if (__float_as_uint(c.y) & 0xFFFFu) {
    test_leaf(r, vert, faces, __float_as_uint(b.w), __float_as_uint(c.x), tmin, tmax, cull, h);
    return 0;
  }
  uint32_t cur = root;
  float lim = tmax;
  for (;;) {
    if (++visits > numNodes) {  // a tree visits each node at most once: a cyclic (corrupted) input
      atomicOr(err, kErrBadIndex);
      break;
    }
    const float4 *q = reinterpret_cast<const float4 *>(trav + cur);
    const float4 q0 = __ldg(q), q1 = __ldg(q + 1), q2 = __ldg(q + 2);
    const uint4 q3 = __ldg(reinterpret_cast<const uint4 *>(q + 3));
    float tl, tr;
    bool hl = box_hit(r, q0, make_float4(q1.x, q1.y, 0.0f, 0.0f), tmin, lim, tl);
    bool hr = box_hit(r, make_float4(q1.z, q1.w, q2.x, q2.y), make_float4(q2.z, q2.w, 0.0f, 0.0f), tmin, lim, tr);
    // Leaf children: the lanes of a warp test their next one together, whichever side it is on.
    bool ll = hl && q3.z != 0u, rl = hr && q3.w != 0u;
    hl = hl && !ll;
    hr = hr && !rl;
    if (ll || rl) {
      do {
        test_leaf(r, vert, faces, ll ? q3.x : q3.y, ll ? q3.z : q3.w, tmin, tmax, cull, h);
        rl = rl && ll;
        ll = false;
      } while (rl);
      if (h.prim != kNone) lim = fmul(h.t, kBestSlack);
      hl = hl && tl <= lim;
      hr = hr && tr <= lim;
    }
    const bool lfirst = hl && (!hr || tl <= tr);
    if (hl && hr) {
      if (sp < kStack) stack[sp++] = make_uint2(lfirst ? q3.y : q3.x, __float_as_uint(lfirst ? tr : tl));
      else atomicOr(err, kErrStackOverflow);
    }
    bool go = hl || hr;
    cur = lfirst ? q3.x : q3.y;
    // Pop the next subtree whose entry distance can still beat the best hit.
    while (!go && sp > 0) {
      const uint2 e = stack[--sp];
      go = __uint_as_float(e.y) <= lim;
      cur = e.x;
    }
    if (!go) break;
  }
  return visits;
}

// ---- four-wide records ---------------------------------------------------------------------------
// Record of an inner node for rays whose visits are not counted (bounce, given and random rays): the
// boxes of its up to four grandchildren (a leaf child stands for itself), quantised to 8 bits per
// plane on a power-of-two grid of the record's own, in one 64-byte line. A ray reads one such line
// where it reads three of the binary records (192 bytes), and its chain of dependent loads halves.
// Every plane is rounded outwards, so a box only grows and the closest hit, which does not depend
// on which further boxes are opened, stays the same (the smallest t, then the smallest primitive). Wide trees
// with quantised boxes are the compressed wide BVHs of Ylitie, Karras and Laine (HPG 2017).
struct __align__(64) WideNode {
  float o[3];       // the grid's origin
  uint32_t meta;    // byte k < 3: the exponent of axis k's grid step (biased); bits 24-27: slots with an
                    // inner node, bits 28-31: slots with a leaf
  uint32_t lo[3];   // byte j: slot j's lower plane on the axis
  uint32_t hi[3];
  uint32_t ref[4];  // an inner slot: the node; a leaf: its only face, or the leaf node | kLeafNode
  uint32_t pad[2];
};
static_assert(sizeof(WideNode) == 64, "one line");
constexpr uint32_t kLeafNode = 0x80000000u;
// Stack of the wide traversal: at most three entries are pushed per two levels, so this holds every
// tree that kStack holds for the binary one.
constexpr int kWideSteps = 8;       // records per lane between two rounds of leaf tests
constexpr int kWideStack = kStack * 3 / 2 + 3 * kWideSteps;

// A tree's size is the largest coordinate of its root's box. No grid step is finer than kWideFinest of it, and
// boxes that reach twice as far are on no grid (nested boxes don't): that bounds every plane distance of a ray,
// and what a slab test may say about a ray that is all but parallel to the slab (limit_reciprocals).
constexpr float kWideFinest = 9.0949470e-13f;  // 2^-40
__device__ __forceinline__ float wide_extent(float4 a, float4 b) {
  return fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))), fmaxf(fabsf(b.x), fabsf(b.y)));
}
struct WideSize {
  float size;
  bool finite;  // false: the root's box is not, 'size' is any
  __device__ __forceinline__ WideSize(float4 a, float4 b) {
    const float m = wide_extent(a, b);
    finite = m < 1e37f;  // a NaN component drops out
    size = finite ? fmaxf(m, 2.7755576e-17f) : 1.1529215e18f;  // 2^-55, 2^60
  }
};
__device__ __forceinline__ WideSize wide_size(const bvhgb_node *__restrict__ nodes, uint32_t root) {
  const float4 *p = reinterpret_cast<const float4 *>(nodes + root);
  return WideSize(__ldg(p), __ldg(p + 1));
}

// Node x's wide record (none for a leaf). False: a link leads out of the tree, or to an inner node that has no
// record (nodes [0, records) have one); no slot of the record is ever opened then.
__device__ __forceinline__ bool build_wide(const bvhgb_node *__restrict__ nodes, uint32_t numNodes, uint32_t records,
                                           uint32_t x, const WideSize &tree, WideNode *__restrict__ out) {
  const float4 *p = reinterpret_cast<const float4 *>(nodes + x);
  const float4 xb = __ldg(p + 1), xc = __ldg(p + 2);
  if (__float_as_uint(xc.y) & 0xFFFFu) return true;
  const uint32_t child[2] = {__float_as_uint(xb.w), __float_as_uint(xc.x)};
  float mn[4][3], mx[4][3];
  uint32_t ref[4] = {0u, 0u, 0u, 0u}, kinds = 0;
  bool ok = child[0] < numNodes && child[1] < numNodes;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (!ok) break;
    const float4 *q = reinterpret_cast<const float4 *>(nodes + child[c]);
    const float4 a = __ldg(q), b = __ldg(q + 1), d = __ldg(q + 2);
    const uint32_t l = __float_as_uint(b.w), r = __float_as_uint(d.x);
    if (__float_as_uint(d.y) & 0xFFFFu) {
      mn[2 * c][0] = a.x; mn[2 * c][1] = a.y; mn[2 * c][2] = a.z;
      mx[2 * c][0] = a.w; mx[2 * c][1] = b.x; mx[2 * c][2] = b.y;
      if (r != 0u) {
        kinds |= 16u << (2 * c);
        ref[2 * c] = r == 1u && l < kLeafNode ? l : child[c] | kLeafNode;
      }
      continue;
    }
    const uint32_t g[2] = {l, r};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (g[k] >= numNodes) {
        ok = false;
        break;
      }
      const float4 *w = reinterpret_cast<const float4 *>(nodes + g[k]);
      const float4 e = __ldg(w), f = __ldg(w + 1), h = __ldg(w + 2);
      const int s = 2 * c + k;
      mn[s][0] = e.x; mn[s][1] = e.y; mn[s][2] = e.z;
      mx[s][0] = e.w; mx[s][1] = f.x; mx[s][2] = f.y;
      const uint32_t count = __float_as_uint(h.x);
      if (!(__float_as_uint(h.y) & 0xFFFFu)) {
        kinds |= 1u << s;
        ref[s] = g[k];
        ok = ok && g[k] < records;
      } else if (count != 0u) {
        kinds |= 16u << s;
        ref[s] = count == 1u && __float_as_uint(f.w) < kLeafNode ? __float_as_uint(f.w) : g[k] | kLeafNode;
      }
    }
  }
  if (!ok) kinds = 0;
  WideNode n;
  n.meta = kinds << 24;
  n.pad[0] = n.pad[1] = 0u;
#pragma unroll
  for (int s = 0; s < 4; ++s) n.ref[s] = ref[s];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float lo = __int_as_float(0x7f800000), hi = -lo;
    bool finite = true;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      if (!(kinds & (17u << s))) continue;
      lo = fminf(lo, mn[s][k]);
      hi = fmaxf(hi, mx[s][k]);
      finite = finite && isfinite(mn[s][k]) && isfinite(mx[s][k]);
    }
    // The step: 240 of them span the boxes, and none is finer than two units in the last place of
    // the largest coordinate, so that the differences below are exact to a fraction of a step.
    const float far = fmaxf(fabsf(lo), fabsf(hi));
    const float need = fmaxf(fmaxf((hi - lo) * (1.0f / 240.0f), far * 4.76837158e-7f), tree.finite ? tree.size * kWideFinest : 0.0f);
    uint32_t e = (__float_as_uint(need) >> 23) + 1u;  // the next power of two above
    n.lo[k] = n.hi[k] = 0u;
    if (!finite || !(far <= 2.0f * tree.size) || kinds == 0u) {
      // Not on any grid: a step of infinity makes every plane distance NaN, which drops out of the
      // slab test, so the slots pass on this axis.
      n.o[k] = 0.0f;
      n.meta |= 255u << (8 * k);
      continue;
    }
    e = e < 32u ? 32u : e;
    const float step = __uint_as_float(e << 23), inv = __uint_as_float((254u - e) << 23);
    n.o[k] = lo - 4.0f * step;
    n.meta |= e << (8 * k);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      if (!(kinds & (17u << s))) continue;
      // an eighth of a step beyond the plane: more than every rounding on the way back
      const int ql = (int)floorf((mn[s][k] - n.o[k]) * inv - 0.125f), qh = (int)ceilf((mx[s][k] - n.o[k]) * inv + 0.125f);
      n.lo[k] |= (uint32_t)min(max(ql, 0), 255) << (8 * s);
      n.hi[k] |= (uint32_t)min(max(qh, 0), 255) << (8 * s);
    }
  }
  const uint4 *src = reinterpret_cast<const uint4 *>(&n);
  uint4 *dst = reinterpret_cast<uint4 *>(out + x);
#pragma unroll
  for (int w = 0; w < 4; ++w) dst[w] = src[w];
  return ok;
}

// A plane's byte in the middle of the mantissa of 1.0: 1 + q 2^-15, exactly, in one byte permute.
__device__ __forceinline__ float wide_plane(uint32_t packed, int slot) {
  return __uint_as_float(__byte_perm(packed, 0x3F800000u, 0x7604u | ((uint32_t)slot << 4)));
}

// A warp traces a run of rays through the wide records and keeps its lanes busy. Rays differ in
// length by more than the mean (33.5M-triangle scene: 34 records on average, 152 for the longest of
// a warp), so a lane that is done takes the next ray of the run at once; and since a ray tests two
// triangles per 30 records, one lane's test would stop the others each time: leaves wait in a queue
// of the lane's own, and the lanes test theirs together every few records. Rays are made (or read)
// and set up 32 at a time by the whole warp and wait in shared memory until lanes take them. Neither
// changes a hit: the closest one does not depend on when a triangle is tested, only on which
// records are skipped, and those lie behind a hit already found.
//
// Bound: the latency of the record loads (long scoreboard 5.4 of 10.3 cycles per instruction; L1 hits
// 58%, shared with the stacks). 4.19M rays in 33.5M triangles / the 1080p bounce in 4.19M, in ms:
// one thread per ray on binary records 8.6 / 4.2; four-wide records alone 8.4 / 4.3; with refill and
// queued leaves 4.9 / 2.7 (128 rays per run; 64: 5.4 / 2.9, 256: 5.2 / 2.9; 4 or 12 records between
// leaf tests: 5.0 / 2.9, 4.9 / 2.7); with stolen runs 5.0 / 2.5; with 24 warps per SM and 12 stack
// entries in shared memory instead of 32 warps and a local stack 4.4 / 2.5 (the stacks' sectors had
// pushed the records out of L1; 16 and 28 warps: 4.4 / 2.7, 4.7 / 2.5).
constexpr uint32_t kWideWarps = 24; // warps per SM
constexpr int kWideRays = 32;       // rays set up at a time
constexpr uint32_t kWideRun = 128;  // most rays of a block's run
constexpr int kWideQueue = 6;       // leaves a lane can hold; it pauses when four more would not fit
constexpr int kWideTop = 12;        // stack entries per lane in shared memory, the deeper ones are in local memory
constexpr uint32_t kWideRefill = 8; // idle lanes that make a refill worth its instructions

// Work stealing: a block is one warp with one run of rays, and a warp whose run is used up takes the
// run of a block that has not been launched yet (clusterlaunchcontrol) instead of ending, so its
// lanes drain once per launch, not once per run. The request for the next run travels while the
// warp works on this one. A request that finds no block left is the last one made.
struct __align__(16) StolenRun {
  unsigned long long reply[2];
  unsigned long long bar;
};
__device__ __forceinline__ uint32_t shared_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void steal_request(StolenRun &st) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the last reply was read
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], 16;" ::"r"(shared_addr(&st.bar)) : "memory");
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                   shared_addr(st.reply)),
               "r"(shared_addr(&st.bar))
               : "memory");
}

// Waits (bounded) for the reply of phase 'parity': true and the block's index, or false. One lane
// waits and reads the reply, so that its own fence orders the read before the next request.
__device__ __forceinline__ bool steal_wait(StolenRun &st, uint32_t parity, uint32_t &block, uint32_t *err) {
  uint32_t taken = 0, x = 0;
  if ((threadIdx.x & 31u) == 0u) {
    uint32_t ok = 0;
    for (uint32_t i = 0; i < (1u << 18) && !ok; ++i) {
      asm volatile(
          "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
          : "=r"(ok)
          : "r"(shared_addr(&st.bar)), "r"(parity)
          : "memory");
    }
    if (ok) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile(
          "{\n .reg .pred p;\n .reg .b128 h;\n .reg .b64 a, b;\n ld.shared.v2.b64 {a, b}, [%2];\n mov.b128 h, {a, b};\n"
          " clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n selp.u32 %0, 1, 0, p;\n mov.u32 %1, 0;\n"
          " @p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n}\n"
          : "=r"(taken), "=r"(x)
          : "r"(shared_addr(st.reply))
          : "memory");
    } else {
      atomicOr(err, kErrTimeout);
    }
  }
  block = __shfl_sync(0xFFFFFFFFu, x, 0);
  return __shfl_sync(0xFFFFFFFFu, taken, 0) != 0u;
}

struct WideShared {
  StolenRun steal;
  float org[3][kWideRays], inv[3][kWideRays], shear[3][kWideRays];
  uint32_t axes[kWideRays];  // kx | ky << 2 | kz << 4
  uint32_t index[kWideRays];
  uint32_t leaf[kWideQueue][32];
  uint2 stack[kWideTop][32];  // the lanes' first stack entries (node, entry distance)
};

__device__ __forceinline__ WideShared &wide_shared() {
  __shared__ WideShared sm;
  return sm;
}

// What the rays are traced against, one tree for all of them.
struct WideScene {
  static constexpr bool kMany = false;  // several trees: a lane keeps the pointers of its ray's own
  const bvhgb_node *nodesOf;
  const WideNode *wideOf;
  const uint32_t *facesOf;
  const float *vert;
  uint32_t nodeCount, rootNode;
  float tmin, tmax;
  bool cull;
  __device__ __forceinline__ const bvhgb_node *nodes(uint32_t) const { return nodesOf; }
  __device__ __forceinline__ const WideNode *wide(uint32_t) const { return wideOf; }
  __device__ __forceinline__ const uint32_t *faces(uint32_t) const { return facesOf; }
  __device__ __forceinline__ uint32_t numNodes() const { return nodeCount; }
  __device__ __forceinline__ uint32_t root() const { return rootNode; }
};

// Reciprocals of direction components beyond 2^116 over the tree's size (and a thousandth of the ray's reach), which a
// ray all but parallel to an axis has, are not used as they are: products with the largest grid step or the origin's
// distance could overflow, and a distance that is infinite on one side only would drop a box.
//   - An infinite one makes the distances NaN, and every box passes on that axis: true, but nothing is culled.
//   - To keep the ray out of the slabs beside it, 2^80 over the largest component serves (or that limit). A ray
//     inside a slab is an eighth of a step or more from its planes, which then are as far away as 2^77 steps along
//     the ray; and the component moves the ray by a thirty-second of a step at most on its first 2^75 steps. A
//     step is kWideFinest of the size or more, so this holds while the origin is within 2^35 sizes (2^-45 of
//     the reciprocal times the largest component).
// Other rays pass one test (a: the root's box with b.x, b.y): a set-up is as long as its instructions are cold.
__device__ __forceinline__ void limit_reciprocals(RayPre &r, float4 a, float4 b) {
  const float origin = fmaxf(fmaxf(fabsf(r.o[0]), fabsf(r.o[1])), fabsf(r.o[2]));
  const float most = fmaxf(fmaxf(fabsf(r.inv[0]), fabsf(r.inv[1])), fabsf(r.inv[2]));
  if (__builtin_expect(most * fmaxf(origin, wide_extent(a, b)) <= 1.1258999e15f, 1)) return;  // 2^50
  if (pick(r.d, r.kz) == 0.0f) {
    // No direction at all: the triangle test's shears are NaN and nothing is hit, so every box lies behind the ray.
    r.o[0] = 3e38f;
    r.inv[0] = r.inv[1] = r.inv[2] = 1.0f;
    return;
  }
  const WideSize tree(a, b);
  const float reach = origin + tree.size;
  const float limit = __fdividef(8.3076750e34f, fmaf(reach, 0.0009765625f, tree.size));
  const float stand = fminf(1.2089258e24f * fabsf(r.sz), limit);
  const bool near = tree.finite && reach <= tree.size * (stand * fabsf(pick(r.d, r.kz)) * 2.8421709e-14f);  // 2^-45
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (fabsf(r.inv[k]) > limit) r.inv[k] = copysignf(near ? stand : __int_as_float(0x7f800000), r.d[k]);
}

// Block b's run is rays [b * run, ...) of 'total' (< 2^31). gen(i, valid, r), which
// the whole warp calls for 32 rays in a row from a multiple of 32, sets r.o and r.d of a valid ray and
// returns whether there is one to trace; emit(i, hit) takes every ray's result (no hit for those gen
// refused). A block is one warp; every lane calls it.
template <typename Scene, typename Gen, typename Emit>
__device__ __forceinline__ void trace_wide(const Scene &sc, uint32_t total, uint32_t run, const Gen &gen, const Emit &emit,
                                           uint32_t *err) {
  const uint32_t lane = threadIdx.x & 31u, ltMask = (1u << lane) - 1u;
  const WideNode *laneWide = nullptr;
  const uint32_t *laneFaces = nullptr;
  WideShared &sm = wide_shared();
  const bool anyT = sc.tmin < 0.0f;  // negative distances: entries are not pruned by their distance
  uint2 deep[kWideStack - kWideTop];
  int sp = 0;
  uint32_t cur = kNone, ray = kNone, steps = 0, pend = 0;
  RayPre r = {};
  Hit h = {kNone, 0.0f};
  float lim = 0.0f;
  // warp-uniform: the rays waiting, the run's position and end, the steal's state
  uint32_t head = 0, count = 0, next = blockIdx.x * run, end = min(total, next + run), parity = 0;
  bool more = true;  // a request is on its way
  if (lane == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_addr(&sm.steal.bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    steal_request(sm.steal);
  }
  __syncwarp();
  for (;;) {
    const uint32_t idle = __ballot_sync(0xFFFFFFFFu, ray == kNone);
    if (__popc(idle) >= (int)kWideRefill) {
      if (head == count && next >= end && more) {
        uint32_t block;
        more = steal_wait(sm.steal, parity, block, err);
        parity ^= 1u;
        if (more) {
          next = block * run;
          end = min(total, next + run);
          if (lane == 0) steal_request(sm.steal);
        }
        __syncwarp();
      }
      if (head == count && next < end) {
        const uint32_t i = next + lane;
        RayPre g = {};
        bool live = gen(i, i < end, g);
        if (live) {
          setup_ray(g);
          float4 a, b, c;
          load_node(sc.nodes(i), sc.root(), a, b, c);
          float tn;
          live = box_hit(g, a, b, sc.tmin, sc.tmax, tn);
          if (live && (__float_as_uint(c.y) & 0xFFFFu)) {  // the tree is one leaf
            Hit o = {kNone, sc.tmax};
            test_leaf(g, sc.vert, sc.faces(i), __float_as_uint(b.w), __float_as_uint(c.x), sc.tmin, sc.tmax, sc.cull, o);
            emit(i, o);
            live = false;
          } else if (!live) {
            emit(i, Hit{kNone, sc.tmax});
          }
          limit_reciprocals(g, a, b);
        } else if (i < end) {
          emit(i, Hit{kNone, sc.tmax});
        }
        const uint32_t have = __ballot_sync(0xFFFFFFFFu, live);
        __syncwarp();
        if (live) {
          const uint32_t s = __popc(have & ltMask);
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            sm.org[k][s] = g.o[k];
            sm.inv[k][s] = g.inv[k];
          }
          sm.shear[0][s] = g.sx;
          sm.shear[1][s] = g.sy;
          sm.shear[2][s] = g.sz;
          sm.axes[s] = (uint32_t)g.kx | ((uint32_t)g.ky << 2) | ((uint32_t)g.kz << 4);
          sm.index[s] = i;
        }
        head = 0;
        count = __popc(have);
        next = end - next > (uint32_t)kWideRays ? next + kWideRays : end;
        __syncwarp();
      }
      if (head == count && next >= end && !more && idle == 0xFFFFFFFFu) break;
      const uint32_t s = head + __popc(idle & ltMask);
      if (ray == kNone && s < count) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          r.o[k] = sm.org[k][s];
          r.inv[k] = sm.inv[k][s];
        }
        r.sx = sm.shear[0][s];
        r.sy = sm.shear[1][s];
        r.sz = sm.shear[2][s];
        const uint32_t ax = sm.axes[s];
        r.kx = (int)(ax & 3u);
        r.ky = (int)((ax >> 2) & 3u);
        r.kz = (int)(ax >> 4);
        ray = sm.index[s];
        if (Scene::kMany) {
          laneWide = sc.wide(ray);
          laneFaces = sc.faces(ray);
        }
        cur = sc.root();
        sp = 0;
        steps = 0;
        pend = 0;
        h.prim = kNone;
        h.t = lim = sc.tmax;
      }
      head = min(count, head + (uint32_t)__popc(idle));
      __syncwarp();  // the next 32 rays may overwrite these
    }
    if (sp > kWideStack - 3 * kWideSteps || steps > sc.numNodes()) {
      // A deeper stack than any the binary traversal can hold, or a cyclic (corrupted) tree: a tree
      // visits each node at most once.
      if (ray != kNone) atomicOr(err, steps > sc.numNodes() ? kErrBadIndex : kErrStackOverflow);
      cur = kNone;
      sp = 0;
      steps = 0;
    }
#pragma unroll 1
    for (int step = 0; step < kWideSteps; ++step) {
      // the next subtree, if its entry distance can still beat the best hit
      if (cur == kNone && sp > 0) {
        --sp;
        uint2 e;
        if (sp < kWideTop) e = sm.stack[sp][lane];
        else e = deep[sp - kWideTop];
        if (__uint_as_float(e.y) <= lim || anyT) cur = e.x;
      }
      if (cur == kNone || pend > (uint32_t)kWideQueue - 4u) continue;
      ++steps;
      const uint4 *q = reinterpret_cast<const uint4 *>((Scene::kMany ? laneWide : sc.wide(0)) + cur);
      const uint4 w0 = __ldg(q), w1 = __ldg(q + 1), w2 = __ldg(q + 2);
      const uint2 w3 = __ldg(reinterpret_cast<const uint2 *>(q + 3));
      const uint32_t ref[4] = {w2.z, w2.w, w3.x, w3.y};
      const float o[3] = {__uint_as_float(w0.x), __uint_as_float(w0.y), __uint_as_float(w0.z)};
      const uint32_t lo[3] = {w1.x, w1.y, w1.z}, hi[3] = {w1.w, w2.x, w2.y};
      float scale[3], base[3];
      uint32_t pn[3], pf[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float gridStep = __uint_as_float(((w0.w >> (8 * k)) & 0xFFu) << 23);
        scale[k] = (gridStep * 32768.0f) * r.inv[k];
        base[k] = (o[k] - r.o[k]) * r.inv[k] - scale[k];
        const bool neg = __float_as_int(r.inv[k]) < 0;
        pn[k] = neg ? hi[k] : lo[k];
        pf[k] = neg ? lo[k] : hi[k];
      }
      // A slot's near and far plane distances are one packed operation per axis. What follows is
      // predicated, not branched (a slot's outcome differs per lane), but for the leaves: two in
      // thirty records.
      uint32_t key[4], leaves = 0;
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        float2 t[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
          t[k] = fma2(make_float2(wide_plane(pn[k], s), wide_plane(pf[k], s)), make_float2(scale[k], scale[k]),
                      make_float2(base[k], base[k]));
        const float t0 = fmaxf(fmaxf(fmaxf(t[0].x, t[1].x), t[2].x), sc.tmin);
        const float tf = fminf(fminf(t[0].y, t[1].y), t[2].y);
        const bool hit = t0 <= fminf(fmaf(fabsf(tf), 9.5367432e-7f, tf), lim);
        // ordered by entry distance (a negative one is 0), the slot in the low bits
        const uint32_t k = (__float_as_uint(fmaxf(t0, 0.0f)) & ~3u) | (uint32_t)s;
        key[s] = hit && (w0.w & (1u << (24 + s))) ? k : 0xFFFFFFFFu;
        leaves |= hit ? w0.w & (1u << (28 + s)) : 0u;
      }
      while (leaves) {
        const int s = __ffs(leaves) - 29;
        leaves &= leaves - 1u;
        sm.leaf[pend][lane] = s == 0 ? ref[0] : s == 1 ? ref[1] : s == 2 ? ref[2] : ref[3];
        ++pend;
      }
#define BVHGB_ORDER(a, b)                                                             \
  {                                                                                   \
    const uint32_t x_ = min(key[a], key[b]), y_ = max(key[a], key[b]);                \
    key[a] = x_;                                                                      \
    key[b] = y_;                                                                      \
  }
      BVHGB_ORDER(0, 1) BVHGB_ORDER(2, 3) BVHGB_ORDER(0, 2) BVHGB_ORDER(1, 3) BVHGB_ORDER(1, 2)
#undef BVHGB_ORDER
      // The nearest is next, the others go onto the stack, farthest first.
#pragma unroll
      for (int j = 3; j >= 0; --j) {
        const bool live = key[j] != 0xFFFFFFFFu;
        const uint32_t ra = key[j] & 1u ? ref[1] : ref[0], rb = key[j] & 1u ? ref[3] : ref[2];
        const uint32_t rf = key[j] & 2u ? rb : ra;
        if (j == 0) {
          cur = live ? rf : kNone;
        } else {
          const uint2 e = make_uint2(rf, key[j] & ~3u);
          if (live && sp < kWideTop) sm.stack[sp][lane] = e;
          if (live && sp >= kWideTop) deep[sp - kWideTop] = e;
          sp += live ? 1 : 0;
        }
      }
    }
    // The leaves found meanwhile, one per lane at a time.
    while (__any_sync(0xFFFFFFFFu, pend != 0u)) {
      if (pend == 0u) continue;
      const uint32_t e = sm.leaf[--pend][lane];
      uint32_t first = e, faceCount = 1u;
      if (e & kLeafNode) {
        const float4 *p = reinterpret_cast<const float4 *>(sc.nodes(ray) + (e & ~kLeafNode));
        first = __float_as_uint(__ldg(p + 1).w);
        faceCount = __float_as_uint(__ldg(p + 2).x);
      }
      test_leaf(r, sc.vert, Scene::kMany ? laneFaces : sc.faces(0), first, faceCount, sc.tmin, sc.tmax, sc.cull, h);
      if (h.prim != kNone) lim = fmul(h.t, kBestSlack);
    }
    if (ray != kNone && cur == kNone && sp == 0) {
      emit(ray, h);
      ray = kNone;
    }
  }
}

// Rays of a block's run: kWideRun, or fewer (a multiple of the 32 that are set up at a time) where
// that would leave warps of the chip without a run.
inline uint32_t wide_run(uint64_t rays) {
  const uint64_t warps = (uint64_t)sm_count() * kWideWarps, per = rays / warps / kWideRays * kWideRays;
  return (uint32_t)(per < (uint64_t)kWideRays ? (uint64_t)kWideRays : per < kWideRun ? per : kWideRun);
}

// ---- ray bundles ---------------------------------------------------------------------------------
// kTraceRayBundle (CUDAKernels.cu:240-383) traverses the tree once for a block of 64 rays: a node
// is visited when any ray of the block hits it, the nearer child first by a vote of the rays. Here
// the bundle is a warp (32 neighbouring primary rays): each lane tests its own ray against both
// children of the warp's node (the node record is one broadcast load), __any_sync decides whether
// the warp goes down a side, a majority ballot picks the near side, and the stack is warp-uniform
// (each lane keeps its own entry distance of a pushed node, +inf where its ray missed it, so a pop
// is skipped when no lane can still improve). A lane tests a leaf's triangles only where its own
// ray hits the leaf's box. Every lane thus tests a superset of what its own traversal would test,
// and the closest-hit rule (smallest t, then smallest primitive) picks the same hit; the visit
// count (intCount) is the warp's. All lanes of the warp must call it; inactive lanes pass active =
// false and get no hit. REC: traversal records (true) or the node array (false).
template <bool REC>
__device__ __forceinline__ uint32_t traverse_bundle(const RayPre &r, bool active, const bvhgb_node *__restrict__ nodes,
                                                    const TravNode *__restrict__ trav, uint32_t numNodes,
                                                    uint32_t root, const float *__restrict__ vert,
                                                    const uint32_t *__restrict__ faces, float tmin, float tmax,
                                                    bool cull, Hit &h, uint32_t *err) {
  const float kInf = __int_as_float(0x7f800000);
  uint32_t stN[kStack];
  float stT[kStack];
  int sp = 0;
  uint32_t visits = 0;
  h.prim = kNone;
  h.t = tmax;
  float4 a, b, c;
  load_node(nodes, root, a, b, c);
  float tn;
  const bool hitRoot = active && box_hit(r, a, b, tmin, tmax, tn);
  if (!__any_sync(0xFFFFFFFFu, hitRoot)) return 0;
  if (__float_as_uint(c.y) & 0xFFFFu) {
    if (hitRoot) test_leaf(r, vert, faces, __float_as_uint(b.w), __float_as_uint(c.x), tmin, tmax, cull, h);
    return 0;
  }
  uint32_t cur = root;
  for (uint32_t it = 0;; ++it) {
    if (it > numNodes) {  // each node is visited at most once per warp: a cyclic (corrupted) input
      if (active) atomicOr(err, kErrBadIndex);
      break;
    }
    ++visits;
    float4 l0, l1, r0, r1;
    uint32_t lref, rref, lcnt, rcnt;
    bool ok = true;
    if (REC) {
      const float4 *q = reinterpret_cast<const float4 *>(trav + cur);
      const float4 q0 = __ldg(q), q1 = __ldg(q + 1), q2 = __ldg(q + 2);
      const uint4 q3 = __ldg(reinterpret_cast<const uint4 *>(q + 3));
      l0 = q0;
      l1 = make_float4(q1.x, q1.y, 0.0f, 0.0f);
      r0 = make_float4(q1.z, q1.w, q2.x, q2.y);
      r1 = make_float4(q2.z, q2.w, 0.0f, 0.0f);
      lref = q3.x;
      rref = q3.y;
      lcnt = q3.z;
      rcnt = q3.w;
    } else {
      float4 ca, cb, cc;
      load_node(nodes, cur, ca, cb, cc);
      const uint32_t li = __float_as_uint(cb.w), ri = __float_as_uint(cc.x);
      ok = li < numNodes && ri < numNodes;
      float4 lc, rc;
      if (ok) {
        load_node(nodes, li, l0, l1, lc);
        load_node(nodes, ri, r0, r1, rc);
        const bool ll = (__float_as_uint(lc.y) & 0xFFFFu) != 0, rl = (__float_as_uint(rc.y) & 0xFFFFu) != 0;
        lref = ll ? __float_as_uint(l1.w) : li;
        rref = rl ? __float_as_uint(r1.w) : ri;
        lcnt = ll ? __float_as_uint(lc.x) : 0u;
        rcnt = rl ? __float_as_uint(rc.x) : 0u;
      }
    }
    if (!ok) {
      if (active) atomicOr(err, kErrBadIndex);
    } else {
      float lim = h.prim == kNone ? tmax : fmul(h.t, kBestSlack);
      float tl = kInf, tr = kInf;
      bool hl = active && box_hit(r, l0, l1, tmin, lim, tl);
      bool hr = active && box_hit(r, r0, r1, tmin, lim, tr);
      if (hl && lcnt) {
        test_leaf(r, vert, faces, lref, lcnt, tmin, tmax, cull, h);
        hl = false;
      }
      if (hr && rcnt) {
        test_leaf(r, vert, faces, rref, rcnt, tmin, tmax, cull, h);
        hr = false;
      }
      lim = h.prim == kNone ? tmax : fmul(h.t, kBestSlack);
      hl = hl && tl <= lim;
      hr = hr && tr <= lim;
      const bool anyL = __any_sync(0xFFFFFFFFu, hl), anyR = __any_sync(0xFFFFFFFFu, hr);
      if (anyL && anyR) {
        const int wantL = __popc(__ballot_sync(0xFFFFFFFFu, hl && (!hr || tl <= tr)));
        const int wantR = __popc(__ballot_sync(0xFFFFFFFFu, hr && (!hl || tr < tl)));
        const bool lfirst = wantL >= wantR;
        if (sp < kStack) {
          stN[sp] = lfirst ? rref : lref;
          stT[sp] = lfirst ? (hr ? tr : kInf) : (hl ? tl : kInf);
          ++sp;
        } else if (active) {
          atomicOr(err, kErrStackOverflow);
        }
        cur = lfirst ? lref : rref;
        continue;
      }
      if (anyL || anyR) {
        cur = anyL ? lref : rref;
        continue;
      }
    }
    // Pop the next subtree that some lane can still improve on.
    bool found = false;
    while (sp > 0) {
      --sp;
      const float lim = h.prim == kNone ? tmax : fmul(h.t, kBestSlack);
      if (__any_sync(0xFFFFFFFFu, active && stT[sp] <= lim)) {
        cur = stN[sp];
        found = true;
        break;
      }
    }
    if (!found) break;
  }
  return active ? visits : 0u;
}

}  // namespace
}  // namespace bvhgb
