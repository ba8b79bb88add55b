// Closest points on sm_100a, bit-identical to the reference's CPU query
// (src/capi.mojo:522-586: an ordered depth-first walk of the median-split hierarchy
// with strict and non-strict tests in given places), ties included. One thread per
// point; above kAabbSortMin points the threads take them in Morton order (perm).
//
// The reference's walk is a chain in a fixed order, and its order is a poor one: the
// best distance comes down slowly, and FP64 boxes are read at every step. So the
// minimum is found first, in an order and with bounds of its own, and then the face
// that the reference's order would have kept:
//
// 1. aabb_any_order_kernel walks the tree nearer disc centre first, skipping children
//    by FP32 boxes and discs (wn_aabb.h), faces by discs of their own, and evaluates
//    the others with the reference's FP64 arithmetic (wn_aabb.cuh). What it skips is
//    farther than the best, so afterwards `best` is the smallest squared distance B
//    that any face of the mesh evaluates to, and the faces that evaluate to B exactly
//    have all been seen. Of these the walk keeps the first in the reference's order,
//    which two faces' common ancestor decides: the child with the smaller box distance
//    comes first (the right one when they are equal), within a leaf the order of the
//    records.
// 2. The reference's result is that face if it looks at it: a leaf is looked at when its
//    box distance is <= the best at that time, which before that face is above B. So a
//    leaf whose box distance is <= B is.
// 3. Where rounding puts the leaf's box distance above B, the thread does the reference's
//    own walk.
//
// Trees that the library did not build may have boxes that do not hold their faces,
// and closest points on very thin faces lose their digits: no bound of step 1 holds
// then, and aabb_query_kernel does the reference's walk for every point.
//
// Bound by the walks' divergence and load latency, not by HBM or FP64 throughput (the
// tree sits in L2; ncu, 524,288 points inside and around the 327,680-face sphere: 8.2 of
// 32 lanes active, issue 42 %, FP64 pipe 15 %). Measured against the reference's walk
// with box and slab (a range of n.x) alone: 327,680 faces x 2^20 points 10.1 -> 2.3 ms,
// 243,602 (terrain) x 2^20 1.54 -> 1.34 ms, x 10,000 0.18 -> 0.12 ms. The reference's
// order with the discs: 5.1 ms. Ties kept in a list and compared at the end, from the root
// down: 2.76 -> 2.57 ms for the whole call, and 131,072 of the mesh's own vertices 0.70 ->
// 0.45 (the reference's walk: 0.31). Keeping the warp's lanes in step, leaves held until 1, 4,
// 8 or more lanes have one: slower in either order (3.2 ms at best here).
#include <cuda_runtime.h>

#include "wn_aabb.cuh"
#include "wn_aabb.h"
#include "wn_common.cuh"
#include "wn_internal.h"

namespace wn {
namespace {

constexpr int kAabbThreads = 128;
// Consecutive points of the (Morton) order that share a warp; its other lanes take
// points from elsewhere, so that 32 of the longest walks do not meet in one warp, which
// the rest of the GPU then waits for (327,680 faces x 2^20 points, stack in local memory:
// 32 3.17 ms, 16 2.64, 8 2.87, 4 2.95).
constexpr int kGroup = 16;
// Shared memory that a launch gets without asking for more: 48 levels of the any-order
// walk's stack. The library's own trees have at most 30 (2^31 faces); a caller-made one may
// have 63, and takes the reference's walk, whose stack is in local memory.
constexpr size_t kStackBytes = 48 << 10;
// Fewer faces than this are in the reference's order soon enough (1,000 points and 131,072,
// us, its walk and the any-order one: 12 faces 33 and 36, 141 and 157; 40 around one vertex
// 46 and 64, 159 and 213; 80 faces 77 and 62, 213 and 193).
constexpr int64_t kOrderFaces = 64;
// The reference's walk takes the discs' bounds on meshes of at least kDiscFaces of which one
// in kDiscShare is thin at most, else the slabs alone (131,072 points, ms, slabs and discs:
// one thin face in 327,681 3.7 and 2.4, in 20,481 0.96 and 1.00; a tenth of 327,680 10.0 and
// 11.3, since a disc over a thin face has no radius).
constexpr int64_t kDiscFaces = 65536, kDiscShare = 1024;
// A face is thin below |n|^2 = kThin * (longest side)^4: thinner than about 1 : 1000.
constexpr double kThin = 1e-6;

struct AabbArgs {
  const AabbNodeRec* __restrict__ nodes;
  const AabbWalkRec* __restrict__ walk;
  const AabbSpan* __restrict__ spans;
  const AabbTriRec* __restrict__ tris;
  const AabbDisc* __restrict__ face_discs;
  const double* __restrict__ P;
  const uint32_t* __restrict__ perm;
  double* __restrict__ sqrd;
  int64_t* __restrict__ index;
  double* __restrict__ closest;
  int* err;
  int64_t np, nnodes;
  double root[6];
  double scale;
  AabbFrame frame;
  int levels;  // depth of the tree
};

// A point in the tree's frame, with the margin of its bounds; `ok` where they hold (not
// for huge or non-finite points, nor where the coordinates are so large beside the mesh
// that their own rounding outweighs it).
struct Local {
  float x, y, z, margin;
  bool ok;
};
__device__ __forceinline__ Local local_of(const AabbArgs& a, double px, double py, double pz) {
  const double x = (px - a.frame.c[0]) * a.frame.s, y = (py - a.frame.c[1]) * a.frame.s,
               z = (pz - a.frame.c[2]) * a.frame.s;
  const double size = a.frame.ext + fabs(x) + fabs(y) + fabs(z);
  const double round = kWalkRound * (a.scale + fabs(px) + fabs(py) + fabs(pz)) * a.frame.s;
  return Local{static_cast<float>(x), static_cast<float>(y), static_cast<float>(z),
               kWalkMargin * __double2float_ru(size) + __double2float_ru(round),
               a.walk != nullptr && size < 1e15 && round < 1e-3 * size};
}

struct Best {
  double d2, x, y, z;
  int64_t face;
};

__device__ __forceinline__ double2 ldg2(const double* p) {
  return __ldg(reinterpret_cast<const double2*>(p));
}

__device__ __forceinline__ ClosestHit closest_on_record(const AabbTriRec* tr, double px, double py,
                                                        double pz, int64_t& face) {
  const double2 w0 = ldg2(tr->a), w1 = ldg2(tr->a + 2), w2 = ldg2(tr->b + 1);
  const double2 w3 = ldg2(tr->c), w4 = ldg2(tr->c + 2);
  face = __double_as_longlong(w4.y);
  return closest_on_triangle(px, py, pz, w0.x, w0.y, w1.x, w1.y, w2.x, w2.y, w3.x, w3.y, w4.x);
}

__device__ __forceinline__ double box_of(const double* box, double px, double py, double pz) {
  const double2 b0 = ldg2(box), b1 = ldg2(box + 2), b2 = ldg2(box + 4);
  return box_distance2(px, py, pz, b0.x, b0.y, b1.x, b1.y, b2.x, b2.y);
}

// Squared lower bound on the distance from p to the faces inside a disc, less the
// rounding margin `e`; v2 receives the squared distance from its centre.
__device__ __forceinline__ float disc_bound2(float px, float py, float pz, const float4& nt,
                                             const float4& cr, float e, float& v2) {
  const float x = px - cr.x, y = py - cr.y, z = pz - cr.z;
  const float h = nt.x * x + nt.y * y + nt.z * z;
  v2 = x * x + y * y + z * z;
  const float g = fmaxf(fabsf(h) - nt.w - e, 0.0f);
  const float l = fmaxf(sqrtf(fmaxf(v2 * (1.0f - 2e-6f) - h * h, 0.0f)) - cr.w - e, 0.0f);
  return (g * g + l * l) * (1.0f - kWalkRel);
}
// A point in the tree's frame in FP64, the margin of its slab bounds there, and what brings
// their squares back (kSlabMargin for their own rounding among it).
struct Slabs {
  double x, y, z, margin, back;
};
__device__ __forceinline__ double slab_bound2(const Slabs& p, float nx, float ny, float nz, float lo,
                                              float hi) {
  const double h = fma(static_cast<double>(nz), p.z,
                       fma(static_cast<double>(ny), p.y, static_cast<double>(nx) * p.x));
  const double g = fmax(static_cast<double>(lo) - h, h - static_cast<double>(hi)) - p.margin;
  return g > 0.0 ? g * g * p.back : 0.0;
}

// The reference's walk. Each stack entry keeps the box distance computed when it was
// pushed (the reference recomputes the same double from the same box at the pop), or
// the disc bound where that is larger: such a child holds no face that the reference
// would take. The order is decided by the box distances alone.
template <bool DISCS>
__device__ __forceinline__ Best walk_in_order(const AabbArgs& a, double px, double py, double pz) {
  const Local p = local_of(a, px, py, pz);
  const double unit = p.ok ? 1.0 / a.frame.s : 0.0;
  const Slabs s{(px - a.frame.c[0]) * a.frame.s, (py - a.frame.c[1]) * a.frame.s,
                (pz - a.frame.c[2]) * a.frame.s,
                p.ok ? kSlabMargin * (a.scale + fabs(px) + fabs(py) + fabs(pz)) * a.frame.s : INFINITY,
                unit * unit * (1.0 - kSlabMargin)};
  Best r{1.0e300, 0.0, 0.0, 0.0, -1};
  int stack_node[kAabbStack];
  double stack_d2[kAabbStack];
  int sp = 0;
  if (a.nnodes > 0) {
    stack_node[0] = 0;
    stack_d2[0] = box_distance2(px, py, pz, a.root[0], a.root[1], a.root[2], a.root[3],
                                a.root[4], a.root[5]);
    sp = 1;
  }
  while (sp > 0) {
    --sp;
    if (stack_d2[sp] > r.d2) continue;
    const AabbNodeRec* nd = a.nodes + stack_node[sp];
    const int4 meta = __ldg(reinterpret_cast<const int4*>(nd));
    if (meta.w > 0) {
      const AabbTriRec* tr = a.tris + meta.z;
      for (int k = 0; k < meta.w; ++k, ++tr) {
        int64_t face;
        const ClosestHit h = closest_on_record(tr, px, py, pz, face);
        if (h.d2 < r.d2) {
          r.d2 = h.d2;
          r.face = face;
          r.x = h.x;
          r.y = h.y;
          r.z = h.z;
        }
      }
    } else {
      const double dl = box_of(nd->lbox, px, py, pz), dr = box_of(nd->rbox, px, py, pz);
      double kl = dl, kr = dr;
      if (DISCS && p.ok) {
        const float4* disc = reinterpret_cast<const float4*>(a.walk + (nd - a.nodes)) + 1;
        float v2;
        const float l = disc_bound2(p.x, p.y, p.z, __ldg(disc), __ldg(disc + 1), p.margin, v2);
        const float r = disc_bound2(p.x, p.y, p.z, __ldg(disc + 2), __ldg(disc + 3), p.margin, v2);
        kl = fmax(kl, static_cast<double>(l) * unit * unit);
        kr = fmax(kr, static_cast<double>(r) * unit * unit);
      } else if (!DISCS) {
        const float4* w = reinterpret_cast<const float4*>(&nd->lslab);
        const float4 s0 = __ldg(w), s1 = __ldg(w + 1);
        const float2 s2 = __ldg(reinterpret_cast<const float2*>(w + 2));
        kl = fmax(kl, slab_bound2(s, s0.x, s0.y, s0.z, s0.w, s1.x));
        kr = fmax(kr, slab_bound2(s, s1.y, s1.z, s1.w, s2.x, s2.y));
      }
      // Farther child first, so the nearer one is popped next (capi.mojo:571-586).
      const bool left_near = dl < dr;
      const int first = left_near ? meta.y : meta.x, second = left_near ? meta.x : meta.y;
      const double dfirst = left_near ? kr : kl, dsecond = left_near ? kl : kr;
      if (sp + 2 > kAabbStack) {  // cannot happen for a validated tree
        atomicOr(a.err, kErrBadLaunch);
        r.face = -2;
        break;
      }
      if (dfirst <= r.d2) {
        stack_node[sp] = first;
        stack_d2[sp] = dfirst;
        ++sp;
      }
      if (dsecond <= r.d2) {
        stack_node[sp] = second;
        stack_d2[sp] = dsecond;
        ++sp;
      }
    }
  }
  return r;
}

__device__ __noinline__ Best ordered_walk(const AabbArgs& a, double px, double py, double pz) {
  return walk_in_order<true>(a, px, py, pz);
}

__device__ __forceinline__ void store_result(const AabbArgs& a, int64_t qi, const Best& r) {
  a.sqrd[qi] = r.d2;
  a.index[qi] = r.face;
  a.closest[3 * qi] = r.x;
  a.closest[3 * qi + 1] = r.y;
  a.closest[3 * qi + 2] = r.z;
}

template <bool DISCS>
__global__ void __launch_bounds__(kAabbThreads) aabb_query_kernel(const AabbArgs a) {
  const int64_t t = static_cast<int64_t>(blockIdx.x) * kAabbThreads + threadIdx.x;
  if (t >= a.np) return;
  const int64_t qi = a.perm ? static_cast<int64_t>(a.perm[t]) : t;
  store_result(a, qi, walk_in_order<DISCS>(a, a.P[3 * qi], a.P[3 * qi + 1], a.P[3 * qi + 2]));
}

__device__ __forceinline__ float box_bound2(float px, float py, float pz, float lx, float ly,
                                            float lz, float hx, float hy, float hz, float e) {
  const float x = fmaxf(fmaxf(lx - px, px - hx) - e, 0.0f);
  const float y = fmaxf(fmaxf(ly - py, py - hy) - e, 0.0f);
  const float z = fmaxf(fmaxf(lz - pz, pz - hz) - e, 0.0f);
  return (x * x + y * y + z * z) * (1.0f - kWalkRel);
}

// Whether the reference's walk reaches the leaf at slot `at` before face record j of another
// leaf: up to the node that holds both (a vertex's faces lie in leaves a few levels apart;
// from the root down it took three times the loads).
__device__ __forceinline__ bool comes_first(const AabbArgs& a, int at, int j, double px, double py,
                                            double pz) {
  while (at >= 0) {
    const int node = at >> 1;
    const int4 s = __ldg(reinterpret_cast<const int4*>(a.spans + node));
    if (j >= s.x && j < s.y) {
      const AabbNodeRec* nd = a.nodes + node;
      const bool left_near = box_of(nd->lbox, px, py, pz) < box_of(nd->rbox, px, py, pz);
      return left_near == !(at & 1);
    }
    at = s.z;
  }
  return false;  // not reached: the root holds every record
}

__global__ void __launch_bounds__(kAabbThreads) aabb_any_order_kernel(const AabbArgs a) {
  // (node, bound) per level and thread; in local memory it competed with the tree for L1
  // (2.64 -> 2.44 ms).
  extern __shared__ uint2 s_stack[];
  const int64_t slot = static_cast<int64_t>(blockIdx.x) * kAabbThreads + threadIdx.x;
  const int64_t nwarp = (a.np + 31) / 32, warp = slot / 32, lane = slot % 32;
  if (warp >= nwarp) return;
  const int64_t t = (lane / kGroup) * (nwarp * kGroup) + warp * kGroup + lane % kGroup;
  if (t >= a.np) return;
  const int64_t qi = a.perm ? static_cast<int64_t>(a.perm[t]) : t;
  const double px = a.P[3 * qi], py = a.P[3 * qi + 1], pz = a.P[3 * qi + 2];
  const Local p = local_of(a, px, py, pz);
  const float fx = p.x, fy = p.y, fz = p.z, margin = p.margin;
  Best r{1.0e300, 0.0, 0.0, 0.0, -1};
  float bestf = INFINITY;  // r.d2 in the tree's frame, rounded up
  int win = -1, win_slot = -1;  // r's face record, its leaf's place
  uint2* stack = s_stack + threadIdx.x;
  bool complete = p.ok;
  int sp = 0, node = p.ok ? 0 : -1;
  while (node >= 0) {
    const float4* rec = reinterpret_cast<const float4*>(a.walk + node);
    const int4 meta = __ldg(reinterpret_cast<const int4*>(rec));
    int go = -1;
    if (meta.w > 0) {
      // The faces whose own discs do not rule them out, up to 32 at a time, then those
      // exactly.
      for (int k0 = 0; k0 < meta.w; k0 += 32) {
        const int n = min(meta.w - k0, 32);
        const float4* disc = reinterpret_cast<const float4*>(a.face_discs + meta.z + k0);
        unsigned todo = 0;
        for (int k = 0; k < n; ++k) {
          float v2;
          const float lb = disc_bound2(fx, fy, fz, __ldg(disc + 2 * k), __ldg(disc + 2 * k + 1),
                                       margin, v2);
          if (!(lb > bestf)) todo |= 1u << k;
        }
        while (todo) {
          const int k = meta.z + k0 + __ffs(todo) - 1;
          todo &= todo - 1;
          int64_t face;
          const ClosestHit h = closest_on_record(a.tris + k, px, py, pz, face);
          // Of equal distances the one that the reference meets first; a leaf's records come
          // in its order here too.
          if (h.d2 < r.d2 || (h.d2 == r.d2 && meta.x != win_slot &&
                              comes_first(a, meta.x, win, px, py, pz))) {
            r = Best{h.d2, h.x, h.y, h.z, face};
            bestf = __double2float_ru(h.d2 * a.frame.s * a.frame.s);
            win = k;
            win_slot = meta.x;
          }
        }
      }
    } else {
      const float4 ln = __ldg(rec + 1), lc = __ldg(rec + 2), rn = __ldg(rec + 3),
                   rc = __ldg(rec + 4), b0 = __ldg(rec + 5), b1 = __ldg(rec + 6),
                   b2 = __ldg(rec + 7);
      float vl, vr;
      const float kl = fmaxf(disc_bound2(fx, fy, fz, ln, lc, margin, vl),
                             box_bound2(fx, fy, fz, b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, margin));
      const float kr = fmaxf(disc_bound2(fx, fy, fz, rn, rc, margin, vr),
                             box_bound2(fx, fy, fz, b1.z, b1.w, b2.x, b2.y, b2.z, b2.w, margin));
      const bool left = !(kl > bestf), right = !(kr > bestf);
      if (left && right) {
        const bool left_first = vl < vr;
        go = left_first ? meta.x : meta.y;
        if (sp < a.levels) {  // always, in a validated tree
          stack[sp * kAabbThreads] = make_uint2(static_cast<unsigned>(left_first ? meta.y : meta.x),
                                                __float_as_uint(left_first ? kr : kl));
          ++sp;
        } else {
          complete = false;  // not all seen: the reference's walk decides
          atomicOr(a.err, kErrBadLaunch);
        }
      } else if (left || right) {
        go = left ? meta.x : meta.y;
      }
    }
    while (go < 0 && sp > 0) {
      --sp;
      const uint2 e = stack[sp * kAabbThreads];
      if (!(__uint_as_float(e.y) > bestf)) go = static_cast<int>(e.x);
    }
    node = go;
  }
  if (complete && win >= 0) {
    const double d =
        win_slot < 0 ? box_distance2(px, py, pz, a.root[0], a.root[1], a.root[2], a.root[3],
                                     a.root[4], a.root[5])
                     : box_of(win_slot & 1 ? a.nodes[win_slot >> 1].rbox : a.nodes[win_slot >> 1].lbox,
                              px, py, pz);
    complete = d <= r.d2;
  }
  if (!complete || win < 0) r = ordered_walk(a, px, py, pz);
  store_result(a, qi, r);
}

// ---- discs ---------------------------------------------------------------------

template <class T, class F>
__device__ __forceinline__ T block_reduce(T v, T* part, F f) {
  for (int o = 16; o; o >>= 1) v = f(v, __shfl_xor_sync(~0u, v, o));
  const int nw = blockDim.x >> 5;
  if (nw == 1) return v;
  __syncthreads();  // the array's last readers are done
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  v = part[0];
  for (int k = 1; k < nw; ++k) v = f(v, part[k]);
  return v;
}

// A node's walk record, its discs without bounds yet.
__global__ void aabb_walk_kernel(const AabbNodeRec* __restrict__ nodes,
                                 const AabbSpan* __restrict__ spans, int64_t n, const AabbFrame f,
                                 AabbWalkRec* __restrict__ walk) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const AabbNodeRec& r = nodes[i];
  const AabbDisc none{{0.f, 0.f, 0.f}, INFINITY, {0.f, 0.f, 0.f}, INFINITY};
  AabbWalkRec w;
  const bool leaf = r.count > 0;
  w.left = leaf ? spans[i].slot : r.left;
  w.right = r.right;
  w.start = leaf ? r.start : spans[r.right].first;
  w.count = r.count;
  w.ldisc = w.rdisc = none;
  for (int k = 0; k < 3; ++k) {  // unused in a leaf
    w.lbox[k] = __double2float_rd((r.lbox[k] - f.c[k]) * f.s);
    w.rbox[k] = __double2float_rd((r.rbox[k] - f.c[k]) * f.s);
    w.lbox[3 + k] = __double2float_ru((r.lbox[3 + k] - f.c[k]) * f.s);
    w.rbox[3 + k] = __double2float_ru((r.rbox[3 + k] - f.c[k]) * f.s);
  }
  walk[i] = w;
}

__device__ __forceinline__ double3 local_corner(const AabbTriRec& t, int j, const AabbFrame& f) {
  const double* x = j == 0 ? t.a : (j == 1 ? t.b : t.c);
  return make_double3((x[0] - f.c[0]) * f.s, (x[1] - f.c[1]) * f.s, (x[2] - f.c[2]) * f.s);
}

// The disc of one node per CTA: of node list[blockIdx.x], or of node blockIdx.x unless
// it has more than kDiscBig faces. Three passes over its vertices: normal and shape of
// the faces; ranges along the normal and two axes across it (the centre); thickness and
// radius about the centre as rounded to FP32.
__global__ void aabb_disc_kernel(const AabbTriRec* __restrict__ tris,
                                 const AabbSpan* __restrict__ spans, const int32_t* list,
                                 const AabbFrame f, AabbWalkRec* walk, AabbNodeRec* nodes) {
  __shared__ double part[32];
  const int64_t node = list ? list[blockIdx.x] : static_cast<int64_t>(blockIdx.x);
  const AabbSpan s = spans[node];
  if (s.slot < 0 || s.last <= s.first) return;
  if (!list && s.last - s.first > kDiscBig) return;
  const int step = static_cast<int>(blockDim.x);
  const auto add = [](double a, double b) { return a + b; };
  const auto low = [](double a, double b) { return fmin(a, b); };
  const auto high = [](double a, double b) { return fmax(a, b); };
  double nx = 0.0, ny = 0.0, nz = 0.0, thin = 0.0;
  for (int k = s.first + threadIdx.x; k < s.last; k += step) {
    const AabbTriRec& t = tris[k];
    const double ux = (t.b[0] - t.a[0]) * f.s, uy = (t.b[1] - t.a[1]) * f.s,
                 uz = (t.b[2] - t.a[2]) * f.s;
    const double wx = (t.c[0] - t.a[0]) * f.s, wy = (t.c[1] - t.a[1]) * f.s,
                 wz = (t.c[2] - t.a[2]) * f.s;
    const double ex = wx - ux, ey = wy - uy, ez = wz - uz;
    const double cx = uy * wz - uz * wy, cy = uz * wx - ux * wz, cz = ux * wy - uy * wx;
    const double l2 = fmax(fmax(ux * ux + uy * uy + uz * uz, wx * wx + wy * wy + wz * wz),
                           ex * ex + ey * ey + ez * ez);
    if (!(cx * cx + cy * cy + cz * cz >= kThin * l2 * l2)) thin = 1.0;
    nx += cx;
    ny += cy;
    nz += cz;
  }
  nx = block_reduce(nx, part, add);
  ny = block_reduce(ny, part, add);
  nz = block_reduce(nz, part, add);
  thin = block_reduce(thin, part, high);
  const double len = sqrt(nx * nx + ny * ny + nz * nz);
  const bool has = len > 0.0 && len < INFINITY;
  nx = has ? nx / len : 1.0;
  ny = has ? ny / len : 0.0;
  nz = has ? nz / len : 0.0;
  // As floats, shortened until |n| <= 1 (then |n.(p - x)| <= |p - x|).
  const double keep = 1.0 - 1.5e-7;
  const float fx = static_cast<float>(nx * keep), fy = static_cast<float>(ny * keep),
              fz = static_cast<float>(nz * keep);
  // Two axes across n.
  const bool zmost = fabs(nz) < 0.7;
  const double vx0 = zmost ? ny : -nz, vy0 = zmost ? -nx : 0.0, vz0 = zmost ? 0.0 : nx;
  const double vl = 1.0 / sqrt(vx0 * vx0 + vy0 * vy0 + vz0 * vz0);
  const double ux = vx0 * vl, uy = vy0 * vl, uz = vz0 * vl;
  const double wx = ny * uz - nz * uy, wy = nz * ux - nx * uz, wz = nx * uy - ny * ux;
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int k = s.first + threadIdx.x; k < s.last; k += step)
    for (int j = 0; j < 3; ++j) {
      const double3 x = local_corner(tris[k], j, f);
      const double d[3] = {nx * x.x + ny * x.y + nz * x.z, ux * x.x + uy * x.y + uz * x.z,
                           wx * x.x + wy * x.y + wz * x.z};
      for (int i = 0; i < 3; ++i) {
        lo[i] = fmin(lo[i], d[i]);
        hi[i] = fmax(hi[i], d[i]);
      }
    }
  double mid[3];
  for (int i = 0; i < 3; ++i)
    mid[i] = 0.5 * (block_reduce(lo[i], part, low) + block_reduce(hi[i], part, high));
  const float cx = static_cast<float>(nx * mid[0] + ux * mid[1] + wx * mid[2]);
  const float cy = static_cast<float>(ny * mid[0] + uy * mid[1] + wy * mid[2]);
  const float cz = static_cast<float>(nz * mid[0] + uz * mid[1] + wz * mid[2]);
  double t = 0.0, r2 = 0.0, w2 = 0.0, dlo = INFINITY, dhi = -INFINITY;
  for (int k = s.first + threadIdx.x; k < s.last; k += step)
    for (int j = 0; j < 3; ++j) {
      const double3 x = local_corner(tris[k], j, f);
      const double dx = x.x - cx, dy = x.y - cy, dz = x.z - cz;
      const double h = static_cast<double>(fx) * dx + static_cast<double>(fy) * dy +
                       static_cast<double>(fz) * dz;
      const double q = dx * dx + dy * dy + dz * dz;
      const double d = static_cast<double>(fx) * x.x + static_cast<double>(fy) * x.y +
                       static_cast<double>(fz) * x.z;
      t = fmax(t, fabs(h));
      r2 = fmax(r2, q - h * h);
      w2 = fmax(w2, q);
      dlo = fmin(dlo, d);
      dhi = fmax(dhi, d);
    }
  dlo = block_reduce(dlo, part, low);
  dhi = block_reduce(dhi, part, high);
  t = block_reduce(t, part, high);
  r2 = block_reduce(r2, part, high);
  w2 = block_reduce(w2, part, high);
  if (threadIdx.x != 0) return;
  const bool right = s.slot & 1;
  AabbDisc& out = right ? walk[s.slot >> 1].rdisc : walk[s.slot >> 1].ldisc;
  const double pad = 1e-12;  // >> the rounding of the sums above
  out.n[0] = fx;
  out.n[1] = fy;
  out.n[2] = fz;
  out.c[0] = cx;
  out.c[1] = cy;
  out.c[2] = cz;
  out.t = __double2float_ru(t + pad);
  out.r = thin > 0.0 ? INFINITY : __double2float_ru(sqrt(r2 + 1e-14 * w2) * (1.0 + 1e-9) + pad);
  AabbNodeRec& parent = nodes[s.slot >> 1];
  (right ? parent.rslab : parent.lslab) =
      AabbSlab{{fx, fy, fz}, __double2float_rd(dlo - pad), __double2float_ru(dhi + pad)};
}

// The disc of every face: about its centroid, along its own normal.
__global__ void aabb_face_disc_kernel(const AabbTriRec* __restrict__ tris, int64_t n,
                                      const AabbFrame f, AabbDisc* __restrict__ out,
                                      int32_t* __restrict__ thin) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const AabbTriRec& t = tris[i];
  const double ux = (t.b[0] - t.a[0]) * f.s, uy = (t.b[1] - t.a[1]) * f.s,
               uz = (t.b[2] - t.a[2]) * f.s;
  const double wx = (t.c[0] - t.a[0]) * f.s, wy = (t.c[1] - t.a[1]) * f.s,
               wz = (t.c[2] - t.a[2]) * f.s;
  const double ex = wx - ux, ey = wy - uy, ez = wz - uz;
  double nx = uy * wz - uz * wy, ny = uz * wx - ux * wz, nz = ux * wy - uy * wx;
  const double l2 = fmax(fmax(ux * ux + uy * uy + uz * uz, wx * wx + wy * wy + wz * wz),
                         ex * ex + ey * ey + ez * ez);
  const double nn = nx * nx + ny * ny + nz * nz;
  const bool is_thin = !(nn >= kThin * l2 * l2);
  if (is_thin) atomicAdd(thin, 1);
  const double inv = nn > 0.0 && nn < INFINITY ? (1.0 - 1.5e-7) / sqrt(nn) : 0.0;
  AabbDisc d;
  d.n[0] = static_cast<float>(nx * inv);
  d.n[1] = static_cast<float>(ny * inv);
  d.n[2] = static_cast<float>(nz * inv);
  double3 x[3];
  for (int j = 0; j < 3; ++j) x[j] = local_corner(t, j, f);
  d.c[0] = static_cast<float>((x[0].x + x[1].x + x[2].x) / 3.0);
  d.c[1] = static_cast<float>((x[0].y + x[1].y + x[2].y) / 3.0);
  d.c[2] = static_cast<float>((x[0].z + x[1].z + x[2].z) / 3.0);
  double h = 0.0, r2 = 0.0, w2 = 0.0;
  for (int j = 0; j < 3; ++j) {
    const double dx = x[j].x - d.c[0], dy = x[j].y - d.c[1], dz = x[j].z - d.c[2];
    const double p = d.n[0] * dx + d.n[1] * dy + d.n[2] * dz;
    const double q = dx * dx + dy * dy + dz * dz;
    h = fmax(h, fabs(p));
    r2 = fmax(r2, q - p * p);
    w2 = fmax(w2, q);
  }
  const double pad = 1e-12;
  d.t = __double2float_ru(h + pad);
  d.r = is_thin ? INFINITY : __double2float_ru(sqrt(r2 + 1e-14 * w2) * (1.0 + 1e-9) + pad);
  float4* dst = reinterpret_cast<float4*>(out + i);
  dst[0] = make_float4(d.n[0], d.n[1], d.n[2], d.t);
  dst[1] = make_float4(d.c[0], d.c[1], d.c[2], d.r);
}

__global__ void signed_from_winding_kernel(const double* __restrict__ w, double* __restrict__ s,
                                           int64_t n) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double d = __dsqrt_rn(s[i]);
  s[i] = fabs(w[i]) > 0.5 ? -d : d;
}

}  // namespace

cudaError_t aabb_query(const AabbDeviceTree& t, const double* P, int64_t np, const uint32_t* perm,
                       double* sqrd, int64_t* index, double* closest, int* err,
                       cudaStream_t stream) {
  if (np <= 0) return cudaSuccess;
  if (t.depth + 1 > kAabbStack) return cudaErrorInvalidValue;
  AabbArgs a{t.nodes, t.walk, t.spans, t.tris, t.face_discs, P, perm, sqrd, index, closest, err, np,
             t.nnodes, {}, t.scale, t.frame, t.depth};
  for (int k = 0; k < 6; ++k) a.root[k] = t.root[k];
  const int64_t blocks = (np + kAabbThreads - 1) / kAabbThreads;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  const size_t stack_bytes = sizeof(uint2) * kAabbThreads * t.depth;
  if (t.any_order && t.nleaf_faces >= kOrderFaces && stack_bytes <= kStackBytes)
    aabb_any_order_kernel<<<static_cast<unsigned>(blocks), kAabbThreads, stack_bytes, stream>>>(a);
  else if (t.nleaf_faces >= kDiscFaces && t.thin <= t.nleaf_faces / kDiscShare)
    aabb_query_kernel<true><<<static_cast<unsigned>(blocks), kAabbThreads, 0, stream>>>(a);
  else
    aabb_query_kernel<false><<<static_cast<unsigned>(blocks), kAabbThreads, 0, stream>>>(a);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

cudaError_t aabb_discs(const AabbDeviceTree& t, const int32_t* big, int64_t nbig,
                       int32_t* thin, cudaStream_t stream) {
  if (t.nnodes <= 0) return cudaSuccess;
  aabb_walk_kernel<<<static_cast<unsigned>((t.nnodes + 255) / 256), 256, 0, stream>>>(
      t.nodes, t.spans, t.nnodes, t.frame, t.walk);
  aabb_disc_kernel<<<static_cast<unsigned>(t.nnodes), 32, 0, stream>>>(t.tris, t.spans, nullptr,
                                                                       t.frame, t.walk, t.nodes);
  if (nbig > 0)
    aabb_disc_kernel<<<static_cast<unsigned>(nbig), 512, 0, stream>>>(t.tris, t.spans, big, t.frame,
                                                                      t.walk, t.nodes);
  aabb_face_disc_kernel<<<static_cast<unsigned>((t.nleaf_faces + 255) / 256), 256, 0, stream>>>(
      t.tris, t.nleaf_faces, t.frame, t.face_discs, thin);
  g_launches.fetch_add(nbig > 0 ? 4 : 3, std::memory_order_relaxed);
  return cudaGetLastError();
}

cudaError_t signed_from_winding(const double* w, double* s, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  const int64_t blocks = (n + 255) / 256;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  signed_from_winding_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(w, s, n);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

}  // namespace wn
