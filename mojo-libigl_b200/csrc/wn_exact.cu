// Exact generalized winding number without visiting every (query, face) pair.
//
// The same number as the all-pairs kernels (lee101/mojo-libigl,
// src/capi.mojo:205-286): W(o) = sum_f Omega_f(o) / 4 pi. Split the faces at a
// query into the near ones N and the far ones. The far faces are a surface that
// does not come close to the query, and the solid angle of a surface depends on
// its boundary alone up to whole turns (A. Jacobson, L. Kavan, O. Sorkine-Hornung,
// "Robust Inside-Outside Segmentation using Generalized Winding Numbers", 2013,
// replaces far patches by caps on this ground). So
//
//   W(o) = sum_{f in N} Omega_f / 4 pi  +  arg(prod_e z_e) / 2 pi  +  k
//
// 1. Near faces: their FP64 pair terms, with turns counted (wn_pair.cuh), as in the
//    all-pairs kernels. Everything that is sensitive to the last bits (queries on
//    vertices, on edges, in faces) happens here, with the bit-exact terms; faces whose
//    denominator is positive by a margin take the cheaper ones (wn_pair_device.cuh).
// 2. Boundary edges e = u -> v of the far faces: the infinite triangle from the
//    edge towards a direction D closes the surface. Its solid angle is
//    2 arg z_e with, for unit vectors a and b from o to u and v,
//      z_e = 1 + a.b + D.a + D.b + i D.(a x b)
//    (van Oosterom-Strackee with the third corner at infinity). Only the product
//    matters, in FP64; no turn is counted. An edge between two far faces cancels
//    and is never formed: the far boundary is the mesh's own boundary ("root"
//    edges, none on a closed mesh) minus the boundary of N.
// 3. The integer k = round(W_far - arg/2 pi) from an approximate W_far, in FP32:
//    second-order expansions of far nodes of a tree (G. Barill et al., "Fast
//    Winding Numbers for Soups and Clouds", 2018) and FP32 solid angles of the
//    leaves in between. k is certain while the error of W_far stays below 1/2,
//    and that error is bounded, not estimated: the expansion of
//    grad(1/|x - o|) about p has terms |G_n| <= (n + 1) rho^n / d^2 with
//    rho = r/d (d = |p - o|, r bounds the node's vertices about p; the gradient
//    of a solid harmonic of degree m is at most m on the unit sphere, by
//    Bernstein's inequality), so a node of total area A is off by at most
//      A / (4 pi d^2) * rho^3 (4 - 3 rho) / (1 - rho)^2.
//    A warp whose sum of these exceeds kMaxBound walks again with a stricter
//    opening rule; a query for which that fails, whose product comes too close to
//    zero for every D, or whose integer does not fit within the bound is summed
//    over all pairs by exact_fallback_kernel.
//
// Edges cancel by position: two directed sides with bitwise equal endpoints in
// opposite directions are partners, whatever their indices, so triangle soups
// whose faces meet work like meshes, and any input is correct: an unpaired side
// is simply a root edge. Where too many are left (kExactMost*, boundary_pays), or the
// mesh is dense or crowded (kMostDense, kMostCrowded*), the method does not pay and an
// all-pairs kernel does the call.
#include <cub/cub.cuh>

#include <algorithm>

#include "wn_common.cuh"
#include "wn_exact.h"
#include "wn_internal.h"
#include "wn_pair.cuh"
#include "wn_pair_device.cuh"

namespace wn {
namespace {

constexpr int kLeaf = kExactLeafFaces;
constexpr int kLeafEdges = 3 * kLeaf;
constexpr int kWarps = 4;            // warps per CTA
constexpr int kStack = 1536;         // node stack of a warp
constexpr float kPad = 0.05f;        // near box: the leaf's box grown by kPad * diagonal
constexpr float kPadAbs = 1e-6f;     // ... and by this much of the mesh's extent
constexpr float kSlack = 3e-7f;      // FP32 rounding of node centres (|p| <= 1)
constexpr float kBeta = 2.5f;        // a node is far when d >= beta * r
constexpr float kMaxBound = 0.45f;   // proven error of W_far below which k is certain
constexpr int kBetaTries = 4;        // beta = 2.5, 3.25, 4.55, 9.1
constexpr int kDirTries = 4;
constexpr int kMinExp = (1023 - 7) << 20;  // |z_e| >= ~2^-7, else try another direction
constexpr int kChain = 64;           // longest hash chain that is searched for partners
constexpr int kMaxLoop = 8;          // boundary loops of at most this many edges become fans
constexpr double kFarQuery = 1e9;    // queries beyond this many extents: all pairs
// Meshes that the method is the slower one for, whatever their edges:
// Dense ones: the area in a face's coarse cell, in faces of the cell, in the mean over the
// faces. Every query then has surface all around it: expansions are far only under strict
// opening rules, and the second and later walks of exact_eval_kernel cost more than the
// pairs. 65,536 Q, ms, this and the FP64 streaming kernel: 128 concentric spheres (9.9) 52
// and 52 (16,384 Q), 256 (25) 144 and 105; 10,000 spheres of radius 0.1 in a cube of side 2
// (8.9) 52 and 64, 0.15 (18.8) 89 and 64, 0.2 (33) 170 and 64; the tetrahedra of a grid of
// 12^3 (11.8) 19 and 13, 16^3 (10.9) 25 and 32, 24^3 (12.3) 104 and 106, 32^3 (14.5) 101 and
// 62 (16,384 Q); 20,000 tetrahedra of side 0.1 (15.8) 44 and 26.
constexpr double kMostDense = 11.5;
// Crowded ones: faces that share a cell of the order with this share of all faces, in the
// mean (a triangle 1,000 times the rest's size away, or a part of 1 : 1,000). Within a cell
// the order is the input's, and every leaf is near: an outlier at 10^6 61 ms, 26 (FP64
// streaming) and 13 (mixed); at 10^3 (0.12) 40, 26 and 12; a ball of 1 : 1,000 beside a ground
// of its own, half of the queries near either (0.11) 12, 28 and 12.
constexpr double kMostCrowdedFp64 = 0.5, kMostCrowdedMixed = 0.02;

struct Info {
  unsigned long long lo[3], hi[3];    // vertex box, ordered keys
  unsigned long long qlo[3], qhi[3];  // box of the queries clamped to twice the mesh's
  int32_t bad;                        // a vertex is not finite
  int32_t nopen;                      // sides without a partner
  int32_t nroot, nitem, ngroup;       // root edges, the triangles and single edges that
                                      // stand for them, the groups they form
  int32_t nlist;                      // queries left to exact_fallback_kernel
  unsigned long long crowd;           // sum over the order's cells of their faces, squared
  unsigned long long density;         // sum over the faces of their coarse cells' area, in faces
                                      // of a cell (2^-8: below 2^63 for 10^7 of the largest)
};

// Coarse cells, 32 to an axis: the upper half of the order's key.
constexpr int kCoarseShift = 15, kCoarse = 1 << 15;
constexpr double kCoarseUnit = 1 << 16;

// 80-byte face: corners A, B, C (FP64), in sorted order.
struct Face64 {
  double v[9];
  double pad;
};
// Raw moments of a node about its centre p (scaled coordinates): total area, p,
// M0_i = sum a n_i, M1_ji = sum a n_i d_j, M2_jki = 1/2 sum a n_i (d_j d_k + C_jk)
// (jk = 00, 01, 02, 11, 12, 22; C a face's second moment about its centroid).
struct Moments {
  double area, p[3], m0[3], m1[3][3], m2[6][3];
};
// What the walk reads of a node: near box, centre, radius, area / (4 pi r^2), and
// the children (first << 2 | count - 1; -1: a leaf).
struct alignas(16) NodeTest {
  float lo[3], hi[3], p[3], r, area;
  int32_t child;
};
static_assert(sizeof(NodeTest) == 48, "three 16-byte words");
// What the expansion reads: the centre as a float pair, r, and the 19 coefficients
// left of the 23 monomials when z^2 = 1 - x^2 - y^2 on the unit sphere.
struct alignas(16) NodeEval {
  float ph[3], r, pl[3], t0[3], qc, q00, q11, q01, q02, q12, l[3];
  float c000, c111, c001, c011, c002, c112, c012, pad[2];
};
static_assert(sizeof(NodeEval) == 112, "seven 16-byte words");
// FP32 face of a leaf that is neither near nor far: corner A relative to the leaf's
// centre, the sides e1 = B - A and e2 = C - A, n = e1 x e2 and the sides' products
// (the mixed kernel's record, wn_mixed.h). The spare word of faces 0..5 holds the
// leaf's centre as a float pair (ph, pl), so that a leaf is one 512-byte read.
struct alignas(16) Face32 {
  float ax, ay, az, e1x, e1y, e1z, e2x, e2y, e2z, nx, ny, nz, e11, e22, e12, centre;
};
static_assert(sizeof(Face32) == 64, "a leaf's faces are one 16-byte word per lane");
// A boundary loop of the mesh of 3..kMaxLoop edges (fanned from its first vertex when
// none of its leaves is near) or one edge on its own: the box that holds the near
// boxes of the edges' leaves, and the edges.
struct alignas(16) Group {
  float lo[3], hi[3];
  int32_t first, count, triangle, pad[3];  // first edge, edges, first triangle of its fan
};
struct Root {
  double u[3], v[3];
};
// Triangle (A, A + e1, A + e2) of a loop's fan, with n = e1 x e2 and the sides' products:
// with a = A - o the pair needs |a|^2, a.e1, a.e2 and a.n only (50 FP64 operations with
// the product; 63 from the corners).
struct alignas(16) Triangle {
  double a[3], e1[3], e2[3], n[3], e11, e22, e12, pad;
};
static_assert(sizeof(Triangle) == 128, "eight 16-byte words");

__device__ __forceinline__ unsigned long long okey(double x) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(x));
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double okey_inv(unsigned long long k) {
  return __longlong_as_double(
      static_cast<long long>((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k));
}

// Scaled coordinates: x' = (x - c) s, s a power of two, the mesh in [-1, 1]^3.
struct Frame {
  double c[3], s;
};
__device__ __forceinline__ Frame frame_of(const Info* info) {
  Frame f;
  double ext = 0.0;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const double lo = okey_inv(info->lo[x]), hi = okey_inv(info->hi[x]);
    f.c[x] = 0.5 * lo + 0.5 * hi;
    ext = fmax(ext, 0.5 * hi - 0.5 * lo);
  }
  // 2^-ceil(log2 ext): from the exponent; a point mesh keeps scale 1.
  const int e = (__double2hiint(ext) >> 20) & 0x7ff;
  f.s = e > 60 && e < 1980 ? __hiloint2double((2045 - e) << 20, 0) : 1.0;
  return f;
}

__global__ void exact_init_kernel(Info* info) {
  const int t = threadIdx.x;
  if (t < 3) {
    info->lo[t] = info->qlo[t] = ~0ull;
    info->hi[t] = info->qhi[t] = 0ull;
  }
  if (t == 0) {
    info->bad = info->nopen = info->nroot = info->nitem = info->ngroup = info->nlist = 0;
    info->crowd = info->density = 0;
  }
}

// Block-wide min/max of three coordinates into ordered keys: one atomic per block
// and bound (one per warp made the atomics the cost: 24 us at 1M points).
__device__ __forceinline__ void reduce_box(double lo[3], double hi[3], unsigned long long* klo,
                                           unsigned long long* khi) {
  __shared__ double part[2][3][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int x = 0; x < 3; ++x)
    for (int o = 16; o; o >>= 1) {
      lo[x] = fmin(lo[x], __shfl_xor_sync(~0u, lo[x], o));
      hi[x] = fmax(hi[x], __shfl_xor_sync(~0u, hi[x], o));
    }
  if (lane == 0)
    for (int x = 0; x < 3; ++x) {
      part[0][x][warp] = lo[x];
      part[1][x][warp] = hi[x];
    }
  __syncthreads();
  if (threadIdx.x < 3) {
    const int x = threadIdx.x;
    double l = part[0][x][0], h = part[1][x][0];
    for (int k = 1; k < nw; ++k) {
      l = fmin(l, part[0][x][k]);
      h = fmax(h, part[1][x][k]);
    }
    if (l <= h) {
      atomicMin(klo + x, okey(l));
      atomicMax(khi + x, okey(h));
    }
  }
}

__global__ void exact_face_box_kernel(const double* __restrict__ tri, int64_t ld, int64_t nf,
                                      Info* info) {
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  bool bad = false;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nf;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
#pragma unroll
    for (int r = 0; r < 9; ++r) {
      const double v = tri[r * ld + i];
      // Coordinates whose products could overflow, or that are not finite.
      bad |= !(fabs(v) < 1e75);
      lo[r % 3] = fmin(lo[r % 3], v);
      hi[r % 3] = fmax(hi[r % 3], v);
    }
  if (bad) info->bad = 1;
  reduce_box(lo, hi, info->lo, info->hi);
}

__device__ __forceinline__ void scaled_query(const double* q, int64_t i, const Frame& f,
                                             double p[3]) {
#pragma unroll
  for (int x = 0; x < 3; ++x) p[x] = (q[3 * i + x] - f.c[x]) * f.s;
}

// The box that the query order's cells divide: the queries' own, but never more than
// twice the mesh's, so that a few distant points do not coarsen the others' order.
__global__ void exact_query_box_kernel(const double* __restrict__ q, int64_t nq, Info* info) {
  const Frame f = frame_of(info);
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nq;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    double p[3];
    scaled_query(q, i, f, p);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const double v = fmin(fmax(p[x], -2.0), 2.0);
      lo[x] = fmin(lo[x], v);
      hi[x] = fmax(hi[x], v);
    }
  }
  reduce_box(lo, hi, info->qlo, info->qhi);
}

// Position along a Hilbert curve of 2^10 cells per axis (J. Skilling, "Programming
// the Hilbert curve", 2004): consecutive runs are compact patches with a quarter
// less boundary than Morton runs.
__device__ __forceinline__ uint32_t hilbert30(uint32_t x, uint32_t y, uint32_t z) {
  uint32_t X[3] = {x, y, z};
#pragma unroll
  for (uint32_t Q = 512; Q > 1; Q >>= 1) {
    const uint32_t P = Q - 1;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      if (X[i] & Q) {
        X[0] ^= P;
      } else {
        const uint32_t t = (X[0] ^ X[i]) & P;
        X[0] ^= t;
        X[i] ^= t;
      }
    }
  }
  X[1] ^= X[0];
  X[2] ^= X[1];
  uint32_t t = 0;
#pragma unroll
  for (uint32_t Q = 512; Q > 1; Q >>= 1)
    if (X[2] & Q) t ^= Q - 1;
  uint32_t key = 0;
#pragma unroll
  for (int b = 9; b >= 0; --b)
#pragma unroll
    for (int i = 0; i < 3; ++i) key = (key << 1) | (((X[i] ^ t) >> b) & 1u);
  return key;
}

__device__ __forceinline__ uint32_t cell_key(const double p[3], const double lo[3],
                                             const double hi[3]) {
  uint32_t c[3];
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const double ext = hi[x] - lo[x];
    const double u = ext > 0.0 ? (p[x] - lo[x]) / ext : 0.0;
    c[x] = min(static_cast<uint32_t>(fmin(fmax(u, 0.0), 1.0) * 1024.0), 1023u);
  }
  return hilbert30(c[0], c[1], c[2]);
}

__global__ void exact_face_keys_kernel(const double* __restrict__ tri, int64_t ld, int64_t nf,
                                       const Info* __restrict__ info, uint32_t* keys,
                                       uint32_t* vals, unsigned long long* coarse) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= nf) return;
  double p[3], lo[3], hi[3], u[3], v[3];
  double ext = 0.0;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const double a = tri[x * ld + i], b = tri[(3 + x) * ld + i], c = tri[(6 + x) * ld + i];
    p[x] = (a + b + c) * (1.0 / 3.0);
    u[x] = b - a;
    v[x] = c - a;
    lo[x] = okey_inv(info->lo[x]);
    hi[x] = okey_inv(info->hi[x]);
    ext = fmax(ext, hi[x] - lo[x]);
  }
  const uint32_t key = cell_key(p, lo, hi);
  keys[i] = key;
  vals[i] = static_cast<uint32_t>(i);
  const double s = ext > 0.0 ? 32.0 / ext : 0.0;  // sides in cells
  const double nx = (u[1] * s) * (v[2] * s) - (u[2] * s) * (v[1] * s),
               ny = (u[2] * s) * (v[0] * s) - (u[0] * s) * (v[2] * s),
               nz = (u[0] * s) * (v[1] * s) - (u[1] * s) * (v[0] * s);
  const double area = 0.5 * sqrt(nx * nx + ny * ny + nz * nz);
  // In whole units: the sum is the same in any order.
  atomicAdd(coarse + (key >> kCoarseShift),
            static_cast<unsigned long long>(fmin(area, 4096.0) * kCoarseUnit + 0.5));
}

__global__ void exact_query_keys_kernel(const double* __restrict__ q, int64_t nq,
                                        const Info* __restrict__ info, uint32_t* keys,
                                        uint32_t* vals) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  const Frame f = frame_of(info);
  double p[3], lo[3], hi[3];
  scaled_query(q, i, f, p);
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    lo[x] = okey_inv(info->qlo[x]);
    hi[x] = okey_inv(info->qhi[x]);
  }
  keys[i] = cell_key(p, lo, hi);
  vals[i] = static_cast<uint32_t>(i);
}

// ---- edge partners -----------------------------------------------------------

// A. Appleby's 32-bit finaliser (MurmurHash3), a coordinate's halves mixed in between.
__device__ __forceinline__ uint32_t point_hash(const double* v) {
  uint32_t h = 0x9e3779b9u;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const unsigned long long b =
        static_cast<unsigned long long>(__double_as_longlong(v[x] + 0.0));  // -0 -> +0
    h = (h ^ static_cast<uint32_t>(b)) * 0x85ebca6bu;
    h = ((h >> 15) ^ h ^ static_cast<uint32_t>(b >> 32)) * 0xc2b2ae35u;
    h ^= h >> 13;
  }
  return h;
}
__device__ __forceinline__ bool same_point(const double* a, const double* b) {
  return a[0] == b[0] && a[1] == b[1] && a[2] == b[2];
}
__device__ __forceinline__ const double* corner_of(const Face64* faces, uint32_t edge, int end) {
  uint32_t c = edge % 3u + end;
  c = c == 3u ? 0u : c;
  return faces[edge / 3u].v + 3 * c;
}

constexpr int kGatherThreads = 128;
// Sorted faces as 80-byte records; every side enters the chain of its hash slot
// (side e = 3 * sorted face + corner, from that corner to the next).
__global__ void exact_gather_kernel(const double* __restrict__ tri, int64_t ld, int64_t nf,
                                    const uint32_t* __restrict__ order,
                                    const uint32_t* __restrict__ keys,
                                    const unsigned long long* __restrict__ coarse, Face64* faces,
                                    uint32_t* heads, uint32_t mask, uint32_t* next, Info* info) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  unsigned long long around = i < nf ? coarse[keys[i] >> kCoarseShift] : 0;
#pragma unroll
  for (int o = 16; o; o >>= 1) around += __shfl_xor_sync(~0u, around, o);
  __shared__ unsigned long long part[kGatherThreads / 32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = around;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < kGatherThreads / 32; ++k) around += part[k];
    atomicAdd(&info->density, around >> 8);
  }
  if (i >= nf) return;
  const uint32_t f = order[i];
  // The first face of a cell that holds more than 64.
  const uint32_t key = keys[i];
  if (i + 64 < nf && keys[i + 64] == key && (i == 0 || keys[i - 1] != key)) {
    int64_t lo = i + 64, hi = nf;  // key at lo; not at hi
    while (hi - lo > 1) {
      const int64_t mid = lo + (hi - lo) / 2;
      if (keys[mid] == key) lo = mid; else hi = mid;
    }
    const unsigned long long n = static_cast<unsigned long long>(hi - i);
    atomicAdd(&info->crowd, n * n);
  }
  double v[10];
#pragma unroll
  for (int r = 0; r < 9; ++r) v[r] = tri[r * ld + f];
  v[9] = 0.0;
  double2* dst = reinterpret_cast<double2*>(faces + i);
#pragma unroll
  for (int k = 0; k < 5; ++k) dst[k] = make_double2(v[2 * k], v[2 * k + 1]);
  const uint32_t h[3] = {point_hash(v), point_hash(v + 3), point_hash(v + 6)};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const uint32_t slot = hash_slot(h[c] + h[(c + 1) % 3], mask);
    const uint32_t e = static_cast<uint32_t>(3 * i + c);
    next[e] = atomicExch(heads + slot, e);
  }
}

// partner[e]: the side that cancels side e, ~0 for a root edge, ~1 for a side
// without length; nb[e]: the partner's leaf when that is another one, else -1.
// Partners pair the k-th side of one direction with the k-th of the other (by
// number), so any number of faces may share an edge. Sides whose chain is longer
// than kChain stay unpaired, all of them alike: still a valid boundary.
constexpr uint32_t kNoPartner = ~0u, kNoLength = ~1u;

// True if side e stays unpaired.
__device__ __forceinline__ bool pair_side(const Face64* __restrict__ faces, uint32_t e,
                                          const uint32_t* __restrict__ heads, uint32_t mask,
                                          const uint32_t* __restrict__ next,
                                          uint32_t* __restrict__ partner,
                                          int32_t* __restrict__ nb) {
  double u[3], v[3];
  {
    const double *pu = corner_of(faces, e, 0), *pv = corner_of(faces, e, 1);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      u[x] = pu[x];
      v[x] = pv[x];
    }
  }
  if (same_point(u, v)) {
    partner[e] = kNoLength;
    nb[e] = -1;
    return false;
  }
  const uint32_t head = heads[hash_slot(point_hash(u) + point_hash(v), mask)];
  int rank = 0, nopp = 0, steps = 0;
  uint32_t opp = ~0u;
  for (uint32_t o = head; o != ~0u && steps <= kChain; o = next[o], ++steps) {
    if (o == e) continue;
    const double *a = corner_of(faces, o, 0), *b = corner_of(faces, o, 1);
    if (same_point(a, u) && same_point(b, v)) {
      rank += o < e;
    } else if (same_point(a, v) && same_point(b, u)) {
      ++nopp;
      opp = o;
    }
  }
  if (steps > kChain) nopp = 0;
  if (nopp > 1 && rank < nopp) {
    // The opposite side with `rank` smaller ones before it.
    for (uint32_t o = head; o != ~0u; o = next[o]) {
      if (!same_point(corner_of(faces, o, 0), v) || !same_point(corner_of(faces, o, 1), u))
        continue;
      int before = 0;
      for (uint32_t w = head; w != ~0u; w = next[w])
        before += w < o && same_point(corner_of(faces, w, 0), v) &&
                  same_point(corner_of(faces, w, 1), u);
      if (before == rank) {
        opp = o;
        break;
      }
    }
  }
  const uint32_t leaf = e / kLeafEdges, other = opp / kLeafEdges;
  partner[e] = rank < nopp ? opp : kNoPartner;
  nb[e] = rank < nopp && other != leaf ? static_cast<int32_t>(other) : -1;
  return rank >= nopp;
}

__global__ void exact_partner_kernel(const Face64* __restrict__ faces, int64_t nedge,
                                     const uint32_t* __restrict__ heads, uint32_t mask,
                                     const uint32_t* __restrict__ next,
                                     uint32_t* __restrict__ partner, int32_t* __restrict__ nb,
                                     Info* info) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const bool open = i < nedge && pair_side(faces, static_cast<uint32_t>(i), heads, mask, next,
                                           partner, nb);
  const int n = __syncthreads_count(open);
  if (threadIdx.x == 0 && n) atomicAdd(&info->nopen, n);
}

// What a leaf's sides lead, and (exclusive sums) what comes before it.
struct Counts {
  int32_t groups, edges, triangles;
};
struct AddCounts {
  __host__ __device__ __forceinline__ Counts operator()(const Counts& a, const Counts& b) const {
    return Counts{a.groups + b.groups, a.edges + b.edges, a.triangles + b.triangles};
  }
};

__device__ __forceinline__ uint32_t point_slot(const double* v, uint32_t mask) {
  return hash_slot(point_hash(v), mask);
}

// More sides without a partner than faces: the method is not taken (exact_boundary), and the
// kernels that look for loops leave at once.
__device__ __forceinline__ bool too_open(const Info* info, int64_t nedge) {
  return 3ll * info->nopen > nedge;
}

// Root edges into the chains of their first points.
__global__ void exact_root_hash_kernel(const Face64* __restrict__ faces, int64_t nedge,
                                       const uint32_t* __restrict__ partner, uint32_t* heads,
                                       uint32_t mask, uint32_t* next,
                                       const Info* __restrict__ info) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (too_open(info, nedge) || i >= nedge || partner[i] != kNoPartner) return;
  const uint32_t e = static_cast<uint32_t>(i);
  next[e] = atomicExch(heads + point_slot(corner_of(faces, e, 0), mask), e);
}

// Calls f(o) for the root edges that start at `v`; false when the chain is too long.
template <class F>
__device__ __forceinline__ bool each_root(const Face64* faces, const uint32_t* heads,
                                          uint32_t mask, const uint32_t* next, const double* v,
                                          F f) {
  int steps = 0;
  for (uint32_t o = heads[point_slot(v, mask)]; o != ~0u; o = next[o]) {
    if (++steps > kChain) return false;
    if (same_point(corner_of(faces, o, 0), v)) f(o);
  }
  return true;
}

// pick[e] of a root edge u -> v: the edge v -> w of the single missing face (u, v, w)
// that it bounds, the one with the smallest sides if there are several; ~0 if none.
__global__ void exact_pick_kernel(const Face64* __restrict__ faces, int64_t nedge,
                                  const uint32_t* __restrict__ partner,
                                  const uint32_t* __restrict__ heads, uint32_t mask,
                                  const uint32_t* __restrict__ next, uint32_t* __restrict__ pick,
                                  const Info* __restrict__ info) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (too_open(info, nedge) || i >= nedge || partner[i] != kNoPartner) return;
  const uint32_t e = static_cast<uint32_t>(i);
  const double *u = corner_of(faces, e, 0), *v = corner_of(faces, e, 1);
  uint32_t best = ~0u;
  unsigned long long lo = ~0ull;
  uint32_t hi = ~0u;
  each_root(faces, heads, mask, next, v, [&](uint32_t o) {
    each_root(faces, heads, mask, next, corner_of(faces, o, 1), [&](uint32_t r) {
      if (r == e || !same_point(corner_of(faces, r, 1), u)) return;
      // The three numbers in ascending order: every side compares the same keys.
      const uint32_t a = min(e, min(o, r)), c = max(e, max(o, r));
      const uint32_t b = e + o + r - a - c;
      const unsigned long long l = (static_cast<unsigned long long>(a) << 32) | b;
      if (l < lo || (l == lo && c < hi)) {
        lo = l;
        hi = c;
        best = o;
      }
    });
  });
  pick[e] = best;
}

// Whether all three sides of the missing face at root edge e chose it.
__device__ __forceinline__ bool picked(const uint32_t* pick, uint32_t e) {
  const uint32_t o = pick[e];
  if (o == ~0u) return false;
  const uint32_t r = pick[o];
  return r != ~0u && pick[r] == e;
}

// succ[e] of a root edge: the next edge of its loop, around the missing face or else
// the only root edge left that goes on from its end; ~0 if there are several.
__global__ void exact_successor_kernel(const Face64* __restrict__ faces, int64_t nedge,
                                       const uint32_t* __restrict__ partner,
                                       const uint32_t* __restrict__ heads, uint32_t mask,
                                       const uint32_t* __restrict__ next,
                                       const uint32_t* __restrict__ pick,
                                       uint32_t* __restrict__ succ,
                                       const Info* __restrict__ info) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (too_open(info, nedge) || i >= nedge || partner[i] != kNoPartner) return;
  const uint32_t e = static_cast<uint32_t>(i);
  uint32_t s = ~0u;
  if (picked(pick, e)) {
    s = pick[e];
  } else {
    int n = 0;
    const bool whole = each_root(faces, heads, mask, next, corner_of(faces, e, 1),
                                 [&](uint32_t o) {
                                   if (picked(pick, o)) return;
                                   ++n;
                                   s = o;
                                 });
    if (!whole || n != 1) s = ~0u;
  }
  succ[e] = s;
}

// Per leaf: the groups it leads, their edges and their triangles (Counts); and
// per side how many edges the group it leads has (0: leads none). A loop's leader
// is its side of the smallest number. As many root edges enter a point as leave it,
// so a loop is left and entered at one place each.
__global__ void exact_loops_kernel(const uint32_t* __restrict__ partner,
                                   const uint32_t* __restrict__ succ, int64_t nedge,
                                   uint8_t* __restrict__ lead,
                                   Counts* __restrict__ counts, Info* info) {
  if (too_open(info, nedge)) return;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint32_t e = static_cast<uint32_t>(i);
  int count = 0;
  if (i < nedge && partner[e] == kNoPartner) {
    uint32_t s = e;
    bool smallest = true;
    for (int k = 1; k <= kMaxLoop; ++k) {
      s = succ[s];
      if (s == ~0u) break;
      if (s == e) {
        count = k;
        break;
      }
      smallest = smallest && e < s;
    }
    if (count < 3) count = 1;
    else if (!smallest) count = 0;
    if (count) {
      Counts* c = counts + e / kLeafEdges;
      atomicAdd(&c->groups, 1);
      atomicAdd(&c->edges, count);
      if (count > 1) atomicAdd(&c->triangles, count - 2);
    }
  }
  if (i < nedge) lead[e] = static_cast<uint8_t>(count);
  const int edges = __reduce_add_sync(~0u, count);
  const int items = __reduce_add_sync(~0u, count > 1 ? count - 2 : count);
  if ((threadIdx.x & 31) == 0 && edges) {
    atomicAdd(&info->nroot, edges);
    atomicAdd(&info->nitem, items);
  }
}

// ---- tree ----------------------------------------------------------------------

__constant__ const int kSym[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};

__device__ __forceinline__ void finish_node(const Moments& m, float r, NodeEval* out) {
  NodeEval e;
  for (int x = 0; x < 3; ++x) {
    e.ph[x] = static_cast<float>(m.p[x]);
    e.pl[x] = static_cast<float>(m.p[x] - static_cast<double>(e.ph[x]));
  }
  e.r = r;
  const double rd = r;
  const double n2 = r > 0.0f ? 1.0 / (2.0 * kTwoPi * rd * rd) : 0.0;
  const double n3 = r > 0.0f ? n2 / rd : 0.0, n4 = r > 0.0f ? n3 / rd : 0.0;
  double l[3], c[10] = {};
  for (int i = 0; i < 3; ++i) {
    double u = 0.0, v = 0.0;
    for (int j = 0; j < 3; ++j) {
      u += m.m2[kSym[j][i]][j];
      v += m.m2[kSym[j][j]][i];
    }
    l[i] = -3.0 * (2.0 * u + v);
  }
  // 15 sum M2_jki y_i y_j y_k by monomial: 000 111 222 001 002 011 022 112 122 012
  const int slot[3][3][3] = {{{0, 3, 4}, {3, 5, 9}, {4, 9, 6}},
                             {{3, 5, 9}, {5, 1, 7}, {9, 7, 8}},
                             {{4, 9, 6}, {9, 7, 8}, {6, 8, 2}}};
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j)
      for (int k = 0; k < 3; ++k) c[slot[i][j][k]] += 15.0 * m.m2[kSym[j][k]][i];
  const double tr = m.m1[0][0] + m.m1[1][1] + m.m1[2][2];
  const double q22 = -3.0 * m.m1[2][2];
  for (int i = 0; i < 3; ++i) e.t0[i] = static_cast<float>(n2 * m.m0[i]);
  e.qc = static_cast<float>(n3 * (tr + q22));
  e.q00 = static_cast<float>(n3 * (-3.0 * m.m1[0][0] - q22));
  e.q11 = static_cast<float>(n3 * (-3.0 * m.m1[1][1] - q22));
  e.q01 = static_cast<float>(n3 * -3.0 * (m.m1[0][1] + m.m1[1][0]));
  e.q02 = static_cast<float>(n3 * -3.0 * (m.m1[0][2] + m.m1[2][0]));
  e.q12 = static_cast<float>(n3 * -3.0 * (m.m1[1][2] + m.m1[2][1]));
  e.l[0] = static_cast<float>(n4 * (l[0] + c[6]));
  e.l[1] = static_cast<float>(n4 * (l[1] + c[8]));
  e.l[2] = static_cast<float>(n4 * (l[2] + c[2]));
  e.c000 = static_cast<float>(n4 * (c[0] - c[6]));
  e.c011 = static_cast<float>(n4 * (c[5] - c[6]));
  e.c001 = static_cast<float>(n4 * (c[3] - c[8]));
  e.c111 = static_cast<float>(n4 * (c[1] - c[8]));
  e.c002 = static_cast<float>(n4 * (c[4] - c[2]));
  e.c112 = static_cast<float>(n4 * (c[7] - c[2]));
  e.c012 = static_cast<float>(n4 * c[9]);
  e.pad[0] = e.pad[1] = 0.0f;
  *out = e;
}

__device__ __forceinline__ float node_area(const Moments& m, float r) {
  return r > 0.0f ? __double2float_ru(m.area / (2.0 * kTwoPi * static_cast<double>(r) *
                                                 static_cast<double>(r)))
                  : 0.0f;
}

// One thread per leaf: near box, centre, moments and the FP32 faces.
__global__ void __launch_bounds__(64) exact_leaf_kernel(
    const Face64* __restrict__ faces, int64_t nf, int64_t nleaf, const Info* __restrict__ info,
    Moments* __restrict__ moments, NodeTest* __restrict__ test, Face32* __restrict__ faces32) {
  const int64_t leaf = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (leaf >= nleaf) return;
  const Frame f = frame_of(info);
  const int64_t f0 = leaf * kLeaf;
  const int n = static_cast<int>(min(static_cast<int64_t>(kLeaf), nf - f0));
  Moments m = {};
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  double mean[3] = {0, 0, 0};
  for (int k = 0; k < n; ++k) {
    const double* src = faces[f0 + k].v;
    double v[9];
    for (int r = 0; r < 9; ++r) {
      v[r] = (src[r] - f.c[r % 3]) * f.s;
      lo[r % 3] = fmin(lo[r % 3], v[r]);
      hi[r % 3] = fmax(hi[r % 3], v[r]);
    }
    const double e1[3] = {v[3] - v[0], v[4] - v[1], v[5] - v[2]};
    const double e2[3] = {v[6] - v[0], v[7] - v[1], v[8] - v[2]};
    const double nx = e1[1] * e2[2] - e1[2] * e2[1], ny = e1[2] * e2[0] - e1[0] * e2[2],
                 nz = e1[0] * e2[1] - e1[1] * e2[0];
    const double a = 0.5 * sqrt(nx * nx + ny * ny + nz * nz);
    m.area += a;
    for (int x = 0; x < 3; ++x) {
      const double c = (v[x] + v[3 + x] + v[6 + x]) * (1.0 / 3.0);
      m.p[x] += a * c;
      mean[x] += c;
    }
  }
  float centre[8] = {};
  for (int x = 0; x < 3; ++x) {
    m.p[x] = m.area > 0.0 ? m.p[x] / m.area : mean[x] / n;
    m.p[x] = fmin(fmax(m.p[x], lo[x]), hi[x]);
    centre[x] = static_cast<float>(m.p[x]);
    centre[3 + x] = static_cast<float>(m.p[x] - static_cast<double>(centre[x]));
  }
  for (int k = 0; k < kLeaf; ++k) {
    double v[9] = {};
    if (k < n) {
      const double* src = faces[f0 + k].v;
      for (int r = 0; r < 9; ++r) v[r] = (src[r] - f.c[r % 3]) * f.s - m.p[r % 3];
    }
    double an[3], c[3];
    const double e1[3] = {v[3] - v[0], v[4] - v[1], v[5] - v[2]};
    const double e2[3] = {v[6] - v[0], v[7] - v[1], v[8] - v[2]};
    an[0] = 0.5 * (e1[1] * e2[2] - e1[2] * e2[1]);
    an[1] = 0.5 * (e1[2] * e2[0] - e1[0] * e2[2]);
    an[2] = 0.5 * (e1[0] * e2[1] - e1[1] * e2[0]);
    // Padding faces are points at the centre: their pair term is real.
    float4* dst = reinterpret_cast<float4*>(faces32 + f0 + k);
    auto fl = [](double x) { return static_cast<float>(x); };
    dst[0] = make_float4(fl(v[0]), fl(v[1]), fl(v[2]), fl(e1[0]));
    dst[1] = make_float4(fl(e1[1]), fl(e1[2]), fl(e2[0]), fl(e2[1]));
    dst[2] = make_float4(fl(e2[2]), fl(2.0 * an[0]), fl(2.0 * an[1]), fl(2.0 * an[2]));
    dst[3] = make_float4(fl(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]),
                         fl(e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2]),
                         fl(e1[0] * e2[0] + e1[1] * e2[1] + e1[2] * e2[2]), centre[k]);
    if (k >= n) continue;
    for (int x = 0; x < 3; ++x) c[x] = (v[x] + v[3 + x] + v[6 + x]) * (1.0 / 3.0);
    for (int i = 0; i < 3; ++i) {
      m.m0[i] += an[i];
      for (int j = 0; j < 3; ++j) m.m1[j][i] += an[i] * c[j];
    }
    for (int j = 0; j < 3; ++j)
      for (int k2 = j; k2 < 3; ++k2) {
        double s2 = c[j] * c[k2];
        for (int s = 0; s < 3; ++s)
          s2 += (v[3 * s + j] - c[j]) * (v[3 * s + k2] - c[k2]) * (1.0 / 12.0);
        for (int i = 0; i < 3; ++i) m.m2[kSym[j][k2]][i] += 0.5 * an[i] * s2;
      }
  }
  const double dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
  const double pad = static_cast<double>(kPad) * sqrt(dx * dx + dy * dy + dz * dz) +
                     static_cast<double>(kPadAbs);
  NodeTest t;
  for (int x = 0; x < 3; ++x) {
    t.lo[x] = __double2float_rd(lo[x] - pad);
    t.hi[x] = __double2float_ru(hi[x] + pad);
    t.p[x] = static_cast<float>(m.p[x]);
  }
  t.r = 0.0f;  // exact_radius_kernel
  t.area = 0.0f;
  t.child = -1;
  test[leaf] = t;
  moments[leaf] = m;
}

// A node from its children, by one warp: areas and boxes unite, moments shift to the
// common centre. A lane takes a component (a thread per node took the whole
// chain of loads alone: 83 us for the last six levels of a 20,480-face mesh).
__device__ __forceinline__ void merge_node(int64_t first, int count, Moments* moments,
                                           NodeTest* test, int64_t node) {
  const int lane = threadIdx.x & 31;
  double area = 0.0, p[3] = {0, 0, 0}, mean[3] = {0, 0, 0};
  for (int k = 0; k < count; ++k) {
    const Moments& c = moments[first + k];
    area += c.area;
    for (int x = 0; x < 3; ++x) {
      p[x] += c.area * c.p[x];
      mean[x] += c.p[x];
    }
  }
  for (int x = 0; x < 3; ++x) p[x] = area > 0.0 ? p[x] / area : mean[x] / count;
  Moments& out = moments[node];
  if (lane < 3) {  // m0
    double v = 0.0;
    for (int k = 0; k < count; ++k) v += moments[first + k].m0[lane];
    out.m0[lane] = v;
    out.p[lane] = p[lane];
    if (lane == 0) out.area = area;
  } else if (lane < 12) {  // m1[j][i]
    const int j = (lane - 3) / 3, i = (lane - 3) % 3;
    double v = 0.0;
    for (int k = 0; k < count; ++k) {
      const Moments& c = moments[first + k];
      v += c.m1[j][i] + (c.p[j] - p[j]) * c.m0[i];
    }
    out.m1[j][i] = v;
  } else if (lane < 30) {  // m2[jk][i]
    const int jk = (lane - 12) / 3, i = (lane - 12) % 3;
    const int j = jk < 3 ? 0 : (jk < 5 ? 1 : 2), l = jk < 3 ? jk : (jk < 5 ? jk - 2 : 2);
    double v = 0.0;
    for (int k = 0; k < count; ++k) {
      const Moments& c = moments[first + k];
      const double sj = c.p[j] - p[j], sl = c.p[l] - p[l];
      v += c.m2[jk][i] + 0.5 * (sj * c.m1[l][i] + sl * c.m1[j][i]) + 0.5 * sj * sl * c.m0[i];
    }
    out.m2[jk][i] = v;
  } else if (lane == 30) {
    NodeTest t;
    for (int x = 0; x < 3; ++x) {
      t.lo[x] = INFINITY;
      t.hi[x] = -INFINITY;
      t.p[x] = static_cast<float>(p[x]);
    }
    for (int k = 0; k < count; ++k)
      for (int x = 0; x < 3; ++x) {
        t.lo[x] = fminf(t.lo[x], test[first + k].lo[x]);
        t.hi[x] = fmaxf(t.hi[x], test[first + k].hi[x]);
      }
    t.r = 0.0f;
    t.area = 0.0f;
    t.child = static_cast<int32_t>(first << 2) | (count - 1);
    test[node] = t;
  }
}

__global__ void __launch_bounds__(128) exact_level_kernel(int64_t child_off, int64_t child_n,
                                                          int64_t off, int64_t n,
                                                          Moments* moments, NodeTest* test) {
  const int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / 32;
  if (i >= n) return;
  const int64_t c0 = i * kExactArity;
  merge_node(child_off + c0, static_cast<int>(min(static_cast<int64_t>(kExactArity), child_n - c0)),
             moments, test, off + i);
}

struct Levels {
  int nlevel;
  int64_t off[kExactMaxLevels], n[kExactMaxLevels];
};
// The few nodes of the top levels, one CTA level by level.
__global__ void __launch_bounds__(1024) exact_top_kernel(const Levels a, int first_level,
                                                         Moments* moments, NodeTest* test) {
  for (int l = first_level; l < a.nlevel; ++l) {
    for (int64_t i = threadIdx.x / 32; i < a.n[l]; i += blockDim.x / 32) {
      const int64_t c0 = i * kExactArity;
      merge_node(a.off[l - 1] + c0,
                 static_cast<int>(min(static_cast<int64_t>(kExactArity), a.n[l - 1] - c0)),
                 moments, test, a.off[l] + i);
    }
    __syncthreads();
  }
}

// Every node's exact radius: the largest distance of its vertices from its centre.
// One warp per 32 faces (four leaves, one node of level 1), a maximum per level; a
// bound from the children's balls is a fifth looser and costs the walk half as many
// nodes again. The radius goes into test[].r as the bits of a positive float.
__global__ void __launch_bounds__(256) exact_radius_kernel(const Face64* __restrict__ faces,
                                                           int64_t nf, const Levels a,
                                                           const Info* __restrict__ info,
                                                           const Moments* __restrict__ moments,
                                                           NodeTest* test) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t base = i & ~int64_t(31);
  if (base >= nf) return;
  const int64_t f = min(i, nf - 1);
  const Frame fr = frame_of(info);
  double v[9];
#pragma unroll
  for (int r = 0; r < 9; ++r) v[r] = (faces[f].v[r] - fr.c[r % 3]) * fr.s;
  int64_t node = f / kLeaf;
  for (int l = 0; l < a.nlevel; ++l) {
    const Moments& m = moments[a.off[l] + node];
    double r2 = 0.0;
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const double x = v[3 * s] - m.p[0], y = v[3 * s + 1] - m.p[1], z = v[3 * s + 2] - m.p[2];
      r2 = fmax(r2, x * x + y * y + z * z);
    }
    float r = __double2float_ru(sqrt(r2) * (1.0 + 1e-12));
    for (int o = l == 0 ? 4 : 16; o; o >>= 1) r = fmaxf(r, __shfl_xor_sync(~0u, r, o));
    if ((threadIdx.x & (l == 0 ? 7 : 31)) == 0)
      atomicMax(reinterpret_cast<int*>(&test[a.off[l] + node].r), __float_as_int(r));
    node /= kExactArity;
  }
}

__global__ void __launch_bounds__(64) exact_finish_kernel(int64_t nnode,
                                                          const Moments* __restrict__ moments,
                                                          NodeTest* test, NodeEval* eval) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= nnode) return;
  const float r = test[i].r;
  test[i].area = node_area(moments[i], r);
  finish_node(moments[i], r, eval + i);
}

// The groups, a thread per side: what a leaf's sides lead lies behind each other in side
// order, from `first` (the exclusive sum of the leaves' counts).
__global__ void exact_groups_kernel(const Face64* __restrict__ faces, int64_t nedge, int64_t nleaf,
                                    const uint32_t* __restrict__ succ,
                                    const uint8_t* __restrict__ lead,
                                    const Counts* __restrict__ counts,
                                    const Counts* __restrict__ first, int64_t max_roots,
                                    const NodeTest* __restrict__ test, Group* __restrict__ groups,
                                    Root* __restrict__ roots, int32_t* __restrict__ root_leaf,
                                    Triangle* __restrict__ triangles, Info* info) {
  const int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e == 0) info->ngroup = first[nleaf - 1].groups + counts[nleaf - 1].groups;
  if (e >= nedge) return;
  const int count = lead[e];
  if (count == 0) return;
  const int64_t leaf = e / kLeafEdges;
  Counts at = first[leaf];
  for (int64_t o = leaf * kLeafEdges; o < e; ++o) {
    const int c = lead[o];
    if (c == 0) continue;
    ++at.groups;
    at.edges += c;
    at.triangles += c > 1 ? c - 2 : 0;
  }
  if (at.edges + count > max_roots) return;  // more than that: the result is not used
  Group g;
  for (int x = 0; x < 3; ++x) {
    g.lo[x] = INFINITY;
    g.hi[x] = -INFINITY;
  }
  g.first = at.edges;
  g.count = count;
  g.triangle = at.triangles;
  g.pad[0] = g.pad[1] = g.pad[2] = 0;
  uint32_t s = static_cast<uint32_t>(e);
  double a[3] = {0.0, 0.0, 0.0};
  for (int k = 0; k < count; ++k) {
    const double *u = corner_of(faces, s, 0), *v = corner_of(faces, s, 1);
    const uint32_t l = s / kLeafEdges;
    for (int x = 0; x < 3; ++x) {
      roots[at.edges + k].u[x] = u[x];
      roots[at.edges + k].v[x] = v[x];
      g.lo[x] = fminf(g.lo[x], test[l].lo[x]);
      g.hi[x] = fmaxf(g.hi[x], test[l].hi[x]);
    }
    root_leaf[at.edges + k] = static_cast<int32_t>(l);
    if (k == 0) {
      for (int x = 0; x < 3; ++x) a[x] = u[x];
    } else if (k + 1 < count) {
      // Triangle k of the fan: the loop's first vertex and this edge.
      Triangle t;
      for (int x = 0; x < 3; ++x) {
        t.a[x] = a[x];
        t.e1[x] = u[x] - a[x];
        t.e2[x] = v[x] - a[x];
      }
      t.n[0] = t.e1[1] * t.e2[2] - t.e1[2] * t.e2[1];
      t.n[1] = t.e1[2] * t.e2[0] - t.e1[0] * t.e2[2];
      t.n[2] = t.e1[0] * t.e2[1] - t.e1[1] * t.e2[0];
      t.e11 = t.e1[0] * t.e1[0] + t.e1[1] * t.e1[1] + t.e1[2] * t.e1[2];
      t.e22 = t.e2[0] * t.e2[0] + t.e2[1] * t.e2[1] + t.e2[2] * t.e2[2];
      t.e12 = t.e1[0] * t.e2[0] + t.e1[1] * t.e2[1] + t.e1[2] * t.e2[2];
      t.pad = 0.0;
      triangles[at.triangles + k - 1] = t;
    }
    if (k + 1 < count) s = succ[s];
  }
  groups[at.groups] = g;
}

// ---- evaluation ------------------------------------------------------------------

struct EvalArgs {
  const Face64* faces;
  const Face32* faces32;
  const int32_t* nb;
  const NodeTest* test;
  const NodeEval* eval;
  const Group* groups;
  const Root* roots;
  const int32_t* root_leaf;
  const Triangle* triangles;
  const double* q;
  const uint32_t* perm;
  double* w;
  uint32_t* list;
  Info* info;
  int64_t nf, nq, top;  // top: the root node
  bool mixed;           // stands in for the mixed kernel
};

struct WarpBox {
  float lo[3], hi[3];
};

__device__ __forceinline__ NodeTest load_test(const NodeTest* t) {
  const float4* s = reinterpret_cast<const float4*>(t);
  const float4 a = __ldg(s), b = __ldg(s + 1), c = __ldg(s + 2);
  NodeTest o;
  o.lo[0] = a.x; o.lo[1] = a.y; o.lo[2] = a.z; o.hi[0] = a.w;
  o.hi[1] = b.x; o.hi[2] = b.y; o.p[0] = b.z; o.p[1] = b.w;
  o.p[2] = c.x; o.r = c.y; o.area = c.z; o.child = __float_as_int(c.w);
  return o;
}

// Whether the near box of a node meets the warp's box. For a leaf this IS the
// definition of near; an ancestor's box holds its leaves' boxes, so a near leaf is
// always reached, and a neighbour may be tested on its own.
__device__ __forceinline__ bool meets(const float lo[3], const float hi[3], const WarpBox& b) {
  return lo[0] <= b.hi[0] && hi[0] >= b.lo[0] && lo[1] <= b.hi[1] && hi[1] >= b.lo[1] &&
         lo[2] <= b.hi[2] && hi[2] >= b.lo[2];
}
// `t` starts with a box (a leaf's NodeTest or a Group).
__device__ __forceinline__ bool box_near(const void* t, const WarpBox& b) {
  const float4* s = reinterpret_cast<const float4*>(t);
  const float4 u = __ldg(s);
  const float2 v = __ldg(reinterpret_cast<const float2*>(s + 1));
  const float lo[3] = {u.x, u.y, u.z}, hi[3] = {u.w, v.x, v.y};
  return meets(lo, hi, b);
}

__device__ __forceinline__ float rsq(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// A node's expansion (in shared memory) at the query (float pairs qh + ql), in units
// of W.
__device__ __forceinline__ float far_value(const float4* s, const float qh[3],
                                           const float ql[3]) {
  const float4 a = s[0], b = s[1], c = s[2], d = s[3], e = s[4], f = s[5], g = s[6];
  // a: ph r | b: pl t0.x | c: t0.yz qc q00 | d: q11 q01 q02 q12 | e: l c000
  // f: c111 c001 c011 c002 | g: c112 c012
  float x = (a.x - qh[0]) + (b.x - ql[0]);
  float y = (a.y - qh[1]) + (b.y - ql[1]);
  float z = (a.z - qh[2]) + (b.z - ql[2]);
  const float inv = rsq(x * x + y * y + z * z);
  x *= inv;
  y *= inv;
  z *= inv;
  const float t = a.w * inv;
  const float xx = x * x, yy = y * y, xy = x * y;
  const float lin = b.w * x + c.x * y + c.y * z;
  const float quad = c.z + c.w * xx + d.x * yy + d.y * xy + z * (d.z * x + d.w * y);
  const float cub = x * (e.x + e.w * xx + f.z * yy) + y * (e.y + f.x * yy + f.y * xx) +
                    z * (e.z + f.w * xx + g.x * yy + g.y * xy);
  return t * t * (lin + t * (quad + t * cub));
}

// FP32 sum of the solid angles of every SUB-th face (from `sub`) of a leaf that is
// neither near nor far (its 512 bytes in shared memory), in units of W: the running
// product of the pairs' unit-scaled complex terms with turns counted (the sign rule
// of wn_pair.cuh), one atan2f.
template <int SUB>
__device__ __forceinline__ float mid_value(const float4* s, int sub, const float qh[3],
                                           const float ql[3]) {
  const float px = (s[3].w - qh[0]) + (s[15].w - ql[0]);
  const float py = (s[7].w - qh[1]) + (s[19].w - ql[1]);
  const float pz = (s[11].w - qh[2]) + (s[23].w - ql[2]);
  float zr = 1.0f, zi = 0.0f;
  int turns = 0;
#pragma unroll
  for (int j = 0; j < kLeaf / SUB; ++j) {
    const float4* r = s + 4 * (j * SUB + sub);
    const float4 f0 = r[0], f1 = r[1], f2 = r[2], f3 = r[3];
    const float ax = f0.x + px, ay = f0.y + py, az = f0.z + pz;
    const float aa = ax * ax + ay * ay + az * az;
    const float a1 = ax * f0.w + ay * f1.x + az * f1.y;
    const float a2 = ax * f1.z + ay * f1.w + az * f2.x;
    const float an = ax * f2.y + ay * f2.z + az * f2.w;
    const float ab = aa + a1, ac = aa + a2, bc = ab + a2 + f3.z;
    const float ra = rsq(aa), rb = rsq(ab + a1 + f3.x), rc = rsq(ac + a2 + f3.y);
    const float rab = ra * rb;
    const float re = 1.0f + ab * rab + bc * (rb * rc) + ac * (rc * ra);
    const float im = an * (rab * rc);
    const float nr = zr * re - zi * im, ni = zr * im + zi * re;
    const bool s0 = signbit(zi), st = signbit(im), s1 = signbit(ni);
    turns += (s0 == st && s0 != s1) ? (s0 ? -1 : 1) : 0;
    zr = nr;
    zi = ni;
  }
  return atan2f(zi, zr) * static_cast<float>(1.0 / kTwoPi) + static_cast<float>(turns);
}

// Running product of the boundary's z; `cond` keeps the smallest exponent seen.
struct EdgeProduct {
  double re, im;
  int cond;
};
__device__ __forceinline__ void multiply(EdgeProduct& p, double re, double im) {
  const int m = max(__double2hiint(re) & 0x7fffffff, __double2hiint(im) & 0x7fffffff);
  p.cond = min(p.cond, m < 0x7ff00000 ? m : 0);
  const double t = p.re * re - p.im * im;
  p.im = p.re * im + p.im * re;
  p.re = t;
}
// |z| lies in [2^-7, 4.01] while `cond` holds, so 64 factors move the product by at
// most 2^448.
__device__ __forceinline__ void rescale(EdgeProduct& p) {
  const int e = max(__double2hiint(p.re) & 0x7ff00000, __double2hiint(p.im) & 0x7ff00000);
  if (e == 0 || e == 0x7ff00000) p.cond = 0;
  const double f = __hiloint2double(0x7fe00000 - e, 0);
  p.re *= f;
  p.im *= f;
}

struct Dir {
  double x, y, z, sx, sy;  // unit direction; x/z and y/z
};
__device__ __forceinline__ Dir direction(int k) {
  // Four directions in general position (no axis, no diagonal of a grid):
  // permutations and signs of (2, 3, 4) / sqrt(29).
  const double a = 0.37139067635410372, b = 0.55708601453115558, c = 0.74278135270820744;
  const double x = k == 0 ? a : (k == 1 ? -c : (k == 2 ? b : -a));
  const double y = k == 0 ? b : (k == 1 ? a : (k == 2 ? -a : -c));
  const double z = k == 0 ? c : (k == 1 ? b : (k == 2 ? -c : -b));
  return Dir{x, y, z, x / z, y / z};
}

// Multiplies in the infinite triangle (u, v, D).
__device__ __forceinline__ void push_edge(EdgeProduct& p, const Dir& D, double qx, double qy,
                                          double qz, double ux, double uy, double uz, double vx,
                                          double vy, double vz) {
  ux -= qx; uy -= qy; uz -= qz;
  vx -= qx; vy -= qy; vz -= qz;
  const double ru = rsqrt64(ux * ux + uy * uy + uz * uz);
  const double rv = rsqrt64(vx * vx + vy * vy + vz * vz);
  const double s = ru * rv;
  const double uv = ux * vx + uy * vy + uz * vz;
  const double du = D.x * ux + D.y * uy + D.z * uz, dv = D.x * vx + D.y * vy + D.z * vz;
  // D.(u x v) = D.z times the cross product of u and v sheared along D to z = 0.
  const double px = ux - D.sx * uz, py = uy - D.sy * uz;
  const double wx = vx - D.sx * vz, wy = vy - D.sy * vz;
  multiply(p, 1.0 + uv * s + du * ru + dv * rv, (px * wy - py * wx) * (s * D.z));
}

// Multiplies in the pair term of a fan triangle, scaled by its lengths.
__device__ __forceinline__ void push_triangle(EdgeProduct& p, double qx, double qy, double qz,
                                              const Triangle* t) {
  const double2* s = reinterpret_cast<const double2*>(t);
  const double2 s0 = s[0], s1 = s[1], s2 = s[2], s3 = s[3], s4 = s[4], s5 = s[5], s6 = s[6];
  const double e12 = t->e12;
  const double ax = s0.x - qx, ay = s0.y - qy, az = s1.x - qz;
  const double aa = ax * ax + ay * ay + az * az;
  const double a1 = ax * s1.y + ay * s2.x + az * s2.y;
  const double a2 = ax * s3.x + ay * s3.y + az * s4.x;
  const double an = ax * s4.y + ay * s5.x + az * s5.y;
  const double ab = aa + a1, ac = aa + a2;
  const double ra = rsqrt64(aa), rb = rsqrt64(ab + a1 + s6.x), rc = rsqrt64(ac + a2 + s6.y);
  const double rab = ra * rb;
  multiply(p, 1.0 + ab * rab + (ab + a2 + e12) * (rb * rc) + ac * (rc * ra), an * (rab * rc));
}

enum WalkMode : int { kWalkFar = 1, kWalkNear = 2, kWalkEdges = 4 };

constexpr int kStage = 32 * 8;  // 16-byte words: 32 triangles or expansions, a leaf's faces

struct WarpMem {
  float4 stage[kStage];
  uint32_t stack[kStack];
  uint32_t farl[64], midl[64];
  uint8_t emit[32];
};

__device__ __forceinline__ bool at_infinity(double x, double y, double z) {
  return !isnan(x) && !isnan(y) && !isnan(z) && (isinf(x) || isinf(y) || isinf(z));
}

__global__ void exact_infinite_kernel(const double* __restrict__ q, int64_t nq,
                                      double* __restrict__ w) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < nq && at_infinity(q[3 * i], q[3 * i + 1], q[3 * i + 2])) w[i] = 0.0;
}

// One warp per 32 / SUB consecutive queries of the Hilbert order, SUB lanes to a
// query. The walk is the warp's: its lanes test 32 nodes at a time against the box
// of its queries, and what is accepted goes through shared memory, 32 expansions or
// one leaf at a time, to all lanes, which share a query's items among them. More
// lanes per query make the box, and with it the lists, smaller, at less work per
// read: the launch chooses by the queries' spacing.
//
// 327,680 faces x 2^20 queries: a warp of 16 queries takes ~550 expansions, ~48 leaves
// in FP32, ~10 near leaves and ~60 edges in place of 327,680 faces; 4.6 ms with the
// preparation, where the all-pairs kernels take 410 (mixed) and 1,884 (FP64). 18,842
// faces with 1,638 holes x 2^20 queries: ~1,607 fan triangles a query, 9.2 ms against
// 108 (FP64 pairs). Bound by FP64 and latency there (ncu, 131,072 queries: FP64 pipe
// 44 %, issue 49 %). Reading each expansion's seven words with every lane instead of
// staging 32 of them cost 11.6 against 6.4 ms. Four CTAs per SM of 128 registers: with
// five of 96 spills cost 5.7 against 5.4 ms, with six of 80 6.3. kPad: 0.2 / 0.1 / 0.05 /
// 0.03 of the diagonal 6.1 / 5.7 / 5.5 / 5.4 ms, at the price of nearer FP32 leaves; kBeta
// 2.25 / 2.5 / 2.75 7.3 / 5.7 / 5.3 ms (too many second walks below), with kMaxBound 0.45
// in place of 0.4 5.1 at 2.5; 18,842 faces prefer the smaller kBeta (9.5 / 9.8 / 10.0).
template <int SUB>
__global__ void __launch_bounds__(32 * kWarps, 4) exact_eval_kernel(const EvalArgs a) {
  __shared__ WarpMem mem[kWarps];
  constexpr int kQueries = 32 / SUB;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % SUB;
  WarpMem& m = mem[warp];
  const int64_t base = (static_cast<int64_t>(blockIdx.x) * kWarps + warp) * kQueries;
  if (base >= a.nq) return;
  const int64_t at = base + lane / SUB;
  const bool valid = at < a.nq;
  const uint32_t qi = a.perm[valid ? at : a.nq - 1];
  const double qx = a.q[3 * static_cast<int64_t>(qi)], qy = a.q[3 * static_cast<int64_t>(qi) + 1],
               qz = a.q[3 * static_cast<int64_t>(qi) + 2];
  bool failed = false;
  float qh[3], ql[3];
  WarpBox box;
  {
    const Frame f = frame_of(a.info);
    const double p[3] = {(qx - f.c[0]) * f.s, (qy - f.c[1]) * f.s, (qz - f.c[2]) * f.s};
    failed = !(fabs(p[0]) < kFarQuery && fabs(p[1]) < kFarQuery && fabs(p[2]) < kFarQuery);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const double v = failed ? 0.0 : p[x];
      qh[x] = static_cast<float>(v);
      ql[x] = static_cast<float>(v - static_cast<double>(qh[x]));
      float l = failed ? INFINITY : __double2float_rd(v), h = failed ? -INFINITY : __double2float_ru(v);
      for (int o = 16; o; o >>= 1) {
        l = fminf(l, __shfl_xor_sync(~0u, l, o));
        h = fmaxf(h, __shfl_xor_sync(~0u, h, o));
      }
      box.lo[x] = l;
      box.hi[x] = h;
    }
  }
  ArgAcc acc;
  argacc_init(acc);
  EdgeProduct fans{1.0, 0.0, 0x7fffffff};  // loops of the mesh's boundary: the same for every D
  float wfar = 0.0f, bound = 0.0f;
  bool bounded = false, settled = false;  // W_far accurate enough; boundary product usable
  double argument = 0.0;
  int dir = 0, beta_try = 0;
  float beta = kBeta;
  int mode = kWalkFar | kWalkNear | kWalkEdges;
  bool overflow = false;
  // At most kBetaTries + kDirTries walks (uniform over the warp).
  for (int round = 0; round < kBetaTries + kDirTries && mode; ++round) {
    const Dir D = direction(dir);
    EdgeProduct prod{1.0, 0.0, 0x7fffffff};
    if (mode & kWalkFar) wfar = bound = 0.0f;
    int nfar = 0, nmid = 0, sp = 1;
    if (lane == 0) m.stack[0] = static_cast<uint32_t>(a.top);
    __syncwarp();
    while (sp > 0) {
      const int n = min(sp, 32);
      const uint32_t id = lane < n ? m.stack[sp - 1 - lane] : ~0u;
      sp -= n;
      __syncwarp();
      bool is_far = false, is_mid = false, is_near = false, open = false;
      int32_t child = -1;
      if (id != ~0u) {
        const NodeTest t = load_test(a.test + id);
        child = t.child;
        if (meets(t.lo, t.hi, box)) {
          is_near = child < 0;
          open = child >= 0;
        } else if (mode & kWalkFar) {
          const float dx = fmaxf(fmaxf(box.lo[0] - t.p[0], t.p[0] - box.hi[0]), 0.0f);
          const float dy = fmaxf(fmaxf(box.lo[1] - t.p[1], t.p[1] - box.hi[1]), 0.0f);
          const float dz = fmaxf(fmaxf(box.lo[2] - t.p[2], t.p[2] - box.hi[2]), 0.0f);
          const float d = sqrtf(dx * dx + dy * dy + dz * dz) - kSlack;
          if (d > beta * t.r) {
            is_far = true;
            const float rho = t.r / d;
            bound += t.area * rho * rho * (rho * rho * rho * (4.0f - 3.0f * rho) /
                                           ((1.0f - rho) * (1.0f - rho)) + 1e-5f);
          } else {
            is_mid = child < 0;
            open = child >= 0;
            if (is_mid) bound += 2e-5f;
          }
        }
      }
      const unsigned below = (1u << lane) - 1u;
      const unsigned mopen = __ballot_sync(~0u, open);
      if (mopen) {
        if (sp + 4 * __popc(mopen) > kStack) {
          overflow = true;
          break;
        }
        if (open) {
          const int to = sp + 4 * __popc(mopen & below);
          const uint32_t first = static_cast<uint32_t>(child) >> 2;
          const int cnt = (child & 3) + 1;
#pragma unroll
          for (int k = 0; k < 4; ++k) m.stack[to + k] = k < cnt ? first + k : ~0u;
        }
        sp += 4 * __popc(mopen);
      }
      const unsigned mfar = __ballot_sync(~0u, is_far), mmid = __ballot_sync(~0u, is_mid);
      if (is_far) m.farl[nfar + __popc(mfar & below)] = id;
      if (is_mid) m.midl[nmid + __popc(mmid & below)] = id;
      nfar += __popc(mfar);
      nmid += __popc(mmid);
      __syncwarp();
      unsigned mnear = __ballot_sync(~0u, is_near);
      if (mode & kWalkEdges) {
        while (mnear) {
          const uint32_t leaf = __shfl_sync(~0u, id, __ffs(mnear) - 1);
          mnear &= mnear - 1;
          const int nface =
              static_cast<int>(min(static_cast<int64_t>(kLeaf), a.nf - static_cast<int64_t>(leaf) * kLeaf));
          const Face64* f = a.faces + static_cast<int64_t>(leaf) * kLeaf;
          if (mode & kWalkNear) {
#pragma unroll 1
            for (int k = sub; k < nface; k += SUB) {
              const double2* s = reinterpret_cast<const double2*>(f + k);
              const double2 s0 = __ldg(s), s1 = __ldg(s + 1), s2 = __ldg(s + 2), s3 = __ldg(s + 3);
              const double s4 = __ldg(&f[k].v[8]);
              const double v[9] = {s0.x, s0.y, s1.x, s1.y, s2.x, s2.y, s3.x, s3.y, s4};
              push_one(acc, qx, qy, qz, v);
            }
          }
          // The sides towards leaves that are not near, reversed.
          bool emit = false;
          if (lane < 3 * nface) {
            const int32_t o = __ldg(a.nb + static_cast<int64_t>(leaf) * kLeafEdges + lane);
            emit = o >= 0 && !box_near(a.test + o, box);
          }
          const unsigned todo = __ballot_sync(~0u, emit);
          if (emit) m.emit[__popc(todo & below)] = static_cast<uint8_t>(lane);
          __syncwarp();
          const int nemit = __popc(todo);
#pragma unroll 1
          for (int k = sub; k < nemit; k += SUB) {
            const int e = m.emit[k], c = e % 3;
            const double* u = f[e / 3].v + 3 * c;
            const double* v = f[e / 3].v + (c == 2 ? 0 : 3 * c + 3);
            push_edge(prod, D, qx, qy, qz, __ldg(v), __ldg(v + 1), __ldg(v + 2), __ldg(u),
                      __ldg(u + 1), __ldg(u + 2));
          }
          rescale(prod);
          __syncwarp();
        }
      }
      while (nfar >= 32 || (sp == 0 && nfar > 0)) {
        const int cnt = min(nfar, 32);
        nfar -= cnt;
        if (lane < cnt) {
          const float4* src = reinterpret_cast<const float4*>(a.eval + m.farl[nfar + lane]);
#pragma unroll
          for (int k = 0; k < 7; ++k) m.stage[7 * lane + k] = __ldg(src + k);
        }
        __syncwarp();
#pragma unroll 2
        for (int k = sub; k < cnt; k += SUB) wfar += far_value(m.stage + 7 * k, qh, ql);
        __syncwarp();
      }
      if (nmid > 32 || (sp == 0 && nmid > 0)) {
        const float4* src = reinterpret_cast<const float4*>(a.faces32);
        float4 ahead = __ldg(src + static_cast<int64_t>(m.midl[0]) * 32 + lane);
        for (int k = 0; k < nmid; ++k) {
          m.stage[lane] = ahead;
          __syncwarp();
          if (k + 1 < nmid) ahead = __ldg(src + static_cast<int64_t>(m.midl[k + 1]) * 32 + lane);
          wfar += mid_value<SUB>(m.stage, sub, qh, ql);
          __syncwarp();
        }
        nmid = 0;
      }
    }
    if (overflow) break;
    if (mode & kWalkFar) {
      for (int o = 16; o; o >>= 1) bound += __shfl_xor_sync(~0u, bound, o);
      bounded = bound < kMaxBound;
    }
    if (mode & kWalkEdges) {
      // The mesh's own boundary, but for the edges of near leaves: loops away from
      // the near leaves as fans (in the first walk), the others edge by edge.
      const int32_t ngroup = a.info->ngroup;
      for (int32_t g0 = 0; g0 < ngroup; g0 += 32) {
        // A lane's group: as a fan when it is not near; else its edges one by one, but
        // for those of near leaves (bit j of `edges`: edge j).
        int fan = 0, first = 0, triangle = 0;
        unsigned edges = 0;
        if (g0 + lane < ngroup) {
          const Group* g = a.groups + g0 + lane;
          const bool near = box_near(g, box);
          const int2 fc = __ldg(reinterpret_cast<const int2*>(&g->first));
          first = fc.x;
          triangle = __ldg(&g->triangle);
          if (fc.y == 1) {
            edges = near ? 0u : 1u;
          } else if (!near) {
            fan = mode & kWalkNear ? fc.y - 2 : 0;
          } else {
            for (int j = 0; j < fc.y; ++j)
              edges |= box_near(a.test + __ldg(a.root_leaf + first + j), box) ? 0u : 1u << j;
          }
        }
        // Both kinds as lists in shared memory, 64 entries at a time. `mine` places a
        // lane's entries behind those of the lanes before it.
        auto place = [&](int count, int& total) {
          int upto = count;
          for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(~0u, upto, o);
            upto += lane >= o ? v : 0;
          }
          total = __shfl_sync(~0u, upto, 31);
          return upto - count;
        };
        int total = 0;
        int mine = place(fan, total);
        for (int t0 = 0; t0 < total; t0 += 64) {
          for (int k = 0; k < fan; ++k) {
            const int to = mine + k - t0;
            if (to >= 0 && to < 64) m.farl[to] = static_cast<uint32_t>(triangle + k);
          }
          __syncwarp();
          const int n = min(total - t0, 64);
          if constexpr (SUB >= 4) {
            // Few queries to a warp: every lane reads its own.
#pragma unroll 2
            for (int k = sub; k < n; k += SUB)
              push_triangle(fans, qx, qy, qz, a.triangles + m.farl[k]);
            __syncwarp();
          } else {
            // Through shared memory, 32 at a time (read by every lane from L1 they cost
            // 12.3 ms instead of 9.8, 18,842 F with 1,638 holes x 2^20 Q).
            for (int u0 = 0; u0 < n; u0 += 32) {
              const int cnt = min(n - u0, 32);
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const int word = 32 * k + lane;
                if (word / 8 < cnt)
                  m.stage[word] = __ldg(reinterpret_cast<const float4*>(
                                            a.triangles + m.farl[u0 + word / 8]) + word % 8);
              }
              __syncwarp();
#pragma unroll 2
              for (int k = sub; k < cnt; k += SUB)
                push_triangle(fans, qx, qy, qz, reinterpret_cast<const Triangle*>(m.stage) + k);
              __syncwarp();
            }
          }
          rescale(fans);
        }
        mine = place(__popc(edges), total);
        for (int t0 = 0; t0 < total; t0 += 64) {
          unsigned left = edges;
          for (int to = mine - t0; left; ++to, left &= left - 1)
            if (to >= 0 && to < 64) m.farl[to] = static_cast<uint32_t>(first + __ffs(left) - 1);
          __syncwarp();
          const int n = min(total - t0, 64);
#pragma unroll 2
          for (int k = sub; k < n; k += SUB) {
            const double2* s = reinterpret_cast<const double2*>(a.roots + m.farl[k]);
            const double2 s0 = __ldg(s), s1 = __ldg(s + 1), s2 = __ldg(s + 2);
            push_edge(prod, D, qx, qy, qz, s0.x, s0.y, s1.x, s1.y, s2.x, s2.y);
          }
          rescale(prod);
          __syncwarp();
        }
      }
#pragma unroll
      for (int o = 1; o < SUB; o <<= 1) {
        const double re = __shfl_xor_sync(~0u, prod.re, o), im = __shfl_xor_sync(~0u, prod.im, o);
        const int c = __shfl_xor_sync(~0u, prod.cond, o);
        const double t = prod.re * re - prod.im * im;
        prod.im = prod.re * im + prod.im * re;
        prod.re = t;
        prod.cond = min(prod.cond, c);
      }
      if (!settled && prod.cond >= kMinExp) {
        settled = true;
        argument = atan2(prod.im, prod.re);
      }
    }
    mode = 0;
    if (!bounded && ++beta_try < kBetaTries) {
      mode |= kWalkFar;
      beta *= beta_try == 1 ? 1.3f : (beta_try == 2 ? 1.4f : 2.0f);
    }
    if (__any_sync(~0u, !settled && !failed) && ++dir < kDirTries) mode |= kWalkEdges;
  }
  // A query's lanes together.
  double near_angle = atan2(acc.zi, acc.zr) + static_cast<double>(acc.k) * kTwoPi;
  double fan_angle = atan2(fans.im, fans.re);
  bool ok = !acc.bad && fans.cond >= kMinExp;
#pragma unroll
  for (int o = 1; o < SUB; o <<= 1) {
    wfar += __shfl_xor_sync(~0u, wfar, o);
    near_angle += __shfl_xor_sync(~0u, near_angle, o);
    fan_angle += __shfl_xor_sync(~0u, fan_angle, o);
    ok = __shfl_xor_sync(~0u, static_cast<int>(ok), o) && ok;
  }
  if (!valid || sub != 0) return;
  argument += fan_angle;
  const double frac = argument * (1.0 / kTwoPi);
  const double k = rint(static_cast<double>(wfar) - frac);
  const double off = fabs(static_cast<double>(wfar) - frac - k);
  ok = ok && !failed && !overflow && bounded && settled &&
       off <= static_cast<double>(bound) + 0.02;
  if (ok)
    a.w[qi] = (near_angle + argument) / kTwoPi + k;
  else if (isfinite(qx) && isfinite(qy) && isfinite(qz))
    a.list[atomicAdd(&a.info->nlist, 1)] = qi;
  else  // as every pair term is, and the mixed kernel's sum
    a.w[qi] = a.mixed && at_infinity(qx, qy, qz) ? 0.0 : NAN;
}

// All pairs for the listed queries, one CTA per query: per-thread running products
// over the faces, added in thread order.
__global__ void __launch_bounds__(256) exact_fallback_kernel(const Face64* __restrict__ faces,
                                                             int64_t nf,
                                                             const double* __restrict__ q,
                                                             const uint32_t* __restrict__ list,
                                                             const Info* __restrict__ info,
                                                             double* __restrict__ w) {
  __shared__ double part[256];
  const int n = info->nlist;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int64_t qi = list[i];
    const double qx = q[3 * qi], qy = q[3 * qi + 1], qz = q[3 * qi + 2];
    ArgAcc acc;
    argacc_init(acc);
    for (int64_t f = threadIdx.x; f < nf; f += 256) {
      const double* v = faces[f].v;
      double det, denom;
      pair_terms_exact(qx, qy, qz, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], det,
                       denom);
      argacc_push(acc, denom, det);
    }
    double angle = atan2(acc.zi, acc.zr) + static_cast<double>(acc.k) * kTwoPi;
    if (acc.bad) {
      angle = 0.0;
      for (int64_t f = threadIdx.x; f < nf; f += 256) {
        const double* v = faces[f].v;
        double det, denom;
        pair_terms_exact(qx, qy, qz, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], det,
                         denom);
        angle += atan2(det, denom);
      }
    }
    part[threadIdx.x] = angle;
    __syncthreads();
    for (int s = 128; s; s >>= 1) {
      if (threadIdx.x < s) part[threadIdx.x] += part[threadIdx.x + s];
      __syncthreads();
    }
    if (threadIdx.x == 0) w[qi] = part[0] / kTwoPi;
    __syncthreads();
  }
}

unsigned blocks(int64_t n, int threads) {
  return static_cast<unsigned>(std::max<int64_t>(1, (n + threads - 1) / threads));
}

}  // namespace

// Where the method starts to pay (one B200, meshes of 1,280 to 327,680 faces, closed,
// open and terrain grids; ms, the streaming all-pairs kernel -> this one): 1,280 F x
// 131,072 Q 0.88 -> 0.42, 20,480 F x 8,192 Q 0.86 -> 0.43, 19,456 F with holes x 8,192 Q
// 0.85 -> 0.65, 28,322 F (grid) x 8,192 Q 1.16 -> 0.57, 77,824 F with holes x 4,096 Q
// 1.58 -> 1.30; below the line 5,120 F x 8,192 Q 0.24 -> 0.38.
// Fewer queries than 4,096 leave too few warps and wide boxes: 243,602 F (grid) x
// 2,048 Q 2.4 -> 4.1.
bool exact_pays(int64_t nf, int64_t nq) {
  return nf >= 1024 && nf <= (int64_t(1) << 29) && nq >= 4096 && nq <= 0x7fffffffLL &&
         static_cast<double>(nf) * static_cast<double>(nq) >= 1.5e8;
}

// A warp goes over the whole boundary for its queries, which takes about 0.23 us an item
// however few the warps are: with few queries that, and not the work, is what the boundary
// costs. 301,466 F with 26,214 holes x 4,096 Q: 7.3 ms against 6.7 (FP64 streaming) and 4.7
// (mixed), x 8,192 8.5 against 13.4 and 7.7, x 16,384 9.6 against 25 and 11.5; 1,205,862 F
// with 104,858 holes x 4,096 27 against 25 and 12, x 16,384 38 against 99 and 36; 75,366 F
// with 6,554 x 4,096 1.9 against 1.6 and 2.6. So it matters to mixed calls, whose own
// preparation counts too (about 1.5 ms and 5 ns a face; 0.8 and 1 on a faster host, where the
// last of these takes 1.4 ms).
bool boundary_pays(int64_t items, int64_t nf, int64_t nq, bool mixed) {
  const double n = static_cast<double>(items), f = static_cast<double>(nf),
               q = static_cast<double>(nq);
  if (!mixed) return n <= kExactMostFp64 * f;
  return n <= kExactMostMixed * f &&
         n * (0.23e-6 + 4.8e-12 * q) <= 1.5e-3 + 5e-9 * f + 1.5e-12 * f * q;
}

ExactPlan plan_exact(int64_t nf, int64_t nq) {
  ExactPlan p;
  p.nf = nf;
  p.nq = nq;
  p.nleaf = (nf + kLeaf - 1) / kLeaf;
  int64_t n = p.nleaf, off = 0;
  for (;;) {
    p.level_off[p.nlevel] = off;
    p.level_n[p.nlevel++] = n;
    off += n;
    if (n == 1) break;
    n = (n + kExactArity - 1) / kExactArity;
  }
  p.nnode = off;
  uint32_t slots = 1024;
  while (slots < 3 * nf && slots < (1u << 30)) slots <<= 1;
  p.hash_slots = slots;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += (bytes + 255) & ~size_t(255);
    return here;
  };
  const size_t f = static_cast<size_t>(nf), q = static_cast<size_t>(nq);
  const size_t leaf = static_cast<size_t>(p.nleaf), node = static_cast<size_t>(p.nnode);
  p.info = take(sizeof(Info));
  p.faces64 = take(sizeof(Face64) * f);
  p.faces32 = take(sizeof(Face32) * kLeaf * leaf);
  p.partner = take(sizeof(uint32_t) * 3 * f);
  p.nb = take(sizeof(int32_t) * 3 * f);
  p.lead = take(3 * f);
  p.moments = take(sizeof(Moments) * node);
  p.test = take(sizeof(NodeTest) * node);
  p.eval = take(sizeof(NodeEval) * node);
  p.counts = take(sizeof(Counts) * leaf);  // set to 0 together with the next
  p.coarse = take(sizeof(unsigned long long) * kCoarse);
  p.first = take(sizeof(Counts) * leaf);
  p.perm = take(sizeof(uint32_t) * q);
  p.list = take(sizeof(uint32_t) * q);
  const size_t m = std::max(f, q);
  p.keys_in = take(sizeof(uint32_t) * m);
  p.keys_out = take(sizeof(uint32_t) * m);
  p.vals_in = take(sizeof(uint32_t) * m);
  p.vals_out = take(sizeof(uint32_t) * f);
  p.heads = take(sizeof(uint32_t) * p.hash_slots);
  p.next = take(sizeof(uint32_t) * 3 * f);
  p.pick = take(sizeof(uint32_t) * 3 * f);
  p.succ = take(sizeof(uint32_t) * 3 * f);
  size_t sort_bytes = 0, scan_bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, static_cast<uint32_t*>(nullptr),
                                  static_cast<uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr),
                                  static_cast<uint32_t*>(nullptr), static_cast<int>(m), 0, 30);
  cub::DeviceScan::ExclusiveScan(nullptr, scan_bytes, static_cast<Counts*>(nullptr),
                                 static_cast<Counts*>(nullptr), AddCounts(), Counts{0, 0, 0},
                                 static_cast<int>(p.nleaf));
  p.cub_bytes = std::max(sort_bytes, scan_bytes);
  p.cub = take(p.cub_bytes);
  p.bytes = at;
  return p;
}

namespace {
template <class T>
T* at(void* scratch, size_t offset) {
  return reinterpret_cast<T*>(static_cast<unsigned char*>(scratch) + offset);
}

// The boundary's block. Every group is at least one item, and so is every triangle.
struct Edges {
  Group* groups;
  Triangle* triangles;
  Root* roots;
  int32_t* leaf;
  size_t bytes;

  Edges(const ExactBoundary& b, void* block) {
    const size_t items = static_cast<size_t>(b.items), edges = static_cast<size_t>(b.edges);
    size_t end = 0;
    auto take = [&](size_t size) {
      const size_t here = end;
      end += (size + 255) & ~size_t(255);
      return here;
    };
    groups = at<Group>(block, take(sizeof(Group) * items));
    triangles = at<Triangle>(block, take(sizeof(Triangle) * items));
    roots = at<Root>(block, take(sizeof(Root) * edges));
    leaf = at<int32_t>(block, take(sizeof(int32_t) * edges));
    bytes = end;
  }
};
}  // namespace

size_t exact_boundary_bytes(const ExactBoundary& boundary) {
  return boundary.items > 0 ? Edges(boundary, nullptr).bytes : 0;
}

cudaError_t exact_boundary(const ExactPlan& p, const double* tri, int64_t ld, void* scratch,
                           bool mixed, ExactBoundary* boundary, cudaStream_t stream) {
  Info* info = at<Info>(scratch, p.info);
  Face64* faces = at<Face64>(scratch, p.faces64);
  uint32_t* partner = at<uint32_t>(scratch, p.partner);
  uint8_t* lead = at<uint8_t>(scratch, p.lead);
  Counts* counts = at<Counts>(scratch, p.counts);
  unsigned long long* coarse = at<unsigned long long>(scratch, p.coarse);
  uint32_t *keys_in = at<uint32_t>(scratch, p.keys_in), *keys_out = at<uint32_t>(scratch, p.keys_out);
  uint32_t *vals_in = at<uint32_t>(scratch, p.vals_in), *vals_out = at<uint32_t>(scratch, p.vals_out);
  uint32_t *heads = at<uint32_t>(scratch, p.heads), *next = at<uint32_t>(scratch, p.next);
  void* temp = at<unsigned char>(scratch, p.cub);
  const uint32_t mask = p.hash_slots - 1;
  const int th = 256;
  size_t tb = p.cub_bytes;
  cudaError_t e;
  exact_init_kernel<<<1, 32, 0, stream>>>(info);
  if ((e = cudaMemsetAsync(heads, 0xff, sizeof(uint32_t) * p.hash_slots, stream)) != cudaSuccess ||
      (e = cudaMemsetAsync(counts, 0, p.coarse - p.counts + sizeof(unsigned long long) * kCoarse,
                           stream)) != cudaSuccess)
    return e;
  exact_face_box_kernel<<<std::min(blocks(p.nf, th), 592u), th, 0, stream>>>(tri, ld, p.nf, info);
  exact_face_keys_kernel<<<blocks(p.nf, th), th, 0, stream>>>(tri, ld, p.nf, info, keys_in,
                                                              vals_in, coarse);
  if ((e = cub::DeviceRadixSort::SortPairs(temp, tb, keys_in, keys_out, vals_in, vals_out,
                                           static_cast<int>(p.nf), 0, 30, stream)) != cudaSuccess)
    return e;
  exact_gather_kernel<<<blocks(p.nf, kGatherThreads), kGatherThreads, 0, stream>>>(
      tri, ld, p.nf, vals_out, keys_out, coarse, faces, heads, mask, next, info);
  exact_partner_kernel<<<blocks(3 * p.nf, th), th, 0, stream>>>(
      faces, 3 * p.nf, heads, mask, next, partner, at<int32_t>(scratch, p.nb), info);
  uint32_t *pick = at<uint32_t>(scratch, p.pick), *succ = at<uint32_t>(scratch, p.succ);
  if ((e = cudaMemsetAsync(heads, 0xff, sizeof(uint32_t) * p.hash_slots, stream)) != cudaSuccess)
    return e;
  exact_root_hash_kernel<<<blocks(3 * p.nf, th), th, 0, stream>>>(faces, 3 * p.nf, partner, heads,
                                                                  mask, next, info);
  exact_pick_kernel<<<blocks(3 * p.nf, th), th, 0, stream>>>(faces, 3 * p.nf, partner, heads, mask,
                                                             next, pick, info);
  exact_successor_kernel<<<blocks(3 * p.nf, th), th, 0, stream>>>(faces, 3 * p.nf, partner, heads,
                                                                  mask, next, pick, succ, info);
  exact_loops_kernel<<<blocks(3 * p.nf, th), th, 0, stream>>>(partner, succ, 3 * p.nf, lead,
                                                              counts, info);
  // Whether it pays is known here: a mesh whose edges do not cancel goes no further.
  Info host;
  if ((e = cudaGetLastError()) != cudaSuccess ||
      (e = cudaMemcpyAsync(&host, info, sizeof(Info), cudaMemcpyDeviceToHost, stream)) !=
          cudaSuccess ||
      (e = cudaStreamSynchronize(stream)) != cudaSuccess)
    return e;
  g_launches.fetch_add(9, std::memory_order_relaxed);
  const double nf = static_cast<double>(p.nf);
  const bool dense = static_cast<double>(host.density) > kMostDense * (kCoarseUnit / 256.0) * nf;
  const bool crowded = static_cast<double>(host.crowd) >
                       (mixed ? kMostCrowdedMixed : kMostCrowdedFp64) * nf * nf;
  const bool fit = !host.bad && !dense && !crowded && host.nopen <= p.nf &&
                   boundary_pays(host.nitem, p.nf, p.nq, mixed);
  boundary->dense = dense && !host.bad;
  boundary->edges = host.nroot;
  boundary->items = fit ? host.nitem : -1;
  boundary->loops = (host.nroot - host.nitem) / 2;  // a loop of n edges: n - 2 triangles
  return cudaSuccess;
}

namespace {
cudaError_t build_tree(const ExactPlan& p, const ExactBoundary& boundary, const Edges& edges,
                       const double* q, void* scratch, cudaStream_t stream) {
  Info* info = at<Info>(scratch, p.info);
  Face64* faces = at<Face64>(scratch, p.faces64);
  uint8_t* lead = at<uint8_t>(scratch, p.lead);
  Moments* moments = at<Moments>(scratch, p.moments);
  NodeTest* test = at<NodeTest>(scratch, p.test);
  Counts *counts = at<Counts>(scratch, p.counts), *first = at<Counts>(scratch, p.first);
  uint32_t *keys_in = at<uint32_t>(scratch, p.keys_in), *keys_out = at<uint32_t>(scratch, p.keys_out);
  uint32_t *vals_in = at<uint32_t>(scratch, p.vals_in), *succ = at<uint32_t>(scratch, p.succ);
  void* temp = at<unsigned char>(scratch, p.cub);
  const int th = 256;
  Levels levels;
  levels.nlevel = p.nlevel;
  for (int k = 0; k < kExactMaxLevels; ++k) {
    levels.off[k] = p.level_off[k];
    levels.n[k] = p.level_n[k];
  }
  cudaError_t e;
  size_t tb = p.cub_bytes;
  if ((e = cub::DeviceScan::ExclusiveScan(temp, tb, counts, first, AddCounts(), Counts{0, 0, 0},
                                          static_cast<int>(p.nleaf), stream)) != cudaSuccess)
    return e;
  exact_leaf_kernel<<<blocks(p.nleaf, 64), 64, 0, stream>>>(faces, p.nf, p.nleaf, info, moments,
                                                            test, at<Face32>(scratch, p.faces32));
  int l = 1;
  for (; l < p.nlevel && p.level_n[l] > 64; ++l) {
    exact_level_kernel<<<blocks(p.level_n[l], 4), 128, 0, stream>>>(
        p.level_off[l - 1], p.level_n[l - 1], p.level_off[l], p.level_n[l], moments, test);
    g_launches.fetch_add(1, std::memory_order_relaxed);
  }
  if (l < p.nlevel) {
    exact_top_kernel<<<1, 1024, 0, stream>>>(levels, l, moments, test);
    g_launches.fetch_add(1, std::memory_order_relaxed);
  }
  exact_radius_kernel<<<blocks(p.nf, th), th, 0, stream>>>(faces, p.nf, levels, info, moments,
                                                           test);
  exact_finish_kernel<<<blocks(p.nnode, 64), 64, 0, stream>>>(p.nnode, moments, test,
                                                              at<NodeEval>(scratch, p.eval));
  exact_groups_kernel<<<blocks(3 * p.nf, th), th, 0, stream>>>(
      faces, 3 * p.nf, p.nleaf, succ, lead, counts, first, boundary.edges, test, edges.groups,
      edges.roots, edges.leaf, edges.triangles, info);
  exact_query_box_kernel<<<std::min(blocks(p.nq, th), 592u), th, 0, stream>>>(q, p.nq, info);
  exact_query_keys_kernel<<<blocks(p.nq, th), th, 0, stream>>>(q, p.nq, info, keys_in, vals_in);
  tb = p.cub_bytes;
  if ((e = cub::DeviceRadixSort::SortPairs(temp, tb, keys_in, keys_out, vals_in,
                                           at<uint32_t>(scratch, p.perm), static_cast<int>(p.nq),
                                           0, 30, stream)) != cudaSuccess)
    return e;
  g_launches.fetch_add(6, std::memory_order_relaxed);
  return cudaGetLastError();
}

template <int SUB>
void launch_eval(const EvalArgs& a, cudaStream_t stream) {
  const int per_block = kWarps * (32 / SUB);
  exact_eval_kernel<SUB><<<blocks(a.nq, per_block), 32 * kWarps, 0, stream>>>(a);
}
}  // namespace

// Lanes per query. More of them shrink the warp's box and fill the GPU where queries are few
// beside the mesh, but every warp walks the tree and reads the mesh's boundary for itself. Each
// line is the number of queries from which fewer lanes are the quicker ones, between the sizes
// where both were measured (ms at 1 / 2 / 4 / 8 lanes):
//   closed   5,120 F x 32,768 Q 0.50 / 0.42 / 0.42 / 0.45   x 80,000 0.52 / 0.50 / 0.55 / 0.64
//            x 180,000 0.66 / 0.67 / 0.78; 20,480 F x 24,000 0.68 / 0.55 / 0.50 / 0.51
//            x 50,000 0.68 / 0.57 / 0.56 / 0.64   x 400,000 1.26 / 1.27 / 1.62; 81,920 F x 32,768
//            1.41 / 1.00 / 0.75 / 0.72   x 80,000 1.36 / 0.94 / 0.88 / 0.99   x 600,000 2.24 /
//            2.16 / 2.83; 327,680 F x 80,000 2.8 / 1.9 / 1.7 / 1.6   x 180,000 3.1 / 2.2 / 2.0
//            x 400,000 3.6 / 2.9 / 3.1   x 2^20 5.1 / 4.6 / 5.6 / 7.8
//   edges    (terrain) 28,322 F x 16,384 2.0 / 1.04 / 0.79 / 0.78   x 50,000 1.6 / 1.19 / 1.12 /
//            1.25   x 262,144 2.8 / 2.6 / 3.0   x 600,000 4.8 / 4.7 / 5.9   x 2^20 7.3 / 7.6 / 9.6;
//            243,602 F x 24,000 8.9 / 4.4 / 2.8 / 2.6   x 131,072 8.7 / 5.7 / 5.7   x 600,000 16.3 /
//            15.0 / 17.3; 498,002 F x 50,000 13 / 8.2 / 6.2 / 5.4   x 262,144 17.7 / 14.0 / 13.7
//   holes    18,842 F, 0.087 items a face, x 12,000 1.29 / 0.93 / 0.92 / 1.23   x 24,000 1.28 /
//            0.96 / 1.32   x 100,000 1.74 / 1.68 / 3.2   x 131,072 1.90 / 1.99   x 2^20 6.5 / 7.8;
//            79,462 F, 0.03 a face, x 100,000 2.8 / 2.4 / 4.6   x 180,000 3.4 / 3.5
static int lanes_per_query(const ExactPlan& p, const ExactBoundary& boundary) {
  struct Lines {
    double eight, four, two;  // below these
  };
  const double f = static_cast<double>(p.nf), q = static_cast<double>(p.nq);
  Lines l;
  if (boundary.items < 64)
    l = {std::max(24e3, 0.41 * f), std::max(32768.0, std::min(1.4 * f, 300e3)),
         std::max(180e3, 8.0 * f)};
  else if (4 * boundary.loops <= boundary.items)
    l = {std::max(20e3, 0.15 * f), 40e3 + 0.45 * f, std::max(500e3, 6.0 * f)};
  else
    l = {8192.0, 16384.0, 20 * boundary.items > p.nf ? 120e3 : 180e3};
  return q < l.eight ? 8 : (q < l.four ? 4 : (q < l.two ? 2 : 1));
}

cudaError_t exact_eval(const ExactPlan& p, const ExactBoundary& boundary, const double* q, double* w,
                       void* scratch, void* block, bool mixed, int sms, cudaStream_t stream) {
  const Edges edges(boundary, block);
  const cudaError_t e = build_tree(p, boundary, edges, q, scratch, stream);
  if (e != cudaSuccess) return e;
  EvalArgs a;
  a.faces = at<Face64>(scratch, p.faces64);
  a.faces32 = at<Face32>(scratch, p.faces32);
  a.nb = at<int32_t>(scratch, p.nb);
  a.test = at<NodeTest>(scratch, p.test);
  a.eval = at<NodeEval>(scratch, p.eval);
  a.groups = edges.groups;
  a.roots = edges.roots;
  a.root_leaf = edges.leaf;
  a.triangles = edges.triangles;
  a.q = q;
  a.perm = at<uint32_t>(scratch, p.perm);
  a.w = w;
  a.list = at<uint32_t>(scratch, p.list);
  a.info = at<Info>(scratch, p.info);
  a.nf = p.nf;
  a.nq = p.nq;
  a.top = p.nnode - 1;
  a.mixed = mixed;
  switch (lanes_per_query(p, boundary)) {
    case 1: launch_eval<1>(a, stream); break;
    case 2: launch_eval<2>(a, stream); break;
    case 4: launch_eval<4>(a, stream); break;
    default: launch_eval<8>(a, stream); break;
  }
  exact_fallback_kernel<<<static_cast<unsigned>(std::max(sms, 1) * 4), 256, 0, stream>>>(
      a.faces, p.nf, q, a.list, a.info, w);
  g_launches.fetch_add(2, std::memory_order_relaxed);
  return cudaGetLastError();
}

cudaError_t exact_infinite(const double* q, int64_t nq, double* w, cudaStream_t stream) {
  exact_infinite_kernel<<<blocks(nq, 256), 256, 0, stream>>>(q, nq, w);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

}  // namespace wn
