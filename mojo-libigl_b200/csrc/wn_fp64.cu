// Plain FP64 forward: the exact generalized winding number of a triangle soup.
//
// Replaces the reference's two-kernel GPU path (lee101/mojo-libigl,
// src/capi.mojo:297-398: one thread per (face, query) writing an nf x nq FP64
// angle buffer, then one thread per query summing it). Here one fused kernel:
//   * each CTA owns 128 queries, one per thread, held in registers;
//   * the CTA streams the face SoA (9 rows x ld doubles) through a ring of
//     shared-memory tiles filled by 1-D bulk copies (cp.async.bulk, completion on
//     an mbarrier; no cluster multicast);
//   * every thread evaluates its query against each face of the tile, reading the
//     face by shared-memory broadcast;
//   * pair terms are bit-identical to the reference (wn_pair.cuh) wherever their
//     last bits can matter, and rounded about as well where they cannot
//     (pair_terms_far); the angles are summed either by the argument-of-product
//     accumulator (default) or by one atan2 per pair, bit-identical terms only;
//   * no nf x nq buffer exists. When there are too few queries to fill the
//     GPU the face range is split over grid.y and a second kernel sums the
//     per-split partial angles in a fixed order (deterministic, no atomics);
//   * few queries (fp64_few_kernel) leave most threads of such a CTA idle: there
//     the threads stand for faces and the queries are common to the CTA.
#include <algorithm>

#include "wn_common.cuh"
#include "wn_internal.h"
#include "wn_mixed.h"
#include "wn_pair.cuh"
#include "wn_pair_device.cuh"

namespace wn {
namespace {

struct Fp64Args {
  const double* tri;
  int64_t ld;
  int64_t nf;
  const double* q;
  int64_t nq;
  int64_t f_chunk;
  double* w;        // final output when gridDim.y == 1
  double* partial;  // [gridDim.y][nq] angle sums when gridDim.y > 1
  int* err;
};

// Sum of atan2 over faces [f_begin, f_end) read straight from global memory;
// the recovery path for an accumulator marked bad.
__device__ double direct_sum_global(const Fp64Args& a, int64_t f_begin, int64_t f_end, double ox,
                                    double oy, double oz) {
  double s = 0.0;
  for (int64_t f = f_begin; f < f_end; ++f) {
    const double* t = a.tri + f;
    double det, denom;
    pair_terms_exact(ox, oy, oz, t[0], t[a.ld], t[2 * a.ld], t[3 * a.ld], t[4 * a.ld],
                     t[5 * a.ld], t[6 * a.ld], t[7 * a.ld], t[8 * a.ld], det, denom);
    s += atan2(det, denom);
  }
  return s;
}

constexpr int kFwdThreads = 128, kFwdStages = 3;
constexpr int kFwdTileBytes = 9 * kTileFaces * 8;

// Bound by the FP64 pipe: about 115 operations a bit-identical pair (three correctly
// rounded roots among them), 65 one of pair_terms_far. Two
// faces a step: their far factors are multiplied first, which saves half of the product's
// bookkeeping (120 -> 95 instructions a pair) and gives every warp a second chain (92
// registers, 20 warps an SM). One query a thread and 64-face tiles keep the split fine.
// On one B200, before (two queries a thread, bit-identical terms only) and now, us:
// 28,322 F x 1,024 Q 235 -> 159, 20,480 F x 1,024 Q 196 -> 121, 243,602 F x 2,048 Q
// 3,491 -> 2,448; one face a step 182, 137, 2,996. Corners shared with the face before
// were tried instead: a third of them at best in a mesh's own order, no gain.
template <int MODE>
__global__ void __launch_bounds__(kFwdThreads) fp64_forward_kernel(const Fp64Args a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  constexpr int TF = kTileFaces, STAGES = kFwdStages;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + STAGES * kFwdTileBytes);

  const int tid = threadIdx.x;
  const int64_t qi = static_cast<int64_t>(blockIdx.x) * kFwdThreads + tid;
  const int64_t f_begin = static_cast<int64_t>(blockIdx.y) * a.f_chunk;
  const int64_t f_end = min(a.nf, f_begin + a.f_chunk);
  const int ntiles = f_end > f_begin ? static_cast<int>((f_end - f_begin + TF - 1) / TF) : 0;
  const bool valid = qi < a.nq;
  const double ox = valid ? a.q[3 * qi] : 0.0;
  const double oy = valid ? a.q[3 * qi + 1] : 0.0;
  const double oz = valid ? a.q[3 * qi + 2] : 0.0;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 1);
    fence_barrier_init();
  }
  __syncthreads();

  // Tile t covers faces [f_begin + t*TF, +n); each of the 9 rows is one bulk
  // copy of round_up(n, 2) doubles. Alignment: ld and f_chunk are even and TF
  // is even, so every source offset is a multiple of 2 doubles (16 bytes).
  auto issue = [&](int t) {
    const int slot = t % STAGES;
    const int64_t f0 = f_begin + static_cast<int64_t>(t) * TF;
    const int64_t n = min(static_cast<int64_t>(TF), f_end - f0);
    const uint32_t bytes = static_cast<uint32_t>(((n + 1) & ~int64_t(1)) * sizeof(double));
    mbar_arrive_expect_tx(&full[slot], 9u * bytes);
#pragma unroll
    for (int r = 0; r < 9; ++r)
      bulk_g2s(smem_raw + slot * kFwdTileBytes + r * TF * 8, a.tri + r * a.ld + f0, bytes,
               &full[slot]);
  };
  int issued = 0;
  if (tid == 0) {
    for (; issued < min(STAGES, ntiles); ++issued) issue(issued);
  }

  ArgAcc acc;
  argacc_init(acc);
  double sum = 0.0;

  bool failed = false;
  int t = 0;
  for (; t < ntiles; ++t) {
    const int slot = t % STAGES;
    const bool landed = mbar_wait(&full[slot], (t / STAGES) & 1, a.err);
    // Every thread has finished tile t-1 past this barrier, so its slot is free.
    if (!__syncthreads_and(landed)) {
      failed = true;
      break;
    }
    if (tid == 0 && t >= 1 && issued < ntiles) issue(issued++);

    const double* s = reinterpret_cast<const double*>(smem_raw + slot * kFwdTileBytes);
    const int64_t f0 = f_begin + static_cast<int64_t>(t) * TF;
    const int n = static_cast<int>(min(static_cast<int64_t>(TF), f_end - f0));
    auto face = [&](int j, double(&v)[9]) {
#pragma unroll
      for (int r = 0; r < 9; ++r) v[r] = s[r * TF + j];
    };
    double u[9], v[9];
    if (MODE == kFp64ArgProd) {
      int j = 0;
#pragma unroll 1
      for (; j + 1 < n; j += 2) {
        face(j, u);
        face(j + 1, v);
        push_two(acc, ox, oy, oz, u, v);
      }
      if (j < n) {
        face(j, u);
        push_one(acc, ox, oy, oz, u);
      }
    } else {
#pragma unroll 1
      for (int j = 0; j < n; ++j) {
        face(j, u);
        double det, denom;
        pair_terms_exact(ox, oy, oz, u[0], u[1], u[2], u[3], u[4], u[5], u[6], u[7], u[8], det,
                         denom);
        sum += atan2(det, denom);
      }
    }
  }

  if (failed) {
    // Leave no bulk copy in flight into this CTA's shared memory.
    if (tid == 0)
      for (int u = t; u < issued; ++u) mbar_wait(&full[u % STAGES], (u / STAGES) & 1, nullptr);
    __syncthreads();
    return;
  }

  if (!valid) return;
  double angle = sum;
  if (MODE == kFp64ArgProd)
    angle = acc.bad ? direct_sum_global(a, f_begin, f_end, ox, oy, oz)
                    : atan2(acc.zi, acc.zr) + static_cast<double>(acc.k) * kTwoPi;
  if (gridDim.y == 1)
    a.w[qi] = angle / kTwoPi;
  else
    a.partial[static_cast<int64_t>(blockIdx.y) * a.nq + qi] = angle;
}

// Few queries: kFewQueries of them a CTA, common to its threads, which take faces
// f_begin + tid, + kFewThreads, ... The threads' products are multiplied pairwise in a
// fixed order (their turns add; a product that went bad makes the CTA sum one atan2 per
// pair). Bound by latency at the few: 1,178 F x 1 Q 78 -> 24 us on one B200 (with the sum
// of the splits), 28,322 F x 64 Q 105 -> 27, 243,602 F x 64 Q 532 -> 102.
constexpr int kFewThreads = 128, kFewQueries = 4;

__device__ void argacc_join(ArgAcc& s, double zr, double zi, int k, int bad) {
  argacc_push(s, zr, zi);
  s.k += k;
  s.bad |= bad;
}

template <int MODE>
__global__ void __launch_bounds__(kFewThreads) fp64_few_kernel(const Fp64Args a) {
  __shared__ double part[kFewThreads / 32][kFewQueries][2];
  __shared__ int turns[kFewThreads / 32][kFewQueries];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t q0 = static_cast<int64_t>(blockIdx.x) * kFewQueries;
  const int64_t f_begin = static_cast<int64_t>(blockIdx.y) * a.f_chunk;
  const int64_t f_end = min(a.nf, f_begin + a.f_chunk);
  const int nq = static_cast<int>(min(static_cast<int64_t>(kFewQueries), a.nq - q0));
  double o[kFewQueries][3];
  ArgAcc acc[kFewQueries];
  double sum[kFewQueries];
#pragma unroll
  for (int k = 0; k < kFewQueries; ++k) {
    for (int x = 0; x < 3; ++x) o[k][x] = k < nq ? a.q[3 * (q0 + k) + x] : 0.0;
    argacc_init(acc[k]);
    sum[k] = 0.0;
  }
  auto walk = [&](bool product) {
    for (int64_t f = f_begin + tid; f < f_end; f += kFewThreads) {
      double v[9];
#pragma unroll
      for (int r = 0; r < 9; ++r) v[r] = a.tri[r * a.ld + f];
#pragma unroll
      for (int k = 0; k < kFewQueries; ++k) {
        if (k >= nq) break;
        if (product) {
          push_one(acc[k], o[k][0], o[k][1], o[k][2], v);
        } else {
          double det, denom;
          pair_terms_exact(o[k][0], o[k][1], o[k][2], v[0], v[1], v[2], v[3], v[4], v[5], v[6],
                           v[7], v[8], det, denom);
          sum[k] += atan2(det, denom);
        }
      }
    }
  };
  bool product = MODE == kFp64ArgProd;
  walk(product);
  if (product) {
    int bad = 0;
#pragma unroll
    for (int k = 0; k < kFewQueries; ++k) {
      if (k >= nq) break;
      for (int off = 16; off; off >>= 1)
        argacc_join(acc[k], __shfl_down_sync(0xffffffffu, acc[k].zr, off),
                    __shfl_down_sync(0xffffffffu, acc[k].zi, off),
                    __shfl_down_sync(0xffffffffu, acc[k].k, off),
                    __shfl_down_sync(0xffffffffu, acc[k].bad, off));
      bad |= acc[k].bad;
      if (lane == 0) {
        part[warp][k][0] = acc[k].zr;
        part[warp][k][1] = acc[k].zi;
        turns[warp][k] = acc[k].k;
      }
    }
    if (__syncthreads_or(bad)) {
      product = false;
      walk(false);
      __syncthreads();  // part is read by no one: it is written again below
    }
  }
  if (!product) {
#pragma unroll
    for (int k = 0; k < kFewQueries; ++k) {
      for (int off = 16; off; off >>= 1) sum[k] += __shfl_down_sync(0xffffffffu, sum[k], off);
      if (lane == 0) part[warp][k][0] = sum[k];
    }
    __syncthreads();
  }
  if (tid >= nq) return;
  double angle = 0.0;
  bool done = false;
  if (product) {
    ArgAcc s;
    argacc_init(s);
    for (int w = 0; w < kFewThreads / 32; ++w)
      argacc_join(s, part[w][tid][0], part[w][tid][1], turns[w][tid], 0);
    angle = atan2(s.zi, s.zr) + static_cast<double>(s.k) * kTwoPi;
    done = true;
  }
  if (!done)
    for (int w = 0; w < kFewThreads / 32; ++w) angle += part[w][tid][0];
  if (gridDim.y == 1)
    a.w[q0 + tid] = angle / kTwoPi;
  else
    a.partial[static_cast<int64_t>(blockIdx.y) * a.nq + q0 + tid] = angle;
}

// 32 queries x 8 slices of the splits a CTA: one thread for all of a query's splits is a
// chain of their loads.
__global__ void __launch_bounds__(256) sum_splits_kernel(const double* __restrict__ partial,
                                                         int64_t nsplit, int64_t nq,
                                                         double* __restrict__ w) {
  __shared__ double slice[8][32];
  const int64_t qi = static_cast<int64_t>(blockIdx.x) * 32 + threadIdx.x;
  double s = 0.0;
  if (qi < nq)
    for (int64_t y = threadIdx.y; y < nsplit; y += 8) s += partial[y * nq + qi];
  slice[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y != 0 || qi >= nq) return;
  for (int k = 1; k < 8; ++k) s += slice[k][threadIdx.x];
  w[qi] = s / kTwoPi;
}

cudaError_t launch_sum_splits(const double* partial, int64_t nsplit, int64_t nq, double* w,
                              cudaStream_t stream) {
  sum_splits_kernel<<<static_cast<unsigned>((nq + 31) / 32), dim3(32, 8), 0, stream>>>(
      partial, nsplit, nq, w);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

// ---- FP64 over a prepared mesh, with corner reuse ---------------------------
// Same bit-exact pair terms and argument-of-product sum, but the faces come from a
// prepared mesh (wn_mixed.cu): Morton-ordered 64-face tiles whose faces are
// ordered as strips, with a per-face code telling which corners equal a corner
// of the previous face. a = v - o and |a| (three subtractions, three products,
// two sums and a correctly rounded sqrt) depend only on the vertex and the
// query, so a repeated corner is copied instead of recomputed: the same bits,
// about 40% fewer FP64 instructions per pair on a typical mesh.
struct Fp64TiledArgs {
  const double* tri64;  // 9 x ld64, tile-major sorted soup
  int64_t ld64;
  const uint8_t* reuse;  // ld64 codes
  int64_t ntiles;
  const double* q;
  int64_t nq;
  int64_t tiles_per_split;
  double* w;
  double* partial;
  int* err;
};

constexpr int kFp64TileBytes = 9 * kTileFaces * 8 + kTileFaces;  // coordinates + codes

__device__ __forceinline__ Corner pick_corner(unsigned code, const Corner& c0, const Corner& c1,
                                              const Corner& c2) {
  return code == 0 ? c0 : (code == 1 ? c1 : c2);
}

// Corner `pos` of face j when its reuse code M is known at compile time: one of
// the previous face's corners (M = 0..2) or a new one computed from the tile.
template <unsigned M>
__device__ __forceinline__ Corner corner_of(const Corner& p0, const Corner& p1, const Corner& p2,
                                            double ox, double oy, double oz, const double* s,
                                            int pos, int j) {
  if constexpr (M == 3)
    return corner_exact(ox, oy, oz, s[(3 * pos) * kTileFaces + j],
                        s[(3 * pos + 1) * kTileFaces + j], s[(3 * pos + 2) * kTileFaces + j]);
  else if constexpr (M == 0)
    return p0;
  else if constexpr (M == 1)
    return p1;
  else
    return p2;
}

// The three corners of face j. The code is the same for every lane (all lanes
// walk the same face), so a switch over it is a uniform branch, and each case
// names its corners at compile time: no per-register selects. The cases are
// the 28 codes whose reused corners are distinct with at most two of them (a
// face that shares all three corners with the previous one is a duplicate and
// takes the generic path).
__device__ __forceinline__ void face_corners(unsigned code, const Corner& p0, const Corner& p1,
                                             const Corner& p2, double ox, double oy, double oz,
                                             const double* s, int j, Corner& c0, Corner& c1,
                                             Corner& c2) {
#define WN_FACE_CASE(A, B, C)                                 \
  case (A) | ((B) << 2) | ((C) << 4):                         \
    c0 = corner_of<A>(p0, p1, p2, ox, oy, oz, s, 0, j);       \
    c1 = corner_of<B>(p0, p1, p2, ox, oy, oz, s, 1, j);       \
    c2 = corner_of<C>(p0, p1, p2, ox, oy, oz, s, 2, j);       \
    return;
  switch (code) {
    WN_FACE_CASE(3, 3, 3)
    WN_FACE_CASE(0, 3, 3) WN_FACE_CASE(1, 3, 3) WN_FACE_CASE(2, 3, 3)
    WN_FACE_CASE(3, 0, 3) WN_FACE_CASE(3, 1, 3) WN_FACE_CASE(3, 2, 3)
    WN_FACE_CASE(3, 3, 0) WN_FACE_CASE(3, 3, 1) WN_FACE_CASE(3, 3, 2)
    WN_FACE_CASE(3, 0, 1) WN_FACE_CASE(3, 0, 2) WN_FACE_CASE(3, 1, 0)
    WN_FACE_CASE(3, 1, 2) WN_FACE_CASE(3, 2, 0) WN_FACE_CASE(3, 2, 1)
    WN_FACE_CASE(0, 3, 1) WN_FACE_CASE(0, 3, 2) WN_FACE_CASE(1, 3, 0)
    WN_FACE_CASE(1, 3, 2) WN_FACE_CASE(2, 3, 0) WN_FACE_CASE(2, 3, 1)
    WN_FACE_CASE(0, 1, 3) WN_FACE_CASE(0, 2, 3) WN_FACE_CASE(1, 0, 3)
    WN_FACE_CASE(1, 2, 3) WN_FACE_CASE(2, 0, 3) WN_FACE_CASE(2, 1, 3)
    default:
      break;
  }
#undef WN_FACE_CASE
  Corner c[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const unsigned cm = (code >> (2 * m)) & 3u;
    c[m] = cm == 3u ? corner_exact(ox, oy, oz, s[(3 * m) * kTileFaces + j],
                                   s[(3 * m + 1) * kTileFaces + j],
                                   s[(3 * m + 2) * kTileFaces + j])
                    : pick_corner(cm, p0, p1, p2);
  }
  c0 = c[0];
  c1 = c[1];
  c2 = c[2];
}

template <int THREADS, int QPT, int STAGES>
__global__ void __launch_bounds__(THREADS) fp64_tiled_kernel(const Fp64TiledArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* ring = smem_raw;  // [STAGES][kFp64TileBytes]
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + STAGES * kFp64TileBytes);
  const int tid = threadIdx.x;
  const int64_t q_base = static_cast<int64_t>(blockIdx.x) * (THREADS * QPT);
  const int64_t t_begin = static_cast<int64_t>(blockIdx.y) * a.tiles_per_split;
  const int64_t t_left = a.ntiles - t_begin < a.tiles_per_split ? a.ntiles - t_begin
                                                                 : a.tiles_per_split;
  const int ntiles = static_cast<int>(t_left > 0 ? t_left : 0);
  double ox[QPT], oy[QPT], oz[QPT];
#pragma unroll
  for (int k = 0; k < QPT; ++k) {
    const int64_t qi = q_base + k * THREADS + tid;
    const bool valid = qi < a.nq;
    ox[k] = valid ? a.q[3 * qi] : 0.0;
    oy[k] = valid ? a.q[3 * qi + 1] : 0.0;
    oz[k] = valid ? a.q[3 * qi + 2] : 0.0;
  }
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 1);
    fence_barrier_init();
  }
  __syncthreads();
  // Tile t: 9 coordinate rows of 64 doubles (512 bytes each, 16-byte aligned since
  // ld64 is a multiple of 64) and 64 reuse codes.
  auto issue = [&](int t) {
    const int slot = t % STAGES;
    unsigned char* dst = ring + slot * kFp64TileBytes;
    const int64_t base = (t_begin + t) * kTileFaces;
    mbar_arrive_expect_tx(&full[slot], kFp64TileBytes);
#pragma unroll
    for (int r = 0; r < 9; ++r)
      bulk_g2s(dst + r * kTileFaces * 8, a.tri64 + r * a.ld64 + base, kTileFaces * 8, &full[slot]);
    bulk_g2s(dst + 9 * kTileFaces * 8, a.reuse + base, kTileFaces, &full[slot]);
  };
  int issued = 0;
  if (tid == 0)
    for (; issued < min(STAGES, ntiles); ++issued) issue(issued);
  ArgAcc acc[QPT];
  Corner p0[QPT], p1[QPT], p2[QPT];
#pragma unroll
  for (int k = 0; k < QPT; ++k) {
    argacc_init(acc[k]);
    p0[k] = p1[k] = p2[k] = Corner{0, 0, 0, 0};
  }
  bool failed = false;
  int t = 0;
  for (; t < ntiles; ++t) {
    const int slot = t % STAGES;
    const bool landed = mbar_wait(&full[slot], (t / STAGES) & 1, a.err);
    if (!__syncthreads_and(landed)) {
      failed = true;
      break;
    }
    if (tid == 0 && t >= 1 && issued < ntiles) issue(issued++);
    const double* s = reinterpret_cast<const double*>(ring + slot * kFp64TileBytes);
    const uint8_t* codes = ring + slot * kFp64TileBytes + 9 * kTileFaces * 8;
#pragma unroll 1
    for (int j = 0; j < kTileFaces; ++j) {
      const unsigned code = codes[j];
      if (code == 0xffu) break;  // padding: the rest of the tile is empty
#pragma unroll
      for (int k = 0; k < QPT; ++k) {
        Corner c0, c1, c2;
        face_corners(code, p0[k], p1[k], p2[k], ox[k], oy[k], oz[k], s, j, c0, c1, c2);
        double det, denom;
        face_exact(c0, c1, c2, det, denom);
        argacc_push(acc[k], denom, det);
        p0[k] = c0;
        p1[k] = c1;
        p2[k] = c2;
      }
    }
  }
  if (failed) {
    if (tid == 0)
      for (int u = t; u < issued; ++u) mbar_wait(&full[u % STAGES], (u / STAGES) & 1, nullptr);
    __syncthreads();
    return;
  }
#pragma unroll
  for (int k = 0; k < QPT; ++k) {
    const int64_t qi = q_base + k * THREADS + tid;
    if (qi >= a.nq) continue;
    double angle;
    if (!acc[k].bad) {
      angle = atan2(acc[k].zi, acc[k].zr) + static_cast<double>(acc[k].k) * kTwoPi;
    } else {
      // Recovery: one atan2 per pair over this slice, from global memory.
      angle = 0.0;
      for (int64_t f = t_begin * kTileFaces; f < (t_begin + ntiles) * kTileFaces; ++f) {
        if (a.reuse[f] == 0xffu) continue;
        const double* v = a.tri64 + f;
        const int64_t L = a.ld64;
        double det, denom;
        pair_terms_exact(ox[k], oy[k], oz[k], v[0], v[L], v[2 * L], v[3 * L], v[4 * L],
                         v[5 * L], v[6 * L], v[7 * L], v[8 * L], det, denom);
        angle += atan2(det, denom);
      }
    }
    if (gridDim.y == 1)
      a.w[qi] = angle / kTwoPi;
    else
      a.partial[static_cast<int64_t>(blockIdx.y) * a.nq + qi] = angle;
  }
}

template <int MODE>
cudaError_t launch_variant(const Fp64Plan& p, const Fp64Args& a, cudaStream_t stream) {
  const dim3 grid(static_cast<unsigned>(p.qblocks), static_cast<unsigned>(p.nsplit));
  if (p.few) {
    fp64_few_kernel<MODE><<<grid, kFewThreads, 0, stream>>>(a);
  } else {
    const int smem = kFwdStages * (kFwdTileBytes + static_cast<int>(sizeof(uint64_t)));
    fp64_forward_kernel<MODE><<<grid, kFwdThreads, smem, stream>>>(a);
  }
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

}  // namespace

// The shape that leaves the busiest SM the least to do. A CTA costs its tiles and half of
// one for its start; fewer than kFwdLeast CTAs an SM do not fill the FP64 pipe, and more
// than some waves of them need no better split.
Fp64Plan plan_fp64(int64_t nf, int64_t nq, int sms, int force_nsplit) {
  constexpr int64_t kFwdLeast = 8, kFwdMost = 16;
  Fp64Plan p;
  auto round_up = [](int64_t n, int64_t m) { return (std::max<int64_t>(n, 1) + m - 1) / m * m; };
  // A few-query CTA pads the queries to 4, the other to 128, but spends up to 1.5 times as
  // long on a pair (28,322 F, us: 80 Q 30 against 42 padded, 150 Q 42 against 52; 96 Q
  // would tie, 200 Q 56 against 52).
  p.few = 3 * round_up(nq, kFewQueries) <= 2 * round_up(nq, kFwdThreads);
  p.tile_faces = p.few ? kFewThreads : kTileFaces;
  p.qblocks = round_up(nq, p.few ? kFewQueries : kFwdThreads) / (p.few ? kFewQueries : kFwdThreads);
  const int64_t tiles = round_up(nf, p.tile_faces) / p.tile_faces;
  sms = std::max(sms, 1);
  int64_t per = tiles;  // tiles of a CTA
  if (force_nsplit > 0) {
    per = (tiles + force_nsplit - 1) / force_nsplit;
  } else if (p.qblocks < kFwdMost * sms) {
    double best = 0.0;
    const int64_t most = (kFwdMost * sms + p.qblocks - 1) / p.qblocks;
    for (int64_t n = 1; n <= std::min(most, tiles); n += 1 + n / 16) {
      const int64_t t = (tiles + n - 1) / n;
      const int64_t ctas = p.qblocks * ((tiles + t - 1) / t);
      const double cost = static_cast<double>(std::max<int64_t>((ctas + sms - 1) / sms, kFwdLeast)) *
                          (static_cast<double>(t) + 0.5);
      if (best == 0.0 || cost < best) {
        best = cost;
        per = t;
      }
    }
  }
  p.f_chunk = per * p.tile_faces;
  p.nsplit = std::max<int64_t>(1, (nf + p.f_chunk - 1) / p.f_chunk);
  p.scratch_doubles = p.nsplit > 1 ? p.nsplit * nq : 0;
  return p;
}

constexpr int kTiledThreads = 128, kTiledQpt = 1, kTiledStages = 4;

Fp64TiledPlan plan_fp64_tiled(int64_t ntiles, int64_t nq, int sms) {
  Fp64TiledPlan p;
  const int64_t per = static_cast<int64_t>(kTiledThreads) * kTiledQpt;
  const int64_t qblocks = std::max<int64_t>(1, (nq + per - 1) / per);
  const int64_t target = static_cast<int64_t>(std::max(sms, 1)) * 8;
  int64_t nsplit = qblocks < target ? (target + qblocks - 1) / qblocks : 1;
  nsplit = std::max<int64_t>(1, std::min(nsplit, std::max<int64_t>(ntiles, 1)));
  p.tiles_per_split = (std::max<int64_t>(ntiles, 1) + nsplit - 1) / nsplit;
  p.nsplit = std::max<int64_t>(1, (std::max<int64_t>(ntiles, 1) + p.tiles_per_split - 1) /
                                      p.tiles_per_split);
  p.qblocks = qblocks;
  p.scratch_doubles = p.nsplit > 1 ? p.nsplit * nq : 0;
  return p;
}

cudaError_t launch_fp64_tiled(const Fp64TiledPlan& p, const MixedMesh& m, const double* q,
                              int64_t nq, double* w, double* scratch, int* err,
                              cudaStream_t stream) {
  if (nq <= 0) return cudaSuccess;
  if (!m.reuse || (p.nsplit > 1 && !scratch) || p.nsplit > 65535)
    return cudaErrorInvalidValue;
  constexpr int kThreads = kTiledThreads, kStages = kTiledStages;
  Fp64TiledArgs a{m.tri64, m.ld64, m.reuse, m.ntiles, q, nq, p.tiles_per_split, w, scratch, err};
  auto kernel = fp64_tiled_kernel<kThreads, kTiledQpt, kStages>;
  const size_t smem = static_cast<size_t>(kStages) * kFp64TileBytes + sizeof(uint64_t) * kStages;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  kernel<<<dim3(static_cast<unsigned>(p.qblocks), static_cast<unsigned>(p.nsplit)), kThreads,
           smem, stream>>>(a);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if ((e = cudaGetLastError()) != cudaSuccess || p.nsplit == 1) return e;
  return launch_sum_splits(scratch, p.nsplit, nq, w, stream);
}

cudaError_t launch_fp64(const Fp64Plan& p, int mode, const double* tri, int64_t ld, int64_t nf,
                        const double* q, int64_t nq, double* w, double* scratch, int* err,
                        cudaStream_t stream) {
  if (nq <= 0) return cudaSuccess;
  if ((ld & 1) || ld < nf || (p.f_chunk % p.tile_faces) || p.qblocks > 0x7fffffff ||
      p.nsplit > 65535 || (p.nsplit > 1 && scratch == nullptr) ||
      (reinterpret_cast<uintptr_t>(tri) & 15))
    return cudaErrorInvalidValue;
  Fp64Args a{tri, ld, nf, q, nq, p.f_chunk, w, scratch, err};
  cudaError_t e;
  if (p.tile_faces != (p.few ? kFewThreads : kTileFaces)) return cudaErrorInvalidConfiguration;
  if (mode == kFp64Direct)
    e = launch_variant<kFp64Direct>(p, a, stream);
  else
    e = launch_variant<kFp64ArgProd>(p, a, stream);
  if (e != cudaSuccess || p.nsplit == 1) return e;
  return launch_sum_splits(scratch, p.nsplit, nq, w, stream);
}

}  // namespace wn
