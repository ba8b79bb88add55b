// Exact generalized winding number from near faces, boundary edges and an
// integer (see wn_exact.cu for the method).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace wn {

constexpr int kExactLeafFaces = 8;
constexpr int kExactArity = 4;
constexpr int kExactMaxLevels = 16;

// Where the device arrays of one evaluation lie in its scratch block.
struct ExactPlan {
  int64_t nf = 0, nq = 0;
  int64_t nleaf = 0, nnode = 0;
  int nlevel = 0;
  int64_t level_off[kExactMaxLevels] = {}, level_n[kExactMaxLevels] = {};
  uint32_t hash_slots = 0;  // a power of two
  size_t info, faces64, faces32, partner, nb, lead, moments, test, eval, counts, first;
  size_t keys_in, keys_out, vals_in, vals_out, coarse, heads, next, pick, succ, perm, list, cub;
  size_t cub_bytes = 0, bytes = 0;
};

// Slot of a 32-bit hash in a table of mask + 1 <= 2^32 slots: the high half of its product
// with 2^64 / golden ratio (D. Knuth, TAOCP vol. 3, 6.4), every bit of which depends on the
// hash. A 32-bit product left 25 bits, so tables of more slots (above 11 million faces) had
// chains as long as one of 2^25 has.
#if defined(__CUDACC__)
__host__ __device__
#endif
inline uint32_t hash_slot(uint32_t h, uint32_t mask) {
  return static_cast<uint32_t>(h * 0x9e3779b97f4a7c15ull >> 32) & mask;
}

// Whether a call of this size should take the method (the mesh's edges still decide).
bool exact_pays(int64_t nf, int64_t nq);

ExactPlan plan_exact(int64_t nf, int64_t nq);

// The boundary's triangles and single edges that the method may take per face, at most. Each
// costs every query about 5.5e-12 s, a pair 4.9e-12 s in the FP64 streaming kernel and 1.2e-12 s
// in the mixed one (327,680-face mesh with 8 % of its faces deleted, 0.087 per face, x
// 262,144 queries: 38 ms against 385 and 100; 81,920 faces with 20 % deleted x 65,536: 15.5
// against 21.0 and 11.6). Few queries take fewer still (boundary_pays).
constexpr double kExactMostFp64 = 0.55, kExactMostMixed = 0.13;

// Whether all pairs cost less in FP64 than in mixed precision with the mesh's preparation,
// whose allocations and waits take the host 0.75 ms at least (two hosts, ms, FP64 and mixed:
// 20,480 F without shared edges x 8,192 Q 0.9 and 0.9 to 1.5, x 16,384 1.7 and 1.3 to 1.9,
// x 65,536 6.6 and 3.0 to 3.6; 57,344 F x 4,096 Q 1.2 and 1.0 to 2.2; up to 16,384 F it is half
// as much: 14,336 F x 16,384 Q 1.2 and 0.9).
inline bool fp64_pairs_pay(int64_t nf, int64_t nq) {
  const double pairs = static_cast<double>(nf) * static_cast<double>(nq);
  return 4.9e-12 * pairs <= (nf > 16384 ? 0.75e-3 : 0.4e-3) + 1.55e-12 * pairs;
}

// Whether a boundary of `items` costs less than all pairs of an FP64 or a mixed call.
bool boundary_pays(int64_t items, int64_t nf, int64_t nq, bool mixed);

// The mesh's boundary: its edges, the triangles and single edges that stand for them (what
// it costs a query), and the loops that the triangles fan.
struct ExactBoundary {
  int64_t edges = 0, items = -1, loops = 0;
  bool dense = false;  // surface all around: FP64 pairs cost less than mixed ones, too
};

// Pairs the mesh's edges in `scratch` (plan.bytes), waits for the stream and reports the
// boundary; items = -1 if an all-pairs call (FP64, or mixed) costs less than they or the
// mesh is not fit for the method.
cudaError_t exact_boundary(const ExactPlan& p, const double* tri, int64_t ld, void* scratch,
                           bool mixed, ExactBoundary* boundary, cudaStream_t stream);

// Memory for the boundary itself, known now only: none on a closed mesh, where room for what
// the method takes at most would be 228 bytes a face.
size_t exact_boundary_bytes(const ExactBoundary& boundary);

// Builds the tree and the query order in `scratch` and the boundary in `edges`, after
// exact_boundary, and evaluates W of the queries (in the order given). Infinite queries get
// what the all-pairs kernel that this stands in for gives them: NaN in FP64, 0 in mixed
// precision.
cudaError_t exact_eval(const ExactPlan& p, const ExactBoundary& boundary, const double* q,
                       double* w, void* scratch, void* edges, bool mixed, int sms,
                       cudaStream_t stream);

// Sets w to 0 for infinite queries: FP64 pairs in a mixed call.
cudaError_t exact_infinite(const double* q, int64_t nq, double* w, cudaStream_t stream);

}  // namespace wn
