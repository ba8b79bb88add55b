// Closest-point queries over the reference's median-split hierarchy: the
// device layout of the tree and the host-side builder (internal interface
// between wn_aabb.cu, wn_aabb_host.cpp and the C ABI in wn_capi.cu).
//
// The tree is the one the reference builds in python/igl/__init__.py:286-319
// (boxes lo/hi, nodes left/right/start/count, faces in leaf order, nodes in
// preorder); the reference's traversal is src/capi.mojo:522-586. On the device a
// node has two records. AabbNodeRec holds the FP64 boxes of BOTH children next to the
// child indices, for the reference's own walk. AabbWalkRec holds bounds of both
// children in FP32, for the walk in any order that wn_aabb.cu starts with: the box,
// and a disc.
//
// A disc is a unit normal n (the normalised area-weighted sum of the faces' normals), a
// centre c, and the thickness t and radius r such that every vertex x of the faces has
// |n.(x - c)| <= t and lies within r of the axis c + s n. The faces lie in that
// cylinder, so with h = n.(p - c) and l the distance of p from the axis,
// max(|h| - t, 0)^2 + max(l - r, 0)^2 bounds the squared distance from p to any of
// them from below. A child is skipped when that bound, less a rounding margin, exceeds
// the best squared distance. All of this is in the tree's own frame (AabbFrame), so that
// neither a distant origin nor the unit of length costs the bounds their digits. Points away from a curved surface reach many boxes but
// few discs: inside a 327,680-face sphere the reference's walk tests 595 faces a point
// with the boxes alone, 367 with the range of n.x (a slab) beside them, 46 with the
// discs, 29 when the order is by the discs' centres.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace wn {

struct __align__(16) AabbDisc {
  float n[3], t;  // unit normal (|n| <= 1), half thickness; +inf: no bound along n
  float c[3], r;  // centre, radius; +inf: no bound across n
};

// Faces between two planes: lo <= n.x' <= hi (infinite: no bound), the disc's thickness
// without FP32's margin. The reference's walk needs that: of the leaves that a point away
// from the surface could reach, one in ten is told apart by less than the margin.
struct AabbSlab {
  float n[3], lo, hi;
};

struct __align__(32) AabbNodeRec {
  int32_t left, right, start, count;  // count > 0: a leaf of faces [start, start+count)
  double lbox[6];  // left child's box (lo xyz, hi xyz); unused for a leaf
  double rbox[6];  // right child's box
  AabbSlab lslab, rslab;
  int32_t pad[2];
};
static_assert(sizeof(AabbNodeRec) == 160, "node record is five 32-byte sectors");

struct __align__(16) AabbWalkRec {
  int32_t left, right;  // a leaf: its place beside its parent (AabbSpan::slot), unused
  int32_t start, count;  // as AabbNodeRec's; an internal node: its right child's first face
  AabbDisc ldisc, rdisc;
  float lbox[6], rbox[6];  // rounded outward
};
static_assert(sizeof(AabbWalkRec) == 128, "walk record is one cache line");

// A node's faces (a run [first, last) of the face records; empty if they are not one
// run, possible only in a caller-made tree) and where its disc goes: 2 * parent + side,
// -1 for the root.
struct __align__(16) AabbSpan {
  int32_t first, last, slot, pad;
};

// Where the discs and FP32 boxes live: x' = (x - c) s with the vertices in [-1, 1]^3, s a
// power of two (the products are exact), ext the largest |x'|; s = 0 for a mesh whose
// extent is 0 or out of range: no bounds then.
struct AabbFrame {
  double c[3] = {}, s = 0.0, ext = 0.0;
};

struct __align__(16) AabbTriRec {
  double a[3], b[3], c[3];
  int64_t face;
};
static_assert(sizeof(AabbTriRec) == 80, "face record is five 16-byte words");

// A device-resident tree (immutable once built).
struct AabbDeviceTree {
  AabbNodeRec* nodes = nullptr;
  AabbWalkRec* walk = nullptr;
  AabbSpan* spans = nullptr;
  AabbTriRec* tris = nullptr;
  AabbDisc* face_discs = nullptr;  // one per face record
  int64_t nnodes = 0, nleaf_faces = 0;
  int depth = 0;       // levels, root = 1
  double root[6] = {};  // root box (the traversal tests it when the root is popped)
  double scale = 0.0;   // largest |coordinate| of the mesh (sets the rounding margin)
  AabbFrame frame;
  int32_t thin = 0;    // thin faces (aabb_discs)
  bool any_order = false;  // aabb_pack's *regular, and no thin face (aabb_discs)
};

// Deepest tree the kernels accept (traversal stack of kAabbStack entries,
// which a tree of depth D never exceeds when D + 1 <= kAabbStack).
constexpr int kAabbStack = 64;

// Queries below this count are traversed in input order; above it they are
// Morton-ordered first so that a warp's threads walk nearby paths.
constexpr int64_t kAabbSortMin = 1 << 14;

// Closest point of each query (P: np x 3) over the tree. perm (optional):
// thread t handles query perm[t]. Writes sqrd[i], index[i], closest[3i..3i+2]
// for every query i, in input order. Sets kErrBadLaunch in *err if a
// traversal stack would overflow (never for a validated tree).
cudaError_t aabb_query(const AabbDeviceTree& t, const double* P, int64_t np, const uint32_t* perm,
                       double* sqrd, int64_t* index, double* closest, int* err,
                       cudaStream_t stream);

// Makes the walk records of a tree and its faces' discs, and fills in its slabs; the others are on
// the device (big: the nbig nodes of more than kDiscBig faces,
// device). *thin (device, set to 0 before) receives the number of faces thinner than
// 1 : 1000: the reference's closest point on such a face may lie off it (the barycentric
// quotients lose their digits), so no bound holds for it and only the reference's own
// order says whether it is looked at.
constexpr int kDiscBig = 256;
cudaError_t aabb_discs(const AabbDeviceTree& t, const int32_t* big, int64_t nbig, int32_t* thin,
                       cudaStream_t stream);

// s[i] <- sqrt(s[i]), negated where |w[i]| > 1/2 (inside a closed, consistently
// oriented surface).
cudaError_t signed_from_winding(const double* w, double* s, int64_t n, cudaStream_t stream);

// ---- host side (wn_aabb_host.cpp) -------------------------------------------
// Nodes of the hierarchy over nf faces with at most `leaf` faces per leaf.
int64_t aabb_node_count(int64_t nf, int64_t leaf);

// Builds the tree of python/igl/__init__.py:286-319 into boxes (nnodes x 6),
// nodes (nnodes x 4) and order (nf); returns the stack size (depth + 1), or a
// negative value for invalid input (message in *why). threads <= 0: all cores.
int64_t aabb_build(const double* V, int64_t nv, const int64_t* F, int64_t nf, int64_t leaf,
                   double* boxes, int64_t* nodes, int64_t* order, int threads, const char** why);

// Validates caller-supplied tree arrays and converts them to the device
// records (host memory, caller-sized: nnodes node records and spans, nf face records); the
// slabs are left without bounds, for aabb_discs to fill in on the device.
// *scale receives the largest |coordinate| of the mesh and *frame its frame; *regular
// whether every box holds its children's boxes or its faces and every face lies in one leaf,
// as in the trees that aabb_build makes. Returns the depth (root = 1), or a negative value
// with the reason in *why.
int64_t aabb_pack(const double* V, int64_t nv, const int64_t* F, int64_t nf, const double* boxes,
                  const int64_t* nodes, const int64_t* order, int64_t nnodes,
                  AabbNodeRec* node_out, AabbSpan* span_out, AabbTriRec* tri_out, double* scale,
                  AabbFrame* frame, bool* regular, const char** why);

// The walk's bounds are computed in FP32 in the tree's frame: kWalkMargin * (ext + |px'| +
// |py'| + |pz'|) covers the rounding of p', of the differences and of their products (under
// 20 units of 2^-24), kWalkRel the relative rest. kWalkRound * (scale + |px| + |py| + |pz|),
// brought into the frame, covers the rounding of the closest points' own coordinates in the
// reference's FP64 arithmetic (a few units of 2^-53 of them).
constexpr float kWalkMargin = 2e-6f, kWalkRel = 1e-5f;
constexpr double kWalkRound = 1e-14;
// The slabs' margin (FP64) is kSlabMargin * (scale + |px| + |py| + |pz|): the rounding of n.x'
// and of the reference's closest points, a few units of 2^-53 of the coordinates, with a
// factor above 1000 to spare.
constexpr double kSlabMargin = 4e-12;

}  // namespace wn
