// Edges of a mesh on the device, for the edge adjoints (wn_edges.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace wn {

// Faces and vertices that the kernels take: 32-bit side numbers and vertex pairs in 62 bits.
inline bool edges_fit(int64_t nf, int64_t nv) {
  return nf >= 1 && nv >= 1 && nf <= (int64_t(1) << 28) && nv <= (int64_t(1) << 29);
}

// Scratch of each kind, kept by the caller between the counting and the writing call.
size_t boundary_scratch_bytes(int64_t nf, int64_t nv);
size_t weld_scratch_bytes(int64_t nf, int64_t nv);
size_t gather_scratch_bytes(int64_t entries);

// Counts the net boundary edges and waits for the stream; -1 if a face has an index
// outside [0, nv). The write puts edge i's endpoints and net count into edges (7, le) and
// its vertices into ends[2 i], ends[2 i + 1], in the order of (smaller, larger) vertex.
cudaError_t boundary_count(const int64_t* F, int64_t nf, int64_t nv, void* scratch, int64_t* ne,
                           cudaStream_t stream);
cudaError_t boundary_write(const double* V, int64_t nf, int64_t nv, const void* scratch,
                           double* edges, int64_t le, int64_t* ends, cudaStream_t stream);

// The faces' sides welded by position: counts[0] edges whose sides cancel (net count 0)
// and counts[1] others; counts[0] = -1 for an index outside [0, nv). The write gives the
// first kind as (7, counts[0]) and the others as (7, counts[1]) behind them.
cudaError_t weld_count(const double* V, const int64_t* F, int64_t nf, int64_t nv, void* scratch,
                       int64_t counts[2], cudaStream_t stream);
cudaError_t weld_write(const double* V, int64_t nf, int64_t nv, int64_t cancelled, int64_t others,
                       void* scratch, double* edges, cudaStream_t stream);

// dL/dV (nv, 3) from the edges' (6, le) endpoint terms, a vertex's in the order of ends.
cudaError_t gather_edges(const double* dedge, int64_t le, const int64_t* ends, int64_t ne,
                         int64_t nv, void* scratch, double* dV, cudaStream_t stream);
// The same from welded edges' terms, (6, cancelled) and (6, others) behind them, through
// the sides of weld_scratch.
cudaError_t gather_welded(const double* dedge, int64_t cancelled, int64_t others,
                          const int64_t* F, int64_t nf, int64_t nv, const void* weld_scratch,
                          void* scratch, double* dV, cudaStream_t stream);

}  // namespace wn
