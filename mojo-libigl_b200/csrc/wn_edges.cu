// Net boundary edges, sides welded by position and per-vertex sums for the edge adjoints.
//
// The tensors involved are small (three sides a face) and what bounds these passes is
// launches and the waits between them, so each is a few kernels about one radix sort and
// one wait for the count that sizes the result. As general tensor operations they took,
// on one B200: the 4,572 boundary edges of 18,842 faces 1.15 ms (60 launches, 5 waits),
// now 0.20; the boundary and the welded sides of 20,480 separate faces 2.5 ms, now 0.5;
// the sums of 9,144 edge ends over 10,242 vertices 0.35 ms (2 waits), now 0.06.
//
// A side is keyed by its vertices, (smaller, larger, direction) in one 64-bit word, and
// sorted by the pair: the sides of an edge meet, whatever their faces, in the order that
// the caller's results have. Only integers are added (with atomics or in any order), so
// every result is the same from run to run.
#include <cub/cub.cuh>
#include <cuda/std/functional>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include <algorithm>

#include "wn_common.cuh"
#include "wn_edges.h"
#include "wn_internal.h"

namespace wn {
namespace {

constexpr uint32_t kNone = 0xffffffffu;
constexpr int kThreads = 256;

size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }
unsigned blocks(int64_t n) { return static_cast<unsigned>((n + kThreads - 1) / kThreads); }

// Bits of a vertex number; all of them set is no vertex pair (the smaller one differs).
int vertex_bits(int64_t nv) {
  int b = 1;
  while ((int64_t(1) << b) < nv) ++b;
  return b;
}

__host__ __device__ uint64_t no_side(int bits) { return (uint64_t(1) << (2 * bits + 1)) - 1; }

__device__ uint64_t side_key(uint32_t a, uint32_t b, int bits) {
  if (a == b) return no_side(bits);
  const uint64_t lo = min(a, b), hi = max(a, b);
  return ((lo << bits | hi) << 1) | (a > b ? 1u : 0u);
}

struct EdgeOf {  // a side's edge
  __device__ uint64_t operator()(uint64_t key) const { return key >> 1; }
};
struct SignOf {  // +1 from the smaller to the larger vertex
  __device__ int operator()(uint64_t key) const { return key & 1 ? -1 : 1; }
};
struct Kept {  // runs of sides that do not cancel
  const uint64_t* edge;
  const int* net;
  const int* runs;
  uint64_t none;
  __device__ uint32_t operator()(uint32_t i) const {
    return i < static_cast<uint32_t>(*runs) && edge[i] != none && net[i] != 0 ? 1u : 0u;
  }
};
struct Head {  // first side of an edge in the sorted sides
  const uint64_t* key;
  uint64_t none;
  __device__ uint32_t operator()(uint32_t i) const {
    const uint64_t e = key[i] >> 1;
    return e != none && (i == 0 || e != key[i - 1] >> 1) ? 1u : 0u;
  }
};
struct Cancelled {  // edges whose sides cancel
  const uint32_t* rank;  // of the last side: the number of edges
  const int* net;
  uint32_t n;
  __device__ uint32_t operator()(uint32_t i) const {
    return i < rank[n - 1] && net[i] == 0 ? 1u : 0u;
  }
};

template <class F>
auto over(F f) {
  return thrust::make_transform_iterator(thrust::counting_iterator<uint32_t>(0), f);
}

// Pieces of a scratch block, 256-byte aligned. With a null base only their sizes count.
struct Pieces {
  char* base;
  size_t at = 0;
  template <class T>
  T* take(size_t n) {
    T* p = base ? reinterpret_cast<T*>(base + at) : nullptr;
    at += align256(std::max<size_t>(1, n) * sizeof(T));
    return p;
  }
};

struct Boundary {
  uint64_t *key, *sorted, *edge;
  int *net, *runs;
  uint32_t *pos, *bad;
  void* temp;
  size_t temp_bytes, bytes;
  int bits;

  Boundary(int64_t nf, int64_t nv, void* base) {
    const int n = static_cast<int>(3 * nf);
    Pieces p{static_cast<char*>(base)};
    bits = vertex_bits(nv);
    key = p.take<uint64_t>(n);
    sorted = p.take<uint64_t>(n);
    edge = key;  // the unsorted keys are done with
    net = p.take<int>(n);
    runs = p.take<int>(1);
    pos = p.take<uint32_t>(n + 2);  // the total at [n], the fault flag behind it
    bad = pos + n + 1;
    size_t sort = 0, reduce = 0, scan = 0;
    cub::DeviceRadixSort::SortKeys(nullptr, sort, key, sorted, n, 1, 1 + 2 * bits);
    cub::DeviceReduce::ReduceByKey(
        nullptr, reduce, thrust::make_transform_iterator(sorted, EdgeOf()), edge,
        thrust::make_transform_iterator(sorted, SignOf()), net, runs, cuda::std::plus<>(), n);
    cub::DeviceScan::ExclusiveSum(nullptr, scan, over(Kept{edge, net, runs, 0}), pos, n + 1);
    temp_bytes = std::max(sort, std::max(reduce, scan));
    temp = p.take<char>(temp_bytes);
    bytes = p.at;
  }
};

struct Weld {
  uint64_t *key, *sorted;
  uint32_t *table, *rep, *slot, *side, *by_edge, *rank, *zero, *place, *info;
  int* net;
  void* temp;
  size_t temp_bytes, bytes;
  uint32_t slots;
  int bits;

  Weld(int64_t nf, int64_t nv, void* base) {
    const int n = static_cast<int>(3 * nf);
    Pieces p{static_cast<char*>(base)};
    bits = vertex_bits(nv);
    slots = 2;
    while (slots < 2 * static_cast<uint64_t>(nv)) slots *= 2;
    key = p.take<uint64_t>(n);
    sorted = p.take<uint64_t>(n);
    table = p.take<uint32_t>(2 * static_cast<size_t>(slots));
    rep = table + slots;
    slot = p.take<uint32_t>(nv);
    side = p.take<uint32_t>(n);     // side of each key
    by_edge = p.take<uint32_t>(n);  // sorted
    rank = p.take<uint32_t>(n);     // edges up to a sorted side
    net = p.take<int>(n);
    zero = p.take<uint32_t>(n + 1);  // cancelled edges before an edge
    place = p.take<uint32_t>(n);     // a side's place among the written edges, and direction
    info = p.take<uint32_t>(3);
    size_t sort = 0, scan = 0, scan2 = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, sort, key, sorted, side, by_edge, n, 1, 1 + 2 * bits);
    cub::DeviceScan::InclusiveSum(nullptr, scan, over(Head{sorted, 0}), rank, n);
    cub::DeviceScan::ExclusiveSum(nullptr, scan2, over(Cancelled{rank, net, 1}), zero, n + 1);
    temp_bytes = std::max(sort, std::max(scan, scan2));
    temp = p.take<char>(temp_bytes);
    bytes = p.at;
  }
};

struct Gather {
  uint32_t *vertex, *entry, *vertex_sorted, *entry_sorted;
  void* temp;
  size_t temp_bytes, bytes;

  Gather(int64_t entries, void* base) {
    const int n = static_cast<int>(entries);
    Pieces p{static_cast<char*>(base)};
    vertex = p.take<uint32_t>(n);
    entry = p.take<uint32_t>(n);
    vertex_sorted = p.take<uint32_t>(n);
    entry_sorted = p.take<uint32_t>(n);
    temp_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, temp_bytes, vertex, vertex_sorted, entry,
                                    entry_sorted, n);
    temp = p.take<char>(temp_bytes);
    bytes = p.at;
  }
};

__global__ void __launch_bounds__(kThreads)
    boundary_keys_kernel(const int64_t* __restrict__ F, uint32_t nf, int64_t nv, int bits,
                         uint64_t* __restrict__ key, uint32_t* __restrict__ bad) {
  const uint32_t f = blockIdx.x * kThreads + threadIdx.x;
  if (f >= nf) return;
  const int64_t v[3] = {F[3 * (size_t)f], F[3 * (size_t)f + 1], F[3 * (size_t)f + 2]};
  if (v[0] < 0 || v[1] < 0 || v[2] < 0 || v[0] >= nv || v[1] >= nv || v[2] >= nv) *bad = 1;
  for (int c = 0; c < 3; ++c)
    key[3 * (size_t)f + c] = side_key(static_cast<uint32_t>(v[c]),
                                      static_cast<uint32_t>(v[c == 2 ? 0 : c + 1]), bits);
}

__global__ void __launch_bounds__(kThreads)
    boundary_write_kernel(const double* __restrict__ V, const uint64_t* __restrict__ edge,
                          const int* __restrict__ net, const uint32_t* __restrict__ pos,
                          uint32_t n, int bits, double* __restrict__ edges, int64_t le,
                          int64_t* __restrict__ ends) {
  const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const uint32_t p = pos[i];
  if (pos[i + 1] == p) return;  // cancelled, or behind the last run
  const int64_t u = static_cast<int64_t>(edge[i] >> bits);
  const int64_t v = static_cast<int64_t>(edge[i] & ((uint64_t(1) << bits) - 1));
  for (int x = 0; x < 3; ++x) {
    edges[x * le + p] = V[3 * u + x];
    edges[(3 + x) * le + p] = V[3 * v + x];
  }
  edges[6 * le + p] = static_cast<double>(net[i]);
  ends[2 * static_cast<int64_t>(p)] = u;
  ends[2 * static_cast<int64_t>(p) + 1] = v;
}

// A coordinate's bits, with one zero.
__device__ uint64_t bits_of(double x) {
  return static_cast<uint64_t>(__double_as_longlong(x == 0.0 ? 0.0 : x));
}

__device__ uint64_t mix(uint64_t h) {  // D. Stafford's variant 13 of the 64-bit finaliser
  h ^= h >> 30;
  h *= 0xbf58476d1ce4e5b9ull;
  h ^= h >> 27;
  h *= 0x94d049bb133111ebull;
  return h ^ h >> 31;
}

// Vertices of equal position share a slot of an open hash table at most half full (a probe
// ends at an empty slot); the smallest of them stands for all.
__global__ void __launch_bounds__(kThreads)
    weld_vertices_kernel(const double* __restrict__ V, uint32_t nv, uint32_t slots,
                         uint32_t* __restrict__ table, uint32_t* __restrict__ rep,
                         uint32_t* __restrict__ slot) {
  const uint32_t v = blockIdx.x * kThreads + threadIdx.x;
  if (v >= nv) return;
  const uint64_t x = bits_of(V[3 * (size_t)v]), y = bits_of(V[3 * (size_t)v + 1]),
                 z = bits_of(V[3 * (size_t)v + 2]);
  uint32_t s = static_cast<uint32_t>(mix(mix(mix(x) + y) + z)) & (slots - 1);
  for (uint32_t probe = 0; probe < slots; ++probe) {
    uint32_t o = table[s];
    if (o == kNone) o = atomicCAS(&table[s], kNone, v);
    if (o == kNone || (bits_of(V[3 * (size_t)o]) == x && bits_of(V[3 * (size_t)o + 1]) == y &&
                       bits_of(V[3 * (size_t)o + 2]) == z))
      break;
    s = (s + 1) & (slots - 1);
  }
  slot[v] = s;
  atomicMin(&rep[s], v);
}

__global__ void __launch_bounds__(kThreads)
    weld_keys_kernel(const int64_t* __restrict__ F, uint32_t nf, int64_t nv, int bits,
                     const uint32_t* __restrict__ rep, const uint32_t* __restrict__ slot,
                     uint64_t* __restrict__ key, uint32_t* __restrict__ side,
                     uint32_t* __restrict__ bad) {
  const uint32_t f = blockIdx.x * kThreads + threadIdx.x;
  if (f >= nf) return;
  uint32_t v[3];
  bool in = true;
  for (int c = 0; c < 3; ++c) {
    const int64_t i = F[3 * (size_t)f + c];
    in = in && i >= 0 && i < nv;
    v[c] = in ? rep[slot[i]] : 0;
  }
  if (!in) *bad = 1;
  for (uint32_t c = 0; c < 3; ++c) {
    key[3 * (size_t)f + c] = side_key(v[c], v[c == 2 ? 0 : c + 1], bits);
    side[3 * (size_t)f + c] = 3 * f + c;
  }
}

__global__ void __launch_bounds__(kThreads)
    weld_net_kernel(const uint64_t* __restrict__ sorted, const uint32_t* __restrict__ rank,
                    uint32_t n, uint64_t none, int* __restrict__ net) {
  const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n || sorted[i] >> 1 == none) return;
  atomicAdd(&net[rank[i] - 1], SignOf()(sorted[i]));
}

__global__ void weld_info_kernel(const uint32_t* __restrict__ rank,
                                 const uint32_t* __restrict__ zero, uint32_t n,
                                 uint32_t* __restrict__ info) {
  info[0] = zero[n];
  info[1] = rank[n - 1] - zero[n];
}

__global__ void __launch_bounds__(kThreads)
    weld_write_kernel(const double* __restrict__ V, const uint64_t* __restrict__ sorted,
                      const uint32_t* __restrict__ by_edge, const uint32_t* __restrict__ rank,
                      const int* __restrict__ net, const uint32_t* __restrict__ zero, uint32_t n,
                      int bits, int64_t cancelled, int64_t others, uint32_t* __restrict__ place,
                      double* __restrict__ edges) {
  const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const uint64_t k = sorted[i], e = k >> 1, none = no_side(bits) >> 1;
  if (e == none) {
    place[by_edge[i]] = kNone;
    return;
  }
  const uint32_t r = rank[i] - 1;
  const bool cancel = net[r] == 0;
  const uint32_t p = cancel ? zero[r] : r - zero[r];
  place[by_edge[i]] = ((cancel ? p : static_cast<uint32_t>(cancelled) + p) << 1) | (k & 1);
  if (i != 0 && e == sorted[i - 1] >> 1) return;
  const int64_t u = static_cast<int64_t>(e >> bits);
  const int64_t v = static_cast<int64_t>(e & ((uint64_t(1) << bits) - 1));
  const int64_t ld = cancel ? cancelled : others;
  double* out = edges + (cancel ? 0 : 7 * cancelled) + p;
  for (int x = 0; x < 3; ++x) {
    out[x * ld] = V[3 * u + x];
    out[(3 + x) * ld] = V[3 * v + x];
  }
  out[6 * ld] = static_cast<double>(net[r]);
}

__global__ void __launch_bounds__(kThreads)
    gather_keys_kernel(const int64_t* __restrict__ vertices, uint32_t n,
                       uint32_t* __restrict__ vertex, uint32_t* __restrict__ entry) {
  const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  vertex[i] = static_cast<uint32_t>(vertices[i]);
  entry[i] = i;
}

__device__ uint32_t first_not_below(const uint32_t* __restrict__ a, uint32_t n, uint32_t v) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (a[mid] < v) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__global__ void __launch_bounds__(kThreads)
    gather_edges_kernel(const double* __restrict__ dedge, int64_t le,
                        const uint32_t* __restrict__ vertex, const uint32_t* __restrict__ entry,
                        uint32_t n, uint32_t nv, double* __restrict__ dV) {
  const uint32_t v = blockIdx.x * kThreads + threadIdx.x;
  if (v >= nv) return;
  double s[3] = {0.0, 0.0, 0.0};
  for (uint32_t i = first_not_below(vertex, n, v); i < n && vertex[i] == v; ++i) {
    const double* d = dedge + 3 * (entry[i] & 1) * le + (entry[i] >> 1);
    for (int x = 0; x < 3; ++x) s[x] += d[x * le];
  }
  for (int x = 0; x < 3; ++x) dV[3 * (size_t)v + x] = s[x];
}

// A side a -> b takes its edge's terms (dP, dQ) as (da, db) when it runs as the edge does,
// else as (-dQ, -dP). A face's corner starts one side and ends another.
__global__ void __launch_bounds__(kThreads)
    gather_welded_kernel(const double* __restrict__ dedge, uint32_t cancelled, uint32_t others,
                         const uint32_t* __restrict__ place, const uint32_t* __restrict__ vertex,
                         const uint32_t* __restrict__ corner, uint32_t n, uint32_t nv,
                         double* __restrict__ dV) {
  const uint32_t v = blockIdx.x * kThreads + threadIdx.x;
  if (v >= nv) return;
  double s[3] = {0.0, 0.0, 0.0};
  for (uint32_t i = first_not_below(vertex, n, v); i < n && vertex[i] == v; ++i) {
    const uint32_t out = corner[i], in = out % 3 == 0 ? out + 2 : out - 1;
    for (int end = 0; end < 2; ++end) {
      const uint32_t p = place[end ? in : out];
      if (p == kNone) continue;
      const uint32_t e = p >> 1;
      const bool turned = p & 1;
      const int64_t ld = e < cancelled ? cancelled : others;
      const double* d = dedge + (e < cancelled ? static_cast<int64_t>(e)
                                               : 6 * static_cast<int64_t>(cancelled) + e - cancelled);
      d += 3 * (turned != (end == 1)) * ld;
      for (int x = 0; x < 3; ++x) s[x] += turned ? -d[x * ld] : d[x * ld];
    }
  }
  for (int x = 0; x < 3; ++x) dV[3 * (size_t)v + x] = s[x];
}

cudaError_t sort_entries(const int64_t* vertices, uint32_t n, int64_t nv, Gather& g,
                         cudaStream_t stream) {
  gather_keys_kernel<<<blocks(n), kThreads, 0, stream>>>(vertices, n, g.vertex, g.entry);
  return cub::DeviceRadixSort::SortPairs(g.temp, g.temp_bytes, g.vertex, g.vertex_sorted, g.entry,
                                         g.entry_sorted, static_cast<int>(n), 0, vertex_bits(nv),
                                         stream);
}

}  // namespace

size_t boundary_scratch_bytes(int64_t nf, int64_t nv) { return Boundary(nf, nv, nullptr).bytes; }
size_t weld_scratch_bytes(int64_t nf, int64_t nv) { return Weld(nf, nv, nullptr).bytes; }
size_t gather_scratch_bytes(int64_t entries) { return Gather(entries, nullptr).bytes; }

cudaError_t boundary_count(const int64_t* F, int64_t nf, int64_t nv, void* scratch, int64_t* ne,
                           cudaStream_t stream) {
  Boundary b(nf, nv, scratch);
  const int n = static_cast<int>(3 * nf);
  cudaError_t e = cudaMemsetAsync(b.bad, 0, sizeof(uint32_t), stream);
  if (e != cudaSuccess) return e;
  boundary_keys_kernel<<<blocks(nf), kThreads, 0, stream>>>(F, static_cast<uint32_t>(nf), nv,
                                                            b.bits, b.key, b.bad);
  size_t tb = b.temp_bytes;
  if ((e = cub::DeviceRadixSort::SortKeys(b.temp, tb, b.key, b.sorted, n, 1, 1 + 2 * b.bits,
                                          stream)) != cudaSuccess)
    return e;
  tb = b.temp_bytes;
  if ((e = cub::DeviceReduce::ReduceByKey(
           b.temp, tb, thrust::make_transform_iterator(b.sorted, EdgeOf()), b.edge,
           thrust::make_transform_iterator(b.sorted, SignOf()), b.net, b.runs, cuda::std::plus<>(), n,
           stream)) != cudaSuccess)
    return e;
  tb = b.temp_bytes;
  if ((e = cub::DeviceScan::ExclusiveSum(
           b.temp, tb, over(Kept{b.edge, b.net, b.runs, no_side(b.bits) >> 1}), b.pos, n + 1,
           stream)) != cudaSuccess)
    return e;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  uint32_t host[2];
  if ((e = cudaMemcpyAsync(host, b.pos + n, sizeof(host), cudaMemcpyDeviceToHost, stream)) !=
          cudaSuccess ||
      (e = cudaStreamSynchronize(stream)) != cudaSuccess)
    return e;
  *ne = host[1] ? -1 : static_cast<int64_t>(host[0]);
  return cudaGetLastError();
}

cudaError_t boundary_write(const double* V, int64_t nf, int64_t nv, const void* scratch,
                           double* edges, int64_t le, int64_t* ends, cudaStream_t stream) {
  const Boundary b(nf, nv, const_cast<void*>(scratch));
  boundary_write_kernel<<<blocks(3 * nf), kThreads, 0, stream>>>(
      V, b.edge, b.net, b.pos, static_cast<uint32_t>(3 * nf), b.bits, edges, le, ends);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

cudaError_t weld_count(const double* V, const int64_t* F, int64_t nf, int64_t nv, void* scratch,
                       int64_t counts[2], cudaStream_t stream) {
  Weld w(nf, nv, scratch);
  const uint32_t n = static_cast<uint32_t>(3 * nf);
  const uint64_t none = no_side(w.bits) >> 1;
  cudaError_t e;
  if ((e = cudaMemsetAsync(w.table, 0xff, 2 * sizeof(uint32_t) * static_cast<size_t>(w.slots),
                           stream)) != cudaSuccess ||
      (e = cudaMemsetAsync(w.net, 0, sizeof(int) * n, stream)) != cudaSuccess ||
      (e = cudaMemsetAsync(w.info, 0, 3 * sizeof(uint32_t), stream)) != cudaSuccess)
    return e;
  weld_vertices_kernel<<<blocks(nv), kThreads, 0, stream>>>(V, static_cast<uint32_t>(nv), w.slots,
                                                            w.table, w.rep, w.slot);
  weld_keys_kernel<<<blocks(nf), kThreads, 0, stream>>>(F, static_cast<uint32_t>(nf), nv, w.bits,
                                                        w.rep, w.slot, w.key, w.side, w.info + 2);
  size_t tb = w.temp_bytes;
  if ((e = cub::DeviceRadixSort::SortPairs(w.temp, tb, w.key, w.sorted, w.side, w.by_edge,
                                           static_cast<int>(n), 1, 1 + 2 * w.bits, stream)) !=
      cudaSuccess)
    return e;
  tb = w.temp_bytes;
  if ((e = cub::DeviceScan::InclusiveSum(w.temp, tb, over(Head{w.sorted, none}), w.rank,
                                         static_cast<int>(n), stream)) != cudaSuccess)
    return e;
  weld_net_kernel<<<blocks(n), kThreads, 0, stream>>>(w.sorted, w.rank, n, none, w.net);
  tb = w.temp_bytes;
  if ((e = cub::DeviceScan::ExclusiveSum(w.temp, tb, over(Cancelled{w.rank, w.net, n}), w.zero,
                                         static_cast<int>(n) + 1, stream)) != cudaSuccess)
    return e;
  weld_info_kernel<<<1, 1, 0, stream>>>(w.rank, w.zero, n, w.info);
  g_launches.fetch_add(4, std::memory_order_relaxed);
  uint32_t host[3];
  if ((e = cudaMemcpyAsync(host, w.info, sizeof(host), cudaMemcpyDeviceToHost, stream)) !=
          cudaSuccess ||
      (e = cudaStreamSynchronize(stream)) != cudaSuccess)
    return e;
  counts[0] = host[2] ? -1 : static_cast<int64_t>(host[0]);
  counts[1] = static_cast<int64_t>(host[1]);
  return cudaGetLastError();
}

cudaError_t weld_write(const double* V, int64_t nf, int64_t nv, int64_t cancelled, int64_t others,
                       void* scratch, double* edges, cudaStream_t stream) {
  const Weld w(nf, nv, scratch);
  weld_write_kernel<<<blocks(3 * nf), kThreads, 0, stream>>>(
      V, w.sorted, w.by_edge, w.rank, w.net, w.zero, static_cast<uint32_t>(3 * nf), w.bits,
      cancelled, others, w.place, edges);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

cudaError_t gather_edges(const double* dedge, int64_t le, const int64_t* ends, int64_t ne,
                         int64_t nv, void* scratch, double* dV, cudaStream_t stream) {
  Gather g(2 * ne, scratch);
  const uint32_t n = static_cast<uint32_t>(2 * ne);
  cudaError_t e = sort_entries(ends, n, nv, g, stream);
  if (e != cudaSuccess) return e;
  gather_edges_kernel<<<blocks(nv), kThreads, 0, stream>>>(
      dedge, le, g.vertex_sorted, g.entry_sorted, n, static_cast<uint32_t>(nv), dV);
  g_launches.fetch_add(2, std::memory_order_relaxed);
  return cudaGetLastError();
}

cudaError_t gather_welded(const double* dedge, int64_t cancelled, int64_t others,
                          const int64_t* F, int64_t nf, int64_t nv, const void* weld_scratch,
                          void* scratch, double* dV, cudaStream_t stream) {
  const Weld w(nf, nv, const_cast<void*>(weld_scratch));
  Gather g(3 * nf, scratch);
  const uint32_t n = static_cast<uint32_t>(3 * nf);
  cudaError_t e = sort_entries(F, n, nv, g, stream);
  if (e != cudaSuccess) return e;
  gather_welded_kernel<<<blocks(nv), kThreads, 0, stream>>>(
      dedge, static_cast<uint32_t>(cancelled), static_cast<uint32_t>(others), w.place,
      g.vertex_sorted, g.entry_sorted, n, static_cast<uint32_t>(nv), dV);
  g_launches.fetch_add(2, std::memory_order_relaxed);
  return cudaGetLastError();
}

}  // namespace wn
