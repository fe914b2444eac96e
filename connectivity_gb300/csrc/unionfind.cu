// Weakly connected components by union-find, for inputs where the searches
// of the run kernel would cost more than one look at every edge:
//   sparse device graphs (lattices, road networks, trees: a BFS from the
//   pivot takes as many steps as the graph is wide, cc_bfs.cpp:47-291), and
//   edge lists, which need no CSR for it (cc_main.cpp:86-165 builds one).
//
// The larger root is always hooked under the smaller, so a component's root
// is its smallest id, the canonical label (cc_main.cpp:184-245).
//
// A device graph goes through three passes.  A block first joins the edges
// inside its own range of ids in shared memory, where a find costs tens of
// cycles a hop; graphs that number neighbours closely (lattices by rows,
// chains) keep most edges there.  The second pass joins the edges between
// ranges on the parents in global memory, the third writes every vertex's
// root.
#include <cstdint>

#include "gb_internal.cuh"

namespace gb {
namespace {

constexpr int kUT = 1024;            // threads per block of the range passes
constexpr int kURangeMin = 2048;     // ids per block
constexpr int kURangeMax = 24576;    // 96 KB of parents: two blocks per SM
constexpr int kUBlocks = 304;        // blocks resident at once (2 per SM)
// Edge lists: one part in kUSample^k is joined first, down to parts of about
// kULast edges, the parents flattened after each (see cc_union_edges).
constexpr int64_t kULast = 65536;
constexpr int kUSample = 8;
constexpr int kULaneDeg = 32;        // longer lists are walked by the warp

template <bool kShared>
__device__ __forceinline__ int32_t uf_ld(const int32_t* p) {
  if constexpr (kShared) return *(const volatile int32_t*)p;
  else return __ldcg(p);
}
// Root with path halving.  Parents only ever point at smaller ids, so what a
// concurrent join leaves behind is still an ancestor.
template <bool kShared>
__device__ __forceinline__ int32_t uf_root(int32_t* par, int32_t x) {
  int32_t p = uf_ld<kShared>(par + x);
  while (p != x) {
    const int32_t q = uf_ld<kShared>(par + p);
    if (q == p) return p;
    par[x] = q;
    x = p;
    p = q;
  }
  return x;
}
template <bool kShared>
__device__ __forceinline__ void uf_join(int32_t* par, int32_t a, int32_t b) {
  for (;;) {
    a = uf_root<kShared>(par, a);
    b = uf_root<kShared>(par, b);
    if (a == b) return;
    const int32_t lo = a < b ? a : b, hi = a < b ? b : a;
    if (atomicCAS(par + hi, hi, lo) == hi) return;
  }
}

// Root as the SM's L1 holds it: an ancestor that was a root at some earlier
// time of this kernel.
__device__ __forceinline__ int32_t uf_root_l1(const int32_t* par, int32_t x) {
  for (int32_t p = __ldca(par + x); p != x; p = __ldca(par + x)) x = p;
  return x;
}
// As uf_join<false>, with a first look through L1: equal ancestors, however
// old, mean one tree.  (Joining on stale values too, with the CAS as the only
// check, was slower: every SM's stale view of a hub costs failed atomics on
// one word; 1.5 M R-MAT edges 0.55-1.3 ms against 0.44.)
__device__ __forceinline__ void uf_join_l1(int32_t* par, int32_t a, int32_t b) {
  a = uf_root_l1(par, a);
  b = uf_root_l1(par, b);
  if (a != b) uf_join<false>(par, a, b);
}

// Calls f(v, w) for every out-edge of the block's vertices [v0, v1), of one
// group of 32 in every `stride`: a lane per vertex, the warp together for
// lists of more than kULaneDeg.  (Four vertices per lane with their loads
// together made the range pass slower, 98 -> 224 us on the 2048^2 lattice:
// it is bound by the joins, which then run with less of the block in step.)
template <class F>
__device__ __forceinline__ void uf_lists(const int64_t* __restrict__ off,
                                         const int32_t* __restrict__ adj, int64_t v0, int64_t v1,
                                         int stride, F f) {
  const int lane = threadIdx.x & 31;
  for (int64_t b = v0 + (int64_t)(threadIdx.x & ~31) * stride; b < v1;
       b += (int64_t)kUT * stride) {
    const int64_t v = b + lane;
    int64_t s = 0, d = 0;
    if (v < v1) {
      s = off[v];
      d = off[v + 1] - s;
    }
    unsigned big = __ballot_sync(0xffffffffu, d > kULaneDeg);
    if (d <= kULaneDeg) {
      for (int64_t e = 0; e < d; e += 4) {
        int32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = e + q < d ? adj[s + e + q] : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (w[q] >= 0) f((int32_t)v, w[q]);
      }
    }
    __syncwarp();
    while (big) {
      const int j = __ffs(big) - 1;
      big &= big - 1;
      const int64_t sj = __shfl_sync(0xffffffffu, s, j), dj = __shfl_sync(0xffffffffu, d, j);
      for (int64_t e = lane; e < dj; e += 32) f((int32_t)(b + j), adj[sj + e]);
      __syncwarp();
    }
  }
}

// Edges inside a block's range of `range` ids, on parents in shared memory;
// *cross gets the number of edges that leave their range.
__global__ void __launch_bounds__(kUT, 2) k_uf_range(int32_t n, int32_t range,
                                                     const int64_t* off, const int32_t* adj,
                                                     int32_t* parent, unsigned long long* cross) {
  extern __shared__ int32_t par[];
  __shared__ unsigned s_cross;
  const int64_t v0 = (int64_t)blockIdx.x * range;
  const int64_t v1 = v0 + range < n ? v0 + range : n;
  const int32_t len = (int32_t)(v1 - v0);
  if (threadIdx.x == 0) s_cross = 0;
  for (int i = threadIdx.x; i < len; i += kUT) par[i] = i;
  __syncthreads();
  unsigned leave = 0;
  uf_lists(off, adj, v0, v1, 1, [&](int32_t v, int32_t w) {
    if (w < v0 || w >= v1) ++leave;
    else if (w != v) uf_join<true>(par, (int32_t)(v - v0), (int32_t)(w - v0));
  });
  leave = __reduce_add_sync(0xffffffffu, leave);
  if ((threadIdx.x & 31) == 0 && leave) atomicAdd(&s_cross, leave);
  __syncthreads();
  if (threadIdx.x == 0 && s_cross) atomicAdd(cross, (unsigned long long)s_cross);
  for (int i = threadIdx.x; i < len; i += kUT)
    parent[v0 + i] = (int32_t)(v0 + uf_root<true>(par, i));
}

// Edges between ranges, of one group of 32 vertices in every `stride`.  With
// stride > 1 the kernel is a first look that does nothing when few edges
// cross (*cross < least): see cc_union_csr.
__global__ void __launch_bounds__(kUT, 2) k_uf_cross(int32_t n, int32_t range, int stride,
                                                     const int64_t* off, const int32_t* adj,
                                                     int32_t* parent,
                                                     const unsigned long long* cross,
                                                     unsigned long long least) {
  if (*cross < least) return;
  const int64_t v0 = (int64_t)blockIdx.x * range;
  const int64_t v1 = v0 + range < n ? v0 + range : n;
  uf_lists(off, adj, v0, v1, stride, [&](int32_t v, int32_t w) {
    if (w < v0 || w >= v1) uf_join_l1(parent, v, w);
  });
}

__global__ void k_uf_self(int32_t n, int32_t* parent) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += (int64_t)gridDim.x * blockDim.x)
    parent[v] = (int32_t)v;
}

// The edges of a list, four per thread with their loads together: those of
// one run of 32 in every `stride` (all with stride 1).  An id outside [0, n)
// sets *bad and its edge is left out.
__global__ void k_uf_edges(int32_t n, int64_t m, int64_t stride, const int32_t* __restrict__ src,
                           const int32_t* __restrict__ dst, int32_t* parent, int* bad) {
  constexpr int kU = 4;
  const int64_t nth = (int64_t)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  const int64_t runs = ((m + 31) / 32 + stride - 1) / stride;
  bool ok = true;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < runs * 32; i += nth * kU) {
    int32_t a[kU], b[kU];
#pragma unroll
    for (int q = 0; q < kU; ++q) {
      const int64_t e = ((i + q * nth) >> 5) * stride * 32 + lane;
      a[q] = e < m ? __ldcs(src + e) : 0;
      b[q] = e < m ? __ldcs(dst + e) : 0;
    }
    // the first hop of all eight ends together
#pragma unroll
    for (int q = 0; q < kU; ++q) {
      if ((uint32_t)a[q] >= (uint32_t)n || (uint32_t)b[q] >= (uint32_t)n) {
        ok = false;
        a[q] = b[q] = 0;
      }
      a[q] = __ldca(parent + a[q]);
      b[q] = __ldca(parent + b[q]);
    }
#pragma unroll
    for (int q = 0; q < kU; ++q)
      if (a[q] != b[q]) uf_join_l1(parent, a[q], b[q]);
  }
  if (!ok) atomicOr(bad, 1);
}

// Every vertex to its root (no join runs at the same time), four vertices per
// thread with their loads together.  The walk halves no paths: a late halving
// write would put back a parent that is no root.  Does nothing when cross is
// given and *cross < least, or bad is given and set.  The roots go to out too
// where that is another array.
__global__ void k_uf_roots(int32_t n, int32_t* parent, const unsigned long long* cross,
                           unsigned long long least, int32_t* out, const int* bad) {
  if ((cross != nullptr && *cross < least) || (bad != nullptr && *bad != 0)) return;
  constexpr int kU = 4;
  const int64_t nth = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nth * kU) {
    int32_t r[kU], p[kU];
#pragma unroll
    for (int q = 0; q < kU; ++q) r[q] = i + q * nth < n ? __ldcg(parent + i + q * nth) : 0;
#pragma unroll
    for (int q = 0; q < kU; ++q) p[q] = __ldcg(parent + r[q]);
#pragma unroll
    for (int q = 0; q < kU; ++q) {
      if (i + q * nth >= n) continue;
      const bool moved = p[q] != r[q];
      while (p[q] != r[q]) {
        r[q] = p[q];
        p[q] = __ldcg(parent + r[q]);
      }
      if (moved) parent[i + q * nth] = r[q];
      if (out != parent) out[i + q * nth] = r[q];
    }
  }
}

int uf_grid(int64_t work) {
  int64_t g = (work + 255) / 256;
  if (g > 152 * 8) g = 152 * 8;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace

cudaError_t cc_union_csr(int32_t n, int64_t m, const int64_t* off, const int32_t* adj,
                         int32_t* labels, unsigned long long* d_cross, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64 || !attr_set[dev]) {
    e = cudaFuncSetAttribute(k_uf_range, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kURangeMax * 4);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) attr_set[dev] = true;
  }
  // one wave of blocks while their ranges fit shared memory
  int64_t range = (((int64_t)n + kUBlocks - 1) / kUBlocks + 255) / 256 * 256;
  if (range < kURangeMin) range = kURangeMin;
  if (range > kURangeMax) range = kURangeMax;
  const int blocks = (int)((n + range - 1) / range);
  k_uf_range<<<blocks, kUT, (size_t)range * 4, s>>>(n, (int32_t)range, off, adj, labels, d_cross);
  if (blocks > 1) {
    // Where most edges cross (no locality in the ids), an eighth of the
    // vertices goes first and the parents are flattened: the other edges
    // then mostly find equal parents.  Joining all at once makes thousands of
    // threads walk and hook the same few roots (uniform random graph, 1 M
    // vertices, 3 M edges: 0.74 ms instead of 0.51).
    const unsigned long long most = (unsigned long long)m / 4 + 65536;
    k_uf_cross<<<blocks, kUT, 0, s>>>(n, (int32_t)range, kUSample, off, adj, labels, d_cross, most);
    k_uf_roots<<<uf_grid(n / 4 + 1), 256, 0, s>>>(n, labels, d_cross, most, labels, nullptr);
    k_uf_cross<<<blocks, kUT, 0, s>>>(n, (int32_t)range, 1, off, adj, labels, d_cross, 0ull);
    k_uf_roots<<<uf_grid(n / 4 + 1), 256, 0, s>>>(n, labels, nullptr, 0ull, labels, nullptr);
  }
  return cudaGetLastError();
}

cudaError_t cc_union_edges(int32_t n, int64_t m, const int32_t* src, const int32_t* dst,
                           int32_t* parent, int32_t* labels, int* d_bad, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (m == 0) parent = labels;
  k_uf_self<<<uf_grid(n), 256, 0, s>>>(n, parent);
  if (m > 0) {
    // A few joins first, then ever more with the parents flattened in between:
    // most edges of the later parts find equal parents at the first load.
    // All at once (100,000 vertices, 1.5 M R-MAT edges): 0.44 ms instead of
    // 0.13, spent on the roots that every thread walks to and hooks.
    int64_t stride = 1;
    while (m / stride > kULast) stride *= kUSample;
    for (; stride >= 1; stride /= kUSample) {
      k_uf_edges<<<uf_grid((m / stride + 3) / 4), 256, 0, s>>>(n, m, stride, src, dst, parent,
                                                              d_bad);
      // (the last part has read every id: only then may the labels be written)
      const bool last = stride == 1;
      k_uf_roots<<<uf_grid(n / 4 + 1), 256, 0, s>>>(n, parent, nullptr, 0ull,
                                                    last ? labels : parent, last ? d_bad : nullptr);
    }
  }
  return cudaGetLastError();
}

}  // namespace gb
