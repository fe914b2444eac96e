// CSR of an edge list for a graph that lives for one run (gb_scc_edges, the
// merged runs of a server), where the order within a list is free.
//
// The radix sorts of build_csr keep the input order (create_csr,
// multistep/scc_main.cpp:127-191) and move every pair three times per side.
// Without an order to keep, two moves do: the edges are split into at most
// kPartMaxBuckets ranges of vertices, whose counters fit shared memory, and
// each range is then placed by counting.
//   k_part_hist   both endpoints' range counts (and the id check), one read;
//   k_part_scan   range bases, and the ranges cut into chunks;
//   k_part_split  tiles of kTileE edges, reordered by range in shared memory
//                 and written in runs, both sides from one read of the edges;
//   k_part_count  per chunk, counts per vertex in shared memory, added to the
//                 vertices' degrees (a hub costs one atomic per chunk);
//   k_part_off    per range, the scan of its degrees: offsets and cursors;
//   k_part_place  per chunk, slots reserved at the cursors (again one atomic
//                 per chunk and vertex), entries written.
// 1 M vertices and 16 M R-MAT edges in random order: 29, 5, 136, 48, 13 and
// 231 us, 0.46 ms against 0.89 for the sorts and the offsets between them.
// R-MAT puts 8 % of all edges into one of 512 ranges, hence the chunks.  A
// pair is a vertex's index in its range and the other endpoint: 32 bits when
// both fit, else 64.
#include <algorithm>
#include <cstdint>

#include "gb_internal.cuh"

namespace gb {
namespace {

constexpr int kPartMaxBuckets = 1024;
constexpr int kPartMaxShift = 14;         // vertices per range: 64 KB of counters
constexpr int kPartMinShift = 8;
constexpr int kTileT = 512;               // threads per block: split
constexpr int kTileK = 16;                // edges per thread
constexpr int kTileE = kTileT * kTileK;
static_assert(2 * kTileT >= kPartMaxBuckets, "two ranges per thread");
constexpr int kChunkT = 512;              // threads per block: count, place

struct Part {
  int32_t n;
  int64_t m;
  int shift;
  int buckets;
  int chunk;                // entries per chunk
  const int32_t* key[2];    // src, dst
  unsigned* hist;           // 2 x buckets
  unsigned* base;           // 2 x (buckets + 1): first entry of a range
  unsigned* cursor;         // 2 x buckets
  unsigned* chunk0;         // 2 x (buckets + 1): first chunk of a range
  void* pairs[2];
  unsigned* deg[2];         // n: degrees, then cursors of the place pass
  int64_t* off[2];
  int32_t* adj[2];
  int* bad;
};

template <class P>
__device__ __forceinline__ P part_pack(uint32_t low, uint32_t val, int shift) {
  return ((P)val << shift) | low;
}

// atomicAdd(&cnt[b], 1) on shared memory for the active lanes, one atomic for
// a warp on one counter: edges that come grouped (a union of graphs, a list
// sorted by source) mostly are, and 32 atomics that return a value from one
// word run one after the other (a union of 106 M edges: 709 -> 460 us for the
// split; shuffled edges pay 10 %).  One atomic per distinct counter, by
// __match_any_sync, doubles the time on shuffled edges.  The count passes use
// plain atomics without a result, which the hardware joins by itself (29 us
// against 54 for the ranges of 16 M edges).  All lanes call.
__device__ __forceinline__ unsigned part_rank(unsigned* cnt, int b, bool active) {
  const int b0 = __shfl_sync(0xffffffffu, b, 0);
  if (__all_sync(0xffffffffu, active && b == b0)) {
    const int lane = threadIdx.x & 31;
    unsigned first = 0;
    if (lane == 0) first = atomicAdd(&cnt[b], 32u);
    return __shfl_sync(0xffffffffu, first, 0) + lane;
  }
  return active ? atomicAdd(&cnt[b], 1u) : 0u;
}

__global__ void __launch_bounds__(1024, 2) k_part_hist(Part p) {
  extern __shared__ unsigned h[];
  for (int i = threadIdx.x; i < 2 * p.buckets; i += blockDim.x) h[i] = 0;
  __syncthreads();
  constexpr int kU = 4;
  const int64_t nth = (int64_t)gridDim.x * blockDim.x;
  bool ok = true;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.m; i += nth * kU) {
    int32_t s[kU], d[kU];
#pragma unroll
    for (int q = 0; q < kU; ++q) {
      const bool in = i + q * nth < p.m;
      s[q] = in ? __ldg(p.key[0] + i + q * nth) : 0;
      d[q] = in ? __ldg(p.key[1] + i + q * nth) : 0;
    }
#pragma unroll
    for (int q = 0; q < kU; ++q) {
      if (i + q * nth >= p.m) continue;
      if ((uint32_t)s[q] >= (uint32_t)p.n || (uint32_t)d[q] >= (uint32_t)p.n) {
        ok = false;
        continue;
      }
      atomicAdd(&h[s[q] >> p.shift], 1u);
      atomicAdd(&h[p.buckets + (d[q] >> p.shift)], 1u);
    }
  }
  if (!ok) atomicOr(p.bad, 1);
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * p.buckets; i += blockDim.x)
    if (h[i]) atomicAdd(p.hist + i, h[i]);
}

// One block: thread b scans range b of both sides.
__global__ void __launch_bounds__(kPartMaxBuckets) k_part_scan(Part p) {
  if (*p.bad) return;
  __shared__ unsigned ws[2][33];
  const int b = threadIdx.x, lane = b & 31, wid = b >> 5;
  for (int side = 0; side < 2; ++side) {
    const unsigned cnt = b < p.buckets ? p.hist[side * p.buckets + b] : 0u;
    const unsigned v[2] = {cnt, (cnt + p.chunk - 1) / p.chunk};
    unsigned inc[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      inc[j] = v[j];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, inc[j], o);
        if (lane >= o) inc[j] += y;
      }
      if (lane == 31) ws[j][wid] = inc[j];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2; ++j)
      for (int i = 0; i < wid; ++i) inc[j] += ws[j][i];
    __syncthreads();
    if (b < p.buckets) {
      p.base[side * (p.buckets + 1) + b] = inc[0] - v[0];
      p.cursor[side * p.buckets + b] = inc[0] - v[0];
      p.chunk0[side * (p.buckets + 1) + b] = inc[1] - v[1];
      if (b == p.buckets - 1) {
        p.base[side * (p.buckets + 1) + p.buckets] = inc[0];
        p.chunk0[side * (p.buckets + 1) + p.buckets] = inc[1];
      }
    }
  }
}

template <class P>
__global__ void __launch_bounds__(kTileT, 2) k_part_split(Part p) {
  extern __shared__ unsigned long long dyn[];
  P* stage = reinterpret_cast<P*>(dyn);
  uint16_t* sb = reinterpret_cast<uint16_t*>(stage + kTileE);
  __shared__ unsigned cnt[kPartMaxBuckets], lo[kPartMaxBuckets], go[kPartMaxBuckets];
  __shared__ unsigned ws[32];
  if (*p.bad) return;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t mask = (1u << p.shift) - 1u;
  for (int64_t t0 = (int64_t)blockIdx.x * kTileE; t0 < p.m; t0 += (int64_t)gridDim.x * kTileE) {
    const int len = (int)(p.m - t0 < kTileE ? p.m - t0 : kTileE);
    int32_t e[2][kTileK];
#pragma unroll
    for (int q = 0; q < kTileK; ++q) {
      const int i = q * kTileT + tid;
      e[0][q] = i < len ? __ldcs(p.key[0] + t0 + i) : -1;
      e[1][q] = i < len ? __ldcs(p.key[1] + t0 + i) : -1;
    }
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      for (int i = tid; i < p.buckets; i += kTileT) cnt[i] = 0;
      __syncthreads();
      uint16_t rank[kTileK];
#pragma unroll
      for (int q = 0; q < kTileK; ++q)
        rank[q] = (uint16_t)part_rank(cnt, e[side][q] >> p.shift, e[side][q] >= 0);
      __syncthreads();
      // ranges' places in the tile and, reserved here, in the pairs
      {
        const int b0 = 2 * tid, b1 = 2 * tid + 1;
        const unsigned c0 = b0 < p.buckets ? cnt[b0] : 0u, c1 = b1 < p.buckets ? cnt[b1] : 0u;
        unsigned inc = c0 + c1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned y = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += y;
        }
        if (lane == 31) ws[wid] = inc;
        __syncthreads();
        unsigned pre = lane < wid ? ws[lane] : 0u;
#pragma unroll
        for (int o = 16; o; o >>= 1) pre += __shfl_xor_sync(0xffffffffu, pre, o);
        unsigned* cur = p.cursor + side * p.buckets;
        if (b0 < p.buckets) {
          lo[b0] = pre + inc - c0 - c1;
          go[b0] = c0 ? atomicAdd(cur + b0, c0) : 0u;
        }
        if (b1 < p.buckets) {
          lo[b1] = pre + inc - c1;
          go[b1] = c1 ? atomicAdd(cur + b1, c1) : 0u;
        }
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kTileK; ++q) {
        if (e[side][q] < 0) continue;
        const int b = e[side][q] >> p.shift;
        const unsigned at = lo[b] + rank[q];
        stage[at] = part_pack<P>((uint32_t)e[side][q] & mask, (uint32_t)e[side ^ 1][q], p.shift);
        sb[at] = (uint16_t)b;
      }
      __syncthreads();
      P* out = static_cast<P*>(p.pairs[side]);
      for (int i = tid; i < len; i += kTileT) {
        const int b = sb[i];
        out[go[b] + (unsigned)i - lo[b]] = stage[i];
      }
      __syncthreads();
    }
  }
}

// Chunk c of side `side`: its range and entries.
__device__ __forceinline__ bool part_chunk(const Part& p, int64_t c, int& side, int& b,
                                           unsigned& e0, unsigned& e1) {
  const int64_t c0 = p.chunk0[p.buckets], c1 = p.chunk0[2 * p.buckets + 1];
  if (c >= c0 + c1) return false;
  side = c >= c0;
  const unsigned q = (unsigned)(side ? c - c0 : c);
  const unsigned* ch = p.chunk0 + side * (p.buckets + 1);
  int lo = 0, hi = p.buckets;  // the last range whose first chunk is <= q
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (ch[mid] <= q) lo = mid;
    else hi = mid;
  }
  b = lo;
  const unsigned* base = p.base + side * (p.buckets + 1);
  e0 = base[b] + (q - ch[b]) * (unsigned)p.chunk;
  e1 = min(e0 + (unsigned)p.chunk, base[b + 1]);
  return true;
}

// Calls f(low, value) for the entries [e0, e1) of a chunk, eight per thread
// with their loads together.
template <class P, class F>
__device__ __forceinline__ void part_entries(const Part& p, int side, unsigned e0, unsigned e1,
                                             F f) {
  const P* in = static_cast<const P*>(p.pairs[side]);
  const uint32_t mask = (1u << p.shift) - 1u;
  constexpr int kU = 8;
  for (unsigned i = e0 + threadIdx.x; i < e1; i += kChunkT * kU) {
    P x[kU];
#pragma unroll
    for (int q = 0; q < kU; ++q) x[q] = i + q * kChunkT < e1 ? in[i + q * kChunkT] : (P)0;
#pragma unroll
    for (int q = 0; q < kU; ++q)
      if (i + q * kChunkT < e1) f((uint32_t)x[q] & mask, (int32_t)(x[q] >> p.shift));
  }
}

template <class P>
__global__ void __launch_bounds__(kChunkT) k_part_count(Part p) {
  extern __shared__ unsigned cnt[];
  if (*p.bad) return;
  const int R = 1 << p.shift;
  int side, b;
  unsigned e0, e1;
  for (int64_t c = blockIdx.x; part_chunk(p, c, side, b, e0, e1); c += gridDim.x) {
    for (int i = threadIdx.x; i < R; i += kChunkT) cnt[i] = 0;
    __syncthreads();
    part_entries<P>(p, side, e0, e1, [&](uint32_t low, int32_t) { atomicAdd(&cnt[low], 1u); });
    __syncthreads();
    unsigned* deg = p.deg[side] + ((int64_t)b << p.shift);
    for (int i = threadIdx.x; i < R; i += kChunkT)
      if (cnt[i]) atomicAdd(deg + i, cnt[i]);
    __syncthreads();
  }
}

// Block b of `buckets` per side: offsets of the range's vertices; their
// degrees become the place pass's cursors.
__global__ void __launch_bounds__(1024) k_part_off(Part p) {
  __shared__ unsigned ws[32];
  if (*p.bad) return;
  const int side = blockIdx.x >= p.buckets, b = blockIdx.x - side * p.buckets;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int64_t v0 = (int64_t)b << p.shift;
  const int R = (int)min((int64_t)1 << p.shift, (int64_t)p.n - v0);
  unsigned run = p.base[side * (p.buckets + 1) + b];
  unsigned* deg = p.deg[side];
  int64_t* off = p.off[side];
  for (int r0 = 0; r0 < R; r0 += 1024) {
    const int i = r0 + tid;
    const unsigned c = i < R ? deg[v0 + i] : 0u;
    unsigned inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) ws[wid] = inc;
    __syncthreads();
    unsigned pre = lane < wid ? ws[lane] : 0u, all = ws[lane];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      pre += __shfl_xor_sync(0xffffffffu, pre, o);
      all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    if (i < R) {
      const unsigned at = run + pre + inc - c;
      off[v0 + i] = (int64_t)at;
      deg[v0 + i] = at;
    }
    run += all;
    __syncthreads();
  }
  if (b == p.buckets - 1 && tid == 0) off[p.n] = p.m;
}

// (Entries grouped by vertex in shared memory first, so that a warp writes
// runs of a list, took as long for ranges of 2,048 vertices, 226 against
// 231 us for 2 x 16 M entries, and twice as long for ranges of 8,192.)
template <class P>
__global__ void __launch_bounds__(kChunkT) k_part_place(Part p) {
  extern __shared__ unsigned cnt[];
  if (*p.bad) return;
  const int R = 1 << p.shift;
  int side, b;
  unsigned e0, e1;
  for (int64_t c = blockIdx.x; part_chunk(p, c, side, b, e0, e1); c += gridDim.x) {
    for (int i = threadIdx.x; i < R; i += kChunkT) cnt[i] = 0;
    __syncthreads();
    part_entries<P>(p, side, e0, e1, [&](uint32_t low, int32_t) { atomicAdd(&cnt[low], 1u); });
    __syncthreads();
    unsigned* cur = p.deg[side] + ((int64_t)b << p.shift);
    for (int i = threadIdx.x; i < R; i += kChunkT)
      if (cnt[i]) cnt[i] = atomicAdd(cur + i, cnt[i]);
    __syncthreads();
    int32_t* adj = p.adj[side];
    part_entries<P>(p, side, e0, e1, [&](uint32_t low, int32_t val) {
      adj[atomicAdd(&cnt[low], 1u)] = val;
    });
    __syncthreads();
  }
}

int bits_of32(uint32_t x) {
  int b = 0;
  while (b < 32 && (x >> b) != 0u) ++b;
  return b;
}

template <class P>
cudaError_t part_run(const Part& p, int* h_bad, cudaEvent_t checked, cudaStream_t s) {
  static bool attr_set[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const int split_b = kTileE * ((int)sizeof(P) + 2);
  if (dev < 0 || dev >= 64 || !attr_set[dev]) {
    const int most = 4 << kPartMaxShift;
    if ((e = cudaFuncSetAttribute(k_part_split<P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  split_b)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(k_part_count<P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  most)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(k_part_place<P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  most)) != cudaSuccess)
      return e;
    if (dev >= 0 && dev < 64) attr_set[dev] = true;
  }
  const int cnt_b = 4 << p.shift;
  const int64_t tiles = (p.m + kTileE - 1) / kTileE;
  const int64_t chunks = 2 * (p.m / p.chunk + p.buckets);
  // blocks resident at once
  const int g2 = (int)std::min<int64_t>(tiles, 152 * 2);
  const int gc = (int)std::min<int64_t>(chunks, 152 * (cnt_b > 48 * 1024 ? 3 : 4));
  k_part_hist<<<(int)std::min<int64_t>((p.m + 4095) / 4096, 152 * 2), 1024, 8 * p.buckets, s>>>(p);
  // (the check's verdict is on the host while the other passes still run)
  e = cudaMemcpyAsync(h_bad, p.bad, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaEventRecord(checked, s);
  if (e != cudaSuccess) return e;
  k_part_scan<<<1, kPartMaxBuckets, 0, s>>>(p);
  k_part_split<P><<<g2, kTileT, split_b, s>>>(p);
  k_part_count<P><<<gc, kChunkT, cnt_b, s>>>(p);
  k_part_off<<<2 * p.buckets, 1024, 0, s>>>(p);
  k_part_place<P><<<gc, kChunkT, cnt_b, s>>>(p);
  return cudaGetLastError();
}

size_t up256(size_t x) { return (x + 255) & ~size_t(255); }

// Ranges of n vertices: at most 512, or up to 1024 where that lets a pair
// fit 32 bits.
void part_shape(int32_t n, int& shift, int& buckets, bool& wide) {
  const int idb = std::max(1, bits_of32((uint32_t)(n > 1 ? n - 1 : 1)));
  shift = kPartMinShift;
  while (((n - 1) >> shift) + 1 > 512) ++shift;
  if (idb + shift > 32 && ((n - 1) >> (shift - 1)) + 1 <= kPartMaxBuckets && idb + shift - 1 <= 32 &&
      shift > kPartMinShift)
    --shift;
  buckets = ((n - 1) >> shift) + 1;
  wide = idb + shift > 32;
}

}  // namespace

bool csr_part_fits(int32_t n, int64_t m) {
  return n >= 1 && m >= 1 && m < 0x7fffffffll && (n - 1) >> kPartMaxShift < 512;
}

size_t csr_part_bytes(int32_t n, int64_t m) {
  int shift, buckets;
  bool wide;
  part_shape(n, shift, buckets, wide);
  const size_t b = (size_t)buckets + 1, range = (size_t)buckets << shift;
  return up256(16) + up256(8 * b * 4) + 2 * up256(range * 4) +
         2 * up256((size_t)m * (wide ? 8 : 4));
}

cudaError_t csr_part_build(int32_t n, int64_t m, const int32_t* src, const int32_t* dst,
                           int64_t* out_off, int32_t* out_adj, int64_t* in_off, int32_t* in_adj,
                           void* scratch, int* h_bad, cudaEvent_t checked, cudaStream_t s) {
  Part p{};
  bool wide;
  part_shape(n, p.shift, p.buckets, wide);
  p.n = n;
  p.m = m;
  p.chunk = std::max(16384, 2 << p.shift);
  p.key[0] = src;
  p.key[1] = dst;
  p.off[0] = out_off;
  p.off[1] = in_off;
  p.adj[0] = out_adj;
  p.adj[1] = in_adj;
  char* q = static_cast<char*>(scratch);
  const size_t b = (size_t)p.buckets + 1, range = (size_t)p.buckets << p.shift;
  p.bad = (int*)q;
  q += up256(16);
  p.hist = (unsigned*)q;
  p.base = p.hist + 2 * b;
  p.cursor = p.base + 2 * b;
  p.chunk0 = p.cursor + 2 * b;
  q += up256(8 * b * 4);
  p.deg[0] = (unsigned*)q;
  q += up256(range * 4);
  p.deg[1] = (unsigned*)q;
  q += up256(range * 4);
  const size_t zero = (size_t)(q - (char*)scratch);
  p.pairs[0] = q;
  p.pairs[1] = q + up256((size_t)m * (wide ? 8 : 4));
  cudaError_t e = cudaMemsetAsync(scratch, 0, zero, s);
  if (e != cudaSuccess) return e;
  return wide ? part_run<unsigned long long>(p, h_bad, checked, s)
              : part_run<uint32_t>(p, h_bad, checked, s);
}

}  // namespace gb
