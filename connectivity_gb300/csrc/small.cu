// Connected components of small graphs, one thread block per graph.
//
// A graph of at most kSmallMaxN vertices fits the shared memory of one SM:
// its offsets, labels, flags, live degrees, frontier queues and a prefix
// array (nine int32 per vertex).  One 1024-thread block then runs the whole
// pipeline with block barriers only -- no cooperative grid, no grid
// barrier, no host round trip -- so a small graph costs a few microseconds
// per step instead of a grid-wide step, and a set of small graphs (a batch,
// or the requests of a server) runs as one launch with a block per graph.
//
// SCC (labels: the smallest member id of each component):
//   1. trim to the fixed point (scc_trim_complete, multistep/scc_trim.cpp:
//      141-297): a vertex without a valid in- or out-neighbour (self-loops
//      aside) is a component alone; removals propagate by live-degree
//      counters and a removed-vertex queue;
//   2. FW-BW (scc_fwbw.cpp:47-466) from the valid vertex of largest
//      out x in live degree (lowest id on ties): forward reach, backward
//      reach inside it; their intersection is one component;
//   3. colour rounds (scc_color.cpp:47-373): every vertex takes the
//      smallest id that reaches it (min-colour push to the fixed point),
//      every vertex whose colour is its own id is a root, and the vertices
//      of its colour that reach it (backward search) are its component;
//      after four of them, signature rounds until no vertex is left (the
//      smallest reaching and reached ids inside classes of equal pairs;
//      equal ids label the vertex).
// Under colour_mode 2, graphs with a hub take a shorter way to the same labels
// (hub_scc): two searches from the hub together, then a contraction of what
// they leave; R-MAT of 4,000 vertices and 52,000 edges: 183 -> 48 us a call.
// WCC (cc_main.cpp:184-245): union-find over the edges with hooking of the
// larger root under the smaller, so each root is its component's smallest
// id; no fixed-point loop.
//
// Frontier steps of the general way are edge-balanced: the frontier's degrees
// are scanned, and thread t takes edges t, t + 1024, ... of the concatenated
// edge lists, finding its vertex by a binary search over the scan, so a hub's
// edges are spread over the whole block.
//
// The CSR comes either from the caller (a device graph or a batch union,
// whose ids are offset by id_base) or from an edge list, counted and
// scattered here into a caller-provided scratch area (2m ints).
#include <cstdint>

#include "contract_device.cuh"

namespace gb {
namespace {

constexpr int kST = 1024;
constexpr int kSW = kST / 32;
constexpr uint32_t kValid = 1u, kFw = 2u, kBw = 4u, kInq = 8u;
constexpr int kCtlInts = 160;

// control words (int32 slots of the shared control area)
constexpr int cQn = 0;       // queue lengths [2]
constexpr int cBad = 2;      // an edge id outside [0, n)
constexpr int cStop = 3;     // a loop ran out of steps
constexpr int cLeft = 4;     // steps the contraction of a rest may take
constexpr int cRed = 8;      // reductions: up to 3 * kSW words
constexpr int cScan = 112;   // scans: kSW + 1 words

__device__ __forceinline__ int warp_incl(int x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// Exclusive prefix sum of a[0..len) in place; returns the total.  Thread t
// owns a contiguous chunk.  Starts and ends with a barrier.
__device__ int32_t block_scan(int32_t* a, int len, int32_t* ctl) {
  __syncthreads();
  const int per = (len + kST - 1) / kST;
  const int lo = min(len, (int)threadIdx.x * per), hi = min(len, lo + per);
  int32_t s = 0;
  for (int i = lo; i < hi; ++i) s += a[i];
  const int inc = warp_incl(s);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t* ws = ctl + cScan;
  if (lane == 31) ws[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    const int v = lane < kSW ? ws[lane] : 0;
    const int vi = warp_incl(v);
    if (lane < kSW) ws[lane] = vi - v;
    if (lane == 31) ws[kSW] = vi;
  }
  __syncthreads();
  int32_t run = ws[wid] + inc - s;
  for (int i = lo; i < hi; ++i) {
    const int32_t x = a[i];
    a[i] = run;
    run += x;
  }
  const int32_t total = ws[kSW];
  __syncthreads();
  return total;
}

// Block sum of x.
__device__ int32_t block_sum(int32_t x, int32_t* ctl) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  __syncthreads();
  if (lane == 0) ctl[cRed + wid] = x;
  __syncthreads();
  int32_t t = 0;
  for (int i = 0; i < kSW; ++i) t += ctl[cRed + i];
  __syncthreads();
  return t;
}

// Block minimum of x.
__device__ int32_t block_min(int32_t x, int32_t* ctl) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o; o >>= 1) x = min(x, __shfl_xor_sync(0xffffffffu, x, o));
  __syncthreads();
  if (lane == 0) ctl[cRed + wid] = x;
  __syncthreads();
  int32_t t = x;
  for (int i = 0; i < kSW; ++i) t = min(t, ctl[cRed + i]);
  __syncthreads();
  return t;
}

// The largest key (then the smallest id) over the block: the pivot rule.
__device__ int32_t block_argmax(long long key, int32_t id, int32_t* ctl) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const long long k2 = __shfl_xor_sync(0xffffffffu, key, o);
    const int32_t i2 = __shfl_xor_sync(0xffffffffu, id, o);
    if (k2 > key || (k2 == key && i2 < id)) { key = k2; id = i2; }
  }
  long long* rk = reinterpret_cast<long long*>(ctl + cRed);  // kSW long longs
  int32_t* ri = ctl + cRed + 2 * kSW;                          // then kSW ids
  __syncthreads();
  if (lane == 0) { rk[wid] = key; ri[wid] = id; }
  __syncthreads();
  for (int i = 0; i < kSW; ++i)
    if (rk[i] > key || (rk[i] == key && ri[i] < id)) { key = rk[i]; id = ri[i]; }
  __syncthreads();
  return id;
}

struct SmallCsr {
  const int32_t* ooff;  // n + 1 (shared)
  const int32_t* ioff;
  const int32_t* oadj;  // global
  const int32_t* iadj;
  int32_t base;         // subtracted from every adjacency entry
};

// The block's shared memory for n vertices, derived in every function from
// the array itself, so that accesses are known to be to shared memory.
struct SmallMem {
  int32_t* ctl;
  int32_t* ooff;   // n + 1
  int32_t* ioff;   // n + 1
  int32_t* lab;    // n from here on
  uint32_t* flg;
  int32_t* cnt_o;
  int32_t* cnt_i;
  int32_t* q[2];
  int32_t* pre;    // n + 1
};
extern __shared__ __align__(16) int32_t g_small_smem[];
__device__ __forceinline__ SmallMem small_mem(int n) {
  SmallMem s;
  s.ctl = g_small_smem;
  s.ooff = g_small_smem + kCtlInts;
  s.ioff = s.ooff + (n + 1);
  s.lab = s.ioff + (n + 1);
  s.flg = reinterpret_cast<uint32_t*>(s.lab + n);
  s.cnt_o = s.lab + 2 * n;
  s.cnt_i = s.cnt_o + n;
  s.q[0] = s.cnt_i + n;
  s.q[1] = s.cnt_i + 2 * n;
  s.pre = s.cnt_i + 3 * n;
  return s;
}

// Visits every edge (v, w) of the frontier's adjacency lists, edge-balanced.
// pre: n + 1 ints of scratch.  Ends with a barrier.
template <class F>
__device__ void expand_front(const int32_t* front, int nf, const int32_t* off, const int32_t* adj,
                             int32_t base, int32_t* pre, int32_t* ctl, F f) {
  for (int i = threadIdx.x; i < nf; i += kST) {
    const int32_t v = front[i];
    pre[i] = off[v + 1] - off[v];
  }
  const int32_t total = block_scan(pre, nf, ctl);
  for (int32_t e = threadIdx.x; e < total; e += kST) {
    int lo = 0, hi = nf - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (pre[mid] <= e) lo = mid;
      else hi = mid - 1;
    }
    const int32_t v = front[lo];
    f(v, adj[off[v] + (e - pre[lo])] - base);
  }
  __syncthreads();
}

// Every edge (u, w) of a CSR, edge-balanced over the block (u found by a
// binary search over the offsets).
template <class F>
__device__ void for_each_edge(int n, const int32_t* off, const int32_t* adj, int32_t base, F f) {
  const int32_t m = off[n];
  for (int32_t e = threadIdx.x; e < m; e += kST) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (off[mid] <= e) lo = mid;
      else hi = mid - 1;
    }
    f(lo, adj[e] - base);
  }
}

// Every edge (a, b) of a list, eight per thread with their loads together
// (the list may be in host memory, read over the host link).  f(a, b, index).
template <class F>
__device__ void for_each_listed(const SmallDesc& D, F f) {
  constexpr int kU = 8;
  for (long long e0 = threadIdx.x; e0 < D.m; e0 += kST * kU) {
    int32_t a[kU], b[kU];
#pragma unroll
    for (int q = 0; q < kU; ++q) {
      const bool in = e0 + q * kST < D.m;
      a[q] = in ? D.src[e0 + q * kST] - D.id_base : 0;
      b[q] = in ? D.dst[e0 + q * kST] - D.id_base : 0;
    }
#pragma unroll
    for (int q = 0; q < kU; ++q)
      if (e0 + q * kST < D.m) f(a[q], b[q], e0 + q * kST);
  }
}

__device__ __forceinline__ void push(int32_t* q, int32_t* qn, int32_t v) {
  q[atomicAdd(qn, 1)] = v;
}

// Union-find root with path halving.  Parents only ever point at smaller
// ids, so a grandparent read at any time is still an ancestor.
__device__ __forceinline__ int32_t uf_find(int32_t* p, int32_t x) {
  volatile int32_t* vp = p;
  for (;;) {
    const int32_t px = vp[x];
    if (px == x) return x;
    const int32_t ppx = vp[px];
    if (ppx != px) vp[x] = ppx;
    x = px;
  }
}

__device__ __forceinline__ void uf_unite(int32_t* p, int32_t a, int32_t b) {
  for (;;) {
    const int32_t ra = uf_find(p, a), rb = uf_find(p, b);
    if (ra == rb) return;
    const int32_t lo = ra < rb ? ra : rb, hi = ra < rb ? rb : ra;
    if (atomicCAS(&p[hi], hi, lo) == hi) return;
  }
}

// ---- graphs with a hub ------------------------------------------------------
// A pivot of at least kHubDeg edges on both sides: the graph's large component
// lies within a few hops of it, and most vertices have a neighbour that is
// reached early.  Then, instead of the trim to the fixed point, the frontier
// queues and the colour rounds (a binary search and a chain of L2 loads per
// edge: 156 us for 4,000 vertices and 52,000 edges):
//   - both searches advance in the same passes, from below: a vertex that is
//     not reached looks through its list until it finds one that is;
//   - the edges between the vertices left are listed, and those without both
//     an in- and an out-edge among them labelled;
//   - what remains is contracted (con_solve).
// A rest too large for the contraction goes to the general way's trim and
// colour rounds, and searches that go on for long leave everything to it: a
// pass over all vertices per hop is then the slower way.  R-MAT graphs of this
// size end within 7 passes.  A pass takes 1.05 us per 1,024 vertices, a hop of
// a chain in the trim 1.9 us, so up to 1,024 vertices the passes win as long as
// what they leave fits the contraction; in larger graphs they stop after
// kHubWork turns of 1,024 vertices (at least kHubPasses).  600 vertices with a
// hub and a chain of k behind them (start to end, us):
//     k                     60    300    600   2000   5000
//     general way only     180    612   1164   3711   9267
//     no bound, no trim    122    437   5747  23289 102648
//     with both            125    446   1177   3708   9306
constexpr int32_t kHubDeg = 16;
constexpr int32_t kHubPasses = 8;
constexpr int32_t kHubWork = 32;
constexpr int32_t kSigAfterSmall = 4;  // colour rounds of colour_mode 2

// One pass of a search from below for vertex v of this lane (valid and not
// reached when `need`): whether a neighbour in adj[s, s + d) is reached
// (`bit`).  Eight entries by the lane, the rest by the warp.  All lanes call.
__device__ __forceinline__ bool hub_look(const uint32_t* flg, const int32_t* adj, int32_t base,
                                         uint32_t bit, bool need, int32_t s, int32_t d) {
  bool hit = false;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    int32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = need && !hit && 4 * h + q < d ? adj[s + 4 * h + q] - base : -1;
#pragma unroll
    for (int q = 0; q < 4; ++q) hit = hit || (w[q] >= 0 && (flg[w[q]] & bit));
  }
  unsigned more = __ballot_sync(kFull, need && !hit && d > 8);
  const int lane = threadIdx.x & 31;
  while (more) {
    const int j = __ffs(more) - 1;
    more &= more - 1;
    const int32_t sj = __shfl_sync(kFull, s, j), dj = __shfl_sync(kFull, d, j);
    bool any = false;
    for (int32_t e = 8; e < dj && !any; e += 128) {
      bool h = false;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int32_t i = e + 32 * q + lane;
        const int32_t w = i < dj ? adj[sj + i] - base : -1;
        h = h || (w >= 0 && (flg[w] & bit));
      }
      any = __any_sync(kFull, h);
    }
    if (lane == j) hit = hit || any;
  }
  return hit;
}

// Edges of the residual between local ids (loc).
struct HubRest {
  const uint32_t* e;
  int n;
  const int32_t* loc;
  template <class W, class F>
  __device__ __forceinline__ void edges(const W& w, F f) const {
    for (int b = (int)w.tid() & ~31; b < n; b += (int)w.threads()) {
      const int i = b + (int)(threadIdx.x & 31);
      const uint32_t x = i < n ? e[i] : 0u;
      f(i < n ? loc[x >> 16] : 0, i < n ? loc[x & 0xffffu] : 0, i < n);
    }
  }
};

// SCC of a graph with a hub, up to the vertices that con_solve could not take:
// their number is returned, their flg is kValid, every other vertex has its
// label in lab.  -1: the searches were given up, nothing is labelled.  Uses
// kHubSmem bytes of shared memory past the flags.
// (R-MAT graphs leave a few dozen vertices.  Room for 1,024 took enough from
// the L1 to slow the general path by 7 %, which reads its lists through it.)
constexpr int32_t kHubVerts = 512, kHubEdges = 1536, kHubLog = 1280;
constexpr int32_t kHubCon = con_bytes(kHubVerts, kHubEdges, kHubLog);
constexpr int32_t kHubSmem = kHubCon + kHubVerts * 4 + kHubEdges * 4;
__device__ __noinline__ int32_t hub_scc(int n, int32_t pivot, const int32_t* oadj,
                                        const int32_t* iadj, int32_t base, int32_t cap) {
  const int tid = threadIdx.x, lane = tid & 31;
  const SmallMem s = small_mem(n);
  const int32_t* const ooff = s.ooff;
  const int32_t* const ioff = s.ioff;
  int32_t* const lab = s.lab;
  uint32_t* const flg = s.flg;
  int32_t* const ctl = s.ctl;
  // (16-byte aligned, after the flags)
  int32_t* const tail = g_small_smem + ((kCtlInts + 4 * n + 2 + 3) & ~3);
  int32_t* qn = ctl + cQn;
  // valid: an edge on either side; the pivot's neighbours are reached
  for (int v = tid; v < n; v += kST) {
    const bool valid = ooff[v + 1] > ooff[v] && ioff[v + 1] > ioff[v];
    flg[v] = valid ? kValid : 0u;
    lab[v] = valid ? -1 : v;
  }
  __syncthreads();
  for (int e = ooff[pivot] + tid; e < ooff[pivot + 1]; e += kST)
    atomicOr(&flg[oadj[e] - base], kFw);
  for (int e = ioff[pivot] + tid; e < ioff[pivot + 1]; e += kST)
    atomicOr(&flg[iadj[e] - base], kBw);
  if (tid == 0) atomicOr(&flg[pivot], kFw | kBw);
  const int32_t turns = (n + kST - 1) / kST;
  int32_t pass = 0;
  for (bool open = true; open; ++pass) {
    if (pass >= cap) return -1;
    if (pass >= kHubPasses && pass * turns >= kHubWork) {
      if (turns > 1) return -1;
      if (pass == kHubWork) {
        int32_t most = 0;
        for (int v = tid; v < n; v += kST) {
          const uint32_t f = flg[v];
          if ((f & kValid) && (f & (kFw | kBw)) != (kFw | kBw)) ++most;
        }
        if (block_sum(most, ctl) > kHubVerts) return -1;
      }
    }
    __syncthreads();
    if (tid == 0) qn[0] = 0;
    __syncthreads();
    bool grew = false;
    for (int v0 = tid & ~31; v0 < n; v0 += kST) {
      const int v = v0 + lane;
      const uint32_t f = v < n ? flg[v] : 0u;
      const bool nf = (f & (kValid | kFw)) == kValid, nb = (f & (kValid | kBw)) == kValid;
      const int32_t is = nf ? ioff[v] : 0, id = nf ? ioff[v + 1] - is : 0;
      const int32_t os = nb ? ooff[v] : 0, od = nb ? ooff[v + 1] - os : 0;
      const bool hf = hub_look(flg, iadj, base, kFw, nf, is, id);
      const bool hb = hub_look(flg, oadj, base, kBw, nb, os, od);
      if (hf || hb) {
        flg[v] = f | (hf ? kFw : 0u) | (hb ? kBw : 0u);  // (only this lane writes it)
        grew = true;
      }
    }
    if (__any_sync(kFull, grew) && lane == 0) qn[0] = 1;
    __syncthreads();
    open = qn[0] != 0;
  }
  // the component takes its smallest member; the rest is listed
  int32_t mn = 0x7fffffff;
  for (int v = tid; v < n; v += kST)
    if ((flg[v] & (kValid | kFw | kBw)) == (kValid | kFw | kBw)) mn = min(mn, v);
  mn = block_min(mn, ctl);
  if (tid == 0) qn[0] = qn[1] = 0;
  int32_t left = 0;
  for (int v = tid; v < n; v += kST) {
    const uint32_t f = flg[v];
    if (!(f & kValid)) {
      flg[v] = 0;
    } else if ((f & (kFw | kBw)) == (kFw | kBw)) {
      lab[v] = mn;
      flg[v] = 0;
    } else {
      flg[v] = kValid;
      ++left;
    }
  }
  left = block_sum(left, ctl);
  if (left == 0) return 0;
  int32_t* const rest = tail + kHubCon / 4;
  uint32_t* const edges = reinterpret_cast<uint32_t*>(rest + kHubVerts);
  // edges between the vertices left, a warp per vertex; kFw: has an out-edge,
  // kBw: has an in-edge
  for (int v = tid >> 5; v < n; v += kSW) {
    if (!(flg[v] & kValid)) continue;
    for (int32_t e = ooff[v] + lane; e < ooff[v + 1]; e += 32) {
      const int32_t w = oadj[e] - base;
      if (w == v || !(flg[w] & kValid)) continue;
      atomicOr(&flg[v], kFw);
      atomicOr(&flg[w], kBw);
      const int at = atomicAdd(&qn[1], 1);
      if (at < kHubEdges) edges[at] = ((uint32_t)v << 16) | (uint32_t)w;
    }
  }
  __syncthreads();
  left = 0;
  for (int v = tid; v < n; v += kST) {
    const uint32_t f = flg[v];
    if (!(f & kValid)) continue;
    if ((f & (kFw | kBw)) == (kFw | kBw)) {
      flg[v] = kValid;
      const int at = atomicAdd(&qn[0], 1);
      if (at < kHubVerts) {
        rest[at] = v;
        lab[v] = at;  // its local id until it is labelled
      }
      ++left;
    } else {
      lab[v] = v;
      flg[v] = 0;
    }
  }
  left = block_sum(left, ctl);
  const int ne = qn[1];
  if (left == 0 || left > kHubVerts || ne > kHubEdges) return left;
  __syncthreads();
  if (tid == 0) {
    qn[1] = 0;
    ctl[cLeft] = cap - pass;
  }
  // edges of vertices labelled just now drop out, a stretch of the block at a
  // time (what is kept never passes what is read)
  for (int b0 = 0; b0 < ne; b0 += kST) {
    const int i = b0 + tid;
    const uint32_t x = i < ne ? edges[i] : 0u;
    const bool keep = i < ne && (flg[x >> 16] & kValid) && (flg[x & 0xffffu] & kValid);
    __syncthreads();
    if (keep) edges[atomicAdd(&qn[1], 1)] = x;
    __syncthreads();
  }
  __syncthreads();
  int32_t* comp;
  con_solve<kHubVerts, kHubEdges, kHubLog>(HubRest{edges, qn[1], lab}, left, tail, ctl + cLeft,
                                           &comp);
  __syncthreads();
  if (ctl[cLeft] < 0) return left;  // (out of steps: all of it is left to the rounds)
  int32_t* const small = tail;  // (the contraction's edges are done with)
  for (int i = tid; i < left; i += kST) small[i] = 0x7fffffff;
  __syncthreads();
  for (int i = tid; i < left; i += kST)
    if (comp[i] >= 0) atomicMin(&small[comp[i]], rest[i]);
  __syncthreads();
  int32_t open = 0;
  for (int i = tid; i < left; i += kST) {
    const int32_t v = rest[i];
    lab[v] = comp[i] >= 0 ? small[comp[i]] : -1;
    if (comp[i] >= 0) flg[v] = 0;
    else ++open;
  }
  return block_sum(open, ctl);
}

// The general path: trim to the fixed point, FW-BW, colour and signature
// rounds by frontier queues.  nvalid >= 0: only the trim and the rounds, for
// the vertices that hub_scc left.  (Not inlined, as hub_scc is not: with both
// in the kernel the registers kept across their calls made this path 8 %
// slower.)
__device__ __noinline__ void queue_scc(int n, const int32_t* oadj, const int32_t* iadj,
                                       int32_t base, int32_t cap, int32_t colour_rounds,
                                       int32_t nvalid) {
  const int tid = threadIdx.x;
  const SmallMem s = small_mem(n);
  int32_t* const ctl = s.ctl;
  int32_t* const ooff = s.ooff;
  int32_t* const ioff = s.ioff;
  int32_t* const lab = s.lab;
  uint32_t* const flg = s.flg;
  int32_t* const cnt_o = s.cnt_o;
  int32_t* const cnt_i = s.cnt_i;
  int32_t* const q[2] = {s.q[0], s.q[1]};
  int32_t* const pre = s.pre;
  int32_t* const qn = ctl + cQn;
  int cur = 0;
  // live degrees without self-loops
  const bool rest = nvalid >= 0;
  for (int v = tid; v < n; v += kST) {
    cnt_o[v] = rest ? 0 : ooff[v + 1] - ooff[v];
    cnt_i[v] = rest ? 0 : ioff[v + 1] - ioff[v];
    if (!rest) flg[v] = kValid;
    if (flg[v] & kValid) lab[v] = -1;
  }
  __syncthreads();
  if (rest) {
    for_each_edge(n, ooff, oadj, base, [&](int32_t u, int32_t w) {
      if (u != w && (flg[u] & flg[w] & kValid)) {
        atomicAdd(&cnt_o[u], 1);
        atomicAdd(&cnt_i[w], 1);
      }
    });
  } else {
    for_each_edge(n, ooff, oadj, base, [&](int32_t u, int32_t w) {
      if (u == w) {
        atomicSub(&cnt_o[u], 1);
        atomicSub(&cnt_i[u], 1);
      }
    });
  }
  if (tid == 0) qn[0] = 0;
  __syncthreads();

  // 1. trim to the fixed point
  for (int v = tid; v < n; v += kST) {
    if ((flg[v] & kValid) && (cnt_o[v] == 0 || cnt_i[v] == 0)) {
      flg[v] = 0;
      lab[v] = v;
      push(q[0], &qn[0], v);
    }
  }
  __syncthreads();
  auto claim_trim = [&](int32_t w, int nx) {
    const uint32_t old = atomicAnd(&flg[w], ~kValid);
    if (old & kValid) {
      lab[w] = w;
      push(q[nx], &qn[nx], w);
    }
  };
  cur = 0;
  for (int32_t it = 0;; ++it) {
    const int nf = qn[cur];
    if (nf == 0) break;
    if (it >= cap) {
      ctl[cStop] = 1;
      break;
    }
    const int nx = cur ^ 1;
    if (tid == 0) qn[nx] = 0;
    __syncthreads();
    expand_front(q[cur], nf, ooff, oadj, base, pre, ctl, [&](int32_t v, int32_t w) {
      if (w != v && (flg[w] & kValid) && atomicSub(&cnt_i[w], 1) == 1) claim_trim(w, nx);
    });
    expand_front(q[cur], nf, ioff, iadj, base, pre, ctl, [&](int32_t v, int32_t w) {
      if (w != v && (flg[w] & kValid) && atomicSub(&cnt_o[w], 1) == 1) claim_trim(w, nx);
    });
    cur = nx;
  }
  __syncthreads();

  // 2. FW-BW from the pivot
  {
    long long key = -1;
    int32_t id = 0x7fffffff;
    int32_t cnt = 0;
    for (int v = tid; v < n; v += kST) {
      if (flg[v] & kValid) {
        ++cnt;
        const long long k = (long long)cnt_o[v] * (long long)cnt_i[v];
        if (k > key || (k == key && v < id)) { key = k; id = v; }
      }
    }
    nvalid = block_sum(cnt, ctl);
    const int32_t pivot = block_argmax(key, id, ctl);
    if (!rest && nvalid > 0 && !ctl[cStop]) {
      for (int dir = 0; dir < 2; ++dir) {
        if (tid == 0) {
          flg[pivot] |= dir == 0 ? kFw : kBw;
          q[0][0] = pivot;
          qn[0] = 1;
        }
        __syncthreads();
        const int32_t* off = dir == 0 ? ooff : ioff;
        const int32_t* adj = dir == 0 ? oadj : iadj;
        const uint32_t want = dir == 0 ? kValid : (kValid | kFw);
        const uint32_t mask = dir == 0 ? (kValid | kFw) : (kValid | kFw | kBw);
        const uint32_t bit = dir == 0 ? kFw : kBw;
        cur = 0;
        for (int32_t it = 0;; ++it) {
          const int nf = qn[cur];
          if (nf == 0) break;
          if (it >= cap) {
            ctl[cStop] = 1;
            break;
          }
          const int nx = cur ^ 1;
          if (tid == 0) qn[nx] = 0;
          __syncthreads();
          expand_front(q[cur], nf, off, adj, base, pre, ctl, [&](int32_t v, int32_t w) {
            if ((flg[w] & mask) == want && !(atomicOr(&flg[w], bit) & bit))
              push(q[nx], &qn[nx], w);
          });
          cur = nx;
        }
        __syncthreads();
      }
      // the component: smallest member id as its label
      int32_t mn = 0x7fffffff;
      for (int v = tid; v < n; v += kST)
        if ((flg[v] & (kValid | kFw | kBw)) == (kValid | kFw | kBw)) mn = min(mn, v);
      mn = block_min(mn, ctl);
      int32_t cnt2 = 0;
      for (int v = tid; v < n; v += kST) {
        const uint32_t f = flg[v];
        if ((f & (kValid | kFw | kBw)) == (kValid | kFw | kBw)) {
          lab[v] = mn;
          flg[v] = 0;
          ++cnt2;
        } else {
          flg[v] = f & kValid;
        }
      }
      nvalid -= block_sum(cnt2, ctl);
    }
  }
  __syncthreads();

  // 3. colour rounds (at most colour_rounds), then signature rounds for what
  // is left
  int32_t* col = cnt_o;  // live degrees are not needed any more
  int32_t round = 0;
  for (; nvalid > 0 && !ctl[cStop] && round < colour_rounds; ++round) {
    if (round >= cap) {
      ctl[cStop] = 1;
      break;
    }
    if (tid == 0) qn[0] = 0;
    __syncthreads();
    for (int v = tid; v < n; v += kST) {
      if (flg[v] & kValid) {
        col[v] = v;
        flg[v] = kValid | kInq;
        push(q[0], &qn[0], v);
      }
    }
    __syncthreads();
    // min colour pushed along out-edges to the fixed point
    cur = 0;
    for (int32_t it = 0;; ++it) {
      const int nf = qn[cur];
      if (nf == 0) break;
      if (it >= cap) {
        ctl[cStop] = 1;
        break;
      }
      const int nx = cur ^ 1;
      if (tid == 0) qn[nx] = 0;
      for (int i = tid; i < nf; i += kST) atomicAnd(&flg[q[cur][i]], ~kInq);
      __syncthreads();
      expand_front(q[cur], nf, ooff, oadj, base, pre, ctl, [&](int32_t v, int32_t w) {
        if (!(flg[w] & kValid)) return;
        const int32_t cv = col[v];
        if (col[w] > cv && atomicMin(&col[w], cv) > cv && !(atomicOr(&flg[w], kInq) & kInq))
          push(q[nx], &qn[nx], w);
      });
      cur = nx;
    }
    if (ctl[cStop]) break;
    // roots, then the vertices of each root's colour that reach it
    if (tid == 0) qn[0] = 0;
    __syncthreads();
    for (int v = tid; v < n; v += kST) {
      if ((flg[v] & kValid) && col[v] == v) {
        flg[v] = kValid | kFw;
        push(q[0], &qn[0], v);
      }
    }
    __syncthreads();
    cur = 0;
    for (int32_t it = 0;; ++it) {
      const int nf = qn[cur];
      if (nf == 0) break;
      if (it >= cap) {
        ctl[cStop] = 1;
        break;
      }
      const int nx = cur ^ 1;
      if (tid == 0) qn[nx] = 0;
      __syncthreads();
      expand_front(q[cur], nf, ioff, iadj, base, pre, ctl, [&](int32_t v, int32_t w) {
        if ((flg[w] & (kValid | kFw)) == kValid && col[w] == col[v] &&
            !(atomicOr(&flg[w], kFw) & kFw))
          push(q[nx], &qn[nx], w);
      });
      cur = nx;
    }
    int32_t cnt3 = 0;
    for (int v = tid; v < n; v += kST) {
      if ((flg[v] & (kValid | kFw)) == (kValid | kFw)) {
        lab[v] = col[v];
        flg[v] = 0;
        ++cnt3;
      }
    }
    nvalid -= block_sum(cnt3, ctl);
  }
  // Signature rounds (a deep condensation, such as a long chain between
  // cycles, would take one colour round per component): each round, fw = the
  // smallest id reaching a vertex and bw = the smallest id it reaches, both
  // inside its class (kept in lab[] while the vertex is valid; one class at
  // first); fw == bw labels the vertex with that id, its SCC's smallest
  // member; the others take the pair as their class.
  if (nvalid > 0 && !ctl[cStop]) {
    int32_t* fw = cnt_o;
    int32_t* bw = cnt_i;
    for (int v = tid; v < n; v += kST)
      if (flg[v] & kValid) lab[v] = 0;
    __syncthreads();
    auto propagate = [&](int32_t* val, const int32_t* off, const int32_t* adj) {
      if (tid == 0) qn[0] = 0;
      __syncthreads();
      for (int v = tid; v < n; v += kST) {
        if (flg[v] & kValid) {
          val[v] = v;
          flg[v] = kValid | kInq;
          push(q[0], &qn[0], v);
        }
      }
      __syncthreads();
      cur = 0;
      for (int32_t it = 0;; ++it) {
        const int nf = qn[cur];
        if (nf == 0) break;
        if (it >= cap) {
          ctl[cStop] = 1;
          break;
        }
        const int nx = cur ^ 1;
        if (tid == 0) qn[nx] = 0;
        for (int i = tid; i < nf; i += kST) atomicAnd(&flg[q[cur][i]], ~kInq);
        __syncthreads();
        expand_front(q[cur], nf, off, adj, base, pre, ctl, [&](int32_t v, int32_t w) {
          if (!(flg[w] & kValid) || lab[w] != lab[v]) return;
          const int32_t cv = val[v];
          if (val[w] > cv && atomicMin(&val[w], cv) > cv && !(atomicOr(&flg[w], kInq) & kInq))
            push(q[nx], &qn[nx], w);
        });
        cur = nx;
      }
    };
    for (; nvalid > 0 && !ctl[cStop]; ++round) {
      if (round >= cap) {
        ctl[cStop] = 1;
        break;
      }
      propagate(fw, ooff, oadj);
      if (ctl[cStop]) break;
      propagate(bw, ioff, iadj);
      if (ctl[cStop]) break;
      int32_t cnt4 = 0;
      for (int v = tid; v < n; v += kST) {
        if (flg[v] & kValid) {
          const int32_t f = fw[v], b = bw[v];
          if (f == b) {
            lab[v] = f;
            flg[v] = 0;
            ++cnt4;
          } else {
            uint32_t x = (uint32_t)f * 0x9E3779B1u;
            x ^= (uint32_t)b * 0x85EBCA77u + 0x7F4A7C15u + (x << 6) + (x >> 2);
            lab[v] = (int32_t)x;
          }
        }
      }
      nvalid -= block_sum(cnt4, ctl);
    }
  }
}

// Components of an edge list in lab.  Rounds: every root hooks under the
// smallest root that an edge joins it to, one minimum per edge and no walk,
// then every vertex goes to its root.  A root that stays is the smallest among
// its neighbours and takes them in the round after, so their number falls by a
// constant factor in two rounds; the last round finds no edge between trees.
// Joining edge by edge with finds and compare-and-swaps, from the start or
// after the first round, makes the warps queue at the roots that their edges
// share.  A call with a host list (start to end, us):
//                            edge by edge   first round   rounds
//   R-MAT 4,000 / 52,000          108            78          68
//   R-MAT 6,000 / 56,000          142           109          93
//   random 5,000 / 20,000         108           123          55
//   random 5,000 / 65,000         155           295          70
//   path 5,000 / 4,999            230            38          40
// In CSR order the minima of a list meet in one word, and the plain joins are
// faster (92 against 128 us).  Returns false for an id outside [0, n).
__device__ __forceinline__ bool listed_wcc(const SmallDesc& D, int n, int32_t* lab, int32_t* ctl) {
  const volatile int32_t* const root = lab;
  for (int v = threadIdx.x; v < n; v += kST) lab[v] = v;
  __syncthreads();
  for (bool first = true;; first = false) {
    bool open = false;
    for_each_listed(D, [&](int32_t a, int32_t b, long long) {
      if ((unsigned)a >= (unsigned)n || (unsigned)b >= (unsigned)n) {
        if (first) ctl[cBad] = 1;  // (later: changed since)
        return;
      }
      // (the vertices themselves at first: a minimum of this round is no root)
      const int32_t x = first ? a : root[a], y = first ? b : root[b];
      if (x == y) return;
      atomicMin(&lab[max(x, y)], min(x, y));
      open = true;
    });
    // (every round that goes on has hooked a root: at most n of them)
    if (!__syncthreads_or(open) || ctl[cBad]) break;
    for (int v = threadIdx.x; v < n; v += kST) lab[v] = uf_find(lab, v);
    __syncthreads();
  }
  return !ctl[cBad];
}

// The run's status (one thread calls, once).  The kernel's own stores stand for
// two memsets, a latch kernel and two copies around it, which were 10 of the
// 50 us of a call.
__device__ __forceinline__ void small_status(const SmallStatus& st, bool many, int code) {
  if (many) {
    if (code) atomicCAS(st.err, 0, code);
    return;
  }
  st.err[0] = code;
  st.err[1] = 0;
  if (st.sticky) {
    if (st.clear) st.sticky[0] = st.sticky[1] = 0;
    else if (code && st.sticky[0] == 0) st.sticky[0] = code;
  }
  if (st.host) {
    st.host[0] = code;
    st.host[1] = 0;
  }
  if (st.tphase)
    for (int i = 0; i < 4; ++i) st.tphase[i] = 0;
}

template <int KIND>
__global__ void __launch_bounds__(kST, 1) k_small(SmallDesc one, const SmallDesc* many,
                                                  int32_t max_steps, int32_t colour_rounds,
                                                  SmallStatus st) {
  const SmallDesc D = many ? many[blockIdx.x] : one;
  const int n = D.n;
  if (n <= 0) return;
  const int tid = threadIdx.x;
  const SmallMem s = small_mem(n);
  int32_t* const ctl = s.ctl;
  int32_t* const ooff = s.ooff;
  int32_t* const ioff = s.ioff;
  int32_t* const lab = s.lab;
  int32_t* const cnt_o = s.cnt_o;
  int32_t* const cnt_i = s.cnt_i;
  const int32_t cap = (int32_t)min((long long)max_steps, 4ll * n + 64);
  if (tid == 0) {
    ctl[cBad] = 0;
    ctl[cStop] = 0;
  }

  // ---- WCC from an edge list: union-find over the edges, no CSR ----------
  if (KIND == 1 && D.out_off == nullptr) {
    __syncthreads();
    const bool fine = listed_wcc(D, n, lab, ctl);
    if (tid == 0) small_status(st, many != nullptr, fine ? 0 : (int)kErrInvalid);
    if (!fine) return;
    for (int v = tid; v < n; v += kST) D.labels[v] = uf_find(lab, v);
    return;
  }

  // ---- the CSR ------------------------------------------------------------
  SmallCsr g;
  if (D.out_off != nullptr) {
    const long long ob = D.out_off[0];
    const long long ib = D.in_off ? D.in_off[0] : ob;
    for (int v = tid; v <= n; v += kST) {
      ooff[v] = (int32_t)(D.out_off[v] - ob);
      ioff[v] = D.in_off ? (int32_t)(D.in_off[v] - ib) : ooff[v];
    }
    g.oadj = D.out_adj + ob;
    g.iadj = D.in_off ? D.in_adj + ib : g.oadj;
    g.base = D.id_base;
  } else {
    for (int v = tid; v < n; v += kST) {
      cnt_o[v] = 0;
      cnt_i[v] = 0;
    }
    __syncthreads();
    for_each_listed(D, [&](int32_t a, int32_t b, long long e) {
      D.keep(e, a, b);
      if ((unsigned)a >= (unsigned)n || (unsigned)b >= (unsigned)n) {
        ctl[cBad] = 1;
      } else {
        atomicAdd(&cnt_o[a], 1);
        atomicAdd(&cnt_i[b], 1);
      }
    });
    __syncthreads();
    if (ctl[cBad]) {
      if (tid == 0) small_status(st, many != nullptr, (int)kErrInvalid);
      return;
    }
    for (int v = tid; v < n; v += kST) {
      ooff[v] = cnt_o[v];
      ioff[v] = cnt_i[v];
    }
    if (tid == 0) {
      ooff[n] = 0;
      ioff[n] = 0;
    }
    block_scan(ooff, n + 1, ctl);
    block_scan(ioff, n + 1, ctl);
    for (int v = tid; v < n; v += kST) {
      cnt_o[v] = ooff[v];
      cnt_i[v] = ioff[v];
    }
    __syncthreads();
    int32_t* so = D.adj_scratch;
    int32_t* si = D.adj_scratch + D.m;
    // (each thread reads the pairs that it kept; a call took as long with the
    // list read twice, 45.3 us at 300 vertices and 101 at 3,000)
    for_each_listed(D.again(), [&](int32_t a, int32_t b, long long) {
      so[atomicAdd(&cnt_o[a], 1)] = b;
      si[atomicAdd(&cnt_i[b], 1)] = a;
    });
    __syncthreads();
    g.oadj = so;
    g.iadj = si;
    g.base = 0;
  }
  g.ooff = ooff;
  g.ioff = ioff;

  // ---- WCC on a CSR: union-find over the out-lists ------------------------
  if (KIND == 1) {
    for (int v = tid; v < n; v += kST) lab[v] = v;
    __syncthreads();
    for_each_edge(n, ooff, g.oadj, g.base, [&](int32_t u, int32_t w) { uf_unite(lab, u, w); });
    __syncthreads();
    for (int v = tid; v < n; v += kST) D.labels[v] = uf_find(lab, v);
    if (tid == 0) small_status(st, many != nullptr, 0);
    return;
  }

  // ---- SCC ----------------------------------------------------------------
  __syncthreads();  // the offsets, from here on read across threads
  int32_t nvalid = -1;
  int32_t hub = -1;
  if (colour_rounds == kSigAfterSmall && steps_free(max_steps, n)) {
    // the vertex of largest out x in degree, among those with kHubDeg on
    // both sides
    long long key = -1;
    int32_t id = 0x7fffffff;
    for (int v = tid; v < n; v += kST) {
      const int32_t od = ooff[v + 1] - ooff[v], idg = ioff[v + 1] - ioff[v];
      const long long k = (long long)od * (long long)idg;
      if (min(od, idg) >= kHubDeg && k > key) { key = k; id = v; }
    }
    if (__syncthreads_or(key >= 0)) hub = block_argmax(key, id, ctl);
  }
  if (hub >= 0)
    nvalid = hub_scc(n, hub, g.oadj, g.iadj, g.base, cap);
  if (nvalid != 0) queue_scc(n, g.oadj, g.iadj, g.base, cap, colour_rounds, nvalid);
  __syncthreads();
  const bool stopped = ctl[cStop] != 0;
  if (tid == 0) small_status(st, many != nullptr, stopped ? (int)kErrIterLimit : 0);
  if (stopped) return;
  for (int v = tid; v < n; v += kST) D.labels[v] = lab[v];
}

template <int KIND>
cudaError_t launch_k(const SmallDesc& one, const SmallDesc* many, int count, int32_t max_n,
                     int32_t max_steps, int32_t colour_rounds, const SmallStatus& st,
                     cudaStream_t s) {
  // the shared-memory attribute, once per device
  static bool attr_set[64][2] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const size_t smem = small_smem_bytes(KIND, max_n);
  if (dev < 0 || dev >= 64 || !attr_set[dev][KIND]) {
    e = cudaFuncSetAttribute(k_small<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)small_smem_bytes(KIND, kSmallMaxN));
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) attr_set[dev][KIND] = true;
  }
  k_small<KIND><<<count, kST, smem, s>>>(one, many, max_steps, colour_rounds, st);
  return cudaGetLastError();
}

}  // namespace

size_t small_smem_bytes(int kind, int32_t max_n) {
  const size_t n = (size_t)(max_n > 0 ? max_n : 1);
  const size_t all = (size_t)kCtlInts * 4 + (9 * n + 3) * 4;
  // (offsets, labels and flags stay beside hub_scc's memory)
  const size_t hub = (size_t)kCtlInts * 4 + (4 * n + 2 + 4) * 4 + kHubSmem;
  return kind == 1 || all > hub ? all : hub;
}

cudaError_t launch_small(int kind, const SmallDesc& one, const SmallDesc* many, int count,
                         int32_t max_n, int32_t max_steps, const SmallStatus& st, cudaStream_t s,
                         int32_t colour_mode) {
  if (count <= 0) return cudaSuccess;
  if (max_n > kSmallMaxN) return cudaErrorInvalidValue;
  // colour rounds before the signature rounds: all (0), none (1), four (2)
  const int32_t cr = colour_mode == 0 ? 0x7fffffff : (colour_mode == 1 ? 0 : kSigAfterSmall);
  return kind == 0 ? launch_k<0>(one, many, count, max_n, max_steps, cr, st, s)
                   : launch_k<1>(one, many, count, max_n, max_steps, cr, st, s);
}

}  // namespace gb
