// SCC by graph contraction, for graphs without hubs.
//
// Searches and propagations follow a path one hop at a time, so on a graph
// of high diameter (lattices, road networks, long chains) they are bound by
// the number of hops times the latency of one.  Contraction has no such
// chain: every round removes a constant share of the vertices whatever their
// distance.  The operations are those of Levy and Low, "A contraction
// algorithm for finding small cycle cutsets" (Journal of Algorithms 9, 1988),
// applied to components instead of cutsets:
//   IN0 / OUT0  a vertex without an in-edge (out-edge) is a component alone
//               (scc_trim_complete, multistep/scc_trim.cpp:141-297);
//   LOOP        edges inside a merged vertex are dropped;
//   2-cycle     u -> v and v -> u: both are in one component, merged;
//   IN1 / OUT1  a vertex v whose in-edges all come from one vertex u (whose
//               out-edges all go to one u) is merged into u.  Every path
//               between other vertices that passes v passes u, so no other
//               vertex's reachability changes; whether v itself belongs to
//               u's component is settled afterwards.
// Round t keeps the edge list E_t over the vertices alive in it (A_t), and
// alternates IN1 (t even) and OUT1 (t odd).  Its passes, a barrier after
// each:
//   P1  per edge: smallest and largest in-neighbour of its head and
//       out-neighbour of its tail.  None: IN0 / OUT0; equal: IN1 / OUT1; one
//       of the two in common between the two sides: a 2-cycle (others are
//       found in later rounds, once merging has brought them to an end);
//   P2  per vertex: dead vertices marked, 2-cycles joined by union-find;
//   P3  per vertex: a vertex of a 2-cycle takes its root; any other IN1 /
//       OUT1 vertex v hooks onto u, unless u hooks itself and the order of
//       their ids (by turns rising and falling) or a hash of v says no:
//       hooks then form trees, never cycles, of a depth of a few dozen on
//       average; the others form A_{t+1};
//   P4  per edge: its ends are replaced by their roots, edges inside a root
//       or at a dead one dropped, the rest is E_{t+1}; the edges that will
//       settle this round's hooked vertices (their out-edges for IN1,
//       in-edges for OUT1) go to a log.
// Then the rounds are undone in reverse: with the components of A_{t+1}
// known, a vertex v that IN1 hooked in round t belongs to its root's
// component exactly when one of v's out-edges, or one of a vertex hooked
// below it, leads to a vertex of that component (OUT1: in-edges); otherwise
// it is a component of its own.  Labels are the smallest members.
//
// A round shrinks the 1024^2 lattice of the benchmark by a factor of two to
// three, so about 20 rounds replace some 27,000 dependent hops: 111 ms ->
// 1.1 ms of device time (the first round takes a quarter of it, each of the
// small ones 35 us of grid barriers and dependent L2 reads, the tail in one
// block 110 us).  When a round drops less than a fifth of the edges before the
// tail takes the rest, every vertex goes back to the searches and rounds:
// one-way street lattices, the cores of random graphs, but also lattices of some
// 2,048 a side (for two seeds in five 2.8 ms becomes 155 ms) and more, and
// chains of more than some 65,000 vertices numbered in order, where every other
// pair of rounds runs against the ids.
#pragma once
#include "run_device.cuh"

namespace gb {
namespace {

constexpr int32_t kConInf = 0x7fffffff;
constexpr int32_t kConOpen = -2;  // component not known (left to later phases)
// states of a vertex: kind, and the round it left the contraction in
enum : uint32_t { kConAlive = 0u, kConDead = 1u, kConUnion = 2u, kConHook = 3u };
constexpr uint32_t kConPos = 0x80000000u;  // hooked vertex in its root's component
__device__ __forceinline__ uint32_t con_state(int t, uint32_t kind) {
  return ((uint32_t)(t + 1) << 2) | kind;
}
// From these sizes down one block runs the rounds on a copy of the graph in
// its shared memory: a round then costs a few block barriers and
// shared-memory accesses instead of four grid barriers and chains of L2
// accesses (37 us a round on small lattices).
constexpr int32_t kConTailVerts = 1024;
constexpr int32_t kConTailEdges = 3072;
constexpr int32_t kConTailLog = 2560;
// One hook in kConCut that would extend a chain of hooks is left out, which
// bounds the trees' depth (the marking pass walks it).
constexpr uint32_t kConCut = 64;

// Where the passes run: the whole grid on arrays in global memory (read
// through L2), or one block on arrays in its shared memory.
struct ConGrid {
  static constexpr bool kStaged = true;
  Ctl* c;
  Steps* st;
  int32_t max_steps;
  __device__ __forceinline__ long long tid() const {
    return (long long)blockIdx.x * blockDim.x + threadIdx.x;
  }
  __device__ __forceinline__ long long threads() const {
    return (long long)gridDim.x * blockDim.x;
  }
  // Loads go through L1, where the words every warp ends at (a large
  // component's root, a hub's extremes) are served per SM instead of one
  // request at a time by L2.  The barrier after each pass drops what L1 holds
  // from before it; within a pass a stale value is an older extreme or
  // ancestor, which costs work only.  fresh() is for the union-find.
  template <class T>
  static __device__ __forceinline__ T ld(const T* p) { return __ldca(p); }
  template <class T>
  static __device__ __forceinline__ T fresh(const T* p) { return __ldcg(p); }
  __device__ __forceinline__ bool sync(int where) const {
    if (st->s - st->s0 >= max_steps) {
      set_err(c, kErrIterLimit, where);
      return false;
    }
    return step_sync(c, *st, where);
  }
};
struct ConBlock {
  static constexpr bool kStaged = false;
  volatile int* left;  // shared: steps this block may still take, < 0: too many
  __device__ __forceinline__ long long tid() const { return threadIdx.x; }
  __device__ __forceinline__ long long threads() const { return blockDim.x; }
  template <class T>
  static __device__ __forceinline__ T ld(const T* p) { return *(const volatile T*)p; }
  template <class T>
  static __device__ __forceinline__ T fresh(const T* p) { return *(const volatile T*)p; }
  static __device__ __forceinline__ int2 ld(const int2* p) {
    const volatile int* q = reinterpret_cast<const volatile int*>(p);
    return make_int2(q[0], q[1]);
  }
  __device__ __forceinline__ bool sync(int) const {
    __syncthreads();
    if (threadIdx.x == 0) --*left;
    __syncthreads();
    return *left >= 0;
  }
};

// A warp's staging of pairs in its shared memory, flushed with one atomic.
struct ConStage {
  unsigned long long* buf;
  int cap;
  int n;
};
__device__ __forceinline__ void con_flush(ConStage& s, unsigned long long* arr, long long base,
                                          long long dir, long long cap, append_count* counter,
                                          int32_t* over) {
  __syncwarp();
  if (s.n > 0) {
    append_count pos = 0;
    if (lane_id() == 0) pos = atomicAdd(counter, (append_count)s.n);
    pos = __shfl_sync(kFull, pos, 0);
    for (int i = lane_id(); i < s.n; i += 32) {
      const long long at = append_slot(pos, (unsigned)i, cap);
      if (at >= 0) arr[base + dir * at] = s.buf[i];
      else *over = 1;
    }
  }
  __syncwarp();
  s.n = 0;
}
template <bool kStaged>
__device__ __forceinline__ void con_push(ConStage& s, bool flag, int32_t a, int32_t b,
                                         unsigned long long* arr, long long base, long long dir,
                                         long long cap, append_count* counter, int32_t* over) {
  const unsigned mask = __ballot_sync(kFull, flag);
  if (mask == 0u) return;
  const int cnt = __popc(mask);
  if constexpr (!kStaged) {
    append_count pos = 0;
    if (lane_id() == 0) pos = atomicAdd(counter, (append_count)cnt);
    pos = __shfl_sync(kFull, pos, 0);
    if (flag) {
      const long long at = append_slot(pos, (unsigned)__popc(mask & lanemask_lt()), cap);
      if (at >= 0) arr[base + dir * at] = ((unsigned long long)(uint32_t)a << 32) | (uint32_t)b;
      else *over = 1;
    }
    return;
  }
  if (s.n + cnt > s.cap) con_flush(s, arr, base, dir, cap, counter, over);
  if (flag)
    s.buf[s.n + __popc(mask & lanemask_lt())] =
        ((unsigned long long)(uint32_t)a << 32) | (uint32_t)b;
  s.n += cnt;
}
// One value per flagged lane appended to arr, one atomic per warp.
__device__ __forceinline__ void con_append(bool flag, int32_t v, int32_t* arr, int32_t* counter) {
  const unsigned mask = __ballot_sync(kFull, flag);
  if (mask == 0u) return;
  const int leader = __ffs(mask) - 1;
  int pos = 0;
  if ((int)lane_id() == leader) pos = atomicAdd(counter, __popc(mask));
  pos = __shfl_sync(kFull, pos, leader);
  if (flag) arr[pos + __popc(mask & lanemask_lt())] = v;
}

template <class W>
__device__ __forceinline__ void con_minmax(int2* p, int32_t x) {
  const int2 c = W::ld(p);
  if (x < c.x) atomicMin(&p->x, x);
  if (x > c.y) atomicMax(&p->y, x);
}

// No walk is longer than its tree is deep; the bound ends one over a damaged
// tree too.
constexpr int kConWalk = 1 << 22;

// Root of x (its tree complete), with path halving; dead roots are < 0.
template <class W>
__device__ __forceinline__ int32_t con_root(int32_t* par, int32_t x) {
  int32_t p = W::ld(par + x);
  for (int it = 0; p >= 0 && p != x && it < kConWalk; ++it) {
    const int32_t q = W::ld(par + p);
    if (q < 0) return q;
    if (q != p) par[x] = q;
    x = p;
    p = q;
  }
  return p;
}
// Joins the trees of a and b, the larger root under a smaller vertex of the
// other tree (a root is its tree's smallest id, so a vertex smaller than a
// root is never below it): only the larger side has to be a root now.
template <class W>
__device__ __forceinline__ void con_unite(int32_t* par, int32_t a, int32_t b) {
  a = con_root<W>(par, a);
  b = con_root<W>(par, b);
  while (a != b) {
    const int32_t lo = a < b ? a : b, hi = a < b ? b : a;
    const int32_t p = W::fresh(par + hi);
    if (p == hi && atomicCAS(par + hi, hi, lo) == hi) return;
    a = lo;
    b = p == hi ? W::fresh(par + hi) : p;
  }
}

// The arrays of one contraction.  E_t is arena[i] for t odd and
// arena[acap - 1 - i] for t even (t >= 1), so that E_t and E_{t+1} grow
// towards each other; E_0 is given by the caller.
struct Contract {
  int2* in;    // smallest and largest in-neighbour
  int2* out;   // smallest and largest out-neighbour
  int32_t* par;
  int32_t* tc;      // hooked vertices: the vertex hooked onto; then components
  uint32_t* info;   // con_state, 0 while alive
  int32_t* A[2];    // alive vertices (A_0: list0, or 0..n0-1 when null)
  int32_t* D;       // vertices merged, in order of rounds
  const int32_t* list0;
  int32_t n0;
  unsigned long long* arena;
  long long acap;
  unsigned long long* elog;
  long long lcap;
  // per round: |A_t|, |E_t|, end of D and of the log after round t
  int32_t* cntA;
  append_count* cntE;
  int32_t* cntD;
  append_count* cntL;
  int32_t* over;    // an array ran out: the round is undone
};

template <class W>
__device__ __forceinline__ int32_t con_vertex(const Contract& k, int t, long long i) {
  if (t > 0) return W::ld(k.A[t & 1] + i);
  return k.list0 ? W::ld(k.list0 + i) : (int32_t)i;
}

// Calls f(s, d, active) warp-collectively for every edge of E_t.
// Src::edges(t = 0) enumerates the caller's edges.
template <class Src, class W, class F>
__device__ __forceinline__ void con_edges(const Contract& k, const Src& src, const W& w, int t,
                                          F f) {
  if (t == 0) {
    src.edges(w, f);
    return;
  }
  // (an append past the capacity is counted but not written, and ends the
  // rounds; the bound keeps even its reader inside the array)
  const long long ne = min((long long)W::ld(k.cntE + t), k.acap);
  const long long nth = w.threads();
  constexpr int kU = 4;
  for (long long b = w.tid() & ~31ll; b < ne; b += nth * kU) {
    unsigned long long e[kU];
#pragma unroll
    for (int q = 0; q < kU; ++q) {
      const long long i = b + q * nth + lane_id();
      e[q] = i < ne ? W::ld((t & 1) ? k.arena + i : k.arena + (k.acap - 1 - i)) : ~0ull;
    }
#pragma unroll
    for (int q = 0; q < kU; ++q)
      if (b + q * nth < ne) f((int32_t)(e[q] >> 32), (int32_t)(uint32_t)e[q], e[q] != ~0ull);
  }
}

// Round t.  Returns false on an error.
template <class Src, class W>
__device__ __noinline__ bool con_round(const Contract& k, const Src& src, const W& w, int t,
                                       unsigned long long* stage) {
  const long long tid = w.tid(), nth = w.threads();
  const int32_t na = t == 0 ? k.n0 : W::ld(k.cntA + t);
  // P1
  con_edges(k, src, w, t, [&](int32_t s, int32_t d, bool act) {
    if (act) {
      con_minmax<W>(k.out + s, d);
      con_minmax<W>(k.in + d, s);
    }
  });
  if (!w.sync(410)) return false;
  // P2
  for (long long i = tid; i < na; i += nth) {
    const int32_t v = con_vertex<W>(k, t, i);
    const int2 in = W::ld(k.in + v), out = W::ld(k.out + v);
    if (in.y < 0 || out.y < 0) {
      k.info[v] = con_state(t, kConDead);
      k.par[v] = ~v;
      k.tc[v] = v;
      continue;
    }
    const bool lo = in.x == out.x || in.x == out.y;
    const bool hi = in.y != in.x && (in.y == out.x || in.y == out.y);
    if (lo || hi) {
      k.info[v] = con_state(t, kConUnion);
      if (lo) {
        k.info[in.x] = con_state(t, kConUnion);
        con_unite<W>(k.par, v, in.x);
      }
      if (hi) {
        k.info[in.y] = con_state(t, kConUnion);
        con_unite<W>(k.par, v, in.y);
      }
    }
  }
  if (!w.sync(411)) return false;
  // P3
  const int2* side = (t & 1) ? k.out : k.in;
  const uint32_t stU = con_state(t, kConUnion), stD = con_state(t, kConDead);
  const bool rising = ((t >> 1) & 1) == 0;
  for (long long b = tid & ~31ll; b < na; b += nth) {
    const long long i = b + lane_id();
    bool alive = false, gone = false;
    int32_t v = 0;
    if (i < na) {
      v = con_vertex<W>(k, t, i);
      const uint32_t st = W::ld(k.info + v);
      if (st == stU) {
        const int32_t r = con_root<W>(k.par, v);
        gone = r != v;
        alive = !gone;
        if (gone) k.par[v] = r;
      } else if (st != stD) {
        const int2 sv = W::ld(side + v);
        alive = true;
        if (sv.x == sv.y) {
          const int32_t u = sv.x;
          const uint32_t su = W::ld(k.info + u);
          const int2 uv = W::ld(side + u);
          const bool umoves = su != stU && su != stD && uv.x == uv.y;
          const bool cut = (((uint32_t)v * 0x9E3779B1u) >> 16) % kConCut == 0u;
          if (!umoves || (rising == (u < v) && !cut)) {
            const int32_t g = su == stU ? con_root<W>(k.par, u) : u;
            k.tc[v] = g;
            k.par[v] = g;
            k.info[v] = con_state(t, kConHook);
            alive = false;
            gone = true;
          }
        }
      }
    }
    con_append(alive, v, k.A[(t + 1) & 1], k.cntA + t + 1);
    con_append(gone, v, k.D, k.cntD);
  }
  if (!w.sync(412)) return false;
  // P4
  const int32_t na1 = W::ld(k.cntA + t + 1);
  for (long long i = tid; i < na1; i += nth) {
    const int32_t v = W::ld(k.A[(t + 1) & 1] + i);
    k.in[v] = make_int2(kConInf, -1);
    k.out[v] = make_int2(kConInf, -1);
    k.info[v] = 0u;
  }
  if (tid == 0) k.cntD[t + 1] = W::ld(k.cntD);
  {
    const uint32_t stH = con_state(t, kConHook);
    const long long ebase = (t + 1) & 1 ? 0 : k.acap - 1, edir = (t + 1) & 1 ? 1 : -1;
    const long long ecap = k.acap - (t > 0 ? (long long)W::ld(k.cntE + t) : 0);
    ConStage se{stage, 256, 0}, sl{stage + 256, 160, 0};
    con_edges(k, src, w, t, [&](int32_t s, int32_t d, bool act) {
      bool keep = false, lg = false;
      int32_t rs = 0, rd = 0;
      if (act) {
        rs = con_root<W>(k.par, s);
        rd = con_root<W>(k.par, d);
        keep = rs >= 0 && rd >= 0 && rs != rd;
        // an edge between live vertices that did not move has no say in the log
        const int32_t a = (t & 1) ? d : s, o = (t & 1) ? s : d;
        if ((((t & 1) ? rd : rs) != a) && W::ld(k.info + a) == stH && W::ld(k.info + o) != stH)
          lg = true;
      }
      con_push<W::kStaged>(se, keep, rs, rd, k.arena, ebase, edir, ecap, k.cntE + t + 1, k.over);
      con_push<W::kStaged>(sl, lg, (t & 1) ? d : s, (t & 1) ? s : d, k.elog, 0, 1, k.lcap, k.cntL, k.over);
    });
    if constexpr (W::kStaged) {
      con_flush(se, k.arena, ebase, edir, ecap, k.cntE + t + 1, k.over);
      con_flush(sl, k.elog, 0, 1, k.lcap, k.cntL, k.over);
    }
  }
  if (!w.sync(413)) return false;
  if (tid == 0) k.cntL[t + 1] = W::ld(k.cntL);
  return true;
}

// The vertex that v was merged into in round t (v itself when it was not).
template <class W>
__device__ __forceinline__ int32_t con_root_at(const Contract& k, int t, int32_t v) {
  const uint32_t h = con_state(t, kConHook), u = con_state(t, kConUnion);
  for (int it = 0; it < kConWalk; ++it) {
    const uint32_t s = W::ld(k.info + v) & ~kConPos;
    if (s != h && s != u) break;
    v = W::ld(k.par + v);
  }
  return v;
}

// Undoes round t: the components of the vertices merged in it.
template <class W>
__device__ __noinline__ bool con_undo(const Contract& k, const W& w, int t) {
  const long long tid = w.tid(), nth = w.threads();
  const uint32_t stH = con_state(t, kConHook);
  const long long l0 = t > 0 ? (long long)W::ld(k.cntL + t) : 0;
  const long long l1 = min((long long)W::ld(k.cntL + t + 1), k.lcap);
  const int32_t d0 = t > 0 ? W::ld(k.cntD + t) : 0, d1 = W::ld(k.cntD + t + 1);
  for (long long i = l0 + tid; i < l1; i += nth) {
    const unsigned long long e = W::ld(k.elog + i);
    const int32_t a = (int32_t)(e >> 32), b = (int32_t)(uint32_t)e;
    const int32_t cr = W::ld(k.tc + con_root_at<W>(k, t, a));
    const int32_t cb = W::ld(k.tc + con_root_at<W>(k, t, b));
    if (cr < 0 || cb != cr) continue;
    for (int32_t x = a; (W::ld(k.info + x) & ~kConPos) == stH; x = W::ld(k.tc + x))
      if (atomicOr(k.info + x, kConPos) & kConPos) break;
  }
  if (!w.sync(420)) return false;
  for (long long i = d0 + tid; i < d1; i += nth) {
    const int32_t v = W::ld(k.D + i);
    const int32_t r = con_root_at<W>(k, t, v);
    const int32_t c = W::ld(k.tc + r);
    const uint32_t s = W::ld(k.info + v);
    // (tc of a vertex hooked in this round is read by the marking pass only)
    k.tc[v] = s == stH && c != kConOpen ? v : c;
  }
  return w.sync(421);
}

// Vertices left when the contraction stops have no component yet.
template <class W>
__device__ __forceinline__ void con_open(const Contract& k, const W& w, int t, bool undone) {
  const int32_t na = W::ld(k.cntA + t);
  for (long long i = w.tid(); i < na; i += w.threads()) k.tc[con_vertex<W>(k, t, i)] = kConOpen;
  if (!undone) return;
  // (an array ran out in round t - 1: what it merged stays open too)
  const int32_t d0 = t > 1 ? W::ld(k.cntD + t - 1) : 0, d1 = W::ld(k.cntD + t);
  for (long long i = d0 + w.tid(); i < d1; i += w.threads()) k.tc[W::ld(k.D + i)] = kConOpen;
}

// Whether another round pays after round t - 1 (t >= 1): that round dropped
// a fifth of the edges.  Lattices drop 40 to 60 % of their edges a round,
// uniform random graphs of three or more edges per vertex under 15 %.
template <class W>
__device__ __forceinline__ bool con_pays(const Contract& k, int t, long long e0) {
  if (t >= kConRounds || W::ld(k.over)) return false;
  const long long before = t == 1 ? e0 : (long long)W::ld(k.cntE + t - 1);
  return (long long)W::ld(k.cntE + t) * 5 <= before * 4;
}

// Edges of E_t between the tail's local ids (tc of a vertex alive in round t).
struct ConLocal {
  const Contract* k;
  int t;
  template <class W, class F>
  __device__ __forceinline__ void edges(const W& w, F f) const {
    const int32_t ne = (int32_t)__ldcg(k->cntE + t);  // (at most kConTailEdges)
    for (int32_t b = (int32_t)w.tid() & ~31; b < ne; b += (int32_t)w.threads()) {
      const int32_t i = b + (int32_t)lane_id();
      int32_t s = 0, d = 0;
      if (i < ne) {
        const unsigned long long e = __ldcg((t & 1) ? k->arena + i : k->arena + (k->acap - 1 - i));
        s = __ldcg(k->tc + (e >> 32));
        d = __ldcg(k->tc + (uint32_t)e);
      }
      f(s, d, i < ne);
    }
  }
};

// The components of a core that the rounds do not shrink, by signatures
// (signature_rounds, on the block's own edge list): the smallest id reaching
// a vertex (in.x) and the smallest id it reaches (in.y), inside classes
// (out.x) of equal pairs; a vertex whose two agree is in that id's component.
template <class W>
__device__ __forceinline__ bool con_core(const Contract& k, const W& w, int t, volatile int* flag) {
  const int32_t na = W::ld(k.cntA + t), ne = (int32_t)W::ld(k.cntE + t);
  const int tid = (int)w.tid(), nth = (int)w.threads();
  for (int i = tid; i < na; i += nth) {
    const int32_t v = con_vertex<W>(k, t, i);
    k.out[v].x = 0;
    k.tc[v] = kConOpen;
  }
  for (;;) {
    if (tid == 0) *flag = 0;
    __syncthreads();
    for (int i = tid; i < na; i += nth) {
      const int32_t v = con_vertex<W>(k, t, i);
      if (W::ld(k.tc + v) != kConOpen) continue;
      k.in[v] = make_int2(v, v);
      *flag = 1;
    }
    if (!w.sync(431)) return false;
    if (*flag == 0) return true;
    for (;;) {
      __syncthreads();
      if (tid == 0) *flag = 0;
      __syncthreads();
      for (int i = tid; i < ne; i += nth) {
        const unsigned long long e = W::ld((t & 1) ? k.arena + i : k.arena + (k.acap - 1 - i));
        const int32_t s = (int32_t)(e >> 32), d = (int32_t)(uint32_t)e;
        if (W::ld(&k.out[s].x) != W::ld(&k.out[d].x) || W::ld(k.tc + s) != kConOpen ||
            W::ld(k.tc + d) != kConOpen)
          continue;
        const int32_t f = W::ld(&k.in[s].x), bk = W::ld(&k.in[d].y);
        if (f < W::ld(&k.in[d].x)) {
          atomicMin(&k.in[d].x, f);
          *flag = 1;
        }
        if (bk < W::ld(&k.in[s].y)) {
          atomicMin(&k.in[s].y, bk);
          *flag = 1;
        }
      }
      if (!w.sync(432)) return false;
      if (*flag == 0) break;
    }
    __syncthreads();
    for (int i = tid; i < na; i += nth) {
      const int32_t v = con_vertex<W>(k, t, i);
      if (W::ld(k.tc + v) != kConOpen) continue;
      const int2 p = W::ld(k.in + v);
      if (p.x == p.y) k.tc[v] = p.x;
      else k.out[v].x = sig_class(p.x, p.y);
    }
    __syncthreads();
  }
}

// One block's contraction of a graph of n <= V vertices (ids 0 to n - 1) in
// con_bytes(V, E, L) bytes of its shared memory; src enumerates the edges, at
// most E; L entries of log.  Afterwards comp[i] (in smem, valid until it is reused)
// is the component of vertex i, the id of one of its members, or kConOpen
// when the log ran out.  *left: steps the block may still take; negative
// afterwards when they ran out (comp is then not set).
constexpr int32_t con_bytes(int32_t V, int32_t E, int32_t L) { return V * 40 + (2 * E + L) * 8; }
template <int32_t V, int32_t E, int32_t L, class Src>
__device__ __noinline__ void con_solve(const Src& src, int32_t n, int32_t* smem,
                                       volatile int* left, int32_t** comp) {
  __shared__ int s_flag;
  __shared__ int32_t s_cnt[2][kConRounds + 2];
  __shared__ append_count s_ecnt[2][kConRounds + 2];
  __shared__ int32_t s_over;
  const int tid = threadIdx.x, nth = blockDim.x;
  Contract l;
  l.arena = reinterpret_cast<unsigned long long*>(smem);
  l.acap = 2 * E;  // E_u and E_{u+1} always fit
  l.elog = l.arena + 2 * E;
  l.lcap = L;
  l.in = reinterpret_cast<int2*>(l.elog + L);
  l.out = l.in + V;
  l.par = reinterpret_cast<int32_t*>(l.out + V);
  l.tc = l.par + V;
  l.info = reinterpret_cast<uint32_t*>(l.tc + V);
  l.A[0] = l.tc + 2 * V;
  l.A[1] = l.A[0] + V;
  l.D = l.A[1] + V;
  l.list0 = nullptr;
  l.n0 = n;
  l.cntA = s_cnt[0];
  l.cntD = s_cnt[1];
  l.cntE = s_ecnt[0];
  l.cntL = s_ecnt[1];
  l.over = &s_over;
  *comp = l.tc;
  if (tid == 0) s_over = 0;
  for (int i = tid; i < 2 * (kConRounds + 2); i += nth) {
    (&s_cnt[0][0])[i] = 0;
    (&s_ecnt[0][0])[i] = 0;
  }
  for (int i = tid; i < n; i += nth) {
    l.in[i] = make_int2(kConInf, -1);
    l.out[i] = make_int2(kConInf, -1);
    l.par[i] = i;
    l.info[i] = 0u;
  }
  __syncthreads();
  const ConBlock b{left};
  int u = 0;
  bool ok = true;
  for (;;) {
    if (u > 0 && (ConBlock::ld(l.cntA + u) == 0 || ConBlock::ld(l.over) || u >= kConRounds)) break;
    // (rounds go on while two of them drop a tenth of the vertices)
    if (u > 2 && ConBlock::ld(l.cntA + u) * 10 > ConBlock::ld(l.cntA + u - 2) * 9) break;
    if (!con_round(l, src, b, u, nullptr)) { ok = false; break; }
    ++u;
    __syncthreads();
  }
  const bool undone = ok && s_over != 0;
  if (ok && undone) {
    con_open(l, b, u, true);
    __syncthreads();
  } else if (ok && ConBlock::ld(l.cntA + u) > 0) {
    ok = con_core(l, b, u, &s_flag);
  }
  __syncthreads();
  for (int x = u - (undone ? 2 : 1); ok && x >= 0; --x) ok = con_undo(l, b, x);
}

// The tail: block 0 finishes the graph of round t (at most kConTailVerts
// vertices and kConTailEdges edges) and leaves a component or kConOpen in tc
// for every vertex of A_t.
constexpr int32_t kConTailBytes = con_bytes(kConTailVerts, kConTailEdges, kConTailLog);
static_assert(kConTailBytes + kConTailVerts * 4 <= kDynSmem,
              "the tail's arrays fit the dynamic shared memory");
__device__ __forceinline__ void con_tail(const Contract& k, int t, int32_t steps_left,
                                         int32_t* smem, int32_t* rounds) {
  __shared__ int s_left;
  int32_t* const gid = smem + kConTailBytes / 4;
  const int tid = threadIdx.x, nth = blockDim.x;
  const int32_t n = __ldcg(k.cntA + t);
  if (tid == 0) s_left = steps_left;
  for (int i = tid; i < n; i += nth) {
    const int32_t v = __ldcg(k.A[t & 1] + i);
    gid[i] = v;
    k.tc[v] = i;
  }
  __syncthreads();
  int32_t* comp;
  con_solve<kConTailVerts, kConTailEdges, kConTailLog>(ConLocal{&k, t}, n, smem, &s_left, &comp);
  // (out of steps, all of it is left to the rounds, which have a cap of their own)
  const bool ok = s_left >= 0;
  for (int i = tid; i < n; i += nth) {
    const int32_t x = ok ? comp[i] : kConOpen;
    k.tc[gid[i]] = x < 0 ? kConOpen : gid[x];
  }
  // (all of this is one round to the caller: how many it took depends on the
  // order in which the vertices were appended)
  if (tid == 0) *rounds = t + 1;
}

// The whole contraction: rounds until no vertex is alive or they stop
// paying, then their reversal.  On entry in / out / par / info hold a fresh
// state for the n0 vertices and a barrier has passed; e0 is a bound on the
// edges of E_0.  On return tc holds a component (the id of one of its
// vertices) or kConOpen for every vertex; *rounds the rounds run.  All
// blocks call; returns false on an error.
template <class Src>
__device__ __noinline__ bool contract_run(const Contract& k, const Src& src, Ctl* c, Steps& st,
                                          int32_t max_steps, long long e0, int32_t* smem,
                                          unsigned long long* stage, int32_t* rounds) {
  const ConGrid g{c, &st, max_steps};
  int t = 0;
  bool small = false, pays = true;
  for (;;) {
    const long long na = t == 0 ? (long long)k.n0 : (long long)__ldcg(k.cntA + t);
    if (na == 0) break;
    if (t > 0) {
      pays = con_pays<ConGrid>(k, t, e0);
      small = na <= kConTailVerts && __ldcg(k.cntE + t) <= kConTailEdges && !__ldcg(k.over);
      if (small || !pays) break;
    }
    trace_rec(c, (int32_t)na, 22);
    if (!con_round(k, src, g, t, stage)) return false;
    ++t;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *rounds = t;
  // (an array may run out in the very round that leaves no vertex alive)
  const bool undone = __ldcg(k.over) != 0;
  if (undone || !pays) {
    con_open(k, g, t, undone);
  } else if (small) {
    trace_rec(c, __ldcg(k.cntA + t), 23);
    if (blockIdx.x == 0) con_tail(k, t, max_steps - (st.s - st.s0), smem, rounds);
  }
  trace_rec(c, t, 24);
  if (!g.sync(430)) return false;
  for (int u = t - (undone ? 2 : 1); u >= 0; --u)
    if (!con_undo(k, g, u)) return false;
  return true;
}

// Out-edges of the valid vertices (E_0 of a device graph): a lane per
// vertex, whose degree is at most kConDegree.
struct ConCsr {
  Csr out;
  const int32_t* list;
  int32_t n;
  const uint32_t* valid;
  template <class W, class F>
  __device__ __forceinline__ void edges(const W& w, F f) const {
    for (long long b = w.tid() & ~31ll; b < n; b += w.threads()) {
      const long long i = b + lane_id();
      int32_t v = 0, deg = 0;
      long long s0 = 0;
      if (i < n) {
        v = __ldcg(list + i);
        s0 = __ldg(out.off + v);
        deg = (int32_t)(__ldg(out.off + v + 1) - s0);
      }
      const int32_t most = __reduce_max_sync(kFull, deg);
      for (int32_t e = 0; e < most; ++e) {
        const bool has = e < deg;
        const int32_t d = has ? __ldg(out.adj + s0 + e) : 0;
        f(v, d, has && d != v && bit_get(valid, d));
      }
    }
  }
};

// Contraction of the valid vertices of a device graph, between the trim and
// the searches: for graphs where the searches would pay for their diameter,
// told by the absence of hubs (no valid vertex of more than kConDegree edges
// on a side).  Vertices whose component it finds are labelled and leave the
// valid set; on a lattice that is all of them.
__device__ __noinline__ void contract_phase(const Args& A, Smem& sm) {
  Work w = A.w;
  Ctl* c = w.ctl;
  const GraphView& g = A.g;
  if (ld_vol(&c->err)) return;
  const int32_t nl = __ldcg(&c->nvalid), pivot = __ldcg(&c->pivot);
  if (nl == 0) return;
  if (pivot >= 0 && (g.out.off[pivot + 1] - g.out.off[pivot] > kConDegree ||
                     g.in.off[pivot + 1] - g.in.off[pivot] > kConDegree))
    return;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nth = (long long)gridDim.x * blockDim.x;
  Contract k;
  // (colour and live_in, q and x0 are adjacent in the workspace)
  k.in = reinterpret_cast<int2*>(w.colour);
  k.out = reinterpret_cast<int2*>(w.q);
  k.par = w.x1;
  k.tc = w.candA;
  k.info = reinterpret_cast<uint32_t*>(w.candB);
  k.A[0] = w.h0;
  k.A[1] = w.h1;
  k.D = w.xa;
  int32_t* const small = w.live_out;  // smallest member of a component
  k.list0 = w.listA;
  k.n0 = nl;
  k.arena = w.con_edges;
  k.acap = w.con_cap;
  k.elog = w.con_edges + w.con_cap;
  k.lcap = w.con_cap;
  k.cntA = c->con_cnt[0];
  k.cntD = c->con_cnt[1];
  k.cntE = c->con_ecnt[0];
  k.cntL = c->con_ecnt[1];
  k.over = &c->con_over;
  Steps st = steps_open(c);
  trace_rec(c, nl, 20);
  // Vertices that the first round may merge, among one group of 32 in 16:
  // those with one edge on a side, and those that an out-neighbour points
  // back to.  Fewer than two in three is a uniform random graph, whose core the
  // rounds do not shrink: 71 % of its vertices have one edge on a side at 1.4
  // edges per vertex, 65 % at 1.6, 53 % at 2 (on the lattices a vertex counts
  // 1.2 times).  4 M vertices, with the rounds and without: 1.2 edges per
  // vertex 4.1 and 4.4 ms, 1.4: 3.7 and 3.6, 1.6: 3.6 and 3.0, 2: 3.5 and 2.3;
  // 100,000 vertices, 1.4: 1.65 and 1.89, 1.6: 1.53 and 1.72, 2: 1.44 and 1.52.
  int may = 0;
  for (long long j = tid; j < (nl + 15) / 16 + 31; j += nth) {
    const long long i = (j >> 5) * 512 + (j & 31);
    if (i >= nl) break;
    const int32_t v = __ldcg(w.listA + i);
    const long long s0 = __ldg(g.out.off + v);
    const long long dout = __ldg(g.out.off + v + 1) - s0;
    const long long din = __ldg(g.in.off + v + 1) - __ldg(g.in.off + v);
    if (dout == 1 || din == 1) ++may;
    bool back = false;
    for (long long e = s0; e < s0 + dout && e < s0 + kConDegree && !back; ++e) {
      const int32_t d = __ldg(g.out.adj + e);
      const long long s1 = __ldg(g.out.off + d), e1 = __ldg(g.out.off + d + 1);
      for (long long x = s1; x < e1 && x < s1 + kConDegree && !back; ++x)
        back = d != v && __ldg(g.out.adj + x) == v;
    }
    if (back) ++may;
  }
  if (may) atomicAdd(&c->con_may, may);
  if (!step_sync(c, st, 399)) return;
  // (at most one group of the sample is cut short)
  if (24ll * __ldcg(&c->con_may) < nl) {
    steps_close(c, st);
    return;
  }
  bool big = false;
  for (long long i = tid; i < nl; i += nth) {
    const int32_t v = __ldcg(w.listA + i);
    big = big || __ldg(g.out.off + v + 1) - __ldg(g.out.off + v) > kConDegree ||
          __ldg(g.in.off + v + 1) - __ldg(g.in.off + v) > kConDegree;
    k.in[v] = make_int2(kConInf, -1);
    k.out[v] = make_int2(kConInf, -1);
    k.par[v] = v;
    k.info[v] = 0u;
    small[v] = kConInf;
  }
  if (__any_sync(kFull, big) && lane_id() == 0) c->con_big = 1;
  if (!step_sync(c, st, 400)) return;
  if (__ldcg(&c->con_big)) {
    steps_close(c, st);
    return;
  }
  const ConCsr src{g.out, w.listA, nl, w.vbits};
  unsigned long long* stage = reinterpret_cast<unsigned long long*>(sm.stage(threadIdx.x >> 5, 0));
  if (!contract_run(k, src, c, st, A.p.tune.max_steps, (long long)__ldcg(&c->m_cand),
                    sm.stage_base, stage, &c->ncolour_rounds))
    return;
  // labels: the smallest member of each component
  int open = 0;
  for (long long i = tid; i < nl; i += nth) {
    const int32_t v = __ldcg(w.listA + i), cv = __ldcg(k.tc + v);
    if (cv < 0) ++open;
    else if (v < __ldca(small + cv)) atomicMin(small + cv, v);
  }
  for (int o = 16; o; o >>= 1) open += __shfl_xor_sync(kFull, open, o);
  if (lane_id() == 0 && open) atomicAdd(&c->con_open, open);
  if (!step_sync(c, st, 401)) return;
  open = __ldcg(&c->con_open);
  for (long long i = tid; i < nl; i += nth) {
    const int32_t v = __ldcg(w.listA + i), cv = __ldcg(k.tc + v);
    if (cv < 0) continue;
    w.label[v] = __ldca(small + cv);
    if (open) bit_set_red(w.done, v);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) c->ncolour = nl - open;
  trace_rec(c, nl, 21);
  if (open == 0) {
    if (blockIdx.x == 0 && threadIdx.x == 0) c->nvalid = 0;
    steps_close(c, st);
    return;
  }
  if (!step_sync(c, st, 402)) return;
  Tally ty;
  auto release = [&](int32_t v) { bit_release(w.vbits, v); };
  if (!compact_ordered(w.listA, nl, w.listB, w.done, w, sm, st, 403, &c->nvalid, ty, release)) return;
  if (!step_sync(c, st, 404)) return;
  for (long long i = tid; i < open; i += nth) w.listA[i] = __ldcg(w.listB + i);
  // (a pivot that has its label leaves the rest to the colour rounds)
  if (blockIdx.x == 0 && threadIdx.x == 0 && pivot >= 0 && !bit_get(w.vbits, pivot)) c->pivot = -1;
  steps_close(c, st);
}

}  // namespace
}  // namespace gb
