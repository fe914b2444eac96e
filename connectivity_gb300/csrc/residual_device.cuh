// What FW-BW leaves of an SCC run, before the colour rounds.
//
// On a power-law graph that is thousands of vertices of which nearly all are
// components alone: no edge from another one left, or none to one.  A colour
// round is ten grid steps (reset, propagation, roots, marking, compaction),
// most of them latency; R-MAT-24 took two, 90 us for 12,208 vertices.  Here
// the edges between the vertices left are listed once, everything without
// both an in- and an out-edge among them is labelled (scc_trim,
// multistep/scc_trim.cpp:101-126, on the residual), and what remains, if it
// is small, is contracted by one block in shared memory (con_tail).  A larger
// rest goes on to the colour rounds.  90 -> 44 us on R-MAT-24, 126 -> 44 on
// 2,000 merged graphs (23,862 vertices left).
#pragma once
#include "contract_device.cuh"

namespace gb {
namespace {

// The phase pays while the rest is small.  A large one mostly holds components
// of its own, whose edges would be looked at once more for nothing, two marks
// and a list entry each: it goes straight to the rounds.  Two R-MAT graphs side
// by side (whole call, with and without the phase): of 2^18 vertices each 2.5
// and 2.9 ms, of 2^19 4.8 and 5.4, of 2^20 8.3 and 6.1, of 2^22 49 and 48; 500
// graphs of 1,024 vertices as one 0.69 and 0.57 ms.
constexpr int32_t kResMax = 1 << 18;
// Edges listed at most: what one block takes in the end is far less.
constexpr long long kResList = 1 << 17;

// Lists the edges (v, w) between valid vertices and marks their ends.
struct ResidVisit {
  static constexpr bool kWeighted = false;
  static constexpr bool kLocal = false;
  const uint32_t* valid;
  int32_t* flag;  // bit 0: has an out-edge, bit 1: has an in-edge
  unsigned long long* list;
  long long cap;
  append_count* count;
  int32_t* over;
  mutable bool full;  // the list ran out: no use in counting on
  __device__ __forceinline__ int32_t source(int32_t v) const { return v; }
  __device__ __forceinline__ void edges(const int32_t (&sv)[kEU], const int32_t (&w)[kEU],
                                        const int (&)[kEU], const bool (&act)[kEU],
                                        bool (&out)[kEU]) const {
    bool p[kEU];
#pragma unroll
    for (int q = 0; q < kEU; ++q) p[q] = act[q] && bit_get_l1(valid, w[q]) && w[q] != sv[q];
    // one append for the step's edges
    unsigned mask[kEU], total = 0;
#pragma unroll
    for (int q = 0; q < kEU; ++q) {
      if (p[q]) {
        atomicOr(flag + sv[q], 1);
        atomicOr(flag + w[q], 2);
      }
      mask[q] = __ballot_sync(kFull, p[q]);
      total += __popc(mask[q]);
      out[q] = false;
    }
    if (total == 0u || full) return;
    append_count pos = 0;
    if (lane_id() == 0) pos = atomicAdd(count, (append_count)total);
    pos = __shfl_sync(kFull, pos, 0);
    full = pos + total > (append_count)cap;
    if (full) *over = 1;
#pragma unroll
    for (int q = 0; q < kEU; ++q) {
      const long long at = append_slot(pos, __popc(mask[q] & lanemask_lt()), cap);
      if (p[q] && at >= 0) list[at] = ((unsigned long long)(uint32_t)sv[q] << 32) | (uint32_t)w[q];
      pos += __popc(mask[q]);
    }
  }
  __device__ __forceinline__ unsigned long long weight(int32_t) const { return 0ull; }
};

// Returns whether vertices may be left (after the caller's barrier).
__device__ __noinline__ bool residual_phase(const Args& A, Smem& sm) {
  Work w = A.w;
  Ctl* c = w.ctl;
  if (ld_vol(&c->err)) return false;
  const int32_t nl = __ldcg(&c->nvalid);
  if (nl == 0) return false;
  if (nl > kResMax) return true;
  const int b = blockIdx.x, t = threadIdx.x;
  const long long tid = (long long)b * blockDim.x + t, nth = (long long)gridDim.x * blockDim.x;
  Tally ty;
  Steps st = steps_open(c);
  int32_t* const flag = w.live_in;
  int32_t* const small = w.live_out;
  // (q and x0 are adjacent in the workspace: n pairs)
  unsigned long long* const e0 = reinterpret_cast<unsigned long long*>(w.q);
  Contract k;
  k.A[0] = k.A[1] = w.x1;
  k.tc = w.candA;
  k.arena = reinterpret_cast<unsigned long long*>(w.listB);
  k.acap = w.n / 2;
  k.cntA = c->res_cnt;
  k.cntE = c->res_ecnt;
  int32_t* const over = &c->res_over;
  trace_rec(c, nl, 28);
  if (!__ldcg(&c->res_ready)) {  // (no search ran, so no compaction did)
    for (long long i = tid; i < nl; i += nth) {
      const int32_t v = __ldcg(w.listA + i);
      flag[v] = 0;
      small[v] = kConInf;
    }
    if (!step_sync(c, st, 500)) return false;
  }
  {
    const Adj outs = adj1(A.g.out);
    const ResidVisit rv{w.vbits, flag, e0, min((long long)w.n, kResList), k.cntE, over, false};
    int32_t* hl[2] = {w.h0, w.h1};
    int32_t nfront = nl, nheavy = 0;
    for (int hs = 0;; hs ^= 1) {
      if (st.s - st.s0 >= A.p.tune.max_steps) { set_err(c, kErrIterLimit, 501); return false; }
      const Sink sk = sink_make(w.xa, 0, w.n, step_out(c, st.s), false, nullptr, hl[hs ^ 1], w.n,
                                502);
      expand<1>(w.listA, nfront, hl[hs], nheavy, outs, rv, sk, A.p.tune, sm, c, ty);
      stat_inc(c, kStColourSteps);
      if (!step_sync(c, st, 503)) return false;
      nheavy = step_read(c, st.s).huge;
      if (nheavy == 0) break;
      nfront = 0;
    }
  }
  const bool lost = __ldcg(over) != 0;
  const long long ne0 = (long long)__ldcg(k.cntE);
  for (long long base = tid & ~31ll; base < nl; base += nth) {
    const long long i = base + lane_id();
    int32_t v = 0;
    bool keep = false;
    if (i < nl) {
      v = __ldcg(w.listA + i);
      keep = __ldcg(flag + v) == 3;
      if (!keep) {
        w.label[v] = v;
        bit_release(w.vbits, v);
      }
    }
    con_append(keep, v, k.A[1], k.cntA + 1);
  }
  if (!lost) {
    ConStage none{nullptr, 0, 0};
    for (long long base = tid & ~31ll; base < ne0; base += nth) {
      const long long i = base + lane_id();
      const unsigned long long e = i < ne0 ? __ldcg(e0 + i) : 0ull;
      const int32_t s = (int32_t)(e >> 32), d = (int32_t)(uint32_t)e;
      con_push<false>(none, i < ne0 && __ldcg(flag + s) == 3 && __ldcg(flag + d) == 3, s, d,
                      k.arena, 0, 1, k.acap, k.cntE + 1, over);
    }
  }
  if (!step_sync(c, st, 504)) return false;
  const int32_t na = __ldcg(k.cntA + 1);
  const append_count ne = __ldcg(k.cntE + 1);
  const bool tail = na <= kConTailVerts && ne <= kConTailEdges && __ldcg(over) == 0;
  bool done = na == 0;
  trace_rec(c, na, 29);
  if (na > 0 && tail && ne == 0) {
    // what kept them were edges to and from vertices now labelled
    for (long long i = tid; i < na; i += nth) {
      const int32_t v = __ldcg(k.A[1] + i);
      w.label[v] = v;
    }
    if (tid == 0) {
      c->nvalid = 0;
      c->ncolour = nl;
      c->ncolour_rounds = 1;
    }
    done = true;
  } else if (na > 0 && tail) {
    if (b == 0) {
      __shared__ int s_open;
      if (t == 0) s_open = 0;
      con_tail(k, 1, A.p.tune.max_steps - (st.s - st.s0), sm.stage_base, &c->ncolour_rounds);
      __syncthreads();
      for (int i = t; i < na; i += blockDim.x) {
        const int32_t v = __ldcg(k.A[1] + i), cv = __ldcg(k.tc + v);
        if (cv >= 0) atomicMin(small + cv, v);
      }
      __syncthreads();
      for (int i = t; i < na; i += blockDim.x) {
        const int32_t v = __ldcg(k.A[1] + i), cv = __ldcg(k.tc + v);
        if (cv >= 0) {
          w.label[v] = __ldcg(small + cv);
          bit_release(w.vbits, v);
        } else {
          w.listA[atomicAdd(&s_open, 1)] = v;
        }
      }
      __syncthreads();
      if (t == 0) {
        c->nvalid = s_open;
        c->ncolour = nl - s_open;
      }
    }
  } else {
    for (long long i = tid; i < na; i += nth) w.listA[i] = __ldcg(k.A[1] + i);
    if (tid == 0) {
      c->nvalid = na;
      c->ncolour = nl - na;
      c->ncolour_rounds = 1;
    }
  }
  trace_rec(c, 0, 15);
  tally_flush(ty, c, kKColour, A.p.count_unassigned != 0, sm.red_u);
  steps_close(c, st);
  return !done;
}

}  // namespace
}  // namespace gb
