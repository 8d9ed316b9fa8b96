// Batched independent instances in one persistent launch.
//
// The loaded CSC holds many graphs side by side (instance i owns vertices
// [vbeg[i], vbeg[i+1]) and only edges among them).  One persistent kernel,
// replayed as a CUDA graph, runs for every instance the reference's
// PageRank (comp_pagerank<float>, GraphMP/app/pagerank.cpp:20-84, with
// N = the instance's vertex count) for up to pr_iters supersteps and then
// its min-label CC (comp_cc, GraphMP/app/cc.cpp:20-75) to convergence, each
// with GraphPS::run's stop rule per instance (GraphMP/system/GraphPS.h:383).
// CTAs claim work slots longest instance first.  A small instance is one slot
// and its superstep barrier a CTA barrier; an instance larger than about half
// a CTA's fair share of the batch is split over a team of CTAs (one slot per
// member, claimed consecutively), whose members sweep interleaved tiles and
// meet at a global barrier after every superstep: an arrival counter and
// triple-buffered change counts per instance, polled with a bounded spin (a
// timeout raises an abort flag that every CTA honours, and the host reports
// GX_ERR_TIMEOUT).  The launch holds no more CTAs than fit on the GPU at
// once, so every member of a claimed team is running.
//
// Two things bounded the sweep of an instance's lists as they lie in the CSC:
// the gather of a neighbour's value per edge (from global memory a warp's 32
// addresses cost the L1 a lookup each, even when all hit), and instructions
// spent on lanes whose list had ended or not begun.  So each call first
// rewrites every instance (about 35 supersteps read what it writes once):
//  * its vertices are renumbered by descending list length, and its edges
//    hold the new ids;
//  * the edges are laid out in rounds of 4 per lane, 32 lanes side by side, so
//    that a warp's load of a round is one contiguous piece: lists of up to
//    `lane_max` edges 32 to a tile, a lane each, in edge order; longer lists
//    across the warp, or across half of it when 16 lanes hold them.  Ids are
//    16-bit where they fit, and unused places hold the id of a slot whose
//    value does not count (0 in a sum, the largest label in a minimum).
// A CTA gathers from a table in shared memory, where a gather of 32 costs its
// bank conflicts, three or four cycles: both buffers of an instance that fits
// twice, else the values of its first vertices (the hottest on R-MAT),
// refreshed from global memory after each superstep; other values are gathered
// from there.  Sums are taken in the order of the lists' plain sweep (a lane
// per short list, else 4 consecutive edges per lane per round of 128 aligned
// edges and an xor tree), so results do not depend on the layout.
// 512 instances of scales 10 to 17 (290 M edges, 35 supersteps): 52.6 ms a
// call swept as they lie, 26.0 rewritten (the rewriting's share 2.4 ms); long
// scoreboard stalls on the id loads lead now, at 0.29 of HBM's rate.
// Threads per CTA, lane_max and CTAs per SM come from the autotuner
// (gx_batch_autotune), which times candidate schedules on the batch and
// records the winner in a table file.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdio>
#include <memory>
#include <numeric>
#include <string>
#include <type_traits>
#include <vector>

#include "gx_engine.h"
#include "gx_nvtx.h"

using namespace gx;

namespace {

constexpr int kBatchSortThreads = 512;
constexpr int kSortSmall = 64;       // where no instance has more than four times as many vertices
constexpr int kBatchL1 = 64 * 1024;  // shared-memory bytes per SM left to the L1

// CTAs that share an instance in the kernels that check and rewrite, which take
// the instances in turn: as many as the longest has pieces of `piece` edges and
// vertices, as far as `ctas` in all give every instance that many, but `least`
// of them at any number (the longest instances of many end last).  (With one,
// four and eight at any number, an instance of 2 M vertices and 30 M edges took
// 6.8 ms to sort, 1.9 to check and 4.5 to write out, now 0.06, 0.03 and 0.09,
// and 20000 instances of 8 vertices 0.17, 0.10 and 0.39, now 0.03, 0.03, 0.09.)
int batch_split(int64_t longest, int64_t piece, int64_t ctas, int32_t n, int least) {
  const int64_t most = std::max<int64_t>(least, ctas / n);
  return static_cast<int>(std::max<int64_t>(1, std::min((longest + piece - 1) / piece, most)));
}

// A unit of an instance's sweep: `cnt` vertices from local (new) id `first`
// on, its rounds from round `at` of the instance on.
enum : int { kUnitTile = 0, kUnitHalf = 1, kUnitWarp = 2 };
struct __align__(16) BatchUnit {
  int32_t first;
  int32_t kind_cnt;  // kind << 8 | cnt
  int32_t at;
  int32_t rounds;    // kUnitWarp: rounds per vertex, else of the unit
};

struct BatchArgs {
  const int64_t* off;
  const int32_t* col;
  const int32_t* outdeg;
  const int32_t* vbeg;      // n_inst + 1
  const int2* slots;        // claim order: (instance, member << 16 | team size), longest first
  int32_t n_slots;
  int32_t n_inst;
  unsigned int* ctr;
  unsigned int* team;       // per instance: arrivals, change counts [3]
  unsigned int* abort;      // set when a team barrier times out
  unsigned int spin_limit;  // polls of a team barrier, each a load and a pause of some 64 ns
  float *pr0, *pr1;         // working values, indexed vbeg[i] + new local id
  float *con0, *con1;
  int32_t *lab0, *lab1;
  float* pr_out;            // results, by the caller's vertex
  int32_t* cc_out;
  int32_t* pr_steps;        // per instance
  int32_t* cc_steps;
  int32_t pr_iters, cc_max;
  int32_t lane_max;
  int32_t tab;              // 4-byte values of the CTA's table in dynamic shared memory
  // The rewritten instances.
  int32_t* inv;             // vertex of new id vbeg[i] + k
  int32_t* perm;            // new local id of a vertex
  int32_t* od;              // out-degrees by new id
  BatchUnit* units;         // instance i's at units[vbeg[i]]
  int32_t* n_units;
  unsigned long long* rounds;  // per instance
  const unsigned long long* round_base;  // first block of its rounds
  int* classes;             // split sorts, per instance: vertices of every class, and those placed
  uint2* ids;               // blocks of 32 x 4 16-bit ids; a round of 32-bit ids is two
  double damping;
};

// Ids are 32-bit from this many vertices on (ids run to n, the unused place's).
constexpr int kBatchWide = 65535;

// Vertices of the instance whose values the table holds (besides the unused
// place's), and whether both buffers fit.
__host__ __device__ inline int batch_table(int n, int tab) { return n < tab - 1 ? n : tab - 1; }
__host__ __device__ inline bool batch_dual(int n, int team, int tab) {
  return team == 1 && 2 * (static_cast<int64_t>(n) + 1) <= tab;
}

// The value of id x, as the layout holds it: ids up to tn are table slots (tn
// is the unused place's), those beyond are vertex x - 1's value in global
// memory.  Without a branch: the table is read at a clamped index, global
// memory under a predicate.
template <bool FULL>
__device__ __forceinline__ uint32_t batch_gather(const uint32_t* tab, int tn, const uint32_t* g, int32_t x) {
  if constexpr (FULL) return tab[x];
  uint32_t r = tab[x < tn ? x : tn];
  asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %1, %2;\n\t@p ld.global.b32 %0, [%3];\n\t}"
               : "+r"(r) : "r"(x), "r"(tn), "l"(g + x - 1) : "memory");
  return r;
}

// Folds a value into the sum (PR: contributions) or minimum (labels).
template <bool PR>
__device__ __forceinline__ void batch_fold(uint32_t x, float& f, int32_t& m) {
  if (PR) f += __uint_as_float(x);
  else m = min(m, static_cast<int32_t>(x));
}

// A lane's four ids of a round.
template <bool WIDE>
struct BatchIds {
  uint4 x;
};
template <>
struct BatchIds<false> {
  uint2 x;
};
template <bool WIDE>
__device__ __forceinline__ BatchIds<WIDE> batch_load(const void* ids, int64_t round, int lane) {
  BatchIds<WIDE> r;
  if constexpr (WIDE) r.x = __ldcs(static_cast<const uint4*>(ids) + round * 32 + lane);
  else r.x = __ldcs(static_cast<const uint2*>(ids) + round * 32 + lane);
  return r;
}
template <bool WIDE, bool FULL>
__device__ __forceinline__ void batch_gather4(const BatchIds<WIDE>& c, const uint32_t* tab, int tn, const uint32_t* g,
                                              uint32_t (&v)[4]) {
  uint32_t id[4];
  if constexpr (WIDE) {
    id[0] = c.x.x, id[1] = c.x.y, id[2] = c.x.z, id[3] = c.x.w;
  } else {
    id[0] = c.x.x & 0xffffu, id[1] = c.x.x >> 16, id[2] = c.x.y & 0xffffu, id[3] = c.x.y >> 16;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = batch_gather<FULL>(tab, tn, g, static_cast<int32_t>(id[j]));
}
template <bool PR, bool WIDE, bool FULL>
__device__ __forceinline__ void batch_fold4(const BatchIds<WIDE>& c, const uint32_t* tab, int tn, const uint32_t* g,
                                            float& f, int32_t& m) {
  uint32_t v[4];
  batch_gather4<WIDE, FULL>(c, tab, tn, g, v);
#pragma unroll
  for (int j = 0; j < 4; ++j) batch_fold<PR>(v[j], f, m);
}

// Folds rounds [at, at + n), 32 bytes a lane in flight.
template <bool PR, bool WIDE, bool FULL>
__device__ __forceinline__ void batch_rounds(const void* ids, int64_t at, int n, int lane, const uint32_t* tab, int tn,
                                             const uint32_t* g, float& f, int32_t& m) {
  constexpr int F = WIDE ? 2 : 4;
  int r = 0;
  for (; r + F <= n; r += F) {
    BatchIds<WIDE> c[F];
#pragma unroll
    for (int j = 0; j < F; ++j) c[j] = batch_load<WIDE>(ids, at + r + j, lane);
    uint32_t v[F][4];  // every round's gathers in flight, then their folds in order
#pragma unroll
    for (int j = 0; j < F; ++j) batch_gather4<WIDE, FULL>(c[j], tab, tn, g, v[j]);
#pragma unroll
    for (int j = 0; j < F; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) batch_fold<PR>(v[j][k], f, m);
  }
  if (r < n) {
    BatchIds<WIDE> c[F - 1];
#pragma unroll
    for (int j = 0; j < F - 1; ++j)
      if (r + j < n) c[j] = batch_load<WIDE>(ids, at + r + j, lane);
#pragma unroll
    for (int j = 0; j < F - 1; ++j)
      if (r + j < n) batch_fold4<PR, WIDE, FULL>(c[j], tab, tn, g, f, m);
  }
}

template <bool PR>
__device__ __forceinline__ void batch_tree(int from, float& f, int32_t& m) {
  for (int o = from; o > 0; o >>= 1) {
    if (PR) f += __shfl_xor_sync(0xffffffffu, f, o);
    else m = min(m, __shfl_xor_sync(0xffffffffu, m, o));
  }
}

// Barrier b of a team of `team` CTAs on instance state t[0..3]: adds this
// CTA's change count to t[1 + b % 3] (member 0 first clears the slot barrier
// b + 1 will use) and returns the team's total.  Every thread of the CTA
// calls it, after a CTA barrier.  Returns false when the wait timed out or
// another team aborted.
__device__ bool team_barrier(const BatchArgs& a, unsigned int* t, int team, int member, int b, unsigned changed,
                             unsigned* total) {
  __shared__ unsigned s_tot;
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    int ok = 1;
    if (member == 0) atomicExch(t + 1 + (b + 1) % 3, 0u);
    if (changed) atomicAdd(t + 1 + b % 3, changed);
    __threadfence();
    atomicAdd(t, 1u);
    const unsigned target = static_cast<unsigned>(b + 1) * static_cast<unsigned>(team);
    volatile unsigned* arr = t;
    volatile unsigned* ab = a.abort;
    for (unsigned it = 0; *arr < target; ++it) {
      if (*ab || it >= a.spin_limit) {
        atomicExch(a.abort, 1u);
        ok = 0;
        break;
      }
      __nanosleep(64);
    }
    __threadfence();
    s_tot = *reinterpret_cast<volatile unsigned*>(t + 1 + b % 3);
    s_ok = ok;
  }
  __syncthreads();
  *total = s_tot;
  return s_ok != 0;
}

// What a superstep's sweep needs, in shared memory: the same for the whole
// CTA, and more than the registers of 2048 threads per SM hold.
struct BatchStep {
  const void* ids;
  const BatchUnit* units;
  const uint32_t* g;      // current values (PageRank: contributions) in global memory
  const void* src;        // current ranks or labels
  void* dst;              // next ones
  float* dcon;            // next contributions
  const int32_t* od;
  double damping, inv_n;
  int n_units, member, team, step, dual, tn;
  int tab, next;          // table's current and next buffer
  int s_next;             // next unit of this CTA's share, claimed by warps as they finish
};

// The new value of local vertex k; 1 when it changed.
template <bool PR>
__device__ __forceinline__ unsigned batch_apply(const BatchStep& st, uint32_t* s_tab, int k, float acc, int32_t low,
                                                uint32_t old_bits, int32_t od) {
  if constexpr (PR) {
    const float nv = static_cast<float>(__dadd_rn(__dmul_rn(static_cast<double>(acc), st.damping), st.inv_n));
    const float old = __uint_as_float(old_bits);
    static_cast<float*>(st.dst)[k] = nv;
    const float c = nv / static_cast<float>(od > 0 ? od : 1);
    if (st.dual) s_tab[st.next + k] = __float_as_uint(c);
    else st.dcon[k] = c;
    return nv != (st.step == 0 ? 0.f : old);
  } else {
    const int32_t old = st.dual ? static_cast<int32_t>(s_tab[st.tab + k]) : static_cast<int32_t>(old_bits);
    const int32_t nv = min(old, low);
    if (st.dual) s_tab[st.next + k] = static_cast<uint32_t>(nv);
    else static_cast<int32_t*>(st.dst)[k] = nv;
    return nv != (st.step == 0 ? 0 : old);
  }
}

// One superstep's units of this CTA's share; returns the warp's changes.
// Member `member` of the team takes units member, member + team, ..., claimed
// from st.s_next.
template <bool PR, bool WIDE, bool FULL>
__device__ __forceinline__ unsigned batch_sweep(BatchStep& st, uint32_t* s_tab, int lane) {
  unsigned changed = 0;
  const uint32_t* tab = s_tab + st.tab;
  const uint32_t* g = st.g;
  const void* ids = st.ids;
  const int tn = st.tn;
  auto claim = [&]() -> int {
    int k = 0;
    if (lane == 0) k = atomicAdd(&st.s_next, 1);
    const int64_t t = st.member + static_cast<int64_t>(__shfl_sync(0xffffffffu, k, 0)) * st.team;
    return t < st.n_units ? static_cast<int>(t) : -1;
  };
  int t = claim();
  int4 next = make_int4(0, 0, 0, 0);
  if (t >= 0) next = *reinterpret_cast<const int4*>(st.units + t);
  while (t >= 0) {
    const int4 u = next;
    t = claim();
    if (t >= 0) next = *reinterpret_cast<const int4*>(st.units + t);  // in flight while u is swept
    const int kind = u.y >> 8, cnt = u.y & 255;
    uint32_t old = 0;
    int32_t od = 0;
    if (lane < cnt) {  // likewise
      if (PR) od = st.od[u.x + lane];
      if (PR || !st.dual) old = __ldcg(static_cast<const uint32_t*>(st.src) + u.x + lane);
    }
    float f = 0.f;
    int32_t m = 0x7fffffff;
    if (kind == kUnitTile) {
      batch_rounds<PR, WIDE, FULL>(ids, u.z, u.w, lane, tab, tn, g, f, m);
    } else if (kind == kUnitHalf) {
      BatchIds<WIDE> c[4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (r < u.w) c[r] = batch_load<WIDE>(ids, u.z + r, lane);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (r < u.w) {
          float fl = 0.f;
          int32_t ml = 0x7fffffff;
          batch_fold4<PR, WIDE, FULL>(c[r], tab, tn, g, fl, ml);
          batch_tree<PR>(8, fl, ml);
          const float fr = __shfl_sync(0xffffffffu, fl, (lane & 1) << 4);
          const int32_t mr = __shfl_sync(0xffffffffu, ml, (lane & 1) << 4);
          if ((lane >> 1) == r) {
            f = fr;
            m = mr;
          }
        }
      }
    } else {
      for (int i = 0; i < cnt; ++i) {
        float fl = 0.f;
        int32_t ml = 0x7fffffff;
        batch_rounds<PR, WIDE, FULL>(ids, u.z + static_cast<int64_t>(i) * u.w, u.w, lane, tab, tn, g, fl, ml);
        batch_tree<PR>(16, fl, ml);
        if (lane == i) {
          f = fl;
          m = ml;
        }
      }
    }
    if (lane < cnt) changed += batch_apply<PR>(st, s_tab, u.x + lane, f, m, old, od);
    __syncwarp();
  }
  return __reduce_add_sync(0xffffffffu, changed);
}

__global__ void __launch_bounds__(1024, 1) batch_kernel(const __grid_constant__ BatchArgs a) {
  extern __shared__ __align__(16) uint32_t s_tab[];
  __shared__ BatchStep s_st;
  __shared__ int s_slot;
  __shared__ unsigned int s_changed[2];
  const int lane = threadIdx.x & 31;
  for (;;) {
    if (threadIdx.x == 0)
      s_slot = *reinterpret_cast<volatile unsigned*>(a.abort) ? a.n_slots : static_cast<int>(atomicAdd(a.ctr, 1u));
    __syncthreads();
    const int slot = s_slot;
    __syncthreads();
    if (slot >= a.n_slots) break;
    const int2 sl = a.slots[slot];
    const int inst = sl.x, member = sl.y >> 16, team = sl.y & 0xffff;
    unsigned int* tstate = a.team + 4 * static_cast<int64_t>(inst);
    const int32_t vb = a.vbeg[inst], ve = a.vbeg[inst + 1], n = ve - vb;
    const double inv_n = 1.0 / n;
    const int vt0 = member * blockDim.x + threadIdx.x, vstride = blockDim.x * team;
    // The table: both buffers of an instance that one CTA holds and that fits
    // twice (`dual`: nothing is kept in global memory then), else the current
    // values of the first tn vertices; after each buffer the unused place's.
    const bool dual = batch_dual(n, team, a.tab);
    const int tn = batch_table(n, a.tab);
    int bar = 0;
    // The barrier that ends step `step` (or, -1, what comes before the first): a
    // CTA barrier, or the team's; *total: the step's changes.  Steps count in two
    // places in turn: the next sweep's set-up clears its own, which every thread
    // has read before the barriers of the step between.  (Thousands of tiny
    // instances are little but barriers: a superstep from the table has this one
    // and the sweep's.  __syncthreads_or in place of the count, or two step
    // records in turn to do without the sweep's, cost the sweep more in registers
    // than they saved: 512 instances 26.1 -> 26.9 and 27.5 ms.)
    auto sync_count = [&](int step, unsigned mine, unsigned* total) -> bool {
      unsigned* at = s_changed + (step & 1);
      if (lane == 0 && mine) atomicAdd(at, mine);
      __syncthreads();
      *total = *reinterpret_cast<volatile unsigned*>(at);
      return team == 1 || team_barrier(a, tstate, team, member, bar++, *total, total);
    };
    // The table's copy of the values a finished phase left in g (through L2:
    // other CTAs of the team wrote them).
    auto fill = [&](const uint32_t* g) {
      for (int i = threadIdx.x; i < tn; i += blockDim.x) s_tab[i] = __ldcg(g + i);
      __syncthreads();
    };
    if (threadIdx.x == 0) {
      s_st.ids = a.ids + 32 * a.round_base[inst];
      s_st.units = a.units + vb;
      s_st.n_units = a.n_units[inst];
      s_st.member = member;
      s_st.team = team;
      s_st.dual = dual;
      s_st.tn = tn;
      s_st.od = a.od + vb;
      s_st.damping = a.damping;
      s_st.inv_n = inv_n;
      s_changed[0] = s_changed[1] = 0;
    }
    // Superstep `step` from buffer `cur` (x0, x1: ranks or labels; c0, c1:
    // contributions), after a barrier; the changes of this warp.
    auto sweep = [&](auto pr, int step, int cur, void* x0, void* x1, float* c0, float* c1) -> unsigned {
      constexpr bool PR = decltype(pr)::value;
      if (threadIdx.x == 0) {
        s_st.step = step;
        s_st.src = cur ? x1 : x0;
        s_st.dst = cur ? x0 : x1;
        s_st.dcon = cur ? c0 : c1;
        s_st.g = static_cast<const uint32_t*>(PR ? (cur ? c1 : c0) : (cur ? x1 : x0));
        s_st.tab = dual && cur ? n + 1 : 0;
        s_st.next = cur ? 0 : n + 1;
        s_st.s_next = 0;
        s_changed[step & 1] = 0;
      }
      __syncthreads();
      const bool wide = n >= kBatchWide;
      if (tn == n)
        return wide ? batch_sweep<PR, true, true>(s_st, s_tab, lane) : batch_sweep<PR, false, true>(s_st, s_tab, lane);
      return wide ? batch_sweep<PR, true, false>(s_st, s_tab, lane) : batch_sweep<PR, false, false>(s_st, s_tab, lane);
    };
    auto unused = [&](uint32_t x) {
      if (threadIdx.x == 0) {
        s_tab[tn] = x;
        if (dual) s_tab[2 * n + 1] = x;
      }
    };
    unsigned tot = 0;
    // ---- PageRank ----
    unused(0u);
    for (int k = vt0; k < n; k += vstride) {
      const float r0 = static_cast<float>(inv_n);
      const int32_t od = a.od[vb + k];
      a.pr0[vb + k] = r0;
      const float c = r0 / static_cast<float>(od > 0 ? od : 1);
      if (dual) s_tab[k] = __float_as_uint(c);
      else a.con0[vb + k] = c;
    }
    if (!sync_count(-1, 0, &tot)) return;
    if (!dual) fill(reinterpret_cast<const uint32_t*>(a.con0 + vb));
    int cur = 0, step = 0;
    for (step = 0; step < a.pr_iters; ++step) {
      const unsigned changed = sweep(std::true_type(), step, cur, a.pr0 + vb, a.pr1 + vb, a.con0 + vb, a.con1 + vb);
      if (!sync_count(step, changed, &tot)) return;
      cur ^= 1;
      if (tot == 0 && step > 1) {
        ++step;
        break;
      }
      if (!dual) fill(reinterpret_cast<const uint32_t*>((cur ? a.con1 : a.con0) + vb));
    }
    for (int k = vt0; k < n; k += vstride) a.pr_out[a.inv[vb + k]] = __ldcg((cur ? a.pr1 : a.pr0) + vb + k);
    if (threadIdx.x == 0 && member == 0) a.pr_steps[inst] = step < a.pr_iters ? step : a.pr_iters;
    __syncthreads();
    // ---- CC ----
    unused(0x7fffffffu);
    for (int k = vt0; k < n; k += vstride) {
      const int32_t label = a.inv[vb + k] - vb;
      if (dual) s_tab[k] = static_cast<uint32_t>(label);
      else a.lab0[vb + k] = label;
    }
    if (!sync_count(-1, 0, &tot)) return;
    if (!dual) fill(reinterpret_cast<const uint32_t*>(a.lab0 + vb));
    cur = 0;
    for (step = 0; step < a.cc_max; ++step) {
      const unsigned changed = sweep(std::false_type(), step, cur, a.lab0 + vb, a.lab1 + vb, nullptr, nullptr);
      if (!sync_count(step, changed, &tot)) return;
      cur ^= 1;
      if (tot == 0 && step > 1) {
        ++step;
        break;
      }
      if (!dual) fill(reinterpret_cast<const uint32_t*>((cur ? a.lab1 : a.lab0) + vb));
    }
    for (int k = vt0; k < n; k += vstride)
      a.cc_out[a.inv[vb + k]] =
          dual ? static_cast<int32_t>(s_tab[(cur ? n + 1 : 0) + k]) : __ldcg((cur ? a.lab1 : a.lab0) + vb + k);
    if (threadIdx.x == 0 && member == 0) a.cc_steps[inst] = step < a.cc_max ? step : a.cc_max;
    __syncthreads();
  }
}

// `split` CTAs take the instances in turn: every edge must stay inside its
// instance (read end to end, four ids a thread: a thread per vertex, walking
// its list, took 3.6 ms for 290 M edges).
__global__ void __launch_bounds__(512) batch_check_kernel(const int64_t* off, const int32_t* col, const int32_t* vbeg,
                                                          int32_t n_inst, int split, unsigned int* bad) {
  unsigned c = 0;
  const int64_t part = blockIdx.x % split, stride = 4ll * split * blockDim.x;
  for (int i = blockIdx.x / split; i < n_inst; i += gridDim.x / split) {
    const int32_t vb = vbeg[i], ve = vbeg[i + 1];
    const int64_t b = off[vb], e = off[ve];
    for (int64_t q = (b & ~3ll) + 4 * (part * blockDim.x + threadIdx.x); q < e; q += stride) {
      const int4 x = __ldcs(reinterpret_cast<const int4*>(col + q));
      const int32_t cs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) c += q + j >= b && q + j < e && (cs[j] < vb || cs[j] >= ve);
    }
  }
  if (c) atomicAdd(bad, c);
}

// Length classes of an instance's lists, in the order of its new ids: across
// the warp by rounds (63 or more first), across half a warp, then a lane's by
// rounds.  lo: the first edge's position in its aligned group of four.
constexpr int kClassCap = 63;
constexpr int kClassHalf = kClassCap, kClassLane = kClassHalf + 1, kClasses = kClassLane + kClassCap + 1;
__device__ __forceinline__ int batch_class(int64_t beg, int64_t len, int lane_max) {
  if (len <= lane_max) {
    const int64_t r = (len + 3) / 4;
    return kClassLane + kClassCap - static_cast<int>(r < kClassCap ? r : kClassCap);
  }
  const int64_t q = (beg & 3) + len;
  if (q <= 64) return kClassHalf;
  const int64_t r = (q + 127) / 128;
  return kClassCap - static_cast<int>(r < kClassCap ? r : kClassCap);
}
// Lists across the warp of up to this many rounds share a unit, four to each.
constexpr int kWarpShare = 4;

// Instances (taken in turn) get their vertices in order of their classes, and
// their units.  Within a class the order is that of the atomics, and so is the
// units' place among the rounds: no result depends on them.  An instance per
// CTA in one launch (kSortAll), or `split` CTAs to an instance in three that
// count the classes, place the vertices and make the units.
enum : int { kSortAll = 0, kSortCount = 1, kSortPlace = 2, kSortUnits = 3 };
template <int PHASE>
__global__ void __launch_bounds__(kBatchSortThreads) batch_sort_kernel(const __grid_constant__ BatchArgs a, int split) {
  __shared__ int s_at[kClasses + 1];
  __shared__ __align__(16) int s_cur[kClasses];
  __shared__ unsigned long long s_w[kBatchSortThreads / 32], s_run;
  static_assert(kClasses == 128, "a lane scans four classes");
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int T = blockDim.x, part = blockIdx.x % split, stride = T * split;
  for (int i = blockIdx.x / split; i < a.n_inst; i += gridDim.x / split) {
    const int32_t vb = a.vbeg[i], n = a.vbeg[i + 1] - vb;
    int* classes = PHASE == kSortAll ? nullptr : a.classes + 2 * kClasses * static_cast<int64_t>(i);  // counted; placed
    if (PHASE != kSortUnits) {
      for (int c = threadIdx.x; c < kClasses; c += T) s_cur[c] = 0;
      __syncthreads();
      for (int k = part * T + threadIdx.x; k < n; k += stride) {
        const int64_t beg = a.off[vb + k];
        atomicAdd(&s_cur[batch_class(beg, a.off[vb + k + 1] - beg, a.lane_max)], 1);
      }
      __syncthreads();
    }
    if (PHASE == kSortCount) {
      for (int c = threadIdx.x; c < kClasses; c += T)
        if (s_cur[c]) atomicAdd(classes + c, s_cur[c]);
      __syncthreads();
      continue;
    }
    if (wid == 0) {
      const int4 x = *reinterpret_cast<const int4*>((PHASE == kSortAll ? s_cur : classes) + 4 * lane);
      const int sum = x.x + x.y + x.z + x.w;
      int incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      const int at = incl - sum;
      s_at[4 * lane] = at;
      s_at[4 * lane + 1] = at + x.x;
      s_at[4 * lane + 2] = at + x.x + x.y;
      s_at[4 * lane + 3] = at + x.x + x.y + x.z;
      if (lane == 31) s_at[kClasses] = incl;
      if (lane == 0) s_run = 0;
    }
    __syncthreads();
    if (PHASE != kSortUnits) {
      for (int c = threadIdx.x; c < kClasses; c += T) {
        int at = s_at[c];
        if (PHASE == kSortPlace && s_cur[c]) at += atomicAdd(classes + kClasses + c, s_cur[c]);
        s_cur[c] = at;
      }
      __syncthreads();
      for (int k = part * T + threadIdx.x; k < n; k += stride) {
        const int64_t beg = a.off[vb + k];
        const int p = atomicAdd(&s_cur[batch_class(beg, a.off[vb + k + 1] - beg, a.lane_max)], 1);
        a.perm[vb + k] = p;
        a.inv[vb + p] = vb + k;
        a.od[vb + p] = a.outdeg[vb + k];
      }
      __syncthreads();
    }
    if (PHASE == kSortPlace) continue;
    // Units: the warp lists of many rounds one each, the others four to a
    // unit, the half-warp lists eight to a unit, the lane lists 32.
    const int n_one = s_at[kClassCap - kWarpShare], n_warp = s_at[kClassHalf], n_wide = s_at[kClassLane];
    const int u_one = n_one, u_warp = u_one + (n_warp - n_one + 3) / 4, u_half = u_warp + (n_wide - n_warp + 7) / 8;
    const int u_all = u_half + (n - n_wide + 31) / 32;
    for (int u0 = part * T; u0 < u_all; u0 += stride) {
      const int u = u0 + threadIdx.x;
      BatchUnit x{0, 0, 0, 0};
      unsigned long long total = 0;
      if (u < u_all) {
        int last;
        if (u < u_warp) {
          x.first = u < u_one ? u : n_one + 4 * (u - u_one);
          last = u < u_one ? x.first + 1 : min(x.first + 4, n_warp);
          x.kind_cnt = kUnitWarp << 8 | (last - x.first);
        } else if (u < u_half) {
          x.first = n_warp + 8 * (u - u_warp);
          last = min(x.first + 8, n_wide);
          x.kind_cnt = kUnitHalf << 8 | (last - x.first);
          x.rounds = (last - x.first + 1) / 2;
          total = x.rounds;
        } else {
          x.first = n_wide + 32 * (u - u_half);
          last = min(x.first + 32, n);
          x.kind_cnt = kUnitTile << 8 | (last - x.first);
        }
        if (u < u_warp || u >= u_half) {
          int64_t most = 0;
          for (int k = x.first; k < last; ++k) {
            const int64_t beg = a.off[a.inv[vb + k]], len = a.off[a.inv[vb + k] + 1] - beg;
            const int64_t r = u < u_warp ? ((beg & 3) + len + 127) / 128 : (len + 3) / 4;
            most = r > most ? r : most;
          }
          x.rounds = static_cast<int32_t>(most);
          total = u < u_warp ? static_cast<unsigned long long>(most) * (last - x.first) : most;
        }
      }
      unsigned long long incl = total;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) s_w[wid] = incl;
      __syncthreads();
      unsigned long long before = 0, all = 0;
      for (int w = 0; w < T / 32; ++w) {
        before += w < wid ? s_w[w] : 0;
        all += s_w[w];
      }
      if (PHASE == kSortUnits) {  // the place of these T units among all CTAs'
        if (threadIdx.x == 0) s_run = atomicAdd(a.rounds + i, all);
        __syncthreads();
      }
      before += s_run;
      if (u < u_all) {
        x.at = static_cast<int32_t>(before + incl - total);
        a.units[vb + u] = x;
      }
      __syncthreads();
      if (PHASE == kSortAll) {
        if (threadIdx.x == 0) s_run += all;
        __syncthreads();
      }
    }
    if (threadIdx.x == 0 && part == 0) a.n_units[i] = u_all;
    if (PHASE == kSortAll && threadIdx.x == 0) a.rounds[i] = s_run;
    __syncthreads();
  }
}

// Writes the rounds: `split` CTAs share an instance, a warp per unit.
__global__ void __launch_bounds__(256) batch_fill_kernel(const __grid_constant__ BatchArgs a, int split) {
  const int lane = threadIdx.x & 31;
  const int w0 = (blockIdx.x % split) * 8 + (threadIdx.x >> 5);
  for (int i = blockIdx.x / split; i < a.n_inst; i += gridDim.x / split) {
    const int32_t vb = a.vbeg[i], n = a.vbeg[i + 1] - vb;
    const int tn = batch_table(n, a.tab);
    const bool wide = n >= kBatchWide;
    uint2* ids = a.ids + 32 * a.round_base[i];
    for (int t = w0; t < a.n_units[i]; t += split * 8) {
      const BatchUnit u = a.units[vb + t];
      const int kind = u.kind_cnt >> 8, cnt = u.kind_cnt & 255;
      // The vertex and the position of this lane's first place in each round.
      int64_t beg = 0, len = 0;
      int k_now = -1;
      const int rounds = kind == kUnitWarp ? cnt * u.rounds : u.rounds;
      for (int r = 0; r < rounds; ++r) {
        int k;       // vertex of the unit
        int64_t q;   // first edge of the lane's four, counted from the list's start
        if (kind == kUnitTile) {
          k = lane;
          q = 4ll * r;
        } else if (kind == kUnitHalf) {
          k = 2 * r + (lane >> 4);
          q = 4ll * (lane & 15);
        } else {
          k = r / u.rounds;
          q = 128ll * (r % u.rounds) + 4ll * lane;
        }
        if (k != k_now) {
          k_now = k;
          len = 0;
          if (k < cnt) {
            const int32_t v = a.inv[vb + u.first + k];
            beg = a.off[v];
            len = a.off[v + 1] - beg;
          }
        }
        if (kind != kUnitTile) q -= beg & 3;
        int32_t c[4];
        uint32_t id[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = q + j >= 0 && q + j < len ? __ldg(a.col + beg + q + j) : -1;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int p = c[j] >= 0 ? __ldg(a.perm + c[j]) : tn;
          id[j] = static_cast<uint32_t>(c[j] >= 0 && p >= tn ? p + 1 : p);
        }
        const int64_t at = u.at + static_cast<int64_t>(r);
        if (wide) reinterpret_cast<uint4*>(ids)[at * 32 + lane] = make_uint4(id[0], id[1], id[2], id[3]);
        else ids[at * 32 + lane] = make_uint2(id[0] | id[1] << 16, id[2] | id[3] << 16);
      }
    }
  }
}

// A call's device memory: one block for what depends on the vertices and
// instances alone, the rounds, and the slots.
struct BatchDev {
  unsigned char* block = nullptr;
  uint2* ids = nullptr;
  int2* slots = nullptr;
  float* pr_out = nullptr;
  int32_t *cc_out = nullptr, *pr_steps = nullptr, *cc_steps = nullptr;
  unsigned long long *rounds = nullptr, *round_base = nullptr;
  std::vector<int32_t> order;       // instances, longest first
  std::vector<int64_t> work;        // per instance: edges + vertices
  int32_t most_vertices = 0;        // of an instance
  int sort_split = 1;               // CTAs that sort one
  ~BatchDev() {
    dev_free(&block);
    dev_free(&slots);
    dev_free(&ids);
  }
};

// Every edge must stay inside its instance (a block-diagonal CSC).  d_vbeg:
// room for the n + 1 bounds, copied there first; ctr: a word.
gx_status batch_check(gx_engine* e, int32_t n, const int32_t* vbeg, int32_t* d_vbeg, unsigned int* ctr) {
  int64_t longest = 0;
  for (int32_t i = 0; i < n; ++i) longest = std::max(longest, e->off[vbeg[i + 1]] - e->off[vbeg[i]]);
  GX_CUDA(cudaMemcpyAsync(d_vbeg, vbeg, sizeof(int32_t) * (static_cast<size_t>(n) + 1), cudaMemcpyHostToDevice, e->s_comp));
  GX_CUDA(cudaMemsetAsync(ctr, 0, sizeof(unsigned int), e->s_comp));
  const int ctas = e->n_sm * 4, split = batch_split(longest, 8192, ctas, n, 4);
  batch_check_kernel<<<split * std::min(n, ctas / split), 512, 0, e->s_comp>>>(e->d_off, e->d_col, d_vbeg, n, split, ctr);
  GX_CUDA(cudaGetLastError());
  unsigned int bad = 0;
  GX_CUDA(cudaMemcpyAsync(&bad, ctr, sizeof(bad), cudaMemcpyDeviceToHost, e->s_comp));
  GX_CUDA(cudaStreamSynchronize(e->s_comp));
  if (bad) return fail(GX_ERR_INVALID, "gx_batch: %u edges cross instance boundaries", bad);
  return GX_OK;
}

// Device memory and arguments for instances [0, n) of vbeg, whose first vertex
// need not be the graph's.
gx_status batch_prepare(gx_engine* e, int32_t n, const int32_t* vbeg, bool check, BatchDev& d, BatchArgs& a) {
  const int32_t V = vbeg[n] - vbeg[0];
  std::vector<int32_t>& order = d.order;
  order.resize(n);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) {
    return e->off[vbeg[x + 1]] - e->off[vbeg[x]] > e->off[vbeg[y + 1]] - e->off[vbeg[y]];
  });
  d.work.resize(n);
  for (int32_t i = 0; i < n; ++i) {
    d.work[i] = (e->off[vbeg[i + 1]] - e->off[vbeg[i]]) + (vbeg[i + 1] - vbeg[i]);
    d.most_vertices = std::max(d.most_vertices, vbeg[i + 1] - vbeg[i]);
  }
  size_t at = 0;
  auto place = [&](size_t count, size_t bytes) {
    const size_t x = at;
    at += (count * bytes + 255) & ~size_t(255);
    return x;
  };
  const size_t v = static_cast<size_t>(V), m = static_cast<size_t>(n);
  const size_t o_vbeg = place(m + 1, 4), o_team = place(4 * m, 4), o_abort = place(1, 4), o_ctr = place(1, 4);
  const size_t o_lab0 = place(v, 4), o_lab1 = place(v, 4), o_cc = place(v, 4), o_pr0 = place(v, 4), o_pr1 = place(v, 4),
               o_con0 = place(v, 4), o_con1 = place(v, 4), o_pr = place(v, 4);
  const size_t o_prs = place(m, 4), o_ccs = place(m, 4);
  const size_t o_inv = place(v, 4), o_perm = place(v, 4), o_od = place(v, 4), o_units = place(v, sizeof(BatchUnit));
  const size_t o_nu = place(m, 4), o_rounds = place(m, 8), o_base = place(m, 8);
  // Several CTAs sort an instance where there are few instances, or one that
  // would keep a single CTA long after the others (unless the counts of all
  // of them, 1 KB each, were many).
  if (n < 65536 && d.most_vertices > (n < e->n_sm ? 4 : 64) * kBatchSortThreads)
    d.sort_split = batch_split(d.most_vertices, 4 * kBatchSortThreads, e->n_sm * 4, n, 8);
  const size_t o_classes = place(d.sort_split > 1 ? 2 * kClasses * m : 0, 4);
  GX_TRY(dev_alloc(&d.block, at));
  a = BatchArgs{};
  auto as = [&](size_t o, auto*& p) { p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(d.block + o); };
  int32_t* d_vbeg = nullptr;
  as(o_vbeg, d_vbeg);
  as(o_team, a.team);
  as(o_abort, a.abort);
  as(o_ctr, a.ctr);
  as(o_lab0, a.lab0);
  as(o_lab1, a.lab1);
  as(o_pr0, a.pr0);
  as(o_pr1, a.pr1);
  as(o_con0, a.con0);
  as(o_con1, a.con1);
  as(o_inv, a.inv);
  as(o_perm, a.perm);
  as(o_od, a.od);
  as(o_units, a.units);
  as(o_nu, a.n_units);
  as(o_pr, d.pr_out);
  as(o_cc, d.cc_out);
  as(o_prs, d.pr_steps);
  as(o_ccs, d.cc_steps);
  as(o_rounds, d.rounds);
  as(o_base, d.round_base);
  as(o_classes, a.classes);
  a.vbeg = d_vbeg;
  a.pr_out = d.pr_out;
  a.cc_out = d.cc_out;
  a.pr_steps = d.pr_steps;
  a.cc_steps = d.cc_steps;
  a.rounds = d.rounds;
  a.round_base = d.round_base;
  a.off = e->d_off;
  a.col = e->d_col;
  a.outdeg = e->d_outdeg;
  a.n_inst = n;
  a.spin_limit = e->cfg.wait_limit;
  // Indexed by the graph's vertices, of which they hold these instances'.
  for (float** x : {&a.pr0, &a.pr1, &a.con0, &a.con1, &a.pr_out}) *x -= vbeg[0];
  for (int32_t** x : {&a.lab0, &a.lab1, &a.cc_out, &a.inv, &a.perm, &a.od}) *x -= vbeg[0];
  a.units -= vbeg[0];
  if (check) return batch_check(e, n, vbeg, d_vbeg, a.ctr);
  GX_CUDA(cudaMemcpyAsync(d_vbeg, vbeg, sizeof(int32_t) * (m + 1), cudaMemcpyHostToDevice, e->s_comp));
  return GX_OK;
}

// Shared memory of a CTA's table: the SM's, less what the index loads need as
// L1, shared out among the CTAs wanted (1 KB each is the system's).
gx_status batch_table_bytes(gx_engine* e, const gx_batch_tuning& t, int* bytes) {
  int smem_sm = 0, optin = 0, per_sm = 0;
  GX_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, e->dev));
  GX_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, e->dev));
  cudaFuncAttributes attr{};
  GX_CUDA(cudaFuncGetAttributes(&attr, batch_kernel));
  const int fixed = static_cast<int>(attr.sharedSizeBytes);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_kernel, t.threads, 0);
  const int want = std::max(1, std::min(per_sm, t.ctas_per_sm));
  *bytes = std::max(64, std::min(optin - fixed, (smem_sm - kBatchL1) / want - 1024 - fixed)) & ~15;
  return GX_OK;
}

// The schedule of a call that names none: the default's two CTAs of 512
// threads per SM, or one of 1024 with twice the table where most of the work
// is in instances that the default's table does not hold whole (512 R-MAT
// instances of scales 10 to 17: 32.6 -> 26.8 ms a call; 2000 of scales 6 to
// 12, which it does hold: 2.2 ms against 2.6).  Instances of at most kTinyMost
// vertices are a warp or two of work between barriers: where there are waves of
// them, CTAs of 64 threads, 16 to an SM, keep eight times as many going (20000
// of 8 vertices: a call of 5.0 -> 2.1 ms).
constexpr int kTinyMost = 256;
gx_status batch_default_schedule(gx_engine* e, int32_t n, const int32_t* vbeg, gx_batch_tuning* t) {
  gx_batch_tuning_default(t);
  int smem = 0;
  GX_TRY(batch_table_bytes(e, *t, &smem));
  int64_t in = 0, out = 0;
  int32_t most = 0;
  for (int32_t i = 0; i < n; ++i) {
    const int32_t v = vbeg[i + 1] - vbeg[i];
    (v < smem / 4 ? in : out) += e->off[vbeg[i + 1]] - e->off[vbeg[i]] + v;
    most = std::max(most, v);
  }
  if (out > in) {
    t->threads = 1024;
    t->ctas_per_sm = 1;
  } else if (most <= kTinyMost && n >= 8 * e->n_sm) {
    t->threads = 64;
    t->ctas_per_sm = 16;
  }
  return GX_OK;
}

// One persistent launch (plus its cursor and team-state resets), captured as
// a CUDA graph.  The grid holds no more CTAs than are resident at once.
gx_status batch_launch(gx_engine* e, const int32_t* vbeg, BatchDev& d, BatchArgs& a, const gx_batch_tuning& t, float* ms) {
  cudaStream_t s = e->s_comp;
  int per_sm = 0;
  int smem = 0;
  GX_TRY(batch_table_bytes(e, t, &smem));
  a.tab = smem / 4;
  GX_CUDA(allow_dynamic_smem(e->dev, reinterpret_cast<const void*>(batch_kernel)));
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_kernel, t.threads, smem);
  if (per_sm < 1) return fail(GX_ERR_INVALID, "gx_batch: %d threads per CTA do not fit an SM", t.threads);
  const int blocks = std::min(per_sm, t.ctas_per_sm) * e->n_sm;
  // Work slots: an instance above half a CTA's fair share gets a team of up
  // to 32 CTAs (never more than the grid).
  int64_t total = 0;
  for (int64_t w : d.work) total += w;
  const int64_t share = std::max<int64_t>(1, total / (2 * static_cast<int64_t>(blocks)));
  std::vector<int2> slots;
  slots.reserve(d.order.size());
  for (int32_t inst : d.order) {
    const int team = static_cast<int>(std::min<int64_t>({(d.work[inst] + share - 1) / share, 32, blocks}));
    for (int m = 0; m < std::max(team, 1); ++m) slots.push_back(make_int2(inst, (m << 16) | std::max(team, 1)));
  }
  dev_free(&d.slots);
  GX_TRY(dev_alloc(&d.slots, slots.size()));
  GX_CUDA(cudaMemcpy(d.slots, slots.data(), sizeof(int2) * slots.size(), cudaMemcpyHostToDevice));
  a.slots = d.slots;
  a.n_slots = static_cast<int32_t>(slots.size());
  cudaEvent_t e0, e1;
  GX_CUDA(cudaEventCreate(&e0));
  GX_CUDA(cudaEventCreate(&e1));
  std::unique_ptr<CUevent_st, cudaError_t (*)(cudaEvent_t)> e0_g(e0, cudaEventDestroy), e1_g(e1, cudaEventDestroy);
  cudaEventRecord(e0, s);
  // The instances rewritten for this schedule.
  const int32_t n = a.n_inst;
  const int64_t longest = d.work[d.order[0]];
  if (d.sort_split == 1) {
    const int threads = d.most_vertices <= 4 * kSortSmall ? kSortSmall : kBatchSortThreads;
    batch_sort_kernel<kSortAll><<<std::min(n, e->n_sm * (2048 / threads)), threads, 0, s>>>(a, 1);
  } else {
    const int split = d.sort_split, grid = split * std::min(n, std::max(1, e->n_sm * 4 / split));
    GX_CUDA(cudaMemsetAsync(a.classes, 0, sizeof(int) * 2 * kClasses * n, s));
    GX_CUDA(cudaMemsetAsync(a.rounds, 0, sizeof(unsigned long long) * n, s));
    batch_sort_kernel<kSortCount><<<grid, kBatchSortThreads, 0, s>>>(a, split);
    batch_sort_kernel<kSortPlace><<<grid, kBatchSortThreads, 0, s>>>(a, split);
    batch_sort_kernel<kSortUnits><<<grid, kBatchSortThreads, 0, s>>>(a, split);
  }
  GX_CUDA(cudaGetLastError());
  std::vector<unsigned long long> rounds_of(static_cast<size_t>(a.n_inst)), base(static_cast<size_t>(a.n_inst));
  GX_CUDA(cudaMemcpyAsync(rounds_of.data(), d.rounds, sizeof(unsigned long long) * a.n_inst, cudaMemcpyDeviceToHost, s));
  GX_CUDA(cudaStreamSynchronize(s));
  unsigned long long n_blocks = 0;
  for (int32_t i = 0; i < a.n_inst; ++i) {
    base[i] = n_blocks;
    n_blocks += vbeg[i + 1] - vbeg[i] >= kBatchWide ? 2 * rounds_of[i] : rounds_of[i];
  }
  GX_TRY(dev_alloc(&d.ids, static_cast<size_t>(n_blocks) * 32));
  a.ids = d.ids;
  GX_CUDA(cudaMemcpyAsync(d.round_base, base.data(), sizeof(unsigned long long) * a.n_inst, cudaMemcpyHostToDevice, s));
  const int ctas = e->n_sm * 8, split = batch_split(longest, 4096, ctas, n, 8);
  batch_fill_kernel<<<split * std::min(n, ctas / split), 256, 0, s>>>(a, split);
  GX_CUDA(cudaGetLastError());
  // Every status counts: a graph that lacks the kernel would end well, with
  // the results as the memory happened to be.
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  std::unique_lock<std::shared_mutex> capturing(capture_mutex());
  GX_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  cudaError_t err = cudaMemsetAsync(a.ctr, 0, sizeof(unsigned int), s);
  if (err == cudaSuccess) err = cudaMemsetAsync(a.team, 0, sizeof(unsigned int) * 4 * static_cast<size_t>(a.n_inst), s);
  if (err == cudaSuccess) err = cudaMemsetAsync(a.abort, 0, sizeof(unsigned int), s);
  if (err == cudaSuccess) {
    batch_kernel<<<blocks, t.threads, smem, s>>>(a);
    err = cudaGetLastError();
  }
  const cudaError_t end_err = cudaStreamEndCapture(s, &graph);
  capturing.unlock();
  if (err == cudaSuccess) err = end_err;
  if (err == cudaSuccess) err = cudaGraphInstantiate(&exec, graph, 0);
  if (graph) cudaGraphDestroy(graph);
  if (err != cudaSuccess) {
    cudaGetLastError();
    return fail(GX_ERR_CUDA, "gx_batch: launch: %s", cudaGetErrorString(err));
  }
  err = cudaGraphLaunch(exec, s);
  if (err == cudaSuccess) err = cudaEventRecord(e1, s);
  if (err == cudaSuccess) err = cudaEventSynchronize(e1);
  float t_ms = 0;
  if (err == cudaSuccess) cudaEventElapsedTime(&t_ms, e0, e1);
  cudaGraphExecDestroy(exec);
  if (err != cudaSuccess) return fail(GX_ERR_CUDA, "gx_batch: run failed: %s", cudaGetErrorString(err));
  unsigned int aborted = 0;
  GX_CUDA(cudaMemcpy(&aborted, a.abort, sizeof(aborted), cudaMemcpyDeviceToHost));
  if (aborted) return fail(GX_ERR_TIMEOUT, "gx_batch: a CTA team barrier timed out");
  *ms = t_ms;
  return GX_OK;
}

gx_status check_tuning(const gx_batch_tuning& t) {
  if (t.threads < 64 || t.threads > 1024 || t.threads % 32 || t.lane_max < 0 || t.ctas_per_sm < 1)
    return fail(GX_ERR_INVALID, "gx_batch: bad tuning (threads %d, lane_max %d, ctas_per_sm %d)", t.threads,
                t.lane_max, t.ctas_per_sm);
  return GX_OK;
}

// One call, or one schedule of the autotuner.
struct BatchCall {
  const int32_t* vbeg;
  int32_t n, pr_iters, cc_max;
  double damping;
  gx_batch_tuning tuning;
  float* pr_out = nullptr;         // nullable, as are the others
  int32_t *cc_out = nullptr, *pr_steps = nullptr, *cc_steps = nullptr;
  bool checked = false;            // batch_check
  float ms = 0;
  int32_t launches = 0;
};

gx_status batch_ranges(const gx_engine* e, int32_t n, const int32_t* vbeg) {
  if (vbeg[0] != 0 || vbeg[n] != e->V) return fail(GX_ERR_INVALID, "gx_batch: instance ranges must cover [0, V)");
  for (int32_t i = 0; i < n; ++i)
    if (vbeg[i + 1] <= vbeg[i]) return fail(GX_ERR_INVALID, "gx_batch: instance %d is empty or out of order", i);
  return GX_OK;
}

// Instances [i0, i1) at once, or, where the device has no room for that (the
// rewritten lists take some 4 bytes an edge, the arrays 60 a vertex), one half
// of the work after the other.
gx_status batch_range(gx_engine* e, BatchCall& c, int32_t i0, int32_t i1) {
  const int32_t n = i1 - i0, v0 = c.vbeg[i0], v1 = c.vbeg[i1];
  const int32_t* vbeg = c.vbeg + i0;
  auto run = [&]() -> gx_status {
    BatchDev d;
    BatchArgs a;
    GX_TRY(batch_prepare(e, n, vbeg, !c.checked, d, a));
    c.checked = true;
    a.pr_iters = c.pr_iters;
    a.cc_max = c.cc_max;
    a.lane_max = c.tuning.lane_max;
    a.damping = c.damping;
    float ms = 0;
    GX_TRY(batch_launch(e, vbeg, d, a, c.tuning, &ms));
    c.ms += ms;
    ++c.launches;
    const size_t v = static_cast<size_t>(v1 - v0), m = static_cast<size_t>(n);
    if (c.pr_out) GX_TRY(copy_to_host(e, c.pr_out + v0, d.pr_out, sizeof(float) * v));
    if (c.cc_out) GX_TRY(copy_to_host(e, c.cc_out + v0, d.cc_out, sizeof(int32_t) * v));
    if (c.pr_steps) GX_CUDA(cudaMemcpy(c.pr_steps + i0, d.pr_steps, sizeof(int32_t) * m, cudaMemcpyDeviceToHost));
    if (c.cc_steps) GX_CUDA(cudaMemcpy(c.cc_steps + i0, d.cc_steps, sizeof(int32_t) * m, cudaMemcpyDeviceToHost));
    return GX_OK;
  };
  const gx_status st = run();
  if (st != GX_ERR_OOM || n == 1) return st;
  if (!c.checked) {  // all instances, before any results are written
    struct Words {
      int32_t* p = nullptr;
      ~Words() { dev_free(&p); }
    } w;
    GX_TRY(dev_alloc(&w.p, static_cast<size_t>(c.n) + 2));
    GX_TRY(batch_check(e, c.n, c.vbeg, w.p, reinterpret_cast<unsigned int*>(w.p + c.n + 1)));
    c.checked = true;
  }
  const int64_t half = (e->off[v0] + e->off[v1] + v0 + v1) / 2;
  int32_t mid = i0 + 1;
  while (mid < i1 - 1 && e->off[c.vbeg[mid]] + c.vbeg[mid] < half) ++mid;
  GX_TRY(batch_range(e, c, i0, mid));
  return batch_range(e, c, mid, i1);
}

}  // namespace

extern "C" {

void gx_batch_tuning_default(gx_batch_tuning* t) {
  if (!t) return;
  t->threads = 512;
  t->lane_max = 32;
  t->ctas_per_sm = 2;
}

gx_status gx_batch_run(gx_engine* e, int32_t n_inst, const int32_t* inst_vbegin, int32_t pr_iters, int32_t cc_max_iter,
                       double damping, const gx_batch_tuning* tuning, float* pr_out, int32_t* cc_out,
                       int32_t* pr_steps, int32_t* cc_steps, gx_run_stats* stats) {
  gx::NvtxRange nvtx_range("gx_batch_run");
  if (!e || n_inst < 1 || !inst_vbegin || pr_iters < 0 || cc_max_iter < 0)
    return fail(GX_ERR_INVALID, "gx_batch_run: bad arguments");
  if (!e->loaded || !e->all_resident) return fail(GX_ERR_STATE, "gx_batch_run: load the packed graph first (all resident)");
  if (e->relabeled) return fail(GX_ERR_STATE, "gx_batch_run: the engine renumbered the vertices (config.relabel)");
  gx_batch_tuning t;
  gx_batch_tuning_default(&t);
  if (tuning) t = *tuning;
  GX_TRY(check_tuning(t));
  GX_CUDA(cudaSetDevice(e->dev));
  BlockBound bound(e->block_bound);
  GX_TRY(batch_ranges(e, n_inst, inst_vbegin));
  if (!tuning) GX_TRY(batch_default_schedule(e, n_inst, inst_vbegin, &t));
  std::vector<int32_t> ps(n_inst), cs(n_inst);
  BatchCall c{inst_vbegin, n_inst, pr_iters, cc_max_iter, damping, t};
  c.pr_out = pr_out;
  c.cc_out = cc_out;
  c.pr_steps = ps.data();
  c.cc_steps = cs.data();
  GX_TRY(batch_range(e, c, 0, n_inst));
  if (pr_steps) memcpy(pr_steps, ps.data(), sizeof(int32_t) * n_inst);
  if (cc_steps) memcpy(cc_steps, cs.data(), sizeof(int32_t) * n_inst);
  if (stats) {
    *stats = gx_run_stats{};
    int64_t edges = 0;
    for (int32_t i = 0; i < n_inst; ++i)
      edges += (e->off[inst_vbegin[i + 1]] - e->off[inst_vbegin[i]]) * static_cast<int64_t>(ps[i] + cs[i]);
    stats->iterations = *std::max_element(ps.begin(), ps.end()) + *std::max_element(cs.begin(), cs.end());
    stats->edges_scanned = edges;
    stats->ms_total = c.ms;
    stats->ms_compute = c.ms;
    stats->kernel_launches = c.launches;  // the supersteps; the preparation (check, sort, fill) is not counted
  }
  return GX_OK;
}

gx_status gx_batch_autotune(gx_engine* e, int32_t n_inst, const int32_t* inst_vbegin, int32_t pr_iters,
                            int32_t cc_max_iter, const char* table_path, gx_batch_tuning* best, double* best_ms) {
  gx::NvtxRange nvtx_range("gx_batch_autotune");
  if (!e || !best || n_inst < 1 || !inst_vbegin) return fail(GX_ERR_INVALID, "gx_batch_autotune: bad arguments");
  if (!e->loaded || !e->all_resident) return fail(GX_ERR_STATE, "gx_batch_autotune: load the packed graph first");
  if (e->relabeled) return fail(GX_ERR_STATE, "gx_batch_autotune: the engine renumbered the vertices (config.relabel)");
  GX_CUDA(cudaSetDevice(e->dev));
  BlockBound bound(e->block_bound);
  GX_TRY(batch_ranges(e, n_inst, inst_vbegin));
  bool checked = false;
  const int threads_c[] = {256, 512, 1024};
  const int lane_c[] = {16, 32, 64};
  const int cps_c[] = {1, 2, 4};
  float best_t = 0;
  bool have = false;
  std::string log;
  for (int th : threads_c)
    for (int lm : lane_c)
      for (int cp : cps_c) {
        if (th * cp > 2048) continue;
        gx_batch_tuning t{th, lm, cp};
        float ms = 0;
        for (int warm = 1; warm >= 0; --warm) {
          BatchCall c{inst_vbegin, n_inst, pr_iters, cc_max_iter, 0.85, t};
          c.checked = checked;
          GX_TRY(batch_range(e, c, 0, n_inst));
          checked = true;
          ms = warm ? c.ms : std::min(ms, c.ms);
        }
        char buf[160];
        snprintf(buf, sizeof(buf), "{\"threads\": %d, \"lane_max\": %d, \"ctas_per_sm\": %d, \"ms\": %.4f}", th, lm, cp,
                 ms);
        log += std::string(log.empty() ? "" : ", ") + buf;
        if (!have || ms < best_t) {
          best_t = ms;
          *best = t;
          have = true;
        }
      }
  if (best_ms) *best_ms = best_t;
  if (table_path && *table_path) {
    FILE* f = fopen(table_path, "a");
    if (!f) return fail(GX_ERR_IO, "gx_batch_autotune: cannot append to %s", table_path);
    fprintf(f,
            "{\"instances\": %d, \"vertices\": %d, \"edges\": %lld, \"pr_iters\": %d, \"best\": {\"threads\": %d, "
            "\"lane_max\": %d, \"ctas_per_sm\": %d, \"ms\": %.4f}, \"candidates\": [%s]}\n",
            n_inst, e->V, static_cast<long long>(e->E), pr_iters, best->threads, best->lane_max, best->ctas_per_sm,
            best_t, log.c_str());
    fclose(f);
  }
  return GX_OK;
}

}  // extern "C"
