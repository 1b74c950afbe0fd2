// steps.cu -- solver iterations on small lattices, the scalar steps inside the stencils.
//
// On a small lattice an iteration is a chain of dependent kernels of 2 to 3 us each, and
// the one-block kernels that sum the stencils' partials (k_alpha, k_lambda in msb.cu) cost
// as much as the stencils.  Here each stencil block has one warp more, which sums the
// previous stencil's partials itself -- all blocks alike, while the other warps run the
// stencil -- and hands the epilogue its coefficient; a lead block beyond the stencil's has
// only that warp at work and advances the solver state.  The iteration is then two kernels
// instead of four:
//   M step:   lambda of the step before (gammag), h = M r + gammag h, partials of |h|^2
//   M^ step:  alpha (omega), r_new = r + omega M^dagger h, partials of |r_new|^2
// The sums run in block_sum_partials' order, the stencils and the recurrences are the
// kernel chain's, so the bits are the same.  Measured at 12^2x12, Ls 16 (216 blocks): 7.5 us
// per iteration instead of 14.0 (7.9 with the state advanced by a stencil block, 9.8 while
// its copy took a round trip per four rows and every warp waited for the flag first).
//
// Every block reads every partial and holds its epilogue until the sum is known, which pays
// while the grid is one wave (kMsStepPerSm).  us per multishift iteration, FP64 / FP32, these
// kernels against the chain (one B200): 549 blocks (14^3, Ls 24) 11.4 / 10.6 against 16.4 / 14.2;
// 729 (18^3, Ls 16) 15.5 / 10.9, 17.5 / 16.2; 880 (22x20x16, Ls 16) 19.0 / 13.4, 19.7 / 16.3; and
// past one wave 896 (16^2x14, Ls 32) 21.1 / 17.5 against 19.8 / 16.6; 1331 (22^3, Ls 16) 32.0 /
// 21.1, 25.6 / 18.7; 2048 (32^3, Ls 8) 45.6 / 31.9, 33.0 / 22.8.
//
// Nothing a kernel reads is written by it: the sums' input and output partials alternate
// between two arrays, the M step reads delta from dl[] of one parity and writes the other,
// and the flag that ends the work of later kernels (the M step's lambda may set `done`) is
// read as `done` by the M^dagger step and as `halt`, which that one sets, by the M step.
//
// Congrad's iteration is three kernels instead of six in the same way: M p, the M^dagger
// step with alpha inside, and the x and p update with beta inside (pending_done, set by the
// update, is read by the stencils; done, set by the M^dagger step, by the update).  At
// 12^2x12, Ls 16: 10.7 us per iteration instead of 17.5; its third kernel has the sum ahead of
// a pass over memory, so the line is lower (kCgStepPerSm): 549 blocks 16.6 against 21.3, 729
// 21.8 / 22.6, 768 (16^2x12, Ls 32) 23.0 / 23.0, 880 26.1 / 24.3, 1331 40.0 / 32.3.
#include <algorithm>
#include <type_traits>

#include "ctx.h"
#include "dslash_site.cuh"
#include "ms.h"
#include "steps.h"
#include "thr_kernels.h"

namespace thr {

namespace {
constexpr int kStepThreads = 128;                   // the Shamir stencil's blocks
constexpr int kStepBlock = kStepThreads + 32;       // and the scalar warp
constexpr int kStepMaxParts = 1024;                 // one partial per virtual thread of the sum
// blocks per SM up to which the kernels are taken, the lead block included
constexpr int kMsStepPerSm = 6, kCgStepPerSm = 5;

// sum of p[0..n) (n <= 1024) in every lane of one warp, as block_sum_partials adds them
// with 1024 threads: thread i has p[i], each warp's 32 values go through a halving tree, then
// the 32 warp sums.  A butterfly gives the tree's value (lane 0 of the
// tree; the operands of an addition commute) in all lanes.
__device__ __forceinline__ double warp_sum_partials(const double* p, int n, int lane) {
  constexpr int kU = 8;  // virtual warps in flight
  double keep = 0.0;
  for (int w0 = 0; w0 < 32 && w0 * 32 < n; w0 += kU) {
    double v[kU];
#pragma unroll
    for (int k = 0; k < kU; k++) {
      const int i = (w0 + k) * 32 + lane;
      v[k] = i < n ? p[i] : 0.0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int k = 0; k < kU; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    }
#pragma unroll
    for (int k = 0; k < kU; k++)
      if (lane == w0 + k) keep = v[k];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) keep += __shfl_xor_sync(0xffffffffu, keep, o);
  return keep;
}

// ms_alpha_block and ms_lambda_block (ms.h) by one warp
__device__ __forceinline__ void ms_alpha_warp(MsState* ms, MsHist* rec, int nstep, double alpha, int lane) {
  if (lane == 0) {
    ms_alpha_scalar(ms, alpha);
    rec->lo[nstep] = ms->lo;
    rec->hi[nstep] = ms->hi;
  }
  __syncwarp();
  for (int k = ms->lo + lane; k <= ms->hi; k += 32) {
    ms_alpha_shift(ms, k);
    rec->om[nstep][k] = ms->omegas[k];
    rec->ze[nstep][k] = ms->zeta_iii[k];
  }
  __syncwarp();
}
__device__ __forceinline__ void ms_lambda_warp(MsState* ms, MsHist* rec, int nstep, double lambda, int lane) {
  if (lane == 0) ms_lambda_scalar(ms, lambda);
  __syncwarp();
  const int lo0 = ms->lo, hi0 = ms->hi;
  for (int k = lo0 + lane; k <= hi0; k += 32) {
    ms_lambda_shift(ms, k);
    rec->ga[nstep][k] = ms->gammas[k];
  }
  const int nq = ms->ndiagq, it = ms->it;
  const double delta = ms->delta, res = (double)ms->res;
  int mini = nq, maxi = -1;
  for (int q = lane; q < nq; q += 32) {
    if (q >= lo0 && q <= hi0) ms->cg_returns[q] = it;
    if (ms->flags[q]) {
      if (sqrt(delta * ms->zeta_ii[q] * ms->zeta_ii[q]) * ms->correction[q] < res) {
        ms->flags[q] = 0;
      } else {
        mini = min(mini, q);
        maxi = max(maxi, q);
      }
    }
  }
  mini = __reduce_min_sync(0xffffffffu, mini);
  maxi = __reduce_max_sync(0xffffffffu, maxi);
  for (int q = lane; q < kMaxShift; q += 32) {
    if (q >= mini && q <= maxi) {
      ms->zeta_i[q] = ms->zeta_ii[q];
      ms->zeta_ii[q] = ms->zeta_iii[q];
    }
  }
  if (lane == 0) {
    rec->nsteps = nstep + 1;
    ms->lo = mini;
    ms->hi = maxi;
    ms->delta = ms->lambda;
    if (!(ms->lambda == ms->lambda)) ms->status = THR_ERR_NAN;
    if (maxi < mini || ms->it >= ms->maxcg || ms->status) ms->done = 1;
  }
  __syncwarp();
}

template <class C>
struct StepArgs {
  C* out;
  const C* in;
  const C* aux;
  const C* u;
  Geom g;
  float am, am3;
  int imass;
  const double* pin;  // the previous stencil's partials
  double* pout;
  int np;             // partials = stencil blocks
  int spb;            // sites per block
  unsigned mls;       // geom_magic of Ls for thread indices
  int rev;
};

// One stencil block with its scalar warp: coef(lane) runs in the scalar warp beside the
// stencil and returns the epilogue's coefficient, lead(lane) after it in the lead block
// (the grid's last, which has no sites).  EPI 1: r_new = r + c M(^dagger) h; 3: h_new = M r + c h; 2: h =
// M p (no coefficient, no scalar warp).  stop (this kernel's flag, loaded by every thread)
// is looked at only before the first store, so that the stencil's loads do not wait for it.
// PER: consecutive s per thread (2: FP32 storage with even Ls, k_dslash_pair's arithmetic).
template <class C, int PER, bool DAG, int EPI, bool SHFL, class Coef, class Lead>
__device__ __forceinline__ bool step_block(const StepArgs<C>& a, const int stop, Coef&& coef, Lead&& lead) {
  using R = typename Sto<C>::R;
  constexpr int kThr = kStepThreads / PER;
  __shared__ double s_coef;
  __shared__ double red[kThr];
  const Geom g = a.g;
  const int tid = threadIdx.x;
  const bool scal = tid >= kThr;
  const bool leadb = EPI != 2 && blockIdx.x == gridDim.x - 1;  // the block beyond the stencil's
  const int bid = a.rev ? a.np - 1 - (int)blockIdx.x : (int)blockIdx.x;
  C acc[PER][4], av[PER][4];
  int s = 0, site = 0;
  bool live = false;
  if (scal) {
    const double c = coef(tid & 31);
    if (tid == kThr) s_coef = c;
    if (leadb && !stop) lead(tid & 31);
  } else if (!leadb) {
    const int row = g.ls / PER, sub = geom_div(tid, row, a.mls);
    s = PER * (tid - sub * row);
    site = bid * a.spb + sub;
    live = sub < a.spb && site < g.v3;
    if (SHFL || live) {  // with SHFL every lane takes part (spare rows on a clamped site)
      const int sc = live ? site : g.v3 - 1;
      if (EPI != 2) {
#pragma unroll
        for (int d = 0; d < 4; d++) {
#pragma unroll
          for (int k = 0; k < PER; k++) av[k][d] = a.aux[sidx32(g, s, sc, d) + k];
        }
      }
      if constexpr (PER == 2) shamir_pair<C, DAG>(a.in, a.u, g, s, sc, a.am, a.imass, a.am3, acc[0], acc[1]);
      else shamir_site<C, DAG, SHFL>(a.in, a.u, g, s, sc, a.am, a.imass, a.am3, acc[0]);
    }
  }
  if (stop) return false;
  if (leadb) return true;
  if (EPI != 2) __syncthreads();
  if (!scal) {
    const R om = EPI != 2 ? (R)s_coef : R(0);
    double racc = 0.0;
    if (live) {
#pragma unroll
      for (int d = 0; d < 4; d++) {
        C v[PER];
#pragma unroll
        for (int k = 0; k < PER; k++)
          v[k] = EPI == 1 ? av[k][d] + om * acc[k][d] : EPI == 3 ? acc[k][d] + om * av[k][d] : acc[k][d];
        const unsigned i = sidx32(g, s, site, d);
        if constexpr (PER == 2) {
          st_pair(a.out, i, v[0], v[1]);
          racc += epi_norm<C>(v[0]) + epi_norm<C>(v[1]);
        } else {
          a.out[i] = v[0];
          racc += epi_norm<C>(v[0]);
        }
      }
    }
    red[tid] = racc;
  }
  __syncthreads();
  if (tid < 32) {  // the block's partial in block_partial_sum's order
    const int nthr = a.spb * (g.ls / PER);
    double v = 0.0;
    for (int i = tid; i < nthr; i += 32) v += red[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (tid == 0) a.pout[bid] = v;
  }
  return true;
}

// DAG false: the M step of iteration j (with the lambda step of iteration j - 1, unless it
// is the batch's first: that one's was taken by k_lambda); DAG true: the M^dagger step
// (with the alpha step) of iteration j
template <class C, int PER, bool DAG, bool SHFL, int MINB>
__global__ void __launch_bounds__(kStepThreads / PER + 32, MINB)
    k_ms_step(StepArgs<C> a, MsState* ms, MsHist* rec, int j) {
  pdl_wait();
  pdl_trigger();
  __shared__ MsState st;  // the lead block's working copy of the state
  constexpr int kWords = (int)(sizeof(MsState) / sizeof(double)), kRows = (kWords + 31) / 32;
  const bool due = DAG || j > 0;
  const int stop = DAG ? ms->done : ms->halt;
  double total = 0.0;
  const bool ran = step_block<C, PER, DAG, DAG ? 1 : 3, SHFL>(
      a, stop,
      [&](int lane) -> double {
        if (!due) return ms->gammag;
        const double delta = DAG ? ms->delta : ms->dl[(j + 1) & 1];
        if (blockIdx.x == gridDim.x - 1) {  // every load of the copy in flight at once
          const double* src = reinterpret_cast<const double*>(ms);
          double w[kRows];
#pragma unroll
          for (int i = 0; i < kRows; i++) w[i] = lane + 32 * i < kWords ? src[lane + 32 * i] : 0.0;
          total = warp_sum_partials(a.pin, a.np, lane);
          double* dst = reinterpret_cast<double*>(&st);
#pragma unroll
          for (int i = 0; i < kRows; i++)
            if (lane + 32 * i < kWords) dst[lane + 32 * i] = w[i];
          __syncwarp();
        } else {
          total = warp_sum_partials(a.pin, a.np, lane);
        }
        return DAG ? -delta / total : total / delta;  // omega (:126-127), gammag (:143)
      },
      [&](int lane) {
        if (!due) return;
        if (DAG) {
          ms_alpha_warp(&st, rec, j, total, lane);
          if (lane == 0) {
            ms->it = st.it;
            ms->alpha = st.alpha;
            ms->omega_save = st.omega_save;
            ms->omega = st.omega;
          }
          for (int k = lane; k < kMaxShift; k += 32) {
            ms->zeta_iii[k] = st.zeta_iii[k];
            ms->omegas[k] = st.omegas[k];
          }
        } else {
          ms_lambda_warp(&st, rec, j - 1, total, lane);
          if (lane == 0) {
            ms->lambda = st.lambda;
            ms->active_sum = st.active_sum;
            ms->gammag = st.gammag;
            ms->lo = st.lo;
            ms->hi = st.hi;
            ms->delta = st.delta;
            ms->dl[j & 1] = st.delta;
            ms->status = st.status;
            ms->done = st.done;
          }
          for (int k = lane; k < kMaxShift; k += 32) {
            ms->gammas[k] = st.gammas[k];
            ms->cg_returns[k] = st.cg_returns[k];
            ms->flags[k] = st.flags[k];
            ms->zeta_i[k] = st.zeta_i[k];
            ms->zeta_ii[k] = st.zeta_ii[k];
          }
        }
      });
  if (DAG && !ran && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) ms->halt = 1;
}

// r -= alpha M^dagger h (measure_module.F90:92) with the alpha step (:57, :66-75) of
// iteration k of a chunk
template <bool SHFL, int MINB>
__global__ void __launch_bounds__(kStepBlock, MINB) k_cg_step(StepArgs<double2> a, CgState* cs, int k) {
  pdl_wait();
  pdl_trigger();
  const int stop = cs->pending_done;
  double alpha = 1.0;  // the first iteration's
  const bool ran = step_block<double2, 1, true, 1, SHFL>(
      a, stop,
      [&](int lane) -> double {
        const int started = cs->started;
        const double rr = cs->bd[k & 1];
        const double alphad = warp_sum_partials(a.pin, a.np, lane);
        if (started) alpha = rr / alphad;
        return -alpha;
      },
      [&](int lane) {
        if (lane == 0) {
          cs->nx += 1;
          cs->itercg += 1;
          cs->alpha = alpha;
        }
      });
  if (!ran && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) cs->done = 1;
}
// h = M p (:60) with |h|^2 (:70)
template <bool SHFL, int MINB>
__global__ void __launch_bounds__(kStepThreads, MINB) k_cg_m_step(StepArgs<double2> a, const CgState* cs) {
  pdl_wait();
  pdl_trigger();
  step_block<double2, 1, false, 2, SHFL>(a, cs->pending_done, [](int) { return 0.0; }, [](int) {});
}

// x = x + alpha*p (:77, skipped at nx == 1), p = r + betacg*p (:119) with the beta step
// (:102-110, :120); a thread takes the four spin planes of one (s, site) element, its loads
// issued before the sum
__global__ void __launch_bounds__(256) k_cg_update_step(CgState* cs, double2* x, double2* p, const double2* r,
                                                        unsigned np4, int rev, const double* pin, int np, int k) {
  pdl_wait();
  pdl_trigger();
  const int stop = cs->done;
  __shared__ double s_rr;
  const double alpha = cs->alpha, rr_old = cs->bd[k & 1];
  const int nx = cs->nx;
  const unsigned step = gridDim.x * blockDim.x;
  unsigned e = blockIdx.x * blockDim.x + threadIdx.x;
  double2 pv[4], xv[4], rv[4];
  auto load = [&]() {
#pragma unroll
    for (int d = 0; d < 4; d++) {
      const size_t i = (rev ? np4 - 1 - e : e) + (size_t)d * np4;
      pv[d] = p[i];
      xv[d] = x[i];
      rv[d] = r[i];
    }
  };
  if (e < np4) load();
  if (threadIdx.x < 32) {
    const double v = warp_sum_partials(pin, np, threadIdx.x);
    if (threadIdx.x == 0) s_rr = v;
  }
  if (stop) return;
  __syncthreads();
  const double rr = s_rr;
  const double beta = nx == 1 ? 0.0 : rr / rr_old;
  while (e < np4) {
#pragma unroll
    for (int d = 0; d < 4; d++) {
      const size_t i = (rev ? np4 - 1 - e : e) + (size_t)d * np4;
      if (nx != 1) x[i] = xv[d] + alpha * pv[d];
      p[i] = rv[d] + beta * pv[d];
    }
    e += step;
    if (e < np4) load();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    cs->bd[(k + 1) & 1] = rr;
    cs->started = 1;
    if (!(rr == rr)) {
      cs->status = THR_ERR_NAN;
      cs->pending_done = 1;
    }
    if (rr < cs->resid) {
      cs->pending_done = 1;
    } else if (nx >= cs->niterc) {
      cs->pending_done = 1;
      cs->capped = 1;
    }
  }
}

bool step_shfl(const Geom& g) { return g.ls <= 32 && (g.ls & (g.ls - 1)) == 0; }

template <class C>
StepArgs<C> step_args(thr_ctx* c, C* out, const C* in, const C* aux, float am, int imass, const double* pin,
                      double* pout, int rev, int per = 1) {
  const dim3 blk = stencil_block(c->g, 0);
  const C* u;
  if constexpr (sizeof(C) == sizeof(double2)) u = c->u64;
  else u = c->u32;
  return StepArgs<C>{out,  in,   aux,  u, c->g, am, c->p.am3, imass,
                     pin,  pout, (int)stencil_grid(c->g, 0), (int)blk.y,
                     geom_magic(kStepThreads, c->g.ls / per), rev};
}

constexpr int kStepMaxShflBudget = 4;

// launch(integral_constant<int, MB>): the resident blocks per SM (2 to MOST) that a kernel's
// registers are budgeted for: one wave of blocks with as many registers as that leaves (a
// site's loads in flight at once).  The multishift's lead block is one of them: left over it
// holds the next kernel up (296, 592 and 740 blocks, Ls 16: 11.7, 15.9 and 18.3 us per iteration
// without it in the count, 8.4, 13.4 and 17.6 with); congrad's only counts the iterations (12.8,
// 17.4 and 23.3 without, 13.4, 18.4 and 23.3 with).  FP64 multishift, us per iteration with budgets 2 to 6 (the
// rule's marked): 343 blocks (14^3, Ls 16) 12.6 [8.5] 10.4 12.1 14.8; 549 (14^3, Ls 24) 15.9 16.4
// [12.2] 13.3 15.5; 683 (16^3, Ls 20) 20.8 17.2 18.6 [15.2] 16.4; 820 (16^3, Ls 24) 23.5 19.5 20.3
// 22.5 [18.1].  Congrad's stencils alike (343: 13.8 [12.9] 14.3 15.2 17.4; 683: 24.0 22.4 23.3
// [19.7] 21.1).
// Up to four blocks s -+ 1 comes by shuffles where Ls allows it (343 blocks: 8.5 against 9.4; at
// four, where the M^dagger kernels with shuffles spill 20 bytes, either is within 4 %: 512
// blocks, 16^3, Ls 16, multishift 11.9 against 11.4, congrad 15.3 against 15.8); in the registers
// that five or six leave they spill more, and the neighbours are read (729 blocks, 18^3, Ls 16:
// 15.3 against 16.9; 800, 20^2 x 16, Ls 16: 18.2 against 24.0).
template <int MOST, class F>
void with_budget(int blocks, F&& launch) {
  using std::integral_constant;
  const int sms = device_sms();
  if (blocks <= 2 * sms) launch(integral_constant<int, 2>{});
  else if (blocks <= 3 * sms) launch(integral_constant<int, 3>{});
  else if (blocks <= 4 * sms) launch(integral_constant<int, 4>{});
  else if (MOST == 5 || blocks <= 5 * sms) launch(integral_constant<int, 5>{});
  else if constexpr (MOST > 5) launch(integral_constant<int, MOST>{});
}

template <class C, int PER, bool DAG>
void launch_ms_step(const StepArgs<C>& a, MsState* ms, MsHist* rec, int j, cudaStream_t st, bool pdl) {
  const dim3 grd(a.np + 1), blk(kStepThreads / PER + 32);
  auto go = [&](auto mb) {
    constexpr int MB = decltype(mb)::value;
    if constexpr (PER == 1 && MB <= kStepMaxShflBudget) {
      if (step_shfl(a.g)) {
        launch_k(k_ms_step<C, PER, DAG, true, MB>, grd, blk, 0, st, pdl, a, ms, rec, j);
        return;
      }
    }
    launch_k(k_ms_step<C, PER, DAG, false, MB>, grd, blk, 0, st, pdl, a, ms, rec, j);
  };
  if constexpr (PER == 1) {
    with_budget<kMsStepPerSm>(a.np + 1, go);
  } else {
    // blocks of 96 threads: six of them leave the registers a site needs.  us per iteration with
    // budgets 2 / 4 / 6 (the rule's marked): 216 blocks [8.1] 8.1 8.6; 343 8.7 8.7 [9.3]; 549 10.1
    // 10.1 [10.6]; 729 15.6 15.6 [10.9]; 880 17.9 18.0 [13.3]
    if (a.np <= 2 * device_sms()) go(std::integral_constant<int, 2>{});
    else go(std::integral_constant<int, 6>{});
  }
}
}  // namespace

static bool steps_apply(const thr_ctx* c, bool fp64, int per_sm) {
  const unsigned np = stencil_grid(c->g, 0);
  return c->p.kernel == 0 && c->g.ls <= kStepThreads && np <= (unsigned)kStepMaxParts &&
         np + 1 <= (unsigned)(per_sm * device_sms()) && stencil_parts(c->g, 0, fp64) == np &&
         2 * (size_t)np + 2 <= c->nparts;
}
bool ms_steps_apply(const thr_ctx* c, bool fp64) { return steps_apply(c, fp64, kMsStepPerSm); }
bool cg_steps_apply(const thr_ctx* c) { return steps_apply(c, true, kCgStepPerSm); }

double* steps_partials2(const thr_ctx* c) { return c->partials + ((stencil_grid(c->g, 0) + 1) & ~1u); }

template <class V>
int ms_step_iteration(thr_ctx* c, MsState* ms, MsHist* rec, V* rold, V* rnew, V* hcur, const V* hprev, float am,
                      int imass, int j, int rev_md, cudaStream_t st, bool pdl) {
  double *pa = c->partials, *pl = steps_partials2(c);
  auto run = [&](auto per) {
    constexpr int P = decltype(per)::value;
    launch_ms_step<V, P, false>(step_args<V>(c, hcur, rold, hprev, am, imass, pl, pa, 0, P), ms, rec, j, st,
                                pdl && j > 0);
    launch_ms_step<V, P, true>(step_args<V>(c, rnew, hcur, rold, am, imass, pa, pl, rev_md, P), ms, rec, j, st, pdl);
  };
  if constexpr (sizeof(V) == sizeof(float2)) {
    if (c->g.ls % 2 == 0) run(std::integral_constant<int, 2>{});
    else run(std::integral_constant<int, 1>{});
  } else {
    run(std::integral_constant<int, 1>{});
  }
  return cudaPeekAtLastError() == cudaSuccess ? THR_OK : THR_ERR_CUDA;
}
template int ms_step_iteration<double2>(thr_ctx*, MsState*, MsHist*, double2*, double2*, double2*, const double2*,
                                        float, int, int, int, cudaStream_t, bool);
template int ms_step_iteration<float2>(thr_ctx*, MsState*, MsHist*, float2*, float2*, float2*, const float2*, float,
                                       int, int, int, cudaStream_t, bool);

int cg_step_iteration(thr_ctx* c, CgState* cs, double2* X, double2* p, double2* r, double2* h, float am, int imass,
                      int k, int rev_m, int rev_md, int rev_p, cudaStream_t st, bool pdl) {
  double *pa = c->partials, *pb = steps_partials2(c);
  const StepArgs<double2> a = step_args<double2>(c, r, h, r, am, imass, pa, pb, rev_md);
  const StepArgs<double2> m = step_args<double2>(c, h, p, nullptr, am, imass, nullptr, pa, rev_m);
  with_budget<kCgStepPerSm>(a.np, [&](auto mb) {
    constexpr int MB = decltype(mb)::value;
    auto run = [&](auto sh) {
      constexpr bool SH = decltype(sh)::value;
      launch_k(k_cg_m_step<SH, MB>, dim3(a.np), dim3(kStepThreads), 0, st, pdl && k > 0, m, (const CgState*)cs);
      launch_k(k_cg_step<SH, MB>, dim3(a.np + 1), dim3(kStepBlock), 0, st, pdl, a, cs, k);
    };
    if constexpr (MB <= kStepMaxShflBudget) {
      if (step_shfl(a.g)) {
        run(std::true_type{});
        return;
      }
    }
    run(std::false_type{});
  });
  const unsigned np4 = (unsigned)(c->n4() / 4);
  const unsigned gb = std::min((np4 + 255) / 256, (unsigned)(8 * device_sms()));
  launch_k(k_cg_update_step, dim3(gb), dim3(256), 0, st, pdl, cs, X, p, (const double2*)r, np4, rev_p,
           (const double*)pb, a.np, k);
  return cudaPeekAtLastError() == cudaSuccess ? THR_OK : THR_ERR_CUDA;
}

}  // namespace thr
