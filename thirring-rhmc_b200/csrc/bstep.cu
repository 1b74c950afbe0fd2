// bstep.cu -- one CG step of the batched congrad (bcg.cu) as three dependent kernels, for
// the Shamir operator: h = M p with |h|^2, r -= alpha M^dagger h with |r|^2, and
// e += alpha p with p = r + beta p.
//
// The entries' scalars cost two launches of one warp per entry between these
// (k_alpha, k_beta in bcg.cu: 6 us each, as long as the stencils of a small batch), and the
// five launches are issued from the host one by one.  Here every block sums its entry's
// partials itself: the M^dagger kernel in a warp beside the stencil, the last one in its
// first warp while the others load; the entry's first block alone advances its state.  Each
// kernel is a programmatic dependent of the one before and looks up its work (the table is
// constant during the solve) before it waits.
//
// Measured against the five kernels (one B200): six FP64 lattices of 8^3x8 to 14^3x20 in a
// pack 28 us per iteration instead of 48; eight FP32 right-hand sides on 16^3, Ls 24 66
// instead of 112 (there the pair accesses of even Ls count most).  Entries of more than
// kStepMaxBlocks work blocks keep the five: every block of an entry reads all its partials.
//
// Nothing a kernel reads is written by it: partials alternate between two arrays, rr
// between two slots by the step's parity, and an entry's end is raised in skip by the last
// kernel (read by the stencils) and copied to skip2 by the M^dagger kernel (read by the
// last).
//
// A stencil block is a work block and writes one partial, summed in block_partial's order, and
// the consumer adds an entry's partials in warp_entry_sum's, so FP64 sums keep the bits of the
// five-kernel step.  (Half work blocks with a partial per warp had a finer tail, but every
// block of the next kernel then reads eight times as many partials: 33 instead of 28 us per
// iteration for the pack below.)
#include "batch.h"
#include "bcg.h"
#include "dslash_site.cuh"
#include "thr_kernels.h"

namespace thr {

namespace {
// stencil threads of a block: a work block, one s per thread (PAIR: two)
constexpr int b_threads(bool pair) { return pair ? 128 : 256; }

// loads of fields the kernel also writes (not through the read-only path)
__device__ __forceinline__ void ldw_pair(const float2* p, size_t i, float2& a, float2& b) {
  const float4 v = *reinterpret_cast<const float4*>(p + i);
  a = make_float2(v.x, v.y);
  b = make_float2(v.z, v.w);
}
template <class S>
__device__ __forceinline__ typename Sto<S>::C ldw(const S* p, size_t i) {
  if constexpr (sizeof(S) == sizeof(__nv_bfloat162)) return __bfloat1622float2(p[i]);
  else return p[i];
}

// a work block's entry, as far as the kernels use it
struct Work {
  Geom g;
  long long off, uoff;
  int e, blk0, spb, nblk;
};
__device__ __forceinline__ Work work_of(const BatchEntry* tab, const int* wmap, int wb) {
  Work w;
  w.e = wmap[wb];
  const BatchEntry& E = tab[w.e];
  w.g = E.g;
  w.off = E.off;
  w.uoff = E.uoff;
  w.blk0 = E.blk0;
  w.spb = E.spb;
  w.nblk = E.nblk;
  return w;
}

// sum of the entry's partials (one per work block) in every lane of a warp, in
// warp_entry_sum's order; eight loads in flight
__device__ __forceinline__ double entry_sum(const double* part, int blk0, int nblk, int lane) {
  constexpr int kU = 8;
  part += blk0;
  double v = 0.0;
  for (int i0 = lane; i0 < nblk; i0 += 32 * kU) {
    double w[kU];
#pragma unroll
    for (int r = 0; r < kU; r++) w[r] = i0 + 32 * r < nblk ? __ldcg(part + i0 + 32 * r) : 0.0;
#pragma unroll
    for (int r = 0; r < kU; r++)
      if (i0 + 32 * r < nblk) v += w[r];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <class S>
struct BStep {
  using C = typename Sto<S>::C;
  const BatchEntry* tab;
  const int* wmap;
  BcgState* stt;
  int *skip, *skip2;
  const C* u;
  S *p, *h;
  C *r, *e;
  double *pa, *pb;  // partials of |h|^2 and |r|^2
  float am, am3;
  int imass, step, cap;
};

// The stencils.  DAG false: h = M p, partials of |h|^2.  DAG true: r -= alpha M^dagger h,
// alpha = rr / |h|^2, partials of |r|^2, with a warp more for alpha.  PAIR: two consecutive s
// per thread (FP32, even Ls: 16-byte accesses), else one s per thread.  A block per work
// block.
template <class S, bool DAG, bool PAIR, int MINB>
__global__ void __launch_bounds__(b_threads(PAIR) + (DAG ? 32 : 0), MINB) k_bstencil(BStep<S> a) {
  using C = typename Sto<S>::C;
  using R = typename Sto<S>::R;
  __shared__ R s_alpha;
  constexpr int kPer = PAIR ? 2 : 1, kThr = b_threads(PAIR);
  const int tid = threadIdx.x, lane = tid & 31;
  const int wb = blockIdx.x;
  const Work w = work_of(a.tab, a.wmap, wb);
  const Geom g = w.g;
  const int row = g.ls / kPer;
  const int sub = tid / row, s = kPer * (tid - sub * row);
  const int site = (wb - w.blk0) * w.spb + sub;
  const bool scal = DAG && tid >= kThr;
  const bool live = !scal && sub < w.spb && site < g.v3;
  const bool lead = wb == w.blk0;
  pdl_wait();
  pdl_trigger();
  if (a.skip[w.e]) {
    if (DAG && lead && tid == 0) a.skip2[w.e] = 1;
    return;
  }
  const S* in = (DAG ? a.h : a.p) + w.off;
  C acc[kPer][4];
  if (live) {
    if constexpr (PAIR) shamir_pair<C, DAG>(in, a.u + w.uoff, g, s, site, a.am, a.imass, a.am3, acc[0], acc[1]);
    else shamir_one<S, DAG>(in, a.u + w.uoff, g, s, site, a.am, a.imass, a.am3, acc[0]);
  }
  if constexpr (DAG) {
    if (scal) {
      const double rr = a.stt[w.e].rr2[a.step & 1];
      const double alpha = rr / entry_sum(a.pa, w.blk0, w.nblk, lane);
      if (lane == 0) {
        s_alpha = (R)alpha;
        if (lead) a.stt[w.e].alpha = alpha;
      }
    }
    __syncthreads();
    if (scal) return;
  }
  double racc = 0.0;
  if (live) {
#pragma unroll
    for (int d = 0; d < 4; d++) {
      const unsigned i = sidx32(g, s, site, d);
      if constexpr (DAG) {
        const R al = s_alpha;
        C* r = a.r + w.off;
        if constexpr (PAIR) {
          C r0, r1;
          ldw_pair(r, i, r0, r1);
          r0 = r0 - al * acc[0][d];
          r1 = r1 - al * acc[1][d];
          st_pair(r, i, r0, r1);
          racc += epi_norm<S>(r0) + epi_norm<S>(r1);
        } else {
          const C rn = r[i] - al * acc[0][d];  // r = r - alpha M^dagger M p (measure_module.F90:92)
          r[i] = rn;
          racc += epi_norm<S>(rn);
        }
      } else {
        if constexpr (PAIR) {
          st_pair(reinterpret_cast<C*>(a.h + w.off), i, acc[0][d], acc[1][d]);
          racc += epi_norm<S>(acc[0][d]) + epi_norm<S>(acc[1][d]);
        } else {
          Sto<S>::st(a.h + w.off, i, acc[0][d]);
          racc += epi_norm<S>(acc[0][d]);
        }
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) racc += __shfl_down_sync(0xffffffffu, racc, o);
  double* part = DAG ? a.pb : a.pa;
  __shared__ double red[kThr / 32];
  if (lane == 0) red[tid >> 5] = racc;
  asm volatile("bar.sync 1, %0;" ::"n"(kThr) : "memory");  // the stencil's threads only
  if (tid == 0) {  // in block_partial's order
    if constexpr (PAIR) part[wb] = (red[0] + red[1]) + (red[2] + red[3]);
    else part[wb] = ((red[0] + red[4]) + (red[2] + red[6])) + ((red[1] + red[5]) + (red[3] + red[7]));
  }
}

// e += alpha p (:91), p = r + beta p (:110), beta = |r|^2 / rr; the entry's first block
// advances its state and raises skip when its solve has ended.  A block per work block,
// each thread the four spins of one s (PAIR: two).
template <class S, bool PAIR>
__global__ void __launch_bounds__(b_threads(PAIR), PAIR ? 6 : 3) k_bxp(BStep<S> a) {
  using C = typename Sto<S>::C;
  using R = typename Sto<S>::R;
  __shared__ double s_rn;
  constexpr int kPer = PAIR ? 2 : 1;
  const int tid = threadIdx.x;
  const int wb = blockIdx.x;
  const Work w = work_of(a.tab, a.wmap, wb);
  const Geom g = w.g;
  const int row = g.ls / kPer, sub = tid / row, s = kPer * (tid - sub * row);
  const int site = (wb - w.blk0) * w.spb + sub;
  const bool live = sub < w.spb && site < g.v3;
  pdl_wait();
  pdl_trigger();
  if (a.skip2[w.e]) return;
  BcgState& st = a.stt[w.e];
  const R al = (R)st.alpha;
  const double rr = st.rr2[a.step & 1];
  const bool capped = a.step + 1 >= a.cap || st.iters0 + a.step + 1 >= st.cap;
  const double target = st.target;
  C pv[kPer][4], ev[kPer][4], rv[kPer][4];
  if (live) {
#pragma unroll
    for (int d = 0; d < 4; d++) {
      const size_t i = (size_t)w.off + sidx32(g, s, site, d);
      if constexpr (PAIR) {
        ldw_pair(reinterpret_cast<const C*>(a.p), i, pv[0][d], pv[1][d]);
        ldw_pair(a.e, i, ev[0][d], ev[1][d]);
        ldw_pair(a.r, i, rv[0][d], rv[1][d]);
      } else {
        pv[0][d] = ldw<S>(a.p, i);
        ev[0][d] = a.e[i];
        rv[0][d] = a.r[i];
      }
    }
  }
  if (tid < 32) {
    const double rn = entry_sum(a.pb, w.blk0, w.nblk, tid);
    if (tid == 0) s_rn = rn;
  }
  __syncthreads();
  const double rn = s_rn;
  const double beta = rn / rr;
  const R be = (R)beta;
  const bool last = !(rn > target) || capped || !(rn == rn);
  if (live) {
#pragma unroll
    for (int d = 0; d < 4; d++) {
      const size_t i = (size_t)w.off + sidx32(g, s, site, d);
#pragma unroll
      for (int k = 0; k < kPer; k++) {
        ev[k][d].x += al * pv[k][d].x;
        ev[k][d].y += al * pv[k][d].y;
        pv[k][d] = mk(rv[k][d].x + be * pv[k][d].x, rv[k][d].y + be * pv[k][d].y);
      }
      if constexpr (PAIR) {
        st_pair(a.e, i, ev[0][d], ev[1][d]);
        if (!last) st_pair(reinterpret_cast<C*>(a.p), i, pv[0][d], pv[1][d]);
      } else {
        a.e[i] = ev[0][d];
        if (!last) Sto<S>::st(a.p, i, pv[0][d]);
      }
    }
  }
  if (wb == w.blk0 && tid == 0) {
    st.beta = beta;
    st.rr = rn;
    st.rr2[(a.step + 1) & 1] = rn;
    st.iters += 1;
    st.inner_it += 1;
    if (!(rn == rn)) {
      st.status = THR_ERR_NAN;
      st.done_outer = 1;
    }
    if (last) {
      st.done_inner = 1;
      a.skip[w.e] = 1;
    }
  }
}

// MB, MD: resident blocks per SM of the M and the (larger) M^dagger blocks
template <class S, bool PAIR, int MB, int MD>
void launch_step(const BStep<S>& a, int blocks, cudaStream_t st, bool pdl) {
  constexpr int kThr = b_threads(PAIR);
  launch_k(k_bstencil<S, false, PAIR, MB>, dim3(blocks), dim3(kThr), 0, st, pdl, a);
  launch_k(k_bstencil<S, true, PAIR, MD>, dim3(blocks), dim3(kThr + 32), 0, st, pdl, a);
  launch_k(k_bxp<S, PAIR>, dim3(blocks), dim3(kThr), 0, st, pdl, a);
}
}  // namespace

template <class VS, class VA>
int launch_bcg_step(BcgRun& br, VA* r, VS* p, VS* h, VA* e, int step, int inner_cap) {
  using C = typename Sto<VS>::C;
  const BatchTable& t = *br.tab;
  BStep<VS> a;
  a.tab = t.dev;
  a.wmap = t.wmap;
  a.stt = br.state;
  a.skip = br.skip;
  a.skip2 = br.skip + t.nent;
  a.u = sizeof(VS) == sizeof(double2) ? (const C*)(const void*)br.u64 : (const C*)br.ulow;
  a.p = p;
  a.h = h;
  a.r = reinterpret_cast<C*>(r);
  a.e = reinterpret_cast<C*>(e);
  a.pa = br.partials;
  a.pb = br.partials + t.total_blocks;
  a.am = br.am;
  a.am3 = br.am3;
  a.imass = br.imass;
  a.step = step;
  a.cap = inner_cap;
  if constexpr (sizeof(VS) == sizeof(float2)) {
    // pairs, us per iteration with (M, M^dagger) budgets [8, 6] / 6, 5 / 5, 5 / 6, 4: 64 work blocks
    // 17.1 16.6 16.2 16.4; 864 (eight sources on 12^3, Ls 16) 25.3 27.0 27.8 26.2; 1640 37.2 38.7
    // 39.0 38.8; 3280 (eight on 16^3, Ls 24) 68.2 70.4 70.8 75.0; 4096 85.7 90.0 91.0 96.0
    if (t.even_ls) launch_step<VS, true, 8, 6>(a, t.total_blocks, br.st, br.pdl);
    else launch_step<VS, false, 3, 3>(a, t.total_blocks, br.st, br.pdl);
  } else {
    // as many registers as do not cost a wave of blocks against four per SM.  FP64, us per
    // iteration with 2 / 3 / 4 per SM: 156 blocks 16.7 / 17.9 / 16.8; 432 - / 20.3 / 22.4; 512 - /
    // 28.5 / 25.1; 648 - / 30.6 / 31.4; 1145 - / 46.9 / 43.1; 1832 89 / 79 / 76.5
    const int sms = device_sms();
    auto waves = [&](int per) { return (t.total_blocks + per * sms - 1) / (per * sms); };
    if (t.total_blocks <= sms) launch_step<VS, false, 1, 1>(a, t.total_blocks, br.st, br.pdl);
    else if (waves(2) == waves(4)) launch_step<VS, false, 2, 2>(a, t.total_blocks, br.st, br.pdl);
    else if (waves(3) == waves(4)) launch_step<VS, false, 3, 3>(a, t.total_blocks, br.st, br.pdl);
    else launch_step<VS, false, 4, 4>(a, t.total_blocks, br.st, br.pdl);
  }
  return cudaPeekAtLastError() == cudaSuccess ? THR_OK : THR_ERR_CUDA;
}

template int launch_bcg_step<double2, double2>(BcgRun&, double2*, double2*, double2*, double2*, int, int);
template int launch_bcg_step<float2, float2>(BcgRun&, float2*, float2*, float2*, float2*, int, int);
template int launch_bcg_step<__nv_bfloat162, float2>(BcgRun&, float2*, __nv_bfloat162*, __nv_bfloat162*, float2*, int,
                                                     int);

}  // namespace thr
