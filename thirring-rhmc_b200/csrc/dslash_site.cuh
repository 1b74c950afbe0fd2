// dslash_site.cuh -- the per-site arithmetic of the domain-wall operator and the
// block body of the one-thread-per-5D-site stencil, shared by the stencil kernels
// (dslash.cu) and the persistent solver kernel of the batched multishift (msp.cu),
// so both run the same instructions per site and give the same bits.
#pragma once
#include "ctx.h"
#include "thr_common.cuh"

namespace thr {


// Spinor loads: COH false reads through the read-only path (__ldg), for fields no
// thread writes during the launch; COH true through L2 (__ldcg), for the persistent
// solver kernel, whose blocks read fields other blocks wrote earlier in the same launch.
template <class S, bool COH>
__device__ __forceinline__ typename Sto<S>::C sto_ld(const S* p, size_t i) {
  if constexpr (COH) return Sto<S>::ldcg(p, i);
  else return Sto<S>::ld(p, i);
}

template <class S, bool COH = false>
struct SpinorView {
  const S* p;
  Geom g;
  __device__ __forceinline__ typename Sto<S>::C operator()(int s, int site, int d) const {
    return sto_ld<S, COH>(p, sidx32(g, s, site, d));
  }
};

// Re(conj(aux_i) v) in the working precision, accumulated in FP64 (for FP32
// storage the term is an FP32 value summed in FP64, as reduce_real_dp5d does)
template <class S>
__device__ __forceinline__ double epi_redot(const S* aux, size_t i, typename Sto<S>::C v) {
  using R = typename Sto<S>::R;
  const typename Sto<S>::C a = Sto<S>::ld(aux, i);
  const R t = a.x * v.x + a.y * v.y;
  return (double)t;
}

// |v|^2 in the working precision (x^2 fused onto the rounded y^2), accumulated in FP64
template <class S>
__device__ __forceinline__ double epi_norm(typename Sto<S>::C v) {
  if constexpr (sizeof(v.x) == sizeof(double)) return __fma_rn(v.x, v.x, __dmul_rn(v.y, v.y));
  else return (double)__fmaf_rn(v.x, v.x, __fmul_rn(v.y, v.y));
}

// ---------------------------------------------------------------- Shamir
// One hop of the 3D Wilson-Dirac term, spin-projected.  The reference adds
// -1/2 [T(d) -+ 2gamma(mu,d) T(gin)] with T = W R(neighbour) for each d
// (dirac.F90:49-76, :464-491).  2gamma(mu,.) is a Hermitian unitary permutation
// (entries +-1, +-i) pairing each upper spin with a lower one, so
//   h(d) = R(d) -+ 2gamma(mu,d) R(gin)   for the upper spins d = 0, 1
// carries the whole hop: W h(d) goes to spin d and -+2gamma(mu,gin) W h(d) to
// spin gin.  Two complex multiplies per neighbour instead of four; the result
// differs from the unprojected sum by rounding only.
// The hop in two parts: hop_products forms W h(d) for d = 0, 1 from the neighbour's
// spinor, hop_accumulate adds them into the site's sums (the four-threads-per-site
// stencil runs the two parts in different threads).
template <class C>
__device__ __forceinline__ void hop_products(int mu, bool plus, C W, const C* r, C* wh) {
#pragma unroll
  for (int d = 0; d < 2; d++) {
    const GammaEntry ge = gamma_entry(mu, d);
    const C gr = gp(ge, r[ge.gin]);
    wh[d] = cmul(W, plus ? r[d] - gr : r[d] + gr);
  }
}
template <class C, class R>
__device__ __forceinline__ void hop_accumulate(int mu, bool plus, const C* wh, C* acc) {
#pragma unroll
  for (int d = 0; d < 2; d++) {
    const int gi = gamma_entry(mu, d).gin;
    acc[d] = acc[d] - R(0.5) * wh[d];
    const C gw = gp(gamma_entry(mu, gi), wh[d]);
    acc[gi] = plus ? acc[gi] + R(0.5) * gw : acc[gi] - R(0.5) * gw;
  }
}
// the two parts in one pass, d by d (the one-thread-per-site kernels)
template <class C, class R>
__device__ __forceinline__ void hop_projected(int mu, bool plus, C W, const C* r, C* acc) {
#pragma unroll
  for (int d = 0; d < 2; d++) {
    const GammaEntry ge = gamma_entry(mu, d);
    const int gi = ge.gin;
    const C gr = gp(ge, r[gi]);
    const C wh = cmul(W, plus ? r[d] - gr : r[d] + gr);
    acc[d] = acc[d] - R(0.5) * wh;
    const C gw = gp(gamma_entry(mu, gi), wh);
    acc[gi] = plus ? acc[gi] + R(0.5) * gw : acc[gi] - R(0.5) * gw;
  }
}

// The rounding of diag R(s) - R(s +- 1) is fixed, so that solutions and iteration counts do
// not depend on what the compiler fuses in one kernel or another.  The single-lattice FP64
// kernels round the product by itself (mul_rn); the batched solver's stencils and the FP32
// pairs fuse it with the difference for all but the first A spin (diag_minus; k: the k-th
// spin of A, 2 + k: of B).
__device__ __forceinline__ double2 mul_rn(double d, double2 a) {
  return make_double2(__dmul_rn(d, a.x), __dmul_rn(d, a.y));
}
__device__ __forceinline__ float2 diag_minus(int k, float diag, float2 c, float2 n) {
  if (k == 0) return make_float2(__fsub_rn(__fmul_rn(diag, c.x), n.x), __fsub_rn(__fmul_rn(diag, c.y), n.y));
  return make_float2(__fmaf_rn(diag, c.x, -n.x), __fmaf_rn(diag, c.y, -n.y));
}
__device__ __forceinline__ double2 diag_minus(int k, double diag, double2 c, double2 n) {
  if (k == 0) return make_double2(__dsub_rn(__dmul_rn(diag, c.x), n.x), __dsub_rn(__dmul_rn(diag, c.y), n.y));
  return make_double2(__fma_rn(diag, c.x, -n.x), __fma_rn(diag, c.y, -n.y));
}
// The site-local terms of the Shamir operator (diagonal, fifth-dimension hop, wall mass
// term) into acc.  SHFL: the fifth-dimension neighbours and wall values come from the
// lanes of the same site (blockDim.x = Ls a power of two <= 32, so a site's Ls threads
// are one aligned segment of a warp); every lane must call this.
template <class S, bool DAG, bool SHFL, bool COH = false>
__device__ __forceinline__ void shamir_local(const S* __restrict__ in, const Geom& g, int s, int site, float am,
                                             int imass, float am3, typename Sto<S>::C* acc) {
  using R = typename Sto<S>::R;
  using C = typename Sto<S>::C;
  SpinorView<S, COH> Rv{in, g};
  const int Ls = g.ls;
  const R diag = (R)((3.0f - am3) + 1.0f);  // dirac.F90:45, default real
  C rc[4];
#pragma unroll
  for (int d = 0; d < 4; d++) {
    rc[d] = Rv(s, site, d);
    if constexpr (sizeof(R) == sizeof(double)) acc[d] = mul_rn(diag, rc[d]);
    else acc[d] = diag * rc[d];
  }
  // fifth-dimension hop (np_third == 1), dirac.F90:80-87 (M), :317-324 (M^dagger):
  // spins A take R(s+1), spins B take R(s-1); A = (2,3) for M, (0,1) for M^dagger
  const int a0 = DAG ? 0 : 2, b0 = DAG ? 2 : 0;
  C nxt[2], prv[2], w0[2], wl[2];
  if (SHFL) {
    const unsigned full = 0xffffffffu;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      nxt[k] = mk(__shfl_down_sync(full, rc[a0 + k].x, 1, Ls), __shfl_down_sync(full, rc[a0 + k].y, 1, Ls));
      prv[k] = mk(__shfl_up_sync(full, rc[b0 + k].x, 1, Ls), __shfl_up_sync(full, rc[b0 + k].y, 1, Ls));
      w0[k] = mk(__shfl_sync(full, rc[a0 + k].x, 0, Ls), __shfl_sync(full, rc[a0 + k].y, 0, Ls));
      wl[k] = mk(__shfl_sync(full, rc[b0 + k].x, Ls - 1, Ls), __shfl_sync(full, rc[b0 + k].y, Ls - 1, Ls));
    }
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    if (s < Ls - 1) acc[a0 + k] = acc[a0 + k] - (SHFL ? nxt[k] : Rv(s + 1, site, a0 + k));
    if (s > 0) acc[b0 + k] = acc[b0 + k] - (SHFL ? prv[k] : Rv(s - 1, site, b0 + k));
  }
  // wall mass term: dirac.F90:119-176 (M), :356-402 (M^dagger).  imass 1, 3 couple
  // R(1) into s = Ls (spins A) and R(Ls) into s = 1 (spins B); imass 5 mixes the
  // chiralities at the same s.  Written as acc += c * v with one coefficient per
  // wall: imass 1: am; imass 3: +i am (A), -i am (B); imass 5: +-i am (M / M^dagger).
  const R a = (R)am;
  const bool five = imass == 5;
  const C cA = imass == 1 ? mk(a, R(0)) : mk(R(0), (five && DAG) ? -a : a);
  const C cB = imass == 1 ? mk(a, R(0)) : mk(R(0), five ? (DAG ? -a : a) : -a);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    if (s == Ls - 1)
      acc[a0 + k] = acc[a0 + k] + cmul(cA, five ? rc[b0 + k] : (SHFL ? w0[k] : Rv(0, site, a0 + k)));
    if (s == 0)
      acc[b0 + k] = acc[b0 + k] + cmul(cB, five ? rc[a0 + k] : (SHFL ? wl[k] : Rv(Ls - 1, site, b0 + k)));
  }
}

// The whole Shamir operator at one 5D site: the local terms, then the Wilson and Dirac
// hopping terms, forward (U R(x+mu)) then backward (conj U(x-mu) R(x-mu)) per
// direction; +gamma forward and -gamma backward in M, the opposite in M^dagger.  The
// reference adds them before (M) or after (M^dagger) the fifth-dimension and mass
// terms; the order only affects rounding.
template <class S, bool DAG, bool SHFL, bool COH = false>
__device__ __forceinline__ void shamir_site(const S* __restrict__ in, const typename Sto<S>::C* __restrict__ u,
                                            const Geom& g, int s, int site, float am, int imass, float am3,
                                            typename Sto<S>::C* acc) {
  using R = typename Sto<S>::R;
  using C = typename Sto<S>::C;
  int x, y, t;
  site_coords(g, site, x, y, t);
  const Nbr nb = neighbours(g, site, x, y, t);
  SpinorView<S, COH> Rv{in, g};
  shamir_local<S, DAG, SHFL, COH>(in, g, s, site, am, imass, am3, acc);
#pragma unroll
  for (int mu = 0; mu < 3; mu++) {
#pragma unroll
    for (int dir = 0; dir < 2; dir++) {
      const int ns = dir == 0 ? nb.f[mu] : nb.b[mu];
      const C W = dir == 0 ? __ldg(u + (size_t)mu * g.v3 + site) : cconj(__ldg(u + (size_t)mu * g.v3 + nb.b[mu]));
      C r[4];
#pragma unroll
      for (int d = 0; d < 4; d++) r[d] = Rv(s, ns, d);
      hop_projected<C, R>(mu, (dir == 0) != DAG, W, r, acc);
    }
  }
}

// shamir_site with the batch rounding
template <class S, bool DAG>
__device__ __forceinline__ void shamir_one(const S* __restrict__ in, const typename Sto<S>::C* __restrict__ u,
                                           const Geom& g, int s, int site, float am, int imass, float am3,
                                           typename Sto<S>::C* acc) {
  using R = typename Sto<S>::R;
  using C = typename Sto<S>::C;
  int x, y, t;
  site_coords(g, site, x, y, t);
  const Nbr nb = neighbours(g, site, x, y, t);
  SpinorView<S> Rv{in, g};
  const int Ls = g.ls;
  const R diag = (R)((3.0f - am3) + 1.0f);
  const int A = DAG ? 0 : 2, B = DAG ? 2 : 0;  // spins taking R(s+1) / R(s-1)
  C rc[4];
#pragma unroll
  for (int d = 0; d < 4; d++) {
    rc[d] = Rv(s, site, d);
    acc[d] = diag * rc[d];
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    if (s < Ls - 1) acc[A + k] = diag_minus(k, diag, rc[A + k], Rv(s + 1, site, A + k));
    if (s > 0) acc[B + k] = diag_minus(2 + k, diag, rc[B + k], Rv(s - 1, site, B + k));
  }
  const R a = (R)am;
  const bool five = imass == 5;
  const C cA = imass == 1 ? mk(a, R(0)) : mk(R(0), (five && DAG) ? -a : a);
  const C cB = imass == 1 ? mk(a, R(0)) : mk(R(0), five ? (DAG ? -a : a) : -a);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    if (s == Ls - 1) acc[A + k] = acc[A + k] + cmul(cA, five ? rc[B + k] : Rv(0, site, A + k));
    if (s == 0) acc[B + k] = acc[B + k] + cmul(cB, five ? rc[A + k] : Rv(Ls - 1, site, B + k));
  }
#pragma unroll
  for (int mu = 0; mu < 3; mu++) {
#pragma unroll
    for (int dir = 0; dir < 2; dir++) {
      const int ns = dir == 0 ? nb.f[mu] : nb.b[mu];
      const C W = dir == 0 ? __ldg(u + (size_t)mu * g.v3 + site) : cconj(__ldg(u + (size_t)mu * g.v3 + nb.b[mu]));
      C r[4];
#pragma unroll
      for (int d = 0; d < 4; d++) r[d] = Rv(s, ns, d);
      hop_projected<C, R>(mu, (dir == 0) != DAG, W, r, acc);
    }
  }
}

// Two consecutive s of one site (s0 even, s0 + 1), Ls even, FP32: the Shamir operator with
// every spinor access a pair (one 16-byte load instead of two of 8).
__device__ __forceinline__ void ld_pair(const float2* p, size_t i, float2& a, float2& b) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(p + i));
  a = make_float2(v.x, v.y);
  b = make_float2(v.z, v.w);
}
__device__ __forceinline__ void st_pair(float2* p, size_t i, float2 a, float2 b) {
  *reinterpret_cast<float4*>(p + i) = make_float4(a.x, a.y, b.x, b.y);
}
template <class C, bool DAG>
__device__ __forceinline__ void shamir_pair(const C* __restrict__ in, const C* __restrict__ u, const Geom& g, int s0,
                                            int site, float am, int imass, float am3, C* a0c, C* a1c) {
  using R = typename Sto<C>::R;
  int x, y, t;
  site_coords(g, site, x, y, t);
  const Nbr nb = neighbours(g, site, x, y, t);
  SpinorView<C> Rv{in, g};
  const int Ls = g.ls;
  const R diag = (R)((3.0f - am3) + 1.0f);
  C c0[4], c1[4];
#pragma unroll
  for (int d = 0; d < 4; d++) {
    ld_pair(in, sidx32(g, s0, site, d), c0[d], c1[d]);
    a0c[d] = diag * c0[d];
    a1c[d] = diag * c1[d];
  }
  const int A = DAG ? 0 : 2, B = DAG ? 2 : 0;  // spins taking R(s+1) / R(s-1)
#pragma unroll
  for (int k = 0; k < 2; k++) {
    a0c[A + k] = diag_minus(k, diag, c0[A + k], c1[A + k]);
    if (s0 + 1 < Ls - 1) a1c[A + k] = diag_minus(k, diag, c1[A + k], Rv(s0 + 2, site, A + k));
    if (s0 > 0) a0c[B + k] = diag_minus(2 + k, diag, c0[B + k], Rv(s0 - 1, site, B + k));
    a1c[B + k] = diag_minus(2 + k, diag, c1[B + k], c0[B + k]);
  }
  const R a = (R)am;
  const bool five = imass == 5;
  const C cA = imass == 1 ? mk(a, R(0)) : mk(R(0), (five && DAG) ? -a : a);
  const C cB = imass == 1 ? mk(a, R(0)) : mk(R(0), five ? (DAG ? -a : a) : -a);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    if (s0 + 1 == Ls - 1) a1c[A + k] = a1c[A + k] + cmul(cA, five ? c1[B + k] : Rv(0, site, A + k));
    if (s0 == 0) a0c[B + k] = a0c[B + k] + cmul(cB, five ? c0[A + k] : Rv(Ls - 1, site, B + k));
  }
#pragma unroll
  for (int mu = 0; mu < 3; mu++) {
#pragma unroll
    for (int dir = 0; dir < 2; dir++) {
      const int ns = dir == 0 ? nb.f[mu] : nb.b[mu];
      const C W = dir == 0 ? __ldg(u + (size_t)mu * g.v3 + site) : cconj(__ldg(u + (size_t)mu * g.v3 + nb.b[mu]));
      C r0[4], r1[4];
#pragma unroll
      for (int d = 0; d < 4; d++) ld_pair(in, sidx32(g, s0, ns, d), r0[d], r1[d]);
      hop_projected<C, R>(mu, (dir == 0) != DAG, W, r0, a0c);
      hop_projected<C, R>(mu, (dir == 0) != DAG, W, r1, a1c);
    }
  }
}

// One block's sites of the stencil with its epilogue (blockDim = (Ls, sites per
// block), NT threads at most; the block's sites are bid * blockDim.y + threadIdx.y).
// Epilogues (EPI): 0 store out = M in; 2 also one FP64 partial of |out|^2 into
// partials[bid]; 1 out = aux + om * (M in), with M in never stored, and a partial of
// |out|^2; 3 out = M in + om * aux with a partial of |out|^2.  The partial goes through
// shared memory and the block's first warp in a fixed order.  A caller that runs
// another block body right after this one must __syncthreads() in between (the
// partial's shared array is reused).  COH: spinor loads through L2 (see sto_ld).
// The persistent multishift kernel runs the same pieces (block_sites, epi_element,
// block_partial_sum) with work of its own between the stencil and its epilogue.

// the epilogue of one output element i from the stencil's value v
template <class S, int EPI, bool COH>
__device__ __forceinline__ void epi_element(S* __restrict__ out, const S* __restrict__ aux, typename Sto<S>::R om,
                                            unsigned i, typename Sto<S>::C v, double& racc) {
  using C = typename Sto<S>::C;
  if (EPI == 1) {
    const C rn = sto_ld<S, COH>(aux, i) + om * v;  // r = r + omega*s (multishift_module.F90:137)
    Sto<S>::st(out, i, rn);
    racc += epi_norm<S>(rn);
  } else if (EPI == 3) {
    const C hn = v + om * sto_ld<S, COH>(aux, i);  // h = M r + gamma h (= M p by linearity)
    Sto<S>::st(out, i, hn);
    racc += epi_norm<S>(hn);
  } else {
    Sto<S>::st(out, i, v);
    if (EPI == 2) racc += epi_norm<S>(v);
  }
}

// one FP64 partial per block in a fixed order.  Blocks of Ls x sites need not be
// whole warps (Ls = 12: 120 threads), so the values go through shared memory and
// the first warp -- always complete: every configuration has >= 32 threads -- sums them.
template <int NT>
__device__ __forceinline__ void block_partial_sum(double racc, double* __restrict__ partials, int bid) {
  __shared__ double red[NT];
  const int tid = threadIdx.x + blockDim.x * threadIdx.y;
  const int nthr = blockDim.x * blockDim.y;
  red[tid] = racc;
  __syncthreads();
  if (tid < 32) {
    double v = 0.0;
    for (int i = tid; i < nthr; i += 32) v += red[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (tid == 0) partials[bid] = v;
  }
}

template <class S, bool DAG, int EPI, int NT, bool SHFL, bool COH = false>
__device__ __forceinline__ void dslash_block(S* __restrict__ out, const S* __restrict__ in,
                                             const typename Sto<S>::C* __restrict__ u, const Geom& g, float am,
                                             int imass, float am3, const S* __restrict__ aux,
                                             typename Sto<S>::R om, int bid, double* __restrict__ partials) {
  using C = typename Sto<S>::C;
  const int s = threadIdx.x;
  double racc = 0.0;
  const int site = bid * blockDim.y + threadIdx.y;
  const bool live = site < g.v3;
  if (SHFL || live) {  // with SHFL every lane takes part (the last block's spare rows on a clamped site)
    const int st = live ? site : g.v3 - 1;
    C acc[4];
    shamir_site<S, DAG, SHFL, COH>(in, u, g, s, st, am, imass, am3, acc);
    if (live) {
#pragma unroll
      for (int d = 0; d < 4; d++) epi_element<S, EPI, COH>(out, aux, om, sidx32(g, s, site, d), acc[d], racc);
    }
  }
  if (EPI != 0) block_partial_sum<NT>(racc, partials, bid);
}

// the stencil part of dslash_block alone: the thread's M in (acc); spare rows compute a
// clamped site (SHFL) or nothing
template <class S, bool DAG, bool SHFL, bool COH = false>
__device__ __forceinline__ void block_sites(const S* __restrict__ in, const typename Sto<S>::C* __restrict__ u,
                                            const Geom& g, float am, int imass, float am3, int bid,
                                            typename Sto<S>::C* acc) {
  const int s = threadIdx.x;
  const int site = bid * blockDim.y + threadIdx.y;
  const bool live = site < g.v3;
  if (SHFL || live) {
    const int st = live ? site : g.v3 - 1;
    shamir_site<S, DAG, SHFL, COH>(in, u, g, s, st, am, imass, am3, acc);
  }
}

// ---------------------------------------------------------------- Wilson, overlap
// The hops are diagonal in s and the links do not depend on s, so the 3D operator D_W and
// the s-combinations of the slices commute: each thread applies the six hops to its own
// slice R(s) only -- four loads per neighbour site, as the Shamir kernel -- and the
// neighbouring slices' results are combined afterwards through shared memory.
//   M:     Q(s) = R(s) + wA P+ R(s-1) + wB P- R(s+1).  A = the hops of the upper spins of
//          R(s) (to all four output spins), B those of the lower spins; then
//          D_W Q(s) = [A + B](s) + wA A(s-1) + wB B(s+1).
//   M^dag: the output's upper spins take D_W^dag (R(s) + w R(s+1)), the lower ones
//          D_W^dag (R(s) + w R(s-1)): one spin-projected hop pass, then one exchange.
// (Building Q at every neighbour first costs 8 to 12 loads per neighbour site.)  The
// overlap operator is the same with slice s's D_W scaled by its coefficient c[s].

// hops of the upper (A) and lower (B) spins of r apart, without the common factor -1/2
template <class C>
__device__ __forceinline__ void hop_halves(int mu, bool plus, C W, const C* r, C* A, C* B) {
#pragma unroll
  for (int d = 0; d < 4; d++) {
    const C T = cmul(W, r[d]);
    const int gi = gamma_entry(mu, d).gin;
    const C gt = gp(gamma_entry(mu, gi), T);
    C* X = d < 2 ? A : B;
    X[d] = X[d] + T;
    X[gi] = plus ? X[gi] - gt : X[gi] + gt;
  }
}

// One 5D site of the Wilson (OV false) or overlap (OV true) operator.  Every thread of the
// block calls it (live false: a thread without a site); ex: NT x (DAG ? 4 : 8) values in
// shared memory, read by nobody once every thread has returned from a __syncthreads().
// tid - s .. tid - s + Ls - 1 are the threads of this thread's site.  COH: see sto_ld.
template <class S, bool OV, bool DAG, int NT, bool COH = false>
__device__ __forceinline__ void wilson_exchange(const S* __restrict__ in, const typename Sto<S>::C* __restrict__ u,
                                                const Geom& g, int s, int site, bool live, int tid, float am,
                                                int imass, float am3, const double* __restrict__ zc,
                                                typename Sto<S>::C* ex, typename Sto<S>::C* res) {
  using R = typename Sto<S>::R;
  using C = typename Sto<S>::C;
  const int Ls = g.ls;
  const R a = (R)am;
  const R dgw = (R)(3.0f + (-am3));  // DWilson(..., -am3) diagonal: dirac.F90:191, :505
  C r[4], A[4], B[4];
  const S* pl[4];
#pragma unroll
  for (int d = 0; d < 4; d++) pl[d] = in + (size_t)d * (size_t)g.v5;
  if (live) {
    int x, y, t;
    site_coords(g, site, x, y, t);
    const Nbr nb = neighbours(g, site, x, y, t);
    const unsigned i0 = (unsigned)s + (unsigned)Ls * (unsigned)site;
#pragma unroll
    for (int d = 0; d < 4; d++) {
      r[d] = sto_ld<S, COH>(pl[d], i0);
      A[d] = B[d] = mk(R(0), R(0));
    }
    if (DAG) {
#pragma unroll
      for (int d = 0; d < 4; d++) A[d] = (OV ? dgw : dgw - R(1)) * r[d];
    }
#pragma unroll
    for (int mu = 0; mu < 3; mu++) {
#pragma unroll
      for (int dir = 0; dir < 2; dir++) {
        const int ns = dir == 0 ? nb.f[mu] : nb.b[mu];
        const C W = dir == 0 ? __ldg(u + (size_t)mu * g.v3 + site) : cconj(__ldg(u + (size_t)mu * g.v3 + nb.b[mu]));
        const unsigned i = (unsigned)s + (unsigned)Ls * (unsigned)ns;
        C q[4];
#pragma unroll
        for (int d = 0; d < 4; d++) q[d] = sto_ld<S, COH>(pl[d], i);
        if (DAG) hop_projected<C, R>(mu, dir != 0, W, q, A);
        else hop_halves<C>(mu, dir == 0, W, q, A, B);
      }
    }
    const R cs = OV ? (R)__ldg(zc + s) : R(1);
    if (DAG) {
#pragma unroll
      for (int d = 0; d < 4; d++) {
        if (OV) A[d] = cs * A[d] - r[d];
        ex[d * NT + tid] = A[d];
      }
    } else {
      const R dd = OV ? dgw : dgw - R(1);
#pragma unroll
      for (int d = 0; d < 4; d++) {
        A[d] = (d < 2) ? dd * r[d] - R(0.5) * A[d] : R(-0.5) * A[d];
        B[d] = (d < 2) ? R(-0.5) * B[d] : dd * r[d] - R(0.5) * B[d];
        ex[d * NT + tid] = A[d];
        ex[(4 + d) * NT + tid] = B[d];
      }
    }
  }
  __syncthreads();
  if (!live) return;
  const bool inp = s > 0, inn = s < Ls - 1;
  const int tp = inp ? tid - 1 : tid + Ls - 1, tn = inn ? tid + 1 : tid - (Ls - 1);
  const R sg = OV ? R(-1) : R(1);  // the overlap module's imass 3 walls have the opposite sign
  // wall factors: wp on the slice before (s = 0: the last one), wn on the slice after
  // M: c1, c2 (dirac.F90:274-278, :287-291); M^dag: z, z' (:602-606, :615-619): the same values;
  // overlap: m1, m2 (measure_OWilson.F90:66-83) and z1, z2 (:139-157)
  const C wp = imass == 1 ? mk(-a, R(0)) : mk(R(0), -sg * a);
  const C wn = imass == 1 ? mk(-a, R(0)) : mk(R(0), sg * a);
  if (DAG) {
#pragma unroll
    for (int d = 0; d < 4; d++) {
      const bool lo = d < 2;  // spins 0,1 from the slice after, 2,3 from the one before
      const C v = ex[d * NT + (lo ? tn : tp)];
      const C w = (lo ? inn : inp) ? v : cmul(lo ? wn : wp, v);
      res[d] = A[d] + R(2) * r[d] + w;
    }
  } else {
    const R cs = OV ? (R)__ldg(zc + s) : R(1);
#pragma unroll
    for (int d = 0; d < 4; d++) {
      const C fa = ex[d * NT + tp], gb = ex[(4 + d) * NT + tn];
      const C v = (A[d] + B[d]) + ((inp ? fa : cmul(wp, fa)) + (inn ? gb : cmul(wn, gb)));
      if (OV) {
        const bool lo = d < 2;
        const C n = sto_ld<S, COH>(pl[d], (unsigned)Ls * (unsigned)site +
                                          (unsigned)(lo ? (inp ? s - 1 : Ls - 1) : (inn ? s + 1 : 0)));
        const C wr = (lo ? inp : inn) ? n : cmul(lo ? wp : wn, n);
        res[d] = cs * v + r[d] - wr;
      } else {
        res[d] = v + R(2) * r[d];
      }
    }
  }
}

}  // namespace thr
