// steps.h -- solver iterations on small lattices with the scalar steps inside the
// stencil kernels (steps.cu): Shamir; the multishift in FP64 and FP32, congrad in FP64.
#pragma once
#include "ctx.h"
#include "ms.h"
#include "solver.h"

namespace thr {

// whether the context's lattice takes them (its device is current)
bool ms_steps_apply(const thr_ctx* c, bool fp64);
bool cg_steps_apply(const thr_ctx* c);
// the second array of stencil partials (the first is c->partials)
double* steps_partials2(const thr_ctx* c);

// iteration j of a batch of the batched multishift: h = M r_old + gammag h_prev and
// r_new = r_old + omega M^dagger h, with the lambda step of iteration j - 1 and the alpha
// step of iteration j inside; the batch's last lambda step is the caller's (k_lambda on
// steps_partials2)
template <class V>
int ms_step_iteration(thr_ctx* c, MsState* ms, MsHist* rec, V* rold, V* rnew, V* hcur, const V* hprev, float am,
                      int imass, int j, int rev_md, cudaStream_t st, bool pdl);

// iteration k of a chunk of congrad: h = M p with |h|^2; r -= alpha M^dagger h with |r|^2 and
// the alpha step inside; x += alpha p, p = r + betacg p with the beta step inside
int cg_step_iteration(thr_ctx* c, CgState* cs, double2* X, double2* p, double2* r, double2* h, float am, int imass,
                      int k, int rev_m, int rev_md, int rev_p, cudaStream_t st, bool pdl);

}  // namespace thr
