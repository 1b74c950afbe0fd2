// cg.cu -- congrad (measure_module.F90:9-140) on the device.
//
// Every scalar of the recurrence lives in device memory and is updated by a
// one-thread kernel, so the host only enqueues iterations and polls a
// `done` flag every few iterations; iterations enqueued after convergence
// return immediately (each kernel tests `done` first).  Vector work per
// iteration: x1 = M p | |x1|^2 | x2 = M^dagger x1 | r -= alpha x2, |r|^2 |
// x += alpha p, p = r + beta p.
#include <mutex>

#include "ctx.h"
#include "solver.h"
#include "steps.h"
#include "thr_reduce.cuh"

namespace thr {

namespace {
constexpr int kThreads = 256;

__device__ __forceinline__ double block_sum(double v) {
  __shared__ double sh[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) sh[w] = v;
  __syncthreads();
  int nw = (blockDim.x + 31) >> 5;
  v = (threadIdx.x < nw) ? sh[threadIdx.x] : 0.0;
  if (w == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  return v;
}

__global__ void k_cg_norm2(const CgState* cs, const double2* a, size_t n, double* partials) {
  if (cs->done) return;
  double acc = 0.0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    double2 v = a[i];
    acc += v.x * v.x + v.y * v.y;
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) partials[blockIdx.x] = acc;
}

// measure_module.F90:57, :66-75 (one block; fixed-order reduction of the partials)
__global__ void k_cg_alpha(CgState* cs, const double* partials, int np) {
  pdl_wait();
  pdl_trigger();
  if (cs->done) return;
  const double alphad = block_sum_partials(partials, np);
  if (threadIdx.x != 0) return;
  cs->nx += 1;
  cs->itercg += 1;
  if (cs->nx != 1) cs->alpha = cs->alphan / alphad;
  cs->nalpha = -cs->alpha;
}

// r = r - alpha*x2 (:92) fused with betacgn = |r|^2 (:102)
__global__ void k_cg_rupdate(CgState* cs, double2* r, const double2* x2, size_t n, double* partials) {
  if (cs->done) return;
  const double alpha = cs->alpha;
  double acc = 0.0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    double2 v = r[i] - alpha * x2[i];
    r[i] = v;
    acc += v.x * v.x + v.y * v.y;
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) partials[blockIdx.x] = acc;
}

// :102-110, :120 (one block)
__global__ void k_cg_beta(CgState* cs, const double* partials, int np) {
  pdl_wait();
  pdl_trigger();
  if (cs->done) return;
  const double betacgn = block_sum_partials(partials, np);
  if (threadIdx.x != 0) return;
  double betacg = betacgn / cs->betacgd;
  cs->betacgd = betacgn;
  cs->alphan = betacgn;
  if (cs->nx == 1) betacg = 0.0;
  cs->betacg = betacg;
  cs->betacgn = betacgn;
  if (!(betacgn == betacgn)) { cs->status = THR_ERR_NAN; cs->pending_done = 1; }
  if (betacgn < cs->resid) cs->pending_done = 1;
  else if (cs->nx >= cs->niterc) { cs->pending_done = 1; cs->capped = 1; }
}

// x = x + alpha*p (:77, skipped at nx == 1); p = r + betacg*p (:119); then latch done
// in site order: a thread takes the four spin planes of one (s, site) element of
// the plane (np = n / 4 elements); rev: from the top site down
__global__ void k_cg_xp(CgState* cs, double2* x, double2* p, const double2* r, size_t np, int rev) {
  pdl_wait();
  pdl_trigger();
  if (cs->done) return;
  const double alpha = cs->alpha, beta = cs->betacg;
  const bool upd = cs->nx != 1;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < np; e += (size_t)gridDim.x * blockDim.x) {
    const size_t i0 = rev ? np - 1 - e : e;
#pragma unroll
    for (int d = 0; d < 4; d++) {
      const size_t i = i0 + d * np;
      const double2 pv = p[i];
      if (upd) x[i] = x[i] + alpha * pv;
      p[i] = r[i] + beta * pv;
    }
  }
}
__global__ void k_cg_latch(CgState* cs) {
  pdl_wait();
  pdl_trigger();
  if (cs->pending_done) cs->done = 1;
}

// graph-driven loop: another chunk unless done; max_chunks bounds the loop
// whatever the device state holds (congrad itself stops at niterc)
__global__ void k_cg_loop(CgState* cs, cudaGraphConditionalHandle h) {
  cs->chunks += 1;
  unsigned more = (cs->done || cs->pending_done) ? 0u : 1u;
  if (more && cs->chunks >= cs->max_chunks) {
    cs->status = THR_ERR_MAXITER;
    cs->done = 1;
    more = 0u;
  }
  cudaGraphSetConditional(h, more);
}

inline unsigned vec_grid(size_t n) {
  size_t b = (n + kThreads - 1) / kThreads;
  if (b > device_sms() * 8) b = device_sms() * 8;
  return (unsigned)(b ? b : 1);
}

constexpr int kCgChunk = 8;

// one chunk of kCgChunk iterations (stream order)
int cg_enqueue_chunk(thr_ctx* c, CgState* cs, double2* X, double2* p, double2* r, double2* x1, double2* x2, float am,
                     int imass) {
  const size_t n = c->n4();
  const unsigned gb = vec_grid(n / 4);
  const unsigned gs = stencil_parts(c->g, c->p.kernel, true);
  // every kernel of the chain is a programmatic dependent launch of the one before (the
  // chunk's first, which follows the loop control, excepted; THR_PDL=0: none); each waits
  // for its predecessor before it reads anything, so the results are the same
  const bool pdl = c->use_pdl;
  const bool steps = !c->prof_on && cg_steps_apply(c);  // the chain while kernels are timed, as the multishift
  for (int k = 0; k < kCgChunk; k++) {
    // sweep directions alternate with the iteration's parity (kCgChunk is even): each
    // kernel starts on the sites its predecessor wrote last (results do not depend on it)
    const int odd = c->rev_sweep == 2 ? (k & 1) : 0;
    const int rev_m = odd, rev_md = c->rev_sweep ? 1 - odd : 0, rev_p = odd;
    if (steps) {  // small lattices: three kernels, the scalar steps inside (steps.cu)
      THR_TRY(cg_step_iteration(c, cs, X, p, r, x1, am, imass, k, rev_m, rev_md, rev_p, c->st, pdl));
      continue;
    }
    // x1 = M p with alphad = |x1|^2 (:60, :70) from the stencil's epilogue
    THR_TRY(launch_dslash_norm<double2>(c->g, c->p.kernel, false, x1, p, c->u64, am, imass, c->p.am3, c->st,
                                        &cs->done, c->partials, rev_m, pdl && k > 0));
    launch_k(k_cg_alpha, dim3(1), dim3(1024), 0, c->st, pdl, cs, (const double*)c->partials, (int)gs);
    // x2 = M^dagger x1 is never stored: the epilogue forms r = r - alpha*x2 (:92) and
    // betacgn = |r|^2 (:102)
    THR_TRY(launch_dslash_axpy<double2>(c->g, c->p.kernel, true, r, x1, c->u64, am, imass, c->p.am3, c->st, &cs->done,
                                        r, &cs->nalpha, c->partials, rev_md, pdl));
    launch_k(k_cg_beta, dim3(1), dim3(1024), 0, c->st, pdl, cs, (const double*)c->partials, (int)gs);
    launch_k(k_cg_xp, dim3(gb), dim3(kThreads), 0, c->st, pdl, cs, X, p, (const double2*)r, n / 4, rev_p);
    launch_k(k_cg_latch, dim3(1), dim3(1), 0, c->st, pdl, cs);
  }
  return cudaPeekAtLastError() == cudaSuccess ? THR_OK : THR_ERR_CUDA;
}

// The chain's two stencils once on separate fields (x1, x2 and the partials are scratch), so
// that the tuner settles them: before a graph bakes them in, and before a host-launched chunk
// updates r in place, which is never timed
int cg_settle(thr_ctx* c, CgState* cs, const double2* p, const double2* r, double2* x1, double2* x2, float am,
              int imass) {
  if (c->cg_settled) return THR_OK;
  THR_TRY(launch_dslash_norm<double2>(c->g, c->p.kernel, false, x1, p, c->u64, am, imass, c->p.am3, c->st, &cs->done,
                                      c->partials));
  THR_TRY(launch_dslash_axpy<double2>(c->g, c->p.kernel, true, x2, x1, c->u64, am, imass, c->p.am3, c->st, &cs->done,
                                      r, &cs->nalpha, c->partials, c->rev_sweep ? 1 : 0));
  c->cg_settled = true;
  return THR_OK;
}

// The chunk loop as one CUDA graph (WHILE node), cached per buffers and operator.
struct CgGraph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  const void *X = nullptr, *p = nullptr, *r = nullptr, *x1 = nullptr, *x2 = nullptr, *cs = nullptr;
  const void *u = nullptr, *partials = nullptr;
  float am = 0.f, am3 = 0.f;
  int imass = 0, kernel = -1;
  size_t n = 0;
  void release() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    exec = nullptr;
    graph = nullptr;
  }
};

int cg_graph_build(thr_ctx* c, CgState* cs, double2* X, double2* p, double2* r, double2* x1, double2* x2, float am,
                   int imass, cudaGraphExec_t* exec_out);

// a graph that cannot be built with dependent launches is built without them
int cg_graph(thr_ctx* c, CgState* cs, double2* X, double2* p, double2* r, double2* x1, double2* x2, float am,
             int imass, cudaGraphExec_t* exec_out) {
  int rc = cg_graph_build(c, cs, X, p, r, x1, x2, am, imass, exec_out);
  if (rc != THR_OK && c->use_pdl) {
    c->use_pdl = false;
    rc = cg_graph_build(c, cs, X, p, r, x1, x2, am, imass, exec_out);
  }
  return rc;
}

int cg_graph_build(thr_ctx* c, CgState* cs, double2* X, double2* p, double2* r, double2* x1, double2* x2, float am,
                   int imass, cudaGraphExec_t* exec_out) {
  if (!c->cg_graph) c->cg_graph = new CgGraph();
  CgGraph& G = *static_cast<CgGraph*>(c->cg_graph);
  if (G.exec && G.X == X && G.p == p && G.r == r && G.x1 == x1 && G.x2 == x2 && G.cs == cs && G.u == c->u64 &&
      G.partials == c->partials && G.am == am && G.am3 == c->p.am3 && G.imass == imass && G.kernel == c->p.kernel &&
      G.n == c->n4()) {
    *exec_out = G.exec;
    return THR_OK;
  }
  G.release();
  if (!cg_steps_apply(c)) THR_TRY(cg_settle(c, cs, p, r, x1, x2, am, imass));
  THR_CUDA(cudaGraphCreate(&G.graph, 0));
  cudaGraphConditionalHandle handle;
  THR_CUDA(cudaGraphConditionalHandleCreate(&handle, G.graph, 1, cudaGraphCondAssignDefault));
  cudaGraphNodeParams cp = {};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = handle;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t node;
  THR_CUDA(cudaGraphAddNode(&node, G.graph, nullptr, 0, &cp));
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  THR_CUDA(cudaStreamBeginCaptureToGraph(c->st, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  int rc = cg_enqueue_chunk(c, cs, X, p, r, x1, x2, am, imass);
  if (rc == THR_OK) k_cg_loop<<<1, 1, 0, c->st>>>(cs, handle);
  cudaGraph_t captured = nullptr;
  const cudaError_t ce = cudaStreamEndCapture(c->st, &captured);
  if (rc != THR_OK || ce != cudaSuccess || cudaGraphInstantiate(&G.exec, G.graph, 0) != cudaSuccess) {
    G.release();
    cudaGetLastError();
    return rc != THR_OK ? rc : THR_ERR_CUDA;
  }
  G.X = X; G.p = p; G.r = r; G.x1 = x1; G.x2 = x2; G.cs = cs; G.u = c->u64; G.partials = c->partials;
  G.am = am; G.am3 = c->p.am3; G.imass = imass; G.kernel = c->p.kernel; G.n = c->n4();
  *exec_out = G.exec;
  return THR_OK;
}
}  // namespace

void cg_graph_release(thr_ctx* c) {
  if (c->cg_graph) {
    static_cast<CgGraph*>(c->cg_graph)->release();
    delete static_cast<CgGraph*>(c->cg_graph);
    c->cg_graph = nullptr;
  }
}

// Runs congrad on device fields: Phi (rhs), X (guess in, solution out).
int congrad_dev(thr_ctx* c, const double2* Phi, double2* X, float res, float am, int imass, int niterc, int* itercg,
                int* iterations) {
  const size_t n = c->n4();
  THR_TRY(c->ensure_w64(6));
  double2 *p = c->w64[2], *r = c->w64[3], *x1 = c->w64[4], *x2 = c->w64[5];
  CgState* cs = reinterpret_cast<CgState*>(c->dscal);
  CgState h{};
  // resid = 4*ksize*ksize*ksizet*kthird*res*res in default real (measure_module.F90:41)
  int ivol = 4 * c->g.lx * c->g.ly * c->g.lt * c->g.ls;
  float resid = ((float)ivol * res) * res;
  h.resid = (double)resid;
  h.alpha = 1.0;
  h.alphan = 0.0;
  h.betacgd = h.bd[0] = 1.0;
  h.niterc = niterc;
  h.max_chunks = niterc / kCgChunk + 3;
  THR_CUDA(cudaMemcpyAsync(cs, &h, sizeof(CgState), cudaMemcpyHostToDevice, c->st));
  THR_CUDA(cudaMemcpyAsync(p, X, n * sizeof(double2), cudaMemcpyDeviceToDevice, c->st));
  THR_CUDA(cudaMemcpyAsync(r, Phi, n * sizeof(double2), cudaMemcpyDeviceToDevice, c->st));
  if (c->use_graphs && !c->prof_on) {
    cudaGraphExec_t exec = nullptr;
    THR_TRY(cg_graph(c, cs, X, p, r, x1, x2, am, imass, &exec));
    THR_CUDA(cudaGraphLaunch(exec, c->st));
    THR_CUDA(cudaMemcpyAsync(&h, cs, sizeof(CgState), cudaMemcpyDeviceToHost, c->st));
    THR_CUDA(cudaStreamSynchronize(c->st));
  } else {
    if (c->prof_on || !cg_steps_apply(c)) THR_TRY(cg_settle(c, cs, p, r, x1, x2, am, imass));
    for (int base = 0; base < niterc + kCgChunk; base += kCgChunk) {
      THR_TRY(cg_enqueue_chunk(c, cs, X, p, r, x1, x2, am, imass));
      THR_CUDA(cudaMemcpyAsync(&h, cs, sizeof(CgState), cudaMemcpyDeviceToHost, c->st));
      THR_CUDA(cudaStreamSynchronize(c->st));
      if (h.done || h.pending_done) break;
    }
  }
  if (itercg) *itercg = h.itercg;
  // Fortran DO semantics: nx ends at niterc+1 when the loop runs out (:124)
  if (iterations) *iterations = h.capped ? h.nx + 1 : h.nx;
  if (h.status) return h.status;
  return h.capped ? THR_ERR_MAXITER : THR_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free congrad.  Some callers cannot allocate device memory at the
// point where they solve: a code that must keep its device footprint fixed
// once its fields are placed (memory handed out by its own pool or by an
// OpenACC/OpenMP runtime, with nothing left for a library to cudaMalloc), or
// one that solves where an allocation would synchronise the device or is not
// permitted.  thr_congrad_static takes the fields on the device from the
// caller and keeps everything else it needs -- the four CG work vectors, the
// per-block partial sums and the recurrence scalars -- in one array that is
// part of the library's image (a file-scope __device__ array), so the call
// itself allocates nothing.
namespace {
constexpr size_t kStaticScratchBytes = size_t(32) << 20;  // 32 MiB on every device that loads the library
constexpr int kStaticMaxDevices = 64;
__device__ __align__(256) unsigned char g_cg_scratch[kStaticScratchBytes];
std::mutex g_scratch_mu;
unsigned char* g_scratch_dev[kStaticMaxDevices] = {};  // device address of g_cg_scratch, per device

// device address of the scratch array on the current device (set up once per device)
int static_scratch(unsigned char** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kStaticMaxDevices) return THR_ERR_CUDA;
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (!g_scratch_dev[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_cg_scratch) != cudaSuccess || !p) return THR_ERR_CUDA;
    g_scratch_dev[dev] = static_cast<unsigned char*>(p);
  }
  *out = g_scratch_dev[dev];
  return THR_OK;
}
inline size_t align256(size_t b) { return (b + 255) & ~size_t(255); }
}  // namespace

}  // namespace thr

using namespace thr;

extern "C" int thr_congrad_static(const thr_params* prm, const void* u, const void* Phi, void* X, float res,
                                  int* itercg, float am, int imass, int* iterations, void* stream) {
  if (!prm || !u || !Phi || !X) return THR_ERR_BADARG;
  if (imass != 1 && imass != 3 && imass != 5) return THR_ERR_BADARG;
  if (prm->kernel != 0 && prm->kernel != 1) return THR_ERR_BADARG;
  if (prm->lx < 2 || prm->ly < 2 || prm->lt < 2 || prm->ls < 1 || prm->ls > 1024) return THR_ERR_BADSHAPE;
  if (prm->layout == 1 && prm->lx % 2 != 0) return THR_ERR_BADSHAPE;
  const Geom g = geom_make(prm->lx, prm->ly, prm->lt, prm->ls, prm->layout);
  const size_t n = (size_t)g.v5 * 4;
  const unsigned gb = vec_grid(n);
  // scratch layout: state | partials | p | r | x1 | x2
  const size_t off_parts = align256(sizeof(CgState));
  const size_t off_vec = off_parts + align256((size_t)gb * sizeof(double));
  const size_t vbytes = align256(n * sizeof(double2));
  if (off_vec + 4 * vbytes > kStaticScratchBytes) return THR_ERR_BADSHAPE;  // lattice too large for the fixed scratch
  unsigned char* base = nullptr;
  THR_TRY(static_scratch(&base));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  CgState* cs = reinterpret_cast<CgState*>(base);
  double* partials = reinterpret_cast<double*>(base + off_parts);
  double2* p = reinterpret_cast<double2*>(base + off_vec);
  double2* r = reinterpret_cast<double2*>(base + off_vec + vbytes);
  double2* x1 = reinterpret_cast<double2*>(base + off_vec + 2 * vbytes);
  double2* x2 = reinterpret_cast<double2*>(base + off_vec + 3 * vbytes);
  const double2* ud = static_cast<const double2*>(u);
  double2* Xd = static_cast<double2*>(X);
  // every call starts from a freshly written state (the array keeps the last call's contents)
  CgState h{};
  int ivol = 4 * g.lx * g.ly * g.lt * g.ls;
  float resid = ((float)ivol * res) * res;  // measure_module.F90:41
  h.resid = (double)resid;
  h.alpha = 1.0;
  h.alphan = 0.0;
  h.betacgd = 1.0;
  h.niterc = g.ls * g.v3;  // params.F90:57
  THR_CUDA(cudaMemcpyAsync(cs, &h, sizeof(CgState), cudaMemcpyHostToDevice, st));
  THR_CUDA(cudaMemcpyAsync(p, Xd, n * sizeof(double2), cudaMemcpyDeviceToDevice, st));
  THR_CUDA(cudaMemcpyAsync(r, Phi, n * sizeof(double2), cudaMemcpyDeviceToDevice, st));
  const int chunk = 8;
  for (int base_it = 0; base_it < h.niterc + chunk; base_it += chunk) {
    for (int k = 0; k < chunk; k++) {
      // fixed-footprint stencils: no autotuner timing runs on the caller's stream
      THR_TRY(launch_dslash_untuned<double2>(g, prm->kernel, false, x1, p, ud, am, imass, prm->am3, st, &cs->done));
      k_cg_norm2<<<gb, kThreads, 0, st>>>(cs, x1, n, partials);
      k_cg_alpha<<<1, 1024, 0, st>>>(cs, partials, gb);
      THR_TRY(launch_dslash_untuned<double2>(g, prm->kernel, true, x2, x1, ud, am, imass, prm->am3, st, &cs->done));
      k_cg_rupdate<<<gb, kThreads, 0, st>>>(cs, r, x2, n, partials);
      k_cg_beta<<<1, 1024, 0, st>>>(cs, partials, gb);
      k_cg_xp<<<vec_grid(n / 4), kThreads, 0, st>>>(cs, Xd, p, r, n / 4, 0);
      k_cg_latch<<<1, 1, 0, st>>>(cs);
    }
    THR_CUDA(cudaMemcpyAsync(&h, cs, sizeof(CgState), cudaMemcpyDeviceToHost, st));
    THR_CUDA(cudaStreamSynchronize(st));
    if (h.done) break;
  }
  if (itercg) *itercg = h.itercg;
  if (iterations) *iterations = h.capped ? h.nx + 1 : h.nx;
  if (h.status) return h.status;
  return h.capped ? THR_ERR_MAXITER : THR_OK;
}

extern "C" int thr_congrad(thr_ctx* c, const double* Phi, double* X, float res, int* itercg, float am, int imass,
                           int* iterations) {
  if (!c || !Phi || !X) return THR_ERR_BADARG;
  if (imass != 1 && imass != 3 && imass != 5) return THR_ERR_BADARG;
  cudaSetDevice(c->dev);
  THR_TRY(c->ensure_w64(6));
  THR_TRY(c->use_links(nullptr));
  THR_TRY(c->upload_spinor(c->w64[0], Phi));
  THR_TRY(c->upload_spinor(c->w64[1], X));
  int niterc = c->g.ls * c->g.v3;  // params.F90:57
  int rc = congrad_dev(c, c->w64[0], c->w64[1], res, am, imass, niterc, itercg, iterations);
  if (rc != THR_OK && rc != THR_ERR_MAXITER) return rc;
  THR_TRY(c->download_spinor(X, c->w64[1]));
  int rs = c->sync();
  return rs ? rs : rc;
}
