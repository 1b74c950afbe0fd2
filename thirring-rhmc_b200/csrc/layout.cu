// layout.cu -- gather/scatter between the reference's Fortran arrays (with
// one-site halos, column-major) and the device fields.  The Fortran array is
// first copied verbatim into a device staging buffer; these kernels then
// gather its interior (inputs; halos are ignored because the device uses
// periodic indexing) or write the interior plus the periodic images into
// every halo position (outputs), which is what the reference's halo update
// (comms5.F90:135-194 on a 1x1x1x1 grid) leaves there.
#include "thr_common.cuh"
#include "thr_kernels.h"

namespace thr {

namespace {
__device__ __forceinline__ int wrap(int c, int l) { return c < 0 ? c + l : (c >= l ? c - l : c); }

__device__ __forceinline__ size_t f5(const Geom& g, int s, int x, int y, int t, int d) {
  // 0-based interior coordinates -> offset in (0:Ls+1,0:Lx+1,0:Ly+1,0:Lt+1,4)
  return (size_t)(s + 1) +
         (size_t)(g.ls + 2) * ((size_t)(x + 1) + (size_t)(g.lx + 2) * ((size_t)(y + 1) + (size_t)(g.ly + 2) * ((size_t)(t + 1) + (size_t)(g.lt + 2) * d)));
}

// The spinor kernels take one row of the fifth dimension per blockDim.x threads: the
// coordinates are found once per row in 32-bit arithmetic (an element at a time the 64-bit
// divisions were the kernels' time).
template <class S>
__global__ void __launch_bounds__(256) k_from_fortran_spinor(S* out, const double2* fin, Geom g) {
  const unsigned rows = 4u * (unsigned)g.v3;
  for (unsigned r = blockIdx.x * blockDim.y + threadIdx.y; r < rows; r += gridDim.x * blockDim.y) {
    const unsigned d = r / (unsigned)g.v3;
    int x, y, t;
    site_coords(g, (int)(r - d * (unsigned)g.v3), x, y, t);
    const double2* src = fin + f5(g, 0, x, y, t, (int)d);
    const size_t dst = (size_t)r * g.ls;
    for (int s = threadIdx.x; s < g.ls; s += blockDim.x) {
      const double2 v = src[s];
      Sto<S>::st(out, dst + s, typename Sto<S>::C{(typename Sto<S>::R)v.x, (typename Sto<S>::R)v.y});
    }
  }
}

__global__ void __launch_bounds__(256) k_to_fortran_spinor(double2* fout, const double2* in, Geom g) {
  // every element of the halo'd array, interior and halos, gets its periodic image
  const unsigned LX2 = g.lx + 2, LY2 = g.ly + 2, LT2 = g.lt + 2, rows = 4u * LX2 * LY2 * LT2;
  const int LS2 = g.ls + 2;
  for (unsigned i = blockIdx.x * blockDim.y + threadIdx.y; i < rows; i += gridDim.x * blockDim.y) {
    unsigned r = i / LX2;
    const int x = wrap((int)(i - r * LX2) - 1, g.lx);
    const unsigned q = r / LY2;
    const int y = wrap((int)(r - q * LY2) - 1, g.ly);
    const unsigned d = q / LT2;
    const int t = wrap((int)(q - d * LT2) - 1, g.lt);
    const double2* src = in + sidx(g, 0, site_index(g, x, y, t), (int)d);
    double2* dst = fout + (size_t)i * LS2;
    for (int s = threadIdx.x; s < LS2; s += blockDim.x) dst[s] = src[wrap(s - 1, g.ls)];
  }
}

__global__ void k_to_fortran_noh(double2* fout, const double2* in, Geom g) {
  size_t n = (size_t)g.v5 * 4;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    size_t r = i;
    int s = (int)(r % g.ls); r /= g.ls;
    int x = (int)(r % g.lx); r /= g.lx;
    int y = (int)(r % g.ly); r /= g.ly;
    int t = (int)(r % g.lt);
    int d = (int)(r / g.lt);
    fout[i] = in[sidx(g, s, site_index(g, x, y, t), d)];
  }
}

__global__ void k_from_fortran_noh(double2* out, const double2* fin, Geom g) {
  size_t n = (size_t)g.v5 * 4;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    size_t r = i;
    int s = (int)(r % g.ls); r /= g.ls;
    int x = (int)(r % g.lx); r /= g.lx;
    int y = (int)(r % g.ly); r /= g.ly;
    int t = (int)(r % g.lt);
    int d = (int)(r / g.lt);
    out[sidx(g, s, site_index(g, x, y, t), d)] = fin[i];
  }
}

__global__ void k_from_fortran_links(double2* out, const double2* fin, Geom g) {
  int n = g.v3 * 3;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int site = i % g.v3, mu = i / g.v3;
    int x, y, t;
    site_coords(g, site, x, y, t);
    out[i] = fin[(x + 1) + (size_t)(g.lx + 2) * ((y + 1) + (size_t)(g.ly + 2) * ((t + 1) + (size_t)(g.lt + 2) * mu))];
  }
}

__global__ void k_to_fortran_links(double2* fout, const double2* in, Geom g) {
  const int LX2 = g.lx + 2, LY2 = g.ly + 2, LT2 = g.lt + 2;
  int n = LX2 * LY2 * LT2 * 3;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int r = i;
    int x = r % LX2; r /= LX2;
    int y = r % LY2; r /= LY2;
    int t = r % LT2;
    int mu = r / LT2;
    fout[i] = in[(size_t)mu * g.v3 + site_index(g, wrap(x - 1, g.lx), wrap(y - 1, g.ly), wrap(t - 1, g.lt))];
  }
}

template <class T>
__global__ void k_from_fortran_3(T* out, const T* fin, Geom g) {
  int n = g.v3 * 3;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int r = i;
    int x = r % g.lx; r /= g.lx;
    int y = r % g.ly; r /= g.ly;
    int t = r % g.lt;
    int mu = r / g.lt;
    out[(size_t)mu * g.v3 + site_index(g, x, y, t)] = fin[i];
  }
}
template <class T>
__global__ void k_to_fortran_3(T* fout, const T* in, Geom g) {
  int n = g.v3 * 3;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int r = i;
    int x = r % g.lx; r /= g.lx;
    int y = r % g.ly; r /= g.ly;
    int t = r % g.lt;
    int mu = r / g.lt;
    fout[i] = in[(size_t)mu * g.v3 + site_index(g, x, y, t)];
  }
}

__global__ void k_to_fortran_ps(float* fout, const float* in, Geom g) {
  const int LX2 = g.lx + 2, LY2 = g.ly + 2, LT2 = g.lt + 2;
  int n = LX2 * LY2 * LT2 * 2;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int r = i;
    int x = r % LX2; r /= LX2;
    int y = r % LY2; r /= LY2;
    int t = r % LT2;
    int c = r / LT2;
    fout[i] = in[(size_t)c * g.v3 + site_index(g, wrap(x - 1, g.lx), wrap(y - 1, g.ly), wrap(t - 1, g.lt))];
  }
}

// threads along a row of n elements, and the grid for `rows` of them in 256-thread blocks
inline dim3 row_block(int n) {
  const unsigned tx = n <= 8 ? 8 : n <= 16 ? 16 : 32;
  return dim3(tx, 256 / tx);
}
inline unsigned row_grid(size_t rows, dim3 blk) {
  const size_t b = (rows + blk.y - 1) / blk.y, most = (size_t)device_sms() * 32;
  return (unsigned)(b < most ? b : most);
}
inline unsigned grid_for(size_t n, int threads = 256) {
  size_t b = (n + threads - 1) / threads;
  if (b > device_sms() * 32) b = device_sms() * 32;
  if (b < 1) b = 1;
  return (unsigned)b;
}
}  // namespace

template <class S>
void from_fortran_spinor(const Geom& g, S* out, const double2* fin, cudaStream_t st) {
  const dim3 blk = row_block(g.ls);
  k_from_fortran_spinor<S><<<row_grid((size_t)g.v3 * 4, blk), blk, 0, st>>>(out, fin, g);
}
template void from_fortran_spinor<double2>(const Geom&, double2*, const double2*, cudaStream_t);
template void from_fortran_spinor<float2>(const Geom&, float2*, const double2*, cudaStream_t);

void to_fortran_spinor(const Geom& g, double2* fout, const double2* in, cudaStream_t st) {
  const dim3 blk = row_block(g.ls + 2);
  k_to_fortran_spinor<<<row_grid((size_t)(g.lx + 2) * (g.ly + 2) * (g.lt + 2) * 4, blk), blk, 0, st>>>(fout, in, g);
}
int upload_fortran_spinor(const Geom& g, double2* stage, const double* host, cudaStream_t st) {
  const size_t plane = (size_t)(g.ls + 2) * (g.lx + 2) * (g.ly + 2) * sizeof(double2);
  const size_t pitch = plane * (g.lt + 2);
  cudaError_t e;
  // page-locked arrays: without the t halos (2 of Lt + 2 planes; a pageable array goes through
  // the driver's staging buffers faster in one piece: 688 against 720 us at 18x14x10, Ls 20);
  // 2^31: the largest pitch a 2D copy takes
  const bool pending = cudaPeekAtLastError() != cudaSuccess;  // an earlier launch's error: the caller's to report
  cudaPointerAttributes at;
  const bool known = cudaPointerGetAttributes(&at, host) == cudaSuccess;
  if (!known && !pending) cudaGetLastError();
  const bool locked = known && at.type == cudaMemoryTypeHost;
  if (locked && pitch < (size_t)1 << 31) {
    e = cudaMemcpy2DAsync(reinterpret_cast<char*>(stage) + plane, pitch, reinterpret_cast<const char*>(host) + plane,
                          pitch, plane * g.lt, 4, cudaMemcpyHostToDevice, st);
  } else {
    e = cudaMemcpyAsync(stage, host, 4 * pitch, cudaMemcpyHostToDevice, st);
  }
  return e == cudaSuccess ? THR_OK : THR_ERR_CUDA;
}
void to_fortran_noh(const Geom& g, double2* fout, const double2* in, cudaStream_t st) {
  k_to_fortran_noh<<<grid_for((size_t)g.v5 * 4), 256, 0, st>>>(fout, in, g);
}
void from_fortran_noh(const Geom& g, double2* out, const double2* fin, cudaStream_t st) {
  k_from_fortran_noh<<<grid_for((size_t)g.v5 * 4), 256, 0, st>>>(out, fin, g);
}
void from_fortran_links(const Geom& g, double2* out, const double2* fin, cudaStream_t st) {
  k_from_fortran_links<<<grid_for((size_t)g.v3 * 3), 256, 0, st>>>(out, fin, g);
}
void to_fortran_links(const Geom& g, double2* fout, const double2* in, cudaStream_t st) {
  size_t n = (size_t)(g.lx + 2) * (g.ly + 2) * (g.lt + 2) * 3;
  k_to_fortran_links<<<grid_for(n), 256, 0, st>>>(fout, in, g);
}
void from_fortran_f3(const Geom& g, float* out, const float* fin, cudaStream_t st) {
  k_from_fortran_3<float><<<grid_for((size_t)g.v3 * 3), 256, 0, st>>>(out, fin, g);
}
void to_fortran_f3(const Geom& g, float* fout, const float* in, cudaStream_t st) {
  k_to_fortran_3<float><<<grid_for((size_t)g.v3 * 3), 256, 0, st>>>(fout, in, g);
}
void from_fortran_d3(const Geom& g, double* out, const double* fin, cudaStream_t st) {
  k_from_fortran_3<double><<<grid_for((size_t)g.v3 * 3), 256, 0, st>>>(out, fin, g);
}
void to_fortran_d3(const Geom& g, double* fout, const double* in, cudaStream_t st) {
  k_to_fortran_3<double><<<grid_for((size_t)g.v3 * 3), 256, 0, st>>>(fout, in, g);
}
void to_fortran_ps(const Geom& g, float* fout, const float* in, cudaStream_t st) {
  size_t n = (size_t)(g.lx + 2) * (g.ly + 2) * (g.lt + 2) * 2;
  k_to_fortran_ps<<<grid_for(n), 256, 0, st>>>(fout, in, g);
}

}  // namespace thr
