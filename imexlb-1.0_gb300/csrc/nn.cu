// Convolution kernels of the warm-start neural operator: 3x3 convolutions
// (stride 1 or 2, optional nearest x2 upsampling of the input) on NHWC
// bfloat16 activations, their data and weight gradients, and Adam.
//
// The products run on the 5th-generation tensor cores (tcgen05.mma, bf16
// operands in shared memory, FP32 accumulators in tensor memory), each an
// implicit GEMM over staged halos of the activations (conv_tc.cuh):
//   forward      C[P x Cout]  = im2col(x)[P x 9Cin] * W^T        (P output pixels)
//   data grad    C[G x Cin]   = dz~[G x 9Cout] * Wt^T            (G stencil-grid pixels)
//   weight grad  C[9Cin x Cout] = im2col(x)^T[9Cin x P] * dz[P x Cout]
#include <algorithm>
#include <atomic>
#include <cstdint>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "imexlb_nn.h"
#include "conv_tc.cuh"
#include "pdl.cuh"

namespace {

typedef __nv_bfloat16 bf16;

namespace conv = imx::conv;

// dz = bf16(dy * relu'(y)) over n = pixels*c values, and the bias gradient
// (per-channel sums of dz): block sums in shared memory, one global atomic
// per block and channel.
__global__ void k_act_grad(const float* __restrict__ dy, const bf16* __restrict__ y, int64_t n,
                           int c, int relu, bf16* __restrict__ dz, float* __restrict__ dbias) {
  __shared__ float part[64];
  for (int i = threadIdx.x; i < c; i += blockDim.x) part[i] = 0.0f;
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float g = dy[i];
    if (relu && __bfloat162float(y[i]) <= 0.0f) g = 0.0f;
    dz[i] = __float2bfloat16(g);
    if (dbias) atomicAdd(&part[i % c], g);
  }
  __syncthreads();
  if (dbias)
    for (int i = threadIdx.x; i < c; i += blockDim.x) atomicAdd(&dbias[i], part[i]);
}

// The same for c a multiple of 8 and 16-byte aligned arrays: a thread takes
// 8 channels of one pixel at a time, always the same ones (blockDim is a
// multiple of c/8), and keeps their sums in registers. HBM-bound: 8 bytes a
// value. 16 x 128x256 x 48 (201 MB): 26 us (7.7 TB/s, part of it from L2) against 118 us with a
// shared-memory atomic per value.
constexpr int kActThreads = 256;
__global__ void __launch_bounds__(kActThreads) k_act_grad8(const float4* __restrict__ dy,
                                                           const uint4* __restrict__ y, int64_t n8,
                                                           int groups, int relu, uint4* __restrict__ dz,
                                                           float* __restrict__ dbias) {
  __shared__ float part[kActThreads * 8];
  imx::pdl_wait();
  imx::pdl_trigger();
  const float4* dyp = imx::pdl_fresh(dy);
  const uint4* yp = imx::pdl_fresh(y);
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.0f;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  constexpr int kU = 2;  // items in flight
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += kU * step) {
    float4 a[kU], b[kU];
    uint4 v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int64_t k = i + u * step;
      if (k < n8) {
        a[u] = __ldcs(dyp + 2 * k);
        b[u] = __ldcs(dyp + 2 * k + 1);
        if (relu) v[u] = yp[k];
      }
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int64_t k = i + u * step;
      if (k >= n8) break;
      float g[8] = {a[u].x, a[u].y, a[u].z, a[u].w, b[u].x, b[u].y, b[u].z, b[u].w};
      if (relu) {
        const bf16* e = (const bf16*)&v[u];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (__bfloat162float(e[j]) <= 0.0f) g[j] = 0.0f;
      }
      uint4 o;
      __nv_bfloat162* ob = (__nv_bfloat162*)&o;
#pragma unroll
      for (int j = 0; j < 4; ++j) ob[j] = __floats2bfloat162_rn(g[2 * j], g[2 * j + 1]);
      dz[k] = o;
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += g[j];
    }
  }
  if (!dbias) return;
  // rows of one pixel's channels, summed down the block
#pragma unroll
  for (int j = 0; j < 8; ++j) part[threadIdx.x * 8 + j] = acc[j];
  __syncthreads();
  const int c = groups * 8, rows = blockDim.x / groups;
  for (int i = threadIdx.x; i < c; i += blockDim.x) {
    float s = 0.0f;
    for (int r = 0; r < rows; ++r) s += part[r * c + i];
    atomicAdd(&dbias[i], s);
  }
}

// Sum the 2x2 children of each pixel of an upsampled grid (data grad of the
// nearest x2 upsampling).
__global__ void k_down_sum(const float* __restrict__ du, int n, int h, int w, int c,
                           float* __restrict__ dx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t total = (int64_t)n * h * w * c;
  if (i >= total) return;
  const int ch = (int)(i % c);
  int64_t r = i / c;
  const int x = (int)(r % w);
  r /= w;
  const int y = (int)(r % h);
  const int img = (int)(r / h);
  float s = 0.0f;
  for (int dy2 = 0; dy2 < 2; ++dy2)
    for (int dx2 = 0; dx2 < 2; ++dx2)
      s += du[(((int64_t)img * 2 * h + 2 * y + dy2) * (2 * w) + 2 * x + dx2) * c + ch];
  dx[i] = s;
}

// w to an aligned place, value by value.
__global__ void k_copy_w(const bf16* __restrict__ w, int n, bf16* __restrict__ to) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) to[i] = w[i];
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, bf16* __restrict__ pb, int64_t n, float lr, float b1,
                       float b2, float eps, float bc1, float bc2, float wd) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i] + wd * p[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
  p[i] = pi;
  if (pb) pb[i] = __float2bfloat16(pi);
}

// Mean squared error over the first `used` of `c` channels per pixel, with
// optional per-pixel weights; dy (c channels per pixel, padding channels
// zero) receives d(loss)/dy. Loss partial sums by block into *loss (atomic).
__global__ void k_mse(const float* __restrict__ y, const float* __restrict__ t,
                      const float* __restrict__ w, int64_t npix, int c, int used, float inv_count,
                      float* __restrict__ dy, float* __restrict__ loss) {
  __shared__ float part[256];
  float acc = 0.0f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < npix * c;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t px = i / c;
    const int ch = (int)(i - px * c);
    float g = 0.0f;
    if (ch < used) {
      const float wt = w ? w[px] : 1.0f;
      const float d = y[i] - t[px * used + ch];
      acc += wt * d * d;
      g = 2.0f * wt * d * inv_count;
    }
    dy[i] = g;
  }
  part[threadIdx.x] = acc;
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) part[threadIdx.x] += part[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, part[0] * inv_count);
}

// The same for c a multiple of 4 and 16-byte aligned y, dy: a thread takes
// four channels of a pixel, and reads y only where a used channel is among
// them. 16 x 128x256 x 16 channels, 3 used (57 MB): 10 us against 37 us.
__global__ void __launch_bounds__(256) k_mse4(const float4* __restrict__ y, const float* __restrict__ t,
                                              const float* __restrict__ w, int64_t n4, int cq, int used,
                                              float inv_count, float4* __restrict__ dy,
                                              float* __restrict__ loss) {
  __shared__ float part[8];
  imx::pdl_wait();
  imx::pdl_trigger();
  const float4* yp = imx::pdl_fresh(y);
  const float* tp = imx::pdl_fresh(t);
  const float* wp = imx::pdl_fresh(w);
  float acc = 0.0f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t px;
    if (n4 < (1ll << 31)) px = (int64_t)((uint32_t)i / (uint32_t)cq);
    else px = i / cq;
    const int ch = (int)(i - px * cq) * 4;
    float g[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (ch < used) {
      const float wt = wp ? wp[px] : 1.0f;
      const float4 v = yp[i];
      const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (ch + j < used) {
          const float d = e[j] - tp[px * used + ch + j];
          acc += wt * d * d;
          g[j] = 2.0f * wt * d * inv_count;
        }
    }
    dy[i] = make_float4(g[0], g[1], g[2], g[3]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.0f;
    for (int k = 0; k < 8; ++k) s += part[k];
    atomicAdd(loss, s * inv_count);
  }
}

bool valid(const imexlb_conv_desc* d) {
  if (!d || d->n <= 0 || d->cin <= 0 || d->cin % 16 || d->cout <= 0 || d->cout % 16 || d->cout > 64)
    return false;
  if (d->cout_store < 0 || d->cout_store > d->cout) return false;
  if (d->hin < 0 || d->win < 0) return false;
  if (d->stride != 1 && d->stride != 2) return false;
  const int hg = d->upsample ? 2 * d->hin : d->hin, wg = d->upsample ? 2 * d->win : d->win;
  return d->hout == (hg - 1) / d->stride + 1 && d->wout == (wg - 1) / d->stride + 1;
}

constexpr int kSmemMax = 232448;  // dynamic + static shared memory of a block

// GEMM sizes the calls take (imexlb_nn.h): weights and 128 rows of K within a
// block's shared memory. k_conv_rows stages less than that, so its own check in
// run_rows refuses no more.
bool gemm_fits(int N, int K) {
  return ((N * K * 2 + 1023) / 1024) * 1024 + conv::kTM * K * 2 <= kSmemMax - 16;
}

int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 1;
}

// Launch with `smem` dynamic bytes, as a dependent of the stream's previous
// kernel. The kernel's shared-memory limit is raised once per device, and
// again if a launch is refused (a context made anew): asking for it before
// each launch took 2 to 3 us, as much as the launch.
template <class Args>
cudaError_t launch(void (*kern)(Args), dim3 grid, int threads, int smem, const Args& a, cudaStream_t s) {
  static std::atomic<uint64_t> raised{0};  // per kernel (its Args are its own) and device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  auto raise = [&] {
    cudaFuncAttributes fa;
    cudaError_t r = cudaFuncGetAttributes(&fa, kern);
    if (r == cudaSuccess)
      r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax - (int)fa.sharedSizeBytes);
    if (r == cudaSuccess && dev < 64) raised.fetch_or(1ull << dev);
    return r;
  };
  const bool known = dev < 64 && (raised.load() >> dev & 1u);
  if (!known && (e = raise()) != cudaSuccess) return e;
  e = imx::launch_dependent(kern, grid, (unsigned)threads, (unsigned)smem, s, a);
  if (e == cudaErrorInvalidValue && known) {
    (void)cudaGetLastError();
    if ((e = raise()) == cudaSuccess)
      e = imx::launch_dependent(kern, grid, (unsigned)threads, (unsigned)smem, s, a);
  }
  return e;
}

int odd_up(int v) { return v | 1; }

// The halo of an 8 x 16 tile read by a 3x3 stencil of stride `step` (1, 2).
void stencil_halo(conv::Halo& h, int step) {
  h.step = step;
  h.org = -1;
  h.hh = step * (conv::kTY - 1) + 3;
  h.hw = step * (conv::kTX - 1) + 3;
  h.half = step == 2 ? (h.hw + 1) / 2 : 0;
  h.rp = step == 2 ? 2 * h.half : h.hw;
  h.plane = odd_up(h.hh * h.rp);
}

// Start pixels of the nine taps in that halo.
void stencil_taps(conv::Taps& t, const conv::Halo& h, bool flip) {
  t.n[0] = 9;
  for (int k = 0; k < 9; ++k) {
    const int ky = flip ? 2 - k / 3 : k / 3, kx = flip ? 2 - k % 3 : k % 3;
    t.tap[0][k] = (uint8_t)k;
    t.off[0][k] = (uint16_t)(ky * h.rp + (h.half ? (kx & 1) * h.half + (kx >> 1) : kx));
  }
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }
bool aligned32(const void* p) { return ((uintptr_t)p & 31u) == 0; }

// Shared memory of a kernel's halo table.
uint32_t table_bytes(const conv::Halo& h) { return (uint32_t)((h.hh * h.rp * 8 + 127) / 128 * 128); }

cudaError_t run_rows(conv::RowsArgs& a, cudaStream_t s) {
  const int K = 9 * a.kch, N = a.n_out;
  if (!gemm_fits(N, K)) return cudaErrorInvalidValue;
  a.tab_bytes = table_bytes(a.h);
  const int b_bytes = ((N * K * 2) + 127) / 128 * 128 + (int)a.tab_bytes;
  const int stage = (a.h.ch >> 3) * a.h.plane * 16;
  // two blocks per SM of three stages when they fit, else one block with as
  // many stages as fit
  const int sms = sm_count();
  int per = 1, stages = std::min(conv::kMaxStages, (kSmemMax - 1024 - b_bytes) / stage);
  if (2 * (b_bytes + 3 * stage + 2048) <= kSmemMax) {
    per = 2;
    stages = 3;
  }
  if (stages < 1) return cudaErrorInvalidValue;
  a.stages = stages;
  a.vec = (a.ncols % 16 == 0 && a.ncols == N && aligned32(a.out_f) && aligned32(a.out_b)) ? 1 : 0;
  const int grid = std::max(1, std::min(a.ntiles, sms * per));
  return launch(conv::k_conv_rows, dim3((unsigned)grid), conv::kRowsThreads, b_bytes + stages * stage, a, s);
}

int tiles(int n, int t) { return (n + t - 1) / t; }

}  // namespace

extern "C" {

int imexlb_nn_conv_fwd(const imexlb_conv_desc* d, const void* x, const void* w, const float* bias,
                       int relu, void* y_bf16, float* y_f32, void* stream) {
  if (!valid(d) || !x || !w || (!y_bf16 && !y_f32) || !aligned16(x) || !aligned16(w)) return -1;
  conv::RowsArgs a{};
  a.h.src = (const bf16*)x;
  a.h.sh = d->hin;
  a.h.sw = d->win;
  a.h.ch = d->cin;
  a.h.up = d->upsample ? 1 : 0;
  a.h.gh = d->hin << a.h.up;
  a.h.gw = d->win << a.h.up;
  stencil_halo(a.h, d->stride);
  stencil_taps(a.t, a.h, false);
  a.w = (const bf16*)w;
  a.n_out = d->cout;
  a.kch = d->cin;
  a.images = d->n;
  a.oh = d->hout;
  a.ow = d->wout;
  a.classes = 1;
  a.tiles_x = tiles(d->wout, conv::kTX);
  a.tiles_y = tiles(d->hout, conv::kTY);
  a.ntiles = d->n * a.tiles_x * a.tiles_y;
  a.bias = bias;
  a.relu = relu;
  a.out_b = y_f32 ? nullptr : (bf16*)y_bf16;
  a.out_f = y_f32;
  a.ncols = d->cout_store ? d->cout_store : d->cout;
  return run_rows(a, (cudaStream_t)stream) == cudaSuccess ? 0 : -2;
}

int imexlb_nn_act_grad(const float* dy, const void* y, long long n, int c, int relu, void* dz,
                       float* dbias, void* stream) {
  if (!dy || !dz || n < 0 || c <= 0 || c > 64 || (relu && !y)) return -1;
  if (n == 0) return 0;
  if (c % 8 == 0 && n % 8 == 0 && (((uintptr_t)dy | (uintptr_t)y | (uintptr_t)dz) & 15u) == 0) {
    const int groups = c / 8, threads = kActThreads / groups * groups;
    const int64_t n8 = n / 8, most = 152 * 4;
    const int64_t grid = std::min(most, (n8 + threads - 1) / threads);
    const cudaError_t e =
        imx::launch_pdl(k_act_grad8, (unsigned)grid, (unsigned)threads, (cudaStream_t)stream, (const float4*)dy,
                        (const uint4*)y, n8, groups, relu, (uint4*)dz, dbias);
    return e == cudaSuccess ? 0 : -2;
  }
  int64_t blocks = (n + 255) / 256;
  if (blocks > 152 * 8) blocks = 152 * 8;
  k_act_grad<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(dy, (const bf16*)y, n, c, relu,
                                                                  (bf16*)dz, dbias);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int imexlb_nn_conv_bwd_data(const imexlb_conv_desc* d, const void* dz, const void* w, void* wt_scratch,
                            float* dgrid, float* dx, void* stream) {
  if (!valid(d) || !dz || !w || !wt_scratch || !dgrid || !aligned16(dz)) return -1;
  if (d->cin > 64) return -2;
  cudaStream_t s = (cudaStream_t)stream;
  // the kernel copies w 16 bytes at a time
  if (!aligned16(w)) {
    if ((uintptr_t)w & 1u || !aligned16(wt_scratch)) return -1;
    const int nw = d->cout * 9 * d->cin;
    k_copy_w<<<(nw + 255) / 256, 256, 0, s>>>((const bf16*)w, nw, (bf16*)wt_scratch);
    if (cudaGetLastError() != cudaSuccess) return -2;
    w = wt_scratch;
  }
  const int hg = d->upsample ? 2 * d->hin : d->hin, wg = d->upsample ? 2 * d->win : d->win;
  conv::RowsArgs a{};
  a.h.src = (const bf16*)dz;
  a.h.sh = a.h.gh = d->hout;
  a.h.sw = a.h.gw = d->wout;
  a.h.ch = d->cout;
  if (d->stride == 1) {
    stencil_halo(a.h, 1);
    stencil_taps(a.t, a.h, true);
    a.classes = 1;
    a.tiles_x = tiles(wg, conv::kTX);
    a.tiles_y = tiles(hg, conv::kTY);
  } else {
    // the grid pixels (2j + py, 2i + px) of one parity class read output
    // pixels j, j + 1 and i, i + 1: tap ky of an even row is 1 (row j), of an
    // odd row 0 (j + 1) and 2 (j)
    a.h.step = 1;
    a.h.org = 0;
    a.h.hh = conv::kTY + 1;
    a.h.hw = a.h.rp = conv::kTX + 1;
    a.h.plane = odd_up(a.h.hh * a.h.rp);
    a.classes = 4;
    a.tiles_x = tiles((wg + 1) / 2, conv::kTX);
    a.tiles_y = tiles((hg + 1) / 2, conv::kTY);
    for (int c = 0; c < 4; ++c)
      for (int k = 0; k < 9; ++k) {
        const int ky = k / 3, kx = k % 3, py = c >> 1, px = c & 1;
        if ((py + 1 - ky) & 1 || (px + 1 - kx) & 1) continue;
        const int n = a.t.n[c]++;
        a.t.tap[c][n] = (uint8_t)k;
        a.t.off[c][n] = (uint16_t)((py + 1 - ky) / 2 * a.h.rp + (px + 1 - kx) / 2);
      }
  }
  a.ntiles = d->n * a.tiles_x * a.tiles_y * a.classes;
  a.w = (const bf16*)w;
  a.trans = 1;
  a.wk = d->cin;
  a.n_out = d->cin;
  a.kch = d->cout;
  a.images = d->n;
  a.oh = hg;
  a.ow = wg;
  a.out_f = dgrid;
  a.ncols = d->cin;
  // the 2x2 sums of an upsampled layer come with the tile (16-byte stores),
  // except between parity classes
  const bool sums = d->upsample && dx && d->stride == 1 && ((uintptr_t)dx & 15u) == 0;
  a.dx = sums ? dx : nullptr;
  if (run_rows(a, s) != cudaSuccess) return -2;
  if (d->upsample && !dx) return -1;
  const int64_t n = (int64_t)d->n * d->hin * d->win * d->cin;
  if (d->upsample && n == 0) return -2;  // no sums to form
  if (d->upsample && !sums) {
    k_down_sum<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(dgrid, d->n, d->hin, d->win, d->cin, dx);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int imexlb_nn_conv_bwd_weight(const imexlb_conv_desc* d, const void* x, const void* dz, float* dw,
                              void* stream) {
  if (!valid(d) || !x || !dz || !dw || !aligned16(x) || !aligned16(dz)) return -1;
  conv::WgradArgs a{};
  a.h.src = (const bf16*)x;
  a.h.sh = d->hin;
  a.h.sw = d->win;
  a.h.ch = d->cin;
  a.h.up = d->upsample ? 1 : 0;
  a.h.gh = d->hin << a.h.up;
  a.h.gw = d->win << a.h.up;
  stencil_halo(a.h, d->stride);
  stencil_taps(a.t, a.h, false);
  a.dz = (const bf16*)dz;
  a.images = d->n;
  a.oh = d->hout;
  a.ow = d->wout;
  a.cin = d->cin;
  a.cout = d->cout;
  // rows (64): the side with more channels, else dz's (its sums go out four
  // at a time); one accumulator of n_cols columns per tap, 512 in all
  a.m_is_ci = d->cin > d->cout ? 1 : 0;
  a.vec = ((uintptr_t)dw & 15u) == 0 ? 1 : 0;
  const int n_cols = a.m_is_ci ? d->cout : std::min(d->cin, 64);
  const int zblocks = tiles(d->cin, 64);
  const int yblocks = tiles(9, std::min(9, 512 / n_cols));
  a.taps_per = tiles(9, yblocks);
  for (a.tmem_cols = 32; (int)a.tmem_cols < a.taps_per * n_cols;) a.tmem_cols *= 2;
  a.tiles_x = tiles(d->wout, conv::kTX);
  a.tiles_y = tiles(d->hout, conv::kTY);
  a.ntiles = d->n * a.tiles_x * a.tiles_y;
  if (a.ntiles == 0) return -2;  // every block of the kernel has a tile
  a.dz_plane = odd_up(conv::kTM);
  a.x_bytes = (uint32_t)((std::min(d->cin, 64) >> 3) * a.h.plane * 16);
  const int z_bytes = (d->cout >> 3) * a.dz_plane * 16;
  a.stage_bytes = (uint32_t)((a.x_bytes + z_bytes + 127) / 128 * 128);
  // the 64 rows run past the staged planes of the last stage
  const int over = a.m_is_ci ? (8 - (std::min(d->cin, 64) >> 3)) * a.h.plane * 16 - z_bytes
                             : (8 - (d->cout >> 3)) * a.dz_plane * 16;
  const int pad = std::max(0, over);
  a.tab_bytes = table_bytes(a.h);
  a.stages = std::min(conv::kMaxStages, (kSmemMax - 1024 - pad - (int)a.tab_bytes) / (int)a.stage_bytes);
  if (a.stages < 1) return -2;
  a.dw = dw;
  const int sms = sm_count();
  // A block's accumulators take kWgAccTiles tiles at most, so past one tile
  // per SM the tiles are dealt to as many whole waves of blocks as that needs.
  const int wave = std::max(1, sms / (yblocks * zblocks));
  const int gx = std::min(a.ntiles, wave * tiles(a.ntiles, wave * conv::kWgAccTiles));
  const cudaError_t e = launch(conv::k_conv_wgrad, dim3((unsigned)gx, (unsigned)yblocks, (unsigned)zblocks),
                               conv::kWgThreads,
                               (int)a.tab_bytes + (int)a.stage_bytes * a.stages + pad, a, (cudaStream_t)stream);
  return e == cudaSuccess ? 0 : -2;
}

int imexlb_nn_mse(const float* y, const float* target, const float* weight, long long npix, int c,
                  int used, float* dy, float* loss, void* stream) {
  if (!y || !target || !dy || !loss || npix < 0 || c <= 0 || used <= 0 || used > c) return -1;
  if (npix == 0) return 0;
  if (c % 4 == 0 && (((uintptr_t)y | (uintptr_t)dy) & 15u) == 0) {
    const int64_t n4 = npix * c / 4, most = 152 * 8;
    const cudaError_t e = imx::launch_pdl(k_mse4, (unsigned)std::min(most, (n4 + 255) / 256), 256u,
                                          (cudaStream_t)stream, (const float4*)y, target, weight, n4, c / 4, used,
                                          1.0f / (float)(npix * used), (float4*)dy, loss);
    return e == cudaSuccess ? 0 : -2;
  }
  int64_t blocks = (npix * c + 255) / 256;
  if (blocks > 152 * 8) blocks = 152 * 8;
  k_mse<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(y, target, weight, npix, c, used,
                                                            1.0f / (float)(npix * used), dy, loss);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int imexlb_nn_adam(float* p, const float* g, float* m, float* v, void* p_bf16, long long n, float lr,
                   float beta1, float beta2, float eps, int t, float weight_decay, void* stream) {
  if (!p || !g || !m || !v || n < 0 || t < 1) return -1;
  if (n == 0) return 0;
  const float bc1 = 1.0f - powf(beta1, (float)t), bc2 = 1.0f - powf(beta2, (float)t);
  k_adam<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      p, g, m, v, (bf16*)p_bf16, n, lr, beta1, beta2, eps, bc1, bc2, weight_decay);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int imexlb_nn_status(int* status) {
  if (!status) return -1;
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, conv::g_conv_status, sizeof(int)) != cudaSuccess) return -2;
  *status = v;
  if (v) {
    const int zero = 0;
    if (cudaMemcpyToSymbol(conv::g_conv_status, &zero, sizeof(int)) != cudaSuccess) return -2;
  }
  return 0;
}

}  // extern "C"
