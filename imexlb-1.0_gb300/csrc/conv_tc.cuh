// Implicit-GEMM kernels of the 3x3 convolutions (nn.cu) on the tcgen05 tensor
// cores.
//
// A tile is 8 x 16 output pixels (x fastest), the 128 rows of one MMA. Its
// operand is staged once, as the halo of pixels the nine taps read, instead
// of as an im2col matrix: shared memory holds [8-channel chunk][halo pixel][16
// bytes], so eight consecutive x pixels of a halo row are one core matrix
// (8 x 16 bytes) wherever they start, the next row of the tile is one halo
// row further (the descriptor's stride offset) and the next eight channels
// one plane further (its leading offset). A tap is then only another start
// address in the descriptor, at 16-byte granularity. At stride 2 the halo's
// even and odd columns are kept apart, so that the eight pixels of a core
// matrix stay adjacent.
//
// Both kernels are warp-specialised: loader warps copy halos (cp.async,
// zero-filled outside the grid) several tiles ahead, one warp issues the
// MMAs, and (forward / data gradient) four warps empty one accumulator while
// the next one fills. Every wait is bounded (kConvWaitNs of the global
// timer); a warp that gives up raises the block's abort flag and the status
// word, the others stop at their next wait, and the tensor memory is freed
// on every path.
//
// What bounds it: with an im2col gather (nine copies of every pixel through
// registers into shared memory, one tile at a time) the 16 x 64x128 -> 128x256
// upsampling layer of 48 -> 48 channels (21.7 GFLOP, 63 MB) took 424 us
// forward, 360 + 37 us for the data gradient and its 2x2 sums, 351 us for the
// weight gradient. Staging each pixel once, tiles ahead, took 56, 55 and
// 118 us; with the MMAs issued warp-wide (umma.cuh) 86 us for the first two
// together and 71 us. A 128 x 48 x 16 MMA reads 5.5 KB of shared memory at 128 bytes a
// cycle, 44 cycles, so 27 of them per tile (16 us for the layer) are the floor of
// the forward pass, and 72 MMAs of 64 x 48 x 16 (29 cycles, 27 us) that of the
// weight gradient.
#pragma once

#include <cstdint>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "umma.cuh"

namespace imx {
namespace conv {

typedef __nv_bfloat16 bf16;

constexpr int kTX = 8, kTY = 16;  // output pixels of a tile
constexpr int kTM = kTX * kTY;    // GEMM rows: the MMA's M
constexpr unsigned long long kConvWaitNs = 2000000000ull;

// Where the nine taps of a tile read: start pixels inside the staged halo.
// The data gradient at stride 2 runs each parity class of grid pixels as
// tiles of its own, with the taps that reach it (1, 2, 2 or 4 of the nine).
struct Taps {
  uint8_t n[4];
  uint8_t tap[4][9];
  uint16_t off[4][9];
};

// The source a kernel gathers from and the halo it stages.
struct Halo {
  const bf16* src;   // [n][sh][sw][ch]
  int sh, sw, ch;
  int up;            // 1: the grid is the source upsampled x2 (nearest)
  int gh, gw;        // grid size
  int step, org;     // grid pixel of halo (0, 0): step * (tile pixel) + org
  int hh, hw;        // halo size
  int rp;            // halo pixels per stored row
  int half;          // stride 2: first stored pixel of the odd columns; 0: stride 1
  int plane;         // pixels per chunk plane (odd: consecutive chunks shift banks)
};

struct RowsArgs {
  Halo h;
  Taps t;
  const bf16* w;      // weights [cout][9 cin]
  int n_out;          // GEMM columns (multiple of 16, <= 64)
  int wk;             // channels per tap of the weight rows
  int trans;          // 0: B[n][k] = w[n][k]; 1: B[n = ci][k = (tap, co)] = w[co][tap, ci]
  int kch;            // K channels per tap
  int images, oh, ow; // images, output grid
  int classes;        // 1, or 4 parity classes (output pixel 2 * tile pixel + class)
  int tiles_x, tiles_y;
  int ntiles;         // per class x classes
  int stages;
  const float* bias;
  int relu;
  bf16* out_b;
  float* out_f;
  int ncols;          // columns stored per output pixel
  int vec;            // 32-byte stores
  float* dx;          // data gradient of an upsampled layer: 2x2 sums of the output
};

struct WgradArgs {
  Halo h;             // x
  Taps t;
  const bf16* dz;     // [n][oh][ow][cout]
  int images, oh, ow, cin, cout;
  int m_is_ci;        // GEMM rows: input channels (else output channels)
                      // (64 per z block, which stages only those channels of x)
  int n_cols;         // columns per tap
  int taps_per;       // taps per y block
  int tiles_x, tiles_y, ntiles;
  int stages;
  uint32_t stage_bytes, x_bytes;
  int dz_plane;
  uint32_t tmem_cols;
  float* dw;
};

#ifdef __CUDACC__

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(umma::smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::smem_addr(bar)) : "memory");
}

// Bounded wait for phase `parity`; false when it gave up or (abort_v given)
// the block aborts.
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_v) {
  unsigned long long t0 = 0;
  for (uint32_t n = 0;; ++n) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(done)
        : "r"(umma::smem_addr(bar)), "r"(parity), "r"(100000u)
        : "memory");
    if (done) return true;
    if (abort_v && *abort_v) return false;
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (n == 0) t0 = t;
    else if (t - t0 > kConvWaitNs) return false;
  }
}

__device__ __forceinline__ void give_up(volatile int* abort_v, int* status) {
  *abort_v = 1;
  atomicExch(status, 1);
}

// One loader thread's share of a halo: chunk c of every `stride`-th pixel
// from p0 (the copies of the block's `lanes` = chunks x stride loader lanes).
struct HaloLane {
  int c, ly0, lx0, dly, dlx;
  bool on;
  __device__ __forceinline__ static HaloLane make(const Halo& h, int lane, int lanes, int channels) {
    HaloLane l;
    const int chunks = channels >> 3, stride = lanes / chunks;
    const int p0 = lane / chunks;
    l.c = lane - p0 * chunks;
    l.on = p0 < stride;
    l.ly0 = p0 / h.hw;
    l.lx0 = p0 - l.ly0 * h.hw;
    l.dly = stride / h.hw;
    l.dlx = stride - l.dly * h.hw;
    return l;
  }
  // copy the halo of the tile at tile pixel (py, px) of image img to `dst`,
  // channels from c0
  __device__ __forceinline__ void load(const Halo& h, uint32_t dst, int img, int py, int px, int c0) const {
    if (!on) return;
    const int y0 = h.step * py + h.org, x0 = h.step * px + h.org;
    const bf16* base = h.src + (int64_t)img * h.sh * h.sw * h.ch + c0 + c * 8;
    const uint32_t d0 = dst + (uint32_t)(c * h.plane) * 16u;
    int ly = ly0, lx = lx0;
    while (ly < h.hh) {
      const int gy = y0 + ly, gx = x0 + lx;
      const bool in = (unsigned)gy < (unsigned)h.gh && (unsigned)gx < (unsigned)h.gw;
      const int64_t off = in ? ((int64_t)(gy >> h.up) * h.sw + (gx >> h.up)) * h.ch : 0;
      const int slot = ly * h.rp + (h.half ? (lx & 1) * h.half + (lx >> 1) : lx);
      cp16(d0 + (uint32_t)slot * 16u, base + off, in);
      ly += dly;
      lx += dlx;
      if (lx >= h.hw) {
        lx -= h.hw;
        ++ly;
      }
    }
  }
};

struct TilePos {
  int cls, img, py, px;
};
__device__ __forceinline__ TilePos tile_pos(int t, int classes, int tiles_x, int tiles_y) {
  TilePos p;
  p.cls = classes == 4 ? t & 3 : 0;
  if (classes == 4) t >>= 2;
  const int row = t / tiles_x;
  p.px = (t - row * tiles_x) * kTX;
  p.img = row / tiles_y;
  p.py = (row - p.img * tiles_y) * kTY;
  return p;
}

// Descriptor with explicit offsets (bytes): `lead` and `stride` as in umma.cuh.
__device__ __forceinline__ uint64_t desc(uint32_t addr, uint32_t lead, uint32_t stride) {
  return umma::smem_desc(addr, lead, stride);
}

constexpr int kLoadWarps = 4;  // k_conv_rows: warps 4 .. 7 load, warps 0 .. 3 empty, warp 8 issues
constexpr int kRowsThreads = 32 * (4 + kLoadWarps + 1);
constexpr int kMaxStages = 4;

__device__ __forceinline__ void st32(void* p, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// Issue the TMEM load of 16 columns without waiting for it.
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Forward convolution and data gradient: C[pixels x n_out] = taps(src) * B^T.
// The K slices run in tap order and, within a tap, channel order, 16 at a
// time, each row's sum the same sequence of MMAs whatever the tile shape.
__global__ void __launch_bounds__(kRowsThreads, 2) k_conv_rows(const __grid_constant__ RowsArgs a,
                                                            int* status) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], tfull[2], tempty[2];
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  __shared__ float sbias[64];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (uniform for the compiler too)
  volatile int* abort_v = &abort_flag;
  const int K = 9 * a.kch, N = a.n_out;
  const uint32_t b_bytes = ((uint32_t)(N * K * 2) + 127u) & ~127u;
  const uint32_t stage_bytes = (uint32_t)(a.h.ch >> 3) * (uint32_t)a.h.plane * 16u;
  bf16* sB = (bf16*)smem;
  // B: K-major core matrices of w's rows, or (trans) N-major: [n / 8][k][8 n]
  if (!a.trans) {
    const int kc_n = K >> 3;
    for (int i = tid; i < N * kc_n; i += kRowsThreads) {
      const int n = i / kc_n, c = i - n * kc_n;
      *(uint4*)(sB + umma::cm_off(n, c * 8, N)) = *(const uint4*)(a.w + (int64_t)n * K + c * 8);
    }
  } else {
    const int nc = N >> 3;  // a row of w is [tap][ci]; k = tap * kch + co
    for (int i = tid; i < K * nc; i += kRowsThreads) {
      const int k = i / nc, c = i - k * nc, tap = k / a.kch, co = k - tap * a.kch;
      *(uint4*)(sB + ((int64_t)c * K + k) * 8) =
          *(const uint4*)(a.w + (int64_t)co * 9 * a.wk + tap * a.wk + c * 8);
    }
  }
  if (tid < 64) sbias[tid] = a.bias && tid < N ? a.bias[tid] : 0.0f;
  if (warp == 0) umma::tmem_alloc(&tmem_base, 128);
  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < a.stages; ++s) {
      bar_init(&full[s], 32 * kLoadWarps);
      bar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      bar_init(&tfull[s], 1);
      bar_init(&tempty[s], 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  umma::fence_smem_async();  // B, for the MMAs
  umma::fence_before();
  __syncthreads();
  umma::fence_after();
  const uint32_t tmem = tmem_base;
  const uint32_t baddr = umma::smem_addr(smem), saddr = baddr + b_bytes;
  const int G = (int)gridDim.x;

  if (warp >= 4 && warp < 4 + kLoadWarps) {
    const HaloLane hl = HaloLane::make(a.h, tid - 128, 32 * kLoadWarps, a.h.ch);
    const int lag = a.stages > 2 ? a.stages - 2 : 0;
    int s = 0, sf = 0, issued = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = (int)blockIdx.x; t < a.ntiles; t += G) {
      if (issued >= a.stages) ok = bar_wait(&empty[s], phase ^ 1u, abort_v);
      if (!ok) break;
      const TilePos p = tile_pos(t, a.classes, a.tiles_x, a.tiles_y);
      hl.load(a.h, saddr + (uint32_t)s * stage_bytes, p.img, p.py, p.px, 0);
      cp_commit();
      if (++s == a.stages) {
        s = 0;
        phase ^= 1u;
      }
      ++issued;
      if (issued > lag) {
        // the tile issued `lag` tiles ago is complete
        if (lag == 0) cp_wait<0>();
        else if (lag == 1) cp_wait<1>();
        else cp_wait<2>();
        umma::fence_smem_async();
        bar_arrive(&full[sf]);
        if (++sf == a.stages) sf = 0;
      }
    }
    if (!ok) give_up(abort_v, status);
    cp_wait<0>();
    umma::fence_smem_async();
    for (int left = issued < lag ? issued : lag; left > 0; --left) {
      bar_arrive(&full[sf]);
      if (++sf == a.stages) sf = 0;
    }
  } else if (warp == 4 + kLoadWarps) {
    const uint32_t idesc = umma::idesc_bf16_f32(kTM, N, false, a.trans != 0);
    const uint32_t lead = (uint32_t)a.h.plane * 16u;
    const uint32_t rows = (uint32_t)(a.h.step * a.h.rp) * 16u;
    const uint32_t b_lead = a.trans ? 128u : (uint32_t)(N >> 3) * 128u;
    const uint32_t b_str = a.trans ? (uint32_t)K * 16u : 128u;
    const uint32_t b_step = a.trans ? 256u : 2u * b_lead;  // bytes per K slice
    const int slices = a.kch >> 4;
    int s = 0, k = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = (int)blockIdx.x; t < a.ntiles; t += G, ++k) {
      const int cls = a.classes == 4 ? t & 3 : 0;
      const int acc = k & 1;
      ok = bar_wait(&full[s], phase, abort_v);
      if (ok && k >= 2) ok = bar_wait(&tempty[acc], (uint32_t)((k >> 1) - 1) & 1u, abort_v);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      umma::fence_after();
      const uint32_t d = tmem + (uint32_t)acc * 64u;
      const uint32_t abase = saddr + (uint32_t)s * stage_bytes;
      bool accum = false;
      for (int j = 0; j < a.t.n[cls]; ++j) {
        const uint32_t ad = abase + (uint32_t)a.t.off[cls][j] * 16u;
        const uint32_t bd = baddr + (uint32_t)(a.t.tap[cls][j] * slices) * b_step;
        for (int c = 0; c < slices; ++c) {
          umma::mma_bf16(d, desc(ad + (uint32_t)c * 2u * lead, lead, rows),
                         desc(bd + (uint32_t)c * b_step, b_lead, b_str), idesc, accum);
          accum = true;
        }
      }
      umma::mma_commit(&empty[s]);
      umma::mma_commit(&tfull[acc]);
      if (++s == a.stages) {
        s = 0;
        phase ^= 1u;
      }
    }
    if (!ok) give_up(abort_v, status);
    // the MMAs in flight end before the block gives its memory back
    if (k >= 1) bar_wait(&tfull[(k - 1) & 1], (uint32_t)((k - 1) >> 1) & 1u, nullptr);
  } else {
    int k = 0;
    for (int t = (int)blockIdx.x; t < a.ntiles; t += G, ++k) {
      const int acc = k & 1;
      const bool ok = __all_sync(0xffffffffu, bar_wait(&tfull[acc], (uint32_t)(k >> 1) & 1u, abort_v));
      if (!ok) {
        if (lane == 0) give_up(abort_v, status);
        break;
      }
      umma::fence_after();
      const TilePos p = tile_pos(t, a.classes, a.tiles_x, a.tiles_y);
      const int r = warp * 32 + lane;
      int oy = p.py + (r >> 3), ox = p.px + (r & 7);
      if (a.classes == 4) {
        oy = 2 * oy + (p.cls >> 1);
        ox = 2 * ox + (p.cls & 1);
      }
      const bool in = oy < a.oh && ox < a.ow;
      const int64_t pix = ((int64_t)p.img * a.oh + oy) * a.ow + ox;
      const uint32_t taddr = tmem + (uint32_t)acc * 64u + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
      for (int c0 = 0; c0 < N; c0 += 32) {
        uint32_t v[2][16];
        tmem_ld16_async(taddr + (uint32_t)c0, v[0]);
        if (c0 + 16 < N) tmem_ld16_async(taddr + (uint32_t)(c0 + 16), v[1]);
        tmem_ld_wait();
        if (c0 + 32 >= N) {
          umma::fence_before();
          __syncwarp();
          if (lane == 0) bar_arrive(&tempty[acc]);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int col = c0 + q * 16;
          if (col >= N) break;
          float x[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            x[j] = __uint_as_float(v[q][j]) + sbias[col + j];
            if (a.relu) x[j] = fmaxf(x[j], 0.0f);
          }
          if (in) {
            const int64_t o = pix * a.ncols + col;
            if (a.vec) {
              if (a.out_f) {
#pragma unroll
                for (int hb = 0; hb < 2; ++hb) {
                  uint32_t w[8];
#pragma unroll
                  for (int j = 0; j < 8; ++j) w[j] = __float_as_uint(x[hb * 8 + j]);
                  st32(a.out_f + o + hb * 8, w);
                }
              } else {
                uint32_t w[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const __nv_bfloat162 b2 = __floats2bfloat162_rn(x[2 * j], x[2 * j + 1]);
                  w[j] = *(const uint32_t*)&b2;
                }
                st32(a.out_b + o, w);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                if (col + j >= a.ncols) break;
                if (a.out_f) a.out_f[o + j] = x[j];
                else a.out_b[o + j] = __float2bfloat16(x[j]);
              }
            }
          }
          if (a.dx) {
            // each source pixel's four children: lanes +1 (x) and +8 (y) of the
            // warp's 4 x 8 pixels
            const bool keep = in && !(oy & 1) && !(ox & 1);
            float* o = a.dx + (((int64_t)p.img * (a.oh >> 1) + (oy >> 1)) * (a.ow >> 1) + (ox >> 1)) * N + col;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float b = __shfl_down_sync(0xffffffffu, x[j], 1);
              const float c = __shfl_down_sync(0xffffffffu, x[j], 8);
              const float d = __shfl_down_sync(0xffffffffu, x[j], 9);
              x[j] = (((0.0f + x[j]) + b) + c) + d;
            }
            if (keep) {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                *(float4*)(o + 4 * j) = make_float4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
            }
          }
        }
      }
    }
  }
  umma::fence_before();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 128);
}

// Weight gradient: dW of the taps [taps_per y, ...) as 64 x n_cols products
// over all pixels, D[m][tap, n] += sum_p M(p, m) N(p, n), where one side is
// dz and the other x at the tap's pixel. Both operands are read M-/N-major
// straight from their staged tiles (channels contiguous, eight pixels of a
// tile row per core matrix, 16 pixels = two tile rows per MMA); one
// accumulator per tap stays in tensor memory over all the block's tiles and
// is added to dw at the end. Rows past the channel count run on whatever
// follows the staged planes and are dropped.
constexpr int kWgLoadWarps = 8;
constexpr int kWgThreads = 32 * (kWgLoadWarps + 1);

__global__ void __launch_bounds__(kWgThreads) k_conv_wgrad(const __grid_constant__ WgradArgs a,
                                                           int* status) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], done;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (uniform for the compiler too)
  volatile int* abort_v = &abort_flag;
  if (warp == 0) umma::tmem_alloc(&tmem_base, a.tmem_cols);
  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < a.stages; ++s) {
      bar_init(&full[s], 32 * kWgLoadWarps);
      bar_init(&empty[s], 1);
    }
    bar_init(&done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  umma::fence_before();
  __syncthreads();
  umma::fence_after();
  const uint32_t tmem = tmem_base;
  const uint32_t saddr = umma::smem_addr(smem);
  const int G = (int)gridDim.x;
  const int tap0 = (int)blockIdx.y * a.taps_per, tap1 = tap0 + a.taps_per < 9 ? tap0 + a.taps_per : 9;
  const int m0 = (int)blockIdx.z * 64;

  if (warp < kWgLoadWarps) {
    const HaloLane hl = HaloLane::make(a.h, tid, 32 * kWgLoadWarps, a.m_is_ci && a.cin - m0 > 64 ? 64 : a.cin - m0);
    const int zc = a.cout >> 3, zstride = 32 * kWgLoadWarps / zc;
    const int zp0 = tid / zc, zch = tid - zp0 * zc;
    const int lag = a.stages > 2 ? a.stages - 2 : 0;
    int s = 0, sf = 0, issued = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = (int)blockIdx.x; t < a.ntiles; t += G) {
      if (issued >= a.stages) ok = bar_wait(&empty[s], phase ^ 1u, abort_v);
      if (!ok) break;
      const TilePos p = tile_pos(t, 1, a.tiles_x, a.tiles_y);
      const uint32_t st = saddr + (uint32_t)s * a.stage_bytes;
      hl.load(a.h, st, p.img, p.py, p.px, m0);
      if (zp0 < zstride) {
        const uint32_t d0 = st + a.x_bytes + (uint32_t)(zch * a.dz_plane) * 16u;
        for (int q = zp0; q < kTM; q += zstride) {
          const int oy = p.py + (q >> 3), ox = p.px + (q & 7);
          const bool in = oy < a.oh && ox < a.ow;
          const int64_t off = in ? (((int64_t)p.img * a.oh + oy) * a.ow + ox) * a.cout : 0;
          cp16(d0 + (uint32_t)q * 16u, a.dz + off + zch * 8, in);
        }
      }
      cp_commit();
      if (++s == a.stages) {
        s = 0;
        phase ^= 1u;
      }
      ++issued;
      if (issued > lag) {
        if (lag == 0) cp_wait<0>();
        else if (lag == 1) cp_wait<1>();
        else cp_wait<2>();
        umma::fence_smem_async();
        bar_arrive(&full[sf]);
        if (++sf == a.stages) sf = 0;
      }
    }
    if (!ok) give_up(abort_v, status);
    cp_wait<0>();
    umma::fence_smem_async();
    for (int left = issued < lag ? issued : lag; left > 0; --left) {
      bar_arrive(&full[sf]);
      if (++sf == a.stages) sf = 0;
    }
  } else {
    // both operands with their channels contiguous
    const uint32_t idesc = umma::idesc_bf16_f32(64, a.n_cols, true, true);
    const uint32_t x_chunk = (uint32_t)a.h.plane * 16u, x_row = (uint32_t)(a.h.step * a.h.rp) * 16u;
    const uint32_t z_chunk = (uint32_t)a.dz_plane * 16u, z_row = 128u;
    int s = 0;
    uint32_t phase = 0;
    bool ok = true, accum = false;
    for (int t = (int)blockIdx.x; t < a.ntiles; t += G) {
      ok = __all_sync(0xffffffffu, bar_wait(&full[s], phase, abort_v));
      if (!ok) break;
      umma::fence_after();
      const uint32_t xb = saddr + (uint32_t)s * a.stage_bytes;
      const uint32_t zb = saddr + (uint32_t)s * a.stage_bytes + a.x_bytes;
      for (int tap = tap0; tap < tap1; ++tap) {
        const uint32_t d = tmem + (uint32_t)((tap - tap0) * a.n_cols);
        const uint32_t xt = xb + (uint32_t)a.t.off[0][tap] * 16u;
#pragma unroll
        for (int k = 0; k < kTM / 16; ++k) {
          const uint64_t xd = desc(xt + (uint32_t)(2 * k) * x_row, x_row, x_chunk);
          const uint64_t zd = desc(zb + (uint32_t)(2 * k) * z_row, z_row, z_chunk);
          umma::mma_bf16(d, a.m_is_ci ? xd : zd, a.m_is_ci ? zd : xd, idesc, accum || k > 0);
        }
      }
      accum = true;
      umma::mma_commit(&empty[s]);
      if (++s == a.stages) {
        s = 0;
        phase ^= 1u;
      }
    }
    if (!ok) give_up(abort_v, status);
    umma::mma_commit(&done);
    // the MMAs in flight end before the block gives its memory back
    bar_wait(&done, 0u, nullptr);
  }
  const bool ok = __all_sync(0xffffffffu, bar_wait(&done, 0u, abort_v));
  if (!ok && lane == 0) give_up(abort_v, status);
  umma::fence_after();
  if (ok && warp < 4 && (int)blockIdx.x < a.ntiles) {
    // row 16 w + l of the 64 sits in lane 32 w + l (l < 16)
    const int m = m0 + warp * 16 + lane;
    const int mn = a.m_is_ci ? a.cin : a.cout;
    const int64_t ld = 9 * (int64_t)a.cin;
    for (int tap = tap0; tap < tap1; ++tap)
      for (int c0 = 0; c0 < a.n_cols; c0 += 16) {
        float v[16];
        umma::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((tap - tap0) * a.n_cols + c0), v);
        if (lane < 16 && m < mn) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            float* o = a.m_is_ci ? a.dw + (int64_t)(c0 + j) * ld + (int64_t)tap * a.cin + m
                                 : a.dw + (int64_t)m * ld + (int64_t)tap * a.cin + c0 + j;
            atomicAdd(o, v[j]);
          }
        }
      }
  }
  umma::fence_before();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, a.tmem_cols);
}

#endif  // __CUDACC__

}  // namespace conv
}  // namespace imx
