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
// weight gradient; here 30, 41 and 48 us. A 128 x 48 x 16 MMA reads 5.5 KB of shared
// memory at 128 bytes a cycle, 44 cycles, so 27 of them per tile (16 us for the
// layer) are the floor of the forward pass, and 72 MMAs of 64 x 48 x 16 (29
// cycles, 27 us) that of the weight gradient; the copies and the epilogue
// share the shared-memory port with them. The data gradient also writes 126 MB.
#pragma once

#include <cstdint>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "pdl.cuh"
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
  uint32_t tab_bytes;
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
  int m_is_ci;        // GEMM rows: input channels (columns: output channels); else the reverse.
                      // A z block takes (and stages) 64 input channels.
  int vec;            // dw is 16-byte aligned
  int taps_per;       // taps per y block
  int tiles_x, tiles_y, ntiles;
  int stages;
  uint32_t tab_bytes, stage_bytes, x_bytes;
  int dz_plane;
  uint32_t tmem_cols;
  float* dw;
};

#ifdef __CUDACC__

// Status of the last kernels: 0, or 1 when a bounded wait gave up.
__device__ int g_conv_status = 0;

// (.ca: a .cg copy bypasses L1 and goes piece by piece unless both sides are
// contiguous over the warp, 24 cycles a warp's copy instead of at most 15)
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0)
               : "memory");
}
// The calling thread arrives on `bar` when its copies so far have landed. (A
// thread that waits for a tile's copies and fences them for the MMAs itself
// also waits for the tiles after it: 3300 cycles a tile, no overlap.)
__device__ __forceinline__ void cp_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(umma::smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void cp_drain() { asm volatile("cp.async.wait_all;" ::: "memory"); }

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

// What each slot of a plane holds: its source relative to the tile's first
// pixel, its halo row and column (-1: nothing). Made once per block; a loader
// thread then copies a chunk in a dozen instructions (the index arithmetic
// per chunk instead took longer than the tile's MMAs).
__device__ __forceinline__ void halo_table(const Halo& h, int2* tab, int tid, int threads) {
  for (int p = tid; p < h.hh * h.rp; p += threads) {
    const int ly = p / h.rp, q = p - ly * h.rp;
    const int lx = h.half ? (q < h.half ? 2 * q : 2 * (q - h.half) + 1) : q;
    // (an upsampled grid's tiles start at even pixels)
    const int dy = (ly + h.org) >> h.up, dx = (lx + h.org) >> h.up;
    tab[p] = make_int2((dy * h.sw + dx) * h.ch, lx < h.hw ? ly | lx << 8 : -1);
  }
}

// Copy the halo of the tile at tile pixel (py, px) of image img to `dst`,
// channels from c0: this thread takes chunk c of every stride-th slot from p0.
__device__ __forceinline__ void halo_load(const Halo& h, const int2* tab, uint32_t dst, int img, int py,
                                          int px, int c0, int c, int p0, int stride) {
  const int y0 = h.step * py + h.org, x0 = h.step * px + h.org;
  const bf16* src = h.src + c0 + c * 8;
  const bf16* base = src + (((int64_t)img * h.sh + ((h.step * py) >> h.up)) * h.sw + ((h.step * px) >> h.up)) * h.ch;
  const uint32_t d0 = dst + (uint32_t)(c * h.plane) * 16u;
  const int n = h.hh * h.rp;
  const unsigned gh = (unsigned)h.gh, gw = (unsigned)h.gw;
  constexpr int kU = 5;
  for (int p = p0; p < n; p += kU * stride) {
    int2 e[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) e[u] = p + u * stride < n ? tab[p + u * stride] : make_int2(0, -2);
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (e[u].y == -2) break;
      const bool in = e[u].y >= 0 && (unsigned)(y0 + (e[u].y & 255)) < gh && (unsigned)(x0 + (e[u].y >> 8)) < gw;
      cp16(d0 + (uint32_t)(p + u * stride) * 16u, in ? base + e[u].x : src, in);
    }
  }
}

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

constexpr int kLoadWarps = 4;  // k_conv_rows: warps 4 .. 7 load, warps 0 .. 3 empty, warp 8 issues
constexpr int kRowsThreads = 32 * (4 + kLoadWarps + 1);
constexpr int kMaxStages = 4;

__device__ __forceinline__ void st32(void* p, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

__device__ __forceinline__ void red4(float* p, float x, float y, float z, float w) {
  asm volatile("red.global.add.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
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
//
// It is launched to start while the stream's previous kernel ends (pdl.cuh):
// what comes before pdl_wait() reads no global memory, and pdl_trigger()
// comes after it, with the tensor memory allocated, so that a following kernel's
// blocks can't take what this one's still wait for. The weights come with
// cp.async beside the first halos, waited for by the MMA warp alone (read by
// all threads before the first halo, and with plain launches, the layer above took
// 78.5 us forward and data gradient together, now 71.6, and a 128x256 prediction of six
// layers 67 us, now 52).
__global__ void __launch_bounds__(kRowsThreads, 2) k_conv_rows(const __grid_constant__ RowsArgs a) {
  int* status = &g_conv_status;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], tfull[2], tempty[2], bfull;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  __shared__ float sbias[64];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (uniform for the compiler too)
  volatile int* abort_v = &abort_flag;
  const int K = 9 * a.kch, N = a.n_out;
  const uint32_t b_bytes = ((uint32_t)(N * K * 2) + 127u) & ~127u;
  const uint32_t stage_bytes = (uint32_t)(a.h.ch >> 3) * (uint32_t)a.h.plane * 16u;
  int2* tab = (int2*)smem;  // halo table, then B, then the stages
  bf16* sB = (bf16*)(smem + a.tab_bytes);
  halo_table(a.h, tab, tid, kRowsThreads);
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
    bar_init(&bfull, 128);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  umma::fence_before();
  __syncthreads();
  umma::fence_after();
  pdl_wait();
  pdl_trigger();
  const uint32_t tmem = tmem_base;
  const uint32_t baddr = umma::smem_addr(sB), saddr = baddr + b_bytes;
  const int G = (int)gridDim.x;

  if (warp >= 4 && warp < 4 + kLoadWarps) {
    const int chunks = a.h.ch >> 3, stride = 32 * kLoadWarps / chunks;
    const int hp0 = (tid - 128) / chunks, hc = tid - 128 - hp0 * chunks;
    int s = 0, issued = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = (int)blockIdx.x; t < a.ntiles; t += G) {
      if (issued >= a.stages) ok = bar_wait(&empty[s], phase ^ 1u, abort_v);
      if (!ok) break;
      const TilePos p = tile_pos(t, a.classes, a.tiles_x, a.tiles_y);
      if (hp0 < stride)
        halo_load(a.h, tab, saddr + (uint32_t)s * stage_bytes, p.img, p.py, p.px, 0, hc, hp0, stride);
      cp_arrive(&full[s]);
      if (++s == a.stages) {
        s = 0;
        phase ^= 1u;
      }
      ++issued;
    }
    if (!ok) give_up(abort_v, status);
    cp_drain();
  } else if (warp == 4 + kLoadWarps) {
    const uint32_t idesc = umma::idesc_bf16_f32(kTM, N, false, a.trans != 0);
    const uint32_t lead = (uint32_t)a.h.plane * 16u;
    const uint32_t rows = (uint32_t)(a.h.step * a.h.rp) * 16u;
    const uint32_t b_lead = a.trans ? 128u : (uint32_t)(N >> 3) * 128u;
    const uint32_t b_str = a.trans ? (uint32_t)K * 16u : 128u;
    const uint32_t b_step = (a.trans ? 256u : 2u * b_lead) >> 4;  // a K slice, in 16 bytes
    const int slices = a.kch >> 4;
    const uint64_t ad0 = umma::smem_desc(saddr, lead, rows), bd0 = umma::smem_desc(baddr, b_lead, b_str);
    const uint32_t a_hi = (uint32_t)(ad0 >> 32), b_hi = (uint32_t)(bd0 >> 32);
    uint32_t ta[9], tb[9];  // the taps' start addresses (a class's, at stride 2)
    int s = 0, k = 0, nt = 0;
    uint32_t phase = 0;
    bool ok = true;
    const bool b_ok = bar_wait(&bfull, 0u, abort_v);  // (its copies are fenced with the first halo's)
    for (int t = (int)blockIdx.x; t < a.ntiles; t += G, ++k) {
      if (k == 0 || a.classes == 4) {
        const int cls = a.classes == 4 ? t & 3 : 0;
        nt = a.t.n[cls];
#pragma unroll
        for (int j = 0; j < 9; ++j) {
          ta[j] = (uint32_t)ad0 + a.t.off[cls][j];
          tb[j] = (uint32_t)bd0 + (uint32_t)(a.t.tap[cls][j] * slices) * b_step;
        }
      }
      const int acc = k & 1;
      ok = b_ok && bar_wait(&full[s], phase, abort_v);
      if (ok && k >= 2) ok = bar_wait(&tempty[acc], (uint32_t)((k >> 1) - 1) & 1u, abort_v);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      umma::fence_smem_async();  // the copies, for the MMAs
      umma::fence_after();
      const uint32_t d = tmem + (uint32_t)acc * 64u;
      const uint32_t st = (uint32_t)s * (stage_bytes >> 4);
#pragma unroll
      for (int j = 0; j < 9; ++j) {
        if (j >= nt) break;
        uint32_t alo = ta[j] + st, blo = tb[j];
#pragma unroll 1
        for (int c = 0; c < slices; ++c) {
          umma::mma_bf16(d, alo, a_hi, blo, b_hi, idesc, j + c > 0);
          alo += lead >> 3;
          blo += b_step;
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
    // B: K-major core matrices of w's rows, or (trans) N-major: [n / 8][k][8 n]
    if (!a.trans) {
      const int kc_n = K >> 3;
      for (int i = tid; i < N * kc_n; i += 128) {
        const int n = i / kc_n, c = i - n * kc_n;
        cp16(umma::smem_addr(sB + umma::cm_off(n, c * 8, N)), a.w + (int64_t)n * K + c * 8, true);
      }
    } else {
      const int nc = N >> 3;  // a row of w is [tap][ci]; k = tap * kch + co
      for (int i = tid; i < K * nc; i += 128) {
        const int k = i / nc, c = i - k * nc, tap = k / a.kch, co = k - tap * a.kch;
        cp16(umma::smem_addr(sB + ((int64_t)c * K + k) * 8), a.w + (int64_t)co * 9 * a.wk + tap * a.wk + c * 8,
             true);
      }
    }
    cp_arrive(&bfull);
    // (a caller's bias has as many values as are stored)
    if (tid < 64) sbias[tid] = a.bias && tid < a.ncols ? a.bias[tid] : 0.0f;
    asm volatile("bar.sync 1, 128;" ::: "memory");  // sbias, among these warps
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
            // the four children of a source pixel are this lane, lane ^ 1 (x),
            // ^ 8 (y) and ^ 9: each of the four sums four of the 16 columns
            const int g = (lane & 1) | (lane >> 2 & 2);
            float part[4][4];  // [child][column of mine]
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              // lane g gives the columns of lane g ^ r and takes its own from it
              float got[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const int to = g ^ r;
                const float lo = to & 1 ? x[4 + j] : x[j], hi = to & 1 ? x[12 + j] : x[8 + j];
                const float v1 = to & 2 ? hi : lo;
                got[j] = r ? __shfl_xor_sync(0xffffffffu, v1, (r & 1) | (r & 2) << 2) : v1;
              }
              // (child g ^ r; placed by static index below)
#pragma unroll
              for (int j = 0; j < 4; ++j) part[r][j] = got[j];
            }
            float4 sum;
            float* sp = (float*)&sum;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              // child k came in round k ^ g
              const float p0 = g & 1 ? part[1][j] : part[0][j], p1 = g & 1 ? part[0][j] : part[1][j];
              const float p2 = g & 1 ? part[3][j] : part[2][j], p3 = g & 1 ? part[2][j] : part[3][j];
              const float k0 = g & 2 ? p2 : p0, k1 = g & 2 ? p3 : p1, k2 = g & 2 ? p0 : p2, k3 = g & 2 ? p1 : p3;
              sp[j] = (((0.0f + k0) + k1) + k2) + k3;
            }
            if (in)
              *(float4*)(a.dx + (((int64_t)p.img * (a.oh >> 1) + (oy >> 1)) * (a.ow >> 1) + (ox >> 1)) * N + col +
                         4 * g) = sum;
          }
        }
      }
    }
    cp_drain();
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
// is added to dw at the end (the host starts no block without a tile). Rows past
// the channel count run on whatever follows the staged planes and are dropped.
// Pixels of a tile past the image have dz = 0 and the x that their taps read: a
// NaN or infinity in x's last rows or columns reaches those taps too.
constexpr int kWgLoadWarps = 8;
// Tiles of one accumulator: 4096 output pixels. The tensor cores truncate a sum
// at every MMA, so its error grows with its length. Relative to a 64-bit sum, on
// positive values, without the bound and with it: 64 x 128x256 pixels of 48 -> 48
// channels 6.3e-5 and 1.0e-5 (154 and 176 us), 16 x 128x256 of 64 -> 64 channels
// 2.6e-5 and 1.0e-5 (83 and 90 us).
constexpr int kWgAccTiles = 32;
constexpr int kWgThreads = 32 * (kWgLoadWarps + 1);

__global__ void __launch_bounds__(kWgThreads) k_conv_wgrad(const __grid_constant__ WgradArgs a) {
  int* status = &g_conv_status;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], done;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (uniform for the compiler too)
  volatile int* abort_v = &abort_flag;
  int2* tab = (int2*)smem;  // halo table, then the stages
  halo_table(a.h, tab, tid, kWgThreads);
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
  pdl_wait();
  pdl_trigger();  // as in k_conv_rows
  const uint32_t tmem = tmem_base;
  const uint32_t saddr = umma::smem_addr(smem) + a.tab_bytes;
  const int G = (int)gridDim.x;
  const int tap0 = (int)blockIdx.y * a.taps_per, tap1 = tap0 + a.taps_per < 9 ? tap0 + a.taps_per : 9;
  const int m0 = (int)blockIdx.z * 64;  // first input channel
  const int n_cols = a.m_is_ci ? a.cout : a.cin - m0 > 64 ? 64 : a.cin - m0;

  if (warp < kWgLoadWarps) {
    const int chunks = (a.cin - m0 > 64 ? 64 : a.cin - m0) >> 3, stride = 32 * kWgLoadWarps / chunks;
    const int hp0 = tid / chunks, hc = tid - hp0 * chunks;
    const int zc = a.cout >> 3, zstride = 32 * kWgLoadWarps / zc;
    const int zp0 = tid / zc, zch = tid - zp0 * zc;
    int s = 0, issued = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = (int)blockIdx.x; t < a.ntiles; t += G) {
      if (issued >= a.stages) ok = bar_wait(&empty[s], phase ^ 1u, abort_v);
      if (!ok) break;
      const TilePos p = tile_pos(t, 1, a.tiles_x, a.tiles_y);
      const uint32_t st = saddr + (uint32_t)s * a.stage_bytes;
      if (hp0 < stride) halo_load(a.h, tab, st, p.img, p.py, p.px, m0, hc, hp0, stride);
      if (zp0 < zstride) {
        const bf16* z0 = a.dz + zch * 8;
        const bf16* zb = z0 + (((int64_t)p.img * a.oh + p.py) * a.ow + p.px) * a.cout;
        const uint32_t d0 = st + a.x_bytes + (uint32_t)(zch * a.dz_plane) * 16u;
#pragma unroll 4
        for (int q = zp0; q < kTM; q += zstride) {
          const bool in = p.py + (q >> 3) < a.oh && p.px + (q & 7) < a.ow;
          cp16(d0 + (uint32_t)q * 16u, in ? zb + ((q >> 3) * a.ow + (q & 7)) * a.cout : z0, in);
        }
      }
      cp_arrive(&full[s]);
      if (++s == a.stages) {
        s = 0;
        phase ^= 1u;
      }
      ++issued;
    }
    if (!ok) give_up(abort_v, status);
    cp_drain();
  } else {
    // both operands with their channels contiguous
    const uint32_t idesc = umma::idesc_bf16_f32(64, n_cols, true, true);
    const uint32_t x_chunk = (uint32_t)a.h.plane * 16u, x_row = (uint32_t)(a.h.step * a.h.rp) * 16u;
    const uint32_t z_chunk = (uint32_t)a.dz_plane * 16u, z_row = 128u;
    const uint64_t xd = umma::smem_desc(saddr, x_row, x_chunk);
    const uint64_t zd = umma::smem_desc(saddr + a.x_bytes, z_row, z_chunk);
    const uint32_t a_hi = (uint32_t)((a.m_is_ci ? xd : zd) >> 32), b_hi = (uint32_t)((a.m_is_ci ? zd : xd) >> 32);
    const uint32_t a_lo = (uint32_t)(a.m_is_ci ? xd : zd), b_lo = (uint32_t)(a.m_is_ci ? zd : xd);
    // two tile rows further in either operand, in 16 bytes
    const uint32_t a_k = (a.m_is_ci ? x_row : z_row) >> 3, b_k = (a.m_is_ci ? z_row : x_row) >> 3;
    uint32_t toff[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) toff[j] = a.t.off[0][j];
    int s = 0;
    uint32_t phase = 0;
    bool ok = true, accum = false;
    for (int t = (int)blockIdx.x; t < a.ntiles; t += G) {
      ok = __all_sync(0xffffffffu, bar_wait(&full[s], phase, abort_v));
      if (!ok) break;
      umma::fence_smem_async();  // the copies, for the MMAs
      umma::fence_after();
      const uint32_t st = (uint32_t)s * (a.stage_bytes >> 4);
      uint32_t d = tmem;
#pragma unroll
      for (int tap = 0; tap < 9; ++tap) {
        if (tap < tap0 || tap >= tap1) continue;
        uint32_t alo = a_lo + st + (a.m_is_ci ? toff[tap] : 0u), blo = b_lo + st + (a.m_is_ci ? 0u : toff[tap]);
#pragma unroll
        for (int k = 0; k < kTM / 16; ++k) {
          umma::mma_bf16(d, alo, a_hi, blo, b_hi, idesc, accum || k > 0);
          alo += a_k;
          blo += b_k;
        }
        d += (uint32_t)n_cols;
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
  if (ok && warp < 8) {
    // row 16 w + l of the 64 sits in lane 32 w + l (l < 16); warps w and w + 4
    // take every other tap
    const int w = warp & 3, m = w * 16 + lane;
    const int64_t ld = 9 * (int64_t)a.cin;
    const bool on = lane < 16 && m0 * a.m_is_ci + m < (a.m_is_ci ? a.cin : a.cout);
    float* row = a.m_is_ci ? a.dw + m0 + m : a.dw + (int64_t)m * ld + m0;
    for (int tap = tap0 + (warp >> 2); tap < tap1; tap += 2)
      for (int c0 = 0; c0 < n_cols; c0 += 16) {
        float v[16];
        umma::tmem_ld16(tmem + ((uint32_t)(w * 32) << 16) + (uint32_t)((tap - tap0) * n_cols + c0), v);
        if (!on) continue;
        if (a.m_is_ci) {
          float* o = row + (int64_t)c0 * ld + (int64_t)tap * a.cin;
#pragma unroll
          for (int j = 0; j < 16; ++j) atomicAdd(o + (int64_t)j * ld, v[j]);
        } else {
          float* o = row + (int64_t)tap * a.cin + c0;
          if (a.vec) {
#pragma unroll
            for (int j = 0; j < 16; j += 4) red4(o + j, v[j], v[j + 1], v[j + 2], v[j + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) atomicAdd(o + j, v[j]);
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
