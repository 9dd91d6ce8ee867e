// FP64 lattice Boltzmann kernels for sm_103a with the reference's rounding.
//
// Every floating-point operation is an explicit round-to-nearest intrinsic in
// the evaluation order of lbm.f90 (Collision lbm.f90:64-72, PostProcessing
// lbm.f90:166-179), so no multiply-add is ever fused and results equal the
// reference's serial build. Terms the reference multiplies by an integer
// lattice component in {-1,0,1} are added, subtracted or skipped; that is
// exact (it can change only the sign of an exact zero). A +/- direction pair
// shares |e.u|, e.u squared and 4.5(e.u)^2, which are exactly equal for the
// two members (e_opp = -e).
//
// GB300 has ~0.5 T FP64 add/mul per second against ~7 TB/s of HBM, so these
// kernels are bound by FP64 issue, not memory; the work per node is kept to
// the reference's own operation count.
#include <cstdint>

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "exact_node.cuh"
#include "kernels.h"
#include "lattice.h"
#include "storage.cuh"

namespace imx {
namespace {

// The kernels around the step use the default variant's operations where
// rho0 = 1 (exact_node.cuh: multiplications and the division by 3 in integer
// arithmetic, a run-time loop over the pairs), else the plain ones: the same
// bits, with the FP64 pipe left to the additions.
template <int DIM, bool RHO1>
struct AuxEm {
  static constexpr uint32_t v = RHO1 ? Splits<DIM>::v[Splits<DIM>::kDefault] : 0u;
};

// 256x128x128 sphere, rho0 = 1: 1318 us against 2093 us with the FP64
// pipe's multiplications (Monitor iteration).
template <int DIM, bool RHO1, bool MON>
__global__ void __launch_bounds__(kBlock) k_collide_fpu(DevGrid g, DevCoef c, DevState st,
                                                         const double* __restrict__ fs,
                                                         const double* __restrict__ ps,
                                                         const double* __restrict__ us,
                                                         double* __restrict__ fout,
                                                         unsigned long long* monitor) {
  constexpr uint32_t EM = AuxEm<DIM, RHO1>::v;
  using N_ = Node<DIM, RHO1, EM>;
  const int64_t id = g.id_lo + (int64_t)blockIdx.x * kBlock + threadIdx.x;
  double um = 0.0;
  if (id < g.id_hi) {
    const uint8_t m = st.mask[id];
    if (m & kMaskFluid) {
      double u[DIM];
      sfor<0, DIM>([&](auto K) { u[K] = us[(int64_t)K * g.N + id]; });
      const double p = ps[id];
      if constexpr (MON) {
        if (id != g.skip_id) um = speed2d(u[0], u[1]);
      }
      if constexpr ((EM & kLoopPairs) != 0u) {
        N_::template collide_loop<false, false>(p, u, c, st, fs, g, fout, id, PullFix{0u});
      } else {
        double f[N_::Q];
        sfor<0, N_::Q>([&](auto I) { f[I] = fs[(int64_t)I * g.N + id]; });
        N_::collide(f, p, u, c, fout, g.N, id);
      }
    }
  }
  if constexpr (MON) block_max_to(um, monitor);
}

// fs null: f is not wanted.
template <int DIM, bool RHO1>
__global__ void __launch_bounds__(kBlock) k_finalize(DevGrid g, DevCoef c, DevState st,
                                                      const double* __restrict__ fin,
                                                      double* __restrict__ fs,
                                                      double* __restrict__ ps,
                                                      double* __restrict__ us) {
  using N_ = Node<DIM, RHO1, AuxEm<DIM, RHO1>::v>;
  const int64_t id = g.id_lo + (int64_t)blockIdx.x * kBlock + threadIdx.x;
  if (id >= g.id_hi) return;
  const uint8_t m = st.mask[id];
  if (!(m & kMaskFluid)) return;
  double f[N_::Q];
  N_::pull(fin, g, id, f);
  double p, u[DIM];
  N_::moments(f, p, u, c);
  N_::dirichlet(m, id, g, st.inlet, p, u);
  if (fs) sfor<0, N_::Q>([&](auto I) { fs[(int64_t)I * g.N + id] = f[I]; });
  sfor<0, DIM>([&](auto K) { us[(int64_t)K * g.N + id] = u[K]; });
  ps[id] = p;
}

// 256x128x128 sphere, rho0 = 1: 971 us against 1396 us with the FP64
// pipe's multiplications.
template <int DIM, bool RHO1>
__global__ void __launch_bounds__(kBlock) k_init_pdf(DevGrid g, DevCoef c, DevState st,
                                                      const double* __restrict__ ps,
                                                      const double* __restrict__ us,
                                                      double* __restrict__ fs) {
  constexpr uint32_t EM = AuxEm<DIM, RHO1>::v;
  using N_ = Node<DIM, RHO1, EM>;
  const int64_t id = g.id_lo + (int64_t)blockIdx.x * kBlock + threadIdx.x;
  if (id >= g.id_hi) return;
  if (!(st.mask[id] & kMaskFluid)) return;
  double u[DIM];
  sfor<0, DIM>([&](auto K) { u[K] = us[(int64_t)K * g.N + id]; });
  auto store = [&](int i, double fe) { fs[(int64_t)i * g.N + id] = fe; };
  if constexpr ((EM & kLoopPairs) != 0u) N_::equilibria_loop(ps[id], u, c, st.tq, store);
  else N_::equilibria(ps[id], u, c, store);
}

template <class T, class E>
__global__ void k_fill(const E* __restrict__ fill, int64_t n, T* fout, const T* __restrict__ fin) {
  constexpr auto kNaN = sizeof(E) == sizeof(DevFill32) ? (int64_t)kFillNaN32 : kFillNaN;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const E e = fill[i];
    const int64_t src = e.src;
    T v;
    if (src >= 0) v = fout[src];
    else if (src != kNaN) v = fin[~src];
    else v = Store<T>::nan();
    fout[e.dst] = v;
  }
}

template <int DIM>
__global__ void k_columns(DevGrid g, const int* __restrict__ bl, int nl,
                          const int* __restrict__ br, int nr, const double* __restrict__ inlet,
                          double* p, double* u) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nl) {
    const int64_t id = (int64_t)bl[i] + 1;
    const int64_t r = DIM == 2 ? id / g.dy : id / g.dz;
    u[id] = inlet[r];
    u[g.N + id] = 0.0;
  }
  if (i < nr) p[(int64_t)br[i] - 1] = 0.0;
}

// ---- double-double accumulation (error-free TwoSum), used for the force and
// mass sums so that the result does not depend on the summation order to
// within ~1e-30 relative.
struct DD {
  double hi, lo;
};

__device__ IMX_FI DD dd_add(DD a, double x) {
  const double s = __dadd_rn(a.hi, x);
  const double bp = __dsub_rn(s, a.hi);
  const double e = __dadd_rn(__dsub_rn(a.hi, __dsub_rn(s, bp)), __dsub_rn(x, bp));
  return DD{s, __dadd_rn(a.lo, e)};
}

__device__ IMX_FI DD dd_add(DD a, DD b) {
  DD r = dd_add(a, b.hi);
  r.lo = __dadd_rn(r.lo, b.lo);
  // renormalise (Fast2Sum, |hi| >= |lo|)
  const double s = __dadd_rn(r.hi, r.lo);
  const double e = __dsub_rn(r.lo, __dsub_rn(s, r.hi));
  return DD{s, e};
}

constexpr int kRedThreads = 512;

// Fixed-shape tree reduction of one DD per component across the block.
template <int NC>
__device__ IMX_FI void block_dd_reduce(DD (&v)[NC], DD (*sh)[NC]) {
  const int t = threadIdx.x;
#pragma unroll
  for (int c = 0; c < NC; ++c) sh[t][c] = v[c];
  __syncthreads();
  for (int stride = kRedThreads / 2; stride > 0; stride >>= 1) {
    if (t < stride) {
#pragma unroll
      for (int c = 0; c < NC; ++c) sh[t][c] = dd_add(sh[t][c], sh[t + stride][c]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) v[c] = sh[0][c];
}

// a + b without the renormalisation (the low parts only accumulate).
__device__ IMX_FI DD dd_merge(DD a, DD b) {
  DD r = dd_add(a, b.hi);
  r.lo = __dadd_rn(r.lo, b.lo);
  return r;
}

// The force sum: the links strided over all blocks; each block leaves one
// partial sum per component, and the block that finishes last adds them in
// block order (a fixed tree: the result does not depend on which block that
// is). An FP64 instruction holds an SM's FP64 pipe for ~20 cycles whatever its
// active lanes, so the links are spread over the SMs and the trees keep the
// components of a level in one warp's lanes. One block of 512 threads took
// 201 us a sample on the 256x128x128 sphere (D 24), 777 us on the 512x256x256 one
// and 13 us on the 1024x512 cylinder; now 13, 17 and 8 us.
constexpr int kForceThreads = 128;

// Tree over the block's values, one DD per thread and component; component
// c's sum ends in thread c.
template <int NC>
__device__ IMX_FI DD force_tree(const DD (&v)[NC], DD (*sh)[kForceThreads]) {
  const int t = threadIdx.x;
#pragma unroll
  for (int c = 0; c < NC; ++c) sh[c][t] = v[c];
  __syncthreads();
  DD r{0.0, 0.0};
  auto level = [&](int width) {  // threads c * width + j: four values each
    if (t < NC * width) {
      const int c = t / width, j = t - c * width;
      r = sh[c][j];
#pragma unroll
      for (int k = 1; k < 4; ++k) r = dd_merge(r, sh[c][j + k * width]);
    }
  };
  auto keep = [&](int width) {
    if (t < NC * width) sh[t / width][t - t / width * width] = r;
  };
  level(32);
  __syncthreads();
  keep(32);
  __syncthreads();
  if (t < 32) {
    level(8);
    __syncwarp();
    keep(8);
    __syncwarp();
    level(2);
    __syncwarp();
    keep(2);
    __syncwarp();
    if (t < NC) r = dd_merge(sh[t][0], sh[t][1]);
  }
  return r;
}

template <int DIM, class T>
__global__ void __launch_bounds__(kForceThreads) k_forces(const DevLink* __restrict__ links, int64_t n,
                                                          const T* __restrict__ fb,
                                                          double* __restrict__ partials,
                                                          unsigned* __restrict__ arrived,
                                                          double* __restrict__ out) {
  using Lat = Lattice<DIM>;
  __shared__ DD sh[DIM][kForceThreads];
  __shared__ unsigned last;
  const int t = threadIdx.x;
  DD acc[DIM];
#pragma unroll
  for (int c = 0; c < DIM; ++c) acc[c] = DD{0.0, 0.0};
  constexpr int kU = 4;  // links in flight
  const int64_t step = (int64_t)gridDim.x * kForceThreads;
  for (int64_t i0 = (int64_t)blockIdx.x * kForceThreads + t; i0 < n; i0 += kU * step) {
    DevLink L[kU];
    double v[kU];
#pragma unroll
    for (int k = 0; k < kU; ++k)
      if (i0 + k * step < n) L[k] = links[i0 + k * step];
#pragma unroll
    for (int k = 0; k < kU; ++k)
      if (i0 + k * step < n) v[k] = __dadd_rn(Store<T>::to_d(fb[L[k].a]), Store<T>::to_d(fb[L[k].b]));
#pragma unroll
    for (int k = 0; k < kU; ++k) {
      if (i0 + k * step >= n) break;
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        // e * v with e in {-1, 0, 1} (adding zero is exact)
        const int e = Lat::e(L[k].iq, c);
        acc[c] = dd_add(acc[c], e > 0 ? v[k] : (e < 0 ? -v[k] : 0.0));
      }
    }
  }
  DD r = force_tree<DIM>(acc, sh);
  if (gridDim.x > 1) {
    if (t < DIM) {
      partials[2 * (blockIdx.x * DIM + t)] = r.hi;
      partials[2 * (blockIdx.x * DIM + t) + 1] = r.lo;
      __threadfence();
    }
    __syncthreads();
    if (t == 0) last = atomicAdd(arrived, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
#pragma unroll
    for (int c = 0; c < DIM; ++c) acc[c] = DD{0.0, 0.0};
    for (int b = t; b < (int)gridDim.x; b += kForceThreads) {
#pragma unroll
      for (int c = 0; c < DIM; ++c)
        acc[c] = dd_merge(acc[c], DD{__ldcg(partials + 2 * (b * DIM + c)), __ldcg(partials + 2 * (b * DIM + c) + 1)});
    }
    r = force_tree<DIM>(acc, sh);
    if (t == 0) *arrived = 0u;  // for the handle's next sample
  }
  if (t < DIM) out[t] = __dadd_rn(r.hi, r.lo);
}

constexpr int kMassBlock = 256;

template <int DIM, class T>
__global__ void __launch_bounds__(kMassBlock) k_mass_partial(DevGrid g, DevState st,
                                                              const T* __restrict__ fin,
                                                              double* partials) {
  using Lat = Lattice<DIM>;
  const int64_t id = g.id_lo + (int64_t)blockIdx.x * kMassBlock + threadIdx.x;
  DD acc{0.0, 0.0};
  if (id < g.id_hi && (st.mask[id] & kMaskFluid)) {
    sfor<0, Lat::Q>([&](auto I) {
      acc = dd_add(acc, Store<T>::to_d(fin[(int64_t)I * g.N + id - g.off[I]]));
    });
  }
  // fixed-shape block tree
  __shared__ DD sh[kMassBlock];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int stride = kMassBlock / 2; stride > 0; stride >>= 1) {
    if (threadIdx.x < stride) sh[threadIdx.x] = dd_add(sh[threadIdx.x], sh[threadIdx.x + stride]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = sh[0].hi;
    partials[2 * blockIdx.x + 1] = sh[0].lo;
  }
}

__global__ void __launch_bounds__(kRedThreads) k_mass_final(const double* __restrict__ partials,
                                                             int64_t nb, double* out) {
  __shared__ DD sh[kRedThreads][1];
  DD acc[1] = {DD{0.0, 0.0}};
  for (int64_t i = threadIdx.x; i < nb; i += kRedThreads)
    acc[0] = dd_add(acc[0], DD{partials[2 * i], partials[2 * i + 1]});
  block_dd_reduce<1>(acc, sh);
  if (threadIdx.x == 0) out[0] = __dadd_rn(acc[0].hi, acc[0].lo);
}

// Layout conversions through a tile of `tile` cells in shared memory. Vector
// fields (K <= 3) take 256 cells, so that a block's 256 threads move whole rows: u of
// 256x128x128 47 us against 137 us with 32 cells a block.
inline int transpose_tile(int K) { return K <= 3 ? 256 : 32; }

template <class T>
__global__ void k_aos_to_soa(const double* __restrict__ aos, T* __restrict__ soa, int64_t N,
                             int64_t stride, int K, int ntile) {
  extern __shared__ double tile[];
  const int64_t c0 = (int64_t)blockIdx.x * ntile;
  const int ncell = (int)((N - c0) < ntile ? (N - c0) : ntile);
  for (int j = threadIdx.x; j < ncell * K; j += blockDim.x) tile[j] = aos[c0 * K + j];
  __syncthreads();
  for (int j = threadIdx.x; j < ncell * K; j += blockDim.x) {
    const int k = j / ncell, c = j - k * ncell;
    soa[(int64_t)k * stride + c0 + c] = Store<T>::from_d(tile[c * K + k]);
  }
}

template <class T>
__global__ void k_soa_to_aos(const T* __restrict__ soa, double* __restrict__ aos, int64_t N,
                             int64_t stride, int K, int ntile) {
  extern __shared__ double tile[];
  const int64_t c0 = (int64_t)blockIdx.x * ntile;
  const int ncell = (int)((N - c0) < ntile ? (N - c0) : ntile);
  for (int j = threadIdx.x; j < ncell * K; j += blockDim.x) {
    const int k = j / ncell, c = j - k * ncell;
    tile[c * K + k] = Store<T>::to_d(soa[(int64_t)k * stride + c0 + c]);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < ncell * K; j += blockDim.x) aos[c0 * K + j] = tile[j];
}

inline unsigned grid_for(const DevGrid& g) {
  return (unsigned)((g.id_hi - g.id_lo + kBlock - 1) / kBlock);
}

}  // namespace

cudaError_t launch_collide_fpu(int dim, bool rho_one, const DevGrid& g, const DevCoef& c,
                               const DevState& st, const double* f, const double* p,
                               const double* u, double* fout, unsigned long long* monitor,
                               cudaStream_t s) {
  const unsigned grid = grid_for(g);
  const bool mon = monitor != nullptr;
#define L_(D, R, M) k_collide_fpu<D, R, M><<<grid, kBlock, 0, s>>>(g, c, st, f, p, u, fout, monitor)
  if (dim == 2) {
    if (rho_one) { if (mon) L_(2, true, true); else L_(2, true, false); }
    else { if (mon) L_(2, false, true); else L_(2, false, false); }
  } else {
    if (rho_one) { if (mon) L_(3, true, true); else L_(3, true, false); }
    else { if (mon) L_(3, false, true); else L_(3, false, false); }
  }
#undef L_
  return cudaGetLastError();
}

// FP64 fused multiply-add throughput: eight independent chains per thread
// (x = x*y + z with y < 1, so the values stay bounded); the result is kept
// live through one conditional store.
__global__ void __launch_bounds__(256) k_dfma_rate(double* out, double y, double z, int iters) {
  double x[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] = (double)(threadIdx.x + j);
#pragma unroll 1
  for (int k = 0; k < iters; ++k) {
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = fma(x[j], y, z);
  }
  double s = 0.0;
#pragma unroll
  for (int j = 0; j < 8; ++j) s += x[j];
  if (s == -1.0) out[0] = s;
}

int step_splits() { return Splits<3>::n; }
int step_split_default(int dim) { return dim == 2 ? Splits<2>::kDefault : Splits<3>::kDefault; }

cudaError_t launch_step(int dim, bool rho_one, const DevGrid& g, const DevCoef& c,
                        const DevState& st, const double* fin, double* fout,
                        unsigned long long* monitor, cudaStream_t s, int split) {
  const unsigned grid = grid_for(g);
  const bool mon = monitor != nullptr;
  if (split < 0 || split >= step_splits()) return cudaErrorInvalidValue;
  if (st.bnd) {  // boundary copies folded in: the default variant only
    if (rho_one && split != step_split_default(dim)) return cudaErrorInvalidValue;
    return launch_step_fused(dim, rho_one, grid, g, c, st, fin, fout, monitor, s);
  }
  if (rho_one) {
    return dim == 2 ? launch_step_split2(split, grid, g, c, st, fin, fout, monitor, s)
                    : launch_step_split3(split, grid, g, c, st, fin, fout, monitor, s);
  }
#define L_(D, M) k_step<D, false, M><<<grid, kBlock, 0, s>>>(g, c, st, fin, fout, monitor)
  if (dim == 2) { if (mon) L_(2, true); else L_(2, false); }
  else { if (mon) L_(3, true); else L_(3, false); }
#undef L_
  return cudaGetLastError();
}

namespace {

__global__ void k_fill_group(const DevGroupFill* __restrict__ fill, int64_t n,
                             double* const* __restrict__ bufs, int out_parity) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const DevGroupFill e = fill[i];
    double v;
    if (e.src_code < 0) {
      v = __longlong_as_double(0x7ff8000000000000ll);
    } else {
      const int r = e.src_code & 0xffff;
      const int k = (e.src_code & kGroupPrev) ? 1 - out_parity : out_parity;
      v = bufs[2 * r + k][e.src];
    }
    bufs[2 * e.dst_rank + out_parity][e.dst] = v;
  }
}

}  // namespace

namespace {

// The reference's InitUP: u_x = prof(row) * r(id mod 100), both factors made on
// the host in its order (profile: (((uu*4)*y)*(n-y))/n**2, times geo(id) = 1 on
// fluid nodes). 512x256x256: 175 us against 1384 us with the profile's
// division per node.
template <int DIM>
__global__ void k_init_up(DevGrid g, const uint8_t* __restrict__ mask, RVec r,
                          const double* __restrict__ prof, double* __restrict__ u) {
  __shared__ double rs[100];
  if (threadIdx.x < 100) rs[threadIdx.x] = r.v[threadIdx.x];
  __syncthreads();
  // fluid nodes are listed as 32-bit ids
  const uint32_t id = (uint32_t)g.id_lo + blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= (uint32_t)g.id_hi || !(mask[id] & kMaskFluid)) return;
  const uint32_t row = DIM == 2 ? id / (uint32_t)g.dy : id / (uint32_t)g.dz;
  u[id] = __dmul_rn(prof[row], rs[id % 100u]);
}

}  // namespace

cudaError_t launch_init_up(int dim, const DevGrid& g, const uint8_t* mask, const RVec& r,
                           const double* prof, double* u, cudaStream_t s) {
  const int64_t cells = g.id_hi - g.id_lo;
  if (cells <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)((cells + 255) / 256);
  if (dim == 2) k_init_up<2><<<grid, 256, 0, s>>>(g, mask, r, prof, u);
  else k_init_up<3><<<grid, 256, 0, s>>>(g, mask, r, prof, u);
  return cudaGetLastError();
}

cudaError_t launch_fill_group(const DevGroupFill* fill, int64_t n, double* const* bufs,
                              int out_parity, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  if (blocks > 152 * 32) blocks = 152 * 32;
  k_fill_group<<<(unsigned)blocks, 256, 0, s>>>(fill, n, bufs, out_parity);
  return cudaGetLastError();
}

cudaError_t launch_fill(int store, const void* fill, bool narrow, int64_t n, void* fout,
                        const void* fin, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  if (blocks > 152 * 32) blocks = 152 * 32;
  return dispatch_store(store, [&](auto tag) {
    using T = decltype(tag);
    if (narrow)
      k_fill<T, DevFill32><<<(unsigned)blocks, 256, 0, s>>>((const DevFill32*)fill, n, (T*)fout,
                                                          (const T*)fin);
    else
      k_fill<T, DevFill><<<(unsigned)blocks, 256, 0, s>>>((const DevFill*)fill, n, (T*)fout,
                                                        (const T*)fin);
    return cudaGetLastError();
  });
}

cudaError_t launch_finalize(int dim, bool rho_one, const DevGrid& g, const DevCoef& c,
                            const DevState& st, const double* fin, double* f, double* p,
                            double* u, cudaStream_t s) {
  const unsigned grid = grid_for(g);
#define L_(D, R) k_finalize<D, R><<<grid, kBlock, 0, s>>>(g, c, st, fin, f, p, u)
  if (dim == 2) { if (rho_one) L_(2, true); else L_(2, false); }
  else { if (rho_one) L_(3, true); else L_(3, false); }
#undef L_
  return cudaGetLastError();
}

cudaError_t launch_columns(int dim, const DevGrid& g, const int* bl, int nl, const int* br,
                           int nr, const double* inlet, double* p, double* u, cudaStream_t s) {
  const int n = nl > nr ? nl : nr;
  if (n <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)((n + 255) / 256);
  if (dim == 2) k_columns<2><<<grid, 256, 0, s>>>(g, bl, nl, br, nr, inlet, p, u);
  else k_columns<3><<<grid, 256, 0, s>>>(g, bl, nl, br, nr, inlet, p, u);
  return cudaGetLastError();
}

cudaError_t launch_init_pdf(int dim, bool rho_one, const DevGrid& g, const DevCoef& c,
                            const DevState& st, const double* p, const double* u, double* f,
                            cudaStream_t s) {
  const unsigned grid = grid_for(g);
#define L_(D, R) k_init_pdf<D, R><<<grid, kBlock, 0, s>>>(g, c, st, p, u, f)
  if (dim == 2) { if (rho_one) L_(2, true); else L_(2, false); }
  else { if (rho_one) L_(3, true); else L_(3, false); }
#undef L_
  return cudaGetLastError();
}

cudaError_t launch_forces(int dim, int store, const DevLink* links, int64_t n, const void* fb,
                          double* partials, unsigned* arrived, double* out, cudaStream_t s) {
  // one block while its threads have at most eight links each: the second
  // stage (fence, counter, reload, tree) costs about as much as the first
  int64_t blocks = n <= 8 * kForceThreads ? 1 : (n + kForceThreads - 1) / kForceThreads;
  blocks = blocks < 1 ? 1 : (blocks > kForceBlocks ? kForceBlocks : blocks);
  return dispatch_store(store, [&](auto tag) {
    using T = decltype(tag);
    const unsigned g = (unsigned)blocks;
    if (dim == 2) k_forces<2, T><<<g, kForceThreads, 0, s>>>(links, n, (const T*)fb, partials, arrived, out);
    else k_forces<3, T><<<g, kForceThreads, 0, s>>>(links, n, (const T*)fb, partials, arrived, out);
    return cudaGetLastError();
  });
}

int64_t mass_partials_size(const DevGrid& g) {
  return 2 * ((g.id_hi - g.id_lo + kMassBlock - 1) / kMassBlock);
}

cudaError_t launch_mass(int dim, int store, const DevGrid& g, const DevState& st, const void* fin,
                        double* partials, double* out, cudaStream_t s) {
  const int64_t nb = (g.id_hi - g.id_lo + kMassBlock - 1) / kMassBlock;
  return dispatch_store(store, [&](auto tag) {
    using T = decltype(tag);
    if (dim == 2) k_mass_partial<2, T><<<(unsigned)nb, kMassBlock, 0, s>>>(g, st, (const T*)fin, partials);
    else k_mass_partial<3, T><<<(unsigned)nb, kMassBlock, 0, s>>>(g, st, (const T*)fin, partials);
    k_mass_final<<<1, kRedThreads, 0, s>>>(partials, nb, out);
    return cudaGetLastError();
  });
}

cudaError_t launch_aos_to_soa(int store, const double* aos, void* soa, int64_t N, int64_t stride,
                              int K, cudaStream_t s) {
  const int nt = transpose_tile(K);
  const unsigned grid = (unsigned)((N + nt - 1) / nt);
  return dispatch_store(store, [&](auto tag) {
    using T = decltype(tag);
    k_aos_to_soa<T><<<grid, 256, sizeof(double) * nt * K, s>>>(aos, (T*)soa, N, stride, K, nt);
    return cudaGetLastError();
  });
}

cudaError_t launch_soa_to_aos(int store, const void* soa, double* aos, int64_t N, int64_t stride,
                              int K, cudaStream_t s) {
  const int nt = transpose_tile(K);
  const unsigned grid = (unsigned)((N + nt - 1) / nt);
  return dispatch_store(store, [&](auto tag) {
    using T = decltype(tag);
    k_soa_to_aos<T><<<grid, 256, sizeof(double) * nt * K, s>>>((const T*)soa, aos, N, stride, K, nt);
    return cudaGetLastError();
  });
}

cudaError_t measure_dfma_rate(double* fma_per_s) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  double* out = nullptr;
  cudaEvent_t a = nullptr, b = nullptr;
  e = cudaMalloc((void**)&out, sizeof(double));
  if (e == cudaSuccess) e = cudaEventCreate(&a);
  if (e == cudaSuccess) e = cudaEventCreate(&b);
  const unsigned grid = (unsigned)sms * 16;
  const int iters = 2048;
  if (e == cudaSuccess) {
    k_dfma_rate<<<grid, 256>>>(out, 0.999999, 1e-3, 64);  // warm-up
    cudaEventRecord(a);
    k_dfma_rate<<<grid, 256>>>(out, 0.999999, 1e-3, iters);
    cudaEventRecord(b);
    e = cudaEventSynchronize(b);
  }
  float ms = 0.f;
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, a, b);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess && ms > 0.f) *fma_per_s = (double)grid * 256.0 * 8.0 * iters / (ms * 1e-3);
  if (a) cudaEventDestroy(a);
  if (b) cudaEventDestroy(b);
  if (out) cudaFree(out);
  return e;
}

}  // namespace imx
