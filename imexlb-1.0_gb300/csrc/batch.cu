// Lockstep stepping of many independent cases (an ensemble of lattices): one
// launch per iteration for up to kBatchPart cases, boundary copies included,
// and one for the boundary refresh of those whose boundary program does not
// fold into the step. Each case keeps its own geometry and buffers; the
// launch's parameters map its blocks onto them, and a device counter (advanced
// by a one-thread kernel after a run of iterations) lets a captured CUDA graph
// replay them while cases with a smaller budget drop out.
#include <cstdint>

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "batch.h"
#include "boundary_fused.cuh"
#include "lattice.h"
#include "node_fast.cuh"
#include "pair_node.cuh"
#include "pdl.cuh"
#include "storage.cuh"

namespace imx {
namespace {

// One node of a case; boundary copies folded in (boundary_fused.cuh) where
// the case has the plan, as in the single-case kernels.
template <int DIM, class T>
__device__ IMX_FI void update_node(const BatchNode& c, const T* __restrict__ fin, T* fout, uint32_t id,
                                   uint8_t m) {
  using N_ = NodeFast<DIM, float>;
  using L = Lattice<DIM>;
  constexpr int Q = N_::Q;
  const DevState st{c.mask, c.inlet, nullptr, nullptr, c.bnd, c.bnd_at, c.push, c.pshift};
  const PullFix fx = PullFix::make(st, (m & kMaskFluid) ? m : (uint8_t)0);
  const bool bwarp = __any_sync(0xffffffffu, fx.other());
  if (!(m & kMaskFluid)) return;
  const int64_t N = c.N;
  auto off = [&](int i) { return L::ex(i) + c.dy * L::ey(i) + (DIM == 3 ? c.dz * L::ez(i) : (int64_t)0); };
  const T* node = fin + id;
  float f[Q];
  if (!bwarp) {
    const uint32_t inl = fx.inl();
    const bool o = fx.outl() != 0u;
    sfor<0, Q>([&](auto I) {
      constexpr int i = I, ex = L::ex(I);
      const T* p = node + (i * N - off(i));
      if constexpr (ex == 1) p += inl;
      else if constexpr (ex == -1) p = o ? node + i * N : p;
      f[I] = Store<T>::to_f(*p);
    });
  } else if (!fx.record()) {
    sfor<0, Q>([&](auto I) {
      constexpr int i = I;
      bool opp;
      int64_t sh;
      fx.form<DIM>(L::ex(i), L::ey(i), L::ez(i), off(i), c.pshift, opp, sh);
      f[I] = Store<T>::to_f(node[(opp ? (Q - 1 - i) * N + off(i) : i * N - off(i)) + sh]);
    });
  } else {
    const uint32_t* row = PullFix::row<Q>(st, id);
    sfor<0, Q>([&](auto I) {
      constexpr int i = I;
      const uint32_t r = row[I];
      f[I] = Store<T>::to_f(r != kNoRedirect ? fin[r] : node[i * N - off(i)]);
    });
  }
  float u[DIM];
  float S3 = N_::moments(f, u, c.k.inv_rho0);
  // PostProcessing's Dirichlet conditions (NodeFast::dirichlet)
  if (m & kMaskInlet) {
    u[0] = (float)c.inlet[id / (uint32_t)(DIM == 2 ? c.dy : c.dz)];
    u[1] = 0.0f;
  }
  if (m & kMaskOutlet) S3 = 0.0f;
  T* out = fout + id;
  N_::collide(f, S3, u, c.k, [&](int i, float v) { out[i * N] = Store<T>::from_f(v); });
  if (fx.record()) push_copies(st.push, PullFix::row<Q>(st, id)[Q], fin, fout);
}

// One iteration of every active case: block b serves the BLOCK*CPT cells
// b - first[j] of case j. The case comes from the launch's parameters (a
// search of at most four steps in the constant bank): from tables in memory a
// block took two dependent L2 latencies to its first load (24 cylinder
// cases: 43.7 against 35.3 ms per 500 iterations). 40 registers for 48 warps per SM.
template <int DIM, class T, int BLOCK, int CPT, int CAP>
__global__ void __launch_bounds__(BLOCK, DIM == 2 ? 1536 / BLOCK : 0) k_step_batch(const __grid_constant__ BatchArgs<CAP> a,
                                                       const BatchCase* __restrict__ cases,
                                                       const int* __restrict__ counter, int k0) {
  int j = 0, hi = a.n;
  while (hi - j > 1) {
    const int mid = (j + hi) >> 1;
    if (blockIdx.x >= a.first[mid]) j = mid;
    else hi = mid;
  }
  j = __shfl_sync(0xffffffffu, j, 0);  // (uniform for the compiler too)
  const BatchNode& c = a.c[j];
  const uint32_t id0 = c.id_lo + (blockIdx.x - a.first[j]) * (uint32_t)(BLOCK * CPT) + threadIdx.x;
  uint8_t m = id0 < c.id_hi ? c.mask[id0] : (uint8_t)0;
  const BatchCase& cs = cases[c.case_id];
  const int it = *counter + k0;
  if (it >= cs.nsteps) return;
  const int par = (cs.parity0 + it) & 1;
  const T* fin = (const T*)(par ? c.fb[1] : c.fb[0]);
  T* fout = (T*)(par ? c.fb[0] : c.fb[1]);
  update_node<DIM, T>(c, fin, fout, id0, m);
#pragma unroll 1
  for (int k = 1; k < CPT; ++k) {
    const uint32_t id = id0 + (uint32_t)(k * BLOCK);
    m = id < c.id_hi ? c.mask[id] : (uint8_t)0;
    update_node<DIM, T>(c, fin, fout, id, m);
  }
}

// A D2Q9 case as pair_update takes it.
template <class T>
struct PairCase {
  const DevState st;
  const CoefR<float>& k;
  const T* src;
  T* dst;
  int64_t N, dy;
  uint32_t id_hi;
  template <int I>
  __device__ IMX_FI int64_t off() const { return Lattice<2>::ex(I) + dy * Lattice<2>::ey(I); }
  template <int I>
  __device__ IMX_FI const T* in() const { return src + (I * N - off<I>()); }
  __device__ IMX_FI const T* fin() const { return src; }
  __device__ IMX_FI T* fout() const { return dst; }
  __device__ IMX_FI T* out(int i) const { return dst + i * N; }
};

// k_step_batch on D2Q9 with two neighbouring cells per thread (pair_node.cuh):
// block b serves the 2 BLOCK cells b - first[j] of case j.
// The counter and the cases' budgets don't change between the launches of a
// run, so they too are read before the previous iteration ends; a run's first
// launch is a plain one.
template <class T, int BLOCK, int CAP>
__global__ void __launch_bounds__(BLOCK, 1280 / BLOCK) k_step_batch_pair(const __grid_constant__ BatchArgs<CAP> a,
                                                                         const BatchCase* __restrict__ cases,
                                                                         const int* __restrict__ counter, int k0) {
  int j = 0, hi = a.n;
  while (hi - j > 1) {
    const int mid = (j + hi) >> 1;
    if (blockIdx.x >= a.first[mid]) j = mid;
    else hi = mid;
  }
  j = __shfl_sync(0xffffffffu, j, 0);  // (uniform for the compiler too)
  const BatchNode& c = a.c[j];
  const uint32_t id = c.id_lo + 2u * ((blockIdx.x - a.first[j]) * (uint32_t)BLOCK + threadIdx.x);
  const BatchCase& cs = cases[c.case_id];
  const int it = *counter + k0;
  if (it >= cs.nsteps) return;
  const int par = (cs.parity0 + it) & 1;
  const PairCase<T> lat{DevState{c.mask, c.inlet, nullptr, nullptr, c.bnd, c.bnd_at, c.push, c.pshift}, c.k,
                        (const T*)(par ? c.fb[1] : c.fb[0]), (T*)(par ? c.fb[0] : c.fb[1]), c.N, c.dy, c.id_hi};
  auto none = [](uint32_t, float) {};
  if (c.dy & 1) pair_update<T, true, false>(lat, id, [] { pdl_wait(); pdl_trigger(); }, none);
  else pair_update<T, false, false>(lat, id, [] { pdl_wait(); pdl_trigger(); }, none);
}

// Boundary refresh of every active case: a block serves 256 entries of a
// case's fill list.
template <class T>
__global__ void __launch_bounds__(256) k_fill_batch(const BatchCase* __restrict__ cases,
                                                     const BatchBlock* __restrict__ fills,
                                                     const int* __restrict__ counter, int k0) {
  const BatchBlock bb = fills[blockIdx.x];
  const BatchCase& cs = cases[bb.case_id];
  const int it = *counter + k0;
  if (it >= cs.nsteps) return;
  const int par = (cs.parity0 + it) & 1;
  const T* fin = (const T*)cs.fb[par];
  T* fout = (T*)cs.fb[1 - par];
  const int64_t i = (int64_t)bb.item * 256 + threadIdx.x;
  if (i >= cs.n_fill) return;
  int64_t dst, src;
  if (cs.fill_narrow) {
    const DevFill32 e = ((const DevFill32*)cs.fill)[i];
    dst = e.dst;
    src = e.src == kFillNaN32 ? kFillNaN : (int64_t)e.src;
  } else {
    const DevFill e = ((const DevFill*)cs.fill)[i];
    dst = e.dst;
    src = e.src;
  }
  T v;
  if (src >= 0) v = fout[src];
  else if (src != kFillNaN) v = fin[~src];
  else v = Store<T>::nan();
  fout[dst] = v;
}

__global__ void k_tick(int* counter, int n) { *counter += n; }

template <class F>
cudaError_t dispatch_lp_b(int store, F&& fn) {
  switch (store) {
    case kStoreF32: return fn(float{});
    case kStoreBF16: return fn(__nv_bfloat16{});
    case kStoreF16: return fn(__half{});
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

const BatchShape kBatchShapes[kNumBatchShapes] = {
    {128, 1}, {256, 1}, {512, 1}, {128, 2}, {256, 2}, {128, 4}};

namespace {

// fn(kernel, threads per block, dependent) of a launch shape; a dependent
// kernel waits for the previous one by itself.
template <int DIM, class T, int CAP, class F>
cudaError_t with_step_kernel(int shape, F&& fn) {
  if constexpr (DIM == 2) {
    switch (shape) {
      case 3: return fn(k_step_batch_pair<T, 128, CAP>, 128, true);
      case 4: return fn(k_step_batch_pair<T, 256, CAP>, 256, true);
      default: break;
    }
  } else {
    switch (shape) {
      case 3: return fn(k_step_batch<DIM, T, 128, 2, CAP>, 128, false);
      case 4: return fn(k_step_batch<DIM, T, 256, 2, CAP>, 256, false);
      default: break;
    }
  }
  switch (shape) {
    case 0: return fn(k_step_batch<DIM, T, 128, 1, CAP>, 128, false);
    case 1: return fn(k_step_batch<DIM, T, 256, 1, CAP>, 256, false);
    case 2: return fn(k_step_batch<DIM, T, 512, 1, CAP>, 512, false);
    default: return fn(k_step_batch<DIM, T, 128, 4, CAP>, 128, false);
  }
}

}  // namespace

template <int CAP>
cudaError_t launch_batch_iteration(int dim, int store, int shape, const BatchArgs<CAP>& a,
                                   const BatchCase* cases, const BatchBlock* fills, int64_t nfills,
                                   const int* counter, int k, cudaStream_t s) {
  return dispatch_lp_b(store, [&](auto tag) {
    using T = decltype(tag);
    auto launch = [&](auto kern, int threads, bool dependent) {
      // (the first launch of a run follows the counter's writer)
      if (dependent && k > 0) return launch_pdl(kern, a.first[a.n], (unsigned)threads, s, a, cases, counter, k);
      kern<<<a.first[a.n], threads, 0, s>>>(a, cases, counter, k);
      return cudaGetLastError();
    };
    const cudaError_t e =
        dim == 2 ? with_step_kernel<2, T, CAP>(shape, launch) : with_step_kernel<3, T, CAP>(shape, launch);
    if (e != cudaSuccess) return e;
    if (nfills > 0) k_fill_batch<T><<<(unsigned)nfills, 256, 0, s>>>(cases, fills, counter, k);
    return cudaGetLastError();
  });
}

template <int CAP>
cudaError_t load_batch_kernel(int dim, int store, int shape) {
  return dispatch_lp_b(store, [&](auto tag) {
    using T = decltype(tag);
    auto load = [](auto kern, int, bool) {
      cudaFuncAttributes fa;
      return cudaFuncGetAttributes(&fa, kern);
    };
    return dim == 2 ? with_step_kernel<2, T, CAP>(shape, load) : with_step_kernel<3, T, CAP>(shape, load);
  });
}

#define I_(CAP)                                                                                             \
  template cudaError_t launch_batch_iteration<CAP>(int, int, int, const BatchArgs<CAP>&, const BatchCase*,  \
                                                   const BatchBlock*, int64_t, const int*, int, cudaStream_t); \
  template cudaError_t load_batch_kernel<CAP>(int, int, int);
I_(kBatchFew)
I_(kBatchPart)
#undef I_

cudaError_t launch_batch_tick(int* counter, int n, cudaStream_t s) {
  k_tick<<<1, 1, 0, s>>>(counter, n);
  return cudaGetLastError();
}

}  // namespace imx
