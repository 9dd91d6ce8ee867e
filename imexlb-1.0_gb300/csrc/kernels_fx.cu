// Step kernel of the fixed-point kind (IMEXLB_FIX64): populations stored as
// Q3.60 integers, the whole node update on the integer pipes
// (node_fixed.cuh). Pull, boundary handling and obstacle copies are those of
// the other step kernels (kernels_lp.cu, boundary_fused.cuh): one thread per
// padded interior cell, the pulled population of direction i read from the
// direction's plane shifted by its pull offset (Propagation, lbm.f90:80-92),
// the moments and Dirichlet conditions of PostProcessing (lbm.f90:159-201),
// Monitor (lbm.f90:205-227) and Collision (lbm.f90:52-76).
#include <cstdint>

#include <cuda_runtime.h>

#include "boundary_fused.cuh"
#include "fixed64.cuh"
#include "kernels.h"
#include "lattice.h"
#include "node_fixed.cuh"

namespace imx {
namespace {

constexpr int kBlockFx = 128;

// How a launch's coefficients let the collision be formed (NodeFixed): any
// weights, or the lattice's own with 1 - ome >= 0 or < 0.
enum FxForm { kFxAny = 0, kFxPos = 1, kFxNeg = 2 };

// Resident blocks per SM the kernel is compiled for. D3Q27 holds 54 words of
// populations: at 96 registers (a few bytes spilled) five blocks hide the
// pulls best. Measured on 256x128x128 (us an iteration): two blocks of 256 threads
// 382, four of 128 357, five 340, six 370. The any-weights form needs 128
// registers. D2Q9 fits its 64 registers (4096x2048: 256-thread blocks 229, these 225).
template <int DIM, int FORM>
constexpr int kFxBlocks = FORM == kFxAny ? 4 : (DIM == 2 ? 8 : 5);

// Max over the block of non-negative values or NaN (their bit patterns order
// like the values, NaN above all), one atomicMax per block.
__device__ __forceinline__ void block_max_fx(double v, unsigned long long* dst) {
  unsigned long long b = (unsigned long long)__double_as_longlong(v);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long x = __shfl_xor_sync(0xffffffffu, b, o);
    b = x > b ? x : b;
  }
  __shared__ unsigned long long wmax[kBlockFx / 32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) wmax[w] = b;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long m = wmax[0];
    for (int i = 1; i < kBlockFx / 32; ++i) m = wmax[i] > m ? wmax[i] : m;
    atomicMax(dst, m);
  }
}

// max of two non-negative values (or NaN) through their bit patterns: NaN
// stays the maximum, as in the block reduction
__device__ __forceinline__ double fx_bitmax(double a, double b) {
  const unsigned long long x = (unsigned long long)__double_as_longlong(a);
  const unsigned long long y = (unsigned long long)__double_as_longlong(b);
  return __longlong_as_double((long long)(x > y ? x : y));
}

// The node update after the pull: moments, PostProcessing's inlet velocity
// (lbm.f90:186-191) and zero outlet pressure (lbm.f90:195-198), the range
// check, [Monitor: um takes the max with |(u_x, u_y)|], Collision, stores.
template <int DIM, bool MON, int FORM>
__device__ __forceinline__ void fx_node_finish(const long long (&F)[Lattice<DIM>::Q],
                                               const DevGrid& g, const CoefFix& c, const DevState& st,
                                               const DevPlanes& pl, uint32_t id, uint8_t m,
                                               double& um) {
  using NF = NodeFixed<DIM>;
  constexpr int Q = Lattice<DIM>::Q;
  long long J[DIM];
  long long S = NF::moments(F, J);
  if (m & kMaskInlet) {
    const int64_t r = DIM == 2 ? (int64_t)id / g.dy : (int64_t)id / g.dz;
    J[0] = fix_from_double(st.inlet[r]);
    J[1] = 0;
  }
  if (m & kMaskOutlet) S = 0;
  const bool ok = NF::in_range(F, S, J);
  if constexpr (MON) {
    if (id != g.skip_id) {
      const double ux = fix_to_double(J[0]), uy = fix_to_double(J[1]);
      um = fx_bitmax(um, ok ? sqrt(__dadd_rn(__dmul_rn(ux, ux), __dmul_rn(uy, uy)))
                            : __longlong_as_double(0x7ff8000000000000LL));
    }
  }
  if (ok) {
    auto store = [&](int i, long long v) { ((long long*)pl.out[i])[id] = v; };
    if constexpr (FORM == kFxAny) NF::collide_any(F, S, J, c.k, c.om1, store);
    else NF::template collide<FORM == kFxNeg>(F, S, J, c.kf, c.m, store);
  } else {
#pragma unroll
    for (int i = 0; i < Q; ++i) ((long long*)pl.out[i])[id] = kFixInvalid;
  }
}

// The general pull of one fluid cell (closed forms of its boundary bits, or
// its record's source row), the node update, and the record's push copies.
template <int DIM, bool MON, int FORM>
__device__ __forceinline__ void fx_node_general(const DevGrid& g, const CoefFix& c,
                                                const DevState& st, const DevPlanes& pl,
                                                uint32_t id, uint8_t m, const PullFix& fx,
                                                double& um) {
  using L = Lattice<DIM>;
  constexpr int Q = L::Q;
  long long F[Q];
  const long long* fin = (const long long*)pl.in[0] + g.off[0];
  long long* fout = (long long*)pl.out[0];
  if (!fx.record()) {
    sfor<0, Q>([&](auto I) {
      constexpr int i = I;
      bool opp;
      int64_t sh;
      fx.form<DIM>(L::ex(i), L::ey(i), L::ez(i), g.off[i], st.pshift, opp, sh);
      const long long* base = (const long long*)(opp ? pl.in[Q - 1 - i] : pl.in[i]);
      F[I] = base[(uint32_t)(id + (uint32_t)sh)];
    });
  } else {
    const uint32_t* row = PullFix::row<Q>(st, id);
    sfor<0, Q>([&](auto I) {
      const uint32_t r = row[I];
      F[I] = r != kNoRedirect ? fin[r] : ((const long long*)pl.in[I])[id];
    });
  }
  fx_node_finish<DIM, MON, FORM>(F, g, c, st, pl, id, m, um);
  if (fx.record()) push_copies(st.push, PullFix::row<Q>(st, id)[Q], fin, fout);
}

template <int DIM, bool MON, int FORM>
__global__ void __launch_bounds__(kBlockFx, (kFxBlocks<DIM, FORM>)) k_step_fx(DevGrid g, CoefFix c, DevState st,
                                                      DevPlanes pl, unsigned long long* monitor) {
  using L = Lattice<DIM>;
  constexpr int Q = L::Q;
  const uint32_t id = (uint32_t)(g.id_lo + (int64_t)pl.block() * kBlockFx + threadIdx.x);
  double um = 0.0;
  const uint8_t m = (int64_t)id < g.id_hi ? st.mask[id] : (uint8_t)0;
  const PullFix fx = PullFix::make(st, (m & kMaskFluid) ? m : (uint8_t)0);
  const bool bwarp = __any_sync(0xffffffffu, fx.other());
  if (m & kMaskFluid) {
    if (!bwarp) {
      long long F[Q];
      const uint32_t id_in = id + fx.inl(), o = fx.outl();
      sfor<0, Q>([&](auto I) {
        constexpr int ex = L::ex(I);
        const uint32_t a = ex == 1 ? id_in : (ex == -1 ? id + o * (uint32_t)g.off[I] : id);
        F[I] = ((const long long*)pl.in[I])[a];
      });
      fx_node_finish<DIM, MON, FORM>(F, g, c, st, pl, id, m, um);
    } else {
      fx_node_general<DIM, MON, FORM>(g, c, st, pl, id, m, fx, um);
    }
  }
  if constexpr (MON) block_max_fx(um, monitor);
}

}  // namespace

cudaError_t launch_step_fx(int dim, const DevGrid& g, const CoefFix& c, const DevState& st,
                           const DevPlanes& pl, unsigned long long* monitor, cudaStream_t s) {
  const unsigned grid = (unsigned)((g.id_hi - g.id_lo + kBlockFx - 1) / kBlockFx);
  // the lattices' own weights fail `own` only where ome t_i is no multiple of
  // 2^-63 (ome < 0.11), or with a caller's other weights
  const int form = !c.own ? kFxAny : (c.om1 < 0 ? kFxNeg : kFxPos);
#define F_(D, M, F) k_step_fx<D, M, F><<<grid, kBlockFx, 0, s>>>(g, c, st, pl, monitor)
#define L_(D, M)                                     \
  do {                                               \
    if (form == kFxAny) F_(D, M, kFxAny);            \
    else if (form == kFxPos) F_(D, M, kFxPos);       \
    else F_(D, M, kFxNeg);                           \
  } while (0)
  if (dim == 2) { if (monitor) L_(2, true); else L_(2, false); }
  else { if (monitor) L_(3, true); else L_(3, false); }
#undef L_
#undef F_
  return cudaGetLastError();
}

}  // namespace imx
