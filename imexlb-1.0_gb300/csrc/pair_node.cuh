// One D2Q9 step of two neighbouring cells by one thread (FP32, BF16 or FP16
// populations), with packed f32x2 arithmetic: per cell the rounded operations of
// NodeFast<2, float>. Shared by the single-lattice step (k_step_pair) and the
// batched one (k_step_batch_pair).
#pragma once

#include <cstdint>
#include <type_traits>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "boundary_fused.cuh"
#include "f32x2.cuh"
#include "kernels.h"
#include "lattice.h"
#include "node_fast.cuh"
#include "storage.cuh"

namespace imx {

// Two neighbouring values of a plane from an even element on (ld_early).
template <class T>
__device__ IMX_FI F2 ld_pair(const T* p) {
  if constexpr (sizeof(T) == 2) {
    unsigned v;
    asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p));
    float2 w;
    if constexpr (std::is_same<T, __half>::value) w = __half22float2(*(const __half2*)&v);
    else w = __bfloat1622float2(*(const __nv_bfloat162*)&v);
    return F2(w.x, w.y);
  } else {
    float a, b;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "l"(p));
    return F2(a, b);
  }
}

template <class T>
__device__ IMX_FI void st_pair(T* p, F2 v) {
  if constexpr (sizeof(T) == 2) {
    if constexpr (std::is_same<T, __half>::value) *(__half2*)p = __floats2half2_rn(v.lo(), v.hi());
    else *(__nv_bfloat162*)p = __floats2bfloat162_rn(v.lo(), v.hi());
  } else {
    *(float2*)p = make_float2(v.lo(), v.hi());
  }
}

// Cells id (even) and id + 1 of the lattice `c` (a class with st, k, N, dy,
// id_hi, off<I>(), in<I>(), fin(), fout() and out(i)); ODD: dy is odd. A word
// holds both cells' pulls of direction I where its offset e_x + dy e_y is even,
// and always both cells' stores: planes, their stride (plane_stride) and id are even. What no
// step writes is read before wait(); speed(cell, |u|) is called per fluid cell if MON.
template <class T, bool ODD, bool MON, class C, class W, class S>
__device__ IMX_FI void pair_update(const C& c, uint32_t id, W&& wait, S&& speed) {
  using N2 = NodeFast<2, F2>;
  using L = Lattice<2>;
  constexpr int Q = L::Q;
  const DevState& st = c.st;
  const bool in = id < c.id_hi;
  uint8_t ma = 0, mb = 0;
  if (in) {
    ma = st.mask[id];
    if (id + 1 < c.id_hi) mb = st.mask[id + 1];
  }
  const bool fla = (ma & kMaskFluid) != 0, flb = (mb & kMaskFluid) != 0;
  const PullFix xa = PullFix::make(st, fla ? ma : (uint8_t)0), xb = PullFix::make(st, flb ? mb : (uint8_t)0);
  // in a warp with a cell that is not plain: every cell's source slots (of a
  // plain one its own pulls), and the obstacle copies of its records
  const bool special = __any_sync(0xffffffffu, (xa.bits | xb.bits) != 0u);
  uint32_t sa[Q], sb[Q], wa = 0, wb = 0;
  if (special && in) {
    auto slots = [&](const PullFix& x, uint32_t cell, uint32_t (&s)[Q], uint32_t& w) {
      sfor<0, Q>([&](auto I) {
        constexpr int i = I;
        bool opp;
        int64_t sh;
        const int64_t o = c.template off<i>();
        x.form<2>(L::ex(i), L::ey(i), L::ez(i), o, st.pshift, opp, sh);
        const uint32_t n = (uint32_t)c.N, off = (uint32_t)o;
        s[I] = cell + (uint32_t)sh + (opp ? (uint32_t)(Q - 1 - i) * n + off : (uint32_t)i * n - off);
      });
      if (x.record()) {
        const uint32_t* row = PullFix::row<Q>(st, cell);
        w = row[Q];
        sfor<0, Q>([&](auto I) {
          const uint32_t r = row[I];
          s[I] = r != kNoRedirect ? r : s[I];
        });
      }
    };
    slots(xa, id, sa, wa);
    slots(xb, id + 1, sb, wb);
  }
  wait();
  const T* fin = c.fin();
  F2 f[Q];
  if (special) {
    if (in) sfor<0, Q>([&](auto I) { f[I] = F2(Store<T>::to_f(fin[sa[I]]), Store<T>::to_f(fin[sb[I]])); });
  } else if (in) {
    sfor<0, Q>([&](auto I) {
      constexpr int i = I;
      const T* p = c.template in<i>() + id;
      if constexpr (((L::ex(i) + (ODD ? L::ey(i) : 0)) & 1) == 0) {
        f[I] = ld_pair(p);
      } else {
        const T a = ld_early(p), b = ld_early(p + 1);
        f[I] = F2(Store<T>::to_f(a), Store<T>::to_f(b));
      }
    });
  }
  if (!(fla || flb)) return;
  CoefR<F2> c2;
  sfor<0, Q>([&](auto I) { c2.k[I] = F2(c.k.k[I]); });
  c2.om1 = F2(c.k.om1);
  c2.inv_rho0 = F2(c.k.inv_rho0);
  F2 u[2];
  F2 S3 = N2::moments(f, u, c2.inv_rho0);
  if (((ma | mb) & (kMaskInlet | kMaskOutlet)) != 0) {
    // PostProcessing's Dirichlet conditions per cell (NodeFast::dirichlet)
    float s3[2] = {S3.lo(), S3.hi()};
    float ua[2] = {u[0].lo(), u[1].lo()}, ub[2] = {u[0].hi(), u[1].hi()};
    auto cond = [&](uint8_t m, uint32_t cell, float& s, float (&v)[2]) {
      if (m & kMaskInlet) {
        v[0] = (float)st.inlet[cell / (uint32_t)c.dy];
        v[1] = 0.0f;
      }
      if (m & kMaskOutlet) s = 0.0f;
    };
    if (fla) cond(ma, id, s3[0], ua);
    if (flb) cond(mb, id + 1, s3[1], ub);
    S3 = F2(s3[0], s3[1]);
    u[0] = F2(ua[0], ub[0]);
    u[1] = F2(ua[1], ub[1]);
  }
  if constexpr (MON) {
    const F2 v = N2::speed(u);
    if (fla) speed(id, v.lo());
    if (flb) speed(id + 1, v.hi());
  }
  if (fla && flb) {
    N2::collide(f, S3, u, c2, [&](int i, F2 v) { st_pair(c.out(i) + id, v); });
  } else {
    N2::collide(f, S3, u, c2, [&](int i, F2 v) {
      c.out(i)[fla ? id : id + 1] = Store<T>::from_f(fla ? v.lo() : v.hi());
    });
  }
  if (wa & 0xffu) push_copies(st.push, wa, fin, c.fout());
  if (wb & 0xffu) push_copies(st.push, wb, fin, c.fout());
}

}  // namespace imx
