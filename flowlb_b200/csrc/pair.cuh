// pair.cuh -- two cells at a time with packed FP32 arithmetic (f32x2).  Each
// half of a packed operation rounds as the scalar one does, so the results
// are those of collide_fused / collide_fused_dev bit for bit; an instruction
// slot does two cells' work (same FP32 rate, half the issue slots: measured on
// a B200, 37.0 T lane operations per second either way).  both() of a literal
// or of a scalar kernel parameter costs no instruction: the packed operations
// take it as an operand (measured: 64 of them issue 64 instructions; with the
// pair stored as a 64-bit parameter, 80).
#pragma once

#include "common.cuh"

namespace flb {

struct f2 {
  unsigned long long v;
};
__device__ __forceinline__ f2 pack(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float lo(f2 a) { return __uint_as_float((uint32_t)a.v); }
__device__ __forceinline__ float hi(f2 a) { return __uint_as_float((uint32_t)(a.v >> 32)); }
__device__ __forceinline__ f2 both(float a) { return pack(a, a); }
__device__ __forceinline__ f2 operator+(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 operator-(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 operator*(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 fmac(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ f2 ld_pair(const float* q) {
  f2 r;
  r.v = *reinterpret_cast<const unsigned long long*>(q);
  return r;
}
__device__ __forceinline__ void st_pair(float* q, f2 a) { *reinterpret_cast<unsigned long long*>(q) = a.v; }

// -1/x of both halves, each the correctly rounded quotient (the negative of
// what __frcp_rn returns).  x away from the ends of the exponent range: the hardware's
// approximation and one Newton step with the residual taken in a fused
// multiply-add (Markstein, IBM J. Res. Dev. 34, 1990).  His theorem has the step
// round the quotient correctly if the starting value is within an ulp of it and
// the significand of x is not all ones; that the approximation serves, and for
// those x too, is tested against __frcp_rn for every float in either half
// (tests/test_gpu_pair_rcp.py).  Otherwise __frcp_rn itself.
__device__ __forceinline__ f2 neg_rcp(f2 x) {
  // biased exponents in [2, 251]: neither x nor 1/x is subnormal, zero, infinite or NaN
  const uint32_t ea = __float_as_uint(lo(x)) << 1, eb = __float_as_uint(hi(x)) << 1;
  if (ea - 0x02000000u < 0xfa000000u && eb - 0x02000000u < 0xfa000000u) {
    float ya, yb;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ya) : "f"(-lo(x)));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yb) : "f"(-hi(x)));
    const f2 y = pack(ya, yb);
    return fmac(fmac(x, y, both(1.0f)), y, y);
  }
  return pack(-__frcp_rn(lo(x)), -__frcp_rn(hi(x)));
}

struct PairMacro {
  f2 rho, ux, uy;
};

// moments_fused and collide_fused (lattice.cuh), operation by operation.
__device__ __forceinline__ PairMacro collide_fused_pair(f2* f, const KParams& p) {
  const f2 s12 = f[1] + f[2], s34 = f[3] + f[4], s56 = f[5] + f[6], s78 = f[7] + f[8];
  // the momentum and 1 / rho negated (the products are the same)
  const f2 d12 = f[2] - f[1], d34 = f[4] - f[3], d56 = f[6] - f[5], d78 = f[8] - f[7];
  PairMacro m;
  m.rho = ((f[0] + s12) + (s34 + s56)) + s78;
  const f2 jx = (d12 + d56) + d78, jy = (d34 + d56) - d78;
  const f2 inv = neg_rcp(m.rho);
  f2 ux = fmac(both(p.fu_nhfx), inv, jx * inv), uy = fmac(both(p.fu_nhfy), inv, jy * inv);
  if (p.u_max > 0.0f) {
    float ax = lo(ux), ay = lo(uy), bx = hi(ux), by = hi(uy);
    limit_u(p.u_max, ax, ay);
    limit_u(p.u_max, bx, by);
    ux = pack(ax, bx);
    uy = pack(ay, by);
  }
  m.ux = ux;
  m.uy = uy;
  const f2 usq = fmac(ux, ux, uy * uy);
  const f2 uF = fmac(ux, both(p.fu_fx), uy * both(p.fu_fy));
  const f2 A = both(p.inv_tau) * m.rho;
  const f2 t1 = fmac(both(-1.5f), usq, both(1.0f));
  const f2 B = fmac(A, t1, both(p.fu_nk3) * uF);
  const f2 A3 = both(3.0f) * A, A45 = both(4.5f) * A;
  f[0] = fmac(both(p.fu_omc), f[0], both(wgt<float>(0)) * B);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int i = 2 * q + 1;
    const f2 cu = q == 0 ? ux : (q == 1 ? uy : (q == 2 ? ux + uy : ux - uy));
    const f2 E = fmac(cu, fmac(A45, cu, both(p.fu_h[q])), B);
    const f2 O = fmac(A3, cu, both(p.fu_g[q]));
    const f2 wi = both(wgt<float>(i));
    f[i] = fmac(both(p.fu_omc), f[i], wi * (E + O));
    f[i + 1] = fmac(both(p.fu_omc), f[i + 1], wi * (E - O));
  }
  return m;
}

// collide_fused_dev (lattice.cuh), operation by operation.
template <bool LIM>
__device__ __forceinline__ PairMacro collide_fused_dev_pair(f2* h, const KParams& p) {
  const f2 s12 = h[1] + h[2], s34 = h[3] + h[4], s56 = h[5] + h[6], s78 = h[7] + h[8];
  const f2 d12 = h[2] - h[1], d34 = h[4] - h[3], d56 = h[6] - h[5], d78 = h[8] - h[7];
  const f2 dS = ((h[0] + s12) + (s34 + s56)) + s78;
  const f2 jx = (d12 + d56) + d78, jy = (d34 + d56) - d78;
  const f2 invS = both(p.f16_inv);
  const f2 delta = dS * invS;
  PairMacro m;
  m.rho = fmac(dS, invS, both(1.0f));
  const f2 inv = neg_rcp(m.rho);
  const f2 invs = inv * invS;
  f2 ux = fmac(both(p.fu_nhfx), inv, jx * invs), uy = fmac(both(p.fu_nhfy), inv, jy * invs);
  if (LIM) {
    float ax = lo(ux), ay = lo(uy), bx = hi(ux), by = hi(uy);
    limit_u(p.u_max, ax, ay);
    limit_u(p.u_max, bx, by);
    ux = pack(ax, bx);
    uy = pack(ay, by);
  }
  m.ux = ux;
  m.uy = uy;
  const f2 usq = fmac(ux, ux, uy * uy);
  const f2 uF = fmac(ux, both(p.fu_fx), uy * both(p.fu_fy));
  const f2 A = both(p.inv_tau) * m.rho;
  const f2 t1 = fmac(both(-1.5f), usq, both(1.0f));
  const f2 x = fmac(delta, t1, both(-1.5f) * usq);
  const f2 Bd = fmac(both(p.inv_tau), x, both(p.fu_nk3) * uF);
  const f2 A3 = both(3.0f) * A, A45 = both(4.5f) * A;
  h[0] = fmac(both(p.fu_omc), h[0], both(p.fu_sw[0]) * Bd);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int i = 2 * q + 1;
    const f2 cu = q == 0 ? ux : (q == 1 ? uy : (q == 2 ? ux + uy : ux - uy));
    const f2 E = fmac(cu, fmac(A45, cu, both(p.fu_h[q])), Bd);
    const f2 O = fmac(A3, cu, both(p.fu_g[q]));
    const f2 swi = both(p.fu_sw[q < 2 ? 1 : 2]);
    h[i] = fmac(both(p.fu_omc), h[i], swi * (E + O));
    h[i + 1] = fmac(both(p.fu_omc), h[i + 1], swi * (E - O));
  }
  return m;
}

}  // namespace flb
