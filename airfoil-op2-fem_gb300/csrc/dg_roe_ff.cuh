// The Roe flux with its dissipation in pairs of single-precision numbers (host and device code).
//
// On GB300 an FP64 instruction holds its scheduler's FP64 pipe for 64 clocks per warp, a
// single-precision or integer one takes an issue slot of one, and the face kernels are bound by
// the FP64 pipe (roe_flux2: 96 FP64 instructions and three root / reciprocal sequences).  The
// dissipation |A| (qR - qL) needs the jumps exactly, but everything that multiplies them only to
// a relative accuracy of 2^-53 times flux / jump: where the jumps are below 2^-8 of the state, a
// pair (h, l) of floats with about 47 bits is enough to leave the flux's own FP64 rounding the
// larger error.  roe_flux2_small takes the four jumps in FP64, forms the Roe averages and the
// dissipation in pairs, and keeps in FP64 the two sides' fluxes and the final subtraction: 53
// FP64 instructions per face node instead of 109 (counted with the stores' scaling).
//
// Measured (stage launches alone, GB300): K = 32768 O-grid, N = 3 49.5 -> 28.5 us; K = 18990,
// N = 5 41 -> 26.6 us; K = 524288 square, N = 4 790 -> 404 us (FP64 floors at 109 and 53
// instructions: 34 / 17, 30 / 15 and 683 / 332 us).
//
// Accuracy.  Against 113-bit arithmetic, random states at Mach numbers to 0.1, 0.8 and 1.9, the
// components' errors at jumps up to the line, in units of 2^-53 of the flux's scale, rms (roe_flux2's
// in brackets): gamma = 1.4 0.11-0.77 (0.54-0.84), 0.28-0.52 (0.46-0.71), 0.43-0.59 (0.56-0.95); no
// component's rms is above roe_flux2's from gamma = 1.00001 to 8 (with the seeds below moved by a unit
// (reciprocal) or two (root) in the last place as the hardware's are).  Three things make it so:
//   - the seeds are refined to second order: with one correction e of 2^-22 cut at e^2, the roots
//     and reciprocals were known to 2^-44 only (momentum 1.04 rms at jumps up to the line);
//   - the halves of a dissipation component are joined in FP64 before they are subtracted, one
//     rounding at the flux's full size less (the pressure term added last would save another, but
//     takes 77 registers instead of 64: vortex steps of K = 2048 10 % and of K = 524288 2 % slower);
//   - the rule below measures jumps and Mach numbers by the sound speed, not by sqrt(E / rho), which
//     is far above it as gamma nears 1 (errors of 30 units there).
//
// roe_small_jump decides per face node, from the states alone (so every launch form gives a node
// the same path): jumps of rho, rho (u, v) and E below 2^-8 of rho, sqrt(g rho E) and E, both sides
// physical with |rho (u, v)|^2 below g rho E, g = min(1, 5 (gamma - 1) / 2) (at gamma = 1.4 a Mach
// number below 1.9, at 1.01 below 1.6), and magnitudes for which no float over- or underflows.
// Everything else (strong jumps, non-finite or non-physical states, extreme scales) takes roe_flux2.
//
// Pair arithmetic after Dekker, "A floating-point technique for extending the available
// precision", Numer. Math. 18 (1971), the sums by Knuth's six-operation form (The Art of Computer
// Programming, vol. 2, 4.2.2), with fused multiply-adds for the product's error.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define DG_HD __host__ __device__ __forceinline__
#else
#define DG_HD inline
#endif

namespace dg {

struct ff {
  float h, l;
};

// Rounded single operations: written out so that neither compiler contracts or reorders them.
DG_HD float ff_mulf(const float a, const float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rn(a, b);
#else
  return a * b;
#endif
}
DG_HD float ff_addf(const float a, const float b) {
#ifdef __CUDA_ARCH__
  return __fadd_rn(a, b);
#else
  return a + b;
#endif
}
DG_HD float ff_fmaf(const float a, const float b, const float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}
// Approximate reciprocal and reciprocal square root of normal numbers (the hardware's, good to a
// few units in the last place; the callers correct them).
DG_HD float ff_rcpf(const float a) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
  return y;
#else
  return 1.0f / a;
#endif
}
DG_HD float ff_rsqrtf(const float a) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
  return y;
#else
  return 1.0f / std::sqrt(a);
#endif
}
DG_HD uint64_t dbl_bits(const double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, sizeof b);
  return b;
#endif
}
DG_HD double bits_dbl(const uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  std::memcpy(&x, &b, sizeof x);
  return x;
#endif
}
DG_HD uint32_t flt_bits(const float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  uint32_t b;
  std::memcpy(&b, &x, sizeof b);
  return b;
#endif
}
DG_HD float bits_flt(const uint32_t b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float x;
  std::memcpy(&x, &b, sizeof x);
  return x;
#endif
}

// h + l with |l| small against |h|, renormalised so that h is the rounded sum.
DG_HD ff ff_norm(const float h, const float l) {
  const float s = ff_addf(h, l);
  return ff{s, ff_addf(l, -ff_addf(s, -h))};
}
DG_HD ff ff_mul(const ff a, const ff b) {
  const float p = ff_mulf(a.h, b.h);
  float e = ff_fmaf(a.h, b.h, -p);
  e = ff_fmaf(a.h, b.l, e);
  e = ff_fmaf(a.l, b.h, e);
  return ff_norm(p, e);
}
DG_HD ff ff_add(const ff a, const ff b) {
  const float s = ff_addf(a.h, b.h);
  const float t = ff_addf(s, -a.h);
  const float e = ff_addf(ff_addf(a.h, -ff_addf(s, -t)), ff_addf(b.h, -t));
  return ff_norm(s, ff_addf(e, ff_addf(a.l, b.l)));
}
DG_HD ff ff_neg(const ff a) { return ff{-a.h, -a.l}; }
DG_HD ff ff_sub(const ff a, const ff b) { return ff_add(a, ff_neg(b)); }
// a * b + c
DG_HD ff ff_fma(const ff a, const ff b, const ff c) {
  const float p = ff_mulf(a.h, b.h);
  float e = ff_fmaf(a.h, b.h, -p);
  e = ff_fmaf(a.h, b.l, e);
  e = ff_fmaf(a.l, b.h, e);
  const float s = ff_addf(p, c.h);
  const float t = ff_addf(s, -p);
  const float d = ff_addf(ff_addf(p, -ff_addf(s, -t)), ff_addf(c.h, -t));
  return ff_norm(s, ff_addf(d, ff_addf(e, c.l)));
}
DG_HD ff ff_half(const ff a) { return ff{ff_mulf(0.5f, a.h), ff_mulf(0.5f, a.l)}; }
// 1 / a, from a single-precision reciprocal y: y (1 + e + e^2), e = 1 - a y by fused multiply-adds
DG_HD ff ff_rcp(const ff a) {
  const float y = ff_rcpf(a.h);
  const float e = ff_fmaf(-a.l, y, ff_fmaf(-a.h, y, 1.0f));
  return ff_norm(y, ff_mulf(y, ff_fmaf(e, e, e)));
}
// sqrt(a) for a > 0: y ~ 1 / sqrt(a) after one Newton step in single precision, s = a y, corrected
// by (a - s^2) y / 2
DG_HD ff ff_sqrt(const ff a) {
  const float y0 = ff_rsqrtf(a.h), s0 = ff_mulf(a.h, y0);
  const float y = ff_fmaf(ff_mulf(0.5f, y0), ff_fmaf(-s0, y0, 1.0f), y0);
  const float s = ff_mulf(a.h, y);
  const float r = ff_addf(ff_fmaf(-s, s, a.h), a.l);
  return ff_norm(s, ff_mulf(ff_mulf(0.5f, y), r));
}

// A double as a pair, with integer instructions and one float subtraction: h takes the leading 24
// bits of the significand, l the next 23 (the last 6 are cut: 2^-47).  |x| must be below 2^100;
// below 2^-100 it becomes 0.
DG_HD ff ff_from(const double x) {
  const uint64_t b = dbl_bits(x);
  const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b, a = hi & 0x7FFFFFFFu;
  const uint32_t m = ((a - (896u << 20)) << 3) | (lo >> 29);
  const uint32_t fh = (hi & 0x80000000u) | m;
  const uint32_t base = (fh & 0xFF800000u) - (23u << 23);
  const float l = ff_addf(bits_flt(base | ((lo >> 6) & 0x7FFFFFu)), -bits_flt(base));
  const bool z = a < ((1023u - 100u) << 20);
  return ff{z ? 0.0f : bits_flt(fh), z ? 0.0f : l};
}
// The leading 24 bits alone, as above.
DG_HD float ff_lead(const double x) {
  const uint64_t b = dbl_bits(x);
  const uint32_t hi = (uint32_t)(b >> 32), a = hi & 0x7FFFFFFFu;
  const uint32_t m = ((a - (896u << 20)) << 3) | ((uint32_t)b >> 29);
  return a < ((1023u - 100u) << 20) ? 0.0f : bits_flt((hi & 0x80000000u) | m);
}
// A float as a double (integer instructions; subnormal floats become 0)
DG_HD double dbl_from(const float v) {
  const uint32_t b = flt_bits(v), a = b & 0x7FFFFFFFu;
  const uint32_t hi = (b & 0x80000000u) | ((a >> 3) + (896u << 20));
  const uint64_t r = ((uint64_t)hi << 32) | (uint32_t)(a << 29);
  return bits_dbl(a < 0x00800000u ? 0ull : r);
}

// 1 / x from a float seed y by one step of Householder's third-order iteration (The Numerical Treatment of a
// Single Nonlinear Equation, 1970): y (1 + e + e^2), e = 1 - x y.  x cut to 24 bits and a seed good to a
// unit in its last place leave |e| < 2^-22, so the cut e^3 and the roundings of e and e + e^2 are below
// 2^-65 and the one rounding that counts is the last: within 0.5 + 2^-12 units in the last place, the
// correctly rounded reciprocal but for about one argument in four thousand.  Three FP64
// instructions; __drcp_rn takes five and is used outside 2^-100 .. 2^100 (zero, non-finite values among
// the rest).
DG_HD double rcp_seeded(const double x) {
  const uint32_t a = (uint32_t)(dbl_bits(x) >> 32) & 0x7FFFFFFFu;
  if (a - ((1023u - 100u) << 20) >= (200u << 20)) {
#ifdef __CUDA_ARCH__
    return __drcp_rn(x);
#else
    return 1.0 / x;
#endif
  }
  const double y0 = dbl_from(ff_rcpf(ff_lead(x)));
  const double e = fma(-x, y0, 1.0);
  return fma(y0, fma(e, e, e), y0);
}

// Largest relative jump that takes the pair path.
constexpr float kRoeJump = 0.00390625f;  // 2^-8

// Whether roe_flux2_small may take this face node (see the head of this file); gm1: gamma - 1.  Written in
// single rounded operations, so that every kernel decides alike.
DG_HD bool roe_small_jump(const double qm[4], const double qp[4], const float gm1) {
  // rho and E of both sides positive, in 2^-30 .. 2^30; momenta below 2^60 (the float squares
  // below stay finite, the conversions in range)
  const uint32_t lim = 60u << 20, off = (1023u - 30u) << 20;
  auto hw = [](const double x) { return (uint32_t)(dbl_bits(x) >> 32); };
  const uint32_t r0 = hw(qm[0]) - off, r1 = hw(qp[0]) - off, r2 = hw(qm[3]) - off, r3 = hw(qp[3]) - off;
  const uint32_t m0 = hw(qm[1]) & 0x7FFFFFFFu, m1 = hw(qm[2]) & 0x7FFFFFFFu, m2 = hw(qp[1]) & 0x7FFFFFFFu,
                 m3 = hw(qp[2]) & 0x7FFFFFFFu;
  const uint32_t mlim = (1023u + 60u) << 20;
  if (!((r0 < lim) & (r1 < lim) & (r2 < lim) & (r3 < lim) & (m0 < mlim) & (m1 < mlim) & (m2 < mlim) & (m3 < mlim)))
    return false;
  const float rL = ff_lead(qm[0]), aL = ff_lead(qm[1]), bL = ff_lead(qm[2]), eL = ff_lead(qm[3]);
  const float rR = ff_lead(qp[0]), aR = ff_lead(qp[1]), bR = ff_lead(qp[2]), eR = ff_lead(qp[3]);
  const float rmin = rL < rR ? rL : rR, emin = eL < eR ? eL : eR;
  const float dr = std::fabs(ff_addf(rL, -rR)), de = std::fabs(ff_addf(eL, -eR)), da = ff_addf(aL, -aR),
              db = ff_addf(bL, -bR);
  const float g25 = ff_mulf(2.5f, gm1), g = g25 < 1.0f ? g25 : 1.0f;
  const float jm = ff_mulf(kRoeJump * kRoeJump, ff_mulf(g, ff_mulf(rmin, emin)));
  return (dr <= ff_mulf(kRoeJump, rmin)) & (de <= ff_mulf(kRoeJump, emin)) &
         (ff_fmaf(da, da, ff_mulf(db, db)) <= jm) &
         (ff_fmaf(aL, aL, ff_mulf(bL, bL)) <= ff_mulf(g, ff_mulf(rL, eL))) &
         (ff_fmaf(aR, aR, ff_mulf(bR, bR)) <= ff_mulf(g, ff_mulf(rR, eR)));
}

// Twice the Roe flux (as roe_flux2) of a face node that roe_small_jump accepts.  gm1, gf: gamma - 1
// as a double and as a pair.
//
// Dissipation from the conservative jumps D = qR - qL and the Roe averages (u, v), H, with
// un = n . (u, v) and q2 = u^2 + v^2 (the identities rho du = D(rho u) - u D rho and
// dp = (gamma - 1) (D E - u . D(rho u) + q2 D rho / 2) hold exactly for Roe's averages):
//   w = D(rho u) - (u, v) D rho,  du = n . w (= rho d un),  s = w - n du (= t rho d ut)
//   P = dp / c^2 = (D E - (u, v) . w - q2 D rho / 2) / (H - q2 / 2),  U = du / c
//   (|un - c| + |un + c|) / 2 = S = max(|un|, c),  (|un + c| - |un - c|) / 2 = T = sign(un) min(|un|, c)
//   d14 = S P + T U,  ce = c (T P + S U),  W2 = |un| (D rho - P)
//   d = (d14 + W2,  (u, v) (d14 + W2) + n ce + |un| s,  H d14 + un ce + q2 W2 + |un| (u, v) . s)
// (src/euler_rhs.h:181-208; its energy term takes W2 with u^2 + v^2, not half of it).
DG_HD void roe_flux2_small(const double qm[4], const double qp[4], const double nx, const double ny,
                           const double gm1, const ff gf, double f2[4]) {
  // jumps, exact or rounded in FP64
  const ff dr = ff_from(qp[0] - qm[0]), da = ff_from(qp[1] - qm[1]), db = ff_from(qp[2] - qm[2]),
           de = ff_from(qp[3] - qm[3]);
  const ff rL = ff_from(qm[0]), rR = ff_from(qp[0]);
  // 1 / rho of both sides from one reciprocal of the product (in 2^-60 .. 2^60; as rcp_seeded)
  const double x = qm[0] * qp[0];
  const double y0 = dbl_from(ff_rcpf(ff_lead(x)));
  const double e0 = fma(-x, y0, 1.0);
  const double y = fma(y0, fma(e0, e0, e0), y0);
  const double irL = qp[0] * y, irR = qm[0] * y;
  // the two sides' fluxes along n, in FP64
  const double mL = fma(nx, qm[1], ny * qm[2]), mR = fma(nx, qp[1], ny * qp[2]);
  const double uL = mL * irL, uR = mR * irR;
  const double kL = fma(-0.5, fma(qm[1], qm[1], qm[2] * qm[2]) * irL, qm[3]);  // p / (gamma - 1)
  const double kR = fma(-0.5, fma(qp[1], qp[1], qp[2] * qp[2]) * irR, qp[3]);
  const double EL = fma(gm1, kL, qm[3]), ER = fma(gm1, kR, qp[3]);  // E + p
  const double ps = fma(gm1, kL, gm1 * kR);
  const double f0 = mL + mR, f1 = fma(nx, ps, fma(qm[1], uL, qp[1] * uR)), f2y = fma(ny, ps, fma(qm[2], uL, qp[2] * uR)),
               f3 = fma(uL, EL, uR * ER);
  // Roe averages in pairs: x = wL (rho x)_L + wR (rho x)_R, wL = 1 / (rho_L + g), wR = 1 / (rho_R + g),
  // g = sqrt(rho_L rho_R)
  const ff g = ff_sqrt(ff_mul(rL, rR));
  const ff wL = ff_rcp(ff_add(rL, g)), wR = ff_rcp(ff_add(rR, g));
  const ff u = ff_fma(wL, ff_from(qm[1]), ff_mul(wR, ff_from(qp[1])));
  const ff v = ff_fma(wL, ff_from(qm[2]), ff_mul(wR, ff_from(qp[2])));
  const ff H = ff_fma(wL, ff_from(EL), ff_mul(wR, ff_from(ER)));
  const ff nxf = ff_from(nx), nyf = ff_from(ny);
  const ff q2 = ff_fma(u, u, ff_mul(v, v));
  const ff hh = ff_sub(H, ff_half(q2));  // c^2 / (gamma - 1)
  const ff c = ff_sqrt(ff_mul(gf, hh));
  const ff un = ff_fma(nxf, u, ff_mul(nyf, v));
  // the jumps' components
  const ff ndr = ff_neg(dr);
  const ff wa = ff_fma(ndr, u, da), wb = ff_fma(ndr, v, db);
  const ff du = ff_fma(nxf, wa, ff_mul(nyf, wb));
  const ff ndu = ff_neg(du);
  const ff sa = ff_fma(ndu, nxf, wa), sb = ff_fma(ndu, nyf, wb);
  const ff k = ff_fma(u, wa, ff_mul(v, wb));
  const ff us = ff_fma(ndu, un, k);  // (u, v) . s
  const ff P = ff_mul(ff_sub(ff_fma(ndr, ff_half(q2), de), k), ff_rcp(hh));
  const ff U = ff_mul(du, ff_rcp(c));
  const bool neg = un.h < 0.0f;
  const ff au = neg ? ff_neg(un) : un;
  const bool sub = au.h < c.h;
  const ff S = sub ? c : au, T = sub ? un : (neg ? ff_neg(c) : c);
  const ff d14 = ff_fma(S, P, ff_mul(T, U));
  const ff ce = ff_mul(c, ff_fma(T, P, ff_mul(S, U)));
  const ff W2 = ff_mul(au, ff_sub(dr, P));
  const ff d0 = ff_add(d14, W2);
  const ff d1 = ff_fma(u, d0, ff_fma(nxf, ce, ff_mul(au, sa)));
  const ff d2 = ff_fma(v, d0, ff_fma(nyf, ce, ff_mul(au, sb)));
  const ff d3 = ff_fma(H, d14, ff_fma(un, ce, ff_fma(q2, W2, ff_mul(au, us))));
  f2[0] = f0 - (dbl_from(d0.h) + dbl_from(d0.l));
  f2[1] = f1 - (dbl_from(d1.h) + dbl_from(d1.l));
  f2[2] = f2y - (dbl_from(d2.h) + dbl_from(d2.l));
  f2[3] = f3 - (dbl_from(d3.h) + dbl_from(d3.l));
}

}  // namespace dg
