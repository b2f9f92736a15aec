// tor_warp_dd.cuh -- double-word pieces of the torontonian's double-double walk
// (tor_rec.cuh) and the radius of its certified tier.
//
// Pivot reciprocals 1 / sqrt(s) are one Newton step from the binary64 rsqrt seed:
// y = y0 + y0 (1 - s y0^2) / 2 in double-word.  The diagonal 1 - O_ii is formed
// exactly (TwoSum), so M enters the walk without rounding.
//
// Certified double-double tier (kTierCertDD): the same walk (the value equals the
// dd tier's bit for bit) with the a-posteriori radius of tor_warp.cuh re-derived for
// double-word operations.  Per-operation relative error bounds (u = 2^-53):
//   dd_add (the accurate double-word sum, Joldes-Muller-Popescu 2017, Alg. 6): 3u^2;
//   dd_mul (TwoProd of the heads, both cross terms by FMA into the tail, Fast2Sum):
//     error = xl*yh*d3 + (xh*yl + e1)(d2 + d3 + d2*d3) - xl*yl, at most 6u^2 + O(u^3)
//     relative (|xl| <= u|xh|, |yl| <= u|yh|, |e1| <= u|xh*yh|); charged 7u^2;
//   dd_mul_d: 2u^2 + O(u^3), charged 3u^2;
//   dd_rsqrt: the Newton step leaves (3/2) e0^2 of the seed's relative error e0 <= 4u
//     (rsqrt taken as 2 ulp) plus the roundings of its four operations: charged 40u^2.
// Every factor entry is an inner product of <= m terms, each a dd_mul and a dd_add,
// plus one scaling; the diagonal carries (1 + 40u^2)^2 from the pivot reciprocal:
// gamma_{2m+20}(7u^2) covers all of it, the last block's determinant (two products, one
// sum) included.  With sigma from the same binary64 eigenvalue
// proof, rho_m follows as in tor_warp.cuh but evaluated as small quantities (1 + rho
// is not representable in binary64): tor_cert_rho_dd.
#pragma once

#include "gbs_common.cuh"
#include "tor_warp.cuh"

namespace gbsb {

// entry of M = I - O as a double-word (the diagonal 1 - O_ii exact by TwoSum)
__device__ __forceinline__ dd tor_m_dd(const double* __restrict__ Oc, int dim, int a, int b) {
  const double o = Oc[2 * (a * dim + b)];
  return a == b ? dd_add_d(dd_make(1.0), -o) : dd_make(-o);
}

__device__ __forceinline__ dd ld_dd(const double* p) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  return dd{v.x, v.y};
}
__device__ __forceinline__ void st_dd(double* p, dd v) { *reinterpret_cast<double2*>(p) = make_double2(v.hi, v.lo); }
// a - b c
__device__ __forceinline__ dd dd_fms(dd a, dd b, dd c) { return dd_sub(a, dd_mul(b, c)); }
// 1 / sqrt(s), s > 0: binary64 seed, one Newton step in double-word
__device__ __forceinline__ dd dd_rsqrt(dd s) {
  const double y0 = rsqrt(s.hi);
  const dd t = dd_mul_d(dd_mul_d(s, y0), y0);  // s y0^2
  const dd r = dd_sub(dd_make(1.0), t);       // 1 - s y0^2 (small)
  return dd_add(dd_make(y0), dd_mul_d(r, 0.5 * y0));
}
// rho_m for m = 0..2k in double-double (see the header): all terms are small, so the
// bound is assembled as small quantities in upward rounding,
//   Up - 1 <= x + y + x y,  x = (gp + m eta) / (2 (1 - m eta)),  y = (m er + er) / (1 - m er - er)
//   1 - Lo <= z/2 + z^2/2 + m er + er,  z = gp + m eta
// y covers the product of the t's too: (m + 1) 40u^2 against m 7u^2 + 45u^2.
// (sqrt(1 + w) <= 1 + w/2; sqrt(1 - w) >= 1 - w/2 - w^2/2 for w <= 1/2).
static __device__ __noinline__ void tor_cert_rho_dd(double sigma, double dmin2, int k, double* rho, int lane) {
  const double u2 = 7.0 * kU * kU;
  const double er = 40.0 * kU * kU;
  for (int m = lane; m <= 2 * k; m += 32) {
    double out;
    if (m == 0) {
      out = 0.0;
    } else if (!(sigma > 0.0) || !(dmin2 > 0.0)) {
      out = INFINITY;
    } else {
      const double md = (double)m;
      const double g = gamma_ru(2.0 * md + 20.0, u2);
      double cm = ru_div(g, rd_sub(1.0, g));
      cm = ru_div(cm, __dmul_rd(rd_sub(1.0, kU), rd_sub(1.0, kU)));
      cm = ru_add(cm, ru_div(ru_mul(2.0 * md + 16.0, 16.0 * kUfl), dmin2));
      const double meta = ru_mul(md, ru_div(ru_mul(md, cm), sigma));
      const double gp = gamma_ru(md + 1.0, u2);
      const double mer = ru_add(ru_mul(md, er), er);
      if (!(meta < 0.25) || !(mer < 0.25)) {
        out = INFINITY;
      } else {
        const double z = ru_add(gp, meta);
        const double x = ru_div(z, ru_mul(2.0, rd_sub(1.0, meta)));
        const double y = ru_div(mer, rd_sub(1.0, mer));
        const double up = ru_add(ru_add(x, y), ru_mul(x, y));
        const double lo = ru_add(ru_add(ru_mul(0.5, z), ru_mul(0.5, ru_mul(z, z))), mer);
        out = fmax(up, lo);
      }
    }
    rho[m] = out;
  }
  __syncwarp();
}

}  // namespace gbsb
