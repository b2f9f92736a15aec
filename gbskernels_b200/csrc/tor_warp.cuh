// tor_warp.cuh -- the certificate of the torontonian's binary64 walk (tor_rec.cuh), and
// the entries of M = I - O.
//
// tor(O) = sum_{S subset [k]} (-1)^(k-|S|) / sqrt(det((I - O)_S)); the walk factors every
// minor by Cholesky with 1 / L[j][j] = rsqrt(s_j) (s_j the pivot before the root), the last
// mode of a subset by its 2 x 2 determinant, and a term is the product of the reciprocal
// pivots.  CUDA documents double rsqrt to 1 ulp; the bound below assumes 2 ulp (relative
// error <= 4u), so it does not lean on the last ulp of that figure.
//
// Each term gets an a-posteriori radius.  Define L^_jj := 1 / rsqrt(s_j) (exact real).  For
// a subset of dimension m the computed factor then satisfies L^L^T = A + F with
// |F_ij| <= c_m D_i D_j (Cholesky backward error: each entry is an inner product of
// <= m fused terms and one scaling, the diagonal carries (1 + 4u)^2 from rsqrt, the last
// block's product Z_aa Z_bb one rounding, a change of Z_bb by at most u Z_bb <= u D_b^2, so
// gamma_{m+12} covers it; D_i = fl(sqrt(fl(1 - O_ii)))), hence det(L^)^2 =
// det(A) det(I + X) with ||X|| <= eta_m = m c_m / sigma, sigma a rigorous lower bound
// of lambda_min(D^-1 M D^-1) -- valid for every principal submatrix by Cauchy
// interlacing, so ONE bound per instance certifies all 2^k subsets.  sigma is proved
// per instance by a binary64 Cholesky of D^-1 M D^-1 - sigma I that succeeds (success
// implies lambda_min >= -g tr / (1 - g), g = gamma_{2k+10}; Weyl for the rounding of
// the scaled matrix), at a sigma guessed by inverse iteration.  The term radius is
// |t^| rho_m (tor_cert_rho).
#pragma once

#include "cert.cuh"
#include "gbs_common.cuh"

namespace gbsb {

__device__ __forceinline__ double tor_m(const double* __restrict__ Oc, int dim, int a, int b) {
  // entry of M = I - O from the complex-interleaved input (real part)
  const double o = Oc[2 * (a * dim + b)];
  return a == b ? 1.0 - o : -o;
}

// ------------------------------------------------------------ certified prologue
// Rigorous lower bound sigma of lambda_min(D^-1 M D^-1), D_i = fl(sqrt(fl(1 - O_ii))),
// for the whole 2k x 2k matrix; <= 0 when none could be proved.  Also returns a lower
// bound of min D_i^2 for the underflow term.  Scratch (warp-private shared memory):
// the packed lower (2k)(2k+1)/2 matrix at S, then 2k scalings.
//   H^_ij = fl(fl(m_ij * fl(1/D_i)) * fl(1/D_j)) is within gamma_5 |h_ij| of the exact
//   scaled entry, so ||H^ - H||_2 <= ||H^ - H||_F <= gamma_5 / (1 - gamma_5) ||H^||_F.
//   A binary64 Cholesky of B = fl(H^ - s I) that completes proves lambda_min(B) >=
//   -g tr(B) / (1 - g), g = gamma_{2k+10} (backward error of the factorisation, the
//   rsqrt pivots included); with the rounding of the diagonal shift (u sum |b_ii|),
//   lambda_min(H) >= s - g tr / (1 - g) - ||E||.
//   The trial shift comes from inverse iteration with the factor of H^ itself.
static __device__ __noinline__ double tor_cert_sigma(const double* __restrict__ Oc, int k, double* S, int lane, double& dmin2) {
  const int dim = 2 * k;
  const int np = dim * (dim + 1) / 2;
  double* dinv = S + np;
  double dm = 1e300;
  bool okd = true;
  for (int i = lane; i < dim; i += 32) {
    const double mii = 1.0 - Oc[2 * (i * dim + i)];
    if (!(mii > 0.0)) okd = false;
    const double di = mii > 0.0 ? sqrt(mii) : 1.0;
    dinv[i] = 1.0 / di;
    dm = fmin(dm, __dmul_rd(di, di));
  }
  okd = __all_sync(0xffffffffu, okd);
#pragma unroll
  for (int mm = 16; mm > 0; mm >>= 1) dm = fmin(dm, shfl_xor_d(dm, mm));
  dmin2 = dm;
  __syncwarp();
  if (!okd) return -1.0;
  auto unpack = [&](int e, int& i, int& jj) {
    i = (int)((sqrt(8.0 * e + 1.0) - 1.0) * 0.5);
    while (i * (i + 1) / 2 > e) --i;
    while ((i + 1) * (i + 2) / 2 <= e) ++i;
    jj = e - i * (i + 1) / 2;
  };
  auto hval = [&](int i, int jj) { return (tor_m(Oc, dim, i, jj) * dinv[i]) * dinv[jj]; };
  double fro2 = 0.0;
  for (int e = lane; e < np; e += 32) {
    int i, jj;
    unpack(e, i, jj);
    const double h = hval(i, jj);
    fro2 = ru_fma(h, h, fro2);
    if (i != jj) fro2 = ru_fma(h, h, fro2);
  }
  fro2 = warp_sum_ru(fro2);
  const double g5 = gamma_ru(5.0, kU);
  const double eh = ru_mul(ru_div(g5, rd_sub(1.0, g5)), ru_sqrt(fro2));
  const double gm = gamma_ru((double)(dim + 10), kU);
  // factor B = fl(H^ - sig I) in place (right-looking, packed lower; the diagonal
  // slot of column j ends holding rsqrt of its pivot); on success return the proved
  // bound sig - tau - ||E||, else -1
  auto attempt = [&](double sig) -> double {
    double trace = 0.0;
    for (int e = lane; e < np; e += 32) {
      int i, jj;
      unpack(e, i, jj);
      double h = hval(i, jj);
      if (i == jj) {
        h = h - sig;
        trace = ru_add(trace, fabs(h));
      }
      S[e] = h;
    }
    trace = warp_sum_ru(trace);
    __syncwarp();
    for (int jc = 0; jc < dim; ++jc) {
      const double p = S[jc * (jc + 1) / 2 + jc];
      if (!(p > 0.0)) {  // warp-uniform (every lane read the same word)
        __syncwarp();
        return -1.0;
      }
      const double id = rsqrt(p);
      __syncwarp();
      if (lane == 0) S[jc * (jc + 1) / 2 + jc] = id;
      for (int i = jc + 1 + lane; i < dim; i += 32) S[i * (i + 1) / 2 + jc] *= id;
      __syncwarp();
      for (int i = jc + 1; i < dim; ++i) {
        const double lij = S[i * (i + 1) / 2 + jc];
        for (int l = jc + 1 + lane; l <= i; l += 32)
          S[i * (i + 1) / 2 + l] = fma(-lij, S[l * (l + 1) / 2 + jc], S[i * (i + 1) / 2 + l]);
      }
      __syncwarp();
    }
    const double tau = ru_div(ru_mul(gm, trace), rd_sub(1.0, gm));
    const double err = ru_add(eh, ru_mul(kUc, trace));
    return rd_sub(rd_sub(sig, tau), err);
  };
  if (attempt(0.0) < -0.5) return -1.0;  // H^ itself does not factor
  // inverse iteration x <- (L L^T)^{-1} x with the factor in S (slots x = lane, lane + 32)
  double x0 = lane < dim ? 1.0 + 0.01 * lane : 0.0;
  double x1 = lane + 32 < dim ? 1.0 + 0.01 * (lane + 32) : 0.0;
  double mu = 1.0;
  for (int it = 0; it < 5; ++it) {
    for (int j = 0; j < dim; ++j) {  // L y = x
      const double yj = __shfl_sync(0xffffffffu, (j >> 5) ? x1 : x0, j & 31) * S[j * (j + 1) / 2 + j];
      if (lane == (j & 31)) {
        if (j >> 5) x1 = yj;
        else x0 = yj;
      }
      if (lane > j && lane < dim) x0 = fma(-S[lane * (lane + 1) / 2 + j], yj, x0);
      if (lane + 32 > j && lane + 32 < dim) x1 = fma(-S[(lane + 32) * (lane + 33) / 2 + j], yj, x1);
    }
    for (int j = dim - 1; j >= 0; --j) {  // L^T z = y
      const double zj = __shfl_sync(0xffffffffu, (j >> 5) ? x1 : x0, j & 31) * S[j * (j + 1) / 2 + j];
      if (lane == (j & 31)) {
        if (j >> 5) x1 = zj;
        else x0 = zj;
      }
      const int r0 = j * (j + 1) / 2;
      if (lane < j) x0 = fma(-S[r0 + lane], zj, x0);
      if (lane + 32 < j) x1 = fma(-S[r0 + lane + 32], zj, x1);
    }
    double nn = x0 * x0 + x1 * x1;
#pragma unroll
    for (int mm = 16; mm > 0; mm >>= 1) nn += shfl_xor_d(nn, mm);
    mu = sqrt(nn);  // ~ 1 / lambda_min once converged (x had unit norm)
    if (!(mu > 0.0) || !isfinite(mu)) return -1.0;
    x0 /= mu;
    x1 /= mu;
  }
  const double est = 1.0 / mu;  // >= lambda_min(H^) up to rounding
  double best = -1.0;
  const double fr[6] = {0.9, 0.7, 0.45, 0.2, 0.05, 0.01};
  for (int t = 0; t < 6 && best <= 0.0; ++t) best = attempt(fr[t] * est);
  return best;
}

// rho_m for m = 0..2k (a-posteriori relative radius of one term of dimension m),
// written to rho[]; +inf where m * eta_m is not below 1/2.  e_r = 4u bounds the
// relative error of rsqrt (2 ulp).
//   c_m   = (g/(1-g) + u/(1-u)) / (1-u)^2 + (m+10) ufl / dmin2,  g = gamma_{m+12}
//   eta_m = m c_m / sigma,   gp = gamma_{m+1}
//   t^ is the product of the reciprocal pivots: at most m roundings, and for the last
//   mode one rsqrt (e_r) of a determinant with one rounding; charged, with room, as the
//   square root of a pivot product (gp) and m + 1 reciprocal roots of error e_r each
//   (m + 1 >= 3: (m + 1) 4u against the m u + 4.5u needed):
//   Up = sqrt((1+gp) / (1 - m eta)) / ((1 - m e_r)(1 - e_r))
//   Lo = sqrt((1-gp)(1 - m eta)) (1 - m e_r) / (1 + e_r)
//   and rho = max(Up - 1, 1 - Lo) bounds |t - t^| / |t^|.
static __device__ __noinline__ void tor_cert_rho(double sigma, double dmin2, int k, double* rho, int lane) {
  const double er = 4.0 * kU;
  for (int m = lane; m <= 2 * k; m += 32) {
    double out;
    if (m == 0) {
      out = 0.0;  // empty minor: t = 1 exactly
    } else if (!(sigma > 0.0) || !(dmin2 > 0.0)) {
      out = INFINITY;
    } else {
      const double md = (double)m;
      const double g = gamma_ru(md + 12.0, kU);
      double cm = ru_add(ru_div(g, rd_sub(1.0, g)), ru_div(kU, rd_sub(1.0, kU)));
      cm = ru_div(cm, __dmul_rd(rd_sub(1.0, kU), rd_sub(1.0, kU)));
      cm = ru_add(cm, ru_div(ru_mul(md + 10.0, kUfl), dmin2));
      const double eta = ru_div(ru_mul(md, cm), sigma);
      const double meta = ru_mul(md, eta);
      const double mer = ru_mul(md, er);
      if (!(meta < 0.5) || !(mer < 0.5)) {
        out = INFINITY;
      } else {
        const double gp = gamma_ru(md + 1.0, kU);
        const double one_meta = rd_sub(1.0, meta);
        const double one_mer = rd_sub(1.0, mer);
        double up = ru_sqrt(ru_div(ru_add(1.0, gp), one_meta));
        up = ru_div(up, __dmul_rd(one_mer, rd_sub(1.0, er)));
        double lo = rd_sqrt(__dmul_rd(rd_sub(1.0, gp), one_meta));
        lo = __ddiv_rd(__dmul_rd(lo, one_mer), ru_add(1.0, er));
        out = fmax(ru_add(up, -1.0), ru_add(1.0, -lo));
      }
    }
    rho[m] = out;
  }
  __syncwarp();
}

}  // namespace gbsb
