// haf_rec.cuh -- hafnian and loop hafnian by the recursion over pairs, binary64 and
// double-double, one warp per block of 2^m0 subsets (m0 <= 7) with every partial state in shared memory.
//
// haf(A) = [z^n] sum_{S subset [n]} (-1)^(n-|S|) f_S(z), the pairs (2u, 2u+1) taken in
// or left out one after the other (Bjorklund, "Counting perfect matchings as fast as
// Ryser", SODA 2012).  A state with m pairs left holds, for every pair of remaining
// vertices, the polynomial b_jk(z) of the paths j..k through the pairs taken so far
// (at the root b_jk = A_jk) and the polynomial g(z) of the closed ones (g = 1):
//   leave the pair (p, q) out:  the same polynomials, two vertices fewer;
//   take it in:  b'_jk = b_jk + z (b_jp b_kq + b_jq b_kp),   g' = g (1 + z e),
//                e = b_pq   (loop hafnian: e = b_pq + d_p d_q).
// Loop weights ride along as one more vertex D that is never taken: b_jD = d_j (the
// path from j to a loop) obeys the same rule.
//
// Two facts make it cheap.  Every remaining pair must contribute one z to [z^n] of the
// alternating sum, so a state with m pairs left matters only up to z^(n-m): the
// polynomials are short where the states are large.  And the last pair telescopes:
//   F_1 = [z^n] (g (1 + z e) - g) = [z^(n-1)] g e.
// A subset costs about 570 complex multiply-adds at n = 14 (shared between subsets),
// against about 20,000 for its own chain of matrix powers.  The alternating sum
// cancels less too: the terms hold each pair at most once per path.
//
// B200 mapping:
//   * FP64 FMA pipe, not the tensor cores: the contractions are 2 x (1 .. 26) vectors
//     of polynomials, mostly under 6 wide -- padding them to m16n8k8 tiles would waste
//     more than the two pipes (same peak) could give back;
//   * one lane computes one whole output polynomial (T + 2 coefficients, T = n - m):
//     its accumulators and one operand sit in registers, the other operand is read
//     once per coefficient, about 14 FMAs per 16-byte shared load at T = 12, and the
//     2 (T + 2) accumulators are independent chains, so one or two warps per scheduler
//     suffice.  T is a template parameter: a rolled loop (Horner's rule, P <- z P + a v)
//     spent as many register moves as FMAs on the shift
//     (measured, complex 28 x 28, 256 instances: 19 us each, 33 us rolled, 47 us with a
//     branch instead of an address select around every load; 250 us by power traces; 16 us
//     since e is kept where g' goes, which makes room for another warp);
//   * coefficient-major planes [c][pair] with pair index j(j-1)/2 + k, the pair taken
//     next being the two highest vertices: leaving a pair out is a view (shorter
//     planes), the operands of a lane are rows of the two taken vertices (contiguous
//     in k, broadcast in j);
//   * the highest n - m0 pairs are a fixed pattern per block (one state, taken in
//     place of the former), the next m0 - 5 a depth-first walk, and the last 5 pairs
//     are walked breadth-first, so that the small states of up to 16 siblings fill the
//     32 lanes.
#pragma once

#include <type_traits>

#include "cert.cuh"
#include "gbs_common.cuh"

namespace gbsb {

extern __shared__ __align__(128) double smem[];

constexpr int kHafRecBlock = 7;      // pairs of one block's subtree at most
constexpr int kHafRecWide = 5;       // of which walked breadth-first

// Polynomials b_jk of a state with m pairs left (L = 1: the loop vertex D on top).
__host__ __device__ inline int haf_rec_polys(int m, int L) {
  const int V = 2 * m + L;
  return V * (V - 1) / 2;
}
// One state (planes 0 .. n - m of the b_jk and g), in scalars.
__host__ __device__ inline int haf_rec_size(int n, int m, int L) { return (n - m + 1) * (haf_rec_polys(m, L) + 1); }

// Workspace of one warp, offsets in scalars (complex or real) from its start.
struct HafRecLayout {
  int m0, mB;                        // pairs of the block, of its breadth-first part
  int pz;                            // the prefix states alternate between 0 and pz
  int b5;                            // the state behind (leave, take) of a 7-pair block
  int lev[kHafRecWide];              // lev[m]: states with m pairs left, 2^(mB-1-m) of them
  int zero;                          // one cell that holds zero
  int e;                             // loop hafnian: e polynomials (of a step in place; dd: of a level)
  int total;
};
__host__ __device__ inline HafRecLayout haf_rec_layout(int n, int m0, int L, bool is_dd = false) {
  HafRecLayout R;
  R.m0 = m0;
  R.mB = m0 < kHafRecWide ? m0 : kHafRecWide;
  // the block's root state, with room for the pairs taken in place down to mB
  int o = (n - R.mB + 1) * (haf_rec_polys(m0, L) + 1);
  R.b5 = o;
  if (m0 > kHafRecWide + 1) o += haf_rec_size(n, kHafRecWide, L);
#pragma unroll
  for (int m = kHafRecWide - 1; m >= 1; --m) {
    R.lev[m] = o;
    if (m < R.mB) o += haf_rec_size(n, m, L) << (R.mB - 1 - m);
  }
  R.lev[0] = o;
  int pz = 0;
  for (int m = m0; m <= n; ++m) {
    const int s = haf_rec_size(n, m, L);
    pz = s > pz ? s : pz;
  }
  R.pz = pz;
  o = o > 2 * pz ? o : 2 * pz;
  R.zero = o++;
  R.e = o;
  if (L) {
    // a step out of place keeps e where it will put g' (only the lane that forms g' reads
    // it, before it writes); the double-double steps, whose lanes take single coefficients
    // of g', keep those of a whole level
    int es = n;
    for (int m = 2; is_dd && m <= R.mB; ++m) {
      const int x = (n - m + 1) << (R.mB - m);
      es = x > es ? x : es;
    }
    o += es;
  }
  R.total = o;
  return R;
}
// Workspace (doubles) for matrices of side 2n, whatever the split into blocks; `width`
// doubles per scalar (1 real, 2 complex, 4 complex double-double).
__host__ __device__ inline int haf_rec_ws(int n, bool loop, int width) {
  int t = 0;
  for (int m0 = 0; m0 <= n && m0 <= kHafRecBlock; ++m0) {
    const int w = haf_rec_layout(n, m0, loop ? 1 : 0, width == 4).total;
    t = w > t ? w : t;
  }
  return (width * t + 5) & ~3;
}

// ------------------------------------------------------------------ scalars
template <typename Z> __device__ __forceinline__ Z hz_zero();
template <> __device__ __forceinline__ cplx hz_zero<cplx>() { return mkc(0.0, 0.0); }
template <> __device__ __forceinline__ double hz_zero<double>() { return 0.0; }
template <> __device__ __forceinline__ ddc hz_zero<ddc>() { return ddc{dd_make(0.0), dd_make(0.0)}; }
__device__ __forceinline__ cplx hz_fma(cplx a, cplx b, cplx c) { return cfma(a, b, c); }
__device__ __forceinline__ ddc hz_fma(const ddc& a, const ddc& b, const ddc& c) { return ddc_add(c, ddc_mul(a, b)); }
__device__ __forceinline__ cplx hz_neg(cplx a) { return cneg(a); }
__device__ __forceinline__ double hz_neg(double a) { return -a; }
__device__ __forceinline__ ddc hz_neg(const ddc& a) { return ddc_neg(a); }
__device__ __forceinline__ cplx hz_sum(cplx a) { return warp_sum_c(a); }
__device__ __forceinline__ double hz_sum(double a) { return warp_sum_d(a); }
__device__ __forceinline__ ddc hz_sum(const ddc& a) { return warp_sum_ddc(a); }
__device__ __forceinline__ double hz_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ cplx hz_add(cplx a, cplx b) { return cadd(a, b); }
__device__ __forceinline__ double hz_add(double a, double b) { return a + b; }
__device__ __forceinline__ ddc hz_add(const ddc& a, const ddc& b) { return ddc_add(a, b); }
__device__ __forceinline__ cplx hz_bias(cplx a, double) { return a; }
__device__ __forceinline__ double hz_bias(double a, double t) { return a + t; }
template <typename Z> __device__ __forceinline__ Z hz_ld(int i);
template <> __device__ __forceinline__ double hz_ld<double>(int i) { return smem[i]; }
template <> __device__ __forceinline__ cplx hz_ld<cplx>(int i) {
  const double2 v = reinterpret_cast<const double2*>(smem)[i];
  return mkc(v.x, v.y);
}
template <> __device__ __forceinline__ ddc hz_ld<ddc>(int i) { return ld_ddc(smem + 4 * i); }
__device__ __forceinline__ void hz_st(int i, double v) { smem[i] = v; }
__device__ __forceinline__ void hz_st(int i, const ddc& v) { st_ddc(smem + 4 * i, v); }
__device__ __forceinline__ void hz_st(int i, cplx v) { reinterpret_cast<double2*>(smem)[i] = make_double2(v.re, v.im); }

// Loads by shared-memory byte address (an address select per load, no branch).  The compiler
// does not see that they read what hz_st wrote: haf_rec_op keeps its stores behind them.
__device__ __forceinline__ uint32_t hz_addr(int i, int bytes) {
  return (uint32_t)__cvta_generic_to_shared(smem) + (uint32_t)(i * bytes);
}
template <typename Z> __device__ __forceinline__ Z hz_lds(uint32_t a);
template <> __device__ __forceinline__ double hz_lds<double>(uint32_t a) {
  double x;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(a));
  return x;
}
template <> __device__ __forceinline__ cplx hz_lds<cplx>(uint32_t a) {
  cplx x;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x.re), "=d"(x.im) : "r"(a));
  return x;
}

// What one lane computes in a step: out = own + z (a1 b1 + a2 b2), offsets (scalars,
// from the start of shared memory) of the coefficient-0 entries, in planes of `str`
// (b1: of `bstr`), of which 0..lim are held (b1: 0..limb, a2 and b2: 0..lim2); the
// rest are read from a cell that holds zero (`zero`), without a branch.
struct HafRecLane {
  int own, a1, b1, a2, b2;
  int str, bstr, lim, limb, lim2;
  int zero;
  int dst, dstr;  // dst < 0: idle lane
};

// One output polynomial, coefficients 0 .. T + 1.  `bias` (real scalars): added to every
// coefficient (the majorant's underflow floor).
template <int T, typename Z>
__device__ __noinline__ void haf_rec_op(HafRecLane L, double bias) {
  constexpr int B = (int)sizeof(Z);
  asm volatile("" ::: "memory");  // stores before the step stay before its loads
  const uint32_t zero = hz_addr(L.zero, B);
  const uint32_t str = (uint32_t)(L.str * B);
  Z acc[T + 2];
  {
    uint32_t p = hz_addr(L.own, B);
#pragma unroll
    for (int c = 0; c <= T; ++c, p += str) acc[c] = hz_bias(hz_lds<Z>(c <= L.lim ? p : zero), bias);
    acc[T + 1] = hz_bias(hz_zero<Z>(), bias);
  }
  uint32_t a0 = hz_addr(L.a1, B), b0 = hz_addr(L.b1, B), bstr = (uint32_t)(L.bstr * B);
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    Z v[T + 1];
#pragma unroll
    for (int c = 0; c <= T; ++c, b0 += bstr) v[c] = hz_lds<Z>(c <= L.limb ? b0 : zero);
#pragma unroll
    for (int u = 0; u <= T; ++u, a0 += str) {
      const Z a = hz_lds<Z>(u <= L.lim ? a0 : zero);
#pragma unroll
      for (int w = 0; w + u <= T; ++w) acc[u + w + 1] = hz_fma(a, v[w], acc[u + w + 1]);
    }
    a0 = hz_addr(L.a2, B);
    b0 = hz_addr(L.b2, B);
    bstr = str;
    L.lim = L.limb = L.lim2;
  }
  asm volatile("" ::: "memory");  // a step in place overwrites words that it has read
  if (L.dst >= 0) {
#pragma unroll
    for (int c = 0; c < T + 2; ++c) hz_st(L.dst + c * L.dstr, acc[c]);
  }
}

// F_1 = [z^(n-1)] g e of one state with one pair left, the even (h = 0) or odd (h = 1)
// coefficients u of one factor: e = b_pq + d_p d_q (loop) or b_pq.  T = n - 1.
// b: b_pq; d0, d1: the loop paths; g: all coefficient-0 offsets in planes of str.
template <int T, typename Z, bool LOOP>
__device__ __noinline__ Z haf_rec_f1(int b, int d0, int d1, int g, int str, int lim, int h, int zero) {
  Z f = hz_zero<Z>();
  if constexpr (LOOP) {
    // acc = sum_i d0[2 i + h] z^(2 i) d1, so [z^(T - h)] g acc is this half of g d0 d1
    Z acc[T + 1], v[T + 1];
#pragma unroll
    for (int c = 0; c <= T; ++c) {
      acc[c] = hz_zero<Z>();
      v[c] = hz_ld<Z>(c <= lim ? d1 + c * str : zero);
    }
#pragma unroll
    for (int i = 0; 2 * i <= T; ++i) {
      const Z a = hz_ld<Z>(2 * i + h <= lim ? d0 + (2 * i + h) * str : zero);
#pragma unroll
      for (int w = 0; w + 2 * i <= T; ++w) acc[2 * i + w] = hz_fma(a, v[w], acc[2 * i + w]);
    }
#pragma unroll
    for (int c = 0; c <= T; ++c) {
      // of the odd half acc[T] lies beyond z^(n-1), perhaps beyond the number range: left out,
      // not multiplied by zero
      const int k = T - h - c;
      f = hz_fma(c < T || k == 0 ? acc[c] : hz_zero<Z>(), hz_ld<Z>(k >= 0 && k <= lim ? g + k * str : zero), f);
    }
  }
#pragma unroll
  for (int i = 0; 2 * i <= T; ++i) {
    const int u = 2 * i + h, k = T - u;
    const bool use = k >= 0 && u <= lim && k <= lim;
    f = hz_fma(hz_ld<Z>(use ? b + u * str : zero), hz_ld<Z>(use ? g + k * str : zero), f);
  }
  return f;
}

template <typename Z>
__device__ __forceinline__ void haf_rec_dispatch(int T, const HafRecLane& L, double bias) {
  switch (T) {
#define GBSB_REC_CASE(K) \
  case K: haf_rec_op<K, Z>(L, bias); break;
    GBSB_REC_CASE(0) GBSB_REC_CASE(1) GBSB_REC_CASE(2) GBSB_REC_CASE(3) GBSB_REC_CASE(4) GBSB_REC_CASE(5)
    GBSB_REC_CASE(6) GBSB_REC_CASE(7) GBSB_REC_CASE(8) GBSB_REC_CASE(9) GBSB_REC_CASE(10) GBSB_REC_CASE(11)
    GBSB_REC_CASE(12) GBSB_REC_CASE(13) GBSB_REC_CASE(14) GBSB_REC_CASE(15)
#undef GBSB_REC_CASE
    default: break;
  }
}
template <typename Z, bool LOOP>
__device__ __forceinline__ Z haf_rec_f1_dispatch(int T, int b, int d0, int d1, int g, int str, int lim, int h,
                                                 int zero) {
  switch (T) {
#define GBSB_REC_CASE(K) \
  case K: return haf_rec_f1<K, Z, LOOP>(b, d0, d1, g, str, lim, h, zero);
    GBSB_REC_CASE(0) GBSB_REC_CASE(1) GBSB_REC_CASE(2) GBSB_REC_CASE(3) GBSB_REC_CASE(4) GBSB_REC_CASE(5)
    GBSB_REC_CASE(6) GBSB_REC_CASE(7) GBSB_REC_CASE(8) GBSB_REC_CASE(9) GBSB_REC_CASE(10) GBSB_REC_CASE(11)
    GBSB_REC_CASE(12) GBSB_REC_CASE(13) GBSB_REC_CASE(14) GBSB_REC_CASE(15)
#undef GBSB_REC_CASE
    default: return hz_zero<Z>();
  }
}

// Vertex pair (j, k), j > k, of pair index q = j (j - 1) / 2 + k.
struct HafRecTri {
  unsigned char j[(kHafMaxN + 1) * kHafMaxN / 2];
};
constexpr HafRecTri haf_rec_tri_table() {
  HafRecTri t{};
  for (int j = 1, q = 0; j <= kHafMaxN; ++j)
    for (int k = 0; k < j; ++k, ++q) t.j[q] = (unsigned char)j;
  return t;
}
static __device__ const HafRecTri kHafRecTri = haf_rec_tri_table();
__host__ __device__ inline int haf_rec_row(int q) {
#ifdef __CUDA_ARCH__
  return kHafRecTri.j[q];
#else
  return haf_rec_tri_table().j[q];
#endif
}

// A state: offset of its plane 0, plane stride (g last in a plane), planes held - 1.
struct HafRecState {
  int off, str, lim;
};

// Lane descriptor of output q (a pair index below np, np = g) of a step that takes the
// two highest vertices of state s with m pairs left.  e: the state's e polynomial (loop),
// its coefficients estr apart.
__host__ __device__ inline HafRecLane haf_rec_lane(const HafRecState& s, int m, int loop, int np, int q, bool active,
                                                   int zero, int e, int estr, int dst, int dstr) {
  HafRecLane L;
  const int V = 2 * m + loop;
  const int r1 = s.off + (V - 1) * (V - 2) / 2, r0 = s.off + (V - 2) * (V - 3) / 2;  // rows of vertices V-1, V-2
  L.str = L.bstr = s.str;
  L.lim = L.limb = L.lim2 = s.lim;
  L.zero = zero;
  L.dst = dst + q;
  L.dstr = dstr;
  if (!active) {
    L.lim = L.limb = L.lim2 = L.dst = -1;
    L.own = L.a1 = L.b1 = L.a2 = L.b2 = s.off;
  } else if (q == np) {
    L.own = L.a1 = L.a2 = L.b2 = s.off + s.str - 1;  // g
    L.lim2 = -1;
    L.b1 = r1 + V - 2;
    if (loop) {
      L.b1 = e;
      L.bstr = estr;
      L.limb = kHafMaxN;  // every coefficient up to T
    }
    L.dst = dst + dstr - 1;
  } else {
    // q = j (j - 1) / 2 + k, j > k
    const int j = haf_rec_row(q), k = q - j * (j - 1) / 2;
    L.own = s.off + q;
    L.a1 = r0 + j;
    L.b1 = r1 + k;
    L.a2 = r1 + j;
    L.b2 = r0 + k;
  }
  return L;
}

// Coefficient c of e = b_pq + d_p d_q for the two highest vertices p, q of state s.
template <typename Z>
__device__ __forceinline__ Z haf_rec_e(const HafRecState& s, int m, int c) {
  const int V = 2 * m + 1;
  const int r1 = s.off + (V - 1) * (V - 2) / 2, r0 = s.off + (V - 2) * (V - 3) / 2;
  Z x = hz_zero<Z>();
  if (c <= s.lim) x = hz_ld<Z>(r1 + V - 2 + c * s.str);
  const int u1 = c < s.lim ? c : s.lim;
#pragma unroll 2
  for (int u = c > s.lim ? c - s.lim : 0; u <= u1; ++u)
    x = hz_fma(hz_ld<Z>(r0 + u * s.str), hz_ld<Z>(r1 + (c - u) * s.str), x);
  return x;
}

// Coefficient c of one output (see HafRecLane): the double-double steps give a lane single
// coefficients, since a product there is a hundred FP64 instructions against the two loads
// of its operands, and a whole polynomial would not fit its registers.
template <typename Z>
__device__ __forceinline__ Z haf_rec_coef(const HafRecLane& L, int c) {
  Z x = c <= L.lim ? hz_ld<Z>(L.own + c * L.str) : hz_zero<Z>();
  const int top = c - 1;
#pragma unroll 1
  for (int u = max(0, top - L.limb); u <= min(L.lim, top); ++u)
    x = hz_fma(hz_ld<Z>(L.a1 + u * L.str), hz_ld<Z>(L.b1 + (top - u) * L.bstr), x);
#pragma unroll 1
  for (int u = max(0, top - L.lim2); u <= min(L.lim2, top); ++u)
    x = hz_fma(hz_ld<Z>(L.a2 + u * L.str), hz_ld<Z>(L.b2 + (top - u) * L.str), x);
  return x;
}

// One step: outputs 0 .. cnt - 1 (of(q, active) describes output q), np polynomials and g
// per state.
template <typename Z, typename Of>
__device__ __forceinline__ void haf_rec_step(int T, int cnt, int np, Of of, double bias, int lane) {
  if constexpr (!std::is_same_v<Z, ddc>) {
    for (int q0 = 0; q0 < cnt; q0 += 32) haf_rec_dispatch<Z>(T, of(q0 + lane, q0 + lane < cnt), bias);
  } else {
    // a lane takes the coefficients h and T + 1 - h of a polynomial: equal work
    const int H = (T + 3) / 2;
    for (int x = lane; x < cnt * H; x += 32) {
      const int q = x / H, h = x - q * H;
      const HafRecLane L = of(q, true);
      if (L.a1 == L.own) continue;  // g, below
      const int h2 = T + 1 - h;
      hz_st(L.dst + h * L.dstr, haf_rec_coef<Z>(L, h));
      if (h2 != h) hz_st(L.dst + h2 * L.dstr, haf_rec_coef<Z>(L, h2));
    }
    // g: every coefficient reads the lower ones, which a step in place (one state)
    // overwrites, so they are all formed before any is stored
    const int states = cnt / (np + 1);
    for (int x0 = 0; x0 < states * (T + 2); x0 += 32) {
      const int x = x0 + lane;
      const bool act = x < states * (T + 2);
      const int p = act ? x / (T + 2) : 0, c = act ? x - p * (T + 2) : 0;
      const HafRecLane L = of(p * (np + 1) + np, true);
      Z v = hz_zero<Z>();
      if (act) v = haf_rec_coef<Z>(L, c);
      __syncwarp();
      if (act) hz_st(L.dst + c * L.dstr, v);
    }
  }
  __syncwarp();
}

// Take the two highest vertices of state s (m pairs left) into the planes at dst
// (stride dstr; dst == s.off with dstr == s.str works in place: the rows of the taken
// vertices lie behind every output).
template <typename Z>
__device__ __forceinline__ HafRecState haf_rec_take(const HafRecState& s, const HafRecLayout& R, int wo, int n, int m,
                                                    int loop, int dst, int dstr, double bias, int lane) {
  const int np = haf_rec_polys(m - 1, loop);
  const bool own_e = std::is_same_v<Z, ddc> || dst == s.off;
  const int e = own_e ? wo + R.e : dst + dstr - 1, estr = own_e ? 1 : dstr;
  if (loop) {
    if (lane <= n - m) hz_st(e + lane * estr, haf_rec_e<Z>(s, m, lane));
    __syncwarp();
  }
  haf_rec_step<Z>(
      n - m, np + 1, np,
      [&](int q, bool act) { return haf_rec_lane(s, m, loop, np, q, act, wo + R.zero, e, estr, dst, dstr); }, bias,
      lane);
  return HafRecState{dst, dstr, n - m + 1};
}

// Node p of level m of the breadth-first part: bit i of p = pair m + i taken.  Pairs
// left out since the last one taken make it a view of that state.
__host__ __device__ inline HafRecState haf_rec_node(const HafRecState& root, const HafRecLayout& R, int wo, int n,
                                                    int loop, int m, int p) {
  if (p == 0) return root;
  int t = 0;
  while (!((p >> t) & 1)) ++t;
  const int mm = m + t;
  const int str = haf_rec_polys(mm, loop) + 1;
  return HafRecState{wo + R.lev[mm] + (p >> (t + 1)) * ((n - mm + 1) * str), str, n - mm};
}

// Sum of one block's breadth-first part: the states behind the 2^mB subsets of the last
// mB >= 1 pairs of `root`, and F_1 of each.  MAJ adds every F_1 (majorant), otherwise
// with the sign of the pairs left out (`odd`: parity so far).
template <typename Z, bool MAJ>
__device__ __forceinline__ Z haf_rec_wide(const HafRecState& root, const HafRecLayout& R, int wo, int n, int loop,
                                          int odd, double bias, int lane) {
  const int mB = R.mB;
  for (int m = mB; m >= 2; --m) {
    const int np = haf_rec_polys(m - 1, loop);
    const int cnt = (np + 1) << (mB - m);
    const int dstr = np + 1, dsz = (n - m + 2) * dstr;
    const int ec = n - m + 1;  // coefficients of e
    const unsigned inv = (65536u + np) / (unsigned)(np + 1);  // q / (np + 1) for q < 16 (np + 1), np < 46
    constexpr bool own_e = std::is_same_v<Z, ddc>;
    const int eo = own_e ? wo + R.e : wo + R.lev[m - 1] + dstr - 1;  // node 0's e; the next ones epn behind
    const int epn = own_e ? ec : dsz, estr = own_e ? 1 : dstr;
    if (loop) {
      for (int q = lane; q < (ec << (mB - m)); q += 32) {
        const int p = q / ec, c = q - p * ec;
        hz_st(eo + p * epn + c * estr, haf_rec_e<Z>(haf_rec_node(root, R, wo, n, loop, m, p), m, c));
      }
      __syncwarp();
    }
    haf_rec_step<Z>(
        n - m, cnt, np,
        [&](int qq, bool act) {
          const int p = act ? (int)((unsigned)qq * inv >> 16) : 0;
          const int q = act ? qq - p * (np + 1) : 0;
          return haf_rec_lane(haf_rec_node(root, R, wo, n, loop, m, p), m, loop, np, q, act, wo + R.zero,
                              eo + p * epn, estr, wo + R.lev[m - 1] + p * dsz, dstr);
        },
        bias, lane);
  }
  Z f = hz_zero<Z>();
  // vertices: haf 0, 1 (b index 0); loop D = 0, then 1, 2 (d: 0 and 1, b: 2)
  if constexpr (std::is_same_v<Z, ddc>) {
    // lane: node p, coefficient k of e
    for (int x = lane; x < (n << (mB - 1)); x += 32) {
      const int p = x / n, k = x - p * n;
      const HafRecState s = haf_rec_node(root, R, wo, n, loop, 1, p);
      const int g = n - 1 - k;
      if (g > s.lim) continue;
      const Z e = loop ? haf_rec_e<Z>(s, 1, k) : (k <= s.lim ? hz_ld<Z>(s.off + k * s.str) : hz_zero<Z>());
      const Z t = ddc_mul(hz_ld<Z>(s.off + s.str - 1 + g * s.str), e);
      f = ddc_add(f, ((__popc(p) + odd) & 1) ? ddc_neg(t) : t);
    }
  } else {
    const int p = lane >> 1, h = lane & 1;
    const bool act = p < (1 << (mB - 1));
    const HafRecState s = haf_rec_node(root, R, wo, n, loop, 1, act ? p : 0);
    const int g = s.off + s.str - 1;
    const int lim = act ? s.lim : -1;
    f = loop ? haf_rec_f1_dispatch<Z, true>(n - 1, s.off + 2, s.off, s.off + 1, g, s.str, lim, h, wo + R.zero)
             : haf_rec_f1_dispatch<Z, false>(n - 1, s.off, s.off, s.off, g, s.str, lim, h, wo + R.zero);
    if (!MAJ && ((__popc(p) + odd) & 1)) f = hz_neg(f);
  }
  __syncwarp();
  return f;
}

// Stage the root: the symmetric part (A + A^T) / 2 (exact for a symmetric A; the sum
// over perfect matchings does not see the antisymmetric part to first order), or an
// upper bound of its modulus (MAJ); loop weights A_vv as they are.  `tiny`: a halving
// that could round absolutely (certified tiers: no radius relative to the entries covers
// that).  Binary64: a sum of unequal entries below twice the smallest normal number.
// Double-double: halves that do not double back, in either word -- the low one can be
// subnormal where the high one is normal.
template <typename Z, bool MAJ>
__device__ __forceinline__ void haf_rec_stage(const double* __restrict__ A, int N, int loop, int off, int lane,
                                              bool& tiny) {
  const int V = N + loop, np = V * (V - 1) / 2;
  for (int q = lane; q < np; q += 32) {
    const int j = haf_rec_row(q), k = q - j * (j - 1) / 2;
    if constexpr (std::is_same_v<Z, ddc>) {
      // the symmetric part exactly: TwoSum, halved
      ddc w;
      if (loop && k == 0) {
        w = ddc_make(ld_c(A + ((size_t)(j - 1) * N + (j - 1)) * 2));
      } else {
        const int r = j - loop, c = k - loop;
        const cplx x = ld_c(A + ((size_t)r * N + c) * 2), y = ld_c(A + ((size_t)c * N + r) * 2);
        double er, ei;
        const double sr = two_sum(x.re, y.re, er), si = two_sum(x.im, y.im, ei);
        w = ddc{dd{0.5 * sr, 0.5 * er}, dd{0.5 * si, 0.5 * ei}};
        if (2.0 * w.re.hi != sr || 2.0 * w.re.lo != er || 2.0 * w.im.hi != si || 2.0 * w.im.lo != ei) tiny = true;
      }
      hz_st(off + q, w);
      continue;
    }
    cplx w;
    if (loop && k == 0) {
      w = ld_c(A + ((size_t)(j - 1) * N + (j - 1)) * 2);
    } else {
      const int r = j - loop, c = k - loop;
      const cplx x = ld_c(A + ((size_t)r * N + c) * 2), y = ld_c(A + ((size_t)c * N + r) * 2);
      const cplx sum = cadd(x, y);
      w = cscale(sum, 0.5);
      if ((x.re != y.re || x.im != y.im) &&
          fmin(fabs(sum.re) > 0.0 ? fabs(sum.re) : 1.0, fabs(sum.im) > 0.0 ? fabs(sum.im) : 1.0) < 4.450147717014403e-308)
        tiny = true;
    }
    if constexpr (std::is_same_v<Z, cplx>) hz_st(off + q, w);
    if constexpr (std::is_same_v<Z, double>) hz_st(off + q, MAJ ? ru_abs_c(w) : w.re);
  }
  if (lane == 0) {
    if constexpr (std::is_same_v<Z, ddc>) hz_st(off + np, ddc_make(mkc(1.0, 0.0)));
    if constexpr (std::is_same_v<Z, cplx>) hz_st(off + np, mkc(1.0, 0.0));
    if constexpr (std::is_same_v<Z, double>) hz_st(off + np, 1.0);
  }
  __syncwarp();
}

// Signed sum (every lane gets it) over the subsets [lo, lo + count), both powers of two
// aligned as the planner cuts them.  MAJ: every term with a plus and every entry by its
// modulus.
template <typename Z, bool MAJ>
__device__ __noinline__ Z haf_rec_sum(const double* __restrict__ A, int N, int loop, unsigned lo, unsigned count,
                                      double* ws, int lane, bool& tiny) {
  const int n = N / 2;
  const int clog = 31 - __clz(count);
  const int m0 = clog < kHafRecBlock ? clog : kHafRecBlock;
  const HafRecLayout R = haf_rec_layout(n, m0, loop, std::is_same_v<Z, ddc>);
  const double bias = MAJ ? 0x1p-960 : 0.0;
  const int wo = (int)((ws - smem) / (sizeof(Z) / sizeof(double)));
  const int str0 = haf_rec_polys(m0, loop) + 1;
  const int g0 = str0 - 1;
  Z sum = hz_zero<Z>();
  if (lane == 0) hz_st(wo + R.zero, hz_zero<Z>());
#pragma unroll 1
  for (unsigned b = 0; b < (count >> m0); ++b) {
    const unsigned pat = (lo >> m0) + b;  // bit i: pair m0 + i
    const int left = (n - m0) - __popc(pat);
    // ---- the block's fixed pattern
    HafRecState s{wo, haf_rec_polys(n, loop) + 1, 0};
    haf_rec_stage<Z, MAJ>(A, N, loop, wo, lane, tiny);
#pragma unroll 1
    for (int m = n; m > m0; --m)
      if ((pat >> (m - 1 - m0)) & 1u)
        s = haf_rec_take<Z>(s, R, wo, n, m, loop, s.off == wo ? wo + R.pz : wo, haf_rec_polys(m - 1, loop) + 1, bias,
                            lane);
    if (s.off != wo || s.str != str0) {
      // move the root of the block to the front, its planes str0 apart
#pragma unroll 1
      for (int c = 0; c <= s.lim; ++c)
        for (int q0 = 0; q0 < str0; q0 += 32) {
          const int q = q0 + lane;
          Z x = hz_zero<Z>();
          if (q < str0) x = hz_ld<Z>(s.off + c * s.str + (q == g0 ? s.str - 1 : q));
          __syncwarp();
          if (q < str0) hz_st(wo + c * str0 + q, x);
        }
      __syncwarp();
      s.off = wo;
      s.str = str0;
    }
    if (m0 == 0) {  // no pair left: [z^n] g
      Z f = hz_zero<Z>();
      if (lane == 0 && s.lim >= n) f = hz_ld<Z>(wo + n * str0 + g0);
      sum = hz_add(sum, (!MAJ && (left & 1)) ? hz_neg(f) : f);
      __syncwarp();
      continue;
    }
    // ---- the walk over the block's highest m0 - mB pairs; a state no longer needed is
    // overwritten by its own successor
    const int d = m0 - R.mB;
    const int par = left + d + R.mB - 1;  // pairs left out if none of the block's is taken, F_1's own apart
#pragma unroll 1
    for (int t = 0; t < (1 << d); ++t) {
      HafRecState r = s;
      if (d == 2 && t == 1) {
        r = haf_rec_take<Z>(s, R, wo, n, 6, loop, wo + R.b5, haf_rec_polys(5, loop) + 1, bias, lane);
      } else if (t > 0) {
        s = r = haf_rec_take<Z>(s, R, wo, n, (d == 2 && t == 2) ? 7 : 6, loop, wo, str0, bias, lane);
      }
      const Z f = haf_rec_wide<Z, MAJ>(r, R, wo, n, loop, (par - __popc(t)) & 1, bias, lane);
      sum = hz_add(sum, f);
    }
  }
  return hz_sum(sum);
}

// ------------------------------------------------------------------ certified radius
// Every coefficient the walk computes is a fixed polynomial of the inputs, evaluated by
// complex multiply-adds; the majorant walk evaluates the polynomial with every
// coefficient and every input replaced by its modulus.  One multiply-add errs by
//   |fl(acc + a v) - (acc + a v)| <= 3u (|acc| + |a||v|)
// (two fused steps per component: u(1 + u)(2|acc| + 2 sqrt(2) |a||v|)), so if acc, a, v
// are within ((1 + 3u)^k - 1) of their majorants (k = ka, kb, ...), the result is within
// (1 + 3u)^(max(k_acc, k_a + k_v) + 1) - 1 of its own.  Subnormal roundings (below
// 2^-1065 per coefficient) are covered by one more unit, since every majorant
// coefficient of a taken pair is at least 2^-960.  haf_rec_units runs that recurrence
// of k over the levels:
//   b'[c]: max(b[c], b[u] + b[v]) + 2 c + 2    (u + v = c - 1; 2 c products, one sum)
//   e[c] : max(b[c], b[u] + b[v]) + c + 2      (loop: u + v = c)
//   g'[c]: max(g[c], g[u] + e[v]) + c + 2
// and ends with F_1 (at most 3 n + 2 additions).  Input entries carry one unit (the
// rounding of the symmetric part).
__host__ __device__ constexpr double haf_rec_units(int n, bool loop) {
  double b[kHafMaxN / 2 + 2] = {}, g[kHafMaxN / 2 + 2] = {}, e[kHafMaxN / 2 + 2] = {};
  double nb[kHafMaxN / 2 + 2] = {}, ng[kHafMaxN / 2 + 2] = {};
  b[0] = 1.0;
  double top = 0.0;
  for (int T = 0; T < n; ++T) {
    for (int c = 0; c <= T; ++c) {
      double x = b[c];
      if (loop)
        for (int u = 0; u <= c; ++u) x = b[u] + b[c - u] > x ? b[u] + b[c - u] : x;
      e[c] = loop ? x + c + 2 : x;
    }
    if (T == n - 1) {
      for (int c = 0; c <= T; ++c) top = g[c] + e[T - c] > top ? g[c] + e[T - c] : top;
      break;
    }
    for (int c = 0; c <= T + 1; ++c) {
      double x = c <= T ? b[c] : 0.0, y = c <= T ? g[c] : 0.0;
      for (int u = 0; u < c; ++u) {
        x = b[u] + b[c - 1 - u] > x ? b[u] + b[c - 1 - u] : x;
        y = g[u] + e[c - 1 - u] > y ? g[u] + e[c - 1 - u] : y;
      }
      nb[c] = x + 2 * c + 2;
      ng[c] = y + c + 2;
    }
    for (int c = 0; c <= T + 1; ++c) {
      b[c] = nb[c];
      g[c] = ng[c];
    }
  }
  return top + 3 * n + 2;
}
struct HafRecUnits {
  float k[2][kHafMaxN / 2 + 1];  // small whole numbers
};
constexpr HafRecUnits haf_rec_units_table() {
  HafRecUnits t{};
  for (int n = 1; n <= kHafMaxN / 2; ++n) {
    t.k[0][n] = (float)haf_rec_units(n, false);
    t.k[1][n] = (float)haf_rec_units(n, true);
  }
  return t;
}
static __device__ const HafRecUnits kHafRecUnits = haf_rec_units_table();

// Radius of the sum over `count` subsets from its majorant sum `maj` (computed to
// nearest: at most as many roundings, all of positive terms, hence the factor).
// Double-double: one multiply-add errs by at most 21u^2 |a||v| (product) and 6u^2 of the
// sum, 28u^2 (|acc| + |a||v|) in all, and its inputs are exact; the same recurrence counts
// the units.  A lane adds up to 9 terms per breadth-first part there.
__device__ __forceinline__ double haf_rec_radius(int n, int loop, unsigned count, double maj, bool is_dd) {
  const double blocks = count >> kHafRecBlock ? (double)(count >> kHafRecBlock) : 1.0;
  const double k = (double)kHafRecUnits.k[loop][n] + (is_dd ? 40.0 : 4.0) * blocks + 8.0;  // + the sums
  const double g = gamma_ru(k, 3.0 * kU);
  const double up = ru_div(ru_add(maj, 1e-300), rd_sub(1.0, g));
  return ru_mul(is_dd ? gamma_ru(k, 28.0 * kU * kU) : g, up);
}

}  // namespace gbsb
