// tor_rec.cuh -- torontonian by a recursion over modes on Schur complements, one warp per
// work item, binary64 (fp64, indicator, certified) and double-double tiers.
//
// tor(O) = sum_{S subset [k]} (-1)^(k-|S|) / sqrt(det((I - O)_S)),  xxpp ordering, where
// including mode j puts rows / columns j and j + k of M = I - O in the minor.
// Reference algorithm: the recursive prefix Cholesky of core/tor_recursive.cu:41-115
// (cpu_ref/tor_recursive.py:46-100): the subsets form a binary tree over the modes, and
// including a mode appends its two rows to one Cholesky factor.
//
// Here a node of that tree is the Schur complement Z of the modes included so far on the
// modes still undecided (packed lower triangle) and t = the product of 1 / L_jj so far.
// Leaving a mode out is a view (two rows fewer); including it is one right-looking
// Cholesky step on its two rows a, b:
//   i0 = rsqrt(Z_aa), l_j = Z_aj i0;  i1 = rsqrt(Z_bb - l_b^2), l'_j = (Z_bj - l_j l_b) i1;
//   Z'_ij = (Z_ij - l_i l_j) - l'_i l'_j,  t' = t i0 i1,
// so each entry sees the operations of the left-looking factorisation, in its order, but
// shared by every subset below the node: near the leaves, where the nodes are, the blocks
// are 2 x 2 to 8 x 8.
//
// B200 mapping: mode k - 1 owns rows 0, 1 and mode j rows 2 (k - 1 - j), so the undecided
// modes are the leading block and the mode decided next its last two rows.
//   * the item's fixed pattern over the first g modes: in place on the whole matrix;
//   * the next modes depth-first in binary-counter order, one shared buffer per level;
//   * five modes breadth-first: up to 32 nodes, lanes over (node, entry);
//   * the last kTail modes (4; double-double 3) per lane in registers: lane = node, the
//     2^kTail subsets by a compile-time recursion, the last mode by its 2 x 2 determinant.
// Bound by latency and the issue of its instruction stream (about 3,200 warp instructions
// per 512 subsets, a quarter of them FP64), not by the FP64 pipe.  Measured, against one
// 10 x 10 factorisation per lane and subset: 64 x 20 modes 5.98 -> 1.43 ms, 512 x 12 modes
// 0.340 -> 0.091 ms.
//
// Certified tiers: see tor_warp.cuh (the a-posteriori radius |t| rho_m of a term of
// dimension m); the step above satisfies its premises: every factor entry is an inner
// product of at most m fused terms and one scaling, the last block's determinant adds
// one rounding of Z_bb, and the product of the t's takes fewer roundings than rho
// charges.  Value and radius are carried through the same sums.
#pragma once

#include "tor_warp.cuh"
#include "tor_warp_dd.cuh"

namespace gbsb {

constexpr int kTorRecWide = 5;  // modes walked breadth-first

template <typename S> struct TorRec;
template <> struct TorRec<double> {
  static constexpr int kTail = 4, W = 1, kOrder = 5;  // modes per lane, doubles per scalar, tor_rec_source's tail
};
template <> struct TorRec<dd> {
  static constexpr int kTail = 3, W = 2, kOrder = 4;
};

// Row i of packed entry e = i (i + 1) / 2 + j, i < 64 (32 modes).
struct TorRecTri {
  unsigned char i[64 * 65 / 2];
};
constexpr TorRecTri tor_rec_tri_table() {
  TorRecTri t{};
  for (int i = 0, e = 0; i < 64; ++i)
    for (int j = 0; j <= i; ++j, ++e) t.i[e] = (unsigned char)i;
  return t;
}
static __device__ const TorRecTri kTorRecTri = tor_rec_tri_table();
__host__ __device__ inline int tor_rec_row(int e) {
#ifdef __CUDA_ARCH__
  return kTorRecTri.i[e];
#else
  return tor_rec_tri_table().i[e];
#endif
}

__host__ __device__ constexpr int tor_rec_entries(int m) { return m * (2 * m + 1); }
// sum of tor_rec_entries(1 .. m)
__host__ __device__ inline int tor_rec_below(int m) { return m * (m + 1) * (2 * m + 1) / 3 + m * (m + 1) / 2; }

// Workspace of one item (k modes, f of them free), offsets in scalars.
struct TorRecLayout {
  int f, mW, mt;           // free modes, breadth-first from mW down to mt
  int lev;                 // breadth-first states: levels mW - 1 .. mt one after the other
  int lc, piv, t;          // columns l, l'; (i0, l_b, i1) per node; t per state
  int noff;                // offsets of a level's nodes (ints, two to a double)
  int rho;                 // certified: rho_m (doubles, from 2x this offset in double-double)
  int total;
};
__host__ __device__ inline TorRecLayout tor_rec_layout(int k, int f, int tail, bool cert, int W) {
  TorRecLayout R;
  R.f = f;
  R.mt = f < tail ? f : tail;
  R.mW = f < tail + kTorRecWide ? f : tail + kTorRecWide;
  // depth-first states behind the leading f-mode block, over the rest of the matrix
  int o = tor_rec_entries(f) + tor_rec_below(f > 0 ? f - 1 : 0) - tor_rec_below(R.mW > 0 ? R.mW - 1 : 0);
  if (o < tor_rec_entries(k)) o = tor_rec_entries(k);
  R.lev = o;
  for (int m = R.mW - 1; m >= R.mt; --m) o += tor_rec_entries(m) << (R.mW - 1 - m);
  o = (o + 1) & ~1;  // l, l' pairs on 16 bytes
  R.lc = o;
  int lc = 4 * k;  // one node of the whole matrix, or a breadth-first level
  for (int m = R.mW; m > R.mt; --m) {
    const int x = (4 * (m - 1)) << (R.mW - m);
    lc = x > lc ? x : lc;
  }
  o += lc;
  R.piv = o;
  o += 3 << kTorRecWide;
  R.t = o;
  o += f + 1 + (1 << kTorRecWide);
  R.noff = o;
  o += (1 << kTorRecWide) / 2;
  if (cert) {  // the eigenvalue proof factors a packed 2k x 2k matrix (+ 2k scalings)
    const int need = (k * (2 * k + 1) + 2 * k + 8 + W - 1) / W;
    if (o < need) o = need;
  }
  R.rho = o;
  if (cert) o += (2 * k + 2 + W - 1) / W;
  R.total = o;
  return R;
}
__host__ __device__ inline int tor_rec_dfs(const TorRecLayout& R, int m) {  // depth-first state of m modes
  return tor_rec_entries(R.f) + tor_rec_below(R.f - 1) - tor_rec_below(m);
}
__host__ __device__ inline int tor_rec_lev(const TorRecLayout& R, int m, int slot) {  // breadth-first state
  int o = R.lev;
  for (int x = R.mW - 1; x > m; --x) o += tor_rec_entries(x) << (R.mW - 1 - x);
  return o + slot * tor_rec_entries(m);
}
// Free modes walked at a time; an item with more (a tuned split) runs its patterns of the
// others one after another.  12 would keep two depth-first states fewer and fit 9 warps an
// SM instead of 7, but stages the matrix four times as often: 20 modes 1.89 against 1.60 ms.
constexpr int kTorRecFree = 14;
__host__ __device__ inline int tor_rec_free(int k, int g) { return k - g < kTorRecFree ? k - g : kTorRecFree; }
// Pattern p over the first g2 modes of an item that starts at pattern `lo` of the first g: the
// other g2 - g modes, above them in the word, change fastest.
__host__ __device__ inline uint32_t tor_rec_pattern(unsigned long long lo, unsigned long long p, int g, int g2) {
  const int more = g2 - g;
  return (uint32_t)((lo + (p >> more)) | ((p & ((1ull << more) - 1)) << g));
}
// Workspace (doubles) of an instance of k modes whose items fix the first g.
__host__ __device__ inline int tor_rec_ws(int k, int g, bool is_dd, bool cert) {
  const int t = tor_rec_layout(k, tor_rec_free(k, g), is_dd ? TorRec<dd>::kTail : TorRec<double>::kTail, cert,
                               is_dd ? 2 : 1).total;
  return ((is_dd ? 2 * t : t) + 3) & ~3;
}

// Entry maps of the breadth-first levels when all five are walked (mW = tail + 5): word q of
// a level that leaves states of m - 1 modes holds the positions of its entry's two columns
// (l, l' pairs) and its node: (p rows + i) | (p rows + j) << 12 | p << 24.
__host__ __device__ constexpr int tor_rec_map_size(int tail) {
  int n = 0;
  for (int m = tail + kTorRecWide; m > tail; --m) n += tor_rec_entries(m - 1) << (tail + kTorRecWide - m);
  return n;
}
__host__ __device__ constexpr int tor_rec_map_off(int tail, int m) {  // first word of level m
  int n = 0;
  for (int x = tail + kTorRecWide; x > m; --x) n += tor_rec_entries(x - 1) << (tail + kTorRecWide - x);
  return n;
}
template <int TAIL>
struct TorRecMap {
  unsigned w[tor_rec_map_size(TAIL)];
};
template <int TAIL>
constexpr TorRecMap<TAIL> tor_rec_map_table() {
  TorRecMap<TAIL> t{};
  int q = 0;
  for (int m = TAIL + kTorRecWide; m > TAIL; --m)
    for (int p = 0; p < (1 << (TAIL + kTorRecWide - m)); ++p)
      for (int i = 0; i < 2 * m - 2; ++i)
        for (int j = 0; j <= i; ++j)
          t.w[q++] = (unsigned)(p * (2 * m - 2) + i) | (unsigned)(p * (2 * m - 2) + j) << 12 | (unsigned)p << 24;
  return t;
}
static __device__ const TorRecMap<4> kTorRecMap4 = tor_rec_map_table<4>();
static __device__ const TorRecMap<3> kTorRecMap3 = tor_rec_map_table<3>();
template <int TAIL>
__host__ __device__ inline unsigned tor_rec_map(int q) {
#ifdef __CUDA_ARCH__
  return TAIL == 4 ? kTorRecMap4.w[q] : kTorRecMap3.w[q];
#else
  return tor_rec_map_table<TAIL>().w[q];
#endif
}

// A state: offset of its packed block, index of its t.
struct TorRecState {
  int off, t;
};
// Node p of level m of the breadth-first part (bit i of p = the mode decided at level
// m + i + 1 was included); left-out modes make it a view.
__host__ __device__ inline TorRecState tor_rec_node(const TorRecLayout& R, const TorRecState& root, int m, int p) {
  if (p == 0) return root;
  int s = 0;
  while (!((p >> s) & 1)) ++s;
  const int mm = m + s, slot = p >> (s + 1);
  return TorRecState{tor_rec_lev(R, mm, slot), R.f + (1 << (R.mW - 1 - mm)) + slot};
}
// State at level mW of the depth-first walk after Tm (bit i: the mode decided at level
// mW + 1 + i was included).
__host__ __device__ inline TorRecState tor_rec_walked(const TorRecLayout& R, const TorRecState& root, uint32_t Tm) {
  if (Tm == 0) return root;
  int s = 0;
  while (!((Tm >> s) & 1u)) ++s;
  return TorRecState{tor_rec_dfs(R, R.mW + s), R.f - (R.mW + s)};
}

// The entry of O read for row i, column j <= i of M, which belong to the modes mi <= mj.  O is
// meant to be symmetric; of one that is not, the torontonian reads the lower triangle in the
// order (mode, x before p), as the reference does, but for the block of the last `tail`
// modes (5, double-double 4) against the modes before them, where it reads the upper one.
__host__ __device__ inline void tor_rec_source(int k, int tail, int i, int mi, int j, int mj, int& row, int& col) {
  const int a = mi + (i & 1) * k, b = mj + (j & 1) * k;
  const bool upper = mi == mj || (mi < k - tail && mj >= k - tail);
  row = upper ? a : b;
  col = upper ? b : a;
}
// ------------------------------------------------------------------ scalars
__device__ __forceinline__ double ts_ld(const double* ws, int i, double) { return ws[i]; }
__device__ __forceinline__ dd ts_ld(const double* ws, int i, dd) { return ld_dd(ws + 2 * i); }
__device__ __forceinline__ void ts_st(double* ws, int i, double v) { ws[i] = v; }
__device__ __forceinline__ void ts_st(double* ws, int i, dd v) { st_dd(ws + 2 * i, v); }
__device__ __forceinline__ double ts_fms(double a, double b, double c) { return fma(-b, c, a); }
__device__ __forceinline__ dd ts_fms(dd a, dd b, dd c) { return dd_fms(a, b, c); }
__device__ __forceinline__ double ts_mul(double a, double b) { return a * b; }
__device__ __forceinline__ dd ts_mul(dd a, dd b) { return dd_mul(a, b); }
__device__ __forceinline__ double ts_add(double a, double b) { return a + b; }
__device__ __forceinline__ dd ts_add(dd a, dd b) { return dd_add(a, b); }
__device__ __forceinline__ double ts_neg(double a) { return -a; }
__device__ __forceinline__ dd ts_neg(dd a) { return dd_neg(a); }
__device__ __forceinline__ double ts_hi(double a) { return a; }
__device__ __forceinline__ double ts_hi(dd a) { return a.hi; }
__device__ __forceinline__ double ts_make(double a, double) { return a; }
__device__ __forceinline__ dd ts_make(double a, dd) { return dd_make(a); }
__device__ __forceinline__ double ts_m(const double* Oc, int dim, int a, int b, double) { return tor_m(Oc, dim, a, b); }
__device__ __forceinline__ dd ts_m(const double* Oc, int dim, int a, int b, dd) { return tor_m_dd(Oc, dim, a, b); }
// rsqrt of a pivot; a pivot that is not positive clears ok and counts as 1
__device__ __forceinline__ double ts_rsqrt(double s, bool& ok) {
  if (!(s > 0.0)) {
    ok = false;
    s = 1.0;
  }
  return rsqrt(s);
}
__device__ __forceinline__ dd ts_rsqrt(dd s, bool& ok) {
  if (!(s.hi > 0.0)) {
    ok = false;
    s = dd_make(1.0);
  }
  return dd_rsqrt(s);
}
// radius of one rounded sum v
__device__ __forceinline__ double ts_sum_err(double v) { return ru_mul(kUc, fabs(v)); }
__device__ __forceinline__ double ts_sum_err(dd v) { return ru_add(ru_mul(4.0 * kU * kU, fabs(v.hi)), kUfl); }
// radius of one term
__device__ __forceinline__ double ts_term_err(double t, double rho) { return ru_add(ru_mul(fabs(t), rho), kUfl); }
__device__ __forceinline__ double ts_term_err(dd t, double rho) {
  return ru_add(ru_mul(ru_mul(fabs(t.hi), 1.0 + 4.0 * kU), rho), kUfl);
}

// ------------------------------------------------------------------ one level
// Include the mode on the last two rows of each of N states (m modes each, node p given
// by src(p)); successor p goes to dst + p * entries(m - 1), its t to index dt + p.
template <typename S, typename Src>
__device__ __forceinline__ void tor_rec_include(double* ws, const TorRecLayout& R, int m, int N, Src src, int dst,
                                                int dt, int lane, bool& ok) {
  const S z{};
  const int ra = (2 * m - 2) * (2 * m - 1) / 2, rb = (2 * m - 1) * m;  // packed rows a = 2m - 2, b = 2m - 1
  int* noff = reinterpret_cast<int*>(ws + R.noff * TorRec<S>::W);
  if (lane < N) {
    const TorRecState s = src(lane);
    const S i0 = ts_rsqrt(ts_ld(ws, s.off + ra + 2 * m - 2, z), ok);
    const S lb = ts_mul(ts_ld(ws, s.off + rb + 2 * m - 2, z), i0);
    const S i1 = ts_rsqrt(ts_fms(ts_ld(ws, s.off + rb + 2 * m - 1, z), lb, lb), ok);
    noff[lane] = s.off;
    ts_st(ws, R.piv + 3 * lane, i0);
    ts_st(ws, R.piv + 3 * lane + 1, lb);
    ts_st(ws, R.piv + 3 * lane + 2, i1);
    ts_st(ws, R.t + dt + lane, ts_mul(ts_mul(ts_ld(ws, R.t + s.t, z), i0), i1));
  }
  __syncwarp();
  const int rows = 2 * m - 2, E = tor_rec_entries(m - 1);
  // q / rows, q / E for the node of a lane's column or entry: N <= 16 nodes of at most
  // 136 entries (one node: any size), exact as (q inv) >> 20
  const unsigned invr = (1048575u + rows) / rows, invE = (1048575u + E) / E;
#pragma unroll 2
  for (int q = lane; q < N * rows; q += 32) {
    const int p = N == 1 ? 0 : (int)((unsigned)q * invr >> 20), j = q - p * rows;
    const int o = noff[p], v = R.piv + 3 * p;
    const S l0 = ts_mul(ts_ld(ws, o + ra + j, z), ts_ld(ws, v, z));
    const S l1 = ts_mul(ts_fms(ts_ld(ws, o + rb + j, z), l0, ts_ld(ws, v + 1, z)), ts_ld(ws, v + 2, z));
    ts_st(ws, R.lc + 2 * q, l0);
    ts_st(ws, R.lc + 2 * q + 1, l1);
  }
  __syncwarp();
#pragma unroll 4
  for (int q = lane; q < N * E; q += 32) {
    const int p = N == 1 ? 0 : (int)((unsigned)q * invE >> 20), e = q - p * E;
    const int i = tor_rec_row(e), j = e - i * (i + 1) / 2;
    const int cp = R.lc + 2 * p * rows;
    S v = ts_fms(ts_ld(ws, noff[p] + e, z), ts_ld(ws, cp + 2 * i, z), ts_ld(ws, cp + 2 * j, z));
    v = ts_fms(v, ts_ld(ws, cp + 2 * i + 1, z), ts_ld(ws, cp + 2 * j + 1, z));
    ts_st(ws, dst + q, v);
  }
  __syncwarp();
}

// l, l' of one column
__device__ __forceinline__ void ts_ld_pair(const double* ws, int i, double& a, double& b) {
  const double2 v = *reinterpret_cast<const double2*>(ws + i);
  a = v.x;
  b = v.y;
}
__device__ __forceinline__ void ts_ld_pair(const double* ws, int i, dd& a, dd& b) {
  a = ld_dd(ws + 2 * i);
  b = ld_dd(ws + 2 * i + 2);
}

// The breadth-first levels M .. tail + 1 of a full walk (root w at mW = tail + 5), every
// size a constant and the entries from the map: index arithmetic on runtime sizes was half
// of the walk's instructions (16 modes, 512 instances: 838 us before, 704 with the entry
// loops unrolled whole).
template <typename S, int M>
__device__ __forceinline__ void tor_rec_levels(double* ws, const TorRecLayout& R, const TorRecState& w, int lane,
                                               bool& ok) {
  constexpr int TAIL = TorRec<S>::kTail, MW = TAIL + kTorRecWide;
  if constexpr (M > TAIL) {
    constexpr int N = 1 << (MW - M), rows = 2 * M - 2, E = tor_rec_entries(M - 1);
    constexpr int ra = (2 * M - 2) * (2 * M - 1) / 2, rb = (2 * M - 1) * M;
    const S z{};
    int* noff = reinterpret_cast<int*>(ws + R.noff * TorRec<S>::W);
    if (lane < N) {
      const TorRecState s = tor_rec_node(R, w, M, lane);
      const S i0 = ts_rsqrt(ts_ld(ws, s.off + ra + 2 * M - 2, z), ok);
      const S lb = ts_mul(ts_ld(ws, s.off + rb + 2 * M - 2, z), i0);
      const S i1 = ts_rsqrt(ts_fms(ts_ld(ws, s.off + rb + 2 * M - 1, z), lb, lb), ok);
      noff[lane] = s.off;
      ts_st(ws, R.piv + 3 * lane, i0);
      ts_st(ws, R.piv + 3 * lane + 1, lb);
      ts_st(ws, R.piv + 3 * lane + 2, i1);
      ts_st(ws, R.t + R.f + N + lane, ts_mul(ts_mul(ts_ld(ws, R.t + s.t, z), i0), i1));
    }
    __syncwarp();
#pragma unroll
    for (int q0 = 0; q0 < N * rows; q0 += 32) {
      const int q = q0 + lane;
      if (q0 + 32 <= N * rows || q < N * rows) {
        const int p = q / rows, j = q - p * rows;
        const int o = noff[p], v = R.piv + 3 * p;
        const S l0 = ts_mul(ts_ld(ws, o + ra + j, z), ts_ld(ws, v, z));
        const S l1 = ts_mul(ts_fms(ts_ld(ws, o + rb + j, z), l0, ts_ld(ws, v + 1, z)), ts_ld(ws, v + 2, z));
        ts_st(ws, R.lc + 2 * q, l0);
        ts_st(ws, R.lc + 2 * q + 1, l1);
      }
    }
    __syncwarp();
    constexpr int mo = tor_rec_map_off(TAIL, M);
    const int dst = R.lev + mo;
    // double-word steps are thirty times as long: unrolled they only miss the instruction cache
    constexpr int UN = TorRec<S>::W == 1 ? 32 : 1;
#pragma unroll UN
    for (int q0 = 0; q0 < N * E; q0 += 32) {
      const int q = q0 + lane;
      if (q0 + 32 <= N * E || q < N * E) {
        const unsigned x = tor_rec_map<TAIL>(mo + q);
        const int p = (int)(x >> 24);
        S l0i, l1i, l0j, l1j;
        ts_ld_pair(ws, R.lc + 2 * (int)(x & 0xfffu), l0i, l1i);
        ts_ld_pair(ws, R.lc + 2 * (int)(x >> 12 & 0xfffu), l0j, l1j);
        ts_st(ws, dst + q, ts_fms(ts_fms(ts_ld(ws, noff[p] - p * E + q, z), l0i, l0j), l1i, l1j));
      }
    }
    __syncwarp();
    tor_rec_levels<S, M - 1>(ws, R, w, lane, ok);
  }
}

// ------------------------------------------------------------------ the last modes, per lane
// Sum over the subsets of the leading M modes of Z (packed, M (2M + 1) entries in
// registers) of (-1)^(M - |T|) t(T), with the sum of |t| (AUX 1) or the radius (AUX 2;
// `dim` rows included so far).
template <typename S, int AUX>
struct TorRecSum {
  S v;
  double a;
};
template <typename S, int AUX, int M, int E>
__device__ __forceinline__ TorRecSum<S, AUX> tor_rec_tail(const S (&Z)[E], S t, int dim, const double* rho, bool& ok) {
  if constexpr (M == 0) {
    return {t, AUX == 1 ? fabs(ts_hi(t)) : (AUX == 2 ? ts_term_err(t, rho[dim]) : 0.0)};
  } else {
    TorRecSum<S, AUX> in;
    constexpr int ra = (2 * M - 2) * (2 * M - 1) / 2, rb = (2 * M - 1) * M;
    if constexpr (M == 1) {
      // det of the 2 x 2 block: one rsqrt instead of two.  A first pivot that is not
      // positive is refused like any other.
      if (!(ts_hi(Z[0]) > 0.0)) ok = false;
      const S det = ts_fms(ts_mul(Z[0], Z[2]), Z[1], Z[1]);
      const S ti = ts_mul(t, ts_rsqrt(det, ok));
      in = {ti, AUX == 1 ? fabs(ts_hi(ti)) : (AUX == 2 ? ts_term_err(ti, rho[dim + 2]) : 0.0)};
    } else {
      constexpr int R = 2 * M - 2;
      const S i0 = ts_rsqrt(Z[ra + R], ok);
      const S lb = ts_mul(Z[rb + R], i0);
      const S i1 = ts_rsqrt(ts_fms(Z[rb + R + 1], lb, lb), ok);
      S l0[R], l1[R], Y[R * (R + 1) / 2];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        l0[j] = ts_mul(Z[ra + j], i0);
        l1[j] = ts_mul(ts_fms(Z[rb + j], l0[j], lb), i1);
      }
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j)
          Y[i * (i + 1) / 2 + j] = ts_fms(ts_fms(Z[i * (i + 1) / 2 + j], l0[i], l0[j]), l1[i], l1[j]);
      in = tor_rec_tail<S, AUX, M - 1>(Y, ts_mul(ts_mul(t, i0), i1), dim + 2, rho, ok);
    }
    const TorRecSum<S, AUX> out = tor_rec_tail<S, AUX, M - 1>(Z, t, dim, rho, ok);
    TorRecSum<S, AUX> r;
    r.v = ts_add(in.v, ts_neg(out.v));
    r.a = AUX == 1 ? in.a + out.a : (AUX == 2 ? ru_add(ru_add(in.a, out.a), ts_sum_err(r.v)) : 0.0);
    return r;
  }
}
template <typename S, int AUX, int M>
__device__ __forceinline__ TorRecSum<S, AUX> tor_rec_tail_load(const double* ws, int off, S t, int dim,
                                                               const double* rho, bool& ok) {
  constexpr int E = M == 0 ? 1 : M * (2 * M + 1);
  S Z[E];
  const S z{};
  if constexpr (M > 0) {
#pragma unroll
    for (int e = 0; e < E; ++e) Z[e] = ts_ld(ws, off + e, z);
  }
  return tor_rec_tail<S, AUX, M>(Z, t, dim, rho, ok);
}

// ------------------------------------------------------------------ one work item
// Pattern `pat` over the first g modes, then every subset of the other f = k - g.  AUX
// 0: value, 1: and sum |term|, 2: and the radius.  Returns false when a pivot was not
// positive.
template <typename S, int AUX>
static __device__ __noinline__ bool tor_rec_item(const double* __restrict__ Oc, int k, int g, uint32_t pat, double* ws,
                                                 const TorRecLayout R, const double* rho, int lane, S& total,
                                                 double& aux) {
  constexpr int TAIL = TorRec<S>::kTail;
  const S z{};
  const int dim = 2 * k;
  const uint32_t inc = pat & (g < 32 ? (1u << g) - 1u : 0xffffffffu);
  const int inc0 = __popc(inc), ks = R.f + inc0;
  if (g == 0) {
    for (int e = lane; e < tor_rec_entries(k); e += 32) {
      const int i = tor_rec_row(e), j = e - i * (i + 1) / 2;
      int r, c;
      tor_rec_source(k, TorRec<S>::kOrder, i, k - 1 - (i >> 1), j, k - 1 - (j >> 1), r, c);
      ts_st(ws, e, ts_m(Oc, dim, r, c, z));
    }
  } else {
    // the modes that the pattern leaves out are not staged at all: their rows lie behind those
    // of every later step (20 modes in 2^14 items of 2^6 subsets: 0.75 ms, 0.79 with them)
    int* modes = reinterpret_cast<int*>(ws + R.noff * TorRec<S>::W);  // included modes, the last first
    if ((inc >> lane) & 1u) modes[inc0 - 1 - __popc(inc & ((1u << lane) - 1u))] = lane;
    __syncwarp();
    for (int e = lane; e < tor_rec_entries(ks); e += 32) {
      const int i = tor_rec_row(e), j = e - i * (i + 1) / 2, si = i >> 1, sj = j >> 1;
      int r, c;
      tor_rec_source(k, TorRec<S>::kOrder, i, si < R.f ? k - 1 - si : modes[si - R.f], j,
                     sj < R.f ? k - 1 - sj : modes[sj - R.f], r, c);
      ts_st(ws, e, ts_m(Oc, dim, r, c, z));
    }
  }
  if (lane == 0) ts_st(ws, R.t, ts_make(1.0, z));
  __syncwarp();
  bool ok = true;
  const TorRecState root{0, 0};
  for (int m = ks; m > R.f; --m) tor_rec_include<S>(ws, R, m, 1, [&](int) { return root; }, 0, 0, lane, ok);
  S sum = ts_make(0.0, z);
  double acc = 0.0;
  const uint32_t nT = 1u << (R.f - R.mW);
  for (uint32_t Tm = 0; Tm < nT; ++Tm) {
    if (Tm) {
      const int s = __ffs(Tm) - 1;  // the mode decided at level mW + 1 + s is included now
      const int m = R.mW + 1 + s;
      const uint32_t up = Tm & (Tm - 1);
      const TorRecState from = tor_rec_walked(R, root, up);
      tor_rec_include<S>(ws, R, m, 1, [&](int) { return from; }, tor_rec_dfs(R, m - 1), R.f - (m - 1), lane, ok);
    }
    const TorRecState w = tor_rec_walked(R, root, Tm);
    if (R.mW == TAIL + kTorRecWide) {
      tor_rec_levels<S, TAIL + kTorRecWide>(ws, R, w, lane, ok);
    } else {
      for (int m = R.mW; m > R.mt; --m)
        tor_rec_include<S>(ws, R, m, 1 << (R.mW - m), [&](int p) { return tor_rec_node(R, w, m, p); },
                           tor_rec_lev(R, m - 1, 0), R.f + (1 << (R.mW - m)), lane, ok);
    }
    if (lane < (1 << (R.mW - R.mt))) {
      const TorRecState s = tor_rec_node(R, w, R.mt, lane);
      const int in = inc0 + __popc(Tm) + __popc(lane);
      const S t = ts_ld(ws, R.t + s.t, z);
      TorRecSum<S, AUX> f;
      switch (R.mt) {
        case 0: f = tor_rec_tail_load<S, AUX, 0>(ws, s.off, t, 2 * in, rho, ok); break;
        case 1: f = tor_rec_tail_load<S, AUX, 1>(ws, s.off, t, 2 * in, rho, ok); break;
        case 2: f = tor_rec_tail_load<S, AUX, 2>(ws, s.off, t, 2 * in, rho, ok); break;
        default:
          if (TAIL == 3 || R.mt == 3) f = tor_rec_tail_load<S, AUX, 3>(ws, s.off, t, 2 * in, rho, ok);
          else f = tor_rec_tail_load<S, AUX, TAIL>(ws, s.off, t, 2 * in, rho, ok);
      }
      sum = ts_add(sum, ((k - R.mt - in) & 1) ? ts_neg(f.v) : f.v);
      if (AUX == 1) acc += f.a;
      if (AUX == 2) acc = ru_add(ru_add(acc, f.a), ts_sum_err(sum));
    }
    __syncwarp();
  }
  // butterfly over the lanes
#pragma unroll
  for (int mm = 16; mm > 0; mm >>= 1) {
    S o;
    if constexpr (sizeof(S) == sizeof(dd)) o = S{shfl_xor_d(sum.hi, mm), shfl_xor_d(sum.lo, mm)};
    else o = shfl_xor_d(sum, mm);
    sum = ts_add(sum, o);
    if (AUX == 1) acc += shfl_xor_d(acc, mm);
    if (AUX == 2) acc = ru_add(ru_add(acc, shfl_xor_d(acc, mm)), ts_sum_err(sum));
  }
  total = sum;
  aux = acc;
  return __all_sync(0xffffffffu, ok);
}

}  // namespace gbsb
