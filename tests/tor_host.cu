// Host restatement of the torontonian recursion's walk (gbskernels_b200/csrc/tor_rec.cuh):
// the kernel's own layout and node functions (all __host__ __device__) drive a sequential
// walk over a workspace of exactly the size the planner asks for, every access checked
// against it, every word read checked to have been written.  The CPU test
// tests/test_tor_rec_walk.py compares the sums with the oracle.
#include <cmath>
#include <vector>

#include "tor_rec.cuh"

using namespace gbsb;

namespace {
struct Walk {
  TorRecLayout R;
  int bad = 0;
  std::vector<double> w;
  std::vector<char> set;
  double get(int i) {
    if (i < 0 || i >= (int)w.size() || !set[i]) { ++bad; return 1.0; }
    return w[i];
  }
  void put(int i, double v) {
    if (i < 0 || i >= (int)w.size()) { ++bad; return; }
    w[i] = v;
    set[i] = 1;
  }
  template <typename Src>
  void include(int m, int N, Src src, int dst, int dt) {  // tor_rec_include
    const int ra = (2 * m - 2) * (2 * m - 1) / 2, rb = (2 * m - 1) * m, rows = 2 * m - 2, E = tor_rec_entries(m - 1);
    if (N > (1 << (kTorRecWide - 1)) && N > 1) ++bad;
    for (int p = 0; p < N; ++p) {
      const TorRecState s = src(p);
      const double i0 = 1 / std::sqrt(get(s.off + ra + 2 * m - 2)), lb = get(s.off + rb + 2 * m - 2) * i0;
      const double i1 = 1 / std::sqrt(get(s.off + rb + 2 * m - 1) - lb * lb);
      put(R.piv + 3 * p, i0);
      put(R.piv + 3 * p + 1, lb);
      put(R.piv + 3 * p + 2, i1);
      put(R.t + dt + p, get(R.t + s.t) * i0 * i1);
    }
    for (int p = 0; p < N; ++p)
      for (int j = 0; j < rows; ++j) {
        const TorRecState s = src(p);
        const double l0 = get(s.off + ra + j) * get(R.piv + 3 * p);
        put(R.lc + 2 * (p * rows + j), l0);
        put(R.lc + 2 * (p * rows + j) + 1, (get(s.off + rb + j) - l0 * get(R.piv + 3 * p + 1)) * get(R.piv + 3 * p + 2));
      }
    for (int q0 = 0; q0 < N * E; q0 += 32) {  // 32 lanes read, then write
      double v[32];
      for (int q = q0; q < N * E && q < q0 + 32; ++q) {
        const int p = q / E, e = q - p * E, i = tor_rec_row(e), j = e - i * (i + 1) / 2;
        const int ci = R.lc + 2 * (p * rows + i), cj = R.lc + 2 * (p * rows + j);
        v[q - q0] = get(src(p).off + e) - get(ci) * get(cj) - get(ci + 1) * get(cj + 1);
      }
      for (int q = q0; q < N * E && q < q0 + 32; ++q) put(dst + q, v[q - q0]);
    }
  }
  double tail(std::vector<double> Z, int M, double t) {
    if (M == 0) return t;
    const int ra = (2 * M - 2) * (2 * M - 1) / 2, rb = (2 * M - 1) * M, r = 2 * M - 2;
    const double i0 = 1 / std::sqrt(Z[ra + r]), lb = Z[rb + r] * i0, i1 = 1 / std::sqrt(Z[rb + r + 1] - lb * lb);
    std::vector<double> Y(r * (r + 1) / 2 + 1), l0(r + 1), l1(r + 1);
    for (int j = 0; j < r; ++j) {
      l0[j] = Z[ra + j] * i0;
      l1[j] = (Z[rb + j] - l0[j] * lb) * i1;
    }
    for (int i = 0; i < r; ++i)
      for (int j = 0; j <= i; ++j) Y[i * (i + 1) / 2 + j] = Z[i * (i + 1) / 2 + j] - l0[i] * l0[j] - l1[i] * l1[j];
    return tail(Y, M - 1, t * i0 * i1) - tail(Z, M - 1, t);
  }
};
}  // namespace

// Sum over the patterns [lo, lo + 1) of the first g modes of the torontonian of O (2k x 2k);
// tail, W: the scalar type's (4, 1 binary64; 3, 2 double-double).  Returns the number of
// accesses outside the workspace or of unwritten words.
extern "C" int t_tor_rec_item(const double* O, int k, int g, unsigned lo, int is_dd, int cert, double* out) {
  const int f = tor_rec_free(k, g), dim = 2 * k, W = is_dd ? 2 : 1;
  Walk x;
  x.R = tor_rec_layout(k, f, is_dd ? 3 : 4, cert != 0, W);
  const TorRecLayout& R = x.R;
  if (R.total * W > tor_rec_ws(k, g, is_dd != 0, cert != 0)) ++x.bad;
  // the certificate's scratch (a packed matrix and its scalings) stays below rho
  if (cert && (k * (2 * k + 1) + 2 * k > R.rho * W || 2 * k + 1 > (R.total - R.rho) * W)) ++x.bad;
  // the entry maps of a full breadth-first walk: columns, node and place of every entry
  const int tail = is_dd ? 3 : 4;
  if (R.mW == tail + kTorRecWide)
    for (int m = R.mW; m > tail; --m) {
      const int E = tor_rec_entries(m - 1), N = 1 << (R.mW - m), mo = tor_rec_map_off(tail, m);
      if (R.lev + mo != tor_rec_lev(R, m - 1, 0)) ++x.bad;
      for (int q = 0; q < N * E; ++q) {
        const unsigned w = is_dd ? tor_rec_map<3>(mo + q) : tor_rec_map<4>(mo + q);
        const int p = q / E, e = q - p * E, i = tor_rec_row(e), j = e - i * (i + 1) / 2;
        if ((int)(w & 0xfffu) != p * (2 * m - 2) + i || (int)(w >> 12 & 0xfffu) != p * (2 * m - 2) + j || (int)(w >> 24) != p)
          ++x.bad;
      }
    }
  if (R.lc & 1) ++x.bad;  // column pairs on 16 bytes
  double sum = 0.0;
  const int g2 = k - f;
  for (unsigned p = 0; p < (1u << (g2 - g)); ++p) {
    const unsigned pat = tor_rec_pattern(lo, p, g, g2);
    x.w.assign(R.rho, 0.0);
    x.set.assign(R.rho, 0);
    const int inc0 = __builtin_popcount(pat), ks = f + inc0;
    std::vector<int> modes;  // included ones of the first g2, the last first
    for (int j = g2 - 1; j >= 0; --j)
      if ((pat >> j) & 1u) modes.push_back(j);
    if (inc0 > 2 * (1 << kTorRecWide) / 2 || R.noff + (1 << kTorRecWide) / 2 > R.rho) ++x.bad;  // the list's place
    auto mode = [&](int r) { return r / 2 < f ? k - 1 - r / 2 : modes[r / 2 - f]; };
    for (int e = 0; e < tor_rec_entries(ks); ++e) {
      const int i = tor_rec_row(e), j = e - i * (i + 1) / 2;
      int a, b;
      tor_rec_source(k, is_dd ? TorRec<dd>::kOrder : TorRec<double>::kOrder, i, mode(i), j, mode(j), a, b);
      x.put(e, (a == b ? 1.0 : 0.0) - O[a * dim + b]);
    }
    x.put(R.t, 1.0);
    const TorRecState root{0, 0};
    for (int m = ks; m > f; --m) x.include(m, 1, [&](int) { return root; }, 0, 0);
    for (unsigned Tm = 0; Tm < (1u << (R.f - R.mW)); ++Tm) {
      if (Tm) {
        const int s = __builtin_ctz(Tm), m = R.mW + 1 + s;
        const TorRecState from = tor_rec_walked(R, root, Tm & (Tm - 1));
        x.include(m, 1, [&](int) { return from; }, tor_rec_dfs(R, m - 1), R.f - (m - 1));
      }
      const TorRecState w = tor_rec_walked(R, root, Tm);
      for (int m = R.mW; m > R.mt; --m)
        x.include(m, 1 << (R.mW - m), [&](int p) { return tor_rec_node(R, w, m, p); }, tor_rec_lev(R, m - 1, 0),
                  R.f + (1 << (R.mW - m)));
      for (int p = 0; p < (1 << (R.mW - R.mt)); ++p) {
        const TorRecState s = tor_rec_node(R, w, R.mt, p);
        std::vector<double> Z;
        for (int e = 0; e < tor_rec_entries(R.mt); ++e) Z.push_back(x.get(s.off + e));
        Z.push_back(0.0);
        const double v = x.tail(Z, R.mt, x.get(R.t + s.t));
        sum += ((k - R.mt - inc0 - __builtin_popcount(Tm) - __builtin_popcount(p)) & 1) ? -v : v;
      }
    }
  }
  *out = sum;
  return x.bad;
}
