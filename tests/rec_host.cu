// Host restatement of the hafnian recursion's walk (gbskernels_b200/csrc/haf_rec.cuh):
// the kernel's own layout, lane and node functions (all __host__ __device__) drive a
// sequential walk over a workspace of exactly the size the planner asks for, every
// access checked against it, every coefficient read checked to have been written.  With
// is_dd the double-double steps' memory behaviour: e polynomials apart (of a whole level in
// the breadth-first part), a lane per coefficient with no lane writing what another one
// reads or writes before the next barrier, g last.  (The arithmetic is binary64 either
// way.)  The CPU test tests/test_haf_rec_walk.py compares the sums with the oracle.
#include <algorithm>
#include <complex>
#include <cstdio>
#include <vector>

#include "haf_rec.cuh"

using namespace gbsb;
typedef std::complex<double> Z;

namespace {
struct Walk {
  int n, loop, is_dd = 0, bad = 0;
  std::vector<Z> w;
  std::vector<char> set;
  // accesses since the last barrier: the one task that read / wrote a word (0 none, -1
  // several readers); `task` 0 switches the check off
  int task = 0;
  std::vector<int> reader, writer;
  Z get(int i) {
    if (i < 0 || i >= (int)w.size() || !set[i]) { ++bad; return 0.0; }
    if (task) {
      if (writer[i] && writer[i] != task) ++bad;
      reader[i] = reader[i] == 0 || reader[i] == task ? task : -1;
    }
    return w[i];
  }
  void put(int i, Z v) {
    if (i < 0 || i >= (int)w.size()) { ++bad; return; }
    if (task) {
      if ((writer[i] && writer[i] != task) || (reader[i] && reader[i] != task)) ++bad;
      writer[i] = task;
    }
    w[i] = v;
    set[i] = 1;
  }
  void barrier() {
    reader.assign(w.size(), 0);
    writer.assign(w.size(), 0);
    task = 0;
  }
  // haf_rec_coef
  Z coef(const HafRecLane& L, int c) {
    Z x = c <= L.lim ? get(L.own + c * L.str) : Z(0.0);
    const int top = c - 1;
    for (int u = std::max(0, top - L.limb); u <= std::min(L.lim, top); ++u)
      x += get(L.a1 + u * L.str) * get(L.b1 + (top - u) * L.bstr);
    for (int u = std::max(0, top - L.lim2); u <= std::min(L.lim2, top); ++u)
      x += get(L.a2 + u * L.str) * get(L.b2 + (top - u) * L.str);
    return x;
  }
  // the double-double branch of haf_rec_step
  void coefs(int T, int np, const std::vector<HafRecLane>& ls) {
    barrier();
    const int cnt = (int)ls.size(), H = (T + 3) / 2;
    for (int x = 0; x < cnt * H; ++x) {
      const HafRecLane& L = ls[x / H];
      const int h = x % H, h2 = T + 1 - h;
      if (L.a1 == L.own) continue;
      task = 1 + x;
      put(L.dst + h * L.dstr, coef(L, h));
      if (h2 != h) put(L.dst + h2 * L.dstr, coef(L, h2));
    }
    const int states = cnt / (np + 1), all = states * (T + 2);
    std::vector<Z> v(all);
    for (int x0 = 0; x0 < all; x0 += 32) {  // 32 lanes form theirs, a barrier, then they store
      for (int x = x0; x < all && x < x0 + 32; ++x) {
        task = 1 + cnt * H + x;
        v[x] = coef(ls[(x / (T + 2)) * (np + 1) + np], x % (T + 2));
      }
      for (int x = x0; x < all && x < x0 + 32; ++x) {
        const HafRecLane& L = ls[(x / (T + 2)) * (np + 1) + np];
        task = 0;
        const int i = L.dst + (x % (T + 2)) * L.dstr;
        put(i, v[x]);
        if (i >= 0 && i < (int)w.size()) writer[i] = -2;  // no barrier before the next round's reads
      }
    }
    barrier();
  }
  std::vector<Z> poly(int o, int str, int lim, int T) {
    std::vector<Z> v(T + 1, 0.0);
    for (int c = 0; c <= T && c <= lim; ++c) v[c] = get(o + c * str);
    return v;
  }
  // one lane of haf_rec_op
  std::vector<Z> op(int T, const HafRecLane& L) {
    std::vector<Z> acc = poly(L.own, L.str, L.lim, T + 1);
    auto add = [&](const std::vector<Z>& a, const std::vector<Z>& b) {
      for (int u = 0; u <= T; ++u)
        for (int v = 0; u + v <= T; ++v) acc[u + v + 1] += a[u] * b[v];
    };
    add(poly(L.a1, L.str, L.lim, T), poly(L.b1, L.bstr, L.limb, T));
    add(poly(L.a2, L.str, L.lim2, T), poly(L.b2, L.str, L.lim2, T));
    return acc;
  }
  // haf_rec_e of every coefficient
  void e(const HafRecState& s, int m, int eo, int estr) {
    const int V = 2 * m + 1, T = n - m;
    const int r1 = s.off + (V - 1) * (V - 2) / 2, r0 = s.off + (V - 2) * (V - 3) / 2;
    std::vector<Z> x = poly(r1 + V - 2, s.str, s.lim, T), a = poly(r0, s.str, s.lim, T), b = poly(r1, s.str, s.lim, T);
    for (int u = 0; u <= T; ++u)
      for (int v = 0; u + v <= T; ++v) x[u + v] += a[u] * b[v];
    for (int c = 0; c <= T; ++c) put(eo + c * estr, x[c]);
  }
  void lanes(int T, const std::vector<HafRecLane>& ls) {  // 32 lanes at a time: all read, then all write
    for (size_t q0 = 0; q0 < ls.size(); q0 += 32) {
      std::vector<std::vector<Z>> r;
      for (size_t q = q0; q < ls.size() && q < q0 + 32; ++q) r.push_back(op(T, ls[q]));
      for (size_t q = q0; q < ls.size() && q < q0 + 32; ++q)
        for (int c = 0; c < T + 2; ++c) put(ls[q].dst + c * ls[q].dstr, r[q - q0][c]);
    }
  }
  HafRecState take(const HafRecState& s, int m, int scratch, int dst, int dstr) {
    const int np = haf_rec_polys(m - 1, loop);
    const bool own_e = is_dd || dst == s.off;  // in place (and double-double): e apart, else where g' goes
    const int eo = own_e ? scratch : dst + dstr - 1, estr = own_e ? 1 : dstr;
    if (loop) e(s, m, eo, estr);
    std::vector<HafRecLane> ls;
    for (int q = 0; q <= np; ++q) ls.push_back(haf_rec_lane(s, m, loop, np, q, true, 0, eo, estr, dst, dstr));
    if (is_dd) coefs(n - m, np, ls);
    else lanes(n - m, ls);
    return HafRecState{dst, dstr, n - m + 1};
  }
  Z wide(const HafRecState& root, const HafRecLayout& R, int odd) {
    for (int m = R.mB; m >= 2; --m) {
      const int np = haf_rec_polys(m - 1, loop), dstr = np + 1, dsz = (n - m + 2) * dstr, ec = n - m + 1;
      const int eo = is_dd ? R.e : R.lev[m - 1] + dstr - 1, epn = is_dd ? ec : dsz, estr = is_dd ? 1 : dstr;
      std::vector<HafRecLane> ls;
      if (loop)
        for (int p = 0; p < (1 << (R.mB - m)); ++p) e(haf_rec_node(root, R, 0, n, loop, m, p), m, eo + p * epn, estr);
      for (int p = 0; p < (1 << (R.mB - m)); ++p)
        for (int q = 0; q <= np; ++q)
          ls.push_back(haf_rec_lane(haf_rec_node(root, R, 0, n, loop, m, p), m, loop, np, q, true, 0, eo + p * epn, estr,
                                    R.lev[m - 1] + p * dsz, dstr));
      if (is_dd) coefs(n - m, np, ls);
      else lanes(n - m, ls);
    }
    Z f = 0.0;
    for (int p = 0; p < (1 << (R.mB - 1)); ++p) {
      const HafRecState s = haf_rec_node(root, R, 0, n, loop, 1, p);
      std::vector<Z> g = poly(s.off + s.str - 1, s.str, s.lim, n - 1), e = poly(s.off + (loop ? 2 : 0), s.str, s.lim, n - 1);
      if (loop) {
        std::vector<Z> x = poly(s.off, s.str, s.lim, n - 1), y = poly(s.off + 1, s.str, s.lim, n - 1);
        for (int u = 0; u < n; ++u)
          for (int v = 0; u + v < n; ++v) e[u + v] += x[u] * y[v];
      }
      Z t = 0.0;
      for (int c = 0; c < n; ++c) t += g[c] * e[n - 1 - c];
      f += ((__builtin_popcount(p) + odd) & 1) ? -t : t;
    }
    return f;
  }
};
}  // namespace

// Signed sum over the subsets [lo, lo + 2^clog) of the (loop) hafnian of A (2n x 2n).
// Returns the number of accesses outside the workspace, of unwritten words or (is_dd)
// between two lanes without a barrier.
extern "C" int t_haf_rec_sum(const double* A, int n, int loop, int is_dd, unsigned lo, int clog, double* out) {
  const int N = 2 * n;
  const int m0 = clog < kHafRecBlock ? clog : kHafRecBlock;
  const HafRecLayout R = haf_rec_layout(n, m0, loop, is_dd != 0);
  Walk W;
  W.n = n;
  W.loop = loop;
  W.is_dd = is_dd;
  const int width = is_dd ? 4 : 2;
  if (width * R.total > haf_rec_ws(n, loop != 0, width)) ++W.bad;
  auto a = [&](int r, int c) { return Z(A[2 * (r * N + c)], A[2 * (r * N + c) + 1]); };
  const int str0 = haf_rec_polys(m0, loop) + 1;
  Z sum = 0.0;
  for (unsigned b = 0; b < (1u << (clog - m0)); ++b) {
    W.w.assign(R.total, 0.0);
    W.set.assign(R.total, 0);
    const unsigned pat = (lo >> m0) + b;
    const int left = (n - m0) - __builtin_popcount(pat);
    HafRecState s{0, haf_rec_polys(n, loop) + 1, 0};
    for (int j = 1; j < N + loop; ++j)
      for (int k = 0; k < j; ++k)
        W.put(j * (j - 1) / 2 + k, loop && k == 0 ? a(j - 1, j - 1) : 0.5 * (a(j - loop, k - loop) + a(k - loop, j - loop)));
    W.put(haf_rec_polys(n, loop), 1.0);
    for (int m = n; m > m0; --m)
      if ((pat >> (m - 1 - m0)) & 1u) s = W.take(s, m, R.e, s.off == 0 ? R.pz : 0, haf_rec_polys(m - 1, loop) + 1);
    if (s.off != 0 || s.str != str0) {
      for (int c = 0; c <= s.lim; ++c)
        for (int q = 0; q < str0; ++q) W.put(c * str0 + q, W.get(s.off + c * s.str + (q == str0 - 1 ? s.str - 1 : q)));
      s.off = 0;
      s.str = str0;
    }
    if (m0 == 0) {
      const Z f = s.lim >= n ? W.get(n * str0 + str0 - 1) : Z(0.0);
      sum += (left & 1) ? -f : f;
      continue;
    }
    const int d = m0 - R.mB, par = left + d + R.mB - 1;
    for (int t = 0; t < (1 << d); ++t) {
      HafRecState r = s;
      if (d == 2 && t == 1) r = W.take(s, 6, R.e, R.b5, haf_rec_polys(5, loop) + 1);
      else if (t > 0) s = r = W.take(s, (d == 2 && t == 2) ? 7 : 6, R.e, 0, str0);
      sum += W.wide(r, R, (par - __builtin_popcount(t)) & 1);
    }
  }
  out[0] = sum.real();
  out[1] = sum.imag();
  return W.bad;
}
