// eo.cpp -- host side of the even / odd operator form (see eo.hpp).
#include "eo.hpp"

#include <algorithm>
#include <cmath>

namespace dgc {

namespace {

// index of lattice node (i, j): i along s, j along r (setup.cpp's node order)
int node(int N, int i, int j) { return i * (N + 1) - i * (i - 1) / 2 + j; }

// face-node list position -> its image under the reflection
int face_image(int N, int m) {
  const int f = m / (N + 1), d = m % (N + 1);
  return (f == 1 ? 1 : 2 - f) * (N + 1) + N - d;
}

std::vector<int> node_image(int N) {
  std::vector<int> s((size_t)(N + 1) * (N + 2) / 2);
  for (int i = 0; i <= N; ++i)
    for (int j = 0; i + j <= N; ++j) s[node(N, i, j)] = node(N, j, i);
  return s;
}

}  // namespace

std::vector<uint8_t> eo_tables(int N, bool rest) {
  const dgk::EoDims d(N);
  std::vector<uint8_t> t;
  for (int i = 0; i <= N; ++i)
    for (int j = i + 1; i + j <= N; ++j) {
      t.push_back((uint8_t)node(N, i, j));
      t.push_back((uint8_t)node(N, j, i));
    }
  for (int i = 0; 2 * i <= N; ++i) {
    t.push_back((uint8_t)node(N, i, i));
    t.push_back((uint8_t)node(N, i, i));
  }
  for (int c = 0; c < d.fE; ++c) {
    const int m = c;  // face 0, then the first half of face 1
    t.push_back((uint8_t)m);
    t.push_back((uint8_t)face_image(N, m));
  }
  for (int i = 0; i < d.Np; ++i)
    for (int c = 0; c < d.nE; ++c)
      if (t[2 * c] == i || t[2 * c + 1] == i) {
        t.push_back((uint8_t)(c | (t[2 * c] == i ? 0 : 128)));
        break;
      }
  t.push_back(rest ? 1 : 0);
  t.resize((size_t)d.tabBytes(), 0);
  return t;
}

bool eo_symmetric(int N, const std::vector<double>& Dr, const std::vector<double>& Ds, const std::vector<double>& L,
                  const std::vector<double>* M) {
  const dgk::EoDims d(N);
  const std::vector<int> s = node_image(N);
  double big[3] = {0, 0, 0}, off[3] = {0, 0, 0};
  auto see = [&](int w, double x, double y) {
    if (!(std::isfinite(x) && std::isfinite(y))) off[w] = INFINITY;
    big[w] = std::max(big[w], std::fabs(x));
    off[w] = std::max(off[w], std::fabs(x - y));
  };
  for (int i = 0; i < d.Np; ++i) {
    for (int j = 0; j < d.Np; ++j) {
      see(0, Dr[(size_t)i * d.Np + j], Ds[(size_t)s[i] * d.Np + s[j]]);
      if (M) see(2, (*M)[(size_t)i * d.Np + j], (*M)[(size_t)s[i] * d.Np + s[j]]);
    }
    const int NF = 3 * d.Nfp;
    for (int m = 0; m < NF; ++m) see(1, L[(size_t)i * NF + m], L[(size_t)s[i] * NF + face_image(N, m)]);
  }
  for (int w = 0; w < 3; ++w)
    if (!(off[w] <= 1e-13 * big[w])) return false;
  return true;
}

bool eo_constants_cancel(int N, const std::vector<double>& Dr, const std::vector<double>& Ds,
                         const std::vector<double>& L) {
  const dgk::EoDims d(N);
  double big = 0.0, off = 0.0;
  auto see = [&](double x) {
    off = std::isfinite(x) ? std::max(off, std::fabs(x)) : INFINITY;
  };
  for (int i = 0; i < d.Np; ++i) {
    double vr = 0.0, vs = 0.0, l[3] = {0.0, 0.0, 0.0};
    for (int j = 0; j < d.Np; ++j) {
      vr += Dr[(size_t)i * d.Np + j];
      vs += Ds[(size_t)i * d.Np + j];
    }
    for (int m = 0; m < 3 * d.Nfp; ++m) l[m / d.Nfp] += L[(size_t)i * 3 * d.Nfp + m];
    for (double v : l) big = std::max(big, std::fabs(v));
    see(vr - (l[1] - l[2]));
    see(vs - (l[1] - l[0]));
  }
  return off <= 1e-10 * big;
}

std::vector<double> eo_pack(int N, const std::vector<double>& Dr, const std::vector<double>& Ds,
                            const std::vector<double>& L, const std::vector<double>* M, bool rest) {
  const dgk::EoDims d(N);
  const std::vector<uint8_t> t = eo_tables(N);
  const int NF = 3 * d.Nfp;
  // coefficient of output (row c, sum or difference) from input (column k, sum
  // or difference) of the matrix f(i, j), tables rt (rows) and ct (columns)
  auto coef = [](auto&& f, const uint8_t* rt, bool ro, const uint8_t* ct, bool co) {
    const int a = rt[0], b = rt[1], x = ct[0], y = ct[1];
    const double rs = ro ? -1.0 : 1.0, cs = co ? -1.0 : 1.0;
    if (a == b && x == y) return f(a, x);
    if (a == b) return (f(a, x) + cs * f(a, y)) / 2;
    if (x == y) return (f(a, x) + rs * f(b, x)) / 2;
    return (f(a, x) + cs * f(a, y) + rs * (f(b, x) + cs * f(b, y))) / 4;
  };
  const uint8_t* nt = t.data();
  const uint8_t* ft = t.data() + 2 * d.nE;
  std::vector<double> out((size_t)d.kK() + d.kL() + (M ? d.kM() : 0), 0.0);
  for (int c = 0; c < d.Np; ++c)
    for (int r = 0; r < d.Np; ++r) {
      const bool co = c >= d.nE, ro = r >= d.nE;
      const double sg = (co == ro) != rest ? 1.0 : -1.0;  // D+ keeps the parity, D- flips it
      auto D = [&](int i, int j) {
        return 0.5 * (Dr[(size_t)i * d.Np + j] + sg * Ds[(size_t)i * d.Np + j]);
      };
      out[(size_t)c * d.Np + r] =
          coef(D, nt + 2 * (ro ? r - d.nE : r), ro, nt + 2 * (co ? c - d.nE : c), co);
    }
  double* l = out.data() + d.kK();
  auto Lf = [&](int i, int m) { return L[(size_t)i * NF + m]; };
  for (int r = 0; r < d.Np; ++r) {
    const bool ro = r >= d.nE, co = ro != rest;
    for (int c = 0; c < (co ? d.fO : d.fE); ++c)
      l[(size_t)c * d.Np + r] = coef(Lf, nt + 2 * (ro ? r - d.nE : r), ro, ft + 2 * c, co);
  }
  if (M) {
    double* m = out.data() + d.kK() + d.kL();
    auto Mf = [&](int i, int j) { return (*M)[(size_t)i * d.Np + j]; };
    for (int r = 0; r < d.Np; ++r) {
      const bool ro = r >= d.nE;
      for (int c = 0; c < (ro ? d.nO : d.nE); ++c)
        m[(size_t)c * d.Np + r] =
            ((c < d.nO ? 2 : 1) * coef(Mf, nt + 2 * (ro ? r - d.nE : r), ro, nt + 2 * c, ro));
    }
  }
  return out;
}

}  // namespace dgc
