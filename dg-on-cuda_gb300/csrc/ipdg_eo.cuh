// ipdg_eo.cuh -- the two passes of laplace_2d (ipdg.cuh) in the even / odd basis
// of the reflection r <-> s (eo.hpp): the FP64 path of the operator, of its CG
// iteration and of the refinement residuals.
//
// Bound by the FP64 pipe like the FP64 stage kernel (dg_rhs_eo.cuh): the
// node-by-node passes kept it over 90 % busy.  FP64 instructions per element at
// N = 4, grad + div + mass: 1.4k instead of 2.7k --
//   * D+ and D- of a field take Np^2 products where Dr and Ds took 2 Np^2, and
//     the divergence is one D+ p + D- m, p and m combined from (qx, qy) with the
//     element's constant geometry: 2 Np^2 instead of 6 Np^2 for both passes, LIFT
//     and M half of theirs;
//   * -1/J (the SPD form: J (1/J) = 1), faceJ, normals and penalties are
//     multiplied into per-element constants, once per laplace handle.
// One tile per CTA (eo_pick_tiles); set-up data are fetched
// before the wait for the previous launch, exterior traces while the tile's own
// fields arrive.
#pragma once

#include "eo.hpp"
#include "ipdg.cuh"

namespace dgk {

template <int N>
struct IpdgEo {
  using R = double;
  using O = Order<N>;
  static constexpr EoDims D{N};
  static constexpr int Np = O::Np, NpP = O::NpP, Nfp = O::Nfp;
  static constexpr int nE = D.nE, nO = D.nO, fE = D.fE, fO = D.fO;
  static constexpr int TE = 256 / Np;
  static constexpr int FSTR = 4 * fE;  // grad: x | y, div: one, each [fE sums | fE differences]
  static constexpr int CSTR = 16;
  static constexpr uint32_t kOpsG = (D.kK() + D.kL()) * 8, kOpsD = kOpsG + D.kM() * 8, kTab = D.tabBytes();
  static constexpr uint32_t kF = TE * NpP * 8;  // one field
  static constexpr uint32_t oBar = 0, oTab = 32, oGeom = oTab + kTab, oNbr = oGeom + TE * 16 * 8, oC = oNbr + TE * 16,
                            oFld = oC + TE * CSTR * 8, oIn = oFld + 3 * kF,
                            oF = oIn + TE * 2 * Np * 8, oRed = (oF + TE * FSTR * 8 + 15) / 16 * 16, oOps = oRed + 16 * 8;
  static constexpr uint32_t kSmemGrad = oOps + kOpsG, kSmemDiv = oOps + kOpsD;
  static_assert(TE * fE <= 256, "one face-node pair per thread");
  static_assert(oGeom % 16 == 0 && oFld % 16 == 0 && kF % 16 == 0 && oRed % 16 == 0 && kOpsG % 16 == 0, "alignment");
  // FP64 instructions per item (eo_pick_tiles)
  static constexpr EoCost kCostGrad{Np + 2 * fE + 6, 12, 2, 0}, kCostDiv{Np + fE + nE + 5, 14, 8, 0};
};

// Per-element constants, in the strong form's signs or with the SPD form's rows
// times -J: (rx +- sx, ry +- sy) s, then per face h nx, h ny and 2 tau h with
// h = faceJ / 2 times -1/J (SPD: J (1/J) = 1), and -J.  The weak form is minus the strong one.
// Laplace handles keep both forms (k_eo_consts), 128 bytes per element and form, read
// in place of geometry and penalties: forming them in every launch was a tenth of a
// pass's FP64 instructions (SPD apply, K = 65522, N = 5: 309 -> 294 us; gradient and
// divergence, K = 131072, N = 4: 373 -> 338 us).
enum IpdgEoConst : int { IC_P1 = 0, IC_P2 = 1, IC_Q1 = 2, IC_Q2 = 3, IC_F = 4, IC_MJ = 13 };

// value group v (0 .. 7: the volume factors, the faces, -J) of an element's constants
__device__ __forceinline__ void eo_const(int v, bool spd, const double* g, const double* tau, double* c) {
  const double sv = spd ? g[14] : 1.0, sf = spd ? 1.0 : g[4];  // g[14] = -J, g[4] = -1/J
  if (v < 2) c[IC_P1 + v] = sv * (v ? g[0] - g[2] : g[0] + g[2]);
  else if (v < 4) c[IC_Q1 + v - 2] = sv * (v == 3 ? g[1] - g[3] : g[1] + g[3]);
  else if (v < 7) {
    const int f = v - 4;
    const double h = 0.5 * g[5 + f] * sf;
    c[IC_F + 3 * f] = h * g[8 + f];
    c[IC_F + 3 * f + 1] = h * g[11 + f];
    c[IC_F + 3 * f + 2] = tau ? 2.0 * tau[f] * h : 0.0;
  } else {
    c[IC_MJ] = g[14];
    c[IC_MJ + 1] = c[IC_MJ + 2] = 0.0;
  }
}

// views of a CTA's shared memory, and the parts both passes share
template <int N>
struct IpdgEoTile {
  using C = IpdgEo<N>;
  unsigned char* smem;
  __device__ uint64_t* bar() const { return reinterpret_cast<uint64_t*>(smem + C::oBar); }
  __device__ const uint8_t* nodes() const { return smem + C::oTab; }
  __device__ const uint8_t* faces() const { return smem + C::oTab + 2 * C::nE; }
  __device__ const uint8_t* inverse() const { return smem + C::oTab + 2 * C::nE + 2 * C::fE; }
  __device__ const double* geom() const { return reinterpret_cast<const double*>(smem + C::oGeom); }
  __device__ const int4* nbr() const { return reinterpret_cast<const int4*>(smem + C::oNbr); }
  __device__ double* consts() const { return reinterpret_cast<double*>(smem + C::oC); }
  __device__ double* field(int i) const { return reinterpret_cast<double*>(smem + C::oFld + i * C::kF); }
  __device__ double* in() const { return reinterpret_cast<double*>(smem + C::oIn); }
  __device__ double* flux() const { return reinterpret_cast<double*>(smem + C::oF); }
  __device__ double* red() const { return reinterpret_cast<double*>(smem + C::oRed); }
  __device__ const double* K() const { return reinterpret_cast<const double*>(smem + C::oOps); }
  __device__ const double* L() const { return K() + C::D.kK(); }
  __device__ const double* M() const { return L() + C::D.kL(); }

  // operators without the symmetry: their rest's row r (eo.hpp), NULL without one
  __device__ const double* rest(const IpdgParams& p, int r) const {
    return smem[C::oTab + C::D.flag()] ? reinterpret_cast<const double*>(p.tab_eo + C::kTab) + r : nullptr;
  }

  // set-up data of the elements k0 .. k0 + ne - 1; false if a wait expired
  __device__ bool setup(const IpdgParams& p, int k0, int ne, uint32_t ops, bool spd) const {
    if (threadIdx.x == 0) {
      mbar_init(bar(), 1);
      mbar_init(bar() + 1, 1);
      fence_barrier_init();
      mbar_arrive_expect_tx(bar(), ops + C::kTab + ne * (16 * 8 + 16));
      bulk_g2s(smem + C::oOps, p.mats_eo, ops, bar());
      bulk_g2s(smem + C::oTab, p.tab_eo, C::kTab, bar());
      // the constants, or the geometry they are formed from
      if (p.consts) bulk_g2s(smem + C::oC, p.consts + ((size_t)(spd ? p.K : 0) + k0) * 16, ne * 16 * 8, bar());
      else bulk_g2s(smem + C::oGeom, static_cast<const double*>(p.geom) + (size_t)k0 * 16, ne * 16 * 8, bar());
      bulk_g2s(smem + C::oNbr, p.nbr + k0, ne * 16, bar());
    }
    __syncthreads();
    return __syncthreads_and(mbar_wait(bar(), 0, p.status));
  }
  // the constants of handles that keep none (gradient and divergence of advection handles)
  __device__ void constants(const IpdgParams& p, int ne) const {
    if (p.consts) return;
    for (int x = 255 - (int)threadIdx.x; x < ne * 8; x += 256)
      eo_const(x & 7, false, geom() + (x >> 3) * 16, nullptr, consts() + (x >> 3) * C::CSTR);
  }

  // inputs of the gradient rows: sums and differences of the field u
  __device__ void sum_diff(const double* u, int ne) const {
    constexpr int nE = C::nE;
    for (int x = 255 - (int)threadIdx.x; x < ne * nE; x += 256) {
      const int e = x / nE, c = x - e * nE;
      double* i = in() + e * 2 * C::Np + c;
      const double ua = u[e * C::NpP + nodes()[2 * c]];
      if (c < C::nO) {
        const double ub = u[e * C::NpP + nodes()[2 * c + 1]];
        i[0] = ua + ub;
        i[nE] = ua - ub;
      } else {
        i[0] = ua;
      }
    }
  }
  // inputs of the divergence rows: p | m, the combinations of the fields (x, y)
  // that D+ and D- act on
  __device__ void combine(const double* fx, const double* fy, int ne) const {
    constexpr int nE = C::nE, Np = C::Np;
    for (int x = 255 - (int)threadIdx.x; x < ne * nE; x += 256) {
      const int e = x / nE, c = x - e * nE;
      const double* cc = consts() + e * C::CSTR;
      const double p1 = cc[IC_P1], p2 = cc[IC_P2], q1 = cc[IC_Q1], q2 = cc[IC_Q2];
      double* i = in() + e * 2 * Np + c;
      const int na = e * C::NpP + nodes()[2 * c], nb = e * C::NpP + nodes()[2 * c + 1];
      const double xa = fx[na], ya = fy[na];
      if (c < C::nO) {
        const double xb = fx[nb], yb = fy[nb];
        const double xs = xa + xb, ys = ya + yb, xd = xa - xb, yd = ya - yb;
        i[0] = fma(p1, xs, q1 * ys);
        i[Np] = fma(p2, xs, q2 * ys);
        i[nE] = fma(p1, xd, q1 * yd);
        i[Np + nE] = fma(p2, xd, q2 * yd);
      } else {
        i[0] = fma(p1, xa, q1 * ya);
        i[Np] = fma(p2, xa, q2 * ya);
      }
    }
  }
  // node r's value from the sums and differences ro[Np] of its element's rows
  // (NEG: minus it)
  template <bool NEG = false>
  __device__ double node(const double* ro, int r) const {
    const int inv = inverse()[r], c = inv & 127;
    const double v = NEG ? -ro[c] : ro[c];
    if (c >= C::nO) return v;
    const double o = ro[C::nE + c];
    return ((inv & 128) != 0) != NEG ? v - o : v + o;
  }
  // gradient rows of the tile from sum_diff's inputs and the x | y flux sums and
  // differences, then both components by node
  template <bool NEG = false>
  __device__ void grad_rows(const IpdgParams& p, int ne, int k0, double* ox, double* oy) const {
    constexpr int Np = C::Np, nE = C::nE, nO = C::nO, fE = C::fE;
    const int e = (int)threadIdx.x / Np, r = (int)threadIdx.x - e * Np;
    const bool act = e < ne;
    double qx = 0.0, qy = 0.0;
    if (act) {
      const bool sum = r < nE;
      const double* k = K() + r;
      const double* x = in() + e * 2 * Np;
      const double* c = consts() + e * C::CSTR;
      double s1 = 0.0, s2 = 0.0;
#pragma unroll 4
      for (int j = 0; j < nE; ++j) s1 = fma(k[j * Np], x[j], s1);
      k += nE * Np;
      x += nE;
#pragma unroll 4
      for (int j = 0; j < nO; ++j) s2 = fma(k[j * Np], x[j], s2);
      if (const double* k2 = rest(p, r)) {
        x = in() + e * 2 * Np;
#pragma unroll 1
        for (int j = 0; j < Np; ++j) (j < nE ? s2 : s1) = fma(k2[j * Np], x[j], j < nE ? s2 : s1);
      }
      const int ia = sum ? 0 : 1;  // D+ u is s1 in a sum row, s2 in a difference row
      qx = fma(c[IC_P1 + ia], s1, c[IC_P2 - ia] * s2);
      qy = fma(c[IC_Q1 + ia], s1, c[IC_Q2 - ia] * s2);
      const double* l = L() + r;
      const double* f = flux() + e * C::FSTR + (sum ? 0 : fE);
#pragma unroll 4
      for (int m = 0; m < fE; ++m) {
        const double ll = l[m * Np];
        qx = fma(ll, f[m], qx);
        qy = fma(ll, f[2 * fE + m], qy);
      }
      if (const double* l2 = rest(p, r)) {
        f = flux() + e * C::FSTR + (sum ? fE : 0);
#pragma unroll 1
        for (int m = 0; m < (sum ? C::fO : fE); ++m) {
          qx = fma(l2[C::D.kK() + m * Np], f[m], qx);
          qy = fma(l2[C::D.kK() + m * Np], f[2 * fE + m], qy);
        }
      }
    }
    __syncthreads();
    double* ro = in() + e * 2 * Np;
    if (act) {
      ro[r] = qx;
      ro[Np + r] = qy;
    }
    __syncthreads();
    if (act) {
      const size_t o = (size_t)(k0 + e) * C::NpP + r;
      ox[o] = node<NEG>(ro, r);
      oy[o] = node<NEG>(ro + Np, r);
    }
  }
  // divergence row r of element e from combine's inputs and the flux sums and differences
  __device__ double div_row(const IpdgParams& p, int e, int r) const {
    constexpr int Np = C::Np, nE = C::nE, nO = C::nO, fE = C::fE;
    const bool sum = r < nE;
    const double* k = K() + r;
    const double* x = in() + e * 2 * Np;
    // sum rows take p's sums and m's differences, difference rows the others
    const double* u = x + (sum ? 0 : Np);
    const double* v = x + (sum ? Np : 0) + nE;
    double s1 = 0.0, s2 = 0.0;
#pragma unroll 4
    for (int j = 0; j < nE; ++j) s1 = fma(k[j * Np], u[j], s1);
    k += nE * Np;
#pragma unroll 4
    for (int j = 0; j < nO; ++j) s2 = fma(k[j * Np], v[j], s2);
    const double* l = L() + r;
    const double* f = flux() + e * C::FSTR + (sum ? 0 : fE);
#pragma unroll 4
    for (int m = 0; m < fE; ++m) s1 = fma(l[m * Np], f[m], s1);
    if (const double* k2 = rest(p, r)) {
      // sum rows: m's sums and p's differences, difference rows the others
#pragma unroll 1
      for (int j = 0; j < Np; ++j) s2 = fma(k2[j * Np], x[((j < nE) == sum ? Np : 0) + j], s2);
      f = flux() + e * C::FSTR + (sum ? fE : 0);
#pragma unroll 1
      for (int m = 0; m < (sum ? C::fO : fE); ++m) s2 = fma(k2[C::D.kK() + m * Np], f[m], s2);
    }
    return s1 + s2;
  }
};

// ---------------------------------------------------------------- grad pass
template <int N, int MODE>
__global__ void __launch_bounds__(256) ipdg_grad_eo_kernel(const IpdgParams p) {
  using C = IpdgEo<N>;
  constexpr int Np = C::Np, NpP = C::NpP, Nfp = C::Nfp, nE = C::nE, nO = C::nO, fE = C::fE, fO = C::fO;
  constexpr bool PCG = MODE == GRAD_PCG;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ double s_beta;
  const IpdgEoTile<N> t{smem};
  const int tid = threadIdx.x;
  const TileCut tiles(p.K, gridDim.x);
  const int k0 = tiles.start(blockIdx.x), ne = tiles.size(blockIdx.x);
  if (!t.setup(p, k0, ne, C::kOpsG, false)) return;
  const double* u_in = static_cast<const double*>(p.u);
  const double* pold = static_cast<const double*>(p.p_old);
  grid_dep_wait();
  grid_dep_launch();
  if (PCG) {
    const int d = p.first ? p.cg->done : cg_decide(*p.cg, p.slot);
    if (d) {
      if (blockIdx.x == 0 && tid == 0) p.cg->done = d;
      return;
    }
  }
  if (tid == 0) {
    mbar_arrive_expect_tx(t.bar() + 1, (PCG ? 2 : 1) * ne * NpP * 8);
    bulk_g2s(t.field(0), u_in + (size_t)k0 * NpP, ne * NpP * 8, t.bar() + 1);
    if (PCG) bulk_g2s(t.field(1), pold + (size_t)k0 * NpP, ne * NpP * 8, t.bar() + 1);
    // beta = rz_new / rz_old, one division per CTA
    s_beta = PCG && !p.first ? p.cg->rz[p.slot] / p.cg->rz[(p.slot + 2) % 3] : 0.0;
    if (PCG && blockIdx.x == 0) p.cg->pAp = 0.0;
  }
  // exterior values of the face-node pair
  const int fe = tid / fE, fc = tid - fe * fE;
  const bool fact = fe < ne, ftwo = fc < fO;
  double bz[2] = {0.0, 0.0}, bp[2] = {0.0, 0.0};
  int kind[2] = {0, 0};  // 0 interior, 1 Dirichlet, 2 Neumann
  if (fact) {
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      if (w && !ftwo) break;
      const int m = t.faces()[2 * fc + w], f = m / Nfp, d = m - f * Nfp;
      const int nb = nb_of<double, N>(t.nbr()[fe], f);
      if (nb >= 0) {
        const size_t o = (size_t)(nb >> 2) * NpP + fmask<N>(nb & 3, Nfp - 1 - d);
        bz[w] = __ldg(u_in + o);
        if (PCG) bp[w] = __ldg(pold + o);
      } else {
        kind[w] = bc_dirichlet<N>(p, nb, d) ? 1 : 2;
      }
    }
  }
  if (!__syncthreads_and(mbar_wait(t.bar() + 1, 0, p.status))) return;
  double* sU = t.field(0);
  const double beta = s_beta;
  if (PCG) {
    // p = z + beta p_old on the tile, written out
    double* pv = static_cast<double*>(p.p);
    for (int x = tid; x < ne * NpP; x += 256) {
      const double v = fma(beta, t.field(1)[x], sU[x]);
      sU[x] = v;
      pv[(size_t)k0 * NpP + x] = v;
    }
    __syncthreads();
  }
  // lifted jumps: sums and differences of the face-node pairs
  if (fact) {
    const double* c = t.consts() + fe * C::CSTR + IC_F;
    double lx[2] = {0.0, 0.0}, ly[2] = {0.0, 0.0};
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      if (w && !ftwo) break;
      const int m = t.faces()[2 * fc + w], f = m / Nfp, d = m - f * Nfp;
      const double um = sU[fe * NpP + fmask<N>(f, d)];
      double up = PCG ? fma(beta, bp[w], bz[w]) : bz[w];
      if (kind[w]) up = kind[w] == 1 ? -um : um;
      const double du = um - up;
      lx[w] = c[3 * f] * du;
      ly[w] = c[3 * f + 1] * du;
    }
    double* fo = t.flux() + fe * C::FSTR + fc;
    fo[0] = ftwo ? lx[0] + lx[1] : lx[0];
    fo[fE] = ftwo ? lx[0] - lx[1] : 0.0;
    fo[2 * fE] = ftwo ? ly[0] + ly[1] : ly[0];
    fo[3 * fE] = ftwo ? ly[0] - ly[1] : 0.0;
  }
  t.sum_diff(sU, ne);
  __syncthreads();
  t.grad_rows(p, ne, k0, static_cast<double*>(p.qx), static_cast<double*>(p.qy));
}

// ---------------------------------------------------------------- div pass
template <int N, int MODE>
__global__ void __launch_bounds__(256) ipdg_div_eo_kernel(const IpdgParams p) {
  using C = IpdgEo<N>;
  constexpr int Np = C::Np, NpP = C::NpP, Nfp = C::Nfp, nE = C::nE, nO = C::nO, fE = C::fE, fO = C::fO;
  constexpr bool SPD = MODE != DIV_LAPLACE;
  extern __shared__ __align__(128) unsigned char smem[];
  const IpdgEoTile<N> t{smem};
  const int tid = threadIdx.x;
  const TileCut tiles(p.K, gridDim.x);
  const int k0 = tiles.start(blockIdx.x), ne = tiles.size(blockIdx.x);
  if (!t.setup(p, k0, ne, SPD ? C::kOpsD : C::kOpsG, SPD)) return;
  const double* qx = static_cast<const double*>(p.qx);
  const double* qy = static_cast<const double*>(p.qy);
  const double* uj = static_cast<const double*>(p.du_src);
  double* out = static_cast<double*>(p.out);
  grid_dep_wait();
  grid_dep_launch();
  if (MODE == DIV_SPD_DOT && p.cg->done) return;
  if (tid == 0) {
    mbar_arrive_expect_tx(t.bar() + 1, 3 * ne * NpP * 8);
    bulk_g2s(t.field(0), qx + (size_t)k0 * NpP, ne * NpP * 8, t.bar() + 1);
    bulk_g2s(t.field(1), qy + (size_t)k0 * NpP, ne * NpP * 8, t.bar() + 1);
    bulk_g2s(t.field(2), uj + (size_t)k0 * NpP, ne * NpP * 8, t.bar() + 1);
    if (MODE == DIV_SPD_DOT && blockIdx.x == 0) {
      const int s1 = (p.slot + 1) % 3;
      p.cg->rz[s1] = 0.0;
      p.cg->rr[s1] = 0.0;
    }
  }
  // exterior traces of the face-node pair
  const int fe = tid / fE, fc = tid - fe * fE;
  const bool fact = fe < ne, ftwo = fc < fO;
  double bx[2], by[2], bu[2];
  int kind[2] = {0, 0};
  if (fact) {
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      if (w && !ftwo) break;
      const int m = t.faces()[2 * fc + w], f = m / Nfp, d = m - f * Nfp;
      const int nb = nb_of<double, N>(t.nbr()[fe], f);
      if (nb >= 0) {
        const size_t o = (size_t)(nb >> 2) * NpP + fmask<N>(nb & 3, Nfp - 1 - d);
        bx[w] = __ldg(qx + o);
        by[w] = __ldg(qy + o);
        bu[w] = __ldg(uj + o);
      } else {
        kind[w] = bc_dirichlet<N>(p, nb, d) ? 1 : 2;
      }
    }
  }
  const int e = tid / Np, r = tid - e * Np;
  const bool act = e < ne;
  const size_t o = (size_t)(k0 + e) * NpP + r;
  double bv = 0.0;
  if (MODE == DIV_RESID && act) bv = static_cast<const double*>(p.b)[o];
  if (!__syncthreads_and(mbar_wait(t.bar() + 1, 0, p.status))) return;
  const double *sX = t.field(0), *sY = t.field(1), *sU = t.field(2);
  if (fact) {
    const double* c = t.consts() + fe * C::CSTR + IC_F;
    double fl[2] = {0.0, 0.0};
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      if (w && !ftwo) break;
      const int m = t.faces()[2 * fc + w], f = m / Nfp, d = m - f * Nfp;
      const int nd = fe * NpP + fmask<N>(f, d);
      const double xm = sX[nd], ym = sY[nd], um = sU[nd];
      if (kind[w]) {  // Dirichlet: [q] = 0, du = 2 u-; Neumann: [q] = 2 q-, du = 0
        const bool dir = kind[w] == 1;
        bx[w] = dir ? xm : -xm;
        by[w] = dir ? ym : -ym;
        bu[w] = dir ? -um : um;
      }
      fl[w] = fma(c[3 * f], xm - bx[w], fma(c[3 * f + 1], ym - by[w], c[3 * f + 2] * (um - bu[w])));
    }
    double* fo = t.flux() + fe * C::FSTR + fc;
    fo[0] = ftwo ? fl[0] + fl[1] : fl[0];
    fo[fE] = ftwo ? fl[0] - fl[1] : 0.0;
  }
  t.combine(sX, sY, ne);
  __syncthreads();
  double au = 0.0;
  const bool sum = r < nE;
  if (act) {
    au = t.div_row(p, e, r);
    if (SPD && p.shift != 0.0) {  // (A - shift I) u, scaled by -J like the rest
      const int c = sum ? r : r - nE;
      const double ua = sU[e * NpP + t.nodes()[2 * c]], ub = sU[e * NpP + t.nodes()[2 * c + 1]];
      const double uh = sum ? (c < nO ? 0.5 * (ua + ub) : ua) : 0.5 * (ua - ub);
      au = fma(-p.shift * t.consts()[e * C::CSTR + IC_MJ], uh, au);
    }
  }
  __syncthreads();
  double* ro = t.in() + e * 2 * Np;
  if (act) ro[r] = au;
  __syncthreads();
  if (SPD) {
    if (act) {
      // mass rows: half sums from half sums, half differences from half differences
      const double* m = t.M() + r;
      const double* w = ro + (sum ? 0 : nE);
      const int n = sum ? nE : nO;
      au = 0.0;
#pragma unroll 4
      for (int j = 0; j < n; ++j) au = fma(m[j * Np], w[j], au);
      ro[Np + r] = au;
    }
    __syncthreads();
    ro += Np;
  }
  double dot = 0.0;
  if (act) {
    double v = t.node(ro, r);
    if (MODE == DIV_RESID) {
      v = bv - v;
      dot = v * v;
    } else if (MODE == DIV_SPD_DOT) {
      dot = sU[e * NpP + r] * v;
    }
    out[o] = v;
  }
  // padded output nodes are written as 0 (callers sum over whole vectors)
  constexpr int kPad = NpP - Np;
  if constexpr (kPad > 0)
    for (int q = tid; q < ne * kPad; q += 256) out[(size_t)(k0 + q / kPad) * NpP + Np + q % kPad] = 0.0;
  if (MODE == DIV_SPD_DOT || MODE == DIV_RESID) {
    const double s = block_sum(dot, t.red());
    if (tid == 0) atomicAdd(MODE == DIV_SPD_DOT ? &p.cg->pAp : p.dot_out, s);
  }
}

}  // namespace dgk
