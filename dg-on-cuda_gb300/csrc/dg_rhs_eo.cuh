// dg_rhs_eo.cuh -- fused RHS + stage kernel in the even / odd basis of the
// reflection r <-> s (eo.hpp): the operator, fluxes and epilogues of
// dg_rhs.cuh with half the products.  It is the FP64 stage kernel.
//
// What bounds it: the FP64 pipe.  GB300 issues about two FP64 lanes per cycle
// and SM, so a stage costs its FP64 instructions and next to nothing else
// (the node-by-node kernel: 413 us per stage at Maxwell TE, K = 32768, N = 6,
// with that pipe 95.7 % busy and 1.5 % of the DRAM bandwidth).  Every choice
// here removes FP64 instructions, counted per element at N = 6, Maxwell:
//   * even / odd operators: D+ and D- of one field take Np^2 products where Dr
//     and Ds took 2 Np^2; the curl of the first two fields is one D+ p + D- m,
//     p and m their combination with the element's constant geometry (formed
//     once per node): 2 Np^2 instead of 6 Np^2, LIFT half: 2456 instead of 6468;
//   * -1/J, faceJ, the normals and the time step are multiplied into per-element
//     constants once, so rows, fluxes and the epilogue apply none of them;
//   * the upwind fluxes through x = q2- + (n x q)-, y = q2+ - (n x q)+: 9
//     operations per face node instead of 15.
// About 3.3k FP64 instructions per element instead of 7.4k.
//
// A CTA takes one tile of at most 256 / Np elements (see eo_pick_tiles).  One
// CTA per tile lets the hardware hand out tiles as SMs become free; persistent
// CTAs, with their fixed share of tiles, took 206.9 instead of 203.5 us per stage
// at K = 32768, N = 6 and 28.4 instead of 27.0 us at K = 8192, N = 4 (Maxwell TE).
// Phases, a CTA barrier between them:
//   constants  thread (element, value); the exterior face values and the
//              update's own operands are loaded meanwhile
//   inputs     thread (element, face-node pair): both fluxes, sum and difference;
//              thread (element, node pair): sums and differences of q2, p, m
//   rows       thread (element, row): the contraction and LIFT of one sum or
//              difference row
//   nodes      thread (element, node): f = E +- O, stage update
// Operators, geometry and neighbours are set-up data and are fetched before the
// wait for the previous stage.
#pragma once

#include "dg_rhs.cuh"
#include "eo.hpp"

namespace dgk {

template <typename R, int N, int P>
struct EoConfig {
  using O = Order<N>;
  static constexpr EoDims D{N};
  static constexpr int Np = O::Np, NpP = O::NpP, Nfp = O::Nfp;
  static constexpr int Nf = PhysTraits<P>::Nf;
  static constexpr int nE = D.nE, nO = D.nO, fE = D.fE, fO = D.fO;
  static constexpr int kThreads = 256;
  static constexpr int TE = kThreads / Np;            // most elements per tile
  static constexpr int ESTR = Nf * NpP;
  // inputs of an element: Maxwell [q2 | p | m], advection [q], each [nE | nO];
  // the row results [Nf][Np] take their place
  static constexpr int ISTR = Nf * Np;
  static constexpr int FSTR = Nf * 2 * fE;            // [field][fE sums | fE differences (last may be unused)]
  static constexpr int CSTR = 16;                     // per-element constants
  static constexpr uint32_t kOps = (D.kK() + D.kL()) * sizeof(R), kTab = D.tabBytes();
  static constexpr uint32_t oBar = 0;
  static constexpr uint32_t oOps = 32;
  static constexpr uint32_t oTab = oOps + kOps;
  static constexpr uint32_t oQ = oTab + kTab;
  static constexpr uint32_t oGeom = oQ + TE * ESTR * sizeof(R);
  static constexpr uint32_t oNbr = oGeom + TE * 16 * sizeof(R);
  static constexpr uint32_t oC = oNbr + TE * 16;
  static constexpr uint32_t oIn = oC + TE * CSTR * sizeof(R);
  static constexpr uint32_t oF = oIn + TE * ISTR * sizeof(R);
  static constexpr uint32_t kSmem = (oF + TE * FSTR * sizeof(R) + 15) / 16 * 16;
  // one face-node pair per thread and tile
  static_assert(TE * fE <= kThreads, "flux items");
  static_assert(kOps % 16 == 0 && ESTR * sizeof(R) % 16 == 0 && oIn % 8 == 0, "16-byte bulk copies");
};

// slots of the per-element constants (s: 1, or the time step of an LSERK stage;
// sg = +1 TE, -1 TM)
enum EoConst : int {
  EC_P1 = 0, EC_P2 = 1,  // Maxwell sg s (rx +- sx) | advection s (cx +- cy-combination of D+ and D-)
  EC_Q1 = 2, EC_Q2 = 3,  // Maxwell -sg s (ry +- sy)
  EC_H = 4,              // faces 0..2: -s faceJ / (2 J) | advection: -s an faceJ / J
  EC_X = 7,              // Maxwell, faces 0..2: sg H nx
  EC_Y = 10,             // Maxwell, faces 0..2: -sg H ny
};

// tiles of the stage kernel, from its FP64 instructions per row,
// flux, input and constant item
template <typename R, int N, int P>
inline int eo_tiles(int K, int sm_count) {
  using C = EoConfig<R, N, P>;
  constexpr bool adv = P == PHYS_ADV;
  return eo_pick_tiles(C::D, K, sm_count, C::TE,
                       adv ? EoCost{C::Np + C::fE + 7, 5, 2, 6} : EoCost{2 * C::Np + 3 * C::fE + 14, 24, 14, 10});
}

template <typename R, int N, int P>
__global__ void __launch_bounds__(256) dg_rhs_eo_kernel(const RhsParams p) {
  using C = EoConfig<R, N, P>;
  constexpr int Np = C::Np, NpP = C::NpP, Nfp = C::Nfp, NF = C::Nf, ESTR = C::ESTR;
  constexpr int nE = C::nE, nO = C::nO, fE = C::fE, fO = C::fO;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + C::oBar);  // [0] set-up data, [1] state
  const R* sK = reinterpret_cast<const R*>(smem + C::oOps);
  const R* sL = sK + C::D.kK();
  const uint8_t* nt = smem + C::oTab;  // node pairs
  const uint8_t* ft = nt + 2 * nE;     // face-node pairs
  R* sQ = reinterpret_cast<R*>(smem + C::oQ);
  const R* sG = reinterpret_cast<const R*>(smem + C::oGeom);
  const int4* sN = reinterpret_cast<const int4*>(smem + C::oNbr);
  R* sC = reinterpret_cast<R*>(smem + C::oC);
  R* sI = reinterpret_cast<R*>(smem + C::oIn);
  R* sF = reinterpret_cast<R*>(smem + C::oF);
  // inflow boundary nodes of the tile: listed by their flux threads, evaluated
  // by consecutive threads (a boundary row touches a few lanes of every flux
  // warp, and the FP64 pipe pays per warp)
  constexpr int kBnd = P == PHYS_ADV ? C::TE * C::O::Nface : 1;
  __shared__ int s_nbnd, s_bnode[kBnd];
  __shared__ R s_bval[kBnd];
  const int tid = threadIdx.x;
  const int rtid = 255 - tid;  // phases that share a barrier interval start from opposite ends of the CTA
  const R* qin = static_cast<const R*>(p.q_in);
  R* out = static_cast<R*>(p.out);
  R* aux = static_cast<R*>(p.aux);
  R* q0 = static_cast<R*>(p.q0);
  const R cca = (R)p.ca, ccb = (R)p.cb;
  const R scale = p.mode == MODE_LSERK ? (R)p.dt : (R)1;
  const TileCut tiles(p.K, gridDim.x);
  const int k0 = tiles.start(blockIdx.x), ne = tiles.size(blockIdx.x);
  if (tid == 0) {
    s_nbnd = 0;
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_barrier_init();
    mbar_arrive_expect_tx(&bar[0], C::kOps + C::kTab + ne * 16 * (sizeof(R) + 1));
    bulk_g2s(const_cast<R*>(sK), p.mats_eo, C::kOps, &bar[0]);
    bulk_g2s(smem + C::oTab, p.tab_eo, C::kTab, &bar[0]);
    bulk_g2s(const_cast<R*>(sG), static_cast<const R*>(p.geom) + (size_t)k0 * 16, ne * 16 * sizeof(R), &bar[0]);
    bulk_g2s(const_cast<int4*>(sN), p.nbr + k0, ne * 16, &bar[0]);
  }
  __syncthreads();  // barrier initialisation seen by all
  if (!__syncthreads_and(mbar_wait(&bar[0], 0, p.status))) return;
  // operators and geometry are set-up data; everything from here on reads the
  // previous launch's results.  The next stage may be scheduled now (it waits
  // likewise).
  grid_dep_wait();
  grid_dep_launch();
  if (tid == 0) {
    mbar_arrive_expect_tx(&bar[1], ne * ESTR * sizeof(R));
    bulk_g2s(sQ, qin + (size_t)k0 * ESTR, ne * ESTR * sizeof(R), &bar[1]);
  }
  const double tnow = P == PHYS_ADV ? (p.t_dev ? *p.t_dev + p.t : p.t) : 0.0;

  // ---- exterior values of this thread's face-node pair, and the update's own
  //      loads: in flight while the state tile arrives
  const int fe = tid / fE, fc = tid - fe * fE;  // element and pair
  const bool fact = fe < ne, ftwo = fc < fO;
  R b[2][NF];
  bool wall[2] = {false, false};
  int bslot[2] = {-1, -1};
  if (fact) {
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      if (w && !ftwo) break;
      const int m = ft[2 * fc + w], f = m / Nfp, d = m - f * Nfp;
      const int nb = f == 0 ? sN[fe].x : (f == 1 ? sN[fe].y : sN[fe].z);
      if (nb >= 0) {
        const R* qb = qin + (size_t)(nb >> 2) * ESTR + fmask<N>(nb & 3, Nfp - 1 - d);
#pragma unroll
        for (int i = 0; i < NF; ++i) b[w][i] = __ldg(qb + i * NpP);
      } else if (P == PHYS_ADV) {
        // the boundary value enters the flux only where the wind blows in
        const R* g = sG + fe * 16;
        b[w][0] = (R)0;
        if (!((R)p.ax * g[8 + f] + (R)p.ay * g[11 + f] >= (R)0)) {
          bslot[w] = atomicAdd(&s_nbnd, 1);
          s_bnode[bslot[w]] = (-1 - nb) * Nfp + d;
        }
      } else {
        wall[w] = true;
      }
    }
  }
  const int e = tid / Np, r = tid - e * Np;  // element and row (then node) of this thread
  const bool act = e < ne;
  const size_t base = (size_t)(k0 + e) * ESTR + r;
  R av[NF], bv[NF];
  if (act) {
    if (p.mode == MODE_LSERK || (p.mode == MODE_RK4 && p.stage > 0))
#pragma unroll
      for (int i = 0; i < NF; ++i) av[i] = aux[base + i * NpP];
    if (p.mode == MODE_RK4 && p.stage > 0)
#pragma unroll
      for (int i = 0; i < NF; ++i) bv[i] = q0[base + i * NpP];
  }

  // ---- constants
  for (int x = rtid; x < ne * 8; x += 256) {
    const int ce = x >> 3, v = x & 7;
    const R* g = sG + ce * 16;
    R* c = sC + ce * C::CSTR;
    if (P == PHYS_ADV) {
      if (v < 2) {
        const R ca = (R)p.ax * g[0] + (R)p.ay * g[1], cb = (R)p.ax * g[2] + (R)p.ay * g[3];
        c[EC_P1 + v] = scale * (v ? ca - cb : ca + cb);
      } else if (v < 5) {
        const int f = v - 2;
        c[EC_H + f] = ((R)p.ax * g[8 + f] + (R)p.ay * g[11 + f]) * (g[5 + f] * (scale * g[4]));
      }
    } else {
      const R sg = P == PHYS_TE ? scale : -scale;
      if (v < 2) c[EC_P1 + v] = sg * (v ? g[0] - g[2] : g[0] + g[2]);
      else if (v < 4) c[EC_Q1 + v - 2] = -sg * (v == 3 ? g[1] - g[3] : g[1] + g[3]);
      else if (v < 7) {
        const int f = v - 4;
        const R h = (R)0.5 * (g[5 + f] * (scale * g[4]));
        c[EC_H + f] = h;
        c[EC_X + f] = P == PHYS_TE ? h * g[8 + f] : -h * g[8 + f];
        c[EC_Y + f] = P == PHYS_TE ? -h * g[11 + f] : h * g[11 + f];
      }
    }
  }
  if (P == PHYS_ADV) {
    __syncthreads();
    for (int x = tid; x < s_nbnd; x += 256) {
      const double* xy = p.bxy + (size_t)s_bnode[x] * 2;
      s_bval[x] = (R)adv_exact(p, tnow, xy[0], xy[1]);
    }
  }
  if (!__syncthreads_and(mbar_wait(&bar[1], 0, p.status))) return;

  // ---- fluxes of the face-node pair, scaled for LIFT, as sum and difference
  if (fact) {
    const R* cc = sC + fe * C::CSTR;
    const R* g = sG + fe * 16;
    const R* qa = sQ + fe * ESTR;
    R fl[2][NF];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      if (w && !ftwo) break;
      const int m = ft[2 * fc + w], f = m / Nfp, d = m - f * Nfp, nd = fmask<N>(f, d);
      if (P == PHYS_ADV) {
        const R h = cc[EC_H + f];
        if (bslot[w] >= 0) b[w][0] = s_bval[bslot[w]];
        // upwind side by the sign of a.n: h carries -s an faceJ / J, so
        // a.n >= 0 exactly where h <= 0 (h >= 0 for a negative time step)
        fl[w][0] = (scale >= (R)0 ? h <= (R)0 : h >= (R)0) ? qa[nd] * h : b[w][0] * h;
      } else {
        const R nx = g[8 + f], ny = g[11 + f];
        const R a0 = qa[nd], a1 = qa[NpP + nd], a2 = qa[2 * NpP + nd];
        if (wall[w]) {  // PEC: E+ = -E-, Hz+ = Hz- | H+ = H-, Ez+ = -Ez-
          b[w][0] = P == PHYS_TE ? -a0 : a0;
          b[w][1] = P == PHYS_TE ? -a1 : a1;
          b[w][2] = P == PHYS_TE ? a2 : -a2;
        }
        R xx, yy;
        if (P == PHYS_TE) {
          xx = fma(nx, a1, fma(-ny, a0, a2));
          yy = fma(-nx, b[w][1], fma(ny, b[w][0], b[w][2]));
        } else {
          xx = fma(ny, a0, fma(-nx, a1, a2));
          yy = fma(-ny, b[w][0], fma(nx, b[w][1], b[w][2]));
        }
        const R ww = xx + yy;
        fl[w][0] = cc[EC_Y + f] * ww;
        fl[w][1] = cc[EC_X + f] * ww;
        fl[w][2] = cc[EC_H + f] * (xx - yy);
      }
    }
    R* fo = sF + fe * C::FSTR + fc;
#pragma unroll
    for (int i = 0; i < NF; ++i) {
      fo[i * 2 * fE] = ftwo ? fl[0][i] + fl[1][i] : fl[0][i];
      // an unpaired face node has no difference; its column is 0
      fo[i * 2 * fE + fE] = ftwo ? fl[0][i] - fl[1][i] : (R)0;
    }
  }
  // ---- inputs of node pairs
  for (int x = rtid; x < ne * nE; x += 256) {
    const int ie = x / nE, c = x - ie * nE;
    const int na = nt[2 * c], nb = nt[2 * c + 1];
    const bool two = c < nO;
    const R* qa = sQ + ie * ESTR;
    R* in = sI + ie * C::ISTR + c;
    R s[NF], d[NF];
#pragma unroll
    for (int i = 0; i < NF; ++i) {
      const R u = qa[i * NpP + na];
      if (two) {
        const R v = qa[i * NpP + nb];
        s[i] = u + v;
        d[i] = u - v;
      } else {
        s[i] = u;
        d[i] = (R)0;
      }
    }
    if (P == PHYS_ADV) {
      in[0] = s[0];
      if (two) in[nE] = d[0];
    } else {
      const R* cc = sC + ie * C::CSTR;
      const R p1 = cc[EC_P1], p2 = cc[EC_P2], q1 = cc[EC_Q1], q2 = cc[EC_Q2];
      in[0] = s[2];
      in[Np] = fma(p1, s[1], q1 * s[0]);
      in[2 * Np] = fma(p2, s[1], q2 * s[0]);
      if (two) {
        in[nE] = d[2];
        in[Np + nE] = fma(p1, d[1], q1 * d[0]);
        in[2 * Np + nE] = fma(p2, d[1], q2 * d[0]);
      }
    }
  }
  __syncthreads();

  // ---- rows: sum row (r < nE) or difference row of element e
  const bool rest = nt[C::D.flag()] != 0;  // operators without the symmetry (eo.hpp)
  auto rest_row = [&] { return reinterpret_cast<const R*>(p.tab_eo + C::kTab) + r; };
  R rr[NF];
  if (act) {
    const bool sum = r < nE;
    const R* k = sK + r;
    const R* x = sI + e * C::ISTR;
    const R* cc = sC + e * C::CSTR;
    if (P == PHYS_ADV) {
      R s1 = (R)0, s2 = (R)0;
#pragma unroll 4
      for (int c = 0; c < nE; ++c) s1 = fma(k[c * Np], x[c], s1);
      k += nE * Np;
      x += nE;
#pragma unroll 4
      for (int c = 0; c < nO; ++c) s2 = fma(k[c * Np], x[c], s2);
      if (rest) {
        const R* k2 = rest_row();
        x = sI + e * C::ISTR;
#pragma unroll 1
        for (int c = 0; c < Np; ++c) (c < nE ? s2 : s1) = fma(k2[c * Np], x[c], c < nE ? s2 : s1);
      }
      const R p1 = cc[EC_P1], p2 = cc[EC_P2];
      rr[0] = sum ? fma(p1, s1, p2 * s2) : fma(p2, s1, p1 * s2);
    } else {
      // sum rows take p's sums and m's differences, difference rows the others
      const R* u = x + (sum ? Np : 2 * Np);
      const R* v = x + (sum ? 2 * Np : Np) + nE;
      R s1 = (R)0, s2 = (R)0, cu = (R)0, cv = (R)0;
#pragma unroll 4
      for (int c = 0; c < nE; ++c) {
        const R kk = k[c * Np];
        s1 = fma(kk, x[c], s1);
        cu = fma(kk, u[c], cu);
      }
      k += nE * Np;
      x += nE;
#pragma unroll 4
      for (int c = 0; c < nO; ++c) {
        const R kk = k[c * Np];
        s2 = fma(kk, x[c], s2);
        cv = fma(kk, v[c], cv);
      }
      if (rest) {
        const R* k2 = rest_row();
        x = sI + e * C::ISTR;
#pragma unroll 1
        for (int c = 0; c < Np; ++c) {
          const R kk = k2[c * Np];
          (c < nE ? s2 : s1) = fma(kk, x[c], c < nE ? s2 : s1);
          // sum rows: m's sums and p's differences, difference rows the others
          cu = fma(kk, x[((c < nE) == sum ? 2 * Np : Np) + c], cu);
        }
      }
      const int ia = sum ? 0 : 1;  // D+ q2 is s1 in a sum row, s2 in a difference row
      rr[0] = fma(cc[EC_Q1 + ia], s1, cc[EC_Q2 - ia] * s2);
      rr[1] = fma(cc[EC_P1 + ia], s1, cc[EC_P2 - ia] * s2);
      rr[2] = cu + cv;
    }
    const R* l = sL + r;
    const R* f = sF + e * C::FSTR + (sum ? 0 : fE);
#pragma unroll 4
    for (int m = 0; m < fE; ++m) {
      const R ll = l[m * Np];
#pragma unroll
      for (int i = 0; i < NF; ++i) rr[i] = fma(ll, f[i * 2 * fE + m], rr[i]);
    }
    if (rest) {
      l = rest_row() + C::D.kK();
      f = sF + e * C::FSTR + (sum ? fE : 0);
#pragma unroll 1
      for (int m = 0; m < (sum ? fO : fE); ++m)
        for (int i = 0; i < NF; ++i) rr[i] = fma(l[m * Np], f[i * 2 * fE + m], rr[i]);
    }
  }
  __syncthreads();
  if (act)
#pragma unroll
    for (int i = 0; i < NF; ++i) sI[e * C::ISTR + i * Np + r] = rr[i];
  __syncthreads();

  // ---- nodes: f = E + O at a pair's first node, E - O at its second
  if (act) {
    const int inv = nt[2 * nE + 2 * fE + r];
    const int c = inv & 127;
    const R* ro = sI + e * C::ISTR;
    const R* qe = sQ + e * ESTR + r;
#pragma unroll
    for (int i = 0; i < NF; ++i) {
      R v = ro[i * Np + c];
      if (c < nO) v = inv & 128 ? v - ro[i * Np + nE + c] : v + ro[i * Np + nE + c];
      rr[i] = v;
    }
    if (p.mode == MODE_RHS) {
#pragma unroll
      for (int i = 0; i < NF; ++i) out[base + i * NpP] = rr[i];
    } else if (p.mode == MODE_LSERK) {
#pragma unroll
      for (int i = 0; i < NF; ++i) {
        const R w = fma(cca, av[i], rr[i]);  // the row results carry the time step
        aux[base + i * NpP] = w;
        out[base + i * NpP] = fma(ccb, w, qe[i * NpP]);
      }
    } else {  // classical RK4 stage
#pragma unroll
      for (int i = 0; i < NF; ++i) {
        const size_t o = base + i * NpP;
        if (p.stage == 0) {
          aux[o] = rr[i];
          out[o] = fma(cca, rr[i], qe[i * NpP]);
        } else if (p.stage < 3) {
          aux[o] = fma(ccb, rr[i], av[i]);
          out[o] = fma(cca, rr[i], bv[i]);
        } else {
          q0[o] = fma(cca, av[i] + rr[i], bv[i]);
        }
      }
    }
  }
}

}  // namespace dgk
