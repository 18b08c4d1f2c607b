// dg_rhs_sym.cuh -- FP32 stage kernel in the even / odd basis of the reflection
// r <-> s (eo.hpp), one element per lane: the operator, fluxes and epilogues of
// dg_rhs_blk.cuh.
//
// What it saves: shared-memory wavefronts (one per cycle and SM).  In
// dg_rhs_blk.cuh the operator loads alone take 8 of the ~11 wavefronts per
// operator column and warp: with the node groups of an element in consecutive
// lanes a 16-byte operator load serves 8 lanes per wavefront.  Here
//   * D+ / D- and the half-sized LIFT (eo.hpp) halve the operator columns;
//   * a warp holds one group of G rows of 32 elements, so an operator load is
//     uniform (2 wavefronts for 4 rows x 32 elements) and an input load is one
//     word per lane at an odd element stride (1 wavefront);
//   * rows are sums only or differences only within a group.
// Wavefronts per element, Maxwell N = 6: volume and LIFT 37 instead of 99.  What
// bounds it then is the chain of a tile's phases: half of the issue slots and 46 %
// of the wavefronts are in use.
//
// A CTA takes one tile of TE elements: bulk copy of state, geometry and neighbours;
// exterior face values into registers; fluxes of face-node pairs and inputs of
// node pairs (sums and differences) to shared memory; rows; results back as
// E +- O, four nodes of an element per thread.  It needs many CTAs per SM to hide
// its phases: inside the batched launch (2-3 CTAs per SM) these tiles were 5-20 %
// slower than dg_rhs_blk.cuh's, which the batch keeps.
//
// us per stage, graphed, against the blocked kernel: advection K = 32768, N = 6
// 12.2 / 15.1, N = 4 7.9 / 11.7, K = 24200, N = 8 15.8 / 28.2, but K = 2048, N = 4
// 5.0 / 5.0; Maxwell K = 32768, N = 6 17.8 / 18.9, N = 4 11.5 / 11.6, K = 12800, N = 7
// 14.4 / 18.1, N = 8 14.8 / 19.5, but N = 3 6.2 / 4.7 and K = 2048, N = 6 5.6 / 4.4: the
// autotuner decides.
#pragma once

#include <type_traits>

#include "dg_rhs.cuh"
#include "eo.hpp"

namespace dgk {

// rows per group: nE = gE G and nO = gO G for most orders, few padded rows otherwise
constexpr int sym_rows(int N) { return N == 1 ? 1 : N == 2 ? 2 : N == 3 ? 2 : N == 4 ? 3 : N == 5 ? 3 : N == 6 ? 4 : N == 7 ? 5 : 7; }

constexpr int sym_pad(int G) { return G <= 2 ? G : (G + 3) / 4 * 4; }  // rows of a group, padded for vector loads

template <int N, int P>
struct SymConfig {
  using O = Order<N>;
  static constexpr EoDims D{N};
  static constexpr int Np = O::Np, NpP = O::NpP, Nfp = O::Nfp, NF = PhysTraits<P>::Nf;
  static constexpr int nE = D.nE, nO = D.nO, fE = D.fE, fO = D.fO;
  static constexpr int G = sym_rows(N), GP = sym_pad(G);
  static constexpr int gE = (nE + G - 1) / G, gO = (nO + G - 1) / G, NG = gE + gO;
  static constexpr int KS = NG * GP;                                        // operator row stride
  static constexpr int MW = 8 / NG > 0 ? 8 / NG : 1;                        // 32-element blocks per tile
  static constexpr int TE = 32 * MW, kThreads = 32 * NG * MW;
  static constexpr int ESTR = NF * NpP;
  static constexpr int IN = NF * Np;                                        // inputs, then row results
  static constexpr int ISTR = (IN + 4) | 1;                                 // odd; 4 constants behind the inputs
  static constexpr int FSTR = (NF * (fE + fO)) | 1;
  static constexpr uint32_t kOps = ((Np + fE) * KS * 4 + 15) / 16 * 16, kTab = D.tabBytes();
  static constexpr uint32_t oBar = 0, oOps = 32, oTab = oOps + kOps, oQ = oTab + kTab, oGeom = oQ + TE * ESTR * 4,
                            oNbr = oGeom + TE * 64, oIn = oNbr + TE * 16, oF = oIn + TE * ISTR * 4,
                            oBnd = oF + TE * FSTR * 4;
  // inflow boundary nodes of the tile (advection): indices and values
  static constexpr int kBnd = P == PHYS_ADV ? TE * O::Nface : 0;
  static constexpr uint32_t kSmem = (oBnd + kBnd * 8 + 8 + 15) / 16 * 16;
  static_assert(NG * MW <= 8 && oQ % 16 == 0 && oGeom % 16 == 0 && oIn % 16 == 0, "layout");
};

template <int G, int GP>
__device__ __forceinline__ void sym_ops(const float* k, float (&o)[G]) {
  if constexpr (GP % 4 == 0) {
#pragma unroll
    for (int q = 0; q < GP / 4; ++q) {
      const float4 v = reinterpret_cast<const float4*>(k)[q];
      if (4 * q < G) o[4 * q] = v.x;
      if (4 * q + 1 < G) o[4 * q + 1] = v.y;
      if (4 * q + 2 < G) o[4 * q + 2] = v.z;
      if (4 * q + 3 < G) o[4 * q + 3] = v.w;
    }
  } else if constexpr (GP == 2) {
    const float2 v = *reinterpret_cast<const float2*>(k);
    o[0] = v.x;
    o[1] = v.y;
  } else {
    o[0] = k[0];
  }
}

// Each element's state is taken relative to its value at node 0 (c below), and so
// are the exterior values on its faces: a constant state has no right-hand side
// (volume and flux terms cancel on a straight-sided element), so c drops out, and
// with it the part of the operators' FP32 rounding that acts on the state's
// magnitude.  Without it that part, larger here than in the node basis because the
// operators are rounded after the change of basis, grew with the time integrated:
// error against FP64 after the same run, blocked kernel / here without / here with:
// Maxwell TE to T = 1, K = 32768, N = 6 5.8e-6 / 6.6e-6 / 3.9e-6, to T = 0.5, K = 4608,
// N = 7 9.2e-6 / 1.2e-5 / 2.5e-6, advection to T = 0.5, K = 8192, N = 4 1.1e-6 / 2.0e-6 /
// 1.1e-6.  It costs the Maxwell stage 1-3 % (K = 32768, N = 6: 17.4 -> 17.7 us).
// Operators or geometry without that cancellation run the blocked kernel.
//
// The tile of ne elements from k0.  Operators, geometry and neighbours are in
// shared memory; the state arrives on `bar`, phase 0.
template <int N, int P>
__device__ __forceinline__ void sym_tile(const RhsParams& p, unsigned char* smem, uint64_t* bar, int k0, int ne,
                                         double tnow) {
  using C = SymConfig<N, P>;
  constexpr int NT = C::kThreads;
  constexpr int Np = C::Np, NpP = C::NpP, Nfp = C::Nfp, NF = C::NF, ESTR = C::ESTR, ISTR = C::ISTR, FSTR = C::FSTR;
  constexpr int nE = C::nE, nO = C::nO, fE = C::fE, fO = C::fO, G = C::G, GP = C::GP, KS = C::KS;
  constexpr int kItems = (C::TE * fE + NT - 1) / NT;
  const float* sK = reinterpret_cast<const float*>(smem + C::oOps);
  const uint8_t* nt = smem + C::oTab;
  const uint8_t* ft = nt + 2 * nE;
  const uint8_t* inv = ft + 2 * fE;
  const float* sQ = reinterpret_cast<const float*>(smem + C::oQ);
  const float* sG = reinterpret_cast<const float*>(smem + C::oGeom);
  const int4* sN = reinterpret_cast<const int4*>(smem + C::oNbr);
  float* sI = reinterpret_cast<float*>(smem + C::oIn);
  float* sF = reinterpret_cast<float*>(smem + C::oF);
  int* bcount = reinterpret_cast<int*>(smem + C::oBnd + C::kBnd * 8);
  int* bnode = reinterpret_cast<int*>(smem + C::oBnd);
  float* bval = reinterpret_cast<float*>(smem + C::oBnd + C::kBnd * 4);
  const int tid = threadIdx.x;
  const float* qin = static_cast<const float*>(p.q_in);
  const float cax = p.fax, cay = p.fay;
  // operators that have lost the symmetry (eo.hpp) or the cancellation
  const bool rest = nt[C::D.flag()] != 0;
  auto rest_ops = [&] { return reinterpret_cast<const float*>(p.tab_eo + C::kTab); };

  // ---- exterior values of the face-node pairs
  float b[kItems][2][NF];
  int bs[kItems][2];  // -1 given in b, -2 wall, else a slot of the inflow list
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int x = tid + q * NT;
    bs[q][0] = bs[q][1] = -1;
    if (x < ne * fE) {
      const int e = x / fE, c = x - e * fE;
      const int4 n4 = sN[e];
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        if (w && c >= fO) break;
        const int m = ft[2 * c + w], f = m / Nfp, d = m - f * Nfp;
        const int nb = f == 0 ? n4.x : (f == 1 ? n4.y : n4.z);
        if (nb >= 0) {
          const float* qb = qin + (size_t)(nb >> 2) * ESTR + fmask<N>(nb & 3, Nfp - 1 - d);
#pragma unroll
          for (int i = 0; i < NF; ++i) b[q][w][i] = __ldg(qb + i * NpP);
        } else if (P == PHYS_ADV) {
          b[q][w][0] = 0.0f;  // enters only where the wind blows in
          if (!(cax * sG[e * 16 + 8 + f] + cay * sG[e * 16 + 11 + f] >= 0.0f)) {
            const int sl = atomicAdd(bcount, 1);
            bnode[sl] = (-1 - nb) * Nfp + d;
            bs[q][w] = sl;
          }
        } else {
          bs[q][w] = -2;
        }
      }
    }
  }
  if (P == PHYS_ADV) {
    __syncthreads();
    for (int x = tid; x < *bcount; x += NT) {
      const double* xy = p.bxy + (size_t)bnode[x] * 2;
      bval[x] = (float)adv_exact(p, tnow, xy[0], xy[1]);
    }
  }
  if (!__syncthreads_and(mbar_wait(bar, 0, p.status))) return;

  // the two phases that take the constant off (compiled twice: a test at each value
  // cost up to 5 % of the stage)
  auto prepare = [&](auto cancels) {
    // the element's constant
    auto level = [&](const float* qa, int i) { return decltype(cancels)::value ? qa[i * NpP] : 0.0f; };
    // ---- fluxes of the pairs, scaled by -faceJ / J, as sums and differences
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
      const int x = tid + q * NT;
      if (x < ne * fE) {
        const int e = x / fE, c = x - e * fE;
        const float* g = sG + e * 16;
        const float* qa = sQ + e * ESTR;
        const bool two = c < fO;
        float fl[2][NF];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          if (w && !two) break;
          const int m = ft[2 * c + w], f = m / Nfp, d = m - f * Nfp, nd = fmask<N>(f, d);
          const float nx = g[8 + f], ny = g[11 + f], sc = g[5 + f] * g[4];  // g[4] = -1/J
          float a[NF];
#pragma unroll
          for (int i = 0; i < NF; ++i) a[i] = qa[i * NpP + nd];
          float* bb = b[q][w];
          if (P == PHYS_ADV) {
            const float an = cax * nx + cay * ny;
            const float bx = bs[q][w] >= 0 ? bval[bs[q][w]] : bb[0];
            fl[w][0] = (((an >= 0.0f) ? a[0] : bx) - level(qa, 0)) * an * sc;
          } else {
            if (bs[q][w] == -2) {  // PEC: E+ = -E-, Hz+ = Hz- | H+ = H-, Ez+ = -Ez-
              bb[0] = P == PHYS_TE ? -a[0] : a[0];
              bb[1] = P == PHYS_TE ? -a[1] : a[1];
              bb[2] = P == PHYS_TE ? a[2] : -a[2];
            }
#pragma unroll
            for (int i = 0; i < NF; ++i) {
              a[i] -= level(qa, i);
              bb[i] -= level(qa, i);
            }
            if (P == PHYS_TM) {
              const float w3 = (a[2] + bb[2]) + ny * (a[0] - bb[0]) - nx * (a[1] - bb[1]);
              fl[w][0] = 0.5f * ny * w3 * sc;
              fl[w][1] = -0.5f * nx * w3 * sc;
              fl[w][2] = 0.5f * (ny * (a[0] + bb[0]) - nx * (a[1] + bb[1]) + a[2] - bb[2]) * sc;
            } else {
              const float w3 = (a[2] + bb[2]) - ny * (a[0] - bb[0]) + nx * (a[1] - bb[1]);
              fl[w][0] = -0.5f * ny * w3 * sc;
              fl[w][1] = 0.5f * nx * w3 * sc;
              fl[w][2] = 0.5f * (nx * (a[1] + bb[1]) - ny * (a[0] + bb[0]) + a[2] - bb[2]) * sc;
            }
          }
        }
        float* fo = sF + e * FSTR + c;
#pragma unroll
        for (int i = 0; i < NF; ++i) {
          fo[i * (fE + fO)] = two ? fl[0][i] + fl[1][i] : fl[0][i];
          if (two) fo[i * (fE + fO) + fE] = fl[0][i] - fl[1][i];
        }
      }
    }
    // ---- inputs of the node pairs: Maxwell [q2 | p | m], advection [q], each [sums | differences];
    //      the element's constants behind them
    for (int x = tid; x < ne * nE; x += NT) {
      const int e = x / nE, c = x - e * nE;
      const float* qa = sQ + e * ESTR;
      const float4 g = *reinterpret_cast<const float4*>(sG + e * 16);  // rx ry sx sy
      const int na = nt[2 * c], nb = nt[2 * c + 1];
      const bool two = c < nO;
      float* in = sI + e * ISTR;
      if (P == PHYS_ADV) {
        const float c0 = level(qa, 0), u = qa[na] - c0, v = qa[nb] - c0;
        in[c] = two ? u + v : u;
        if (two) in[nE + c] = u - v;
        if (c == 0) {
          const float al = cax * g.x + cay * g.y, be = cax * g.z + cay * g.w;
          in[C::IN] = al + be;
          in[C::IN + 1] = al - be;
        }
      } else {
        const float sg = P == PHYS_TE ? 1.0f : -1.0f;
        const float p1 = sg * (g.x + g.z), p2 = sg * (g.x - g.z), q1 = -sg * (g.y + g.w), q2 = -sg * (g.y - g.w);
        const float c0 = level(qa, 0), c1 = level(qa, 1), c2 = level(qa, 2);
        const float u0 = qa[na] - c0, u1 = qa[NpP + na] - c1, u2 = qa[2 * NpP + na] - c2;
        if (two) {
          const float v0 = qa[nb] - c0, v1 = qa[NpP + nb] - c1, v2 = qa[2 * NpP + nb] - c2;
          const float s0 = u0 + v0, s1 = u1 + v1, d0 = u0 - v0, d1 = u1 - v1;
          in[c] = u2 + v2;
          in[nE + c] = u2 - v2;
          in[Np + c] = p1 * s1 + q1 * s0;
          in[Np + nE + c] = p1 * d1 + q1 * d0;
          in[2 * Np + c] = p2 * s1 + q2 * s0;
          in[2 * Np + nE + c] = p2 * d1 + q2 * d0;
        } else {
          in[c] = u2;
          in[Np + c] = p1 * u1 + q1 * u0;
          in[2 * Np + c] = p2 * u1 + q2 * u0;
        }
        if (c == 0) {
          in[C::IN] = p1;
          in[C::IN + 1] = p2;
          in[C::IN + 2] = q1;
          in[C::IN + 3] = q2;
        }
      }
    }
  };
  if (rest) prepare(std::false_type{});
  else prepare(std::true_type{});
  __syncthreads();

  // ---- rows: warp = (block of 32 elements, row group), lane = element
  const int wrp = tid >> 5, sub = wrp / C::NG, grp = wrp - sub * C::NG;
  const int re = sub * 32 + (tid & 31);
  const bool ract = wrp < C::NG * C::MW && re < ne;
  const bool sum = grp < C::gE;
  const int row0 = sum ? grp * G : (grp - C::gE) * G, nrow = sum ? nE : nO;
  float rr[NF][G];
  if (ract) {
    const float* k = sK + grp * GP;
    const float* x = sI + re * ISTR;
    float s1[G], s2[G];
#pragma unroll
    for (int g = 0; g < G; ++g) s1[g] = s2[g] = 0.0f;
    if (P == PHYS_ADV) {
#pragma unroll 4
      for (int c = 0; c < nE; ++c) {
        float o[G];
        sym_ops<G, GP>(k + c * KS, o);
        const float xv = x[c];
#pragma unroll
        for (int g = 0; g < G; ++g) s1[g] = fmaf(o[g], xv, s1[g]);
      }
#pragma unroll 4
      for (int c = nE; c < Np; ++c) {
        float o[G];
        sym_ops<G, GP>(k + c * KS, o);
        const float xv = x[c];
#pragma unroll
        for (int g = 0; g < G; ++g) s2[g] = fmaf(o[g], xv, s2[g]);
      }
      if (rest) {
        const float* k2 = rest_ops() + grp * GP;
#pragma unroll 1
        for (int c = 0; c < Np; ++c) {
          float o[G];
          sym_ops<G, GP>(k2 + c * KS, o);
          const float xe = c < nE ? x[c] : 0.0f, xo = c < nE ? 0.0f : x[c];
#pragma unroll
          for (int g = 0; g < G; ++g) {
            s2[g] = fmaf(o[g], xe, s2[g]);
            s1[g] = fmaf(o[g], xo, s1[g]);
          }
        }
      }
      const float p1 = x[C::IN], p2 = x[C::IN + 1];
      const float ca = sum ? p1 : p2, cb = sum ? p2 : p1;
#pragma unroll
      for (int g = 0; g < G; ++g) rr[0][g] = ca * s1[g] + cb * s2[g];
    } else {
      // sum rows take p's sums and m's differences, difference rows the others
      const float* u = x + (sum ? Np : 2 * Np);
      const float* v = x + (sum ? 2 * Np : Np);
      float cu[G];
#pragma unroll
      for (int g = 0; g < G; ++g) cu[g] = 0.0f;
#pragma unroll 4
      for (int c = 0; c < nE; ++c) {
        float o[G];
        sym_ops<G, GP>(k + c * KS, o);
        const float xv = x[c], uv = u[c];
#pragma unroll
        for (int g = 0; g < G; ++g) {
          s1[g] = fmaf(o[g], xv, s1[g]);
          cu[g] = fmaf(o[g], uv, cu[g]);
        }
      }
#pragma unroll 4
      for (int c = nE; c < Np; ++c) {
        float o[G];
        sym_ops<G, GP>(k + c * KS, o);
        const float xv = x[c], vv = v[c];
#pragma unroll
        for (int g = 0; g < G; ++g) {
          s2[g] = fmaf(o[g], xv, s2[g]);
          cu[g] = fmaf(o[g], vv, cu[g]);
        }
      }
      if (rest) {
        const float* k2 = rest_ops() + grp * GP;
#pragma unroll 1
        for (int c = 0; c < Np; ++c) {
          float o[G];
          sym_ops<G, GP>(k2 + c * KS, o);
          // sum rows: m's sums and p's differences, difference rows the others
          const float xv = x[c], uv = x[((c < nE) == sum ? 2 * Np : Np) + c];
          const float xe = c < nE ? xv : 0.0f, xo = c < nE ? 0.0f : xv;
#pragma unroll
          for (int g = 0; g < G; ++g) {
            s2[g] = fmaf(o[g], xe, s2[g]);
            s1[g] = fmaf(o[g], xo, s1[g]);
            cu[g] = fmaf(o[g], uv, cu[g]);
          }
        }
      }
      const float p1 = x[C::IN], p2 = x[C::IN + 1], q1 = x[C::IN + 2], q2 = x[C::IN + 3];
      // D+ q2 is s1 in a sum row, s2 in a difference row
      const float pa = sum ? p1 : p2, pb = sum ? p2 : p1, qa = sum ? q1 : q2, qb = sum ? q2 : q1;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        rr[0][g] = qa * s1[g] + qb * s2[g];
        rr[NF - 2][g] = pa * s1[g] + pb * s2[g];
        rr[NF - 1][g] = cu[g];
      }
    }
    const float* l = sK + Np * KS + grp * GP;
    const float* f = sF + re * FSTR + (sum ? 0 : fE);
    const int nf = sum ? fE : fO;
#pragma unroll 2
    for (int m = 0; m < nf; ++m) {
      float o[G];
      sym_ops<G, GP>(l + m * KS, o);
#pragma unroll
      for (int i = 0; i < NF; ++i) {
        const float fv = f[i * (fE + fO) + m];
#pragma unroll
        for (int g = 0; g < G; ++g) rr[i][g] = fmaf(o[g], fv, rr[i][g]);
      }
    }
    if (rest) {
      l = rest_ops() + Np * KS + grp * GP;
      f = sF + re * FSTR + (sum ? fE : 0);
#pragma unroll 1
      for (int m = 0; m < (sum ? fO : fE); ++m) {
        float o[G];
        sym_ops<G, GP>(l + m * KS, o);
#pragma unroll
        for (int i = 0; i < NF; ++i)
#pragma unroll
          for (int g = 0; g < G; ++g) rr[i][g] = fmaf(o[g], f[i * (fE + fO) + m], rr[i][g]);
      }
    }
  }
  // the next stage may be scheduled: its set-up overlaps the rest of this one
  grid_dep_launch();
  __syncthreads();
  if (ract) {
    // a pair's sum goes to its first node's place, its difference to the second's
    float* in = sI + re * ISTR;
#pragma unroll
    for (int g = 0; g < G; ++g)
      if (row0 + g < nrow) {
        const int n = nt[2 * (row0 + g) + (sum ? 0 : 1)];
#pragma unroll
        for (int i = 0; i < NF; ++i) in[i * Np + n] = rr[i][g];
      }
  }
  __syncthreads();

  // ---- nodes: E + O, E - O; four nodes of an element per thread
  float* out = static_cast<float*>(p.out);
  float* aux = static_cast<float*>(p.aux);
  float* q0 = static_cast<float*>(p.q0);
  const float cca = p.fca, ccb = p.fcb, cdt = p.fdt;
  constexpr int NQ = NpP / 4;
  for (int x = tid; x < ne * NQ; x += NT) {
    const int e = x / NQ, n0 = 4 * (x - e * NQ);
    const float* ro = sI + e * ISTR;
    int other[4];     // the pair's other node
    float sgn[4];     // 1: E + O, -1: E - O with E the other's entry, 0: a node on the axis
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int me = n0 + n < Np ? n0 + n : 0, v = inv[me], c = v & 127;
      other[n] = nt[2 * c + (v & 128 ? 0 : 1)];
      sgn[n] = c >= nO ? 0.0f : (v & 128 ? -1.0f : 1.0f);
    }
#pragma unroll
    for (int i = 0; i < NF; ++i) {
      const size_t o = (size_t)(k0 + e) * ESTR + i * NpP + n0;
      float r[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const float a = ro[i * Np + (n0 + n < Np ? n0 + n : 0)], c = ro[i * Np + other[n]];
        r[n] = sgn[n] == 0.0f ? a : (sgn[n] > 0.0f ? a + c : c - a);
      }
      const float4 qv = *reinterpret_cast<const float4*>(sQ + e * ESTR + i * NpP + n0);
      const float qq[4] = {qv.x, qv.y, qv.z, qv.w};
      float w0[4], w1[4];  // values for out and for aux / q0
      bool wr_out = true, wr_aux = true, wr_q0 = false;
      if (p.mode == MODE_RHS) {
#pragma unroll
        for (int n = 0; n < 4; ++n) w0[n] = w1[n] = r[n];
        wr_aux = false;
      } else if (p.mode == MODE_LSERK) {
        const float4 av = *reinterpret_cast<const float4*>(aux + o);
        const float aa[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          w1[n] = cca * aa[n] + cdt * r[n];
          w0[n] = qq[n] + ccb * w1[n];
        }
      } else if (p.stage == 0) {  // classical RK4, first stage
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          w1[n] = r[n];
          w0[n] = qq[n] + cca * r[n];
        }
      } else {
        const float4 av = *reinterpret_cast<const float4*>(aux + o), bv = *reinterpret_cast<const float4*>(q0 + o);
        const float aa[4] = {av.x, av.y, av.z, av.w}, ba[4] = {bv.x, bv.y, bv.z, bv.w};
        if (p.stage < 3) {
#pragma unroll
          for (int n = 0; n < 4; ++n) {
            w1[n] = aa[n] + ccb * r[n];
            w0[n] = ba[n] + cca * r[n];
          }
        } else {  // last stage updates the base state only
#pragma unroll
          for (int n = 0; n < 4; ++n) w0[n] = w1[n] = ba[n] + cca * (aa[n] + r[n]);
          wr_out = wr_aux = false;
          wr_q0 = true;
        }
      }
      // padding nodes are written as 0
#pragma unroll
      for (int n = 1; n < 4; ++n)
        if (n0 + n >= Np) w0[n] = w1[n] = 0.0f;
      if (wr_out) *reinterpret_cast<float4*>(out + o) = make_float4(w0[0], w0[1], w0[2], w0[3]);
      if (wr_aux) *reinterpret_cast<float4*>(aux + o) = make_float4(w1[0], w1[1], w1[2], w1[3]);
      if (wr_q0) *reinterpret_cast<float4*>(q0 + o) = make_float4(w1[0], w1[1], w1[2], w1[3]);
    }
  }
}

template <int N, int P>
__global__ void __launch_bounds__(SymConfig<N, P>::kThreads, SymConfig<N, P>::kThreads <= 160 ? 6 : 4)
    dg_rhs_sym_kernel(const RhsParams p) {
  using C = SymConfig<N, P>;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + C::oBar);  // [0] set-up data, [1] state
  const int k0 = blockIdx.x * C::TE, ne = min(C::TE, p.K - k0);
  if (threadIdx.x == 0) {
    *reinterpret_cast<int*>(smem + C::oBnd + C::kBnd * 8) = 0;
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_barrier_init();
    mbar_arrive_expect_tx(&bar[0], C::kOps + C::kTab + ne * 80);
    bulk_g2s(smem + C::oOps, p.mats_sym, C::kOps, &bar[0]);
    bulk_g2s(smem + C::oTab, p.tab_eo, C::kTab, &bar[0]);
    bulk_g2s(smem + C::oGeom, static_cast<const float*>(p.geom) + (size_t)k0 * 16, ne * 64, &bar[0]);
    bulk_g2s(smem + C::oNbr, p.nbr + k0, ne * 16, &bar[0]);
  }
  __syncthreads();
  if (!__syncthreads_and(mbar_wait(&bar[0], 0, p.status))) return;
  // operators and geometry are set-up data; the state, the residual and the
  // device time are the previous launch's output
  grid_dep_wait();
  if (threadIdx.x == 0) {
    const uint32_t bytes = ne * C::ESTR * 4;
    mbar_arrive_expect_tx(&bar[1], bytes);
    bulk_g2s(smem + C::oQ, static_cast<const float*>(p.q_in) + (size_t)k0 * C::ESTR, bytes, &bar[1]);
  }
  const double tnow = P == PHYS_ADV ? (p.t_dev ? *p.t_dev + p.t : p.t) : 0.0;
  sym_tile<N, P>(p, smem, &bar[1], k0, ne, tnow);
}

}  // namespace dgk
