// grad_div.cu -- weak-form gradient and divergence with central fluxes on the
// handle's mesh (C ABI: dgc_grad_apply, dgc_div_apply, dgc_boundary_nodes).
//
// grad_2d::operator() (src/grad_2d.h:141-187), per element k, node i:
//   gx = -(Dx u)_i + (1/J) sum_m LIFT_im faceJ_m nx_m (u- + u+)_m / 2
//   gy = -(Dy u)_i + (1/J) sum_m LIFT_im faceJ_m ny_m (u- + u+)_m / 2
// div_2d::operator() (src/div_2d.h:148-190):
//   d  = -(Dx ux + Dy uy)_i + (1/J) sum_m LIFT_im faceJ_m (n.(u- + u+))_m / 2
// with the weak Dr, Ds, LIFT of the advection operator, Dx = rx Dr + sx Ds,
// Dy = ry Dr + sy Ds, and the exterior trace u+ taken from the face neighbour
// (its face nodes in reverse order) or, on the boundary, from the caller's
// boundary data u+ = g + sign u- (the exterior_val callbacks of the
// reference's boundary-condition objects all have this form).
//
// FP64: even / odd form on the tile layout of ipdg_eo.cuh (k_grad_eo, k_div_eo),
// bound by the FP64 pipe: at K = 131072, N = 4 a gradient and a divergence take
// 338 us together on laplace handles, 522 us node by node (that pipe 94.6 % busy).  FP32, FP64
// operators without the reflection symmetry and inputs off a 16-byte boundary:
//
// Kernel: one CTA of 256 threads holds E = 256 / NpP elements; their fields are
// staged in shared memory, one thread per face node computes the central flux
// into shared memory, then one thread per (element, node) applies the
// operators (read from L1-resident global memory) and writes the result.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "dgc_gb300.h"
#include "dgc_internal.hpp"
#include "ipdg_eo.cuh"

namespace dgk {

template <typename R, int N, bool DIV>
__global__ void __launch_bounds__(256) k_grad_div(int K, const R* __restrict__ geom, const int4* __restrict__ nbr,
                                                  const R* __restrict__ mats, const R* __restrict__ u0,
                                                  const R* __restrict__ u1, const double* __restrict__ g0,
                                                  const double* __restrict__ g1, R sign, R* __restrict__ out0,
                                                  R* __restrict__ out1) {
  constexpr int Np = (N + 1) * (N + 2) / 2, Nfp = N + 1, NF = 3 * Nfp, NpP = (Np + 3) / 4 * 4;
  constexpr int E = 256 / NpP;
  constexpr int kD = (Np * Np + 3) / 4 * 4;
  __shared__ R sU[2][E * NpP];
  __shared__ R sF[E * NF];
  const int t = threadIdx.x;
  const int k0 = blockIdx.x * E;
  const int ne = min(E, K - k0);
  for (int q = t; q < ne * NpP; q += 256) {
    sU[0][q] = u0[(size_t)k0 * NpP + q];
    if (DIV) sU[1][q] = u1[(size_t)k0 * NpP + q];
  }
  __syncthreads();
  // central fluxes, pre-multiplied by faceJ (and by nothing else: grad applies n per component)
  for (int q = t; q < ne * NF; q += 256) {
    const int e = q / NF, m = q % NF, f = m / Nfp, d = m % Nfp;
    const int k = k0 + e;
    const R* G = geom + (size_t)k * 16;
    const int nd = fmask<N>(f, d);
    const R a0 = sU[0][e * NpP + nd];
    const R a1 = DIV ? sU[1][e * NpP + nd] : R(0);
    R b0, b1 = R(0);
    const int nb = (&nbr[k].x)[f];
    if (nb >= 0) {
      const int kn = nb >> 2, nd2 = fmask<N>(nb & 3, Nfp - 1 - d);
      b0 = u0[(size_t)kn * NpP + nd2];
      if (DIV) b1 = u1[(size_t)kn * NpP + nd2];
    } else {
      const size_t bi = (size_t)(-1 - nb) * Nfp + d;
      b0 = (g0 ? (R)g0[bi] : R(0)) + sign * a0;
      if (DIV) b1 = (g1 ? (R)g1[bi] : R(0)) + sign * a1;
    }
    const R fJ = G[5 + f];
    sF[q] = DIV ? (R(0.5) * ((a0 + b0) * G[8 + f] + (a1 + b1) * G[11 + f])) * fJ : (R(0.5) * (a0 + b0)) * fJ;
  }
  __syncthreads();
  const int e = t / NpP, i = t % NpP;
  if (e >= ne || i >= Np) return;
  const int k = k0 + e;
  const R* G = geom + (size_t)k * 16;
  const R rx = G[0], ry = G[1], sx = G[2], sy = G[3], invJ = -G[4];
  const R* DrT = mats;
  const R* DsT = mats + kD;
  const R* LT = mats + 2 * kD;
  const R* ua = sU[0] + e * NpP;
  const R* ub = sU[1] + e * NpP;
  R dr0 = R(0), ds0 = R(0), dr1 = R(0), ds1 = R(0);
#pragma unroll 4
  for (int j = 0; j < Np; ++j) {
    const R dr = __ldg(DrT + j * Np + i), ds = __ldg(DsT + j * Np + i);
    dr0 += dr * ua[j];
    ds0 += ds * ua[j];
    if (DIV) {
      dr1 += dr * ub[j];
      ds1 += ds * ub[j];
    }
  }
  const R* F = sF + e * NF;
  if (DIV) {
    R l = R(0);
#pragma unroll 4
    for (int m = 0; m < NF; ++m) l += __ldg(LT + m * Np + i) * F[m];
    out0[(size_t)k * NpP + i] = -(rx * dr0 + sx * ds0) - (ry * dr1 + sy * ds1) + invJ * l;
  } else {
    R lx = R(0), ly = R(0);
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      R lf = R(0);
      for (int d = 0; d < Nfp; ++d) lf += __ldg(LT + (f * Nfp + d) * Np + i) * F[f * Nfp + d];
      lx += lf * G[8 + f];
      ly += lf * G[11 + f];
    }
    out0[(size_t)k * NpP + i] = -(rx * dr0 + sx * ds0) + invJ * lx;
    out1[(size_t)k * NpP + i] = -(ry * dr0 + sy * ds0) + invJ * ly;
  }
}

template <typename R, bool DIV>
cudaError_t launch_grad_div(int N, int K, const R* geom, const int4* nbr, const R* mats, const R* u0, const R* u1,
                            const double* g0, const double* g1, R sign, R* out0, R* out1, cudaStream_t s) {
  auto go = [&](auto kern, int NpP) {
    const int E = 256 / NpP;
    kern<<<(K + E - 1) / E, 256, 0, s>>>(K, geom, nbr, mats, u0, u1, g0, g1, sign, out0, out1);
    return cudaGetLastError();
  };
  switch (N) {
    case 1: return go(k_grad_div<R, 1, DIV>, 4);
    case 2: return go(k_grad_div<R, 2, DIV>, 8);
    case 3: return go(k_grad_div<R, 3, DIV>, 12);
    case 4: return go(k_grad_div<R, 4, DIV>, 16);
    case 5: return go(k_grad_div<R, 5, DIV>, 24);
    case 6: return go(k_grad_div<R, 6, DIV>, 28);
    case 7: return go(k_grad_div<R, 7, DIV>, 36);
    case 8: return go(k_grad_div<R, 8, DIV>, 48);
    default: return cudaErrorInvalidValue;
  }
}

// Boundary data of k_grad_eo / k_div_eo: u+ = g[b] + sign u- (g may be NULL).
struct GradDivBc {
  const double *g0, *g1;
  double sign;
};

// gradient of p.u into p.qx, p.qy
template <int N>
__global__ void __launch_bounds__(256) k_grad_eo(const IpdgParams p, const GradDivBc bc) {
  using C = IpdgEo<N>;
  constexpr int Np = C::Np, NpP = C::NpP, Nfp = C::Nfp, nE = C::nE, nO = C::nO, fE = C::fE, fO = C::fO;
  extern __shared__ __align__(128) unsigned char smem[];
  const IpdgEoTile<N> t{smem};
  const int tid = threadIdx.x;
  const TileCut tiles(p.K, gridDim.x);
  const int k0 = tiles.start(blockIdx.x), ne = tiles.size(blockIdx.x);
  if (!t.setup(p, k0, ne, C::kOpsG, false)) return;
  const double* u = static_cast<const double*>(p.u);
  grid_dep_wait();
  grid_dep_launch();
  if (tid == 0) {
    mbar_arrive_expect_tx(t.bar() + 1, ne * NpP * 8);
    bulk_g2s(t.field(0), u + (size_t)k0 * NpP, ne * NpP * 8, t.bar() + 1);
  }
  const int fe = tid / fE, fc = tid - fe * fE;
  const bool fact = fe < ne, ftwo = fc < fO;
  double b[2] = {0.0, 0.0};
  bool bnd[2] = {false, false};
  if (fact) {
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      if (w && !ftwo) break;
      const int m = t.faces()[2 * fc + w], f = m / Nfp, d = m - f * Nfp;
      const int nb = nb_of<double, N>(t.nbr()[fe], f);
      if (nb >= 0) {
        b[w] = __ldg(u + (size_t)(nb >> 2) * NpP + fmask<N>(nb & 3, Nfp - 1 - d));
      } else {
        bnd[w] = true;
        if (bc.g0) b[w] = bc.g0[(size_t)(-1 - nb) * Nfp + d];
      }
    }
  }
  t.constants(p, ne);
  if (!__syncthreads_and(mbar_wait(t.bar() + 1, 0, p.status))) return;
  const double* sU = t.field(0);
  if (fact) {
    const double* c = t.consts() + fe * C::CSTR + IC_F;
    double lx[2] = {0.0, 0.0}, ly[2] = {0.0, 0.0};
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      if (w && !ftwo) break;
      const int m = t.faces()[2 * fc + w], f = m / Nfp, d = m - f * Nfp;
      const double um = sU[fe * NpP + fmask<N>(f, d)];
      const double us = um + (bnd[w] ? fma(bc.sign, um, b[w]) : b[w]);
      lx[w] = c[3 * f] * us;
      ly[w] = c[3 * f + 1] * us;
    }
    double* fo = t.flux() + fe * C::FSTR + fc;
    fo[0] = ftwo ? lx[0] + lx[1] : lx[0];
    fo[fE] = ftwo ? lx[0] - lx[1] : 0.0;
    fo[2 * fE] = ftwo ? ly[0] + ly[1] : ly[0];
    fo[3 * fE] = ftwo ? ly[0] - ly[1] : 0.0;
  }
  t.sum_diff(sU, ne);
  __syncthreads();
  t.template grad_rows<true>(p, ne, k0, static_cast<double*>(p.qx), static_cast<double*>(p.qy));
}

// divergence of (p.qx, p.qy) into p.out
template <int N>
__global__ void __launch_bounds__(256) k_div_eo(const IpdgParams p, const GradDivBc bc) {
  using C = IpdgEo<N>;
  constexpr int Np = C::Np, NpP = C::NpP, Nfp = C::Nfp, nE = C::nE, nO = C::nO, fE = C::fE, fO = C::fO;
  extern __shared__ __align__(128) unsigned char smem[];
  const IpdgEoTile<N> t{smem};
  const int tid = threadIdx.x;
  const TileCut tiles(p.K, gridDim.x);
  const int k0 = tiles.start(blockIdx.x), ne = tiles.size(blockIdx.x);
  if (!t.setup(p, k0, ne, C::kOpsG, false)) return;
  const double* u0 = static_cast<const double*>(p.qx);
  const double* u1 = static_cast<const double*>(p.qy);
  grid_dep_wait();
  grid_dep_launch();
  if (tid == 0) {
    mbar_arrive_expect_tx(t.bar() + 1, 2 * ne * NpP * 8);
    bulk_g2s(t.field(0), u0 + (size_t)k0 * NpP, ne * NpP * 8, t.bar() + 1);
    bulk_g2s(t.field(1), u1 + (size_t)k0 * NpP, ne * NpP * 8, t.bar() + 1);
  }
  const int fe = tid / fE, fc = tid - fe * fE;
  const bool fact = fe < ne, ftwo = fc < fO;
  double bx[2] = {0.0, 0.0}, by[2] = {0.0, 0.0};
  bool bnd[2] = {false, false};
  if (fact) {
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      if (w && !ftwo) break;
      const int m = t.faces()[2 * fc + w], f = m / Nfp, d = m - f * Nfp;
      const int nb = nb_of<double, N>(t.nbr()[fe], f);
      if (nb >= 0) {
        const size_t o = (size_t)(nb >> 2) * NpP + fmask<N>(nb & 3, Nfp - 1 - d);
        bx[w] = __ldg(u0 + o);
        by[w] = __ldg(u1 + o);
      } else {
        const size_t bi = (size_t)(-1 - nb) * Nfp + d;
        bnd[w] = true;
        if (bc.g0) bx[w] = bc.g0[bi];
        if (bc.g1) by[w] = bc.g1[bi];
      }
    }
  }
  t.constants(p, ne);
  if (!__syncthreads_and(mbar_wait(t.bar() + 1, 0, p.status))) return;
  const double *sX = t.field(0), *sY = t.field(1);
  if (fact) {
    const double* c = t.consts() + fe * C::CSTR + IC_F;
    double fl[2] = {0.0, 0.0};
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      if (w && !ftwo) break;
      const int m = t.faces()[2 * fc + w], f = m / Nfp, d = m - f * Nfp;
      const int nd = fe * NpP + fmask<N>(f, d);
      const double xm = sX[nd], ym = sY[nd];
      const double xs = xm + (bnd[w] ? fma(bc.sign, xm, bx[w]) : bx[w]);
      const double ys = ym + (bnd[w] ? fma(bc.sign, ym, by[w]) : by[w]);
      fl[w] = fma(c[3 * f], xs, c[3 * f + 1] * ys);
    }
    double* fo = t.flux() + fe * C::FSTR + fc;
    fo[0] = ftwo ? fl[0] + fl[1] : fl[0];
    fo[fE] = ftwo ? fl[0] - fl[1] : 0.0;
  }
  t.combine(sX, sY, ne);
  __syncthreads();
  const int e = tid / Np, r = tid - e * Np;
  const bool act = e < ne;
  const double au = act ? t.div_row(p, e, r) : 0.0;
  __syncthreads();
  double* ro = t.in() + e * 2 * Np;
  if (act) ro[r] = au;
  __syncthreads();
  if (act) static_cast<double*>(p.out)[(size_t)(k0 + e) * NpP + r] = t.template node<true>(ro, r);
}

template <int N, bool DIV>
cudaError_t launch_eo(const IpdgParams& p, const GradDivBc& bc, int sm, cudaStream_t s) {
  using C = IpdgEo<N>;
  auto kern = DIV ? k_div_eo<N> : k_grad_eo<N>;
  static std::once_flag once;
  static cudaError_t st = cudaSuccess;
  std::call_once(once, [&] {
    st = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemGrad);
  });
  if (st != cudaSuccess) return st;
  // the passes' cost, without the mass rows and with the constants formed here
  EoCost w = DIV ? EoCost{C::kCostDiv.row - C::nE, C::kCostDiv.flux, C::kCostDiv.in, 0} : C::kCostGrad;
  if (!p.consts) w.cst = 8;
  const int ntiles = eo_pick_tiles(C::D, p.K, sm, C::TE, w);
  if (ntiles <= sm) return launch_stage(kern, ntiles, 256, C::kSmemGrad, s, p, bc);
  kern<<<ntiles, 256, C::kSmemGrad, s>>>(p, bc);
  return cudaGetLastError();
}

template <bool DIV>
cudaError_t launch_grad_div_eo(int N, const IpdgParams& p, const GradDivBc& bc, int sm, cudaStream_t s) {
  switch (N) {
    case 1: return launch_eo<1, DIV>(p, bc, sm, s);
    case 2: return launch_eo<2, DIV>(p, bc, sm, s);
    case 3: return launch_eo<3, DIV>(p, bc, sm, s);
    case 4: return launch_eo<4, DIV>(p, bc, sm, s);
    case 5: return launch_eo<5, DIV>(p, bc, sm, s);
    case 6: return launch_eo<6, DIV>(p, bc, sm, s);
    case 7: return launch_eo<7, DIV>(p, bc, sm, s);
    case 8: return launch_eo<8, DIV>(p, bc, sm, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace dgk

using namespace dgc;

namespace {

int check_scalar_handle(dgc_handle h) {
  if (!h) return set_error(DGC_ERR_ARG, "null handle");
  if (h->Nf != 1) return set_error(DGC_ERR_UNSUPPORTED, "grad / div act on scalar-field (advection, laplace) handles");
  if (h->prec == DGC_F32C) return set_error(DGC_ERR_UNSUPPORTED, "grad / div are not offered for compensated FP32 handles");
  return DGC_OK;
}

template <typename R, bool DIV>
int grad_div(dgc_handle h, const void* u0, const void* u1, const double* g0, const double* g1, double sign,
             void* out0, void* out1, cudaStream_t s) {
  const bool f64 = sizeof(R) == 8;
  const R* geom = static_cast<const R*>(f64 ? (const void*)h->d_kgeom64 : (const void*)h->d_kgeom32);
  // the even / odd kernels copy their input tiles in bulk (16-byte aligned
  // buffers); others, and operators without the symmetry, go node by node
  const bool al = ((reinterpret_cast<uintptr_t>(u0) | reinterpret_cast<uintptr_t>(u1)) & 15u) == 0;
  if (f64 && h->eo_ok[0] && al) {
    dgk::IpdgParams p{};
    p.K = h->K;
    p.geom = h->d_kgeom64;
    p.nbr = reinterpret_cast<const int4*>(h->d_nbr);
    p.mats_eo = h->d_eo64[0];
    p.tab_eo = h->d_eo_tab[0];
    p.consts = ipdg_consts(h);
    p.status = h->d_status;
    p.u = u0;
    p.qx = DIV ? const_cast<void*>(u0) : out0;
    p.qy = DIV ? const_cast<void*>(u1) : out1;
    p.out = out0;
    const cudaError_t e = dgk::launch_grad_div_eo<DIV>(h->N, p, dgk::GradDivBc{g0, g1, sign}, h->sm_count, s);
    if (e != cudaSuccess) return set_error(DGC_ERR_CUDA, cudaGetErrorString(e));
    ++h->launches;
    return DGC_OK;
  }
  const R* mats = static_cast<const R*>(f64 ? (const void*)h->d_mats64[0] : (const void*)h->d_mats32[0]);
  cudaError_t e = dgk::launch_grad_div<R, DIV>(h->N, h->K, geom, reinterpret_cast<const int4*>(h->d_nbr), mats,
                                               static_cast<const R*>(u0), static_cast<const R*>(u1), g0, g1,
                                               (R)sign, static_cast<R*>(out0), static_cast<R*>(out1), s);
  if (e != cudaSuccess) return set_error(DGC_ERR_CUDA, cudaGetErrorString(e));
  ++h->launches;
  return DGC_OK;
}

}  // namespace

extern "C" int dgc_boundary_nodes(dgc_handle h, double* xy) {
  if (!h || !xy) return set_error(DGC_ERR_ARG, "null argument");
  std::copy(h->mesh.bxy.begin(), h->mesh.bxy.end(), xy);
  return DGC_OK;
}

extern "C" int dgc_grad_apply(dgc_handle h, const void* u, void* gx, void* gy, const double* g, double sign,
                              void* stream) {
  if (int rc = check_scalar_handle(h)) return rc;
  if (!u || !gx || !gy || gx == gy || u == gx || u == gy)
    return set_error(DGC_ERR_ARG, "u, gx, gy must be distinct, non-null buffers");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return h->prec == DGC_F64 ? grad_div<double, false>(h, u, nullptr, g, nullptr, sign, gx, gy, s)
                            : grad_div<float, false>(h, u, nullptr, g, nullptr, sign, gx, gy, s);
}

extern "C" int dgc_div_apply(dgc_handle h, const void* ux, const void* uy, void* out, const double* gx,
                             const double* gy, double sign, void* stream) {
  if (int rc = check_scalar_handle(h)) return rc;
  if (!ux || !uy || !out || out == ux || out == uy)
    return set_error(DGC_ERR_ARG, "ux, uy, out must be non-null and out distinct from the inputs");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return h->prec == DGC_F64 ? grad_div<double, true>(h, ux, uy, gx, gy, sign, out, nullptr, s)
                            : grad_div<float, true>(h, ux, uy, gx, gy, sign, out, nullptr, s);
}
