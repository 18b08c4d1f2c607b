// eo.hpp -- even / odd form of the reference element's operators.
//
// The nodes, the face nodes and the operators are symmetric under the
// reflection r <-> s of the reference triangle: with S the node permutation
// (i, j) -> (j, i) of the node lattice, Ds = S Dr S, LIFT = S LIFT S_f (S_f the
// permutation of the face-node list it induces) and M = S M S.  In the basis of
// sums e_c = u_a + u_b and differences o_c = u_a - u_b of the node pairs
// (a, b = S a) -- a node on the axis is its own sum --
//   D+ = (Dr + Ds) / 2 maps sums to sums and differences to differences,
//   D- = (Dr - Ds) / 2 maps sums to differences and differences to sums,
//   LIFT and M map sums to sums and differences to differences,
// so Dr and Ds together take Np^2 products per field instead of 2 Np^2, and
// LIFT and M half of theirs.  Dx = (rx + sx) D+ + (rx - sx) D-, likewise Dy.
//
// Outputs are half sums E_c = (f_a + f_b) / 2 (f_a on the axis) and half
// differences O_c = (f_a - f_b) / 2: f_a = E_c + O_c, f_b = E_c - O_c.
//
// Order: pairs c = 0 .. nP-1 first, then the nF axis nodes (sums only); rows
// and columns are [nE sums | nO differences], nE = nP + nF, nO = nP.  Face-node
// pairs: c < Nfp pairs node c of face 0 with node N - c of face 2, then the
// pairs (d, N - d) of face 1, then its middle node (N even).
//
// Operators without the symmetry (dgc_set_operators) go to the node-by-node
// kernels.  A graph that a caller captured before still holds the kernels of this
// form: for it the tables carry a flag, and the blob the operators' rest, which
// maps where the parts above do not (D+ sums to differences, LIFT difference
// columns to sum rows, ...), in the same layout.  A kernel that finds the flag adds
// it from global memory.
#pragma once

#include <cstdint>
#include <vector>

#if defined(__CUDACC__)
#define DGC_HD __host__ __device__
#else
#define DGC_HD
#endif

namespace dgk {

struct EoDims {
  int N, Np, Nfp, nF, nP, nE, nO, fE, fO;
  DGC_HD constexpr explicit EoDims(int n)
      : N(n), Np((n + 1) * (n + 2) / 2), Nfp(n + 1), nF(n / 2 + 1), nP((Np - (n / 2 + 1)) / 2), nE(nP + nF), nO(nP),
        fE(n + 1 + (n + 2) / 2), fO(n + 1 + (n + 1) / 2) {}
  // operand blob, in elements of the kernel type (each part padded to 16 bytes
  // for FP32 and FP64): K [Np columns][Np rows] (D+ and D-), L [fE][Np] (LIFT),
  // M [nE][Np] (mass, taking the half sums and half differences the rows give;
  // its difference rows have nO columns)
  DGC_HD constexpr int kK() const { return (Np * Np + 3) / 4 * 4; }
  DGC_HD constexpr int kL() const { return (fE * Np + 3) / 4 * 4; }
  DGC_HD constexpr int kM() const { return (nE * Np + 3) / 4 * 4; }
  // tables: pair (a, b) per sum column, pair (m1, m2) per face sum column, per node
  // its pair | 128 for the second member, then the flag: 1 with a rest (which
  // follows the tables in memory)
  DGC_HD constexpr int flag() const { return 2 * nE + 2 * fE + Np; }
  DGC_HD constexpr int tabBytes() const { return (flag() + 1 + 15) / 16 * 16; }
};

// FP64 instructions of a tile kernel per row (contraction to update), per
// face-node pair, per node pair and per item of its constants
struct EoCost {
  int row, flux, in, cst;
};

// Number of tiles (one CTA of 256 threads each, at most te_max elements, cut
// evenly, TileCut): the tile size with the least
// FP64 work on the busiest SM, in warp instructions.  A tile costs its phases'
// warps times their instructions (a partly filled warp costs a full one) plus a
// fixed share for its barriers and copies; an SM gets ceil(tiles / SMs) of them.
// The model follows the measured times within 5 % over tile sizes: stage kernel,
// Maxwell TE, K = 2048, N = 6: 17.3 us at the 7 or 8 elements it picks against
// 20.1 at the largest tile (9), 18.3 at 5 and 22.5 at 4; K = 8192, N = 4: 27.0 us
// at 14 against 31.3 at 17 and 31.3 at 8.  Where one tile per SM is enough, every
// SM gets one (an SM left out draws several CTAs of an overlapped next launch).
inline int eo_pick_tiles(const EoDims& d, int K, int sm_count, int te_max, const EoCost& w) {
  auto warps = [](int lanes) { return (lanes + 31) / 32; };
  int best = 1;
  long long cost = -1;
  for (int te = te_max; te >= 1; --te) {
    const int tile = warps(te * d.Np) * w.row + warps(te * d.fE) * w.flux + warps(te * d.nE) * w.in +
                     warps(te * 8) * w.cst + 64;
    const long long c = (long long)(((K + te - 1) / te + sm_count - 1) / sm_count) * tile;
    if (cost < 0 || c < cost) {
      cost = c;
      best = (K + te - 1) / te;
    }
  }
  return best < sm_count ? (K < sm_count ? K : sm_count) : best;
}

// K elements cut into n tiles of K / n elements, the first K % n tiles one more
struct TileCut {
  int len, rem;
  DGC_HD TileCut(int K, int n) : len((int)((unsigned)K / (unsigned)n)), rem(K - len * n) {}
  DGC_HD int start(int i) const { return i * len + (i < rem ? i : rem); }
  DGC_HD int size(int i) const { return len + (i < rem ? 1 : 0); }
};

// K elements cut into tiles of len elements, the last one shorter
struct TileRun {
  int K, len;
  DGC_HD int start(int i) const { return i * len; }
  DGC_HD int size(int i) const { return K - i * len < len ? K - i * len : len; }
};

// Tiles of the register-blocked kernels (FP32 and compensated stages, FP32 CG), cut
// evenly (TileCut): as many as full tiles make, at least one per SM.  On meshes with
// fewer full tiles than SMs a launch is latency (FP32 stage, Maxwell TE, K = 128,
// N = 3: 3.8 -> 3.0 us; CG iteration, K = 3200, N = 3: 19.8 -> 15.0 us with the
// convergence test in the grad pass); rounding larger counts up to whole waves took
// the CG iteration at K = 131072, N = 4 from 95 to 98 us.
inline int blk_tiles_for(int K, int sm_count, int te_max) {
  const int full = (K + te_max - 1) / te_max;
  return full >= sm_count ? full : (K < sm_count ? K : sm_count);
}

}  // namespace dgk

namespace dgc {

// Node and face-node pair tables of order N, as the blob stores them:
// 2 nE node indices, 2 fE face-node indices (f Nfp + d; the two members of an
// unpaired entry are equal), then per node its pair | 128 for the second member
// and the flag.
std::vector<uint8_t> eo_tables(int N, bool rest = false);

// Whether (Dr, Ds, L, M) have the reflection symmetry to rounding (1e-13 of
// their largest entry); M may be null.  Operators a caller has replaced by ones
// without it keep the general kernels.
bool eo_symmetric(int N, const std::vector<double>& Dr, const std::vector<double>& Ds, const std::vector<double>& L,
                  const std::vector<double>* M);

// Whether the weak form's volume and flux terms cancel for a constant state (to
// 1e-10 of the largest face row sum): Dr 1 = l1 - l2 and Ds 1 = l1 - l0 with l_f the
// sums of LIFT's columns of face f.  With straight-sided geometry (straight_sided)
// the right-hand side of q then equals that of q - c, element by element.
bool eo_constants_cancel(int N, const std::vector<double>& Dr, const std::vector<double>& Ds,
                         const std::vector<double>& L);

// The K, L and M parts of the blob (M left out when null), in FP64; rest: the K and
// L parts of the operators' rest (the mass matrix always has the symmetry).
std::vector<double> eo_pack(int N, const std::vector<double>& Dr, const std::vector<double>& Ds,
                            const std::vector<double>& L, const std::vector<double>* M, bool rest = false);

}  // namespace dgc
