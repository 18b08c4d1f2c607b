// mpnn_tc.cuh -- the message-passing layer of the learned preconditioner on the
// tensor cores (tcgen05, BF16 operands, FP32 accumulation in tensor memory).
//
// Per graph node e the layer computes
//   a_e = Ws h_e + Wn m_e + b,   m_e = sum of h over the face neighbours of e,
//   h'_e = h_e + relu(a_e)   (or h_e + a_e for the linear network),
// i.e. for a tile of 128 nodes the product D[128 x 64] = X[128 x 128] W^T with
// X = [h | m] (FP32) and W = [Ws | Wn] (64 x 128, BF16 copies of the FP32
// master weights).  W is exact in BF16; X is not, so X is split into three
// BF16 parts X = X0 + X1 + X2 (each the leading bits of what the previous
// parts leave; 3 x 8 significand bits cover FP32's 24) and the tile is three
// accumulating products per K step.  The result matches the FP32 SIMT form of
// the same layer to FP32 accumulation round-off.
//
// The backward pass through the layer's input has the same form,
//   dh_e <- dh_e + Ws^T g_e + Wn^T (sum of g over the face neighbours),
// with X = [g | sum g] and the transposed weights.
//
// CTA: 256 threads, one 128-node tile at a time (persistent over tiles).
//   * W is staged once per CTA in shared memory (K-major, no swizzle, core
//     matrices of 8 rows x 16 bytes: element (row, k) at byte
//     (row / 8) * 2048 + (k / 8) * 128 + (row % 8) * 16 + (k % 8) * 2);
//   * a warp gathers 16 rows: 8 rows x 64 contiguous bytes per load instruction
//     (with a thread per row every load touched 32 lines: 187 us per layer at
//     262144 nodes, 73 us with this mapping and the epilogue below), 16 loads in
//     flight per thread;
//     the split is by truncation (exact: 8 + 8 + 8 bits, no conversions);
//   * one thread issues 3 parts x 8 K steps of MMAs (M = 128, N = 64, K = 16) into
//     64 TMEM columns and commits to an mbarrier (bounded wait);
//   * the epilogue moves D through the (now free) operand tile so that bias,
//     activation and the global accesses run on whole 256-byte rows.  The
//     backward form replaces an FP32 SIMT kernel (400 us at 262144 nodes, 86 us).
// Bound by DRAM and the gather's L2 traffic.  Shared memory 112 KB + barriers:
// 2 CTAs per SM, one gathering while the other multiplies; TMEM 64 columns each.
#pragma once

#include <cuda_bf16.h>

#include "dg_rhs_tct.cuh"

namespace dgk {

struct MpnnTc {
  static constexpr int kRows = 128;                 // nodes per tile (MMA M)
  static constexpr int kK = 128;                    // [h | m]
  static constexpr int kN = 64;                     // channels (MMA N)
  static constexpr int kThreads = 256;
  static constexpr uint32_t kSbo = (kK / 8) * 128;  // bytes between 8-row groups
  static constexpr uint32_t kBBytes = (kN / 8) * kSbo;     // 16 KB
  static constexpr uint32_t kABytes = (kRows / 8) * kSbo;  // 32 KB per split
  static constexpr uint32_t oBar = 0;               // mbarrier (8 B) + TMEM address (4 B)
  static constexpr uint32_t oBias = 16;             // 64 FP32 biases
  static constexpr uint32_t oB = 384;
  static constexpr uint32_t oA = oB + kBBytes;
  static constexpr uint32_t kSmem = oA + 3 * kABytes;
  static constexpr uint32_t kTmemCols = 64;
  static constexpr int kDStr = kN + 4;              // floats between rows of the staged D
  // instruction descriptor: D f32 (bits 4-5 = 1), A and B bf16 (bits 7-9, 10-12 = 1),
  // both K-major, N >> 3 at bit 17, M >> 4 at bit 24
  static constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kN >> 3) << 17) |
                                     ((uint32_t)(kRows >> 4) << 24);
  static_assert(kSmem % 16 == 0 && oA % 128 == 0 && kRows * kDStr * 4 <= 3 * kABytes, "operand alignment");
};

// face neighbours of graph node e (sample s = e / K): up to 3 node indices, -1 on the boundary
__device__ __forceinline__ void neighbours(const int4* __restrict__ nbr, int K, int64_t e, int64_t (&j)[3]) {
  const int64_t s = e <= 0x7fffffff ? (int64_t)((uint32_t)e / (uint32_t)K) : e / K;
  const int4 n4 = __ldg(nbr + (e - s * K));
  const int c[3] = {n4.x, n4.y, n4.z};
#pragma unroll
  for (int f = 0; f < 3; ++f) j[f] = c[f] >= 0 ? s * K + (c[f] >> 2) : -1;
}

__device__ __forceinline__ uint32_t tc_off(int row, int k) {  // byte offset of (row, k) in an operand
  return (uint32_t)((row >> 3) * MpnnTc::kSbo + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

__device__ __forceinline__ void tc_mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// four FP32 values -> three 8-byte rows of BF16 parts, x = p0 + p1 + p2 exactly:
// each part is the leading 8 significand bits of what the previous ones leave
// (infinities and NaN come out as NaN)
__device__ __forceinline__ void split3_store(const float4& x, unsigned char* a0) {
  const float v[4] = {x.x, x.y, x.z, x.w};
  uint32_t w[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float r = v[i];
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      w[p][i] = __float_as_uint(r) & 0xffff0000u;
      if (p < 2) r -= __uint_as_float(w[p][i]);
    }
  }
#pragma unroll
  for (int p = 0; p < 3; ++p)
    *reinterpret_cast<uint2*>(a0 + p * MpnnTc::kABytes) =
        make_uint2(__byte_perm(w[p][0], w[p][1], 0x7632), __byte_perm(w[p][2], w[p][3], 0x7632));
}

// BWD false: a_out (may be NULL) = W X + b, out = x + relu(a) (linear: x + a), x = the tile's own rows.
// BWD true:  out = add + W^T X.
template <bool BWD>
__global__ void __launch_bounds__(MpnnTc::kThreads, 2)
    k_layer_tc(int64_t n, int K, const int4* __restrict__ nbr, const __nv_bfloat16* __restrict__ Ws,
               const __nv_bfloat16* __restrict__ Wn, const __nv_bfloat16* __restrict__ bl,
               const float* __restrict__ x, const float* __restrict__ add, float* __restrict__ a_out,
               float* __restrict__ out, int linear, int* __restrict__ status) {
  using C = MpnnTc;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + C::oBar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::oBar + 8);
  unsigned char* sB = smem + C::oB;
  unsigned char* sA = smem + C::oA;
  float* sD = reinterpret_cast<float*>(sA);  // [row][kDStr], after the products
  float* sBias = reinterpret_cast<float*>(smem + C::oBias);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;

  if (t == 0) {
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  if (warp == 0) tmem_alloc_n(tmem_slot, C::kTmemCols);
  if (BWD) {
    // row i = input channel, column c (Ws) or 64 + c (Wn) = output channel
    for (int q = t; q < 2 * C::kN * C::kN; q += C::kThreads) {
      const int k = q / C::kN, i = q % C::kN;
      *reinterpret_cast<__nv_bfloat16*>(sB + tc_off(i, k)) = k < C::kN ? Ws[k * C::kN + i] : Wn[(k - C::kN) * C::kN + i];
    }
  } else {
    // row c = output channel, k < 64 from Ws[c][k], k >= 64 from Wn[c][k - 64];
    // 16-byte chunks of 8 consecutive k
    for (int q = t; q < C::kN * (C::kK / 8); q += C::kThreads) {
      const int c = q / (C::kK / 8), k0 = (q % (C::kK / 8)) * 8;
      const __nv_bfloat16* src = (k0 < C::kN ? Ws + c * C::kN + k0 : Wn + c * C::kN + (k0 - C::kN));
      *reinterpret_cast<uint4*>(sB + tc_off(c, k0)) = *reinterpret_cast<const uint4*>(src);
    }
    if (t < C::kN) sBias[t] = __bfloat162float(bl[t]);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t sA_u = smem_u32(sA), sB_u = smem_u32(sB);
  const int lrow = lane >> 2, lq = lane & 3;  // gather: row within 8, 4-channel quad within 4
  const int erow = (warp & 3) * 32 + lane, ecol = (warp >> 2) * 32;  // TMEM lanes and columns of the epilogue
  uint32_t phase = 0;
  bool ok = true;
  for (int64_t n0 = (int64_t)blockIdx.x * C::kRows; n0 < n && ok; n0 += (int64_t)gridDim.x * C::kRows) {
    // ---- X = [x | sum of x over the neighbours], split into three BF16 parts
#pragma unroll 1
    for (int hh = 0; hh < 2; ++hh) {
      const int row = warp * 16 + hh * 8 + lrow;
      const int64_t e = n0 + row;
      int64_t j[4] = {-1, -1, -1, -1};
      if (e < n) {
        int64_t nb[3];
        neighbours(nbr, K, e, nb);
        j[0] = e;
        j[1] = nb[0];
        j[2] = nb[1];
        j[3] = nb[2];
      }
      float4 v[4][4];
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const float4* src = reinterpret_cast<const float4*>(x + j[f] * C::kN) + lq;
#pragma unroll
        for (int u = 0; u < 4; ++u) v[f][u] = j[f] >= 0 ? __ldg(src + 4 * u) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = 4 * (lq + 4 * u);
        split3_store(v[0][u], sA + tc_off(row, k));
        const float4 m = make_float4((v[1][u].x + v[2][u].x) + v[3][u].x, (v[1][u].y + v[2][u].y) + v[3][u].y,
                                     (v[1][u].z + v[2][u].z) + v[3][u].z, (v[1][u].w + v[2][u].w) + v[3][u].w);
        split3_store(m, sA + tc_off(row, C::kN + k));
      }
    }
    // generic-proxy stores of X -> visible to the tensor core's async proxy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (t == 0) {
      // the small parts first, so that only the leading part's 8 steps round at full
      // magnitude (gradient error against 64 bits at K = 32768, 8 samples: 2.6e-6
      // part by part within each step, 0.7-1.1e-6 so; an FP32 SIMT layer 1.2-2.1e-6)
#pragma unroll
      for (int p = 2; p >= 0; --p)
#pragma unroll
        for (int s = 0; s < C::kK / 16; ++s) {
          const uint64_t db = smem_desc(sB_u + s * 256, 128, C::kSbo);
          const uint64_t da = smem_desc(sA_u + p * C::kABytes + s * 256, 128, C::kSbo);
          tc_mma_bf16(tmem, da, db, C::kIdesc, (s > 0 || p < 2) ? 1u : 0u);
        }
      tc_commit(bar);
    }
    ok = __syncthreads_and(mbar_wait(bar, phase, status));
    if (!ok) {
      // error path (recorded in the status word): give the MMAs in flight one
      // more bounded wait before the tensor memory is released
      mbar_wait(bar, phase, nullptr);
      break;
    }
    phase ^= 1;
    tc_fence_after();
    // ---- epilogue: D to shared memory (the operand tile has been consumed),
    //      then by whole rows
    {
      float d[32];
      tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + ecol, d);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        *reinterpret_cast<float4*>(sD + erow * C::kDStr + ecol + 4 * q) =
            make_float4(d[4 * q], d[4 * q + 1], d[4 * q + 2], d[4 * q + 3]);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
#pragma unroll
    for (int i = 0; i < C::kRows * 16 / C::kThreads; ++i) {
      const int row = (t >> 4) + 16 * i, c = 4 * (t & 15);
      const int64_t e = n0 + row;
      if (e >= n) break;
      const size_t o = (size_t)e * C::kN + c;
      const float4 d = *reinterpret_cast<const float4*>(sD + row * C::kDStr + c);
      if (BWD) {
        const float4 b = *reinterpret_cast<const float4*>(add + o);
        *reinterpret_cast<float4*>(out + o) = make_float4(b.x + d.x, b.y + d.y, b.z + d.z, b.w + d.w);
      } else {
        const float4 bq = *reinterpret_cast<const float4*>(sBias + c);
        const float4 a = make_float4(d.x + bq.x, d.y + bq.y, d.z + bq.z, d.w + bq.w);
        if (a_out) *reinterpret_cast<float4*>(a_out + o) = a;
        const float4 hh = __ldg(reinterpret_cast<const float4*>(x + o));
        *reinterpret_cast<float4*>(out + o) =
            linear ? make_float4(hh.x + a.x, hh.y + a.y, hh.z + a.z, hh.w + a.w)
                   : make_float4(hh.x + fmaxf(a.x, 0.f), hh.y + fmaxf(a.y, 0.f), hh.z + fmaxf(a.z, 0.f),
                                 hh.w + fmaxf(a.w, 0.f));
      }
    }
    __syncthreads();  // the tile's shared rows consumed before the next tile overwrites them
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc_n(tmem, C::kTmemCols);
}

}  // namespace dgk
