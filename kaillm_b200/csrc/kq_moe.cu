// Mixture-of-experts GEMV/GEMM over expert-major GGUF weights W[E][n][row bytes]: every output row z of Y is one
// (token, expert) pair, y[z] = W[expert(z)] * q8_1(x[token(z)]).
//
//   vec    (ggml_moe_a8_vec, vllm_gguf_plugin/csrc/gguf/moe_vec.cuh:4-52, gguf_kernel.cu:395-530): z = token * top_k + j,
//          expert = topk_ids[z]; MMVQ arithmetic (vecdotq.cuh vec_dot_*_q8_1)
//   block  (ggml_moe_a8, csrc/gguf/moe.cuh:9-128, gguf_kernel.cu:292-393): the (token, expert) pairs arrive sorted by
//          expert in blocks of KQ_MOE_BLOCK slots (vLLM's moe_align_block_size with the size ggml_moe_get_block_size
//          returns); block b belongs to expert_ids[b], slot s holds z = sorted_token_ids[s] (z >= tokens * top_k: padding),
//          token = z / top_k; MMQ arithmetic.  A block's weights are decoded once for all of its slots.
//
// Block mode runs here only where the integer GEMM (kq_mmq.cu: a weight decoded once per run of up to 64 slots) does not take
// it: weights that are not 16-byte aligned, or option moe_smem = 0.
//
// One warp per weight row: lanes take 32-weight sub-blocks round-robin, decode them to int8 words and form the exact
// integer dots with dp4a (the same arithmetic as the general GEMV kernel).  Experts outside [0, E) and padding slots are
// skipped, their output rows keep what the caller put there (the reference returns zeros for them).
#include "kq_common.cuh"

namespace kq {

namespace {

__device__ const uint16_t c_iq3s_codes_moe[512] = {
#include "kq_iq3s_codes.inc"
};

struct MoeParams {
  const uint8_t* W;
  int64_t rowbytes, expert_stride;   // bytes per row / per expert
  int n, nsb, experts;
  const __half2* ds;                 // activation scales [tokens][kpad/32]
  const int8_t* qs;                  // activation codes [tokens][kpad]
  int kpad, tokens, top_k;
  const int32_t* ids;                // vec: topk_ids [tokens * top_k]; block: sorted_token_ids
  const int32_t* expert_ids;         // block mode only
  const int32_t* num_post_padded;    // block mode only
  int zero_bad;                      // vec: 1 = the output rows of pairs without a valid expert are written as zeros
  int64_t wbytes;                    // size of the whole weight tensor
  int rows, stage_bytes;             // staged vec kernel: rows per CTA (a multiple of 16), bytes of one stage of a warp's ring
  int64_t nslots;                    // tokens * top_k (vec) / entries of sorted_token_ids (block)
  void* y;
  int64_t stride_y;
};

template <int QT, int MT, bool MMQ, bool BLOCK, typename OutT>
__global__ void __launch_bounds__(128) moe_dp4a_kernel(const MoeParams p) {
  using F = Fmt<QT>;
  __shared__ uint32_t s_grid[QT == KQ_TYPE_IQ3_S ? 512 : 1];
  if constexpr (QT == KQ_TYPE_IQ3_S) {
    for (int i = threadIdx.x; i < 512; i += blockDim.x) s_grid[i] = iq3s_expand(c_iq3s_codes_moe[i], KQ_IQ3S_TOP);
    __syncthreads();
  }
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= p.n) return;
  const int64_t total = (int64_t)p.tokens * p.top_k;
  // the slots of this CTA: their activation rows and output rows (-1: nothing to do)
  int tok[MT], dst[MT];
  int expert;
  if constexpr (BLOCK) {
    const int64_t s0 = (int64_t)blockIdx.y * MT;
    if (s0 > (int64_t)p.num_post_padded[0]) return;   // the reference's bound (moe.cuh:37)
    expert = p.expert_ids[blockIdx.y];
#pragma unroll
    for (int t = 0; t < MT; ++t) {
      const int64_t s = s0 + t;
      const int z = s < p.nslots ? p.ids[s] : -1;
      const bool ok = z >= 0 && z < total;
      dst[t] = ok ? z : -1;
      tok[t] = ok ? z / p.top_k : 0;
    }
  } else {
    const int64_t z = blockIdx.y;
    expert = p.ids[z];
    dst[0] = (int)z;
    tok[0] = (int)(z / p.top_k);
  }
  if (expert < 0 || expert >= p.experts) {
    if (!BLOCK && p.zero_bad && lane == 0) reinterpret_cast<OutT*>(p.y)[(size_t)dst[0] * p.stride_y + row] = from_f32<OutT>(0.f);
    return;
  }
  const uint8_t* wrow = p.W + (size_t)expert * p.expert_stride + (size_t)row * p.rowbytes;
  const int nb8 = p.kpad >> 5;
  constexpr int NG = 32 / F::GROUP;

  float acc[MT];
#pragma unroll
  for (int t = 0; t < MT; ++t) acc[t] = 0.f;
  for (int sb = lane; sb < p.nsb; sb += 32) {
    SubBlock s;
    decode_subblock<QT>(wrow, sb, s_grid, s);
#pragma unroll
    for (int t = 0; t < MT; ++t) {
      if (dst[t] >= 0) {
        const uint4* ap = reinterpret_cast<const uint4*>(p.qs + (size_t)tok[t] * p.kpad + (size_t)sb * 32);
        const uint4 u0 = ap[0], u1 = ap[1];
        const float2 dsf = __half22float2(p.ds[(size_t)tok[t] * nb8 + sb]);
        const uint32_t u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
        int I[2] = {0, 0}, S[2] = {0, 0};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int h = (NG == 2) ? (i >> 2) : 0;
          I[h] = __dp4a((int)s.v[i], (int)u[i], I[h]);
          if (F::HAS_MIN) S[h] = __dp4a(0x01010101, (int)u[i], S[h]);
        }
        float c;
        if constexpr (HalfProd<QT>::value) {
          c = __half2float(__float2half_rn(s.wa[0] * dsf.x)) * (float)I[0] - __half2float(__float2half_rn(s.wb[0] * dsf.y));
        } else if constexpr (NG == 1) {
          c = s.wa[0] * (dsf.x * (float)I[0]);
          if constexpr (F::HAS_MIN) {
            const float z = RawSum<QT, MMQ>::value ? dsf.y : dsf.x * (float)S[0];
            c -= s.wb[0] * z;
          }
        } else {
          c = dsf.x * (s.wa[0] * (float)I[0] + s.wa[1] * (float)I[1]);
          if constexpr (F::HAS_MIN) c -= dsf.x * (s.wb[0] * (float)S[0] + s.wb[1] * (float)S[1]);
        }
        acc[t] += c;
      }
    }
  }
  OutT* y = reinterpret_cast<OutT*>(p.y);
#pragma unroll
  for (int t = 0; t < MT; ++t) {
    float v = acc[t];
#pragma unroll
    for (int mask = 16; mask > 0; mask >>= 1) v += __shfl_xor_sync(0xffffffffu, v, mask);
    if (lane == 0 && dst[t] >= 0) y[(size_t)dst[t] * p.stride_y + row] = from_f32<OutT>(v);
  }
}

// Vec mode: the pair's activations in shared memory.  A CTA of eight warps copies the q8_1 codes and scales of its token
// once and then walks MOE_ROWS_PER_CTA rows of the expert (a warp takes MOE_RW rows at a time), so the activations are read
// from global memory once per 64 rows instead of once per row.  Same arithmetic, same order of additions per row as
// moe_dp4a_kernel (bit-identical results).  Measured on 32 experts x Q4_K 2816x2048, top-4, 8 tokens: 42 -> 38 us (the
// reference's kernel: 63); four rows per warp were slower than two (128 registers).
constexpr int MOE_ROWS_PER_CTA = 64;
#ifndef MOE_RW
#define MOE_RW 2
#endif
template <int QT, bool MMQ, typename OutT>
__global__ void __launch_bounds__(256) moe_vec_smem_kernel(const MoeParams p) {
  using F = Fmt<QT>;
  extern __shared__ __align__(16) uint8_t moe_smem[];
  __shared__ uint32_t s_grid[QT == KQ_TYPE_IQ3_S ? 512 : 1];
  const int nb8 = p.kpad >> 5;
  int8_t* sQ = reinterpret_cast<int8_t*>(moe_smem);                          // [kpad]
  __half2* sDS = reinterpret_cast<__half2*>(moe_smem + p.kpad);              // [kpad / 32]
  if constexpr (QT == KQ_TYPE_IQ3_S) {
    for (int i = threadIdx.x; i < 512; i += blockDim.x) s_grid[i] = iq3s_expand(c_iq3s_codes_moe[i], KQ_IQ3S_TOP);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t z = blockIdx.y;                                              // the grid row is the (token, expert) pair
  const int expert = p.ids[z], tok = (int)(z / p.top_k);
  if (expert < 0 || expert >= p.experts) {
    const int row = blockIdx.x * MOE_ROWS_PER_CTA + threadIdx.x;
    if (p.zero_bad && threadIdx.x < MOE_ROWS_PER_CTA && row < p.n) reinterpret_cast<OutT*>(p.y)[(size_t)z * p.stride_y + row] = from_f32<OutT>(0.f);
    return;
  }
  {
    const uint4* src = reinterpret_cast<const uint4*>(p.qs + (size_t)tok * p.kpad);
    for (int i = threadIdx.x; i < (p.kpad >> 4); i += blockDim.x) reinterpret_cast<uint4*>(sQ)[i] = __ldg(src + i);
    for (int i = threadIdx.x; i < nb8; i += blockDim.x) sDS[i] = p.ds[(size_t)tok * nb8 + i];
  }
  __syncthreads();
  constexpr int NG = 32 / F::GROUP;
  OutT* y = reinterpret_cast<OutT*>(p.y);
  const int row_end = min(p.n, (int)(blockIdx.x + 1) * MOE_ROWS_PER_CTA);
  // a warp takes MOE_RW rows at a time: codes and scales are read from shared memory once for all of them
  constexpr int RW = MOE_RW;
  for (int row = blockIdx.x * MOE_ROWS_PER_CTA + RW * warp; row < row_end; row += 8 * RW) {
    const uint8_t* wrow0 = p.W + (size_t)expert * p.expert_stride + (size_t)row * p.rowbytes;
    float acc[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) acc[r] = 0.f;
    for (int sb = lane; sb < p.nsb; sb += 32) {
      SubBlock sw[RW];
#pragma unroll
      for (int r = 0; r < RW; ++r)   // rows past the end re-read the last row (their sums are not stored)
        decode_subblock<QT>(wrow0 + (size_t)(row + r < row_end ? r : 0) * p.rowbytes, sb, s_grid, sw[r]);
      // never taken: the branch keeps the 5-bit formats' loads of both rows ahead of the first dot.  Without it Q5_0 / Q5_1 / Q5_K
      // calls were 10 / 9 / 5 % slower (mean over eight shapes x 1 to 256 pairs, weights from memory); the others gain nothing
      if ((QT == KQ_TYPE_Q5_0 || QT == KQ_TYPE_Q5_1 || QT == KQ_TYPE_Q5_K) && tok < 0) continue;
      const uint4* ap = reinterpret_cast<const uint4*>(sQ + (size_t)sb * 32);
      const uint4 u0 = ap[0], u1 = ap[1];
      const float2 dsf = __half22float2(sDS[sb]);
      const uint32_t u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
      int S[2] = {0, 0};
      if constexpr (F::HAS_MIN && !RawSum<QT, MMQ>::value) {
#pragma unroll
        for (int i = 0; i < 8; ++i) S[(NG == 2) ? (i >> 2) : 0] = __dp4a(0x01010101, (int)u[i], S[(NG == 2) ? (i >> 2) : 0]);
      }
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        const SubBlock& s = sw[r];
        int I[2] = {0, 0};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int h = (NG == 2) ? (i >> 2) : 0;
          I[h] = __dp4a((int)s.v[i], (int)u[i], I[h]);
        }
        float c;
        if constexpr (HalfProd<QT>::value) {
          c = __half2float(__float2half_rn(s.wa[0] * dsf.x)) * (float)I[0] - __half2float(__float2half_rn(s.wb[0] * dsf.y));
        } else if constexpr (NG == 1) {
          c = s.wa[0] * (dsf.x * (float)I[0]);
          if constexpr (F::HAS_MIN) {
            const float zt = RawSum<QT, MMQ>::value ? dsf.y : dsf.x * (float)S[0];
            c -= s.wb[0] * zt;
          }
        } else {
          c = dsf.x * (s.wa[0] * (float)I[0] + s.wa[1] * (float)I[1]);
          if constexpr (F::HAS_MIN) c -= dsf.x * (s.wb[0] * (float)S[0] + s.wb[1] * (float)S[1]);
        }
        acc[r] += c;
      }
    }
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      float v = acc[r];
#pragma unroll
      for (int mask = 16; mask > 0; mask >>= 1) v += __shfl_xor_sync(0xffffffffu, v, mask);
      if (lane == 0 && row + r < row_end) y[(size_t)z * p.stride_y + row + r] = from_f32<OutT>(v);
    }
  }
}

// A sub-block out of a row staged in shared memory at its global address modulo 16; Q4_K (rows are 16-byte aligned): three
// 16-byte loads.
template <int QT>
__device__ __forceinline__ void decode_staged(const uint8_t* row, int sb, const uint32_t* grid, SubBlock& o) {
  if constexpr (QT == KQ_TYPE_Q4_K) {
    const uint8_t* b = row + (sb >> 3) * 144;
    const int j = sb & 7;
    const uint4 h = *reinterpret_cast<const uint4*>(b);
    const uint4* qp = reinterpret_cast<const uint4*>(b + 16 + 32 * (j >> 1));
    const uint4 q0 = qp[0], q1 = qp[1];
    const uint32_t scw = j < 4 ? h.y & 0x3F3F3F3Fu : (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
    const uint32_t mnw = j < 4 ? h.z & 0x3F3F3F3Fu : ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
    const float2 dd = __half22float2(*reinterpret_cast<const __half2*>(&h.x));
    const int sh = 8 * (j & 3), e4 = 4 * (j & 1);
    o.wa[0] = dd.x * (float)((scw >> sh) & 0xFFu); o.wb[0] = dd.y * (float)((mnw >> sh) & 0xFFu);
    o.wa[1] = 0.f; o.wb[1] = 0.f;
    const uint32_t q[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) o.v[i] = (q[i] >> e4) & 0x0F0F0F0Fu;
  } else {
    decode_subblock<QT, true>(row, sb, grid, o);
  }
}

// Vec mode with the weight rows staged as well: each warp runs its own ring of row pairs, filled by 16-byte cp.async pieces
// of the aligned window around the two rows, so that 2-byte aligned blocks cost coalesced requests and the loads run
// MOE_STAGES - 1 pairs ahead of the arithmetic.  Same arithmetic and order of additions as above (bit-identical).
// A CTA takes 128 rows where that gives four CTAs per SM, otherwise 64 (eight pairs of rows in a row per warp leave few
// calls enough CTAs: Q2_K 512x2048, 24 pairs, 30.9 us with 128 rows and 16.5 unstaged).
// Measured: 32 pairs over 32 experts, Q4_K 2816x2048 and Q8_0 2048x1408 (the rows' bytes are 3.2 and 3.1 MB a pair): the
// feed-forward call of 8 tokens 84.5 -> 61.3 us; unstaged the two kernels took 36 and 35 us, bound by their 2-byte loads.
constexpr int MOE_STAGES = 3;             // row pairs in a warp's ring: one being multiplied, two on their way
template <int QT, typename OutT>
__global__ void __launch_bounds__(256) moe_vec_staged_kernel(const MoeParams p) {
  using F = Fmt<QT>;
  extern __shared__ __align__(16) uint8_t moe_smem[];
  __shared__ uint32_t s_grid[QT == KQ_TYPE_IQ3_S ? 512 : 1];
  const int nb8 = p.kpad >> 5;
  int8_t* sQ = reinterpret_cast<int8_t*>(moe_smem);                          // [kpad]
  __half2* sDS = reinterpret_cast<__half2*>(moe_smem + p.kpad);              // [kpad / 32]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint8_t* ring = moe_smem + p.kpad + nb8 * 4 + warp * MOE_STAGES * p.stage_bytes;
  const uint32_t ring_a = (uint32_t)__cvta_generic_to_shared(ring);
  pdl_trigger();
  if constexpr (QT == KQ_TYPE_IQ3_S) {
    for (int i = threadIdx.x; i < 512; i += blockDim.x) s_grid[i] = iq3s_expand(c_iq3s_codes_moe[i], KQ_IQ3S_TOP);
  }
  pdl_wait();
  OutT* y = reinterpret_cast<OutT*>(p.y);
  const int64_t z = blockIdx.y;                                              // the grid row is the (token, expert) pair
  const int expert = p.ids[z], tok = (int)(z / p.top_k);
  if (expert < 0 || expert >= p.experts) {
    const int row = blockIdx.x * p.rows + threadIdx.x;
    if (p.zero_bad && threadIdx.x < p.rows && row < p.n) y[(size_t)z * p.stride_y + row] = from_f32<OutT>(0.f);
    return;
  }
  const uint8_t* We = p.W + (size_t)expert * p.expert_stride;
  const uint8_t* wend = p.W + p.wbytes;
  const int row_end = min(p.n, (int)(blockIdx.x + 1) * p.rows);
  auto issue = [&](int it) {              // rows row, row + 1 of this warp's it-th pair
    const int row = blockIdx.x * p.rows + 2 * (warp + 8 * it);
    if (16 * it < p.rows && row < row_end) {
      const uint8_t* ga = We + (size_t)row * p.rowbytes;
      const uint8_t* a0 = reinterpret_cast<const uint8_t*>((uintptr_t)ga & ~(uintptr_t)15);
      const int bytes = (int)(ga - a0) + (row + 1 < row_end ? 2 : 1) * (int)p.rowbytes;
      const uint32_t dst = ring_a + (it % MOE_STAGES) * p.stage_bytes;
      for (int c = lane * 16; c < bytes; c += 512) {
        // of the tensor's last piece only the bytes that exist are read (the rest is zero-filled)
        const uint32_t have = a0 + c + 16 <= wend ? 16u : (uint32_t)(wend - (a0 + c));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + c), "l"(a0 + c), "r"(have) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int i = 0; i < MOE_STAGES - 1; ++i) issue(i);
  {
    const uint4* src = reinterpret_cast<const uint4*>(p.qs + (size_t)tok * p.kpad);
    for (int i = threadIdx.x; i < (p.kpad >> 4); i += blockDim.x) reinterpret_cast<uint4*>(sQ)[i] = __ldg(src + i);
    for (int i = threadIdx.x; i < nb8; i += blockDim.x) sDS[i] = p.ds[(size_t)tok * nb8 + i];
  }
  __syncthreads();
  constexpr int NG = 32 / F::GROUP;
  for (int it = 0; 16 * it < p.rows; ++it) {
    const int row = blockIdx.x * p.rows + 2 * (warp + 8 * it);
    if (row >= row_end) break;
    asm volatile("cp.async.wait_group %0;" ::"n"(MOE_STAGES - 2) : "memory");
    __syncwarp();                         // every lane's pieces of this pair have landed; everyone is past the pair before it
    issue(it + MOE_STAGES - 1);           // into the buffer of the pair before it
    const uint8_t* w0 = ring + (it % MOE_STAGES) * p.stage_bytes + (((uint32_t)(uintptr_t)We + (uint32_t)row * (uint32_t)p.rowbytes) & 15u);
    const int step = row + 1 < row_end ? (int)p.rowbytes : 0;               // a missing second row re-reads the first
    float acc[2] = {0.f, 0.f};
    for (int sb = lane; sb < p.nsb; sb += 32) {
      const uint4* ap = reinterpret_cast<const uint4*>(sQ + (size_t)sb * 32);
      const uint4 u0 = ap[0], u1 = ap[1];
      const float2 dsf = __half22float2(sDS[sb]);
      const uint32_t u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
      int S[2] = {0, 0};
      if constexpr (F::HAS_MIN && !RawSum<QT, false>::value) {
#pragma unroll
        for (int i = 0; i < 8; ++i) S[(NG == 2) ? (i >> 2) : 0] = __dp4a(0x01010101, (int)u[i], S[(NG == 2) ? (i >> 2) : 0]);
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        SubBlock s;
        decode_staged<QT>(w0 + r * step, sb, s_grid, s);
        int I[2] = {0, 0};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int h = (NG == 2) ? (i >> 2) : 0;
          I[h] = __dp4a((int)s.v[i], (int)u[i], I[h]);
        }
        float c;
        if constexpr (HalfProd<QT>::value) {
          c = __half2float(__float2half_rn(s.wa[0] * dsf.x)) * (float)I[0] - __half2float(__float2half_rn(s.wb[0] * dsf.y));
        } else if constexpr (NG == 1) {
          c = s.wa[0] * (dsf.x * (float)I[0]);
          if constexpr (F::HAS_MIN) {
            const float zt = RawSum<QT, false>::value ? dsf.y : dsf.x * (float)S[0];
            c -= s.wb[0] * zt;
          }
        } else {
          c = dsf.x * (s.wa[0] * (float)I[0] + s.wa[1] * (float)I[1]);
          if constexpr (F::HAS_MIN) c -= dsf.x * (s.wb[0] * (float)S[0] + s.wb[1] * (float)S[1]);
        }
        acc[r] += c;
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float v = acc[r];
#pragma unroll
      for (int mask = 16; mask > 0; mask >>= 1) v += __shfl_xor_sync(0xffffffffu, v, mask);
      if (lane == 0 && row + r < row_end) y[(size_t)z * p.stride_y + row + r] = from_f32<OutT>(v);
    }
  }
}

// Staged rows (two CTAs share an SM) or the unstaged kernel?  Staging wins by the 2-byte loads it saves and the depth of its
// loads, and loses by fewer warps per SM and a start-up of its own, so it pays where an expert's matrix is large and the block
// awkward.  Staged / unstaged time of one call, geometric mean over eight shapes from 512x1024 to 5632x2048 x 1 to 256 pairs, weights from memory
// and (in brackets) from L2: above the lines drawn here Q6_K 0.70 (0.72), Q3_K 0.71 (0.80), Q4_K 0.79 (0.86), Q5_K 0.80 (0.91), Q8_0 0.81
// (0.82), Q5_1 0.81 (0.88), Q5_0 0.81 (0.94), Q2_K 0.87 (0.96), Q4_0 0.92 (0.94); below them up to 1.5 times slower.  Q4_1, IQ3_S, IQ4_NL
// and IQ4_XS decode from aligned or few words: 1.1 to 1.4 times slower at 64 pairs and more.
static bool moe_staged(int type, int64_t expert_bytes, int64_t pairs) {
  if (options().moe_smem != 1) return options().moe_smem == 2;
  switch (type) {
    case KQ_TYPE_Q8_0: case KQ_TYPE_Q3_K: case KQ_TYPE_Q4_K: case KQ_TYPE_Q5_K: case KQ_TYPE_Q6_K: return expert_bytes >= 1000000;
    case KQ_TYPE_Q4_0: case KQ_TYPE_Q5_1: case KQ_TYPE_Q2_K: return expert_bytes >= 1400000;
    case KQ_TYPE_Q5_0: return expert_bytes >= 1400000 && pairs <= 32;
    default: return false;
  }
}

template <int QT, bool MMQ, typename OutT>
int run_moe(const MoeParams& p, bool block, cudaStream_t st) {
  const unsigned gx = (unsigned)((p.n + 3) / 4);
  if (block) {
    const int64_t nblocks = (p.nslots + KQ_MOE_BLOCK - 1) / KQ_MOE_BLOCK;
    if (nblocks > 65535) { set_error("kq_moe_a8: more than 65535 blocks of sorted tokens"); return KQ_ELIMIT; }
    if (nblocks > 0) moe_dp4a_kernel<QT, KQ_MOE_BLOCK, MMQ, true, OutT><<<dim3(gx, (unsigned)nblocks), 128, 0, st>>>(p);
  } else {
    if (p.nslots > 65535) { set_error("kq_moe_a8_vec: more than 65535 (token, expert) pairs"); return KQ_ELIMIT; }
    const size_t smem = (size_t)p.kpad + (size_t)(p.kpad >> 5) * 4;
    // three stages of a row pair and its aligned window (plus the word that a funnel shift reads past a block) per warp, where two
    // CTAs then share an SM
    MoeParams ps = p;
    ps.stage_bytes = (int)((2 * p.rowbytes + 14 + 4 + 15) / 16 * 16);
    const size_t staged = smem + (size_t)8 * MOE_STAGES * ps.stage_bytes;
    if (p.nslots > 0 && staged <= 112 * 1024 && moe_staged(QT, p.expert_stride, p.nslots) && ((uintptr_t)p.W % 16) == 0) {
      auto kern = moe_vec_staged_kernel<QT, OutT>;
      static DeviceOnce staged_set;
      if (staged_set.first_time()) {
        KQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024));
        staged_set.done();
      }
      ps.rows = (p.n + 127) / 128 * p.nslots >= 4 * sm_count() ? 128 : 64;
      const unsigned gr = (unsigned)((p.n + ps.rows - 1) / ps.rows);
      KQ_CUDA_TRY(launch_pdl(kern, dim3(gr, (unsigned)p.nslots), dim3(256), staged, st, options().pdl != 0, ps));
      options().launches += 1;
      KQ_CUDA_TRY(cudaGetLastError());
      return KQ_OK;
    }
    if (p.nslots > 0 && smem <= 200 * 1024 && options().moe_smem) {
      auto kern = moe_vec_smem_kernel<QT, MMQ, OutT>;
      static DeviceOnce attr_set;
      if (attr_set.first_time()) {
        KQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr_set.done();
      }
      const unsigned gr = (unsigned)((p.n + MOE_ROWS_PER_CTA - 1) / MOE_ROWS_PER_CTA);
      kern<<<dim3(gr, (unsigned)p.nslots), 256, smem, st>>>(p);
    } else if (p.nslots > 0) {
      moe_dp4a_kernel<QT, 1, MMQ, false, OutT><<<dim3(gx, (unsigned)p.nslots), 128, 0, st>>>(p);
    }
  }
  options().launches += 1;
  KQ_CUDA_TRY(cudaGetLastError());
  return KQ_OK;
}

template <int QT, bool MMQ>
int run_moe_out(const MoeParams& p, bool block, int y_dtype, cudaStream_t st) {
  switch (y_dtype) {
    case KQ_F32: return run_moe<QT, MMQ, float>(p, block, st);
    case KQ_F16: return run_moe<QT, MMQ, __half>(p, block, st);
    case KQ_BF16: return run_moe<QT, MMQ, __nv_bfloat16>(p, block, st);
  }
  set_error("unsupported output dtype %d", y_dtype);
  return KQ_EUNSUPPORTED;
}

}  // namespace

// ---------------------------------------------------------------------------------------------- routing and combination
// moe_align_block_size for a call of at most MOE_ALIGN_SLOTS slots and MOE_ALIGN_EXPERTS experts, in one CTA: slots sorted
// by expert (in slot order inside an expert), every run padded to a multiple of `block` with `total`; expert id per block,
// -1 past the padded total; out[0] = padded total, out[1] = 1 if some id is outside [0, experts).  Stands for 25 launches of
// torch ops.  A counting sort: warp w owns the w-th stretch of slots and a row of counters; lanes of one expert find one another
// by match_any, so no counter is written twice at a time and the order stays the slots'.  Work grows with slots + 32 * experts; a
// scan of all slots by every expert (its predecessor) took 9 us at 32
// experts x 1024 slots, 127 at 128 x 8192 and 950 at 1024 x 8192 (the torch ops: 320 to 380).
constexpr int MOE_ALIGN_SLOTS = 8192, MOE_ALIGN_EXPERTS = 1024;
__global__ void __launch_bounds__(1024) moe_align_kernel(const int32_t* __restrict__ ids, int total, int experts, int block,
                                                         int32_t* __restrict__ sorted, int nsorted, int32_t* __restrict__ expert_ids,
                                                         int nblocks, int32_t* __restrict__ out) {
  extern __shared__ __align__(16) uint8_t moe_align_smem[];
  uint16_t* counts = reinterpret_cast<uint16_t*>(moe_align_smem);          // [32 warps][experts]: then offsets inside the run
  __shared__ int s_start[MOE_ALIGN_EXPERTS + 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint16_t* mine = counts + warp * experts;
  const int stretch = (total + 1023) / 1024 * 32;                          // slots of a warp
  const int first = warp * stretch, end = min(total, first + stretch);
  for (int i = lane; i < experts; i += 32) mine[i] = 0;
  for (int i = tid; i < nsorted; i += 1024) sorted[i] = total;
  __syncwarp();
  bool bad = false;
  for (int i0 = first; i0 < end; i0 += 32) {
    const int e = i0 + lane < end ? ids[i0 + lane] : -1;
    const bool ok = e >= 0 && e < experts;
    bad |= i0 + lane < end && !ok;
    const unsigned same = __match_any_sync(0xffffffffu, ok ? e : -1);
    if (ok && lane == __ffs(same) - 1) mine[e] += (uint16_t)__popc(same);
    __syncwarp();
  }
  const int any_bad = __syncthreads_or(bad);
  if (tid < experts) {                   // a thread per expert: the warps' offsets inside its run, then its padded length
    int run = 0;
#pragma unroll 8
    for (int w = 0; w < 32; ++w) {
      const int c = counts[w * experts + tid];
      counts[w * experts + tid] = (uint16_t)run;
      run += c;
    }
    s_start[tid + 1] = (run + block - 1) / block * block;
  }
  __syncthreads();
  if (warp == 0) {                       // running sum over the experts
    int run = 0;
    for (int e0 = 0; e0 < experts; e0 += 32) {
      int v = e0 + lane < experts ? s_start[e0 + lane + 1] : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += u;
      }
      if (e0 + lane < experts) s_start[e0 + lane + 1] = run + v;
      run += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) { s_start[0] = 0; out[0] = run; out[1] = any_bad != 0; }
  }
  __syncthreads();
  for (int i0 = first; i0 < end; i0 += 32) {
    const int e = i0 + lane < end ? ids[i0 + lane] : -1;
    const bool ok = e >= 0 && e < experts;
    const unsigned same = __match_any_sync(0xffffffffu, ok ? e : -1);
    const int base = ok ? mine[e] : 0;
    __syncwarp();
    if (ok) {
      sorted[s_start[e] + base + __popc(same & ((1u << lane) - 1u))] = i0 + lane;
      if (lane == __ffs(same) - 1) mine[e] = (uint16_t)(base + __popc(same));
    }
    __syncwarp();
  }
  for (int b = tid; b < nblocks; b += 1024) {     // the expert whose run holds slot b * block
    const int s = b * block;
    int lo = 0, hi = experts;
    while (lo < hi) {                    // first e with s_start[e + 1] > s
      const int mid = (lo + hi) >> 1;
      if (s_start[mid + 1] > s) hi = mid; else lo = mid + 1;
    }
    expert_ids[b] = lo < experts ? lo : -1;
  }
}

// out[t, c] = sum over the token's experts of T(y[t * top_k + j, c] * w[t, j]): products rounded to T, fp32 sum, as
// `(y.reshape(tokens, top_k, n) * w.to(T)).sum(1)`
template <typename T, typename WT>
__global__ void __launch_bounds__(256) moe_combine_kernel(const T* __restrict__ y, const WT* __restrict__ w, T* __restrict__ out, int n, int top_k) {
  const int c = blockIdx.x * 256 + threadIdx.x;
  const int64_t t = blockIdx.y;
  if (c >= n) return;
  float sum = 0.f;
  for (int j = 0; j < top_k; ++j) {
    const float wj = to_f32<T>(from_f32<T>(to_f32<WT>(w[t * top_k + j])));
    sum += to_f32<T>(from_f32<T>(to_f32<T>(y[(t * top_k + j) * n + c]) * wj));
  }
  out[t * n + c] = from_f32<T>(sum);
}

template <typename T>
static int run_combine(const void* y, const void* w, int w_dtype, void* out, int64_t tokens, int64_t n, int top_k, cudaStream_t st) {
  const dim3 grid((unsigned)((n + 255) / 256), (unsigned)tokens);
  switch (w_dtype) {
    case KQ_F32: moe_combine_kernel<T, float><<<grid, 256, 0, st>>>((const T*)y, (const float*)w, (T*)out, (int)n, top_k); break;
    case KQ_F16: moe_combine_kernel<T, __half><<<grid, 256, 0, st>>>((const T*)y, (const __half*)w, (T*)out, (int)n, top_k); break;
    default: moe_combine_kernel<T, __nv_bfloat16><<<grid, 256, 0, st>>>((const T*)y, (const __nv_bfloat16*)w, (T*)out, (int)n, top_k); break;
  }
  options().launches += 1;
  KQ_CUDA_TRY(cudaGetLastError());
  return KQ_OK;
}

int launch_moe_combine(const void* y, int dtype, const void* w, int w_dtype, void* out, int64_t tokens, int64_t n, int top_k, cudaStream_t st) {
  switch (dtype) {
    case KQ_F32: return run_combine<float>(y, w, w_dtype, out, tokens, n, top_k, st);
    case KQ_F16: return run_combine<__half>(y, w, w_dtype, out, tokens, n, top_k, st);
    default: return run_combine<__nv_bfloat16>(y, w, w_dtype, out, tokens, n, top_k, st);
  }
}

bool moe_align_supported(int64_t total, int64_t experts) { return total > 0 && total <= MOE_ALIGN_SLOTS && experts > 0 && experts <= MOE_ALIGN_EXPERTS; }

int launch_moe_align(const int32_t* ids, int64_t total, int64_t experts, int32_t* sorted, int64_t nsorted, int32_t* expert_ids, int64_t nblocks,
                     int32_t* out, cudaStream_t st) {
  static DeviceOnce attr_set;
  if (attr_set.first_time()) {
    KQ_CUDA_TRY(cudaFuncSetAttribute(moe_align_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * MOE_ALIGN_EXPERTS));
    attr_set.done();
  }
  moe_align_kernel<<<1, 1024, (size_t)(64 * experts), st>>>(ids, (int)total, (int)experts, KQ_MOE_BLOCK, sorted, (int)nsorted, expert_ids, (int)nblocks, out);
  options().launches += 1;
  KQ_CUDA_TRY(cudaGetLastError());
  return KQ_OK;
}

// block = false: ids = topk_ids; block = true: ids = sorted_token_ids (MMQ arithmetic)
int launch_moe(const void* W, int type, int64_t experts, int64_t n, int64_t k, const void* ds, const void* qs, int64_t kpad,
               int64_t tokens, int top_k, const int32_t* ids, int64_t nslots, const int32_t* expert_ids,
               const int32_t* num_post_padded, bool block, void* y, int y_dtype, int64_t stride_y, cudaStream_t st, int zero_bad) {
  int blk, bytes;
  if (!type_geometry(type, &blk, &bytes)) { set_error("unsupported GGML type %d", type); return KQ_EUNSUPPORTED; }
  MoeParams p;
  p.W = (const uint8_t*)W; p.rowbytes = k / blk * bytes; p.expert_stride = p.rowbytes * n; p.wbytes = p.expert_stride * experts; p.rows = 0; p.stage_bytes = 0; p.n = (int)n; p.nsb = (int)(k / 32);
  p.experts = (int)experts; p.ds = (const __half2*)ds; p.qs = (const int8_t*)qs; p.kpad = (int)kpad; p.tokens = (int)tokens;
  p.top_k = top_k; p.ids = ids; p.expert_ids = expert_ids; p.num_post_padded = num_post_padded; p.nslots = nslots;
  p.y = y; p.stride_y = stride_y; p.zero_bad = zero_bad;
  const bool mmq = block;
#define KQ_MOE_CASE(T) case T: return run_moe_out<T, false>(p, block, y_dtype, st)
#define KQ_MOE_CASE2(T) case T: return mmq ? run_moe_out<T, true>(p, block, y_dtype, st) : run_moe_out<T, false>(p, block, y_dtype, st)
  switch (type) {
    KQ_MOE_CASE(KQ_TYPE_Q4_0); KQ_MOE_CASE(KQ_TYPE_Q8_0); KQ_MOE_CASE(KQ_TYPE_Q2_K); KQ_MOE_CASE(KQ_TYPE_Q6_K);
    KQ_MOE_CASE(KQ_TYPE_IQ3_S); KQ_MOE_CASE(KQ_TYPE_Q4_1); KQ_MOE_CASE(KQ_TYPE_Q5_1); KQ_MOE_CASE(KQ_TYPE_Q3_K);
    KQ_MOE_CASE(KQ_TYPE_IQ4_NL); KQ_MOE_CASE(KQ_TYPE_IQ4_XS);
    KQ_MOE_CASE2(KQ_TYPE_Q4_K); KQ_MOE_CASE2(KQ_TYPE_Q5_0); KQ_MOE_CASE2(KQ_TYPE_Q5_K);
  }
#undef KQ_MOE_CASE
#undef KQ_MOE_CASE2
  set_error("unsupported GGML type %d", type);
  return KQ_EUNSUPPORTED;
}

}  // namespace kq
