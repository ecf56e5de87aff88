// Integer-dot GEMM (q8_1 activations, exact int8 dots) for many tokens: linear calls of the formats the tcgen05 GEMM does
// not take, and the expert-sorted mixture-of-experts op.
//
//   y[tok, row] = sum over 32-weight sub-blocks of  wa * (d8 * I) - wb * z      (SubBlock in kq_common.cuh)
//
// The row-streaming GEMV re-reads and re-decodes a weight for every 8 tokens, the old block op for every 8 slots.  Here a
// weight is decoded once per 64 tokens (or slots of one expert): decoding is what bounded both (Q5_K 6144x5120 at 333
// tokens was 42 passes).  The dots stay exact integers and the scales fp32; fp16 operands on tcgen05 (kq_gemm_tc.cu) would not.
//
//   CTA       8 warps; tile 128 (or 64) weight rows x up to 64 tokens; two CTAs share an SM, so that one decodes while
//             another multiplies
//   raw       wire bytes of a 256-weight column of the rows: 16-byte cp.async pieces of the 16-byte aligned window of
//             each row, one column ahead
//   decode    every half column (128 weights): thread = (row, sub-block) -> int8 codes and fp32 scales in shared memory
//   multiply  warp = 32 rows x a share of the tokens: int8 mma.sync m16n8k32 (k16 for 16-weight scale groups).  The accumulator input
//             of the mma is the bit pattern of 12582912.0f, so the integer dot comes out as a float after one subtraction;
//             two outputs per fp32x2 instruction
//   tokens    codes, scales and min-term factors of a half column by cp.async, double buffered
//   sums      The kernels this one replaces add a row in 32 lanes and a tree; one fp32 chain over K would lose against that
//             (relative error against 64 bits, Q5_K, 1e-7: K = 512 1.07 against 0.63, 5120 3.05 against 0.81, 17408 6.1 against
//             1.07).  So a chain ends after 8 sub-blocks (4 where K < 2048, 2 where K < 512: the shorter the row the better
//             that tree) and is added to a sum and its correction in tensor memory, for which no register or shared memory
//             is left: 0.57 / 0.69 / 0.72, and not above the replaced kernels' in any format from K = 256 on.  A
//             sub-block's min term joins its dot before the chain.
//
// Measured (us, whole call, bf16 in and out, before -> now): Q5_K 6144x5120 at 333 tokens 755 -> 219
// (197 with one fp32 chain per output); the fused mixture-of-experts layer (32 experts, top 4, 2048/1408, Q4_K + Q8_0) at
// 256 tokens 1057 -> 300 (275).  What bounds it: latency of the half-column steps (load, decode, multiply behind barriers).
//
// Mixture of experts: a work item is a run of up to 8 consecutive 8-slot blocks of one expert; every CTA finds the items
// from expert_ids itself and takes every gridDim-th of them.
#include "kq_common.cuh"

namespace kq {
namespace {

constexpr int MQ_TOK = 64;          // tokens (slots) per CTA
constexpr int MQ_THREADS = 256;
constexpr int MQ_WARPS = MQ_THREADS / 32;
constexpr int MQ_KH = 128;          // weights per half column
constexpr uint32_t MQ_MAGIC = 0x4B400000u;   // 12582912.0f: exact for |dot| < 2^22 (a 32-weight dot is at most 32 * 128 * 127)

template <int QT, int ROWS> struct Mq {
  using F = Fmt<QT>;
  static constexpr int NG = 32 / F::GROUP;
  static constexpr int COLB = F::BYTES * (256 / F::BLK);           // wire bytes of 256 weights of a row
  static constexpr int PIECES = (COLB + 14 + 15) / 16;             // 16-byte pieces of their aligned window, at the worst offset
  static constexpr int SROW = PIECES * 16 + ((PIECES & 1) ? 0 : 16);   // odd multiple of 16: spreads rows over the banks
  static constexpr int STR = NG == 2 ? MQ_KH + 16 : MQ_KH + 32;    // bytes per staged code row: conflict-free 4 / 8-byte reads
  static constexpr int NS = NG == 2 ? 4 : 2;                       // floats per (sub-block, row): wa[NG], wb[NG]
  static constexpr bool MIN = F::HAS_MIN;
  static constexpr int RAW = ROWS * SROW, A = ROWS * STR, S = 4 * ROWS * NS * 4, B = MQ_TOK * STR;
  static constexpr int DS = MQ_TOK * 16, ZR = NG == 2 ? MQ_TOK * 32 : MQ_TOK * 16;   // raw ds / z pieces of a half column
  static constexpr int D = 4 * MQ_TOK * 4, Z = MIN ? 4 * NG * MQ_TOK * 4 : 0;
  static constexpr int WR = ROWS / 32, WN = MQ_WARPS / WR, NT = 8 / WN;   // warps over rows x tokens; 8-token tiles per warp
  static constexpr int TCOLS = 2 * NT * 16;                        // tensor memory: two warps per lane quarter, {sum, correction} x 8 per tile
  static constexpr int OFF_A = RAW, OFF_S = OFF_A + A, OFF_B = OFF_S + S, OFF_DS = OFF_B + 2 * B, OFF_ZR = OFF_DS + 2 * DS,
                       OFF_D = OFF_ZR + (MIN ? 2 * ZR : 0), OFF_Z = OFF_D + D, OFF_TOK = OFF_Z + Z, SMEM = OFF_TOK + 2 * MQ_TOK * 4 + 16;   // 16: address of the tensor memory
  static_assert(TCOLS >= 32 && (TCOLS & (TCOLS - 1)) == 0 && TCOLS <= 256, "two CTAs per SM share 512 columns");
  static_assert(OFF_TOK >= ROWS * 65 * 4, "the epilogue's transpose tile reuses the buffers");
};

struct MmqParams {
  const uint8_t* W;
  int64_t rowbytes, expert_stride, wbytes;   // wbytes: size of the whole weight tensor
  int n, nsb, experts, row_tiles;
  const __half2* ds;
  const int8_t* qs;
  const float* z32r;
  const float* z16r;
  int kpad, tokens, top_k;
  const int32_t* ids;                        // mixture of experts only
  const int32_t* expert_ids;
  const int32_t* num_post_padded;
  int64_t nslots;
  void* y;
  int64_t stride_y;
  int y_dtype;
};

typedef unsigned long long f2_t;
__device__ __forceinline__ f2_t f2_pack(float a, float b) { f2_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ f2_t f2_bits(int a, int b) { f2_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ float2 f2_unpack(f2_t v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ f2_t f2_add(f2_t a, f2_t b) { f2_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f2_t f2_mul(f2_t a, f2_t b) { f2_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) { f2_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }

__device__ __forceinline__ void mq_mma_k32(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(MQ_MAGIC));
}
__device__ __forceinline__ void mq_mma_k16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a0), "r"(a1), "r"(b0), "r"(MQ_MAGIC));
}
// sixteen 32-bit words per lane of this warp's quarter of tensor memory
__device__ __forceinline__ void mq_tmem_ld16(uint32_t at, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
               "tcgen05.wait::ld.sync.aligned;"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(at) : "memory");
}
__device__ __forceinline__ void mq_tmem_st16(uint32_t at, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(at), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void mq_cp16(uint32_t dst, const void* src, uint32_t have) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(have) : "memory");
}

template <typename OutT, int ROWS>
__device__ __forceinline__ void mq_store(const float* sT, const int* sDst, const MmqParams& p, int row_tile, int ntok, int tid) {
  const int r = tid % ROWS, row = row_tile * ROWS + r;
  if (row >= p.n) return;
  for (int t = tid / ROWS; t < ntok; t += MQ_THREADS / ROWS) {
    const int z = sDst[t];
    if (z >= 0) reinterpret_cast<OutT*>(p.y)[(size_t)z * p.stride_y + row] = from_f32<OutT>(sT[r * 65 + t]);
  }
}

template <int QT, bool MMQ, bool MOE, int ROWS>
__global__ void __launch_bounds__(MQ_THREADS, 2) mmq_kernel(const MmqParams p) {
  using F = Fmt<QT>;
  using M = Mq<QT, ROWS>;
  constexpr int NG = M::NG, NT = M::NT, WN = M::WN;
  extern __shared__ __align__(128) uint8_t mq_smem[];
  uint8_t* sRaw = mq_smem;
  uint8_t* sA = mq_smem + M::OFF_A;
  float* sS = reinterpret_cast<float*>(mq_smem + M::OFF_S);     // [4 sub-blocks][ROWS][NS]
  uint8_t* sB = mq_smem + M::OFF_B;                             // 2 x [64 tokens][STR]
  float* sD = reinterpret_cast<float*>(mq_smem + M::OFF_D);     // [4 sub-blocks][64 tokens]
  float* sZ = reinterpret_cast<float*>(mq_smem + M::OFF_Z);     // [4 * NG][64 tokens]
  int* sTok = reinterpret_cast<int*>(mq_smem + M::OFF_TOK);     // activation row of a slot (-1: none)
  int* sDst = sTok + MQ_TOK;                                    // output row of a slot (-1: none)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int wrow = (warp % M::WR) * 32, wn = warp / M::WR;      // this warp's 32 rows; it takes the 8-token tiles wn, wn + WN, ..
  const uint32_t smem_a = (uint32_t)__cvta_generic_to_shared(mq_smem);
  const int nhalf = (p.nsb + 3) >> 2, nb8 = p.kpad >> 5;
  const uint8_t* wend = p.W + p.wbytes;
  uint32_t* sTmem = reinterpret_cast<uint32_t*>(mq_smem + M::OFF_TOK + 2 * MQ_TOK * 4);
  uint32_t tacc = 0;                                            // this warp's part of the tensor memory
  // After pdl_wait() and before pdl_trigger(): a CTA never holds tensor memory while it waits for another kernel, and a kernel
  // behind this one cannot take it first.
  auto tmem_open = [&]() {
    if (warp == 0) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(sTmem)), "r"(M::TCOLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tacc = *sTmem + ((uint32_t)(warp & 3) << 21) + (uint32_t)((warp >> 2) * NT * 16);
    pdl_trigger();
  };
  auto tmem_close = [&]() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*sTmem), "r"(M::TCOLS));
  };

  int row_tile, expert = 0;
  // raw column `col` of the row tile: pieces are dealt to consecutive threads along a row; rows past n re-read row n - 1,
  // and of a window that reaches past the tensor only the bytes that exist are read (the rest is zero-filled)
  auto issue_raw = [&](int col) {
    const uint8_t* base = p.W + (size_t)expert * p.expert_stride + (size_t)col * M::COLB;
    for (int c = tid; c < ROWS * M::PIECES; c += MQ_THREADS) {
      const int r = c / M::PIECES, part = c - r * M::PIECES;
      int row = row_tile * ROWS + r;
      if (row >= p.n) row = p.n - 1;
      const uint8_t* src = reinterpret_cast<const uint8_t*>((uintptr_t)(base + (size_t)row * p.rowbytes) & ~(uintptr_t)15) + part * 16;
      const uint32_t have = src + 16 <= wend ? 16u : (src < wend ? (uint32_t)(wend - src) : 0u);
      mq_cp16(smem_a + r * M::SROW + part * 16, have ? src : p.W, have);
    }
  };
  // activations of half column h (4 sub-blocks) of the slots: codes, {d, raw sum}, code sums
  auto issue_b = [&](int h, int ntok) {
    const int buf = h & 1;
    for (int c = tid; c < ntok * 8; c += MQ_THREADS) {
      const int s = c >> 3, part = c & 7, tok = sTok[s];
      mq_cp16(smem_a + M::OFF_B + buf * M::B + s * M::STR + part * 16, p.qs + (size_t)(tok < 0 ? 0 : tok) * p.kpad + (size_t)h * MQ_KH + part * 16, tok < 0 ? 0u : 16u);
    }
    for (int s = tid; s < ntok; s += MQ_THREADS) {
      const int tok = sTok[s];
      const size_t at = (size_t)(tok < 0 ? 0 : tok) * nb8 + 4 * h;
      const uint32_t have = tok < 0 ? 0u : 16u;
      mq_cp16(smem_a + M::OFF_DS + buf * M::DS + s * 16, p.ds + at, have);
      if constexpr (F::HAS_MIN && !RawSum<QT, MMQ>::value) {
        if constexpr (NG == 1) {
          mq_cp16(smem_a + M::OFF_ZR + buf * M::ZR + s * 16, p.z32r + at, have);
        } else {
          mq_cp16(smem_a + M::OFF_ZR + buf * M::ZR + s * 32, p.z16r + 2 * at, have);
          mq_cp16(smem_a + M::OFF_ZR + buf * M::ZR + s * 32 + 16, p.z16r + 2 * at + 4, have);
        }
      }
    }
  };

  // one tile: sTok / sDst hold `ntok` slots (a multiple of 8)
  auto run_tile = [&](int ntok, bool raw_issued) {
    const int ntiles = ntok >> 3;
    const int every = p.nsb < 16 ? 1 : p.nsb < 64 ? 3 : 7;   // sums are closed after the sub-blocks whose index has these bits set
    bool opened = false;                       // the tensor memory holds sums of this tile
    f2_t acc[2][NT][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < NT; ++b) { acc[a][b][0] = 0ull; acc[a][b][1] = 0ull; }
    if (!raw_issued) issue_raw(0);
    issue_b(0, ntok);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int h = 0; h < nhalf; ++h) {
      const int buf = h & 1;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();        // column and activations have landed; everyone is past the previous multiplication
      {
        const int sub = tid & 3, sbg = 4 * h + sub, sbl = ((h & 1) << 2) + sub;
        const uint32_t colb = (uint32_t)(h >> 1) * (uint32_t)M::COLB + (uint32_t)((size_t)expert * p.expert_stride);
#pragma unroll
        for (int ri = 0; ri < ROWS * 4 / MQ_THREADS; ++ri) {
          const int r = (tid >> 2) + ri * (MQ_THREADS / 4);
          SubBlock s;
          if (sbg < p.nsb) {
            int row = row_tile * ROWS + r;
            if (row >= p.n) row = p.n - 1;
            const uint32_t off = (colb + (uint32_t)row * (uint32_t)p.rowbytes) & 15u;   // W itself is 16-byte aligned
            decode_subblock<QT>(sRaw + r * M::SROW + off, sbl, nullptr, s);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) s.v[i] = 0;
            s.wa[0] = s.wa[1] = s.wb[0] = s.wb[1] = 0.f;
          }
          uint4* a = reinterpret_cast<uint4*>(sA + r * M::STR + sub * 32);
          a[0] = make_uint4(s.v[0], s.v[1], s.v[2], s.v[3]);
          a[1] = make_uint4(s.v[4], s.v[5], s.v[6], s.v[7]);
          if constexpr (NG == 2) *reinterpret_cast<float4*>(sS + (sub * ROWS + r) * 4) = make_float4(s.wa[0], s.wa[1], s.wb[0], s.wb[1]);
          else *reinterpret_cast<float2*>(sS + (sub * ROWS + r) * 2) = make_float2(s.wa[0], s.wb[0]);
        }
        const __half2* dsr = reinterpret_cast<const __half2*>(mq_smem + M::OFF_DS + buf * M::DS);
        const float* zr = reinterpret_cast<const float*>(mq_smem + M::OFF_ZR + buf * M::ZR);
        for (int c = tid; c < 4 * ntok; c += MQ_THREADS) {
          const int s = c >> 2, b = c & 3;
          const float2 v = __half22float2(dsr[s * 4 + b]);
          sD[b * MQ_TOK + s] = v.x;
          if constexpr (F::HAS_MIN) {
            if constexpr (RawSum<QT, MMQ>::value) sZ[b * MQ_TOK + s] = v.y;
            else if constexpr (NG == 1) sZ[b * MQ_TOK + s] = zr[s * 4 + b];
            else { sZ[(2 * b) * MQ_TOK + s] = zr[s * 8 + 2 * b]; sZ[(2 * b + 1) * MQ_TOK + s] = zr[s * 8 + 2 * b + 1]; }
          }
        }
      }
      __syncthreads();        // decoded; the raw column is free after its second half
      if (h + 1 < nhalf) {
        issue_b(h + 1, ntok);
        if (h & 1) issue_raw((h + 1) >> 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      const uint8_t* bB = sB + buf * M::B;
      const f2_t nmagic = f2_pack(-12582912.0f, -12582912.0f);
#pragma unroll 1
      for (int sub = 0; sub < 4; ++sub) {
        uint32_t a[2][4];
        f2_t wa[2][2][NG], wb[2][2][NG];
        float was[2][2], wbs[2][2];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            const int r = wrow + mt * 16 + hf * 8 + g;
            if constexpr (NG == 1) {
              const uint2 v = *reinterpret_cast<const uint2*>(sA + r * M::STR + sub * 32 + 8 * t4);
              a[mt][hf] = v.x; a[mt][2 + hf] = v.y;
              const float2 w = *reinterpret_cast<const float2*>(sS + (sub * ROWS + r) * 2);
              wa[mt][hf][0] = f2_pack(w.x, w.x); wb[mt][hf][0] = f2_pack(-w.y, -w.y);
              was[mt][hf] = w.x; wbs[mt][hf] = w.y;
            } else {
              a[mt][hf] = *reinterpret_cast<const uint32_t*>(sA + r * M::STR + sub * 32 + 4 * t4);
              a[mt][2 + hf] = *reinterpret_cast<const uint32_t*>(sA + r * M::STR + sub * 32 + 16 + 4 * t4);
              const float4 w = *reinterpret_cast<const float4*>(sS + (sub * ROWS + r) * 4);
              wa[mt][hf][0] = f2_pack(w.x, w.x); wa[mt][hf][NG - 1] = f2_pack(w.y, w.y);
              wb[mt][hf][0] = f2_pack(-w.z, -w.z); wb[mt][hf][NG - 1] = f2_pack(-w.w, -w.w);
            }
          }
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          const int nt = i * WN + wn;
          if (nt < ntiles) {
            const f2_t d = *reinterpret_cast<const f2_t*>(sD + sub * MQ_TOK + nt * 8 + 2 * t4);
            if constexpr (NG == 1) {
              const uint2 b = *reinterpret_cast<const uint2*>(bB + (nt * 8 + g) * M::STR + sub * 32 + 8 * t4);
              f2_t z = 0ull;
              if constexpr (F::HAS_MIN) z = *reinterpret_cast<const f2_t*>(sZ + sub * MQ_TOK + nt * 8 + 2 * t4);
#pragma unroll
              for (int mt = 0; mt < 2; ++mt) {
                int D[4];
                mq_mma_k32(D, a[mt], b.x, b.y);
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                  const f2_t I = f2_add(f2_bits(D[2 * hf], D[2 * hf + 1]), nmagic);
                  if constexpr (HalfProd<QT>::value) {
                    // d * d8 and m * s8 rounded to fp16 before their use, as the reference does for Q4_1 / Q5_1
                    const float2 dv = f2_unpack(d), zv = f2_unpack(z);
                    const float2 pd = __half22float2(__floats2half2_rn(was[mt][hf] * dv.x, was[mt][hf] * dv.y));
                    const float2 pz = __half22float2(__floats2half2_rn(wbs[mt][hf] * zv.x, wbs[mt][hf] * zv.y));
                    acc[mt][i][hf] = f2_add(acc[mt][i][hf], f2_fma(I, f2_pack(pd.x, pd.y), f2_pack(-pz.x, -pz.y)));
                  } else if constexpr (F::HAS_MIN) {
                    acc[mt][i][hf] = f2_add(acc[mt][i][hf], f2_fma(wa[mt][hf][0], f2_mul(I, d), f2_mul(wb[mt][hf][0], z)));
                  } else {
                    acc[mt][i][hf] = f2_fma(wa[mt][hf][0], f2_mul(I, d), acc[mt][i][hf]);
                  }
                }
              }
            } else {
              const uint8_t* bp = bB + (nt * 8 + g) * M::STR + sub * 32 + 4 * t4;
              const uint32_t b0 = *reinterpret_cast<const uint32_t*>(bp), b1 = *reinterpret_cast<const uint32_t*>(bp + 16);
              f2_t z0 = 0ull, z1 = 0ull;
              if constexpr (F::HAS_MIN) {
                z0 = *reinterpret_cast<const f2_t*>(sZ + (2 * sub) * MQ_TOK + nt * 8 + 2 * t4);
                z1 = *reinterpret_cast<const f2_t*>(sZ + (2 * sub + 1) * MQ_TOK + nt * 8 + 2 * t4);
              }
#pragma unroll
              for (int mt = 0; mt < 2; ++mt) {
                int D0[4], D1[4];
                mq_mma_k16(D0, a[mt][0], a[mt][1], b0);
                mq_mma_k16(D1, a[mt][2], a[mt][3], b1);
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                  const f2_t I0 = f2_add(f2_bits(D0[2 * hf], D0[2 * hf + 1]), nmagic), I1 = f2_add(f2_bits(D1[2 * hf], D1[2 * hf + 1]), nmagic);
                  const f2_t dot = f2_fma(wa[mt][hf][NG - 1], I1, f2_mul(wa[mt][hf][0], I0));
                  if constexpr (F::HAS_MIN) acc[mt][i][hf] = f2_add(acc[mt][i][hf], f2_fma(d, dot, f2_fma(wb[mt][hf][NG - 1], z1, f2_mul(wb[mt][hf][0], z0))));
                  else acc[mt][i][hf] = f2_fma(d, dot, acc[mt][i][hf]);
                }
              }
            }
          }
        }
        if (((4 * h + sub) & every) == every || (sub == 3 && h + 1 == nhalf)) {
          // close these sub-blocks' sums: into {sum, correction} pairs in tensor memory, by Dekker's fast two-sum
          if (opened) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll
          for (int i = 0; i < NT; ++i) {
            if (i * WN + wn < ntiles) {
              uint32_t v[16];
              if (opened) {
                mq_tmem_ld16(tacc + i * 16, v);
              } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = 0u;
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                f2_t& c = acc[j >> 1][i][j & 1];
                const f2_t sum = f2_bits((int)v[2 * j], (int)v[2 * j + 1]), minus1 = f2_pack(-1.0f, -1.0f);
                const f2_t t = f2_add(sum, c), err = f2_fma(f2_fma(sum, minus1, t), minus1, c);   // c - (t - sum)
                const f2_t corr = f2_add(f2_bits((int)v[8 + 2 * j], (int)v[9 + 2 * j]), err);
                const float2 tv = f2_unpack(t), cv = f2_unpack(corr);
                v[2 * j] = __float_as_uint(tv.x); v[2 * j + 1] = __float_as_uint(tv.y);
                v[8 + 2 * j] = __float_as_uint(cv.x); v[9 + 2 * j] = __float_as_uint(cv.y);
                c = 0ull;
              }
              mq_tmem_st16(tacc + i * 16, v);
            }
          }
          opened = true;
        }
      }
    }
    // epilogue: transpose through shared memory (the buffers are free), lanes = consecutive rows of one token
    __syncthreads();
    float* sT = reinterpret_cast<float*>(mq_smem);     // [ROWS][65]: lanes = consecutive rows read without conflicts
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int nt = i * WN + wn;
      if (nt < ntiles) {
        uint32_t v[16];
        mq_tmem_ld16(tacc + i * 16, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) {       // j: 16-row half, 8-row half, token of the pair
          const float sum = __uint_as_float(v[j]);
          // an infinite or NaN sum stays what it is
          sT[(wrow + (j >> 2) * 16 + ((j >> 1) & 1) * 8 + g) * 65 + nt * 8 + 2 * t4 + (j & 1)] = isfinite(sum) ? sum + __uint_as_float(v[8 + j]) : sum;
        }
      }
    }
    __syncthreads();
    if (p.y_dtype == KQ_F32) mq_store<float, ROWS>(sT, sDst, p, row_tile, ntok, tid);
    else if (p.y_dtype == KQ_F16) mq_store<__half, ROWS>(sT, sDst, p, row_tile, ntok, tid);
    else mq_store<__nv_bfloat16, ROWS>(sT, sDst, p, row_tile, ntok, tid);
  };

  if constexpr (!MOE) {
    const int ntt = (p.tokens + MQ_TOK - 1) / MQ_TOK;
    row_tile = blockIdx.x / ntt;
    const int t0 = (int)(blockIdx.x % ntt) * MQ_TOK;
    const int ntok = min(MQ_TOK, (p.tokens - t0 + 7) & ~7);
    issue_raw(0);             // the weights do not depend on the previous kernel
    if (tid < MQ_TOK) {
      const int tok = t0 + tid < p.tokens ? t0 + tid : -1;
      sTok[tid] = tok; sDst[tid] = tok;
    }
    pdl_wait();
    tmem_open();
    run_tile(ntok, true);
  } else {
    row_tile = blockIdx.x % p.row_tiles;
    const int first = blockIdx.x / p.row_tiles, step = gridDim.x / p.row_tiles;
    pdl_wait();
    const int64_t total = (int64_t)p.tokens * p.top_k;
    const int64_t npost = p.num_post_padded[0];
    int nblk = (int)((p.nslots + KQ_MOE_BLOCK - 1) / KQ_MOE_BLOCK);
    if (npost < 0) return;
    tmem_open();
    if (npost / KQ_MOE_BLOCK + 1 < nblk) nblk = (int)(npost / KQ_MOE_BLOCK) + 1;   // blocks whose first slot is <= npost (moe.cuh:37)
    int run_start = 0, items = 0;            // of the block before the current one / items seen so far (the same in all warps)
    for (int base = 0; base < nblk; base += 32) {
      // every warp scans the same 32 blocks: an item starts where a run of one expert starts and every 8 blocks after that
      const int b = base + lane;
      const int e = b < nblk ? p.expert_ids[b] : -1;
      const int before = b > 0 && b < nblk ? p.expert_ids[b - 1] : -2;
      const unsigned starts = __ballot_sync(0xffffffffu, b < nblk && (b == 0 || e != before));
      const unsigned upto = starts & (0xffffffffu >> (31 - lane));
      const int start = upto ? base + 31 - __clz(upto) : run_start;
      const bool item = b < nblk && ((b - start) & 7) == 0;
      const unsigned im = __ballot_sync(0xffffffffu, item);
      if (starts) run_start = base + 31 - __clz(starts);
      const int idx = items + __popc(im & ((1u << lane) - 1u));
      const unsigned mine = __ballot_sync(0xffffffffu, item && idx % step == first && e >= 0 && e < p.experts);
      items += __popc(im);
      for (unsigned left = mine; left; left &= left - 1) {
        const int b0 = base + __ffs(left) - 1;
        expert = p.expert_ids[b0];
        int cnt = 1;
        while (cnt < 8 && b0 + cnt < nblk && p.expert_ids[b0 + cnt] == expert) ++cnt;
        __syncthreads();      // the previous item's epilogue has read sDst and the transpose tile
        if (tid < MQ_TOK) {
          const int64_t s = (int64_t)b0 * KQ_MOE_BLOCK + tid;
          const int z = tid < cnt * KQ_MOE_BLOCK && s < p.nslots ? p.ids[s] : -1;
          const bool ok = z >= 0 && z < total;
          sDst[tid] = ok ? z : -1;
          sTok[tid] = ok ? z / p.top_k : -1;
        }
        __syncthreads();
        run_tile(cnt * KQ_MOE_BLOCK, false);
      }
    }
  }
  tmem_close();
}

template <int QT, bool MMQ, bool MOE, int ROWS>
int run_mmq_rows(const MmqParams& p, unsigned grid, cudaStream_t st) {
  auto kern = mmq_kernel<QT, MMQ, MOE, ROWS>;
  constexpr int smem = Mq<QT, ROWS>::SMEM;
  static DeviceOnce attr_set;
  if (attr_set.first_time()) {
    KQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr_set.done();
  }
  KQ_CUDA_TRY(launch_pdl(kern, dim3(grid), dim3(MQ_THREADS), (size_t)smem, st, options().pdl != 0, p));
  options().launches += 1;
  KQ_CUDA_TRY(cudaGetLastError());
  return KQ_OK;
}

template <int QT, bool MMQ, bool MOE>
int run_mmq(MmqParams& p, unsigned grid, int rows, cudaStream_t st) {
  return rows == 64 ? run_mmq_rows<QT, MMQ, MOE, 64>(p, grid, st) : run_mmq_rows<QT, MMQ, MOE, 128>(p, grid, st);
}

void mmq_params(MmqParams& p, const void* W, int type, int64_t experts, int64_t n, int64_t k, const Q8Ptrs& P, int64_t tokens, void* y,
                int y_dtype, int64_t stride_y, int rows) {
  int blk = 1, bytes = 1;
  type_geometry(type, &blk, &bytes);
  p.W = (const uint8_t*)W; p.rowbytes = k / blk * bytes; p.expert_stride = p.rowbytes * n; p.wbytes = p.expert_stride * experts;
  p.n = (int)n; p.nsb = (int)(k / 32); p.experts = (int)experts; p.row_tiles = (int)((n + rows - 1) / rows);
  p.ds = P.ds; p.qs = P.qs; p.z32r = P.z32r; p.z16r = P.z16r; p.kpad = (int)P.kpad; p.tokens = (int)tokens; p.top_k = 1;
  p.ids = nullptr; p.expert_ids = nullptr; p.num_post_padded = nullptr; p.nslots = 0;
  p.y = y; p.stride_y = stride_y; p.y_dtype = y_dtype;
}

}  // namespace

// 16-byte aligned weights (the copy windows start at or after W); formats of the switch in launch_mmq
bool mmq_supported(const void* W, int type) { return ((uintptr_t)W % 16) == 0 && !type_is_core(type); }

int launch_mmq(const void* W, int type, int64_t n, int64_t k, const Q8Ptrs& P, int64_t m, void* y, int y_dtype, int64_t stride_y,
               bool mmq, cudaStream_t st) {
  MmqParams p;
  // 64-row tiles where 128-row tiles would leave SMs without a second CTA
  const int64_t tok_tiles = (m + MQ_TOK - 1) / MQ_TOK;
  const int rows = (n + 127) / 128 * tok_tiles < 3 * sm_count() / 2 ? 64 : 128;
  mmq_params(p, W, type, 1, n, k, P, m, y, y_dtype, stride_y, rows);
  const int64_t grid = (int64_t)p.row_tiles * tok_tiles;
  if (grid > 0x7fffffff) { set_error("integer GEMM: too many tiles"); return KQ_ELIMIT; }
  switch (type) {
    case KQ_TYPE_Q4_1: return run_mmq<KQ_TYPE_Q4_1, false, false>(p, (unsigned)grid, rows, st);
    case KQ_TYPE_Q5_0: return mmq ? run_mmq<KQ_TYPE_Q5_0, true, false>(p, (unsigned)grid, rows, st) : run_mmq<KQ_TYPE_Q5_0, false, false>(p, (unsigned)grid, rows, st);
    case KQ_TYPE_Q5_1: return run_mmq<KQ_TYPE_Q5_1, false, false>(p, (unsigned)grid, rows, st);
    case KQ_TYPE_Q3_K: return run_mmq<KQ_TYPE_Q3_K, false, false>(p, (unsigned)grid, rows, st);
    case KQ_TYPE_Q5_K: return mmq ? run_mmq<KQ_TYPE_Q5_K, true, false>(p, (unsigned)grid, rows, st) : run_mmq<KQ_TYPE_Q5_K, false, false>(p, (unsigned)grid, rows, st);
    case KQ_TYPE_IQ4_NL: return run_mmq<KQ_TYPE_IQ4_NL, false, false>(p, (unsigned)grid, rows, st);
    case KQ_TYPE_IQ4_XS: return run_mmq<KQ_TYPE_IQ4_XS, false, false>(p, (unsigned)grid, rows, st);
  }
  set_error("integer GEMM: GGML type %d is not covered", type);
  return KQ_EUNSUPPORTED;
}

// Expert-sorted blocks of KQ_MOE_BLOCK slots (MMQ flavour).  Every (row tile, item) is one unit of work; the grid has up to
// eight CTAs per SM's worth of them, so that short and long runs even out.
int launch_mmq_moe(const void* W, int type, int64_t experts, int64_t n, int64_t k, const Q8Ptrs& P, int64_t tokens, int top_k,
                   const int32_t* ids, int64_t nslots, const int32_t* expert_ids, const int32_t* num_post_padded, void* y, int y_dtype,
                   int64_t stride_y, cudaStream_t st) {
  if (nslots == 0) return KQ_OK;
  MmqParams p;
  const int rows = 128;
  mmq_params(p, W, type, experts, n, k, P, tokens, y, y_dtype, stride_y, rows);
  p.top_k = top_k; p.ids = ids; p.nslots = nslots; p.expert_ids = expert_ids; p.num_post_padded = num_post_padded;
  const int64_t nblocks = (nslots + KQ_MOE_BLOCK - 1) / KQ_MOE_BLOCK;
  if (nblocks > 65535) { set_error("kq_moe_a8: more than 65535 blocks of sorted tokens"); return KQ_ELIMIT; }
  int64_t groups = (8ll * sm_count() + p.row_tiles - 1) / p.row_tiles;
  if (groups > nblocks) groups = nblocks;
  const unsigned grid = (unsigned)(groups * p.row_tiles);
  switch (type) {
    case KQ_TYPE_Q4_0: return run_mmq<KQ_TYPE_Q4_0, true, true>(p, grid, rows, st);
    case KQ_TYPE_Q4_1: return run_mmq<KQ_TYPE_Q4_1, true, true>(p, grid, rows, st);
    case KQ_TYPE_Q5_0: return run_mmq<KQ_TYPE_Q5_0, true, true>(p, grid, rows, st);
    case KQ_TYPE_Q5_1: return run_mmq<KQ_TYPE_Q5_1, true, true>(p, grid, rows, st);
    case KQ_TYPE_Q8_0: return run_mmq<KQ_TYPE_Q8_0, true, true>(p, grid, rows, st);
    case KQ_TYPE_Q2_K: return run_mmq<KQ_TYPE_Q2_K, true, true>(p, grid, rows, st);
    case KQ_TYPE_Q3_K: return run_mmq<KQ_TYPE_Q3_K, true, true>(p, grid, rows, st);
    case KQ_TYPE_Q4_K: return run_mmq<KQ_TYPE_Q4_K, true, true>(p, grid, rows, st);
    case KQ_TYPE_Q5_K: return run_mmq<KQ_TYPE_Q5_K, true, true>(p, grid, rows, st);
    case KQ_TYPE_Q6_K: return run_mmq<KQ_TYPE_Q6_K, true, true>(p, grid, rows, st);
  }
  set_error("integer GEMM: GGML type %d is not covered", type);
  return KQ_EUNSUPPORTED;
}

}  // namespace kq
