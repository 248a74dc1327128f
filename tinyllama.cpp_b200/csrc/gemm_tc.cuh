// Batched matmul on the 5th-generation tensor cores for batch >= 16 decode and prompt ingestion:
//   Y[t][row] = sum_k W[row][k] * X[t][k]        (W packed Q8_0 / Q4_K / Q6_K, X fp16, fp32 accumulate)
// Replaces matmul_*_f32_batch_cpu (reference utils.cpp:730-782, 890-1044) / smart_gemm_batch_cuda
// (model.cpp:2141-2249). "Swap-AB": the weight rows are the M side of the MMA (128 per tile), the tokens
// the N side (32..256 per tile).
//
// One persistent CTA (608 threads) per SM walks K block by block, four steps of 64 elements to a block:
//   * a weight-producer warp brings the packed units of the tile's 128 rows, one 256-element block at a time as eight
//     contiguous cells (cp.async.bulk), into a ring;
//   * sixteen warps dequantise into TENSOR MEMORY, which is where the MMA takes its A operand from:
//     thread = (weight row = TMEM lane, one 64-element step of the block), 32 columns of packed fp16 pairs a
//     step, two blocks; one wait, one fence and one arrival cover 64 elements of a thread;
//   * an activation-producer lane moves the matching slices of the fp16 activations with TMA
//     (cp.async.bulk.tensor.3d, 128-byte swizzle, tokens beyond T read as zero), one to four steps a copy;
//   * the MMA warp issues sixteen tcgen05.mma (M=128, N=NT, K=16, kind::f16) per block into an
//     fp32 accumulator in tensor memory (two of them when NT <= 128). Its instruction stream is serial: as a
//     branch for one lane, with two waits and a commit a step, it took 860 cycles a step, whatever NT, and everyone
//     waited for it; so the warp runs it together, with few waits, and one lane is elected for the MMAs alone;
//   * after a unit's last step the sixteen warps read their TMEM lanes back (tcgen05.ld 32x32b: thread =
//     weight row, registers = tokens) and run the matvec kernel's epilogues.
// Measured, 7B Q4_K shapes: a step of 16 sequences 8.3 ms with one CTA per tile and the fp16 tile in shared memory, 4.7 ms now;
// a 1024-token prompt 32.7 and 23.1 ms. With few tokens the bound is issue: about 370 instructions per thread and
// block, byte permutes at half rate, 1650 cycles a block and warp beside 1240 of MMA issue, where HBM would need 800. With 256
// tokens it is the activation tiles: 128 KB a block and SM from L2, at about 36 bytes a cycle.
// The roles meet on mbarriers only. Every wait is bounded; on a give-up the kernel sets the error word,
// waits for its MMAs and copies, frees its tensor memory and returns.
//
// Why the A operand goes through tensor memory: with few tokens the kernel should run at the rate the
// packed weights arrive (128 rows x 64 elements of Q4_K in about 200 cycles). Stored to shared memory, the
// fp16 tile costs 128 cycles of it per step to write and 128 to read, on top of the packed bytes.
//
// Why the last partial wave is cut along K: 172 row tiles (a 22016-row gate/up image) on 148 SMs are two
// waves for 1.16 waves of work. Whole waves run tile by tile; the tiles left over are laid end to end
// along K and cut into `ge` equal ranges, one per CTA. A tile's ranges leave their sums in a workspace and
// the last CTA to finish adds them in order of K (deterministic). The host picks ge by what the extra
// traffic costs (tc_plan).
//
// fp16 operands: each weight is computed in FP32 as the reference does and rounded to fp16 once
// (relative 2^-11), activations likewise, so results agree with the FP32 reference dot to about 1e-3 of
// the largest output, not to 1e-3 of each element; the parity tests state that tolerance.
#pragma once
#include <cuda.h>  // CUtensorMap (types only; the encoder is fetched through cudaGetDriverEntryPoint)

#include "gemv.cuh"

namespace b200 {

constexpr int TC_M = 128;        // weight rows per CTA tile (the MMA's M)
constexpr int TC_KC = 64;        // elements along K per step: one 128-byte swizzled row of fp16 activations
constexpr int TC_WORKERS = 512;  // sixteen dequantising warps: thread = (weight row, 64-element quarter of a block)
constexpr int TC_THREADS = TC_WORKERS + 96;  // + the MMA warp, the weight-producer warp and the activation-producer warp
constexpr int TC_MAX_N = 256;    // tokens per tile: half of the tensor memory holds accumulators, half the weight stages

struct TcParams {
  GemvSeg seg[3];
  int nseg;
  int K;
  int nblk;                       // 256-element blocks along K
  const __half* x16;              // [T][K] activations (already normalised when the layer asks for it)
  int T;                          // tokens
  int NT;                         // tokens per tile: a multiple of 32, <= 256
  int epi;                        // EPI_STORE / EPI_RESID / EPI_QKV_ROPE / EPI_SWIGLU
  float* y;                       // [T][y_stride]
  __half* y16;                    // SWIGLU: the next matmul's operand, in place of y (the rounding to_half_kernel would apply)
  int y_stride;
  float* y2;                      // QKV: new K then V rows, [T][y2_stride]
  int y2_stride;
  const float* resid;             // RESID: y = resid + W x (nullptr: y itself)
  const float* rope;
  const int* positions;           // [T]
  int head_dim, max_pos;
  int tiles_n;                    // token tiles; tile = row tile * tiles_n + token tile
  int rem, ge, full;              // tiles 0 .. rem-1 are cut into ge ranges along K, the others run whole, `full` per CTA
  int bk, b_stages;               // steps of an activation stage (1, 2 or 4), stages
  int w_stages, w_stage_bytes;    // packed-weight ring: stages of eight cells
  float* ws;                      // partial sums of cut tiles, [2 * ge][NT][128]
  int* tickets;                   // one per cut tile, zero between launches
  int* error_flag;
};

// ---- tcgen05 / TMEM primitives (inline PTX) ---------------------------------------------------
__device__ __forceinline__ void tc_alloc(uint32_t* smem_dst, int ncols) {  // one full warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, int ncols) {  // the same warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// D[tmem] (+)= A[smem] * B[smem]^T, M = 128, K = 16 16-bit elements per instruction. The whole warp calls it, the leader issues it:
// control flow and addresses stay uniform over the warp (uniform registers, which the instruction wants)
__device__ __forceinline__ void tc_mma_f16(uint32_t leader, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(leader)
      : "memory");
}
// the same with A in tensor memory: lane = row, each 32-bit column two consecutive elements along K
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t leader, uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(leader)
      : "memory");
}
// arrives on the mbarrier once every MMA issued so far by the leader has completed
__device__ __forceinline__ void tc_commit_if(uint32_t leader, void* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(smem_u32(bar)), "r"(leader)
      : "memory");
}
__device__ __forceinline__ uint32_t warp_leader() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r;
}
// thread = lane, 16 consecutive columns from registers
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
               "r"(r[14]), "r"(r[15])
               : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// this warp's 32 TMEM lanes, 8 consecutive columns: thread = lane, registers = columns
__device__ __forceinline__ void tc_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// Shared-memory matrix descriptor of a K-major tile in the 128-byte-swizzle layout: rows of 128
// bytes, 8-row groups 1024 bytes apart, 16-byte chunk c of row r stored at chunk c ^ (r & 7).
// Fields: start address >> 4 [0,14), leading byte offset >> 4 [16,30) (1: unused with this
// swizzle), stride byte offset >> 4 [32,46) (1024 >> 4), descriptor version 1 [46,48), layout
// type 2 = SWIZZLE_128B [61,64). A step of 16 elements along K advances the start by 32 bytes.
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t smem_addr) {
  const uint32_t lo = ((smem_addr & 0x3FFFFu) >> 4) | (1u << 16);
  const uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);
  return ((uint64_t)hi << 32) | lo;
}
// Instruction descriptor, kind::f16: D = F32 [4,6) = 1, A and B = F16 (0) and K-major (0),
// N >> 3 at [17,23), M >> 4 at [24,29).
__host__ __device__ __forceinline__ uint32_t tc_idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TC_M >> 4) << 24); }

__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Byte k of `v` (its top two bits clear, bit 7 pre-set by the caller: v = q | 0x80 per byte) as the
// float 1 + q / 128: the byte lands in mantissa bits 16..22 under the exponent of 1.0 (its bit 7 is
// the exponent's lowest bit). One PRMT, and the affine map back to q folds into the FMA that applies
// the scale: scale * (q - off) = (128 scale) * X - (128 + off) * scale, X = 1 + q/128.
__device__ __forceinline__ uint32_t byte_to_unit_float(uint32_t v, int k) { return __byte_perm(v, 0x3F000000u, 0x7044 | (k << 8)); }

__device__ __forceinline__ uint32_t f2_half2(uint64_t v) {
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
  return pack_h2(__uint_as_float(lo), __uint_as_float(hi));
}

// Four bytes 0x80 | q (q < 64) -> four fp16 weights D * X + C in element order, computed in FP32.
__device__ __forceinline__ void tc_affine4(uint32_t bytes, uint64_t D, uint64_t C, uint32_t& w0, uint32_t& w1) {
  w0 = f2_half2(f2_fma(f2_pack(byte_to_unit_float(bytes, 0), byte_to_unit_float(bytes, 1)), D, C));
  w1 = f2_half2(f2_fma(f2_pack(byte_to_unit_float(bytes, 2), byte_to_unit_float(bytes, 3)), D, C));
}

// The packed bytes one thread needs for its 64 elements [64 c, 64 c + 64) of a block, copied from the ring so that
// the stage can be refilled while they are converted. cell, r: the row's cell and its row in it.
//   Q4_K: r[0] = d, dmin, 12 scale bytes; r[1..2] = 32 nibble pairs (low nibbles = elements 0..31, high = 32..63)
//   Q6_K: r[0..3] = ql bytes, r[4..5] = qh bytes of the 128-element half; aux = four sub-block scales; d = block scale
//   Q8_0: r[0..3] = 64 quants; aux = two fp16 scales
struct TcRaw {
  uint4 r[6];
  uint32_t aux;
  uint16_t d;
};

template <int TYPE>
__device__ __forceinline__ void tc_fetch(const uint8_t* cell, int r, int c, TcRaw& t) {
  const uint8_t* even = cell + 16 * r;                  // chunk 0 of the row; chunk n lies 256 n further,
  const uint8_t* odd = cell + 16 * (r ^ 4);             // odd chunks in the row's swapped place
  if (TYPE == T_Q4_K) {
    t.r[0] = *reinterpret_cast<const uint4*>(even);
    t.r[1] = *reinterpret_cast<const uint4*>(odd + 256 * (1 + 2 * c));
    t.r[2] = *reinterpret_cast<const uint4*>(even + 256 * (2 + 2 * c));
  } else if (TYPE == T_Q6_K) {
    const int hh = c >> 1;
#pragma unroll
    for (int i = 0; i < 4; ++i) t.r[i] = *reinterpret_cast<const uint4*>(((i & 1) ? odd : even) + 256 * (4 * hh + i));
#pragma unroll
    for (int i = 0; i < 2; ++i) t.r[4 + i] = *reinterpret_cast<const uint4*>((i ? odd : even) + 256 * (8 + 2 * hh + i));
    t.aux = *reinterpret_cast<const uint32_t*>(even + 256 * 12 + 4 * c);
    t.d = *reinterpret_cast<const uint16_t*>(cell + 16 * 208 + 2 * r);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) t.r[i] = *reinterpret_cast<const uint4*>(((i & 1) ? odd : even) + 256 * (4 * c + i));
    t.aux = *reinterpret_cast<const uint32_t*>(even + 256 * 16 + 4 * c);
  }
}

// Half hf (32 elements) of the thread's 64 as sixteen fp16 pairs. Each weight is computed in FP32 as the reference
// does and rounded to fp16 once (scaling in fp16 pairs was measured to triple the error of the products: the sub-block
// scale's rounding is shared by 16 or 32 weights and does not average out). Formulas: reference dequantize_q4_k_m /
// dequantize_q6_k / dequantize_q8_0_block (quantization.cpp:171-266, 1047-1052). FP32 pairs (fma.rn.f32x2) halve the
// multiply-adds; what is left per element is one byte permute and half a conversion.
template <int TYPE>
__device__ __forceinline__ void tc_dequant32(const TcRaw& t, int c, int hf, uint32_t (&w)[16]) {
  if (TYPE == T_Q4_K) {
    const uint4 h = t.r[0];
    const float2 dm = __half22float2(*reinterpret_cast<const __half2*>(&h.x));
    // get_scale_min_k4 (quantization.cpp:145-155) of sub-block 2c + hf on the 12 scale bytes h.y h.z h.w
    const int sh = 8 * (2 * (c & 1) + hf);
    const uint32_t a = h.y >> sh, b = h.z >> sh, e = h.w >> sh;
    const uint32_t sc = c < 2 ? (a & 63u) : ((e & 15u) | ((a >> 2) & 48u));
    const uint32_t mn = c < 2 ? (b & 63u) : (((e >> 4) & 15u) | ((b >> 2) & 48u));
    const float d1 = dm.x * (float)sc, m1 = dm.y * (float)mn;
    // d1 * q - m1 = D * X - (D + m1), D = 128 d1 (exact), X = 1 + q/128: the constant's rounding is 2^-24 of
    // 128 d1, far below the fp16 rounding of the result
    const float D = 128.0f * d1;
    const uint64_t D2 = f2_dup(D), C2 = f2_dup(-(D + m1));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t q = u4_word(t.r[1 + (i >> 2)], i & 3);
      tc_affine4(((hf ? q >> 4 : q) & 0x0F0F0F0Fu) | 0x80808080u, D2, C2, w[2 * i], w[2 * i + 1]);
    }
  } else if (TYPE == T_Q6_K) {
    // 32-element group 2 (c & 1) + hf of the 128-element half: low nibbles of ql (high ones for the upper two groups),
    // two bits of qh brought to bits 4-5 by one rotation, one bitwise select, one more clears bits 6-7 and sets bit 7
    const float d = half_bits_to_float(t.d);
    const int lsh = 4 * (c & 1), hrot = (4 - 2 * hf - 4 * (c & 1)) & 31;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const float sc = d * (float)(int)(int8_t)((t.aux >> (16 * hf + 8 * s)) & 0xFF);
      const uint64_t D2 = f2_dup(128.0f * sc), C2 = f2_dup(-160.0f * sc);  // sc * (q - 32) = 128 sc * X - (128 + 32) sc
#pragma unroll
      for (int i = 4 * s; i < 4 * s + 4; ++i) {
        const uint32_t lo = u4_word(t.r[2 * hf + (i >> 2)], i & 3) >> lsh, hw = u4_word(t.r[4 + (i >> 2)], i & 3);
        const uint32_t hi = __funnelshift_l(hw, hw, hrot);
        tc_affine4(((((lo ^ hi) & 0x0F0F0F0Fu) ^ hi) & 0x3F3F3F3Fu) | 0x80808080u, D2, C2, w[2 * i], w[2 * i + 1]);
      }
    }
  } else {
    // 0x4B0000bb is 8388608 + bb; the pairs' subtraction and product are exact, the one rounding is that to fp16
    const float d = scale_field_to_float((uint16_t)((t.aux >> (16 * hf)) & 0xFFFF));
    const uint64_t one = f2_dup(1.0f), off = f2_dup(-8388736.0f), D2 = f2_dup(d), zero = f2_dup(0.0f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t q = u4_word(t.r[2 * hf + (i >> 2)], i & 3) ^ 0x80808080u;  // int8 + 128 as an unsigned byte
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint64_t x = f2_pack(__byte_perm(q, 0x4B000000u, 0x7440 | (2 * k)), __byte_perm(q, 0x4B000000u, 0x7440 | (2 * k + 1)));
        w[2 * i + k] = f2_half2(f2_fma(f2_fma(x, one, off), D2, zero));
      }
    }
  }
}

constexpr int TC_B_STAGES = 8;   // at most: activation tiles in flight (TMA)
constexpr int TC_W_STAGES = 8;   // at most: packed-weight stages in flight (TMA)
constexpr uint32_t TC_A_COL = 256;  // first tensor-memory column of the two weight blocks, 128 columns each (the accumulators lie below)

struct alignas(64) TcMaps {
  CUtensorMap act;  // the fp16 activations
};

struct TcShared {
  unsigned long long a_full[2];              // the sixteen warps have stored a block's weights
  unsigned long long a_empty[2];             // the MMAs that read them have completed
  unsigned long long b_full[TC_B_STAGES];    // the activation tile has landed (TMA transaction bytes)
  unsigned long long b_empty[TC_B_STAGES];   // the MMAs that read it have completed
  unsigned long long acc_full[2];            // all MMAs of a unit have completed
  unsigned long long acc_empty[2];           // the sixteen warps have read the accumulator
  unsigned long long w_full[TC_W_STAGES];    // the packed units of a block have landed
  unsigned long long w_empty[TC_W_STAGES];   // the sixteen warps have copied their part of the stage into registers
  unsigned long long drained;                // all MMAs issued by this CTA have completed
  uint32_t tmem_base;
  int abort_flag;
  int last;       // this CTA is the last one of a cut tile
  int w_issued, b_issued;  // stages whose copies have been requested
};

__device__ __noinline__ bool tc_wait_slow(const TcParams& p, TcShared* sh, void* bar, uint32_t parity) {
  if (*(volatile int*)&sh->abort_flag) return false;
  if (mbar_wait(bar, parity)) return true;
  *(volatile int*)&sh->abort_flag = 1;
  if (p.error_flag) *reinterpret_cast<volatile int*>(p.error_flag) = 1;
  return false;
}
__device__ __forceinline__ bool mbar_try(void* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool tc_wait(const TcParams& p, TcShared* sh, void* bar, uint32_t parity) {
  return mbar_try(bar, parity) ? true : tc_wait_slow(p, sh, bar, parity);
}
__device__ __forceinline__ void tc_workers_sync() { asm volatile("bar.sync 14, %0;" ::"n"(TC_WORKERS) : "memory"); }

// 2-D tiled TMA load (64 elements along K x rows, 128-byte swizzle), issued by the leader of the warp
__device__ __forceinline__ void tc_tma_load_2d(uint32_t leader, void* dst, const void* tmap, int c0, int c1, void* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(leader)
      : "memory");
}
// 3-D tiled TMA load of an activation stage: steps x NT tokens x 64 elements, each step a tile in the 128-byte swizzle
__device__ __forceinline__ void tc_tma_load_3d(void* dst, const void* tmap, int c0, int c1, int c2, void* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
               "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}

// Dynamic shared memory (1024-byte aligned): the activation stages of bk x NT x 128 bytes, then the packed-weight ring.
__host__ __device__ __forceinline__ size_t tc_smem_bytes(int NT, int bk, int b_stages, int w_stages, int w_stage_bytes) {
  return 1024 + (size_t)b_stages * bk * NT * 128 + (size_t)w_stages * w_stage_bytes;
}
constexpr int TC_SMEM_MAX = 226 * 1024;  // dynamic part; the barriers live in static shared memory

// How `tiles` tiles of nblk blocks fall to `sms` CTAs: whole waves, and the tiles left over cut into ge ranges along K.
struct TcPlan {
  int rem, ge, full, grid;
};
inline TcPlan tc_plan(int tiles, int nblk, int NT, int sms, bool cut) {
  TcPlan r;
  r.full = tiles / sms;
  r.rem = tiles - r.full * sms;
  r.ge = r.rem;
  if (r.rem && cut) {
    // Cycles: a block takes four steps, each bound by the MMAs (2 NT cycles) or by dequantisation (about 250); a cut tile's
    // sums travel to the workspace and back at about 32 bytes a cycle, read by its last CTA, behind a ticket (about 1500).
    const double block = 4.0 * std::max(2 * NT, 250), part = NT * 128 * 4 / 32.0;
    double best = block * nblk;
    for (int k = 2; ; ++k) {
      const int ge = std::min({k * r.rem, sms, r.rem * nblk});
      const double t = block * ((r.rem * nblk + ge - 1) / ge) + part * ((ge + r.rem - 1) / r.rem + 1) + 1500;
      if (t < best) { best = t; r.ge = ge; }
      if (ge < k * r.rem) break;
      if (ge == sms || ge == r.rem * nblk) break;
    }
  }
  r.grid = r.full ? sms : r.ge;
  return r;
}

// Workspace of an engine: two parts of a 128 x 256 tile per CTA.
inline size_t tc_part_floats(int sms) { return (size_t)2 * sms * TC_M * TC_MAX_N; }

// One unit of work: blocks b0 .. b0 + nb - 1 of a tile; c0 .. c1: the CTAs that share the tile (c0 == c1: whole).
struct TcWork {
  int tile, b0, nb, c0, c1;
  int seg, row0, t0;
};
__device__ __forceinline__ bool tc_work(const TcParams& p, int cta, int i, TcWork& w) {
  w.c0 = w.c1 = cta;
  bool cut = false;
  if (cta < p.ge) {
    const int W = p.rem * p.nblk, x0 = cta * W / p.ge, x1 = (cta + 1) * W / p.ge;  // at most nblk blocks: one or two tiles
    const int a = x0 / p.nblk, mid = min(x1, (a + 1) * p.nblk);
    const int two = x1 > mid;
    if (i <= two) {
      w.tile = a + i;
      w.b0 = i ? 0 : x0 - a * p.nblk;
      w.nb = i ? x1 - mid : mid - x0;
      w.c0 = ((w.tile * p.nblk + 1) * p.ge - 1) / W;
      w.c1 = ((w.tile + 1) * p.nblk * p.ge - 1) / W;
      cut = true;
    }
    i -= 1 + two;
  }
  if (!cut) {
    if (i >= p.full) return false;
    w.tile = p.rem + i * (int)gridDim.x + cta;
    w.b0 = 0;
    w.nb = p.nblk;
  }
  int m = w.tile / p.tiles_n;
  w.t0 = (w.tile - m * p.tiles_n) * p.NT;
  w.seg = 0;
  while (w.seg + 1 < p.nseg && m >= (p.seg[w.seg].rows + TC_M - 1) / TC_M) { m -= (p.seg[w.seg].rows + TC_M - 1) / TC_M; ++w.seg; }
  w.row0 = m * TC_M;
  return true;
}
// Workspace slot of CTA c's part of a cut tile (a CTA has a part of at most two).
__device__ __forceinline__ int tc_slot(const TcParams& p, int c, int tile) { return 2 * c + (c * (p.rem * p.nblk) / p.ge / p.nblk != tile); }

// Eight finished columns (tokens t .. t+7) of this lane's row: the epilogue.
__device__ __forceinline__ void tc_finish8(const TcParams& p, const TcWork& w, int row, int t, const float (&v)[8]) {
  const int lane = threadIdx.x & 31;
  const bool row_ok = row < p.seg[w.seg].rows;
  const int n = min(8, p.T - t);
  if (p.epi == EPI_SWIGLU) {
    // image rows: eight gate rows then the same eight up rows (reference model.cpp:734-735, batch form
    // cpu_batch_processor.cpp:252-256: (g / (1 + exp(-g))) * u)
    const size_t at = (size_t)t * p.y_stride + (row >> 4) * 8 + (row & 7);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float up = __shfl_sync(0xffffffffu, v[j], (lane & 23) + 8);
      if (row_ok && !(row & 8) && j < n) {
        const float o = (v[j] / (1.0f + expf(-v[j]))) * up;
        if (p.y16) p.y16[at + (size_t)j * p.y_stride] = __float2half_rn(o);
        else p.y[at + (size_t)j * p.y_stride] = o;
      }
    }
  } else if (p.epi == EPI_RESID) {
    if (!row_ok) return;
    const float* rs = (p.resid ? p.resid : p.y) + (size_t)t * p.y_stride + row;
    float* y = p.y + (size_t)t * p.y_stride + row;
    float r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = j < n ? rs[(size_t)j * p.y_stride] : 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < n) y[(size_t)j * p.y_stride] = r[j] + v[j];
  } else if (p.epi == EPI_QKV_ROPE) {
    const int i = (row % p.head_dim) >> 1;
    float* y = w.seg == 0 ? p.y + (size_t)t * p.y_stride + row : p.y2 + (size_t)t * p.y2_stride + (w.seg == 2 ? p.seg[1].rows : 0) + row;
    const int ld = w.seg == 0 ? p.y_stride : p.y2_stride;
    float2 cs[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int pos = w.seg < 2 && j < n ? p.positions[t + j] : -1;
      cs[j] = pos >= 0 && pos < p.max_pos ? *reinterpret_cast<const float2*>(p.rope + ((size_t)pos * (p.head_dim >> 1) + i) * 2) : make_float2(2.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float other = __shfl_xor_sync(0xffffffffu, v[j], 1);
      float o = v[j];
      if (cs[j].x < 1.5f)  // a cosine: the row is rotated
        o = (row & 1) ? __fadd_rn(__fmul_rn(other, cs[j].y), __fmul_rn(v[j], cs[j].x)) : __fsub_rn(__fmul_rn(v[j], cs[j].x), __fmul_rn(other, cs[j].y));
      if (row_ok && j < n) y[(size_t)j * ld] = o;
    }
  } else if (row_ok) {
    float* y = p.y + (size_t)t * p.y_stride + row;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < n) y[(size_t)j * p.y_stride] = v[j];
  }
}

// One unit's blocks by a dequantising warp; blk: blocks of this CTA before it (ring position).
template <int TYPE>
__device__ __forceinline__ void tc_dequant_unit(const TcParams& p, TcShared& sh, const uint8_t* Wbase, uint32_t tmem, const TcWork& w, int blk) {
  constexpr int cell = TYPE == T_Q4_K ? 16 * 144 : TYPE == T_Q6_K ? 16 * 208 + 32 : 16 * 272;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int my_row = threadIdx.x & (TC_M - 1), c = warp >> 2;
  const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
  int stage = blk % p.w_stages;
  uint32_t wpar = (uint32_t)((blk / p.w_stages) & 1);
#pragma unroll 1
  for (int i = 0; i < w.nb; ++i, ++blk) {
    tc_wait(p, &sh, &sh.w_full[stage], wpar);
    TcRaw raw;
    tc_fetch<TYPE>(Wbase + (size_t)stage * p.w_stage_bytes + (size_t)(my_row >> 4) * cell, my_row & 15, c, raw);
    uint32_t v[16];
    tc_dequant32<TYPE>(raw, c, 0, v);
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh.w_empty[stage]);  // the stage may be refilled
    if (++stage == p.w_stages) { stage = 0; wpar ^= 1u; }
    // the MMAs that read this half of the weight columns two blocks ago must be done before it is overwritten
    const int sa = blk & 1;
    if (blk >= 2) tc_wait(p, &sh, &sh.a_empty[sa], (uint32_t)(((blk >> 1) - 1) & 1));
    tc_fence_after();
    const uint32_t dst = tmem + TC_A_COL + 32u * (uint32_t)(4 * sa + c) + lanes;
    __syncwarp();
    tc_st16(dst, v);
    tc_dequant32<TYPE>(raw, c, 1, v);
    tc_st16(dst + 16, v);
    tc_wait_st();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh.a_full[sa]);
  }
}

// grid: tc_plan. 608 threads: warps 0-15 dequantise and run the epilogue, warp 16 issues the MMAs, warp 17
// moves the packed weights, warp 18 the activation tiles. A programmatic dependent launch: only the activation producer and
// the epilogue wait for the previous kernel; weights are fetched and dequantised ahead of it.
__global__ void __launch_bounds__(TC_THREADS, 1) gemm_tc_kernel(const __grid_constant__ TcParams p, const __grid_constant__ TcMaps maps) {
  extern __shared__ uint8_t tc_smem_raw[];
  __shared__ TcShared sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* const Bbase = reinterpret_cast<uint8_t*>(((uintptr_t)tc_smem_raw + 1023) & ~(uintptr_t)1023);  // [b_stages][bk][NT rows][128 B]
  const uint32_t b_stage_bytes = (uint32_t)(p.bk * p.NT) * 128;
  uint8_t* const Wbase = Bbase + (size_t)p.b_stages * b_stage_bytes;  // [w_stages][128 rows][unit bytes]
  const int nbuf = p.NT <= (int)TC_A_COL / 2 ? 2 : 1;                 // accumulators, 128 columns apart
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&sh.a_full[i], TC_WORKERS / 32); mbar_init(&sh.a_empty[i], 1); }
    for (int i = 0; i < TC_B_STAGES; ++i) { mbar_init(&sh.b_full[i], 1); mbar_init(&sh.b_empty[i], 1); }
    for (int i = 0; i < TC_W_STAGES; ++i) { mbar_init(&sh.w_full[i], 1); mbar_init(&sh.w_empty[i], TC_WORKERS / 32); }
    for (int i = 0; i < 2; ++i) { mbar_init(&sh.acc_full[i], 1); mbar_init(&sh.acc_empty[i], TC_WORKERS / 32); }
    mbar_init(&sh.drained, 1);
    sh.abort_flag = 0;
    sh.w_issued = sh.b_issued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tc_alloc(&sh.tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();
  const uint32_t tmem = sh.tmem_base;
  TcWork w;

  if (warp == TC_WORKERS / 32) {
    // ---- MMA warp ----
    const uint32_t leader = warp_leader();
    const uint32_t idesc = tc_idesc(p.NT);
    const uint64_t bdesc0 = tc_smem_desc(smem_u32(Bbase)), b_step = (uint64_t)((p.NT * 128) >> 4);
    int sb = 0, blk = 0;
    uint32_t pb = 0;
    uint64_t bdesc = bdesc0;
    bool ok = true;
    auto wait = [&](void* bar, uint32_t parity) { return __all_sync(0xffffffffu, tc_wait(p, &sh, bar, parity)) != 0; };
    for (int u = 0; ok && tc_work(p, blockIdx.x, u, w); ++u) {
      const int buf = nbuf == 2 ? (u & 1) : 0, use = nbuf == 2 ? (u >> 1) : u;
      if (use > 0 && !(ok = wait(&sh.acc_empty[buf], (uint32_t)((use - 1) & 1)))) break;
      const uint32_t d = tmem + 128u * (uint32_t)buf;
      uint32_t accumulate = 0;
#pragma unroll 1
      for (int i = 0; i < w.nb; ++i, ++blk) {
        const int sa = blk & 1;
        if (!(ok = wait(&sh.a_full[sa], (uint32_t)((blk >> 1) & 1)))) break;
        uint32_t a = tmem + TC_A_COL + 128u * (uint32_t)sa;
#pragma unroll 1
        for (int k = 0; k < 4; k += p.bk) {
          if (!(ok = wait(&sh.b_full[sb], pb))) break;
          tc_fence_after();
#pragma unroll 1
          for (int j = 0; j < p.bk; ++j) {
            tc_mma_f16_ts(leader, d, a, bdesc, idesc, accumulate);  // 16 elements along K = 8 columns of A, 32 bytes = 2 descriptor units of B
            tc_mma_f16_ts(leader, d, a + 8, bdesc + 2, idesc, 1u);
            tc_mma_f16_ts(leader, d, a + 16, bdesc + 4, idesc, 1u);
            tc_mma_f16_ts(leader, d, a + 24, bdesc + 6, idesc, 1u);
            accumulate = 1u;
            a += 32;
            bdesc += b_step;
          }
          tc_commit_if(leader, &sh.b_empty[sb]);
          if (++sb == p.b_stages) { sb = 0; pb ^= 1u; bdesc = bdesc0; }
        }
        if (!ok) break;
        tc_commit_if(leader, &sh.a_empty[sa]);
      }
      if (ok) tc_commit_if(leader, &sh.acc_full[buf]);
    }
    // the block frees the tensor memory that MMAs in flight write: the epilogue waits for them too, but not after a give-up
    tc_commit_if(leader, &sh.drained);
    mbar_wait(&sh.drained, 0);
    __syncwarp();
  } else if (warp == TC_WORKERS / 32 + 2) {
    // ---- activation producer ----
    if (lane == 0) {
      pdl_wait();
      int sb = 0, n = 0;
      uint32_t pb = 1;  // a fresh ring's stages count as empty
      bool ok = true;
      for (int u = 0; ok && tc_work(p, blockIdx.x, u, w); ++u) {
#pragma unroll 1
        for (int k = 4 * w.b0; k < 4 * (w.b0 + w.nb); k += p.bk) {
          if (n >= p.b_stages && !(ok = tc_wait(p, &sh, &sh.b_empty[sb], pb))) break;
          mbar_expect_tx(&sh.b_full[sb], b_stage_bytes);
          tc_tma_load_3d(Bbase + (size_t)sb * b_stage_bytes, &maps.act, 0, w.t0, k, &sh.b_full[sb]);
          *(volatile int*)&sh.b_issued = ++n;
          if (++sb == p.b_stages) { sb = 0; pb ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else if (warp == TC_WORKERS / 32 + 1) {
    // ---- weight producer: eight lanes copy the block's eight cells (row groups past the image repeat its last one; the
    //      results of such rows are dropped) ----
    const int nw = p.w_stages;
    int blk = 0;
    bool ok = true;
    for (int u = 0; ok && tc_work(p, blockIdx.x, u, w); ++u) {
      const GemvSeg& sg = p.seg[w.seg];
      const uint32_t cell = (uint32_t)gemv_cell_bytes(sg.type);
      const int group = min((w.row0 >> 4) + (lane & 7), (sg.rows - 1) >> 4);
      const uint8_t* src = sg.img + ((size_t)group * p.nblk + w.b0) * cell;
#pragma unroll 1
      for (int i = 0; i < w.nb; ++i, ++blk, src += cell) {
        const int stage = blk % nw;
        void* bar = &sh.w_full[stage];
        if (lane == 0) {
          ok = blk < nw || tc_wait(p, &sh, &sh.w_empty[stage], (uint32_t)((blk / nw - 1) & 1));
          if (ok) {
            mbar_expect_tx(bar, 8 * cell);
            *(volatile int*)&sh.w_issued = blk + 1;
          }
        }
        ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        if (!ok) break;
        if (lane < 8) bulk_g2s(Wbase + (size_t)stage * p.w_stage_bytes + (size_t)lane * cell, src, cell, bar);
      }
    }
    __syncwarp();
  } else {
    // ---- dequantising warps, then the epilogue: warp w holds TMEM lanes 32*(w & 3) .. +31 (= weight rows), the four warp
    //      groups split the tokens ----
    const int r = 32 * (warp & 3) + lane;
    const int q_cols = p.NT / 4, c_begin = (warp >> 2) * q_cols;  // NT is a multiple of 32
    int blk = 0;
    for (int u = 0; tc_work(p, blockIdx.x, u, w); ++u) {
      const int type = p.seg[w.seg].type;
      if (type == T_Q4_K) tc_dequant_unit<T_Q4_K>(p, sh, Wbase, tmem, w, blk);
      else if (type == T_Q6_K) tc_dequant_unit<T_Q6_K>(p, sh, Wbase, tmem, w, blk);
      else tc_dequant_unit<T_Q8_0>(p, sh, Wbase, tmem, w, blk);
      blk += w.nb;
      const int buf = nbuf == 2 ? (u & 1) : 0, use = nbuf == 2 ? (u >> 1) : u;
      if (u == 0) pdl_wait();
      tc_wait(p, &sh, &sh.acc_full[buf], (uint32_t)(use & 1));
      __syncwarp();
      tc_fence_after();
      const uint32_t acc = tmem + 128u * (uint32_t)buf + ((uint32_t)(32 * (warp & 3)) << 16);
      const int c_end = min(c_begin + q_cols, p.T - w.t0);
      const bool whole = w.c0 == w.c1;
      float* part = p.ws + (whole ? 0 : (size_t)tc_slot(p, blockIdx.x, w.tile) * p.NT * TC_M) + r;
#pragma unroll 1
      for (int c0 = c_begin; c0 < c_end; c0 += 8) {
        float v[8];
        tc_ld8(acc + (uint32_t)c0, v);
        if (whole) {
          tc_finish8(p, w, w.row0 + r, w.t0 + c0, v);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) __stcg(part + (size_t)(c0 + j) * TC_M, v[j]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.acc_empty[buf]);
      if (!whole) {
        __threadfence();
        tc_workers_sync();
        if (tid == 0) {
          sh.last = atomicAdd(&p.tickets[w.tile], 1) == w.c1 - w.c0;
          if (sh.last) p.tickets[w.tile] = 0;
          __threadfence();
        }
        tc_workers_sync();
        const bool fin = sh.last != 0;
        if (fin) {
#pragma unroll 1
          for (int c0 = c_begin; c0 < c_end; c0 += 8) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = 0.f;
#pragma unroll 2
            for (int c = w.c0; c <= w.c1; ++c) {
              const float* src = p.ws + (size_t)tc_slot(p, c, w.tile) * p.NT * TC_M + r;
#pragma unroll
              for (int j = 0; j < 8; ++j) v[j] += __ldcg(src + (size_t)(c0 + j) * TC_M);
            }
            tc_finish8(p, w, w.row0 + r, w.t0 + c0, v);
          }
        }
        tc_workers_sync();  // sh.last is read before the next unit writes it
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  // Copies are waited for by their readers; only after a give-up may some still be in flight, and the block outlives them.
  if (*(volatile int*)&sh.abort_flag && tid == 0) {
    for (int s = max(0, sh.w_issued - p.w_stages); s < sh.w_issued; ++s) mbar_wait(&sh.w_full[s % p.w_stages], (uint32_t)((s / p.w_stages) & 1));
    for (int s = max(0, sh.b_issued - p.b_stages); s < sh.b_issued; ++s) mbar_wait(&sh.b_full[s % p.b_stages], (uint32_t)((s / p.b_stages) & 1));
  }
  __syncthreads();
  if (warp == 0) tc_dealloc(tmem, 512);
}

// x16[t][k] = fp16(x[t][k]) or, with norm weights, fp16(RMSNorm(x[t])[k]) (reference rmsnorm_batch_cpu,
// utils.cpp:613-646: f = 1/sqrtf(mean(x^2) + eps), out = x * f * w). One block of 512 threads per token;
// the row stays in registers between the two passes (rows of up to 16384 elements, else it is read again).
constexpr int TOH_THREADS = 512;
__global__ void __launch_bounds__(TOH_THREADS) to_half_kernel(const float* __restrict__ x, int x_stride, const float* __restrict__ norm_w, float eps, int K,
                                                              __half* __restrict__ out) {
  __shared__ float red[TOH_THREADS / 32 + 1];
  const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_launch_dependents();
  pdl_wait();
  const float4* xr = reinterpret_cast<const float4*>(x + (size_t)t * x_stride);
  const int n4 = K / 4;  // K is a multiple of 256
  constexpr int KEEP = 8;
  float4 v[KEEP];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    const int j = tid + i * TOH_THREADS;
    v[i] = j < n4 ? xr[j] : make_float4(0.f, 0.f, 0.f, 0.f);
    ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
  }
  for (int j = tid + KEEP * TOH_THREADS; j < n4; j += TOH_THREADS) {
    const float4 a = xr[j];
    ss += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
  }
  float f = 1.0f;
  if (norm_w) {
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    if (tid == 0) {
      float tot = 0.f;
      for (int w = 0; w < TOH_THREADS / 32; ++w) tot += red[w];
      red[TOH_THREADS / 32] = 1.0f / sqrtf(tot / (float)K + eps);
    }
    __syncthreads();
    f = red[TOH_THREADS / 32];
  }
  const float4* wr = reinterpret_cast<const float4*>(norm_w);
  uint2* orow = reinterpret_cast<uint2*>(out + (size_t)t * K);
  auto emit = [&](int j, float4 a) {
    if (norm_w) {
      const float4 w = __ldg(wr + j);
      a.x = a.x * f * w.x; a.y = a.y * f * w.y; a.z = a.z * f * w.z; a.w = a.w * f * w.w;
    }
    orow[j] = make_uint2(pack_h2(a.x, a.y), pack_h2(a.z, a.w));
  };
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    const int j = tid + i * TOH_THREADS;
    if (j < n4) emit(j, v[i]);
  }
  for (int j = tid + KEEP * TOH_THREADS; j < n4; j += TOH_THREADS) emit(j, xr[j]);
}

}  // namespace b200
