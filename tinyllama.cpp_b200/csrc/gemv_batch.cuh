// The matvec kernel (gemv.cuh) for 2 to 8 activation vectors at once: decode batches below the tensor-core matmul.
//
// Same arithmetic (24-bit activations in three digit planes, stored weight integers, exact integer sub-block sums), same
// cells, same producer. What is shared: a weight fragment is unpacked once and multiplied with every vector. One m16n8k32
// integer MMA has eight columns and a vector needs three, so two vectors share an MMA for Q4_K and Q8_0: column 2p + v
// carries plane p of vector v, and lane t receives (plane t, both vectors) in c[0] / c[1] (row g) and c[2] / c[3] (row
// g + 8). Q6_K has two scales per 32 elements and keeps one MMA per vector (column 2p + s: plane p restricted to sub-block s).
//
// What bounds it: instruction issue. One vector takes about 340 warp instructions per (16 rows, 256 elements), which is
// 85 % of the issue slots at the rate HBM delivers the cell; one launch column per vector therefore took 5 x the time for 5
// vectors (62 us a launch for 5 sequences of a 7B Q4_K model, 14 us for one). A further pair costs about 110 instructions
// here (Q6_K: 180): 28 to 45 us a launch, 6.9 -> 4.4 ms for that model's step of 5 sequences over 600 tokens. (The integer
// MMA itself is not the limit: 8.1 cycles per SM quarter.) At the 96 registers that 17 warps leave a
// thread, four pairs spill 176 bytes, three 76, two 16.
//
// Layout: the digit planes of all vectors of the CTA lie in shared memory (13.8 KB a vector at K = 4096, 37 KB at 11008) and
// B fragments are read from there for each cell, not kept in registers. To leave room for a ring, a stage holds at most eight
// cells; the two halves of the sixteen consumer warps take alternate stages. The host gives a CTA as many vectors as
// leave two stages (gvb_split); more go to further CTAs (blockIdx.y), which meet the weights in L2.
#pragma once
#include <algorithm>

#include "gemv.cuh"

namespace b200 {

constexpr int GVB_MAX = 8;     // vectors per CTA
constexpr int GVB_CELLS = 8;   // cells per stage
constexpr int GVB_PART = 4096; // floats of parked partial sums: [2 buffers][tiles][vectors][16 warps][16 rows]
constexpr int GVB_ZERO = 512;  // bytes of zeros: the operand of lanes whose column carries nothing

// Stages of a tile: R row groups x nblk blocks when a row has at most eight blocks, else one row group in nst stages of S blocks.
struct GvbGeom {
  int R, nst, S;
};
__host__ __device__ __forceinline__ GvbGeom gvb_geometry(int nblk) {
  GvbGeom g;
  g.R = nblk <= GVB_CELLS ? GVB_CELLS / nblk : 1;
  g.nst = (nblk + GVB_CELLS - 1) / GVB_CELLS;
  g.S = (nblk + g.nst - 1) / g.nst;
  return g;
}

// Shared-memory image of np pairs: [pair][6 columns = 2 plane + vector][plane stride] | zeros | per vector: scales, digits of the
// 32- and 16-element sums (as ActImage).
__host__ __device__ __forceinline__ size_t gvb_vector_bytes(int K) { return (size_t)act_sx_floats(K) * 4 + 4 * (size_t)(K / 32 + 16) + 4 * (size_t)(K / 16 + 16); }
__host__ __device__ __forceinline__ size_t gvb_ring_offset(int K, int np) {
  return ((size_t)np * 6 * act_plane_stride(K) + GVB_ZERO + 2 * np * gvb_vector_bytes(K) + 127) / 128 * 128;
}
__device__ __forceinline__ ActImage gvb_image(uint8_t* smem, int K, int np, int v) {
  const int stride = act_plane_stride(K);
  ActImage a;
  a.plane_stride = 2 * stride;
  a.planes = smem + (size_t)((v >> 1) * 6 + (v & 1)) * stride;
  uint8_t* p = smem + (size_t)np * 6 * stride + GVB_ZERO + v * gvb_vector_bytes(K);
  a.sx = reinterpret_cast<const float*>(p);
  p += act_sx_floats(K) * 4;
  a.xs32d = p;
  a.n32 = K / 32 + 16;
  p += 4 * a.n32;
  a.xs16d = p;
  a.n16 = K / 16 + 16;
  return a;
}

// A launch as the choice between this kernel and one launch column per vector (gemv_kernel) sees it: its row length, the tiles
// of one column and the largest cell.
struct GvbLaunch {
  int K, tiles, cell;
};
// How `batch` vectors are shared out: `per` to a CTA, np pairs of them, in `groups` groups; np = 0: a CTA has no room for two vectors
// and two ring slots (rows beyond about 22000 elements).
struct GvbSplit {
  int np, groups, per;
};
inline uint32_t gvb_slot_bytes(int K, int cell) {
  const GvbGeom g = gvb_geometry(K / 256);
  return (uint32_t)((g.R * g.S * cell + 127) / 128 * 128);
}
inline GvbSplit gvb_split(const GvbLaunch& l, int batch) {
  GvbSplit r{std::min(GVB_MAX, batch + 1) / 2, 0, 0};
  while (r.np > 0 && gvb_ring_offset(l.K, r.np) + 2 * (size_t)gvb_slot_bytes(l.K, l.cell) > (size_t)GEMV_SMEM_BUDGET) --r.np;
  if (r.np == 0) return r;
  r.groups = (batch + 2 * r.np - 1) / (2 * r.np);
  r.per = (batch + r.groups - 1) / r.groups;
  r.np = (r.per + 1) / 2;
  return r;
}

// Does launch i of n that follow one another (a layer's four, or the lm_head alone) run here? Where one column per vector finds an SM
// for every tile at once, the columns cost what one vector costs, while this kernel's prologue grows with the vectors of a CTA. Chains of
// one launch, us, columns / this kernel, K = 256 to 2048: 2 vectors 4.0 / 4.1, 3: 4.0 / 4.8, 4: 4.0 / 5.4, 6: 4.0 / 6.9, 8: 4.1 / 8.4
// (K = 4096: 4.5 / 11.1); with two waves of columns 7.8 / 4.6, 5.1, 5.7, 7.1, 8.4. So:
//   * columns for all launches where all of them fit at once, or in two waves when a CTA would take seven or eight vectors (a step of
//     15 sequences of a 512-wide model: 83.9 us, 96.5 when its launches of 1.2 waves run here);
//   * otherwise launch by launch, columns where they fit at once;
//   * but not for two vectors: what the columns save there (0.1 to 0.5 us) is less than what the step loses by changing
//     between two kernels (steps of 8 layers, launch by launch / here: 2048 wide, where the O projection alone fits, 320.8 / 311.8
//     us, in Q8_0 329.7 / 315.9; 1024 wide, where QKV, O and down fit, 256.5 / 245).
inline bool gvb_takes(const GvbLaunch* l, int n, int i, int batch, int sms) {
  if (batch < 2 || gvb_split(l[i], batch).np == 0) return false;
  auto waves_fit = [&](const GvbLaunch& x, int waves) { return (long long)x.tiles * batch <= (long long)waves * sms; };
  bool all = true;
  for (int j = 0; j < n; ++j) {
    const GvbSplit s = gvb_split(l[j], batch);
    all = all && (s.np == 0 || waves_fit(l[j], s.per >= 7 ? 2 : 1));
  }
  if (all) return false;
  return batch == 2 || !waves_fit(l[i], 1);
}

struct GvbShared {
  unsigned long long full_bar[GEMV_MAX_STAGES];
  unsigned long long empty_bar[GEMV_MAX_STAGES];
  unsigned long long xready_bar;
  unsigned long long best[GVB_MAX];  // argmax of a vector's rows so far: ordered value | ~index
  float red[GVB_MAX][GEMV_WARPS];
  float part[GVB_PART];
  int abort_flag;
};

__device__ __forceinline__ void gvb_fail(const GemvParams& prm, GvbShared* sh) {
  *(volatile int*)&sh->abort_flag = 1;
  if (prm.error_flag) *reinterpret_cast<volatile int*>(prm.error_flag) = 1;
}
__device__ __forceinline__ bool gvb_wait(const GemvParams& prm, GvbShared* sh, void* bar, uint32_t parity) {
  if (*(volatile int*)&sh->abort_flag) return false;
  if (mbar_wait(bar, parity)) return true;
  gvb_fail(prm, sh);
  return false;
}

// What a lane needs to find its operands of vector pair 0 (further pairs: + step) and of one block (+ 256 block).
struct GvbLane {
  LaneCtx L;
  const uint8_t* pair;  // Q4_K, Q8_0: column g of the pair
  uint32_t pair_step;   // 0 for lanes whose column carries nothing: they stay in the zeros
  const uint8_t* half;  // Q6_K: column g of vector 0 (of vector 1: + half_step)
  uint32_t half_step;
  bool pair_on, half_on;
};

// ph, pq as in compute_q4 / q6 / q8: one cell times all vectors; acc[v][0 / 1] = rows g / g + 8.
template <int NP>
__device__ __forceinline__ void gvb_q4(const uint8_t* ph, const uint8_t* pq, uint8_t* smem, int K, int blk, const GvbLane& G, float (&acc)[2 * NP][2]) {
  const LaneCtx& L = G.L;
  const uint4 h0 = *reinterpret_cast<const uint4*>(ph), h1 = *reinterpret_cast<const uint4*>(ph + 128);
  const uint32_t scA0 = h0.y & 0x3F3F3F3Fu, scB0 = (h0.w & 0x0F0F0F0Fu) | ((h0.y >> 2) & 0x30303030u);
  const uint32_t scA1 = h1.y & 0x3F3F3F3Fu, scB1 = (h1.w & 0x0F0F0F0Fu) | ((h1.y >> 2) & 0x30303030u);
  const uint8_t* bp = G.pair + (G.pair_on ? blk * 256 : 0);
  int J[NP][4];
#pragma unroll
  for (int i = 0; i < NP; ++i) J[i][0] = J[i][1] = J[i][2] = J[i][3] = 0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint2 qa = *reinterpret_cast<const uint2*>(pq + 512 * c), qb = *reinterpret_cast<const uint2*>(pq + 512 * c + 128);
    const uint32_t s0 = c < 2 ? scA0 : scB0, s1 = c < 2 ? scA1 : scB1;
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      const int sh = 4 * hi;
      const uint32_t a0 = (qa.x >> sh) & 0x0F0F0F0Fu, a1 = (qb.x >> sh) & 0x0F0F0F0Fu, a2 = (qa.y >> sh) & 0x0F0F0F0Fu, a3 = (qb.y >> sh) & 0x0F0F0F0Fu;
      const int k0 = byte_u(s0, (2 * c + hi) & 3), k1 = byte_u(s1, (2 * c + hi) & 3);
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        const uint2 b = *reinterpret_cast<const uint2*>(bp + i * G.pair_step + 64 * c + 32 * hi);
        int r[4];
        imma_16x8x32<false>(r, a0, a1, a2, a3, b.x, b.y);
        J[i][0] += k0 * r[0];
        J[i][1] += k0 * r[1];
        J[i][2] += k1 * r[2];
        J[i][3] += k1 * r[3];
      }
    }
  }
  const uint32_t mnA0 = h0.z & 0x3F3F3F3Fu, mnB0 = ((h0.w >> 4) & 0x0F0F0F0Fu) | ((h0.z >> 2) & 0x30303030u);
  const uint32_t mnA1 = h1.z & 0x3F3F3F3Fu, mnB1 = ((h1.w >> 4) & 0x0F0F0F0Fu) | ((h1.z >> 2) & 0x30303030u);
  const float2 dm0 = __half22float2(*reinterpret_cast<const __half2*>(&h0.x)), dm1 = __half22float2(*reinterpret_cast<const __half2*>(&h1.x));
#pragma unroll
  for (int v = 0; v < 2 * NP; ++v) {
    const ActImage a = gvb_image(smem, K, NP, v);
    const uint2 xw = *reinterpret_cast<const uint2*>(a.xs32d + (size_t)L.t * a.n32 + blk * 8);
    const float sx = a.sx[blk];
    const int M0 = dp4a_us(mnB0, xw.y, dp4a_us(mnA0, xw.x, 0)), M1 = dp4a_us(mnB1, xw.y, dp4a_us(mnA1, xw.x, 0));
    acc[v][0] = fmaf(sx, dm0.x * (L.wt * (float)J[v >> 1][v & 1]) - dm0.y * (L.wd * (float)M0), acc[v][0]);
    acc[v][1] = fmaf(sx, dm1.x * (L.wt * (float)J[v >> 1][2 + (v & 1)]) - dm1.y * (L.wd * (float)M1), acc[v][1]);
  }
}

template <int NP>
__device__ __forceinline__ void gvb_q6(const uint8_t* ph, const uint8_t* pq, uint8_t* smem, int K, int blk, const GvbLane& G, float (&acc)[2 * NP][2]) {
  const LaneCtx& L = G.L;
  const uint4 sc0 = *reinterpret_cast<const uint4*>(ph + 12 * 256), sc1 = *reinterpret_cast<const uint4*>(ph + 12 * 256 + 128);
  const float d0 = half_bits_to_float(*reinterpret_cast<const uint16_t*>(ph + 16 * 208 - 14 * L.g));
  const float d1 = half_bits_to_float(*reinterpret_cast<const uint16_t*>(ph + 16 * 208 + 16 - 14 * L.g));
  const uint8_t* bp = G.half + (G.half_on ? blk * 256 : 0);
  int J[2 * NP][2];
#pragma unroll
  for (int v = 0; v < 2 * NP; ++v) J[v][0] = J[v][1] = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint2 ha = *reinterpret_cast<const uint2*>(pq + 8 * 256 + 512 * h), hb = *reinterpret_cast<const uint2*>(pq + 8 * 256 + 512 * h + 128);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint2 la = *reinterpret_cast<const uint2*>(pq + 512 * (2 * h + q)), lb = *reinterpret_cast<const uint2*>(pq + 512 * (2 * h + q) + 128);
#pragma unroll
      for (int hi = 0; hi < 2; ++hi) {
        const int g4 = q + 2 * hi;
        auto six = [&](uint32_t lw, uint32_t hw) -> uint32_t {
          const uint32_t nib = hi ? ((lw >> 4) & 0x0F0F0F0Fu) : (lw & 0x0F0F0F0Fu);
          const uint32_t top = g4 == 0 ? (hw << 4) : g4 == 1 ? (hw << 2) : g4 == 2 ? hw : (hw >> 2);
          return nib | (top & 0x30303030u);
        };
        const uint32_t a0 = six(la.x, ha.x), a1 = six(lb.x, hb.x), a2 = six(la.y, ha.y), a3 = six(lb.y, hb.y);
        const uint32_t w0 = u4_word(sc0, 2 * h + hi), w1 = u4_word(sc1, 2 * h + hi);
        const int k00 = byte_s(w0, 2 * q), k01 = byte_s(w0, 2 * q + 1), k10 = byte_s(w1, 2 * q), k11 = byte_s(w1, 2 * q + 1);
#pragma unroll
        for (int v = 0; v < 2 * NP; ++v) {
          const uint2 b = *reinterpret_cast<const uint2*>(bp + (6 * (v >> 1) + (v & 1)) * G.half_step + 32 * (4 * h + g4));
          int r[4];
          imma_16x8x32<false>(r, a0, a1, a2, a3, b.x, b.y);
          J[v][0] += k00 * r[0] + k01 * r[1];
          J[v][1] += k10 * r[2] + k11 * r[3];
        }
      }
    }
  }
#pragma unroll
  for (int v = 0; v < 2 * NP; ++v) {
    const ActImage a = gvb_image(smem, K, NP, v);
    const uint4 xw = *reinterpret_cast<const uint4*>(a.xs16d + (size_t)L.t * a.n16 + blk * 16);
    const float sx = a.sx[blk];
    const int C0 = dp4a_ss(sc0.w, xw.w, dp4a_ss(sc0.z, xw.z, dp4a_ss(sc0.y, xw.y, dp4a_ss(sc0.x, xw.x, 0))));
    const int C1 = dp4a_ss(sc1.w, xw.w, dp4a_ss(sc1.z, xw.z, dp4a_ss(sc1.y, xw.y, dp4a_ss(sc1.x, xw.x, 0))));
    acc[v][0] = fmaf(sx * d0, L.wt * (float)J[v][0] - 32.f * (L.wd * (float)C0), acc[v][0]);
    acc[v][1] = fmaf(sx * d1, L.wt * (float)J[v][1] - 32.f * (L.wd * (float)C1), acc[v][1]);
  }
}

template <int NP>
__device__ __forceinline__ void gvb_q8(const uint8_t* ph, const uint8_t* pq, uint8_t* smem, int K, int blk, const GvbLane& G, float (&acc)[2 * NP][2]) {
  const LaneCtx& L = G.L;
  const uint4 da = *reinterpret_cast<const uint4*>(ph + 16 * 256), db = *reinterpret_cast<const uint4*>(ph + 16 * 256 + 128);
  const uint8_t* bp = G.pair + (G.pair_on ? blk * 256 : 0);
  float s[NP][4];
#pragma unroll
  for (int i = 0; i < NP; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint2 qa = *reinterpret_cast<const uint2*>(pq + 512 * j), qb = *reinterpret_cast<const uint2*>(pq + 512 * j + 128);
    const float d0 = scale_field_to_float((uint16_t)((u4_word(da, j >> 1) >> (16 * (j & 1))) & 0xFFFF));
    const float d1 = scale_field_to_float((uint16_t)((u4_word(db, j >> 1) >> (16 * (j & 1))) & 0xFFFF));
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const uint2 b = *reinterpret_cast<const uint2*>(bp + i * G.pair_step + 32 * j);
      int r[4];
      imma_16x8x32<true>(r, qa.x, qb.x, qa.y, qb.y, b.x, b.y);
      s[i][0] = fmaf(d0, (float)r[0], s[i][0]);
      s[i][1] = fmaf(d0, (float)r[1], s[i][1]);
      s[i][2] = fmaf(d1, (float)r[2], s[i][2]);
      s[i][3] = fmaf(d1, (float)r[3], s[i][3]);
    }
  }
#pragma unroll
  for (int v = 0; v < 2 * NP; ++v) {
    const float sx = gvb_image(smem, K, NP, v).sx[blk] * L.wt;
    acc[v][0] = fmaf(sx, s[v >> 1][v & 1], acc[v][0]);
    acc[v][1] = fmaf(sx, s[v >> 1][2 + (v & 1)], acc[v][1]);
  }
}

// Prologue: RMSNorm and quantisation of the CTA's nv vectors (act_build for one). All vectors' sums of squares meet at one
// barrier; the second pass reads the vectors again, from L1 or L2.
template <int NP>
__device__ __forceinline__ void gvb_build(const GemvParams& prm, GvbShared* sh, uint8_t* smem, int first, int nv) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = prm.K, nblk = K / 256;
  auto load = [&](int v, int b, float (&x)[8]) {
    const float4* s = reinterpret_cast<const float4*>(prm.x + (size_t)(first + v) * prm.x_stride + b * 256 + lane * 8);
    const float4 p = s[0], q = s[1];
    x[0] = p.x; x[1] = p.y; x[2] = p.z; x[3] = p.w; x[4] = q.x; x[5] = q.y; x[6] = q.z; x[7] = q.w;
  };
  if (prm.norm_w) {
    float ss[2 * NP];
#pragma unroll
    for (int v = 0; v < 2 * NP; ++v) ss[v] = 0.f;
#pragma unroll 1
    for (int b = warp; b < nblk; b += GEMV_WARPS) {
#pragma unroll
      for (int v = 0; v < 2 * NP; ++v) {
        float x[8];
        load(min(v, nv - 1), b, x);
#pragma unroll
        for (int i = 0; i < 8; ++i) ss[v] = fmaf(x[i], x[i], ss[v]);
      }
    }
#pragma unroll
    for (int v = 0; v < 2 * NP; ++v) ss[v] = warp_sum(ss[v]);
    if (lane == 0) {
#pragma unroll
      for (int v = 0; v < 2 * NP; ++v) sh->red[v][warp] = ss[v];
    }
    consumer_sync();
  }
  if (lane == 0) mbar_arrive(&sh->xready_bar);
  // the warp's (vector, block) items, the next one's elements requested before this one is worked on
  float xn[8];
  if (warp < nblk) load(0, warp, xn);
  int v = 0, b = warp;
  float f = 0.f;
#pragma unroll 1
  while (v < nv && warp < nblk) {
    float x[8], amax;
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = xn[i];
    int v2 = v, b2 = b + GEMV_WARPS;
    if (b2 >= nblk) { b2 = warp; ++v2; }
    if (v2 < nv) load(v2, b2, xn);
    float4 w[2];
    w[0] = w[1] = make_float4(1.f, 1.f, 1.f, 1.f);
    if (prm.norm_w) {
      w[0] = __ldg(reinterpret_cast<const float4*>(prm.norm_w + b * 256 + lane * 8));
      w[1] = __ldg(reinterpret_cast<const float4*>(prm.norm_w + b * 256 + lane * 8 + 4));
      if (b == warp) {  // a new vector: fixed-order pairwise sum of the 16 warp partials, as act_build
        float r = sh->red[v][lane & 15];
#pragma unroll
        for (int o = 1; o < GEMV_WARPS; o <<= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        f = rsqrtf(r * (1.0f / (float)K) + prm.eps);
      }
    }
    act_scale_block<3>(x, prm.norm_w, w, f, amax);
    act_quantize_block<3>(gvb_image(smem, K, NP, v), b, lane, x, warp_max(amax));
    v = v2;
    b = b2;
  }
  if (tid < GVB_ZERO / 4) reinterpret_cast<uint32_t*>(smem + (size_t)NP * 6 * act_plane_stride(K))[tid] = 0u;
  if (tid < GVB_MAX) sh->best[tid] = 0ull;
  consumer_sync();
}

// Finishes the rows of the n tiles parked in `part` (numbers first_i .. of this CTA's sequence) for the CTA's nv vectors. There
// are two such buffers and one barrier, on entry: who has no rows to finish goes on, and by the next flush's barrier all
// have read this buffer. The rows go to other warps each time.
template <int NP>
__device__ __forceinline__ void gvb_flush(const GemvParams& prm, GvbShared* sh, const GvbGeom& g, const float* part, int first_i, int n, int first, int nv) {
  consumer_sync();
  const int lane = threadIdx.x & 31, turn = ((threadIdx.x >> 5) + 3 * first_i) & (GEMV_WARPS - 1);
  const int cells = g.nst == 1 ? prm.nblk : g.S;  // warps of a half that hold a row group's sums
  const int total = n * g.R * nv * 16;
#pragma unroll 1
  for (int base = 32 * turn; base < total; base += GEMV_WARPS * 32) {
    const int idx = base + lane, r = idx & 15;
    const bool in = idx < total;
    const int rest = in ? idx >> 4 : 0, v = rest % nv, sg = rest / nv;
    const int slot = sg / g.R, rgi = sg - slot * g.R;
    float tot = 0.f;
    {
      const float* pp = part + ((slot * (2 * NP) + v) * GEMV_WARPS) * 16 + r;
      const int lo = g.nst == 1 ? 8 * ((first_i + slot) & 1) + rgi * prm.nblk : 0;
#pragma unroll 4
      for (int w = 0; w < cells; ++w) tot += pp[(lo + w) * 16];
      if (g.nst > 1) {
#pragma unroll 4
        for (int w = 0; w < cells; ++w) tot += pp[(8 + w) * 16];
      }
    }
    int seg, tl;
    gemv_locate(prm, blockIdx.x + (first_i + slot) * gridDim.x, seg, tl);
    const int row = (tl * g.R + rgi) * 16 + r;  // image row within the segment
    const bool valid = in && row < prm.seg[seg].rows;
    const int b = first + v;
    if (prm.epi == EPI_SWIGLU) {
      const float u = __shfl_sync(0xffffffffu, tot, (lane & 23) + 8);
      if (valid && r < 8) {
        const float sig = 1.0f / (1.0f + expf(-tot));
        prm.y[(size_t)b * prm.y_stride + (row >> 4) * 8 + r] = (tot * sig) * u;
      }
    } else if (prm.epi == EPI_RESID) {
      if (valid) prm.y[(size_t)b * prm.y_stride + row] = (prm.resid ? prm.resid : prm.y)[(size_t)b * prm.y_stride + row] + tot;
    } else if (prm.epi == EPI_QKV_ROPE) {
      const float other = __shfl_xor_sync(0xffffffffu, tot, 1);
      if (valid) {
        float o = tot;
        if (seg < 2) {  // q and k are rotated in adjacent pairs (reference utils.cpp:428-489)
          const int pos = prm.positions[b];
          if (pos >= 0 && pos < prm.max_pos) {
            const int i = (row % prm.head_dim) >> 1;
            const float2 cs = *reinterpret_cast<const float2*>(prm.rope + ((size_t)pos * (prm.head_dim >> 1) + i) * 2);
            o = (row & 1) ? __fadd_rn(__fmul_rn(other, cs.y), __fmul_rn(tot, cs.x)) : __fsub_rn(__fmul_rn(tot, cs.x), __fmul_rn(other, cs.y));
          }
        }
        float* dst = seg == 0 ? prm.y + (size_t)b * prm.y_stride + row : prm.y2 + (size_t)b * prm.y2_stride + (seg == 2 ? prm.seg[1].rows : 0) + row;
        *dst = o;
      }
    } else {
      const int grow = row + prm.amax_row_offset;
      if (valid) {
        if (prm.pen_counts) {
          const int times = prm.pen_counts[(size_t)b * prm.pen_stride + grow];
          if (times) {
            const float pen = *prm.pen_value;
#pragma unroll 1
            for (int k = 0; k < times; ++k) tot = tot > 0.0f ? __fdiv_rn(tot, pen) : __fmul_rn(tot, pen);
          }
        }
        prm.y[(size_t)b * prm.y_stride + row] = tot;
      }
      if (prm.amax_val) {  // the sixteen lanes of a row group hold one vector: its largest value, the first of equal ones; NaN never
        const uint32_t bits = __float_as_uint(tot + 0.0f);
        unsigned long long key = !valid || tot != tot ? 0ull : ((unsigned long long)(bits & 0x80000000u ? ~bits : bits | 0x80000000u) << 32) | (uint32_t)~grow;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
          const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
          key = other > key ? other : key;
        }
        if (r == 0 && key) atomicMax(&sh->best[v], key);
      }
    }
  }
}

template <int NP, int TYPE>
__device__ __forceinline__ void gvb_tiles(const GemvParams& prm, GvbShared* sh, uint8_t* smem, const uint8_t* ring, int nslots, const GvbGeom& g, const GvbLane& G,
                                          int seg_end, int& tile, int& i, int& n, int first, int nv) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = warp >> 3, ci = warp & 7;
  constexpr uint32_t cell = TYPE == T_Q6_K ? 16 * 208 + 32 : TYPE == T_Q4_K ? 16 * 144 : 16 * 272;
  constexpr int NTB = GVB_PART / 2 / (2 * NP * GEMV_WARPS * 16);  // tiles of a buffer
  const uint32_t off_h = (uint32_t)ci * cell + 16u * (uint32_t)G.L.g;
  const uint32_t off_q = (uint32_t)ci * cell + gemv_chunk(G.L.g, (TYPE == T_Q4_K ? 1 : 0) + (G.L.t >> 1)) + 8u * (uint32_t)(G.L.t & 1);
#pragma unroll 1
  for (; tile < seg_end; tile += gridDim.x, ++i) {
    float acc[2 * NP][2];
#pragma unroll
    for (int v = 0; v < 2 * NP; ++v) acc[v][0] = acc[v][1] = 0.f;
    bool mine = false;
#pragma unroll 1
    for (int s = 0; s < g.nst; ++s, ++n) {
      if ((n & 1) != half) continue;
      mine = true;
      const int slot = n % nslots;
      gvb_wait(prm, sh, &sh->full_bar[slot], (uint32_t)((n / nslots) & 1));
      __syncwarp();
      const int blk = g.nst == 1 ? ci % prm.nblk : s * g.S + ci;
      if (g.nst == 1 ? ci < g.R * prm.nblk : (ci < g.S && blk < prm.nblk)) {
        const uint8_t* st = ring + (size_t)slot * prm.slot_bytes;
        if (TYPE == T_Q4_K) gvb_q4<NP>(st + off_h, st + off_q, smem, prm.K, blk, G, acc);
        else if (TYPE == T_Q6_K) gvb_q6<NP>(st + off_h, st + off_q, smem, prm.K, blk, G, acc);
        else gvb_q8<NP>(st + off_h, st + off_q, smem, prm.K, blk, G, acc);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->empty_bar[slot]);
    }
    const int pp = i % NTB;
    float* part = sh->part + (i / NTB & 1) * (GVB_PART / 2);
    if (mine) {
      // sum over the four lanes of a row: lanes 2t and 2t+1 first share out rows g / g + 8, then the pairs the vectors
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        float k[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float keep = (G.L.t & 1) ? acc[2 * p + u][1] : acc[2 * p + u][0], give = (G.L.t & 1) ? acc[2 * p + u][0] : acc[2 * p + u][1];
          k[u] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
        }
        const float keep = (G.L.t & 2) ? k[1] : k[0], give = (G.L.t & 2) ? k[0] : k[1];
        part[((pp * (2 * NP) + 2 * p + (G.L.t >> 1)) * GEMV_WARPS + warp) * 16 + G.L.g + 8 * (G.L.t & 1)] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
      }
    }
    if (pp == NTB - 1 || tile + (int)gridDim.x >= prm.ntiles) gvb_flush<NP>(prm, sh, g, part, i - pp, pp + 1, first, nv);
  }
}

// grid = (CTAs over the tiles, groups of `per` vectors). prm.seg[].tiles and prm.ntiles count tiles of gvb_geometry.
template <int NP>
__global__ void __launch_bounds__(GEMV_THREADS, 1) gemv_batch_kernel(const __grid_constant__ GemvParams prm, int nslots, int per, int batch) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ GvbShared sh;
  uint8_t* ring = smem + gvb_ring_offset(prm.K, NP);
  const GvbGeom g = gvb_geometry(prm.nblk);
  const int first = blockIdx.y * per, nv = min(per, batch - first);
  if (threadIdx.x == 0) {
    for (int s = 0; s < nslots; ++s) {
      mbar_init(&sh.full_bar[s], 1);
      mbar_init(&sh.empty_bar[s], GEMV_WARPS / 2);
    }
    mbar_init(&sh.xready_bar, GEMV_WARPS);
    sh.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_launch_dependents();
  if (threadIdx.x >= GEMV_CONSUMER_THREADS) {
    if (threadIdx.x == GEMV_CONSUMER_THREADS) {
      int n = 0, last_n = -1;
      bool ok = true;
#pragma unroll 1
      for (int tile = blockIdx.x; ok && tile < prm.ntiles; tile += gridDim.x) {
        int s, tl;
        gemv_locate(prm, tile, s, tl);
        const GemvSeg& sg = prm.seg[s];
        const uint32_t cell = (uint32_t)gemv_cell_bytes(sg.type);
        const int groups = min(g.R, (sg.rows + 15) / 16 - tl * g.R);
        const uint8_t* src = sg.img + (size_t)tl * g.R * prm.nblk * cell;
#pragma unroll 1
        for (int k = 0; k < g.nst; ++k, ++n) {
          const int slot = n % nslots;
          if (n == prm.early_stages) ok = gvb_wait(prm, &sh, &sh.xready_bar, 0);
          if (ok && n >= nslots) ok = gvb_wait(prm, &sh, &sh.empty_bar[slot], (uint32_t)((n / nslots - 1) & 1));
          if (!ok) break;
          const uint32_t bytes = cell * (uint32_t)(g.nst == 1 ? groups * prm.nblk : min(g.S, prm.nblk - k * g.S));
          mbar_expect_tx(&sh.full_bar[slot], bytes);
          bulk_g2s(ring + (size_t)slot * prm.slot_bytes, src + (size_t)(k * g.S) * cell, bytes, &sh.full_bar[slot]);
          last_n = n;
        }
      }
      if (!ok)  // only after a give-up: the block outlives its copies in flight
        for (int k = max(0, last_n - nslots + 1); k <= last_n; ++k) mbar_wait(&sh.full_bar[k % nslots], (uint32_t)((k / nslots) & 1));
    }
    return;
  }
  const int lane = threadIdx.x & 31;
  unsigned long long* rec = (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) ? prm.trace : nullptr;
  trace_stamp(rec, 0);
  pdl_wait();
  for (int i = 1; i < 5; ++i) trace_stamp(rec, i);
  gvb_build<NP>(prm, &sh, smem, first, nv);
  trace_stamp(rec, 5);
  GvbLane G;
  G.L.g = lane >> 2;
  G.L.t = lane & 3;
  G.L.wd = __int_as_float((127 + 8 * G.L.t) << 23);  // 256^t
  G.L.wt = G.L.t < 3 ? G.L.wd : 0.f;
  const int stride = act_plane_stride(prm.K);
  const uint8_t* zeros = smem + (size_t)NP * 6 * stride;
  G.pair_on = G.L.g < 6;
  G.pair = G.pair_on ? smem + (size_t)G.L.g * stride + 8 * G.L.t : zeros;
  G.pair_step = G.pair_on ? 6u * (uint32_t)stride : 0u;
  G.half_on = G.L.g < 6 && (G.L.t >> 1) == (G.L.g & 1);
  G.half = G.half_on ? smem + (size_t)(G.L.g & ~1) * stride + 8 * G.L.t : zeros;
  G.half_step = G.half_on ? (uint32_t)stride : 0u;
  int tile = blockIdx.x, i = 0, n = 0, seg_end = 0;
#pragma unroll 1
  for (int s = 0; s < prm.nseg; ++s) {
    seg_end += prm.seg[s].tiles;
    if (tile >= seg_end) continue;
    const int type = prm.seg[s].type;
    if (type == T_Q4_K) gvb_tiles<NP, T_Q4_K>(prm, &sh, smem, ring, nslots, g, G, seg_end, tile, i, n, first, nv);
    else if (type == T_Q6_K) gvb_tiles<NP, T_Q6_K>(prm, &sh, smem, ring, nslots, g, G, seg_end, tile, i, n, first, nv);
    else gvb_tiles<NP, T_Q8_0>(prm, &sh, smem, ring, nslots, g, G, seg_end, tile, i, n, first, nv);
  }
  trace_stamp(rec, 6);
  if (prm.amax_val) consumer_sync();  // all rows are in `best`
  if (prm.amax_val && threadIdx.x < nv) {
    const unsigned long long key = sh.best[threadIdx.x];
    const uint32_t u = (uint32_t)(key >> 32);
    prm.amax_val[(size_t)(first + threadIdx.x) * gridDim.x + blockIdx.x] = key ? __uint_as_float(u & 0x80000000u ? u & 0x7fffffffu : ~u) : -INFINITY;
    prm.amax_idx[(size_t)(first + threadIdx.x) * gridDim.x + blockIdx.x] = key ? (int)~(uint32_t)key : 0x7fffffff;
  }
  trace_stamp(rec, 7);
}

}  // namespace b200
