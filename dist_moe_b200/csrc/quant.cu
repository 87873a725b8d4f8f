// Block-scaled quantisers: MXFP8 E4M3 (E8M0 scale per 32 elements) and NVFP4 (E2M1 data,
// E4M3 scale per 16 elements, fp32 per-token or per-expert scale).  All HBM bound:
// 16-byte loads, byte-exact hardware conversions (cvt.rp.ue8m0, cvt.rn.satfinite.e4m3x2,
// cvt.rn.satfinite.e2m1x2 through the cuda_fp8/cuda_fp4 intrinsics), no fast-math.
//
// Numerics follow the reference's quantisers step by step
// (dist_moe/kernels/blockscaled_quantization_common.py:120-257, 739-752;
//  dist_moe/kernels/triton_quantization/blockscaled_quantize.py:296-493):
//   MXFP8: s = amax * fl(1/448); byte = round-up-to-power-of-two(s); recip = 2^(127-byte);
//          q = e4m3_rn_satfinite(x * recip); a non-finite block gets byte 0xFF and NaN data.
//   NVFP4: raw = (amax * scale) * fl(1/6) clamped to [2^-9, 448]; byte = e4m3_rn(raw);
//          mult = div_rn(scale, f32(byte)); codes = e2m1_rn_satfinite(x * mult), even element
//          in the low nibble.
#include <cuda_fp4.h>

#include "publish.cuh"
#include "quant_common.cuh"
#include "../../include/dist_moe_b200.h"

namespace dm {

// Scale byte and reciprocal of a block of bf16 values from the low 15 bits of its largest magnitude: the byte that
// mxfp8_scale computes through fp32, in integers.  amax / 448 <= 2^(b - 127) holds for bf16 exactly when the
// (exponent, mantissa) pair is <= (b + 8, 0x60), 448 being 1.75 * 2^8; bytes below 0 are 0, a non-finite block is 0xFF.
__device__ __forceinline__ uint32_t mxfp8_scale_bits(uint32_t bits15, float& recip) {
  const int b = static_cast<int>((bits15 + 0x1fu) >> 7) - 8;
  const uint32_t byte = bits15 >= 0x7f80u ? 0xffu : static_cast<uint32_t>(b > 0 ? b : 0);
  recip = byte == 0xffu ? __int_as_float(0x7fc00000) : __uint_as_float((254u - byte) << 23);
  return byte;
}

// The same of two maxima side by side, both finite: the scale bytes in 16 bits each, and the reciprocals (powers of two) as the two
// bf16 of `recip2`.
__device__ __forceinline__ uint32_t mxfp8_scale_bits2(uint32_t bits15x2, uint32_t& recip2) {
  const uint32_t b = __vmaxu2(((bits15x2 + 0x001f001fu) >> 7) & 0x01ff01ffu, 0x00080008u) - 0x00080008u;
  recip2 = (0x00fe00feu - b) << 7;
  return b;
}
__device__ __forceinline__ bool any_nonfinite2(uint32_t bits15x2) { return __vmaxu2(bits15x2, 0x7f7f7f7fu) != 0x7f7f7f7fu; }

// Products of two packed fp32 pairs (one instruction), as two E4M3 bytes.
__device__ __forceinline__ uint32_t e4m3x2_scaled(float lo, float hi, float r_lo, float r_hi) {
  float a, b;
  asm("{\n\t"
      ".reg .b64 x, y, z;\n\t"
      "mov.b64 x, {%2, %3};\n\t"
      "mov.b64 y, {%4, %5};\n\t"
      "mul.rn.f32x2 z, x, y;\n\t"
      "mov.b64 {%0, %1}, z;\n\t"
      "}\n"
      : "=f"(a), "=f"(b)
      : "f"(lo), "f"(hi), "f"(r_lo), "f"(r_hi));
  return __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
}

// ---------------------------------------------------------------------------
// MXFP8 row mode: 1x32 blocks along the contiguous dimension.  HBM bound.  A warp takes 1024 elements of one row (four
// 16-byte loads in flight per lane), four neighbouring lanes hold one block.  `live` (optional, one word per row) names
// the padding rows by a zero: they are neither read nor written, which at decode sizes is nearly all of them (64 routes
// on 42 experts padded to 5376 rows of 2816: 15.6 -> 5.4 us).  4096 x 2816: 11.7 -> 8.4 us.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) mxfp8_row_kernel(const uint4* __restrict__ x, const int32_t* num_rows,
                                                        int64_t max_rows, int vec_per_row, uint8_t* __restrict__ q,
                                                        int64_t q_stride, uint8_t* __restrict__ scales,
                                                        int64_t s_stride, int blocked, int n_col_atoms,
                                                        const int64_t* __restrict__ live, IdPublish ids) {
  publish_ids(ids);
  int64_t rows = num_rows ? *num_rows : max_rows;
  if (rows > max_rows) rows = max_rows;
  const int lane = threadIdx.x & 31;
  const int segs = (vec_per_row + 127) >> 7;
  const int64_t items = rows * segs;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); i < items; i += warps) {
    const int64_t r = segs == 1 ? i : i / segs;
    if (live != nullptr && live[r] == 0) continue;
    const int v0 = static_cast<int>(i - r * segs) * 128 + lane;
    const uint4* xr = x + r * vec_per_row;
    uint4 w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = v0 + 32 * j < vec_per_row ? xr[v0 + 32 * j] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int v = v0 + 32 * j;
      uint32_t m = __vmaxu2(__vmaxu2(w[j].x & 0x7fff7fffu, w[j].y & 0x7fff7fffu),
                            __vmaxu2(w[j].z & 0x7fff7fffu, w[j].w & 0x7fff7fffu));
      m = __vmaxu2(m, __shfl_xor_sync(0xffffffffu, m, 1));
      m = __vmaxu2(m, __shfl_xor_sync(0xffffffffu, m, 2));
      float recip;
      const uint32_t byte = mxfp8_scale_bits((m >> 16) > (m & 0xffffu) ? m >> 16 : m & 0xffffu, recip);
      if (v >= vec_per_row) continue;
      float f[8];
      unpack8f(w[j], f);
      *reinterpret_cast<uint2*>(q + r * q_stride + static_cast<int64_t>(v) * 8) =
          make_uint2(e4m3x2_scaled(f[0], f[1], recip, recip) | (e4m3x2_scaled(f[2], f[3], recip, recip) << 16),
                     e4m3x2_scaled(f[4], f[5], recip, recip) | (e4m3x2_scaled(f[6], f[7], recip, recip) << 16));
      if ((v & 3) == 0) {
        const int blk = v >> 2;
        if (blocked)
          scales[blocked_offset(r, blk, n_col_atoms)] = static_cast<uint8_t>(byte);
        else
          scales[r * s_stride + blk] = static_cast<uint8_t>(byte);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// MXFP8 column mode (32x1 blocks along the rows) and 32x32 tile mode.
// One CTA handles a 32-row x 256-column slab staged in shared memory.
//   col mode : scale[c][r/32]           (natural: [C][ceil(R/32)], or blocked with rows = C)
//   tile mode: one scale per 32x32 tile, written for both GEMM orientations:
//              row_scales[n][k/32] (forward) and col_scales[k][n/32] (input gradient).
// ---------------------------------------------------------------------------
template <bool kTile>
__global__ void __launch_bounds__(256) mxfp8_slab_kernel(const __nv_bfloat16* __restrict__ x, const int32_t* num_rows,
                                                         int64_t max_rows, int C, uint8_t* __restrict__ q,
                                                         uint8_t* __restrict__ s0, uint8_t* __restrict__ s1,
                                                         int blocked, int s0_col_atoms, int s1_col_atoms,
                                                         int64_t batch_rows) {
  __shared__ float tile[32][257];
  __shared__ float col_amax[256];
  int64_t rows = num_rows ? *num_rows : max_rows;
  if (rows > max_rows) rows = max_rows;
  const int64_t row0 = static_cast<int64_t>(blockIdx.y) * 32;
  const int col0 = blockIdx.x * 256;
  if (row0 >= rows) return;
  const int t = threadIdx.x;
  for (int i = t; i < 32 * 256; i += 256) {
    const int r = i >> 8, c = i & 255;
    float v = 0.f;
    if (row0 + r < rows && col0 + c < C) v = __bfloat162float(x[(row0 + r) * C + col0 + c]);
    tile[r][c] = v;
  }
  __syncthreads();
  {
    float a = 0.f;
#pragma unroll 8
    for (int r = 0; r < 32; ++r) a = amax_nonfinite(a, tile[r][t]);
    col_amax[t] = a;
  }
  __syncthreads();
  float amax = col_amax[t];
  if (kTile) {
    const int g = t & ~31;
    amax = 0.f;
    for (int j = 0; j < 32; ++j) {
      const float v = col_amax[g + j];
      amax = (v != v || amax != amax) ? __int_as_float(0x7f800000) : fmaxf(amax, v);
    }
  }
  float recip;
  const uint8_t byte = mxfp8_scale(amax, recip);
  const int c = col0 + t;
  if (c < C) {
    if (kTile) {
      // batch_rows = rows of one expert: scale tensors are per-expert blocked groups.
      const int64_t e = row0 / batch_rows, rl = row0 - e * batch_rows;
      if ((t & 31) == 0) {
        // forward orientation: 32 rows share the byte for k-block c/32
        for (int r = 0; r < 32 && row0 + r < rows; ++r) {
          const int64_t rr = row0 + r;
          if (blocked) {
            const int64_t grp = (batch_rows + 127) / 128 * 128 * static_cast<int64_t>(s0_col_atoms) * 4;
            s0[e * grp + blocked_offset(rl + r, c >> 5, s0_col_atoms)] = byte;
          } else {
            s0[rr * ((C + 31) / 32) + (c >> 5)] = byte;
          }
        }
      }
      if (s1 != nullptr) {
        // input-gradient orientation: row index = k (this column), column = n-block
        const int64_t nb = rl >> 5;
        if (blocked) {
          const int64_t grp = (static_cast<int64_t>(C) + 127) / 128 * 128 * static_cast<int64_t>(s1_col_atoms) * 4;
          s1[e * grp + blocked_offset(c, static_cast<int>(nb), s1_col_atoms)] = byte;
        } else {
          s1[(e * C + c) * ((batch_rows + 31) / 32) + nb] = byte;
        }
      }
    } else {
      const int64_t rb = row0 >> 5;
      if (blocked)
        s0[blocked_offset(c, static_cast<int>(rb), s0_col_atoms)] = byte;
      else
        s0[static_cast<int64_t>(c) * ((max_rows + 31) / 32) + rb] = byte;
    }
  }
  // every thread converts one column of the slab: 32 rows, written as bytes into shared memory first
  __syncthreads();
  for (int r = 0; r < 32; ++r) tile[r][t] = tile[r][t] * recip;
  __syncthreads();
  for (int i = t; i < 32 * 64; i += 256) {
    const int r = i >> 6, c4 = (i & 63) * 4;
    if (row0 + r < rows && col0 + c4 < C) {
      const uint32_t w = e4m3x4(tile[r][c4], tile[r][c4 + 1], tile[r][c4 + 2], tile[r][c4 + 3]);
      *reinterpret_cast<uint32_t*>(q + (row0 + r) * C + col0 + c4) = w;
    }
  }
}

// ---------------------------------------------------------------------------
// MXFP8 column mode, optionally with the row-quantised copy, for activations: the bandwidth-bound form.
//
// Bound: HBM (reads of the source once, two E4M3 copies and their scales written once).  A tile is 128 rows x 128
// columns: exactly one 512-byte scale atom of either orientation, so both atoms are assembled in shared memory and
// leave as whole 128-byte lines (single scale bytes of a narrower tile are partial-sector writes: 2.3 M of them per
// 73 728 x 4096 operand).  A warp owns 32 rows x 64 columns and a lane 8 rows x 8 columns of it, held in registers
// as loaded (16 bytes per row and lane): row blocks are four neighbouring lanes, column blocks the four lanes of a
// stride of eight, so both maxima are shuffles, nothing of the tile is staged and no barrier separates the loads from
// the stores; every lane stores 8 bytes per row and copy (64 contiguous bytes per row of the warp's tile).
// Block maxima are taken on the bit patterns: |x| of a bf16 is its low 15 bits, their unsigned order is the order of
// the magnitudes, and any pattern above 0x7f80 is a NaN, which makes the block non-finite exactly as the fp32 rule
// does (bf16 -> fp32 is exact).  Two 16-bit lanes are compared per instruction.
// The grid is persistent, so that a launch whose predicate or row count leaves nothing to do ends at once.
//
// Measured against the form it replaces (32 x 512 slabs staged in shared memory, two-byte column stores), 73 728 rows,
// one B200: W13 input gather 4096 wide 309 -> 207 us, gradient gather 329 -> 209 us, SwiGLU forward 1536 wide 216 -> 196 us,
// SwiGLU backward 431 -> 316 us; a dense 32 768 x 4096 matrix 148 -> 98 us (5.6 TB/s of algorithmic bytes).  The SwiGLU
// forms are bound by the sigmoid's arithmetic (69 % of the issue slots), the others by HBM.
// Two scales at a time and rows without a question each (see tile_quantise): 65 536 x 4096 gather 207 -> 175 us, from the combine
// buffer 210 -> 209 (HBM), SwiGLU forward 1536 wide 186 -> 168, backward 246 -> 234.
// ---------------------------------------------------------------------------
constexpr int kTileRows = 128;
constexpr int kTileCols = 128;

// Where a tile comes from: a dense [rows, C] matrix; rows named by a pointer table (a null pointer is a row of
// zeros; pointers may address peer memory); or SwiGLU of a dense [rows, 2C] matrix [gate | up], rounded to
// bf16 exactly as the standalone activation kernel rounds it.
enum TileSource : int { kTileDense = 0, kTileGather = 1, kTileSwiglu = 2 };

struct TileOut {
  uint8_t* q_col;
  uint8_t* s_col;
  uint8_t* q_row;
  uint8_t* s_row;
  int64_t rows;
  int64_t max_rows;
  int C;  // row pitch of the outputs
  int blocked, col_atoms, row_atoms;
};

struct TileLane {
  int warp, lane, rg, cg, slab, half;  // rg: which 8 rows of the warp's 32; cg: which 8 columns of its 64
  __device__ __forceinline__ TileLane() {
    warp = threadIdx.x >> 5;
    lane = threadIdx.x & 31;
    rg = lane >> 3;
    cg = lane & 7;
    slab = warp >> 1;
    half = warp & 1;
  }
  __device__ __forceinline__ int row() const { return slab * 32 + rg * 8; }   // first row inside the tile
  __device__ __forceinline__ int col() const { return half * 64 + cg * 8; }   // first column inside the tile
};

// Quantises the lane's 8 x 8 values (`w[r]` = row r, packed bf16, zeros outside the matrix) of the tile at
// (row0, col0).  `limit` bounds the columns this tile may touch.  `atoms` is the CTA's 1 KiB of scale staging; called
// by every thread of the CTA.
__device__ __forceinline__ void tile_quantise(const uint4 (&w)[8], const TileLane& me, int64_t row0, int col0, int limit,
                                              const TileOut& out, uint8_t* atoms) {
  const int c = col0 + me.col();
  const int64_t r0 = row0 + me.row();
  uint8_t* row_atom = atoms;
  uint8_t* col_atom = atoms + 512;
  float rrow[8], rcol[8];
  {
    uint32_t m[4] = {0, 0, 0, 0};  // maxima of columns 2j (low) and 2j + 1 (high)
    uint32_t n[4];                 // maxima of rows 2p (low) and 2p + 1 (high)
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      uint32_t h[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint4 v = w[2 * p + q];
        const uint32_t ax = v.x & 0x7fff7fffu, ay = v.y & 0x7fff7fffu, az = v.z & 0x7fff7fffu, aw = v.w & 0x7fff7fffu;
        m[0] = __vmaxu2(m[0], ax);
        m[1] = __vmaxu2(m[1], ay);
        m[2] = __vmaxu2(m[2], az);
        m[3] = __vmaxu2(m[3], aw);
        h[q] = __vmaxu2(__vmaxu2(ax, ay), __vmaxu2(az, aw));
      }
      n[p] = __vmaxu2(__byte_perm(h[0], h[1], 0x5410), __byte_perm(h[0], h[1], 0x7632));
      n[p] = __vmaxu2(n[p], __shfl_xor_sync(0xffffffffu, n[p], 1));
      n[p] = __vmaxu2(n[p], __shfl_xor_sync(0xffffffffu, n[p], 2));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      m[j] = __vmaxu2(m[j], __shfl_xor_sync(0xffffffffu, m[j], 8));
      m[j] = __vmaxu2(m[j], __shfl_xor_sync(0xffffffffu, m[j], 16));
    }
    uint32_t nb[4], mb[4];  // scale bytes, 16 bits each
    if (!any_nonfinite2(__vmaxu2(__vmaxu2(__vmaxu2(n[0], n[1]), __vmaxu2(n[2], n[3])),
                                 __vmaxu2(__vmaxu2(m[0], m[1]), __vmaxu2(m[2], m[3]))))) {
      // two scales at a time: one by one they were a sixth of the kernel's instructions
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t r2;
        nb[j] = mxfp8_scale_bits2(n[j], r2);
        rrow[2 * j] = __uint_as_float(r2 << 16);
        rrow[2 * j + 1] = __uint_as_float(r2 & 0xffff0000u);
        mb[j] = mxfp8_scale_bits2(m[j], r2);
        rcol[2 * j] = __uint_as_float(r2 << 16);
        rcol[2 * j + 1] = __uint_as_float(r2 & 0xffff0000u);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        nb[j] = mxfp8_scale_bits(n[j] & 0xffffu, rrow[2 * j]);
        nb[j] |= mxfp8_scale_bits(n[j] >> 16, rrow[2 * j + 1]) << 16;
        mb[j] = mxfp8_scale_bits(m[j] & 0xffffu, rcol[2 * j]);
        mb[j] |= mxfp8_scale_bits(m[j] >> 16, rcol[2 * j + 1]) << 16;
      }
    }
    if ((me.lane & 3) == 0) {
      uint8_t* to = row_atom + me.rg * 8 * 16 + me.slab * 4 + me.half * 2 + (me.cg >> 2);
#pragma unroll
      for (int r = 0; r < 8; ++r) to[r * 16] = static_cast<uint8_t>((r & 1) ? nb[r >> 1] >> 16 : nb[r >> 1]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (me.rg == j) {  // the four row groups share the eight columns' bytes between them
        const int ct = me.col() + 2 * j;
        uint8_t* to = col_atom + (ct & 31) * 16 + (ct >> 5) * 4 + me.slab;
        to[0] = static_cast<uint8_t>(mb[j]);
        to[16] = static_cast<uint8_t>(mb[j] >> 16);
      }
  }
  const bool rowq = out.q_row != nullptr, colq = out.q_col != nullptr;
  const bool col_wide = (reinterpret_cast<uintptr_t>(out.q_col) & 7) == 0;  // a caller's own buffer may be 2-byte aligned
  const int64_t left = out.rows - r0;
  const int live = c < limit ? (left < 8 ? static_cast<int>(left) : 8) : 0;
  uint8_t* dr = out.q_row + r0 * out.C + c;
  uint8_t* dc = out.q_col + r0 * out.C + c;
  auto row_bytes = [&](const float (&f)[8], int r) {
    return make_uint2(e4m3x2_scaled(f[0], f[1], rrow[r], rrow[r]) | (e4m3x2_scaled(f[2], f[3], rrow[r], rrow[r]) << 16),
                      e4m3x2_scaled(f[4], f[5], rrow[r], rrow[r]) | (e4m3x2_scaled(f[6], f[7], rrow[r], rrow[r]) << 16));
  };
  auto col_bytes = [&](const float (&f)[8]) {
    return make_uint2(e4m3x2_scaled(f[0], f[1], rcol[0], rcol[1]) | (e4m3x2_scaled(f[2], f[3], rcol[2], rcol[3]) << 16),
                      e4m3x2_scaled(f[4], f[5], rcol[4], rcol[5]) | (e4m3x2_scaled(f[6], f[7], rcol[6], rcol[7]) << 16));
  };
  if (rowq && colq && col_wide && live == 8) {  // both copies of whole rows: nothing to ask per row
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      float f[8];
      unpack8f(w[r], f);
      *reinterpret_cast<uint2*>(dr + static_cast<int64_t>(r) * out.C) = row_bytes(f, r);
      *reinterpret_cast<uint2*>(dc + static_cast<int64_t>(r) * out.C) = col_bytes(f);
    }
  } else {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (r < live) {
        float f[8];
        unpack8f(w[r], f);
        if (rowq) *reinterpret_cast<uint2*>(dr) = row_bytes(f, r);
        if (colq) {
          const uint2 q = col_bytes(f);
          if (col_wide) {
            *reinterpret_cast<uint2*>(dc) = q;
          } else {
            uint16_t* d2 = reinterpret_cast<uint16_t*>(dc);
            d2[0] = static_cast<uint16_t>(q.x);
            d2[1] = static_cast<uint16_t>(q.x >> 16);
            d2[2] = static_cast<uint16_t>(q.y);
            d2[3] = static_cast<uint16_t>(q.y >> 16);
          }
        }
      }
      dr += out.C;
      dc += out.C;
    }
  }
  __syncthreads();
  // Scales.  A tile that lies wholly inside the matrix owns whole atoms; at the edges (or in a buffer that 16-byte
  // stores cannot reach) only the bytes of real blocks are written, one by one: a caller may have zeroed the rest.
  const int t = threadIdx.x;
  const bool whole = out.blocked && row0 + kTileRows <= out.rows && col0 + kTileCols <= limit && (col0 & 127) == 0 &&
                     ((reinterpret_cast<uintptr_t>(out.s_row) | reinterpret_cast<uintptr_t>(out.s_col)) & 15) == 0;
  if (whole) {
    if (t < 32) {
      if (rowq)
        reinterpret_cast<uint4*>(out.s_row + ((row0 >> 7) * out.row_atoms + (col0 >> 7)) * 512)[t] =
            reinterpret_cast<const uint4*>(row_atom)[t];
    } else if (t < 64) {
      if (colq)
        reinterpret_cast<uint4*>(out.s_col + (static_cast<int64_t>(col0 >> 7) * out.col_atoms + (row0 >> 7)) * 512)[t - 32] =
            reinterpret_cast<const uint4*>(col_atom)[t - 32];
    }
  } else {
    for (int i = t; i < 512; i += 256) {
      if (rowq) {
        const int r = i >> 2, b = i & 3;  // row and 32-column block of the tile
        if (row0 + r < out.rows && col0 + b * 32 < limit)
          out.s_row[blocked_offset(row0 + r, (col0 >> 5) + b, out.row_atoms)] = row_atom[(r & 31) * 16 + (r >> 5) * 4 + b];
      }
      if (colq) {
        const int ct = i >> 2, sl = i & 3;  // column and 32-row block of the tile
        const int64_t rb = (row0 >> 5) + sl;
        if (col0 + ct < limit && row0 + sl * 32 < out.rows) {
          const uint8_t byte = col_atom[(ct & 31) * 16 + (ct >> 5) * 4 + sl];
          if (out.blocked)
            out.s_col[blocked_offset(col0 + ct, static_cast<int>(rb), out.col_atoms)] = byte;
          else
            out.s_col[static_cast<int64_t>(col0 + ct) * ((out.max_rows + 31) / 32) + rb] = byte;
        }
      }
    }
  }
  __syncthreads();  // the staging bytes may be written again
}

// ---------------------------------------------------------------------------
// 32x32 tile mode for weights whose sides are multiples of 128 (the general form is the slab kernel above): a CTA takes
// 128 x 128, a warp 32 rows x 64 columns of it (two tiles), a lane 8 rows x 8 columns held in registers as loaded.  The tile
// maximum is four shuffles, nothing of the matrix is staged.  The 4 x 4 scales of a CTA fill one 512-byte atom of either
// orientation, 32 equal 16-byte rows each, which leave as whole lines (the slab form writes single bytes).
// Bound: HBM.  Both weights of 16 experts x 1024 x 640 (63 MB) 95 us in slabs of 32 x 256, 21 us so.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) mxfp8_tile32_kernel(const uint4* __restrict__ x, int64_t expert_rows, int C,
                                                           uint8_t* __restrict__ q, uint8_t* __restrict__ s0,
                                                           uint8_t* __restrict__ s1) {
  __shared__ __align__(16) uint8_t sc[2][16];  // [row block][column block], and transposed
  const TileLane me;
  const int col_tiles = C >> 7;
  const int64_t row_tile = blockIdx.x / col_tiles;
  const int col_tile = static_cast<int>(blockIdx.x - row_tile * col_tiles);
  const int64_t r0 = row_tile * kTileRows + me.row();
  const int c = col_tile * kTileCols + me.col();
  uint4 w[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) w[r] = x[((r0 + r) * C + c) >> 3];
  uint32_t m = 0;
#pragma unroll
  for (int r = 0; r < 8; ++r)
    m = __vmaxu2(m, __vmaxu2(__vmaxu2(w[r].x & 0x7fff7fffu, w[r].y & 0x7fff7fffu), __vmaxu2(w[r].z & 0x7fff7fffu, w[r].w & 0x7fff7fffu)));
  // the four column groups of a tile are neighbouring lanes, its four row groups eight lanes apart
#pragma unroll
  for (int d = 1; d <= 16; d <<= 1)
    if (d != 4) m = __vmaxu2(m, __shfl_xor_sync(0xffffffffu, m, d));
  float recip;
  const uint32_t byte = mxfp8_scale_bits((m >> 16) > (m & 0xffffu) ? m >> 16 : m & 0xffffu, recip);
  const int cb = me.half * 2 + (me.cg >> 2);
  if ((me.lane & 0x1b) == 0) {  // one lane per tile
    sc[0][me.slab * 4 + cb] = static_cast<uint8_t>(byte);
    sc[1][cb * 4 + me.slab] = static_cast<uint8_t>(byte);
  }
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const uint4 v = w[r];
    *reinterpret_cast<uint2*>(q + (r0 + r) * C + c) = make_uint2(
        e4m3x2_scaled(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), recip, recip) |
            (e4m3x2_scaled(__uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u), recip, recip) << 16),
        e4m3x2_scaled(__uint_as_float(v.z << 16), __uint_as_float(v.z & 0xffff0000u), recip, recip) |
            (e4m3x2_scaled(__uint_as_float(v.w << 16), __uint_as_float(v.w & 0xffff0000u), recip, recip) << 16));
  }
  __syncthreads();
  const int t = threadIdx.x;
  if (t < 64) {
    // atoms of either orientation: an expert's row blocks x column blocks, and the other way round
    const int64_t row_blocks = expert_rows >> 7, e = row_tile / row_blocks, rb = row_tile - e * row_blocks;
    const int64_t first = e * row_blocks * col_tiles;
    const int64_t atom = t < 32 ? first + rb * col_tiles + col_tile : first + static_cast<int64_t>(col_tile) * row_blocks + rb;
    reinterpret_cast<uint4*>((t < 32 ? s0 : s1) + atom * 512)[t & 31] = *reinterpret_cast<const uint4*>(sc[t >> 5]);
  }
}

// Placement chosen on the device: each pointer is an allocation base and the byte offset is read from device memory
// when the kernel starts (all null = the pointers are final).  `compact_cols` sizes the column-scale layout from the
// device row count instead of max_rows, so that a column bundle occupies exactly dim * rows / 32 bytes; `cond`
// (optional) turns the whole launch into a no-op when it reads 0.
struct PlacedOffsets {
  const int64_t* x;
  const int64_t* x2;
  const int64_t* q_col;
  const int64_t* s_col;
  const int64_t* q_row;
  const int64_t* s_row;
  const int* cond;
  int compact_cols;
};

template <class T>
__device__ __forceinline__ T* placed(T* base, const int64_t* off) {
  if (base == nullptr || off == nullptr) return base;
  return reinterpret_cast<T*>(reinterpret_cast<uintptr_t>(base) + static_cast<uintptr_t>(*off));
}

// 16 bytes global -> shared without passing through registers; `bytes` 0 fills with zeros and reads nothing.
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem_dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A lane's 8 rows of every input arrive in shared-memory slots of its own through asynchronous copies: the next tile's
// rows are in flight while this tile is converted and stored, without holding registers, and the activation of the SwiGLU
// forms runs in a rolled loop (the exponential and the IEEE reciprocal of 64 unrolled elements did not fit the
// instruction cache: 265 against 196 us).  Slots are private to the thread, so no barrier is involved.
constexpr int kTileSlot = 8 * 256;  // uint4 slots of one input

template <int kSource>
__global__ void __launch_bounds__(256, 3) mxfp8_colrow_kernel(const uint4* __restrict__ x, const int64_t* __restrict__ row_ptrs,
                                                              ActParams act, const int32_t* num_rows,
                                                              int64_t max_rows, int C, uint8_t* __restrict__ q_col,
                                                              uint8_t* __restrict__ s_col, int blocked, int col_atoms,
                                                              uint8_t* __restrict__ q_row, uint8_t* __restrict__ s_row,
                                                              int row_atoms, PlacedOffsets at) {
  __shared__ __align__(16) uint8_t atoms[1024];
  extern __shared__ uint4 slots[];
  if (at.cond != nullptr && *at.cond == 0) return;
  int64_t rows = num_rows ? *num_rows : max_rows;
  if (rows > max_rows) rows = max_rows;
  x = placed(x, at.x);
  if (at.compact_cols) col_atoms = static_cast<int>(((rows + 31) / 32 + 3) / 4);
  const TileOut out{placed(q_col, at.q_col), placed(s_col, at.s_col), placed(q_row, at.q_row), placed(s_row, at.s_row),
                    rows, max_rows, C, blocked, col_atoms, row_atoms};
  const TileLane me;
  const int vec_per_row = C >> 3;
  const int col_tiles = (C + kTileCols - 1) / kTileCols;
  const int64_t tiles = (rows + kTileRows - 1) / kTileRows * col_tiles;
  uint4* slot = slots + threadIdx.x;
  uint4* up = slot + kTileSlot;
  // what a copy of zero bytes names as its source: nothing is read there, but the address has to be on 16 bytes as for any
  // other copy of this width, which a table of 8-byte pointers need not be
  const void* nowhere = reinterpret_cast<const void*>(reinterpret_cast<uintptr_t>(row_ptrs) & ~uintptr_t(15));
  auto fetch = [&](int64_t tile) {  // the lane's 8 rows of a tile on their way into its slots
    const int64_t r0 = tile / col_tiles * kTileRows + me.row();
    const int c = static_cast<int>(tile - tile / col_tiles * col_tiles) * kTileCols + me.col();
    const int v = c >> 3;
    const int64_t left = rows - r0;
    const int live = c < C ? (left < 8 ? static_cast<int>(left) : 8) : 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (kSource == kTileSwiglu) {
        const uint4* src = x + (r0 + r) * 2 * vec_per_row + v;
        cp_async16(slot + 256 * r, r < live ? src : x, r < live ? 16 : 0);
        cp_async16(up + 256 * r, r < live ? src + vec_per_row : x, r < live ? 16 : 0);
      } else if (kSource == kTileDense) {
        cp_async16(slot + 256 * r, r < live ? x + (r0 + r) * vec_per_row + v : x, r < live ? 16 : 0);
      } else {
        const uint4* src = r < live ? reinterpret_cast<const uint4*>(row_ptrs[r0 + r]) : nullptr;
        cp_async16(slot + 256 * r, src != nullptr ? static_cast<const void*>(src + v) : nowhere, src != nullptr ? 16 : 0);
      }
    }
  };
  if (static_cast<int64_t>(blockIdx.x) < tiles) fetch(blockIdx.x);
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t row0 = tile / col_tiles * kTileRows;
    const int col0 = static_cast<int>(tile - tile / col_tiles * col_tiles) * kTileCols;
    cp_async_wait_all();
    if (kSource == kTileSwiglu) {
#pragma unroll 1
      for (int r = 0; r < 8; ++r) {
        float g[8], u[8], z[8];
        unpack8f(slot[256 * r], g);
        unpack8f(up[256 * r], u);
        swiglu_f32(g, u, z, act);
        slot[256 * r] = make_uint4(pack_bf16x2(z[0], z[1]), pack_bf16x2(z[2], z[3]), pack_bf16x2(z[4], z[5]), pack_bf16x2(z[6], z[7]));
      }
    }
    uint4 w[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) w[r] = slot[256 * r];
    if (tile + gridDim.x < tiles) fetch(tile + gridDim.x);  // in flight behind this tile's arithmetic and stores
    tile_quantise(w, me, row0, col0, C, out, atoms);
  }
}

// SwiGLU backward fused in: from h1 = [gate | up] ([rows, 2F]) and dz = dL/dh2 ([rows, F]) a CTA computes the
// gate-gradient tile and the matching up-gradient tile of grad_h1 = [dgate | dup] (rounded to bf16 as the standalone
// backward kernel rounds them) and quantises both; grad_h1 itself is never written.  Either copy may be left out.
__global__ void __launch_bounds__(256, 2) mxfp8_swiglu_bwd_colrow_kernel(const uint4* __restrict__ h1,
                                                                         const uint4* __restrict__ dz, ActParams act,
                                                                         const int32_t* num_rows, int64_t max_rows, int F,
                                                                         uint8_t* __restrict__ q_col,
                                                                         uint8_t* __restrict__ s_col, int col_atoms,
                                                                         uint8_t* __restrict__ q_row,
                                                                         uint8_t* __restrict__ s_row, int row_atoms,
                                                                         PlacedOffsets at) {
  __shared__ __align__(16) uint8_t atoms[1024];
  extern __shared__ uint4 slots[];
  int64_t rows = num_rows ? *num_rows : max_rows;
  if (rows > max_rows) rows = max_rows;
  h1 = placed(h1, at.x);
  dz = placed(dz, at.x2);
  if (at.compact_cols) col_atoms = static_cast<int>(((rows + 31) / 32 + 3) / 4);
  const TileOut out{placed(q_col, at.q_col), placed(s_col, at.s_col), placed(q_row, at.q_row), placed(s_row, at.s_row),
                    rows, max_rows, 2 * F, 1, col_atoms, row_atoms};
  const TileLane me;
  const int vec_per_row = F >> 3;
  const int col_tiles = (F + kTileCols - 1) / kTileCols;
  const int64_t tiles = (rows + kTileRows - 1) / kTileRows * col_tiles;
  uint4* gate = slots + threadIdx.x;
  uint4* up = gate + kTileSlot;
  uint4* grad = up + kTileSlot;
  auto fetch = [&](int64_t tile) {
    const int64_t r0 = tile / col_tiles * kTileRows + me.row();
    const int c = static_cast<int>(tile - tile / col_tiles * col_tiles) * kTileCols + me.col();
    const int v = c >> 3;
    const int64_t left = rows - r0;
    const int live = c < F ? (left < 8 ? static_cast<int>(left) : 8) : 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const uint4* src = h1 + (r0 + r) * 2 * vec_per_row + v;
      cp_async16(gate + 256 * r, r < live ? src : h1, r < live ? 16 : 0);
      cp_async16(up + 256 * r, r < live ? src + vec_per_row : h1, r < live ? 16 : 0);
      cp_async16(grad + 256 * r, r < live ? dz + (r0 + r) * vec_per_row + v : h1, r < live ? 16 : 0);
    }
  };
  if (static_cast<int64_t>(blockIdx.x) < tiles) fetch(blockIdx.x);
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t row0 = tile / col_tiles * kTileRows;
    const int col0 = static_cast<int>(tile - tile / col_tiles * col_tiles) * kTileCols;
    cp_async_wait_all();
#pragma unroll 1
    for (int r = 0; r < 8; ++r) {
      float x[8], y[8], d[8], dx[8], dy[8];
      unpack8f(gate[256 * r], x);
      unpack8f(up[256 * r], y);
      unpack8f(grad[256 * r], d);
      swiglu_bwd_f32(x, y, d, act, dx, dy);
      gate[256 * r] = make_uint4(pack_bf16x2(dx[0], dx[1]), pack_bf16x2(dx[2], dx[3]), pack_bf16x2(dx[4], dx[5]), pack_bf16x2(dx[6], dx[7]));
      up[256 * r] = make_uint4(pack_bf16x2(dy[0], dy[1]), pack_bf16x2(dy[2], dy[3]), pack_bf16x2(dy[4], dy[5]), pack_bf16x2(dy[6], dy[7]));
    }
#pragma unroll 1
    for (int which = 0; which < 2; ++which) {
      uint4 w[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) w[r] = gate[which * kTileSlot + 256 * r];
      if (which == 1 && tile + gridDim.x < tiles) fetch(tile + gridDim.x);
      tile_quantise(w, me, row0, which * F + col0, (which + 1) * F, out, atoms);
    }
  }
}

// ---------------------------------------------------------------------------
// NVFP4
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint8_t nvfp4_block_scale(float amax, float scale, float& mult) {
  if (amax == __int_as_float(0x7f800000)) amax = __int_as_float(0x7fc00000);
  float raw = (amax * scale) * (1.0f / 6.0f);
  raw = raw < 0.001953125f ? 0.001953125f : raw;
  raw = raw > 448.0f ? 448.0f : raw;
  const uint8_t byte =
      static_cast<uint8_t>(__nv_cvt_float2_to_fp8x2(make_float2(raw, 0.f), __NV_SATFINITE, __NV_E4M3) & 0xFF);
  const __half_raw h = __nv_cvt_fp8_to_halfraw(byte, __NV_E4M3);
  const float sf = __half2float(*reinterpret_cast<const __half*>(&h));
  mult = byte != 0 ? __fdiv_rn(scale, sf) : 0.f;
  return byte;
}

__device__ __forceinline__ uint32_t e2m1x8(const float (&f)[8], float m) {
  uint32_t out = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t b = __nv_cvt_float2_to_fp4x2(make_float2(f[2 * i] * m, f[2 * i + 1] * m), __NV_E2M1, cudaRoundNearest);
    out |= (b & 0xFF) << (8 * i);
  }
  return out;
}

// One CTA (128 threads) per token row: row amax, then 16-element blocks (2 threads each).
__global__ void __launch_bounds__(128) nvfp4_token_kernel(const uint4* __restrict__ x, const int32_t* num_rows,
                                                          int64_t max_rows, int vec_per_row, uint8_t* q,
                                                          int64_t q_stride, uint8_t* s, int64_t s_stride,
                                                          uint8_t* inv, int64_t inv_stride, int blocked_atoms,
                                                          const int64_t* __restrict__ live, IdPublish ids) {
  __shared__ float red[4];
  publish_ids(ids);
  int64_t rows = num_rows ? *num_rows : max_rows;
  if (rows > max_rows) rows = max_rows;
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    if (live != nullptr && live[r] == 0) continue;  // a padding row: nothing reads its quantised form
    const uint4* xr = x + r * vec_per_row;
    float amax = 0.f;
    for (int v = threadIdx.x; v < vec_per_row; v += 128) {
      float f[8];
      unpack8f(xr[v], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(f[j]));
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    const float row_scale = 2688.0f * __frcp_rn(fmaxf(amax, 1e-8f));
    if (threadIdx.x == 0 && inv != nullptr) *reinterpret_cast<float*>(inv + r * inv_stride) = __frcp_rn(row_scale);
    for (int v0 = 0; v0 < vec_per_row; v0 += 128) {
      const int v = v0 + threadIdx.x;
      float f[8];
      float bmax = 0.f;
      if (v < vec_per_row) {
        unpack8f(xr[v], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) bmax = amax_nonfinite(bmax, f[j]);
      }
      const float other = __shfl_xor_sync(0xffffffffu, bmax, 1);
      bmax = (other != other) ? other : fmaxf(bmax, other);
      float mult;
      const uint8_t byte = nvfp4_block_scale(bmax, row_scale, mult);
      if (v < vec_per_row) {
        *reinterpret_cast<uint32_t*>(q + r * q_stride + v * 4) = e2m1x8(f, mult);
        if ((v & 1) == 0) {
          if (blocked_atoms > 0)
            s[blocked_offset(r, v >> 1, blocked_atoms)] = byte;
          else
            s[r * s_stride + (v >> 1)] = byte;
        }
      }
    }
  }
}

// The form for rows that fit the registers of their threads: `kThreads` threads (a warp, or a CTA of 256) hold a whole
// row, `kBpt` 16-element blocks per thread, between the row-maximum pass and the quantising pass.  A thread owns whole
// blocks, so the scale (a division and two conversions) is computed once per block, without exchange between lanes.
// Same arithmetic as the kernel above: block maxima are taken on the bf16 bit patterns (their order is the order of the
// magnitudes, a NaN makes the block non-finite); the row maximum ignores NaNs, so a block that holds one is gone through
// again.  Bound: HBM for long inputs (read once, 0.56 bytes per element written).  One B200: 65 536 x 2048 with padding
// rows skipped 68 us (eight elements per lane, the scale computed twice per block: 113 us); 8192 x 7168 into packed
// rows 30 us (a CTA of 128 reading the row twice: 49 us).
template <int kThreads, int kBpt>
__global__ void __launch_bounds__(256) nvfp4_token_reg_kernel(const uint4* __restrict__ x, const int32_t* num_rows,
                                                              int64_t max_rows, int blocks_per_row, uint8_t* q,
                                                              int64_t q_stride, uint8_t* s, int64_t s_stride,
                                                              uint8_t* inv, int64_t inv_stride, int blocked_atoms,
                                                              const int64_t* __restrict__ live, IdPublish ids) {
  __shared__ float red[2][8];
  publish_ids(ids);
  int64_t rows = num_rows ? *num_rows : max_rows;
  if (rows > max_rows) rows = max_rows;
  constexpr int kRowsPerCta = 256 / kThreads;
  const int t = threadIdx.x & (kThreads - 1), lane = threadIdx.x & 31;
  const int64_t step = static_cast<int64_t>(gridDim.x) * kRowsPerCta;
  const bool wide = ((reinterpret_cast<uintptr_t>(q) | static_cast<uintptr_t>(q_stride)) & 7) == 0;
  int parity = 0;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * kRowsPerCta + threadIdx.x / kThreads; r < rows; r += step) {
    if (live != nullptr && live[r] == 0) continue;  // a padding row: nothing reads its quantised form
    const uint4* xr = x + r * blocks_per_row * 2;
    uint4 w[2 * kBpt];
#pragma unroll
    for (int j = 0; j < kBpt; ++j) {
      const int b = j * kThreads + t;
      const bool in = b < blocks_per_row;
      w[2 * j] = in ? xr[2 * b] : make_uint4(0, 0, 0, 0);
      w[2 * j + 1] = in ? xr[2 * b + 1] : make_uint4(0, 0, 0, 0);
    }
    uint32_t top[kBpt];
    float amax = 0.f;
#pragma unroll
    for (int j = 0; j < kBpt; ++j) {
      const uint32_t v[8] = {w[2 * j].x, w[2 * j].y, w[2 * j].z, w[2 * j].w,
                             w[2 * j + 1].x, w[2 * j + 1].y, w[2 * j + 1].z, w[2 * j + 1].w};
      uint32_t m = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) m = __vmaxu2(m, v[i] & 0x7fff7fffu);
      top[j] = (m >> 16) > (m & 0xffffu) ? m >> 16 : m & 0xffffu;
      if (top[j] <= 0x7f80u) {
        amax = fmaxf(amax, __uint_as_float(top[j] << 16));
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          amax = fmaxf(amax, fmaxf(fabsf(__uint_as_float(v[i] << 16)), fabsf(__uint_as_float(v[i] & 0xffff0000u))));
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
    if (kThreads > 32) {
      // two sets of partial maxima in turn: one barrier per row is enough
      if (lane == 0) red[parity][threadIdx.x >> 5] = amax;
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = fmaxf(amax, red[parity][i]);
      parity ^= 1;
    }
    const float row_scale = 2688.0f * __frcp_rn(fmaxf(amax, 1e-8f));
    if (t == 0 && inv != nullptr) *reinterpret_cast<float*>(inv + r * inv_stride) = __frcp_rn(row_scale);
#pragma unroll
    for (int j = 0; j < kBpt; ++j) {
      const int b = j * kThreads + t;
      if (b >= blocks_per_row) continue;
      float mult;
      const uint8_t byte = nvfp4_block_scale(amax_from_bf16_bits(top[j]), row_scale, mult);
      float f[8], g[8];
      unpack8f(w[2 * j], f);
      unpack8f(w[2 * j + 1], g);
      uint32_t* dst = reinterpret_cast<uint32_t*>(q + r * q_stride + b * 8);
      const uint32_t lo = e2m1x8(f, mult), hi = e2m1x8(g, mult);
      if (wide) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(lo, hi);
      } else {
        dst[0] = lo;
        dst[1] = hi;
      }
      if (blocked_atoms > 0)
        s[blocked_offset(r, b, blocked_atoms)] = byte;
      else
        s[r * s_stride + b] = byte;
    }
  }
}

// Weights: per-expert global scale given; rows of K elements; scales natural or blocked per expert.
__global__ void __launch_bounds__(256) nvfp4_weight_kernel(const uint4* __restrict__ w, const float* __restrict__ gs,
                                                           int64_t rows_per_expert, int64_t total_rows,
                                                           int vec_per_row, uint32_t* __restrict__ q,
                                                           uint8_t* __restrict__ s, int blocked, int n_col_atoms) {
  const int64_t total = total_rows * vec_per_row;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < (total + 31) / 32 * 32;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const bool live = i < total;
    const int64_t r = live ? i / vec_per_row : 0;
    const int64_t e = r / rows_per_expert;
    float f[8];
    float bmax = 0.f;
    if (live) {
      unpack8f(w[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) bmax = amax_nonfinite(bmax, f[j]);
    }
    const float other = __shfl_xor_sync(0xffffffffu, bmax, 1);
    bmax = (other != other) ? other : fmaxf(bmax, other);
    if (!live) continue;
    float g = gs[e];
    g = g > 1e-12f ? g : 1e-12f;
    float mult;
    const uint8_t byte = nvfp4_block_scale(bmax, g, mult);
    q[i] = e2m1x8(f, mult);
    if ((i & 1) == 0) {
      const int blk = static_cast<int>(i - r * vec_per_row) >> 1;
      if (blocked) {
        const int64_t rl = r - e * rows_per_expert;
        const int64_t grp = (rows_per_expert + 127) / 128 * 128 * static_cast<int64_t>(n_col_atoms) * 4;
        s[e * grp + blocked_offset(rl, blk, n_col_atoms)] = byte;
      } else {
        s[r * (vec_per_row >> 1) + blk] = byte;
      }
    }
  }
}

// natural [rows][cols] scale bytes -> blocked atoms (padding entries are written as 0)
__global__ void sf_swizzle_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int64_t rows, int cols,
                                  int64_t padded_rows, int n_col_atoms) {
  const int64_t total = padded_rows * n_col_atoms * 4;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / (n_col_atoms * 4);
    const int c = static_cast<int>(i - r * (n_col_atoms * 4));
    dst[blocked_offset(r, c, n_col_atoms)] = (r < rows && c < cols) ? src[r * cols + c] : 0;
  }
}

// Packed dispatch rows [q | natural scales | fp32 inverse scale | pad] fetched through a pointer table
// (sources may be peer memory) and unpacked into GEMM operand form: dense q rows, blocked scales,
// per-row inverse scales.  A null pointer yields a zero row.
//
// Bound: HBM writes (the source rows of a rank fit L2).  A warp copies rows in pieces of 128 vectors.  The scales of a
// 128-row block are written in whole 32-byte sectors: a lane reads one atom's word of the rows l, l + 32, l + 64, l + 96
// and of their neighbours l + 1 ... (128 contiguous bytes of every row per warp, which is also what peer reads want) and
// stores the atom's bytes of both.  A word per row and atom, each in a sector of its own, made 65 536 rows of 448 scales
// take 101 us in all; 76 us now.  The last, partial block of a row count that is no multiple of 128 takes the
// word-wise form.
__global__ void __launch_bounds__(256) gather_packed_kernel(const int64_t* __restrict__ ptrs,
                                                            const int32_t* __restrict__ num_rows, int64_t max_rows,
                                                            int q_vecs, int scale_cols, int has_inv, uint8_t* q_base,
                                                            const int64_t* q_off, uint8_t* sf_base,
                                                            const int64_t* sf_off, uint8_t* inv_base,
                                                            const int64_t* inv_off, const int* cond, int live_only) {
  if (cond != nullptr && *cond == 0) return;
  int64_t rows = *num_rows;
  if (rows > max_rows) rows = max_rows;
  uint4* q = reinterpret_cast<uint4*>(q_base + (q_off ? *q_off : 0));
  uint8_t* sf = sf_base + (sf_off ? *sf_off : 0);
  float* inv = has_inv ? reinterpret_cast<float*>(inv_base + (inv_off ? *inv_off : 0)) : nullptr;
  const int atoms = (scale_cols + 3) / 4;
  const int lane = threadIdx.x & 31;
  const int64_t first = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  const bool whole_atoms = (reinterpret_cast<uintptr_t>(sf) & 15) == 0;
  // scale tasks first (eight rows of one 128-row block, 32 atoms), then row pieces
  const int chunks = (atoms + 31) >> 5;
  const int64_t blocks = whole_atoms ? rows >> 7 : 0;
  for (int64_t i = first; i < blocks * 16 * chunks; i += warps) {
    const int64_t pair = i / chunks;
    const int c4 = static_cast<int>(i - pair * chunks) * 32 + lane;
    const int64_t blk = pair >> 4;
    const int l0 = static_cast<int>(pair & 15) * 2;
    uint32_t w[2][4];
    int64_t srcs[8], any = 0;
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      srcs[g] = ptrs[blk * 128 + 32 * (g >> 1) + l0 + (g & 1)];
      any |= srcs[g];
    }
    if (live_only && any == 0) continue;
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      const int64_t src = srcs[g];
      w[g & 1][g >> 1] = (src != 0 && c4 < atoms)
                             ? __ldcg(reinterpret_cast<const uint32_t*>(src + static_cast<int64_t>(q_vecs) * 16) + c4)
                             : 0;
    }
    if (c4 < atoms) {
      uint4* dst = reinterpret_cast<uint4*>(sf + (blk * atoms + c4) * 512) + l0;
      dst[0] = make_uint4(w[0][0], w[0][1], w[0][2], w[0][3]);
      dst[1] = make_uint4(w[1][0], w[1][1], w[1][2], w[1][3]);
    }
  }
  const int pieces = (q_vecs + 127) >> 7;
  for (int64_t i = first; i < rows * pieces; i += warps) {
    const int64_t r = pieces == 1 ? i : i / pieces;
    const int piece = static_cast<int>(i - r * pieces);
    const uint8_t* src = reinterpret_cast<const uint8_t*>(ptrs[r]);
    if (live_only && src == nullptr) continue;
    const int v0 = piece * 128 + lane;
    uint4 t[4];  // four 16-byte loads in flight per lane
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int v = v0 + 32 * j;
      t[j] = (src && v < q_vecs) ? __ldcg(reinterpret_cast<const uint4*>(src) + v) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int v = v0 + 32 * j;
      if (v < q_vecs) q[r * q_vecs + v] = t[j];
    }
    if (piece != 0) continue;
    const uint8_t* ssrc = src ? src + static_cast<int64_t>(q_vecs) * 16 : nullptr;
    if ((r >> 7) >= blocks) {
      for (int c4 = lane; c4 < atoms; c4 += 32)
        *reinterpret_cast<uint32_t*>(sf + blocked_offset(r, c4 * 4, atoms)) =
            ssrc ? __ldcg(reinterpret_cast<const uint32_t*>(ssrc) + c4) : 0;
    }
    if (inv != nullptr && lane == 0)
      inv[r] = src ? __ldcg(reinterpret_cast<const float*>(ssrc + scale_cols)) : 0.f;
  }
}

// Grid of the persistent 128 x 128 tile quantisers: `per_sm` resident CTAs per SM, never more than there are tiles.
static int tile_grid(int64_t max_rows, int64_t C, int per_sm) {
  const int64_t tiles = ceil_div64(max_rows, kTileRows) * ceil_div64(C, kTileCols);
  const int64_t cap = grid_cap(per_sm);
  return static_cast<int>(tiles < cap ? tiles : cap);
}

static int blocks_for(int64_t items, int threads, int cap) {
  int64_t b = (items + threads - 1) / threads;
  if (b > cap) b = cap;
  return b < 1 ? 1 : static_cast<int>(b);
}

}  // namespace dm

using namespace dm;

static int mxfp8_row_impl(const IdPublish& ids, const int64_t* live, const void* x, const int32_t* num_rows, int64_t max_rows, int64_t C, void* q,
                          int64_t q_row_stride, void* scales, int64_t scale_row_stride, int blocked, void* stream) {
  if (!x || !q || !scales || max_rows < 0 || C <= 0 || (C % 32) != 0) return kRcBadArg;
  if (q_row_stride == 0) q_row_stride = C;
  if (scale_row_stride == 0) scale_row_stride = C / 32;
  if ((q_row_stride % 8) != 0) return kRcBadArg;
  if (max_rows == 0) return kRcOk;
  const int vec = static_cast<int>(C / 8);
  const int atoms = static_cast<int>((C / 32 + 3) / 4);
  mxfp8_row_kernel<<<blocks_for(max_rows * ((vec + 127) / 128), 8, grid_cap(8)), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(x), num_rows, max_rows, vec, static_cast<uint8_t*>(q), q_row_stride,
      static_cast<uint8_t*>(scales), scale_row_stride, blocked, atoms, live, ids);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int dm_quant_mxfp8_row(const void* x, const int32_t* num_rows, int64_t max_rows, int64_t C, void* q,
                                  int64_t q_row_stride, void* scales, int64_t scale_row_stride, int blocked,
                                  void* stream) {
  return mxfp8_row_impl(IdPublish{}, nullptr, x, num_rows, max_rows, C, q, q_row_stride, scales, scale_row_stride, blocked, stream);
}

extern "C" int dm_quant_mxfp8_row_live(const int64_t* row_live, const void* x, const int32_t* num_rows, int64_t max_rows,
                                       int64_t C, void* q, int64_t q_row_stride, void* scales, int64_t scale_row_stride,
                                       int blocked, void* stream) {
  if (!row_live) return kRcBadArg;
  return mxfp8_row_impl(IdPublish{}, row_live, x, num_rows, max_rows, C, q, q_row_stride, scales, scale_row_stride, blocked, stream);
}

extern "C" int dm_quant_mxfp8_col(const void* x, const int32_t* num_rows, int64_t max_rows, int64_t C, void* q,
                                  void* scales, int blocked, void* stream) {
  if (!x || !q || !scales || max_rows < 0 || C <= 0 || (C % 4) != 0) return kRcBadArg;
  if (max_rows == 0) return kRcOk;
  const int atoms = static_cast<int>(((max_rows + 31) / 32 + 3) / 4);
  if ((C % 16) == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(q)) % 16) == 0) {
    const int fast = tile_grid(max_rows, C, 3);
    mxfp8_colrow_kernel<kTileDense><<<fast, 256, kTileSlot * 16, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint4*>(x), nullptr, ActParams{0, 1.0f, 0.0f}, num_rows, max_rows, static_cast<int>(C),
        static_cast<uint8_t*>(q), static_cast<uint8_t*>(scales), blocked, atoms, nullptr, nullptr, 0, PlacedOffsets{});
    return static_cast<int>(cudaGetLastError());
  }
  const dim3 grid(static_cast<unsigned>((C + 255) / 256), static_cast<unsigned>((max_rows + 31) / 32));
  mxfp8_slab_kernel<false><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), num_rows, max_rows, static_cast<int>(C), static_cast<uint8_t*>(q),
      static_cast<uint8_t*>(scales), nullptr, blocked, atoms, 0, max_rows);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int dm_quant_mxfp8_rowcol(const void* x, const int32_t* num_rows, int64_t max_rows, int64_t C, void* q_row,
                                     void* scales_row_blocked, void* q_col, void* scales_col_blocked, void* stream) {
  if (!x || !q_row || !scales_row_blocked || !q_col || !scales_col_blocked || max_rows < 0 || C <= 0 || (C % 32) != 0)
    return kRcBadArg;
  if (max_rows == 0) return kRcOk;
  const int grid = tile_grid(max_rows, C, 3);
  const int col_atoms = static_cast<int>(((max_rows + 31) / 32 + 3) / 4);
  const int row_atoms = static_cast<int>((C / 32 + 3) / 4);
  mxfp8_colrow_kernel<kTileDense><<<grid, 256, kTileSlot * 16, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(x), nullptr, ActParams{0, 1.0f, 0.0f}, num_rows, max_rows, static_cast<int>(C),
      static_cast<uint8_t*>(q_col), static_cast<uint8_t*>(scales_col_blocked), 1, col_atoms,
      static_cast<uint8_t*>(q_row), static_cast<uint8_t*>(scales_row_blocked), row_atoms, PlacedOffsets{});
  return static_cast<int>(cudaGetLastError());
}

static int launch_rowcol_gather(const int64_t* row_ptrs, const int32_t* num_rows, int64_t max_rows, int64_t C,
                                void* q_row, void* sf_row, void* q_col, void* sf_col, PlacedOffsets at, void* stream) {
  if (!row_ptrs || !q_row || !sf_row || (q_col == nullptr) != (sf_col == nullptr) || max_rows < 0 || C <= 0 ||
      (C % 32) != 0)
    return kRcBadArg;  // the column copy may be left out (a forward nothing will differentiate)
  if (max_rows == 0) return kRcOk;
  const int grid = tile_grid(max_rows, C, 3);
  const int col_atoms = static_cast<int>(((max_rows + 31) / 32 + 3) / 4);
  const int row_atoms = static_cast<int>((C / 32 + 3) / 4);
  mxfp8_colrow_kernel<kTileGather><<<grid, 256, kTileSlot * 16, static_cast<cudaStream_t>(stream)>>>(
      nullptr, row_ptrs, ActParams{0, 1.0f, 0.0f}, num_rows, max_rows, static_cast<int>(C), static_cast<uint8_t*>(q_col),
      static_cast<uint8_t*>(sf_col), 1, col_atoms, static_cast<uint8_t*>(q_row), static_cast<uint8_t*>(sf_row),
      row_atoms, at);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int dm_quant_mxfp8_rowcol_gather(const int64_t* row_ptrs, const int32_t* num_rows, int64_t max_rows, int64_t C,
                                            void* q_row, void* scales_row_blocked, void* q_col,
                                            void* scales_col_blocked, void* stream) {
  return launch_rowcol_gather(row_ptrs, num_rows, max_rows, C, q_row, scales_row_blocked, q_col, scales_col_blocked,
                              PlacedOffsets{}, stream);
}

extern "C" int dm_quant_mxfp8_rowcol_gather_at(const int64_t* row_ptrs, const int32_t* num_rows, int64_t max_rows,
                                               int64_t C, dm_operand q_row, dm_operand sf_row, dm_operand q_col,
                                               dm_operand sf_col, const int* cond, void* stream) {
  PlacedOffsets at{nullptr, nullptr, q_col.offset, sf_col.offset, q_row.offset, sf_row.offset, cond, 1};
  return launch_rowcol_gather(row_ptrs, num_rows, max_rows, C, q_row.base, sf_row.base, q_col.base, sf_col.base, at,
                              stream);
}

static int launch_swiglu_fwd_quant(const void* h1, const int32_t* num_rows, int64_t max_rows, int64_t F, int clamped,
                                   float alpha, float limit, void* q_row, void* sf_row, void* q_col, void* sf_col,
                                   PlacedOffsets at, void* stream) {
  if (!h1 || !q_row || !sf_row || (q_col == nullptr) != (sf_col == nullptr) || max_rows < 0 || F <= 0 || (F % 32) != 0)
    return kRcBadArg;
  if (max_rows == 0) return kRcOk;
  constexpr int kSmem = 2 * kTileSlot * 16;
  static PerDeviceOnce attr_set;
  const int rc_attr = once_per_device(attr_set, [] {
    return static_cast<int>(
        cudaFuncSetAttribute(mxfp8_colrow_kernel<kTileSwiglu>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  });
  if (rc_attr != 0) return rc_attr;
  const int grid = tile_grid(max_rows, F, 3);
  const int col_atoms = static_cast<int>(((max_rows + 31) / 32 + 3) / 4);
  const int row_atoms = static_cast<int>((F / 32 + 3) / 4);
  mxfp8_colrow_kernel<kTileSwiglu><<<grid, 256, kSmem, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(h1), nullptr, ActParams{clamped, alpha, limit}, num_rows, max_rows, static_cast<int>(F),
      static_cast<uint8_t*>(q_col), static_cast<uint8_t*>(sf_col), 1, col_atoms, static_cast<uint8_t*>(q_row),
      static_cast<uint8_t*>(sf_row), row_atoms, at);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int dm_swiglu_fwd_quant_mxfp8_rowcol(const void* h1, const int32_t* num_rows, int64_t max_rows, int64_t F,
                                                int clamped, float alpha, float limit, void* q_row,
                                                void* scales_row_blocked, void* q_col, void* scales_col_blocked,
                                                void* stream) {
  return launch_swiglu_fwd_quant(h1, num_rows, max_rows, F, clamped, alpha, limit, q_row, scales_row_blocked, q_col,
                                 scales_col_blocked, PlacedOffsets{}, stream);
}

extern "C" int dm_swiglu_fwd_quant_mxfp8_rowcol_at(dm_operand h1, const int32_t* num_rows, int64_t max_rows, int64_t F,
                                                   int clamped, float alpha, float limit, dm_operand q_row,
                                                   dm_operand sf_row, dm_operand q_col, dm_operand sf_col,
                                                   const int* cond, void* stream) {
  PlacedOffsets at{h1.offset, nullptr, q_col.offset, sf_col.offset, q_row.offset, sf_row.offset, cond, 1};
  return launch_swiglu_fwd_quant(h1.base, num_rows, max_rows, F, clamped, alpha, limit, q_row.base, sf_row.base,
                                 q_col.base, sf_col.base, at, stream);
}

static int launch_swiglu_bwd_quant(const void* h1, const void* grad_h2, const int32_t* num_rows, int64_t max_rows,
                                   int64_t F, int clamped, float alpha, float limit, void* q_row, void* sf_row,
                                   void* q_col, void* sf_col, PlacedOffsets at, void* stream) {
  if (!h1 || !grad_h2 || max_rows < 0 || F <= 0 || (F % 32) != 0) return kRcBadArg;
  if ((q_row == nullptr) != (sf_row == nullptr) || (q_col == nullptr) != (sf_col == nullptr) ||
      (q_row == nullptr && q_col == nullptr))
    return kRcBadArg;
  if (max_rows == 0) return kRcOk;
  constexpr int kSmem = 3 * kTileSlot * 16;
  static PerDeviceOnce attr_set;
  const int rc_attr = once_per_device(attr_set, [] {
    return static_cast<int>(
        cudaFuncSetAttribute(mxfp8_swiglu_bwd_colrow_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  });
  if (rc_attr != 0) return rc_attr;
  const int grid = tile_grid(max_rows, F, 2);
  const int col_atoms = static_cast<int>(((max_rows + 31) / 32 + 3) / 4);
  const int row_atoms = static_cast<int>((2 * F / 32 + 3) / 4);
  mxfp8_swiglu_bwd_colrow_kernel<<<grid, 256, kSmem, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(h1), static_cast<const uint4*>(grad_h2), ActParams{clamped, alpha, limit}, num_rows,
      max_rows, static_cast<int>(F), static_cast<uint8_t*>(q_col), static_cast<uint8_t*>(sf_col), col_atoms,
      static_cast<uint8_t*>(q_row), static_cast<uint8_t*>(sf_row), row_atoms, at);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int dm_swiglu_bwd_quant_mxfp8(const void* h1, const void* grad_h2, const int32_t* num_rows, int64_t max_rows,
                                        int64_t F, int clamped, float alpha, float limit, void* q_row,
                                        void* scales_row_blocked, void* q_col, void* scales_col_blocked, void* stream) {
  return launch_swiglu_bwd_quant(h1, grad_h2, num_rows, max_rows, F, clamped, alpha, limit, q_row, scales_row_blocked,
                                 q_col, scales_col_blocked, PlacedOffsets{}, stream);
}

extern "C" int dm_swiglu_bwd_quant_mxfp8_at(dm_operand h1, dm_operand grad_h2, const int32_t* num_rows,
                                           int64_t max_rows, int64_t F, int clamped, float alpha, float limit,
                                           dm_operand q_row, dm_operand sf_row, dm_operand q_col, dm_operand sf_col,
                                           void* stream) {
  PlacedOffsets at{h1.offset, grad_h2.offset, q_col.offset, sf_col.offset, q_row.offset, sf_row.offset, nullptr, 1};
  return launch_swiglu_bwd_quant(h1.base, grad_h2.base, num_rows, max_rows, F, clamped, alpha, limit, q_row.base,
                                 sf_row.base, q_col.base, sf_col.base, at, stream);
}

extern "C" int dm_quant_mxfp8_tile32(const void* w, int64_t experts, int64_t N, int64_t K, void* q, void* row_scales,
                                     void* col_scales, int blocked, void* stream) {
  if (!w || !q || !row_scales || experts <= 0 || N <= 0 || K <= 0 || (N % 32) != 0 || (K % 32) != 0) return kRcBadArg;
  const int64_t rows = experts * N;
  const uintptr_t all = reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(row_scales) |
                        reinterpret_cast<uintptr_t>(col_scales);
  if (blocked && col_scales && (N % 128) == 0 && (K % 128) == 0 && (all & 15) == 0 && (rows >> 7) * (K >> 7) < (1ll << 31)) {
    mxfp8_tile32_kernel<<<static_cast<unsigned>((rows >> 7) * (K >> 7)), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint4*>(w), N, static_cast<int>(K), static_cast<uint8_t*>(q), static_cast<uint8_t*>(row_scales),
        static_cast<uint8_t*>(col_scales));
    return static_cast<int>(cudaGetLastError());
  }
  const dim3 grid(static_cast<unsigned>((K + 255) / 256), static_cast<unsigned>(rows / 32));
  mxfp8_slab_kernel<true><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(w), nullptr, rows, static_cast<int>(K), static_cast<uint8_t*>(q),
      static_cast<uint8_t*>(row_scales), static_cast<uint8_t*>(col_scales), blocked,
      static_cast<int>((K / 32 + 3) / 4), static_cast<int>((N / 32 + 3) / 4), N);
  return static_cast<int>(cudaGetLastError());
}

static int nvfp4_token_impl(const IdPublish& ids, const int64_t* live, const void* x, const int32_t* num_rows, int64_t max_rows,
                            int64_t C, void* q, int64_t q_row_stride, void* scales, int64_t scale_row_stride,
                            int scales_blocked, void* scale_inv, int64_t inv_row_stride, void* stream) {
  if (!x || !q || !scales || max_rows < 0 || C <= 0 || (C % 16) != 0 || (q_row_stride % 4) != 0) return kRcBadArg;
  if (scale_inv && (inv_row_stride % 4) != 0) return kRcBadArg;
  if (max_rows == 0) return kRcOk;
  // Up to 2048 elements a warp holds the row, up to 8192 a CTA does (launched with as many blocks per thread as the row
  // needs); longer rows are read twice.
  const int blocks = static_cast<int>(C / 16);
  const int atoms = scales_blocked ? static_cast<int>((C / 16 + 3) / 4) : 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
#define DM_TOKEN(THREADS, BPT)                                                                                       \
  nvfp4_token_reg_kernel<THREADS, BPT><<<blocks_for(max_rows, 256 / THREADS, grid_cap(8)), 256, 0, st>>>(              \
      static_cast<const uint4*>(x), num_rows, max_rows, blocks, static_cast<uint8_t*>(q), q_row_stride,                \
      static_cast<uint8_t*>(scales), scale_row_stride, static_cast<uint8_t*>(scale_inv), inv_row_stride, atoms, live, ids)
  if (blocks <= 512) {
    if (blocks <= 32)
      DM_TOKEN(32, 1);
    else if (blocks <= 64)
      DM_TOKEN(32, 2);
    else if (blocks <= 128)
      DM_TOKEN(32, 4);
    else if (blocks <= 256)
      DM_TOKEN(256, 1);
    else
      DM_TOKEN(256, 2);
    return static_cast<int>(cudaGetLastError());
  }
#undef DM_TOKEN
  nvfp4_token_kernel<<<blocks_for(max_rows, 1, grid_cap(16)), 128, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(x), num_rows, max_rows, static_cast<int>(C / 8), static_cast<uint8_t*>(q),
      q_row_stride, static_cast<uint8_t*>(scales), scale_row_stride, static_cast<uint8_t*>(scale_inv),
      inv_row_stride, scales_blocked ? static_cast<int>((C / 16 + 3) / 4) : 0, live, ids);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int dm_quant_nvfp4_token(const void* x, const int32_t* num_rows, int64_t max_rows, int64_t C, void* q,
                                    int64_t q_row_stride, void* scales, int64_t scale_row_stride, int scales_blocked,
                                    void* scale_inv, int64_t inv_row_stride, void* stream) {
  return nvfp4_token_impl(IdPublish{}, nullptr, x, num_rows, max_rows, C, q, q_row_stride, scales, scale_row_stride, scales_blocked,
                          scale_inv, inv_row_stride, stream);
}

extern "C" int dm_quant_nvfp4_token_live(const int64_t* row_live, const void* x, const int32_t* num_rows,
                                         int64_t max_rows, int64_t C, void* q, int64_t q_row_stride, void* scales,
                                         int64_t scale_row_stride, int scales_blocked, void* scale_inv,
                                         int64_t inv_row_stride, void* stream) {
  if (!row_live) return kRcBadArg;
  return nvfp4_token_impl(IdPublish{}, row_live, x, num_rows, max_rows, C, q, q_row_stride, scales, scale_row_stride, scales_blocked,
                          scale_inv, inv_row_stride, stream);
}

extern "C" int dm_quant_nvfp4_weight(const void* w, const float* global_scale, int64_t experts, int64_t N, int64_t K,
                                     void* q, void* scales, int blocked, void* stream) {
  if (!w || !global_scale || !q || !scales || experts <= 0 || N <= 0 || K <= 0 || (K % 16) != 0) return kRcBadArg;
  const int vec = static_cast<int>(K / 8);
  nvfp4_weight_kernel<<<blocks_for(experts * N * vec, 256, grid_cap(16)), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(w), global_scale, N, experts * N, vec, static_cast<uint32_t*>(q),
      static_cast<uint8_t*>(scales), blocked, static_cast<int>((K / 16 + 3) / 4));
  return static_cast<int>(cudaGetLastError());
}

extern "C" int dm_sf_swizzle(const void* natural, void* blocked_out, int64_t rows, int64_t cols, void* stream) {
  if (!natural || !blocked_out || rows <= 0 || cols <= 0) return kRcBadArg;
  const int64_t padded_rows = (rows + 127) / 128 * 128;
  const int atoms = static_cast<int>((cols + 3) / 4);
  sf_swizzle_kernel<<<blocks_for(padded_rows * atoms * 4, 256, grid_cap(8)), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint8_t*>(natural), static_cast<uint8_t*>(blocked_out), rows, static_cast<int>(cols),
      padded_rows, atoms);
  return static_cast<int>(cudaGetLastError());
}

static int gather_packed_impl(int live_only, const int64_t* ptrs, const int32_t* num_rows, int64_t max_rows, int64_t q_bytes,
                              int64_t scale_cols, int has_inv, dm_operand q, dm_operand scales_blocked,
                              dm_operand scale_inv, const int* cond, void* stream) {
  if (!ptrs || !num_rows || !q.base || !scales_blocked.base || q_bytes <= 0 || (q_bytes % 16) != 0 || scale_cols <= 0 ||
      (scale_cols % 4) != 0 || max_rows < 0)
    return kRcBadArg;
  if (has_inv && !scale_inv.base) return kRcBadArg;
  if (max_rows == 0) return kRcOk;
  gather_packed_kernel<<<blocks_for(max_rows * ((q_bytes / 16 + 127) / 128), 8, grid_cap(8)), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      ptrs, num_rows, max_rows, static_cast<int>(q_bytes / 16), static_cast<int>(scale_cols), has_inv,
      static_cast<uint8_t*>(q.base), q.offset, static_cast<uint8_t*>(scales_blocked.base), scales_blocked.offset,
      static_cast<uint8_t*>(scale_inv.base), scale_inv.offset, cond, live_only);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int dm_gather_packed_rows(const int64_t* ptrs, const int32_t* num_rows, int64_t max_rows, int64_t q_bytes,
                                     int64_t scale_cols, int has_inv, dm_operand q, dm_operand scales_blocked,
                                     dm_operand scale_inv, const int* cond, void* stream) {
  return gather_packed_impl(0, ptrs, num_rows, max_rows, q_bytes, scale_cols, has_inv, q, scales_blocked, scale_inv, cond, stream);
}

extern "C" int dm_gather_packed_rows_live(const int64_t* ptrs, const int32_t* num_rows, int64_t max_rows, int64_t q_bytes,
                                          int64_t scale_cols, int has_inv, dm_operand q, dm_operand scales_blocked,
                                          dm_operand scale_inv, const int* cond, void* stream) {
  return gather_packed_impl(1, ptrs, num_rows, max_rows, q_bytes, scale_cols, has_inv, q, scales_blocked, scale_inv, cond, stream);
}

// What an inference call publishes, in one launch: its tokens quantised into the packed dispatch rows [q | natural scales |
// fp32 inverse scale (NVFP4)] and its expert ids.  The launch of the ids alone took 1.4 us and a gap.
extern "C" int dm_publish_quantised(int format, const void* x, const void* ids, int ids_are_int64, void* dispatch_local,
                                    int64_t row_stride, int64_t q_bytes, int64_t scale_bytes, void* routing_local, int64_t T,
                                    int64_t D, int K, int E, int validate, int* status, void* stream) {
  if (!x || !ids || !dispatch_local || !routing_local || T <= 0 || D <= 0 || K <= 0 || E <= 0 || E > 32767 ||
      (format != 0 && format != 1))
    return kRcBadArg;
  const IdPublish publish{ids, static_cast<uint8_t*>(routing_local), T * K, ids_are_int64, static_cast<int>(T), E, validate, status};
  uint8_t* rows = static_cast<uint8_t*>(dispatch_local);
  if (format == 0)
    return mxfp8_row_impl(publish, nullptr, x, nullptr, T, D, rows, row_stride, rows + q_bytes, row_stride, 0, stream);
  return nvfp4_token_impl(publish, nullptr, x, nullptr, T, D, rows, row_stride, rows + q_bytes, row_stride, 0,
                          rows + q_bytes + scale_bytes, row_stride, stream);
}
