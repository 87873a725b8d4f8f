// Persistent grouped MXFP8 GEMMs over routed rows on tcgen05: forward and input gradient.
//
//   fprop  C[r,n] = sum_k (X[r,k] * sfx[r,k/32]) * (W[e][n,k] * sfw[e][n,k/32])
//   dgrad  C[r,n] = sum_k (X[r,k] * sfx[r,k/32]) * (W[e][k,n] * sfw[e][n,k/32])      W N-major
//
// A pair of CTAs (cta_group::2) works on one tile: 256 output columns of the weights are the M side of the MMA (128 per CTA)
// and up to 256 routed rows its N side in steps of 32 (each CTA loads half of them), as in the BF16 kernel.  The accumulator
// holds C transposed (TMEM lane = output column, TMEM column = routed row).  Against 128 x 256 tiles of single CTAs with rows
// on the M side: a stage loads 32 KiB of operands instead of 48 (those tiles ran into 13 to 14 TB/s of L2 reads), and an
// expert pays for its rows rounded up to 32 instead of 128.  One B200, layers: training 8192 tokens, 128 experts x 4096 x 1536
// 7100 -> 6914 us; inference 128 x 2816 x 2816, 4096 tokens (128 rows per expert) 911 -> 859 us, and against the
// swapped-operand kernel below that: 16 tokens 244 -> 220, 256 tokens 580 -> 561; 32 x 4096 x 1536, 8 to 192 tokens 121 to 162
// -> 120 to 160 us.  Bound: power (1.55 GHz) and the epilogue, which takes about 1400 cycles per block of 32 rows next to
// 512 cycles per stage (a tile of W2 has twelve).
//
//   * a stage is 128 bytes of K per row;
//   * scales are stored in 128-row x 4-column atoms of 512 bytes (row r, column c at (r%32)*16 + (r/32)*4 + c), the source
//     shape of tcgen05.cp 32x128b.warpx4, which lands an atom in four TMEM columns of 32 rows each.  A CTA needs the atom of
//     its own 128 weight columns and those of all rows of the tile (at most two, see row_tiles.cuh).
//     A tile that starts at row 32 q of an atom names column q (0 or 2) as its scale address;
//   * the warp that issues the MMAs copies a stage's atoms right before them: copies and MMAs of one thread execute in order,
//     and the copies hide behind the MMAs before them (512 cycles a stage with and without);
//   * TMEM: scale columns of the stage slots at the top, two accumulators below them that overlap where 2 x rows do not fit.
//     The epilogue reads the shared columns first and hands them back, so only that read stands between two tiles.  Reading
//     all blocks before the arithmetic of the first made the plain forms 3 % slower (more registers per thread, spills).
//
// One CTA per SM, 384 threads: warp 0 loads weights, warp 11 rows, warp 1 issues (in the leading CTA), warps 2 to 9 are the
// epilogue (two per TMEM lane quadrant, each group of four takes every other block of 32 rows), warp 10 watches accumulators.
#include "gemm_common.cuh"
#include "quant_common.cuh"
#include "row_tiles.cuh"

namespace dm {

constexpr int kBrBM = 128;       // output columns per CTA of a pair
constexpr int kBrMaxStages = 10;
constexpr int kBrThreads = 384;
constexpr int kBrMaxGroups = 256;
constexpr uint32_t kBrWBytes = kBrBM * 128;   // 16 KiB
constexpr uint32_t kBrTmemCols = 512;
constexpr uint32_t kBrStagePlain = 32 * 256;  // per epilogue group: 32 rows x 128 columns
constexpr uint32_t kBrStageFused = 32 * 384;  // 32 rows x (64 gate, 64 up, 64 h2)
constexpr uint32_t kBrDynSmem = 227 * 1024 - 4096;  // the rest holds the tables and barriers

struct BrParams {
  CUtensorMap tm_w;
  CUtensorMap tm_x[kRwBoxes];  // routed rows, boxes of rw_box_rows(i) rows x 128 bytes
  CUtensorMap tm_sfw;          // scales as lines of 128 bytes, boxes of one atom
  CUtensorMap tm_sfx;          // the rows' scales as lines that overlap: they may start inside a line
  const int64_t* x_off;
  const int64_t* sfx_off;
  const int64_t* c_off;
  const int64_t* h2_off;
  const int64_t* row_inv_off;
  const uint8_t* row_inv_base;  // fp32 per row or null
  const float* expert_inv;      // fp32 per expert or null
  uint8_t* c_base;
  uint8_t* h2_base;
  const int64_t* scatter_ptrs;
  const int32_t* expert_offsets;
  const int32_t* expert_counts;  // real rows of every 128-padded group, or null: all of them
  const int* cond;
  int* status;
  int64_t sfw_group_lines;
  int e_local, max_rows, N, Kw, k_iters, x_col_atoms, w_col_atoms;
  // SwiGLU epilogue that writes h2 as MXFP8 rows (E4M3 bytes + blocked E8M0 scales) instead of bf16
  uint8_t* hq_base;
  const int64_t* hq_off;
  uint8_t* hsf_base;
  const int64_t* hsf_off;
  int h_atoms;
  ActParams act;
};

struct BrTile {
  int e, pair, row0, rows, n, last;  // rows: real rows of the tile, n: the MMA's N (rows rounded up to 32)
};

__device__ __forceinline__ BrTile br_decode(int tile, int& e, const int* tile_start, const int* off, const int* cnt,
                                            const uint16_t* rows_per_tile) {
  while (tile >= tile_start[e + 1]) ++e;
  const int local = tile - tile_start[e];
  const int nt = rw_row_tiles(cnt[e]), per = rows_per_tile[e];
  BrTile t;
  t.e = e;
  t.pair = local / nt;
  const int i = local - t.pair * nt;
  t.row0 = off[e] + i * per;
  const int left = cnt[e] - i * per;
  t.rows = left < per ? (left > 0 ? left : 0) : per;
  t.n = t.rows > 0 ? (t.rows + 31) & ~31 : 32;
  t.last = i == nt - 1;
  return t;
}

// Two neighbouring columns of one row from words of one column of two neighbouring rows (lanes 2p and 2p + 1).
__device__ __forceinline__ uint32_t br_pair(uint32_t w, int odd) {
  const uint32_t o = __shfl_xor_sync(0xffffffffu, w, 1);
  return __byte_perm(w, o, odd ? 0x3276 : 0x5410);
}

template <int kDgrad, bool kSwiglu, bool kPadRows>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kBrThreads, 1)
    blockscaled_rows_kernel(const __grid_constant__ BrParams p) {
  if (p.cond != nullptr && *p.cond == 0) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  __shared__ uint64_t full_bar[kBrMaxStages];
  __shared__ uint64_t empty_bar[kBrMaxStages];
  __shared__ uint64_t tmem_full_bar[2];
  __shared__ uint64_t tmem_empty_bar[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ volatile int s_first_bad;  // first of this CTA's tiles whose accumulator never came
  __shared__ uint32_t s_stop[3];        // where the weight producer, the row producer and the issuer stopped
  __shared__ int s_box;
  __shared__ int s_off[kBrMaxGroups + 1];
  __shared__ int s_cnt[kBrMaxGroups];
  __shared__ int s_tile_start[kBrMaxGroups + 1];
  __shared__ uint16_t s_per[kBrMaxGroups];

  constexpr uint32_t kStaging = kSwiglu ? kBrStageFused : kBrStagePlain;
  constexpr uint32_t kRing = kBrDynSmem - 1024 - 2 * kStaging;
  constexpr uint32_t kSfBytes = 512;  // a stage's atom of 128 rows
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int64_t x_off = p.x_off ? *p.x_off : 0, sfx_off = p.sfx_off ? *p.sfx_off : 0;  // on their way while the tables are built

  // ---- tile table ---------------------------------------------------------------------------------------------------
  const int m_pairs = (p.N + 2 * kBrBM - 1) / (2 * kBrBM);
  if (warp == 2) {
    if (lane < kBrMaxStages) {
      mbar_init(&full_bar[lane], 1);
      mbar_init(&empty_bar[lane], 1);
    }
    if (lane < 2) {
      mbar_init(&tmem_full_bar[lane], 1);
      mbar_init(&tmem_empty_bar[lane], 16);  // the leader's: eight epilogue warps of both CTAs
    }
    if (lane == 0) {
      abort_flag = 0;
      s_first_bad = kNoBadTile;
    }
    mbar_fence_init();
    __syncwarp();
  }
  cluster_arrive();  // this CTA's barriers exist
  if (warp == 1) {
    tmem_alloc_pair(&tmem_base_slot, kBrTmemCols);
    tmem_relinquish_pair();
  }
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&p.tm_w);
      tma_prefetch_desc(&p.tm_sfw);
      tma_prefetch_desc(&p.tm_sfx);
    }
    int box = 0;
    tile_tables(p.expert_offsets, p.expert_counts, p.e_local, p.max_rows, lane, s_off, s_tile_start,
                [&](int e, int lo, int hi, int count) {
      const int rows = bs_group_rows(lo, hi, count);
      s_cnt[e] = rows;
      if (count > 0 && hi > lo && !bs_group_aligned(lo))
        set_status(p.status, kCapacityExceeded, -1, e, lo);  // groups must be 128-padded
      const int nt = rw_row_tiles(rows), per = bs_rows_per_tile(rows);
      s_per[e] = static_cast<uint16_t>(per);
      if (nt > 0) box = max(box, rw_box_index(per));
      return nt * m_pairs;
    });
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) box = max(box, __shfl_xor_sync(0xffffffffu, box, d));
    if (lane == 0) s_box = box;
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_wait();  // both CTAs' barriers exist before either is signalled from the other
  tcgen05_fence_after();
  const uint32_t tmem_base = uniform(tmem_base_slot);
  const int total_tiles = uniform(s_tile_start[p.e_local]);
  // Ring: stages as large as the launch's largest tile needs, as many as shared memory and the scale columns allow.
  const int n_max = 2 * rw_box_rows(uniform(s_box));
  const uint32_t x_groups = bs_tile_atoms(n_max);
  // One B200, 2816 x 2816, all pairs | even rounds, us.  W13 with SwiGLU: 16 tokens on 47 of 128 experts 118.5 | 115.7, 4 rows per
  // expert on average 326.5 | 325.8, 16 327.5 | 327.9; 154 tiles (three rounds, the last with 6) 33.1 | 32.0, 242 43.0 | 40.3, but 132 (two,
  // the last with 58 of 74) 27.7 | 29.0, 198 34.8 | 36.0, 144 of 2048 x 768 25.5 | 26.4.  W2: 62.2 | 59.7, 169.5 | 166.5, 175.6 | 174.0; 66 to
  // 418 tiles 0.5 to 12 % less, 132 24.4 | 24.0, 198 32.2 | 30.9.  From tiles of 64 rows up the epilogues want all pairs: 32 rows on
  // average 343 / 171 | 346 / 172, 64 361 / 175 | 371 / 174, 96 388 / 181 | 397 / 178.
  const int pair = blockIdx.x >> 1;
  const int tile_step = balanced_pairs(total_tiles, gridDim.x >> 1, n_max, 32, kSwiglu);
  const int first_tile = pair < tile_step ? pair : total_tiles;
  // Scale columns of a stage slot: an atom of the weights and those of the rows, at a stride of 8 or 16.  With slots of twelve, all
  // that two atoms of rows need, the four forward and input-gradient launches of a training layer took 0.9 to 1.6 % longer.
  const uint32_t slot_cols = x_groups == 1 ? 8 : 16;
  const uint32_t sf_at = kBrWBytes + static_cast<uint32_t>(n_max / 2) * 128;  // weight atoms, then the rows' atoms
  const uint32_t stage_bytes = sf_at + (((1 + x_groups) * kSfBytes + 1023) & ~1023u);
  const int fit = static_cast<int>(kRing / stage_bytes);
  const int most = n_max <= 128 ? min(kBrMaxStages, static_cast<int>((kBrTmemCols - 2 * n_max) / slot_cols)) : 6;
  const int stages = fit < most ? fit : most;
  // Accumulators [0, n) and [acc1, acc1 + n); they share columns where acc1 < n_max.
  const int acc1 = static_cast<int>(kBrTmemCols - stages * slot_cols - n_max) & ~31;
  const bool shared_cols = acc1 < n_max;
  const uint32_t sf_tmem = tmem_base + kBrTmemCols - stages * slot_cols;

  if (warp == 0 || warp == 11) {
    // ======================= TMA producers: warp 0 the weights, warp 11 the rows =======================
    const bool rows_side = warp == 11;
    const bool elected = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    int e = 0;
    if (rows_side && lane == 0 && ((x_off & 127) | (sfx_off & 15)) != 0) set_status(p.status, kCapacityExceeded, -2, 0, 0);
    const int x_line0 = uniform(static_cast<int>(x_off >> 7)), sfx_line0 = uniform(static_cast<int>(sfx_off >> 7));
    const int sfx_x = uniform(static_cast<int>((sfx_off >> 4) & 7) * 4);  // word of its line that the scales start at
    constexpr int kSfLines = kSfBytes / 128;
    bool ok = true;
    const uint32_t lead_full = uniform(cluster_addr(smem_u32(&full_bar[0]), 0));
    for (int tile = first_tile; tile < total_tiles; tile += tile_step) {
      const BrTile t = br_decode(tile, e, s_tile_start, s_off, s_cnt, s_per);
      const int box = uniform(rw_box_index(t.n));
      const CUtensorMap* tm_x = &p.tm_x[box];
      const int atom0 = uniform(t.row0 >> 7);
      const int x_atoms = uniform(((t.row0 + t.n - 1) >> 7) - (t.row0 >> 7) + 1);
      const uint32_t tx = 2 * (kBrWBytes + static_cast<uint32_t>(rw_box_rows(box)) * 128 + (1 + x_atoms) * kSfBytes);  // both CTAs
      const int m_blk = uniform(2 * t.pair + static_cast<int>(rank));
      const int x_row = uniform(t.row0 + static_cast<int>(rank) * (t.n >> 1));
      const int expert = uniform(t.e);
      const int sfw_line = uniform(static_cast<int>(expert * p.sfw_group_lines) + m_blk * p.w_col_atoms * 4);
      const int sfx_line = uniform(sfx_line0 + atom0 * p.x_col_atoms * 4);
#pragma unroll 1
      for (int kb = 0; kb < p.k_iters; ++kb) {
        ok = warp_mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_flag);
        if (!ok) break;
        uint8_t* sw = smem + stage * stage_bytes;
        const uint32_t full = lead_full + stage * 8;
        if (elected) {
          if (rows_side) {
            tma_load_3d_pair(sw + kBrWBytes, tm_x, 0, x_line0 + kb, x_row, full);
            uint8_t* sf = sw + sf_at + kSfBytes;
            for (int a = 0; a < x_atoms; ++a)
              tma_load_2d_pair(sf + a * kSfBytes, &p.tm_sfx, sfx_x, sfx_line + a * p.x_col_atoms * 4 + kb * kSfLines, full);
          } else {
            if (rank == 0) mbar_arrive_expect_tx(&full_bar[stage], tx);
            if (kDgrad)
              tma_load_2d_pair(sw, &p.tm_w, m_blk * kBrBM, expert * p.Kw + kb * 128, full);
            else
              tma_load_2d_pair(sw, &p.tm_w, kb * 128, expert * p.N + m_blk * kBrBM, full);
            tma_load_2d_pair(sw + sf_at, &p.tm_sfw, 0, sfw_line + kb * kSfLines, full);
          }
        }
        __syncwarp();
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (!ok) break;
    }
    if (lane == 0) s_stop[rows_side ? 1 : 0] = ring_stop(stage, phase);
    __syncwarp();
  } else if (warp == 1) {
    // ======================= MMA issuer =======================
    if (rank == 0) {
      const bool elected = elect_one();
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO 1024, version 1, 128-byte swizzle
      constexpr uint32_t kLbo = (16u >> 4) << 16;
      constexpr uint32_t w_step = kDgrad ? 4096u >> 4 : 32u >> 4, x_step = 32u >> 4;
      const uint32_t ring = uniform(smem_u32(smem));
      const uint32_t full0 = uniform(smem_u32(&full_bar[0])), empty0 = uniform(smem_u32(&empty_bar[0]));
      const uint32_t tfull0 = uniform(smem_u32(&tmem_full_bar[0]));
      int stage = 0;
      uint32_t phase = 0, ready = 0;  // ready: the current stage is known to be full
      int e = 0, it = 0;
      bool ok = true;
      for (int tile = first_tile; tile < total_tiles; tile += tile_step, ++it) {
        const BrTile t = br_decode(tile, e, s_tile_start, s_off, s_cnt, s_per);
        const int n = uniform(t.n);
        const uint32_t q = uniform(static_cast<uint32_t>((t.row0 & 127) >> 5));  // the tile's first 32-row group in its atom
        const int x_atoms = uniform(((t.row0 + t.n - 1) >> 7) - (t.row0 >> 7) + 1);
        uint32_t idesc[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          idesc[j] = umma_idesc_blockscaled(n, 0, j, j, kDgrad, 0, 2 * kBrBM);
        const int buf = it & 1;
        const uint32_t d_tmem = tmem_base + (buf ? acc1 : 0);
        // Shared columns: the tile before has been read where the two overlap (and the one before that altogether).
        // Otherwise: the tile two before, in the same columns, has been read.
        if (shared_cols)
          ok = it == 0 || warp_mbar_wait(&tmem_empty_bar[0], (it - 1) & 1u, &abort_flag);
        else
          ok = warp_mbar_wait(&tmem_empty_bar[buf], ((it >> 1) & 1u) ^ 1u, &abort_flag);
        if (!ok) break;
        tcgen05_fence_after();
        uint32_t acc = 0;
#pragma unroll 1
        for (int kb = 0; kb < p.k_iters; ++kb) {
          if (!__all_sync(0xffffffffu, ready)) {
            ok = warp_mbar_wait(&full_bar[stage], phase, &abort_flag);
            if (!ok) break;
          }
          tcgen05_fence_after();
          const uint32_t w_addr = ring + stage * stage_bytes;
          const uint32_t w_lo = ((w_addr & 0x3ffffu) >> 4) | kLbo, x_lo = w_lo + (kBrWBytes >> 4);
          const uint32_t sf_lo = sf_desc_lo(w_addr + sf_at);
          const uint32_t sfw_t = sf_tmem + stage * slot_cols;
          const uint32_t sfx_t = sfw_t + 4u;
          const uint32_t empty = empty0 + stage * 8;
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
          ready = mbar_test(full0 + stage * 8, phase);
          if (elected) {
            tmem_cp_sf_lo_pair(sfw_t, sf_lo);
            tmem_cp_sf_lo_pair(sfx_t, sf_lo + kSfAtomWords);
            if (x_atoms > 1) tmem_cp_sf_lo_pair(sfx_t + 4, sf_lo + 2 * kSfAtomWords);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              umma_mxf8_lo_pair(d_tmem, w_lo + j * w_step, x_lo + j * x_step, kDescHi, idesc[j], sfw_t, sfx_t + q,
                                j > 0 ? 1u : acc);
            tcgen05_commit_pair(empty);
          }
          __syncwarp();
          acc = 1;
        }
        if (!ok) break;
        if (elected) tcgen05_commit_pair(tfull0 + buf * 8);
        __syncwarp();
      }
      if (lane == 0) s_stop[2] = ring_stop(stage, phase);
    }
    __syncwarp();
  } else if (warp == 10) {
    // ======================= accumulator watcher =======================
    // Polls the accumulator-ready barriers for the epilogue warps and releases them through a hardware named barrier;
    // after a timeout it releases them once more and stops.
    bool ok = true;
    int it = 0;
    for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step, ++it) {
      if (lane == 0) ok = handover_report(&s_first_bad, it, mbar_wait(&tmem_full_bar[it & 1], (it >> 1) & 1u, &abort_flag));
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      asm volatile("bar.arrive %0, %1;" ::"r"(handover_barrier(it)), "r"(8 * 32 + 32) : "memory");
    }
  } else {
    // ======================= epilogue =======================
    // Lane l of quadrant q holds output column 32 q + l (SwiGLU: W13 rows alternate 8 gate and 8 up, so lane l pairs with lane
    // l ^ 8 and a warp has 16 features).  Blocks of 32 rows (TMEM columns) go to the two groups in turn, those in columns that
    // the other accumulator shares first.  The staging tile is laid out row by row; the 16-byte chunks of a row are permuted
    // so that the words the 32 lanes write (two rows, and gate and up) fall into different banks.
    const int ew = warp - 2;
    const int quad = warp & 3;  // TMEM lanes [32 * quad, 32 * quad + 32)
    const int half = ew >> 2;
    uint8_t* stg = smem + kRing + half * kStaging;
    const int bar_id = 1 + kHandoverBarriers + half;
    const uint32_t lead_empty = cluster_addr(smem_u32(&tmem_empty_bar[0]), 0);
    const int odd = lane & 1;
    int e = 0, it = 0;
    bool ok = true;
    const int64_t c_off = p.c_off ? *p.c_off : 0;
    const int64_t h2_off = p.h2_off ? *p.h2_off : 0;
    const float* row_inv =
        p.row_inv_base ? reinterpret_cast<const float*>(p.row_inv_base + (p.row_inv_off ? *p.row_inv_off : 0)) : nullptr;
    const bool scaled = row_inv != nullptr || p.expert_inv != nullptr;
    const bool dense = p.scatter_ptrs == nullptr && p.c_base != nullptr;
    const int F = p.N / 2;
    for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step, ++it) {
      const BrTile t = br_decode(tile, e, s_tile_start, s_off, s_cnt, s_per);
      const int buf = it & 1;
      const int blocks = t.n >> 5;
      const int m_blk = 2 * t.pair + static_cast<int>(rank);
      const float escale = p.expert_inv ? p.expert_inv[t.e] : 1.0f;
      const int d_col = buf ? acc1 : 0;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + d_col;
      auto block_at = [&](int i) { return buf == 0 ? blocks - 1 - i : i; };
      // whether block i (in reading order) lies in columns that the other accumulator may use
      auto in_shared = [&](int i) {
        const int c = block_at(i) * 32;
        return buf == 0 ? c + 32 > acc1 : acc1 + c < n_max;
      };
      // row pointer of this lane's row of a block
      auto row_ptr = [&](int b) -> uint64_t {
        const int r = b * 32 + lane;
        if (kSwiglu ? p.c_base == nullptr : false) return 0;
        if (!kSwiglu && p.scatter_ptrs != nullptr) return r < t.rows ? static_cast<uint64_t>(p.scatter_ptrs[t.row0 + r]) : 0;
        // dense rows up to the next multiple of 32 are computed (padding rows hold zeros)
        if (!kSwiglu && !kPadRows && r >= t.rows) return 0;
        return reinterpret_cast<uint64_t>(p.c_base) + c_off + static_cast<uint64_t>(t.row0 + r) * p.N * 2;
      };
      auto row_scale = [&](int b) -> float { return row_inv != nullptr ? row_inv[t.row0 + b * 32 + lane] : 1.0f; };
      auto finish = [&](uint32_t (&v)[32], int b, uint64_t my_row, float my_scale) {
        if (scaled) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            v[i] = __float_as_uint((__uint_as_float(v[i]) * __shfl_sync(0xffffffffu, my_scale, i)) * escale);
        }
        uint32_t w[16];  // rows (2i, 2i + 1) of this lane's column
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = pack_bf16x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
        asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "r"(128) : "memory");  // the previous block has left the staging tile
        if (kSwiglu) {
          const int up = (lane >> 3) & 1;
          const int word = (((lane >> 4) << 3) | (lane & 7)) >> 1;
          uint32_t o[8], z[8];
          // the gate lane takes rows 0-15 of its feature, the up lane rows 16-31: each sends the half the other one needs
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = __shfl_xor_sync(0xffffffffu, up ? w[i] : w[8 + i], 8);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float gf[8], uf[8], zf[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t gw = up ? o[4 * h + i] : w[4 * h + i], uw = up ? w[8 + 4 * h + i] : o[4 * h + i];
              gf[2 * i] = __uint_as_float(gw << 16);
              gf[2 * i + 1] = __uint_as_float(gw & 0xffff0000u);
              uf[2 * i] = __uint_as_float(uw << 16);
              uf[2 * i + 1] = __uint_as_float(uw & 0xffff0000u);
            }
            swiglu_f32(gf, uf, zf, p.act);
#pragma unroll
            for (int i = 0; i < 4; ++i) z[4 * h + i] = pack_bf16x2(zf[2 * i], zf[2 * i + 1]);
          }
          const int chunk = 2 * quad + (word >> 2);
          if (p.c_base != nullptr) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int r = 2 * i + odd;
              *reinterpret_cast<uint32_t*>(stg + r * 384 + up * 128 + ((chunk ^ (odd << 2) ^ (up << 1)) << 4) + (word & 3) * 4) =
                  br_pair(w[i], odd);
            }
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = up * 16 + 2 * i + odd;
            *reinterpret_cast<uint32_t*>(stg + r * 384 + 256 + ((chunk ^ (odd << 2) ^ (up << 1)) << 4) + (word & 3) * 4) =
                br_pair(z[i], odd);
          }
        } else {
          const int word = lane >> 1;
          const int chunk = 4 * quad + (word >> 2);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int r = 2 * i + odd;
            *reinterpret_cast<uint32_t*>(stg + r * 256 + ((chunk ^ (odd << 2)) << 4) + (word & 3) * 4) = br_pair(w[i], odd);
          }
        }
        asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "r"(128) : "memory");
        if (kSwiglu && p.hq_base != nullptr) {
          // Four lanes per row, 16 features each, two lanes per 1 x 32 block: the bytes the row quantiser would produce from
          // the bf16 values in the staging tile.
          const int r = quad * 8 + (lane >> 2), c4 = lane & 3;
          const uint8_t* src = stg + r * 384 + 256;
          const int sw = ((r & 1) << 2) ^ ((r >> 4) << 1);
          const uint4 a = *reinterpret_cast<const uint4*>(src + (((2 * c4) ^ sw) << 4));
          const uint4 b4 = *reinterpret_cast<const uint4*>(src + (((2 * c4 + 1) ^ sw) << 4));
          const uint32_t zw[8] = {a.x, a.y, a.z, a.w, b4.x, b4.y, b4.z, b4.w};
          uint32_t m = 0;
#pragma unroll
          for (int j = 0; j < 8; ++j) m = __vmaxu2(m, zw[j] & 0x7fff7fffu);
          m = __vmaxu2(m, __shfl_xor_sync(0xffffffffu, m, 1));
          const uint32_t top = (m >> 16) > (m & 0xffffu) ? (m >> 16) : (m & 0xffffu);
          float recip;
          const uint8_t byte = mxfp8_scale(amax_from_bf16_bits(top), recip);
          uint32_t o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            o[j] = e4m3x4(__uint_as_float(zw[2 * j] << 16) * recip, __uint_as_float(zw[2 * j] & 0xffff0000u) * recip,
                          __uint_as_float(zw[2 * j + 1] << 16) * recip, __uint_as_float(zw[2 * j + 1] & 0xffff0000u) * recip);
          const int f = m_blk * 64 + 16 * c4;
          if (b * 32 + r < t.rows && f + 16 <= F) {
            const int64_t row = t.row0 + b * 32 + r;
            store_global16(reinterpret_cast<uint64_t>(p.hq_base) + (p.hq_off ? *p.hq_off : 0) + row * F + f, make_uint4(o[0], o[1], o[2], o[3]));
            if ((c4 & 1) == 0) (p.hsf_base + (p.hsf_off ? *p.hsf_off : 0))[blocked_offset(row, f >> 5, p.h_atoms)] = byte;
          }
        } else if (kSwiglu) {
          const int c = lane & 7, col = m_blk * 64 + c * 8;  // eight lanes per row and 128-byte piece
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int r = quad * 8 + i * 4 + (lane >> 3);
            const uint64_t h1 = __shfl_sync(0xffffffffu, my_row, r);
            if (b * 32 + r < t.rows && col + 8 <= F) {
              const uint8_t* src = stg + r * 384;
              const int sw = (r & 1) << 2;
              if (h1 != 0) {
                store_global16(h1 + static_cast<uint64_t>(col) * 2, *reinterpret_cast<const uint4*>(src + ((c ^ sw) << 4)));
                store_global16(h1 + static_cast<uint64_t>(F + col) * 2,
                               *reinterpret_cast<const uint4*>(src + 128 + ((c ^ sw ^ 2) << 4)));
              }
              store_global16(reinterpret_cast<uint64_t>(p.h2_base) + h2_off +
                                 (static_cast<uint64_t>(t.row0 + b * 32 + r) * F + col) * 2,
                             *reinterpret_cast<const uint4*>(src + 256 + ((c ^ sw ^ ((r >> 4) << 1)) << 4)));
            }
          }
        } else {
          const int c = lane & 15, col = m_blk * kBrBM + c * 8;  // sixteen lanes per row
          uint64_t rp[4];
          uint4 v16[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = quad * 8 + i * 2 + (lane >> 4);
            rp[i] = __shfl_sync(0xffffffffu, my_row, r);
            v16[i] = *reinterpret_cast<const uint4*>(stg + r * 256 + ((c ^ ((r & 1) << 2)) << 4));
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (rp[i] != 0 && col + 8 <= p.N) store_global16(rp[i] + static_cast<uint64_t>(col) * 2, v16[i]);
        }
      };
      uint64_t row_a = half < blocks ? row_ptr(block_at(half)) : 0;
      float scale_a = half < blocks ? row_scale(block_at(half)) : 1.0f;
      asm volatile("bar.sync %0, %1;" ::"r"(handover_barrier(it)), "r"(8 * 32 + 32) : "memory");  // released by the watcher
      ok = handover_good(&s_first_bad, it);  // the same for every epilogue warp
      if (!ok) break;
      tcgen05_fence_after();
      bool held = true;  // this warp has not yet handed the accumulator back
      auto hand_back = [&] {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(lead_empty + (shared_cols ? 0 : buf) * 8);
        held = false;
      };
      for (int i = half; i < blocks; i += 4) {
        const bool two = i + 2 < blocks;
        uint32_t va[32], vb[32];
        tmem_ld_32x32(taddr + block_at(i) * 32, va);
        uint64_t row_b = 0, row_n = 0;
        float scale_b = 1.0f, scale_n = 1.0f;
        if (two) {
          tmem_ld_32x32(taddr + block_at(i + 2) * 32, vb);
          row_b = row_ptr(block_at(i + 2));
          scale_b = row_scale(block_at(i + 2));
        }
        if (i + 4 < blocks) {
          row_n = row_ptr(block_at(i + 4));
          scale_n = row_scale(block_at(i + 4));
        }
        tmem_ld_wait();
        if (held && (i + 4 >= blocks || (shared_cols && !in_shared(i + 4)))) hand_back();
        finish(va, block_at(i), row_a, scale_a);
        if (two) finish(vb, block_at(i + 2), row_b, scale_b);
        row_a = row_n;
        scale_a = scale_n;
      }
      if (held) hand_back();
      if (!kSwiglu && kPadRows && dense && t.last) {
        // rows between the last multiple of 32 and the end of the padded group: zeros, as the product of their zero rows
        const int col = m_blk * kBrBM + (lane & 15) * 8;
        if (col + 8 <= p.N)
          for (int r = t.row0 + t.n + 2 * ew + (lane >> 4); r < s_off[t.e + 1]; r += 16)
            *reinterpret_cast<uint4*>(p.c_base + c_off + (static_cast<int64_t>(r) * p.N + col) * 2) = make_uint4(0, 0, 0, 0);
      }
    }
  }

  // ---- teardown ---------------------------------------------------------------
  tcgen05_fence_before();
  __syncthreads();
  if (abort_flag && rank == 0 && threadIdx.x == 0) {  // the leader's barriers count both CTAs' loads and MMAs
    const uint64_t deadline = globaltimer_ns() + kSettleNs;
    settle_ring(empty_bar, stages, s_stop[2], deadline);
    settle_ring(full_bar, stages, s_stop[0], deadline);
    settle_ring(full_bar, stages, s_stop[1], deadline);
  }
  __syncwarp();
  cluster_sync();  // neither CTA leaves while the other may still signal its barriers, or loads into either are in flight
  if (abort_flag && threadIdx.x == 0) set_status(p.status, kPipelineTimeout, 4, blockIdx.x);
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, kBrTmemCols);
  }
}

// gemm_nvfp4.cu
int nvfp4_forward(const dm_operand& a, const dm_operand& sfa, const void* w, const void* sfb, const dm_operand& c,
                  const dm_operand& h2, const int64_t* scatter_ptrs, const dm_operand& row_scale_inv,
                  const float* expert_scale_inv, const int32_t* expert_offsets, int e_local, int64_t max_rows, int64_t N,
                  int64_t Kd, int swiglu_interleaved, const ActParams& act, const int* cond, int num_sms, int* status,
                  cudaStream_t st);
int mxfp8_forward(const dm_operand& a, const dm_operand& sfa, const void* w, const void* sfb, const dm_operand& c,
                  const dm_operand& h2, const int64_t* scatter_ptrs, const dm_operand& row_scale_inv,
                  const float* expert_scale_inv, const int32_t* expert_offsets, const int32_t* expert_counts, int e_local,
                  int64_t max_rows, int64_t N, int64_t Kd, int swiglu_interleaved, const ActParams& act, bool pad_rows,
                  const int* cond, int num_sms, int* status, cudaStream_t st);

// kPadRows: rows of a dense C past an expert's count are written too.
template <int kDgrad, bool kSwiglu, bool kPadRows = true>
static int br_launch(const BrParams& p, int num_sms, cudaStream_t st) {
  static PerDeviceOnce attr_set;
  const int rc = once_per_device(attr_set, [] {
    return static_cast<int>(cudaFuncSetAttribute(blockscaled_rows_kernel<kDgrad, kSwiglu, kPadRows>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kBrDynSmem)));
  });
  if (rc != 0) return rc;
  blockscaled_rows_kernel<kDgrad, kSwiglu, kPadRows><<<pair_grid(num_sms), kBrThreads, kBrDynSmem, st>>>(p);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace dm

using namespace dm;

// What the three entry points share: operands, scales and the row table.
static int br_setup(BrParams& p, const dm_operand& x, const dm_operand& sfx, const void* sfw, int64_t row_bytes,
                    int64_t scale_cols, const int32_t* expert_offsets, const int32_t* expert_counts, int e_local,
                    int64_t max_rows, int64_t N, const int* cond, int* status) {
  for (int i = 0; i < kRwBoxes; ++i) {
    const int rc = encode_arena_u8(&p.tm_x[i], x, row_bytes, max_rows + 256, rw_box_rows(i));
    if (rc != kRcOk) return rc;
  }
  p.x_col_atoms = p.w_col_atoms = static_cast<int>((scale_cols + 3) / 4);
  p.sfw_group_lines = (N + 127) / 128 * static_cast<int64_t>(p.w_col_atoms) * 4;
  // An extent that does not even hold the layout was never told in earnest (entry points before this kernel did not read
  // it): the loads are then bounded by the rows alone, as they were.
  const int64_t layout_bytes = max_rows / 128 * static_cast<int64_t>(p.x_col_atoms) * 512;
  const int64_t sfx_bytes = sfx.bytes >= layout_bytes ? sfx.bytes : int64_t{1} << 37;
  int rc = encode_sf(&p.tm_sfx, sfx.base, sfx_bytes, true);
  if (rc != kRcOk) return rc;
  rc = encode_sf(&p.tm_sfw, sfw, e_local * p.sfw_group_lines * 128, false);
  if (rc != kRcOk) return rc;
  p.x_off = x.offset;
  p.sfx_off = sfx.offset;
  p.expert_offsets = expert_offsets;
  p.expert_counts = expert_counts;
  p.cond = cond;
  p.status = status;
  p.e_local = e_local;
  p.max_rows = static_cast<int>(max_rows);
  p.N = static_cast<int>(N);
  p.k_iters = static_cast<int>(row_bytes / 128);
  return kRcOk;
}

// The MXFP8 forward of dm_gemm_blockscaled and of dm_gemm_blockscaled_swapped (arguments checked there).
int dm::mxfp8_forward(const dm_operand& a, const dm_operand& sfa, const void* w, const void* sfb, const dm_operand& c,
                      const dm_operand& h2, const int64_t* scatter_ptrs, const dm_operand& row_scale_inv,
                      const float* expert_scale_inv, const int32_t* expert_offsets, const int32_t* expert_counts, int e_local,
                      int64_t max_rows, int64_t N, int64_t Kd, int swiglu_interleaved, const ActParams& act, bool pad_rows,
                      const int* cond, int num_sms, int* status, cudaStream_t st) {
  BrParams p{};
  int rc = br_setup(p, a, sfa, sfb, Kd, Kd / 32, expert_offsets, expert_counts, e_local, max_rows, N, cond, status);
  if (rc != kRcOk) return rc;
  rc = encode_2d_u8(&p.tm_w, w, static_cast<int64_t>(e_local) * N, Kd, kBrBM);
  if (rc != kRcOk) return rc;
  p.c_off = c.offset;
  p.h2_off = h2.offset;
  p.c_base = static_cast<uint8_t*>(c.base);
  p.h2_base = static_cast<uint8_t*>(h2.base);
  p.row_inv_base = static_cast<const uint8_t*>(row_scale_inv.base);
  p.row_inv_off = row_scale_inv.offset;
  p.expert_inv = expert_scale_inv;
  p.scatter_ptrs = scatter_ptrs;
  p.act = act;
  if (swiglu_interleaved) return br_launch<0, true>(p, num_sms, st);
  return pad_rows ? br_launch<0, false>(p, num_sms, st) : br_launch<0, false, false>(p, num_sms, st);
}

extern "C" int dm_gemm_blockscaled_counted(int format, dm_operand a, dm_operand sfa, const void* w, const void* sfb,
                                           dm_operand c, dm_operand h2, const int64_t* scatter_ptrs,
                                           dm_operand row_scale_inv, const float* expert_scale_inv,
                                           const int32_t* expert_offsets, const int32_t* expert_counts, int e_local,
                                           int64_t max_rows, int64_t N, int64_t Kd, int swiglu_interleaved, int clamped,
                                           float alpha, float limit, const int* cond, int num_sms, int* status,
                                           void* stream) {
  if (!a.base || !sfa.base || !w || !sfb || !expert_offsets || e_local <= 0 || max_rows < 0 || N <= 0 || Kd <= 0)
    return kRcBadArg;
  if (format != 0 && format != 1) return kRcBadArg;
  if (!swiglu_interleaved && !c.base && !scatter_ptrs) return kRcBadArg;
  if (swiglu_interleaved && (!h2.base || scatter_ptrs)) return kRcBadArg;
  if (e_local > kBrMaxGroups || max_rows > (1 << 30)) return kRcTooLarge;
  const int fp4 = format == 1;
  const int64_t row_bytes = fp4 ? Kd / 2 : Kd;
  if ((row_bytes % 128) != 0 || (N % 128) != 0 || (max_rows % 128) != 0) return kRcUnsupportedShape;
  if (max_rows == 0) return kRcOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (fp4)
    return nvfp4_forward(a, sfa, w, sfb, c, h2, scatter_ptrs, row_scale_inv, expert_scale_inv, expert_offsets, e_local, max_rows,
                         N, Kd, swiglu_interleaved, ActParams{clamped, alpha, limit}, cond, num_sms, status, st);
  return mxfp8_forward(a, sfa, w, sfb, c, h2, scatter_ptrs, row_scale_inv, expert_scale_inv, expert_offsets, expert_counts,
                       e_local, max_rows, N, Kd, swiglu_interleaved, ActParams{clamped, alpha, limit}, true, cond, num_sms,
                       status, st);
}

extern "C" int dm_gemm_blockscaled(int format, dm_operand a, dm_operand sfa, const void* w, const void* sfb,
                                   dm_operand c, dm_operand h2, const int64_t* scatter_ptrs, dm_operand row_scale_inv,
                                   const float* expert_scale_inv, const int32_t* expert_offsets, int e_local,
                                   int64_t max_rows, int64_t N, int64_t Kd, int swiglu_interleaved, int clamped,
                                   float alpha, float limit, const int* cond, int num_sms, int* status, void* stream) {
  return dm_gemm_blockscaled_counted(format, a, sfa, w, sfb, c, h2, scatter_ptrs, row_scale_inv, expert_scale_inv,
                                     expert_offsets, nullptr, e_local, max_rows, N, Kd, swiglu_interleaved, clamped, alpha,
                                     limit, cond, num_sms, status, stream);
}

// MXFP8 forward W13 GEMM whose SwiGLU epilogue writes h2 already row-quantised (the operand of the W2 GEMM).
extern "C" int dm_gemm_blockscaled_swiglu_mxfp8_counted(dm_operand a, dm_operand sfa, const void* w, const void* sfb,
                                                        dm_operand h2_q, dm_operand h2_sf, const int32_t* expert_offsets,
                                                        const int32_t* expert_counts, int e_local, int64_t max_rows,
                                                        int64_t N, int64_t Kd, int clamped, float alpha, float limit,
                                                        const int* cond, int num_sms, int* status, void* stream) {
  if (!a.base || !sfa.base || !w || !sfb || !h2_q.base || !h2_sf.base || !expert_offsets || e_local <= 0 ||
      max_rows < 0 || N <= 0 || Kd <= 0)
    return kRcBadArg;
  if (e_local > kBrMaxGroups || max_rows > (1 << 30)) return kRcTooLarge;
  if ((Kd % 128) != 0 || (N % 128) != 0 || (max_rows % 128) != 0 || ((N / 2) % 32) != 0) return kRcUnsupportedShape;
  if (max_rows == 0) return kRcOk;
  BrParams p{};
  int rc = br_setup(p, a, sfa, sfb, Kd, Kd / 32, expert_offsets, expert_counts, e_local, max_rows, N, cond, status);
  if (rc != kRcOk) return rc;
  rc = encode_2d_u8(&p.tm_w, w, static_cast<int64_t>(e_local) * N, Kd, kBrBM);
  if (rc != kRcOk) return rc;
  p.hq_base = static_cast<uint8_t*>(h2_q.base);
  p.hq_off = h2_q.offset;
  p.hsf_base = static_cast<uint8_t*>(h2_sf.base);
  p.hsf_off = h2_sf.offset;
  p.h_atoms = static_cast<int>((N / 2 / 32 + 3) / 4);
  p.act = ActParams{clamped, alpha, limit};
  return br_launch<0, true>(p, num_sms, static_cast<cudaStream_t>(stream));
}

extern "C" int dm_gemm_blockscaled_swiglu_mxfp8(dm_operand a, dm_operand sfa, const void* w, const void* sfb,
                                                dm_operand h2_q, dm_operand h2_sf, const int32_t* expert_offsets,
                                                int e_local, int64_t max_rows, int64_t N, int64_t Kd, int clamped,
                                                float alpha, float limit, const int* cond, int num_sms, int* status,
                                                void* stream) {
  return dm_gemm_blockscaled_swiglu_mxfp8_counted(a, sfa, w, sfb, h2_q, h2_sf, expert_offsets, nullptr, e_local, max_rows, N,
                                                  Kd, clamped, alpha, limit, cond, num_sms, status, stream);
}

// Input gradient: W is the same E4M3 qdata as in the forward ([E, Kd, N] bytes, 32x32-tile quantised) read N-major, with the
// scales of the transposed orientation ([N rows, Kd/32 columns] per expert, blocked).
extern "C" int dm_gemm_blockscaled_dgrad_counted(dm_operand dy, dm_operand sf_dy, const void* w, const void* sfb_dgrad,
                                                 dm_operand c, const int64_t* scatter_ptrs, const int32_t* expert_offsets,
                                                 const int32_t* expert_counts, int e_local, int64_t max_rows, int64_t N,
                                                 int64_t Kd, const int* cond, int num_sms, int* status, void* stream) {
  if (!dy.base || !sf_dy.base || !w || !sfb_dgrad || !expert_offsets || e_local <= 0 || max_rows < 0 || N <= 0 || Kd <= 0)
    return kRcBadArg;
  if (!c.base && !scatter_ptrs) return kRcBadArg;
  if (e_local > kBrMaxGroups || max_rows > (1 << 30)) return kRcTooLarge;
  if ((Kd % 128) != 0 || (N % 128) != 0 || (max_rows % 128) != 0) return kRcUnsupportedShape;
  if (max_rows == 0) return kRcOk;
  BrParams p{};
  int rc = br_setup(p, dy, sf_dy, sfb_dgrad, Kd, Kd / 32, expert_offsets, expert_counts, e_local, max_rows, N, cond, status);
  if (rc != kRcOk) return rc;
  rc = encode_2d_u8(&p.tm_w, w, static_cast<int64_t>(e_local) * Kd, N, 128);
  if (rc != kRcOk) return rc;
  p.c_off = c.offset;
  p.c_base = static_cast<uint8_t*>(c.base);
  p.scatter_ptrs = scatter_ptrs;
  p.Kw = static_cast<int>(Kd);
  p.act = ActParams{0, 1.0f, 0.0f};
  return br_launch<1, false>(p, num_sms, static_cast<cudaStream_t>(stream));
}

extern "C" int dm_gemm_blockscaled_dgrad(dm_operand dy, dm_operand sf_dy, const void* w, const void* sfb_dgrad,
                                         dm_operand c, const int64_t* scatter_ptrs, const int32_t* expert_offsets,
                                         int e_local, int64_t max_rows, int64_t N, int64_t Kd, const int* cond,
                                         int num_sms, int* status, void* stream) {
  return dm_gemm_blockscaled_dgrad_counted(dy, sf_dy, w, sfb_dgrad, c, scatter_ptrs, expert_offsets, nullptr, e_local,
                                           max_rows, N, Kd, cond, num_sms, status, stream);
}
