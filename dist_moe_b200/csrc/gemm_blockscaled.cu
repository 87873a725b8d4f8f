// Persistent grouped MXFP8 weight-gradient GEMM on tcgen05 with scale factors in TMEM.
//
//   dW[e][m, n] (+)= sum_{r in expert e}  (dY[r,m] * sfdy[m, r/32]) * (X[r,n] * sfx[n, r/32])
//
// Same warp-specialised skeleton as the BF16 kernels (TMA producer warp, MMA-issuing warp, eight epilogue warps, one
// 128 x 256 fp32 accumulator in TMEM).  Both operands are MN-major: column-quantised rows, K = the expert's rows.
//   * a pipeline stage is 128 rows of K;
//   * next to the operand tiles the producer bulk-copies the stage's scale atoms.  Scales are stored in 128-row x 4-column
//     atoms of 512 bytes (row r, column c at (r%32)*16 + (r/32)*4 + c), which is exactly the 32-row x 16-byte source shape of
//     tcgen05.cp ... 32x128b.warpx4, so an atom goes to TMEM with one instruction and no shuffling;
//   * per K step of 32 the MMA names the scale byte inside the TMEM columns (a_sf_id / b_sf_id);
//   * rows of every expert are padded to 128 by the routing step, so K stages and scale atoms align.
#include "gemm_common.cuh"

namespace dm {

constexpr int kBsBM = 128;
constexpr uint32_t kBsABytes = kBsBM * 128;  // 16 KiB
constexpr uint32_t kBsTmemCols = 512;
constexpr int kBsMaxGroups = 256;

struct BsParams {
  CUtensorMap tm_a;
  CUtensorMap tm_b;
  CUtensorMap tm_c;  // dW as [e_local][rows][cols], boxes of 16 rows x 128 bytes
  const int64_t* a_off;
  const int64_t* b_off;
  const int64_t* sfa_off;
  const int64_t* sfb_off;
  const uint8_t* sfa_base;
  const uint8_t* sfb;
  const int32_t* expert_offsets;
  const int* cond;
  int* status;
  int e_local, max_rows, N, a_col_atoms, b_col_atoms, compact_cols;
  int Kw;  // dW columns (N: its rows)
  int out_fp32, accumulate;
};

struct BsTile {
  int e, m_blk, n_blk, row0, k_iters;
};

__device__ __forceinline__ BsTile bs_decode(int tile, int& e, const int* tile_start, const int* off, int n_tiles) {
  while (tile >= tile_start[e + 1]) ++e;
  const int local = tile - tile_start[e];
  BsTile t;
  t.e = e;
  t.n_blk = local % n_tiles;
  t.m_blk = local / n_tiles;
  t.row0 = off[e];
  t.k_iters = (off[e + 1] - off[e] + 127) / 128;
  return t;
}

// 128 x 256 output tiles.  Per 128 rows of K the tile moves 48 KiB of operands for four MMAs of 128 cycles.  With few rows per
// expert the epilogue bounds it: it takes 6900 cycles a tile and waits 25 of them for an accumulator; staging, proxy fences and
// the copy engine's reads (2100 cycles) are its time, the adding into dW (4.3 to 4.7 TB/s of HBM) is behind them.  685 and
// 1486 us for the W2 and W13 gradients of 128 experts, 73 728 rows, D = 4096, F = 1536.  TMEM holds one 256-column accumulator
// plus the scale columns of the stage slots: the epilogue warps read it into registers and hand it back before they convert and
// store, so only that read stands between a tile's last MMA and the next tile's first.
constexpr int kWdBN = 256;
constexpr int kWdThreads = 352;  // TMA warp, MMA warp, eight epilogue warps, accumulator watcher
constexpr uint32_t kWdBBytes = kWdBN * 128;                            // 32 KiB
constexpr uint32_t kWdSfBytes = 512;                                   // a scale atom
constexpr uint32_t kWdStageBytes = kBsABytes + kWdBBytes + 2048;       // 50 KiB: 1 + 2 scale atoms, padded
constexpr int kWdStages = 4;
constexpr uint32_t kWdSfTmemBase = kWdBN;  // scale columns: 16 per stage slot after the accumulator
static_assert(kWdSfTmemBase + kWdStages * 16 <= kBsTmemCols, "scale columns do not fit");
constexpr size_t kWdSmem = kWdStages * kWdStageBytes + 8 * kStaging64Bytes + 1024;

__global__ void __launch_bounds__(kWdThreads, 1) blockscaled_wide_kernel(const __grid_constant__ BsParams p) {
  if (p.cond != nullptr && *p.cond == 0) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  __shared__ uint64_t full_bar[kWdStages];
  __shared__ uint64_t empty_bar[kWdStages];
  __shared__ uint64_t tmem_full_bar;
  __shared__ uint64_t tmem_empty_bar;
  __shared__ uint32_t tmem_base_slot;
  __shared__ uint32_t s_stop[2];  // where the producer and the issuer stopped
  __shared__ int abort_flag;
  __shared__ volatile int s_first_bad;  // first of this CTA's tiles whose accumulator never came
  __shared__ int s_off[kBsMaxGroups + 1];
  __shared__ int s_tile_start[kBsMaxGroups + 1];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_tiles = (p.Kw + kWdBN - 1) / kWdBN;
  const int m_tiles = (p.N + kBsBM - 1) / kBsBM;

  for (int i = threadIdx.x; i <= p.e_local; i += blockDim.x) {
    const int v = min(p.expert_offsets[i], p.max_rows);
    s_off[i] = v;
    if (i < p.e_local && (v & 127) != 0) set_status(p.status, kCapacityExceeded, -1, i, v);  // rows must be 128-padded
  }
  if (threadIdx.x == 0) {
    abort_flag = 0;
    s_first_bad = kNoBadTile;
    for (int s = 0; s < kWdStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&tmem_full_bar, 1);
    mbar_init(&tmem_empty_bar, 8);
    mbar_fence_init();
  }
  for (int e = threadIdx.x; e <= p.e_local; e += blockDim.x) s_tile_start[e] = e * m_tiles * n_tiles;
  if (warp == 1) {
    tmem_alloc(&tmem_base_slot, kBsTmemCols);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&p.tm_a);
    tma_prefetch_desc(&p.tm_b);
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = uniform(tmem_base_slot);
  const int total_tiles = uniform(s_tile_start[p.e_local]);
  const uint32_t ring = uniform(smem_u32(smem));

  if (warp == 0) {
    // ======================= producer =======================
    {
      const bool elected = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      int e = 0;
      const int a_line0 = static_cast<int>((p.a_off ? *p.a_off : 0) >> 7);
      const int b_line0 = static_cast<int>((p.b_off ? *p.b_off : 0) >> 7);
      const uint8_t* sfa = p.sfa_base + (p.sfa_off ? *p.sfa_off : 0);
      const uint8_t* sfb = p.sfb + (p.sfb_off ? *p.sfb_off : 0);
      const int col_blocks = (p.Kw + 127) >> 7;  // 128-wide blocks of the B side
      int a_col_atoms = p.a_col_atoms, b_col_atoms = p.b_col_atoms;
      // column bundles sized by the device row count: their scale layout has rows/128 column atoms
      if (p.compact_cols) a_col_atoms = b_col_atoms = ((s_off[p.e_local] + 31) / 32 + 3) / 4;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        const BsTile t = bs_decode(tile, e, s_tile_start, s_off, n_tiles);
        // scales of the column-quantised operands: rows = features, columns = 32-row blocks of the packed rows
        const uint8_t* sfa_row = sfa + (static_cast<int64_t>(t.m_blk) * a_col_atoms + (t.row0 >> 7)) * 512;
        const uint8_t* sfb_row0 = sfb + (static_cast<int64_t>(t.n_blk * 2) * b_col_atoms + (t.row0 >> 7)) * 512;
        const uint8_t* sfb_row1 = sfb_row0 + static_cast<int64_t>(b_col_atoms) * 512;
        const bool second = uniform(t.n_blk * 2 + 1 < col_blocks ? 1 : 0) != 0;  // the tile's upper 128 columns exist
        const int t_k = uniform(t.k_iters), t_m = uniform(t.m_blk), t_n = uniform(t.n_blk), t_row = uniform(t.row0);
#pragma unroll 1
        for (int kb = 0; kb < t_k; ++kb) {
          ok = warp_mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_flag);
          if (!ok) break;
          uint8_t* sa = smem + stage * kWdStageBytes;
          uint8_t* sb = sa + kBsABytes;
          uint8_t* ssa = sb + kWdBBytes;
          uint8_t* ssb = ssa + kWdSfBytes;
          if (elected) {
            // B arrives as two 128-byte-wide boxes of 128 K rows; the upper one only where it exists
            mbar_arrive_expect_tx(&full_bar[stage], kBsABytes + (second ? kWdBBytes + 3 * kWdSfBytes : kWdBBytes / 2 + 2 * kWdSfBytes));
            tma_load_3d(sa, &p.tm_a, 0, a_line0 + t_m, t_row + kb * 128, &full_bar[stage]);
            tma_load_3d(sb, &p.tm_b, 0, b_line0 + t_n * 2, t_row + kb * 128, &full_bar[stage]);
            if (second) tma_load_3d(sb + kWdBBytes / 2, &p.tm_b, 0, b_line0 + t_n * 2 + 1, t_row + kb * 128, &full_bar[stage]);
            bulk_load(ssa, sfa_row + static_cast<int64_t>(kb) * kWdSfBytes, kWdSfBytes, &full_bar[stage]);
            bulk_load(ssb, sfb_row0 + static_cast<int64_t>(kb) * kWdSfBytes, kWdSfBytes, &full_bar[stage]);
            if (second) bulk_load(ssb + kWdSfBytes, sfb_row1 + static_cast<int64_t>(kb) * kWdSfBytes, kWdSfBytes, &full_bar[stage]);
          }
          __syncwarp();
          if (++stage == kWdStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (lane == 0) s_stop[0] = ring_stop(stage, phase);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ======================= MMA issuer =======================
    // The scale atoms of a stage are copied to the stage slot's TMEM columns by the warp that issues the MMAs, right before
    // them: copies and MMAs of one thread execute in order, so no barrier stands between them, and the copies run while
    // the MMAs issued before them occupy the pipe.  Columns: the A atom, then the B atoms of the tile's lower and upper 128
    // columns.  The slot's previous MMAs are complete by then: the producer refilled the stage only after their commit.
    {
      const bool elected = elect_one();
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO 1024, version 1, 128-byte swizzle
      constexpr uint32_t kStep = 4096u >> 4;  // 32 rows of K
      constexpr uint32_t kALbo = (16u >> 4) << 16, kBLbo = ((kWdBBytes / 2) >> 4) << 16;  // B's 128-byte-wide halves are 16 KiB apart
      const uint32_t full0 = uniform(smem_u32(&full_bar[0])), empty0 = uniform(smem_u32(&empty_bar[0]));
      const uint32_t tfull = uniform(smem_u32(&tmem_full_bar));
      int stage = 0;
      uint32_t phase = 0, ready = 0;  // ready: the current stage is known to be there
      int e = 0, it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++it) {
        const BsTile t = bs_decode(tile, e, s_tile_start, s_off, n_tiles);
        const int k_iters = uniform(t.k_iters);
        ok = warp_mbar_wait(&tmem_empty_bar, (it & 1u) ^ 1u, &abort_flag);  // the epilogue has drained the accumulator
        if (!ok) break;
        tcgen05_fence_after();
#pragma unroll 1
        for (int kb = 0; kb < k_iters; ++kb) {
          if (!__all_sync(0xffffffffu, ready)) {
            ok = warp_mbar_wait(&full_bar[stage], phase, &abort_flag);
            if (!ok) break;
          }
          tcgen05_fence_after();
          const uint32_t a_addr = ring + stage * kWdStageBytes;
          const uint32_t a_lo = ((a_addr & 0x3ffffu) >> 4) | kALbo, b_lo = (((a_addr + kBsABytes) & 0x3ffffu) >> 4) | kBLbo;
          const uint32_t sf_lo = sf_desc_lo(a_addr + kBsABytes + kWdBBytes);
          const uint32_t sfa_t = tmem_base + kWdSfTmemBase + stage * 16u;
          const uint32_t sfb_t = sfa_t + 4u;
          const uint32_t empty = empty0 + stage * 8;
          if (++stage == kWdStages) {
            stage = 0;
            phase ^= 1u;
          }
          ready = mbar_test(full0 + stage * 8, phase);
          if (elected) {
            tmem_cp_sf_lo(sfa_t, sf_lo);
            tmem_cp_sf_lo(sfb_t, sf_lo + kSfAtomWords);
            tmem_cp_sf_lo(sfb_t + 4, sf_lo + 2 * kSfAtomWords);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              umma_mxf8_lo(tmem_base, a_lo + j * kStep, b_lo + j * kStep, kDescHi, umma_idesc_blockscaled(kWdBN, 0, j, j, 1, 1),
                           sfa_t, sfb_t, (kb > 0 || j > 0) ? 1u : 0u);
            tcgen05_commit_addr(empty);
          }
          __syncwarp();
        }
        if (!ok) break;
        if (elected) {
          if (k_iters > 0)
            tcgen05_commit_addr(tfull);
          else
            mbar_arrive(&tmem_full_bar);
        }
        __syncwarp();
      }
      if (lane == 0) s_stop[1] = ring_stop(stage, phase);
    }
    __syncwarp();
  } else if (warp == 10) {
    // ======================= accumulator watcher =======================
    // Polls the accumulator-ready barrier for the epilogue warps and releases them through a hardware named barrier;
    // after a timeout it releases them once more and stops.
    bool ok = true;
    int it = 0;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++it) {
      if (lane == 0) ok = handover_report(&s_first_bad, it, mbar_wait(&tmem_full_bar, it & 1u, &abort_flag));
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      asm volatile("bar.arrive %0, %1;" ::"r"(handover_barrier(it)), "r"(8 * 32 + 32) : "memory");
    }
  } else {
    // ======================= epilogue =======================
    // Eight warps: two per TMEM lane quadrant, each owning 128 of the tile's 256 columns.  A lane reads its own
    // accumulator row; dW is overwritten or added to (fp32 or bf16) by the copy engine.
    const int ew = warp - 2;
    const int quad = warp & 3;
    const int half = ew >> 2;
    uint8_t* stg = smem + kWdStages * kWdStageBytes + ew * kStaging64Bytes;
    int e = 0, it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++it) {
      const BsTile t = bs_decode(tile, e, s_tile_start, s_off, n_tiles);
      asm volatile("bar.sync %0, %1;" ::"r"(handover_barrier(it)), "r"(8 * 32 + 32) : "memory");  // released by the watcher
      ok = handover_good(&s_first_bad, it);  // the same for every epilogue warp
      if (!ok) break;
      tcgen05_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
      uint32_t ra[32], rb[32], rc[32], rd[32];
      if (t.k_iters > 0) {
        tmem_ld_32x32(taddr + half * (kWdBN / 2), ra);
        tmem_ld_32x32(taddr + half * (kWdBN / 2) + 32, rb);
        tmem_ld_32x32(taddr + half * (kWdBN / 2) + 64, rc);
        tmem_ld_32x32(taddr + half * (kWdBN / 2) + 96, rd);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) ra[j] = rb[j] = rc[j] = rd[j] = 0u;
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty_bar);  // accumulator handed back before the stores
      // 128 bytes of output columns per trip (64 bf16 or 32 fp32).  The staging tile is laid out as a 16-row x
      // 128-byte box in the 128-byte swizzle, so the warp's 32 rows go in two passes; one thread hands each box
      // to the copy engine, which stores it or adds it to dW in L2 in whole 128-byte lines and clips rows and
      // columns past the matrix.
      const int col0 = t.n_blk * kWdBN + half * (kWdBN / 2);
      auto send = [&](int cc, int pass) {
        fence_proxy_async_smem();
        __syncwarp();
        const int box_row = t.m_blk * kBsBM + quad * 32 + pass * 16;
        if (lane == 0 && box_row < p.N && cc < p.Kw) {
          if (p.accumulate)
            tma_reduce_add_3d(&p.tm_c, stg, cc, box_row, t.e);
          else
            tma_store_3d(&p.tm_c, stg, cc, box_row, t.e);
          bulk_commit();
        }
      };
      if (p.out_fp32) {
#pragma unroll
        for (int trip = 0; trip < 4; ++trip) {
          uint32_t (&r)[32] = trip == 0 ? ra : (trip == 1 ? rb : (trip == 2 ? rc : rd));
#pragma unroll
          for (int pass = 0; pass < 2; ++pass) {
            if (lane == 0) bulk_wait_read();  // the engine has read the previous box out of the staging tile
            __syncwarp();
            if ((lane >> 4) == pass) {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                stage_put(stg, lane & 15, j, make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]));
            }
            send(col0 + 32 * trip, pass);
          }
        }
      } else {
#pragma unroll
        for (int trip = 0; trip < 2; ++trip) {
          uint32_t (&r0)[32] = trip == 0 ? ra : rc;
          uint32_t (&r1)[32] = trip == 0 ? rb : rd;
#pragma unroll
          for (int pass = 0; pass < 2; ++pass) {
            if (lane == 0) bulk_wait_read();
            __syncwarp();
            if ((lane >> 4) == pass) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                stage_put(stg, lane & 15, j, pack8_bf16(r0 + 8 * j));
                stage_put(stg, lane & 15, j + 4, pack8_bf16(r1 + 8 * j));
              }
            }
            send(col0 + 64 * trip, pass);
          }
        }
      }
    }
    if (lane == 0) bulk_wait_all();  // weight gradient: staged boxes are out of shared memory and written
  }

  tcgen05_fence_before();
  __syncthreads();
  if (abort_flag) {
    if (threadIdx.x == 0) {
      set_status(p.status, kPipelineTimeout, 4, blockIdx.x);
      const uint64_t deadline = globaltimer_ns() + kSettleNs;
      settle_ring(empty_bar, kWdStages, s_stop[1], deadline);
      settle_ring(full_bar, kWdStages, s_stop[0], deadline);
    }
    __syncthreads();
  }
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, kBsTmemCols);
  }
}

}  // namespace dm

using namespace dm;

// Launches the 128 x 256 kernel.
static int bs_launch(const BsParams& p, int num_sms, cudaStream_t st) {
  const int grid = persistent_grid(num_sms);
  static PerDeviceOnce wide_attr_set;
  const int rc = once_per_device(wide_attr_set, [] {
    return static_cast<int>(cudaFuncSetAttribute(blockscaled_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(kWdSmem)));
  });
  if (rc != 0) return rc;
  blockscaled_wide_kernel<<<grid, kWdThreads, kWdSmem, st>>>(p);
  return static_cast<int>(cudaGetLastError());
}

// Weight gradient: dW[e][m, n] (+)= sum_{r in expert e} dY[r, m] * X[r, n].  Both operands are quantised
// along the row dimension (32 rows share a scale, per column); their scales are blocked with the
// feature as the row index and the 32-row block as the column index.
static int blockscaled_wgrad(dm_operand dy_col, dm_operand sf_dy_col, dm_operand x_col, dm_operand sf_x_col, void* dw,
                             int dw_is_fp32, int accumulate, const int32_t* expert_offsets, int e_local,
                             int64_t max_rows, int64_t M, int64_t N, const int* cond, int num_sms, int* status,
                             void* stream, int compact_cols) {
  if (!dy_col.base || !sf_dy_col.base || !x_col.base || !sf_x_col.base || !dw || !expert_offsets || e_local <= 0 ||
      max_rows < 0 || M <= 0 || N <= 0)
    return kRcBadArg;
  if (e_local > kBsMaxGroups || max_rows > (1 << 30)) return kRcTooLarge;
  if ((M % 128) != 0 || (N % 128) != 0 || (max_rows % 128) != 0) return kRcUnsupportedShape;
  BsParams p{};
  int rc = kRcOk;
  // with no rows at all the kernel still runs so that a non-accumulating call zero-fills dW
  const int64_t rows_extent = max_rows > 0 ? max_rows : 128;
  rc = encode_arena_u8(&p.tm_a, dy_col, M, rows_extent, 128);
  if (rc != kRcOk) return rc;
  rc = encode_arena_u8(&p.tm_b, x_col, N, rows_extent, 128);
  if (rc != kRcOk) return rc;
  p.a_col_atoms = static_cast<int>(((max_rows + 31) / 32 + 3) / 4);
  p.b_col_atoms = p.a_col_atoms;
  p.a_off = dy_col.offset;
  p.b_off = x_col.offset;
  p.sfa_off = sf_dy_col.offset;
  p.sfb_off = sf_x_col.offset;
  p.sfa_base = static_cast<const uint8_t*>(sf_dy_col.base);
  p.sfb = static_cast<const uint8_t*>(sf_x_col.base);
  rc = encode_out_3d(&p.tm_c, dw, e_local, M, N, dw_is_fp32 != 0);
  if (rc != kRcOk) return rc;
  p.expert_offsets = expert_offsets;
  p.cond = cond;
  p.status = status;
  p.e_local = e_local;
  p.max_rows = static_cast<int>(max_rows);
  p.N = static_cast<int>(M);
  p.Kw = static_cast<int>(N);
  p.compact_cols = compact_cols;
  p.out_fp32 = dw_is_fp32 ? 1 : 0;
  p.accumulate = accumulate ? 1 : 0;
  return bs_launch(p, num_sms, static_cast<cudaStream_t>(stream));
}

extern "C" int dm_gemm_blockscaled_wgrad(dm_operand dy_col, dm_operand sf_dy_col, dm_operand x_col, dm_operand sf_x_col,
                                         void* dw, int dw_is_fp32, int accumulate, const int32_t* expert_offsets,
                                         int e_local, int64_t max_rows, int64_t M, int64_t N, const int* cond,
                                         int num_sms, int* status, void* stream) {
  return blockscaled_wgrad(dy_col, sf_dy_col, x_col, sf_x_col, dw, dw_is_fp32, accumulate, expert_offsets, e_local,
                           max_rows, M, N, cond, num_sms, status, stream, 0);
}

// The same product for column bundles whose scale layout was sized by the device row count
// (expert_offsets[e_local] rows, as the *_at quantisers write them) instead of by max_rows.
extern "C" int dm_gemm_blockscaled_wgrad_compact(dm_operand dy_col, dm_operand sf_dy_col, dm_operand x_col,
                                                 dm_operand sf_x_col, void* dw, int dw_is_fp32, int accumulate,
                                                 const int32_t* expert_offsets, int e_local, int64_t max_rows,
                                                 int64_t M, int64_t N, const int* cond, int num_sms, int* status,
                                                 void* stream) {
  return blockscaled_wgrad(dy_col, sf_dy_col, x_col, sf_x_col, dw, dw_is_fp32, accumulate, expert_offsets, e_local,
                           max_rows, M, N, cond, num_sms, status, stream, 1);
}
