// Persistent grouped NVFP4 forward GEMM on tcgen05 with scale factors in TMEM, for experts with many rows.
//
//   C[r, n] = sum_k  (A[r,k] * sfa[r, k/16]) * (W[e][n,k] * sfb[e][n, k/16])
//
// Same warp-specialised skeleton as the BF16 kernels (TMA producer warp, MMA-issuing warp, eight epilogue warps, one
// 128 x 256 fp32 accumulator in TMEM).  Differences:
//   * a pipeline stage is 128 bytes of K per row: 256 packed E2M1 elements;
//   * next to the A/B tiles the producer bulk-copies the stage's scale atoms.  Scales are stored in 128-row x 4-column atoms
//     of 512 bytes (row r, column c at (r%32)*16 + (r/32)*4 + c), which is exactly the 32-row x 16-byte source shape of
//     tcgen05.cp ... 32x128b.warpx4, so an atom goes to TMEM with one instruction and no shuffling: one atom per K = 64 step;
//   * rows of every expert are padded to 128 by the routing step, so tiles and scale atoms align.
//
// Epilogues: plain bf16 rows (optionally scaled by the per-token and per-expert NVFP4 inverse scales, optionally scattered to
// per-row destinations), or SwiGLU over a W13 whose rows were interleaved in groups of 8 gate / 8 up rows at preparation
// time, producing bf16 h2 (and h1).
#include "gemm_common.cuh"
#include "row_tiles.cuh"

namespace dm {

constexpr int kN4BM = 128;
constexpr int kN4BN = 256;
constexpr uint32_t kN4ABytes = kN4BM * 128;  // 16 KiB
constexpr uint32_t kN4BBytes = kN4BN * 128;  // 32 KiB
constexpr uint32_t kN4SfBytes = 4 * 512;     // a stage's atoms of 128 rows
constexpr uint32_t kN4TmemCols = 512;
constexpr int kN4MaxGroups = 256;

struct N4Params {
  CUtensorMap tm_a;
  CUtensorMap tm_b;
  CUtensorMap tm_sfa;  // scales as lines of 128 bytes, boxes of a stage's four atoms
  CUtensorMap tm_sfb;
  const int64_t* a_off;
  const int64_t* sfa_off;
  const int64_t* c_off;
  const int64_t* h2_off;
  const int64_t* row_inv_off;
  const uint8_t* sfa_base;
  const uint8_t* sfb;
  const uint8_t* row_inv_base;  // fp32 per row (token scale inverse) or null
  const float* expert_inv;      // fp32 per expert (weight global scale inverse) or null
  uint8_t* c_base;
  uint8_t* h2_base;
  const int64_t* scatter_ptrs;
  const int32_t* expert_offsets;
  const int32_t* expert_counts;  // real rows of every 128-padded group, or null: all of them
  const int* cond;
  int* status;
  int64_t sfb_group_bytes;
  int e_local, max_rows, N, k_iters, swiglu, col_atoms;
  int direct_store;  // SwiGLU forward without staging tiles (four stages)
  ActParams act;
};

struct N4Tile {
  int e, n_blk, row0, row_end;
};

__device__ __forceinline__ N4Tile n4_decode(int tile, int& e, const int* tile_start, const int* off) {
  while (tile >= tile_start[e + 1]) ++e;
  const int local = tile - tile_start[e];
  const int m_tiles = (off[e + 1] - off[e] + kN4BM - 1) / kN4BM;
  N4Tile t;
  t.e = e;
  t.n_blk = local / m_tiles;
  t.row0 = off[e] + (local - t.n_blk * m_tiles) * kN4BM;
  t.row_end = off[e + 1];
  return t;
}

// 128 x 256 output tiles.  Per 128 bytes of K the tile moves 48 KiB of operands and 6 KiB of scales and needs twelve
// scale-atom copies (16 cycles each, hidden behind the MMAs) and four 128-cycle MMAs.  TMEM holds one 256-column accumulator
// plus the scale columns of every stage slot: the epilogue warps read it into registers and hand it back before they
// convert and store, so only that read stands between a tile's last MMA and the next tile's first.  Bound: operand loads from
// L2, 14 TB/s.  32 experts, 65 536 rows, D = 7168, F = 2048: 1976 us a layer; the kernel that puts rows on the MMA's N side
// over pairs of CTAs (gemm_blockscaled_rows.cu, MXFP8) loads a third less but took 2187 to 2233 us where these tiles took
// 2004, its epilogue of 2 x 256 rows against eight stages of W2.  Experts with few rows take the swapped-operand kernel instead.
constexpr int kN4Threads = 352;  // TMA warp, MMA warp, eight epilogue warps, accumulator watcher
constexpr uint32_t kN4Stage = kN4ABytes + kN4BBytes + 3 * kN4SfBytes;  // 54 KiB
constexpr int kN4Stages = 3;
constexpr uint32_t kN4SfTmemBase = kN4BN;  // scale columns: 64 per stage slot after the accumulator
constexpr size_t kN4Smem = kN4Stages * kN4Stage + 8 * kStaging64Bytes + 1024;
// With the SwiGLU epilogue and no h1 output every lane stores its own 64 bytes of h2 per block straight from registers, the
// staging tiles go, and a fourth stage fits.  Three 54 KiB stages do not cover the load latency; the stores of this form
// are less coalesced but run while the next tile's MMAs do.
constexpr int kN4StagesDirect = 4;
constexpr size_t kN4SmemDirect = kN4StagesDirect * kN4Stage + 1024;
static_assert(kN4SfTmemBase + kN4StagesDirect * 64 <= kN4TmemCols, "scale columns do not fit");
static_assert(kN4SmemDirect >= kN4Smem, "largest shared-memory request");

__global__ void __launch_bounds__(kN4Threads, 1) nvfp4_wide_kernel(const __grid_constant__ N4Params p) {
  if (p.cond != nullptr && *p.cond == 0) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  __shared__ uint64_t full_bar[kN4StagesDirect];
  __shared__ uint64_t empty_bar[kN4StagesDirect];
  __shared__ uint64_t tmem_full_bar;
  __shared__ uint64_t tmem_empty_bar;
  __shared__ uint32_t tmem_base_slot;
  __shared__ uint32_t s_stop[2];  // where the producer and the issuer stopped
  __shared__ int abort_flag;
  __shared__ volatile int s_first_bad;  // first of this CTA's tiles whose accumulator never came
  __shared__ int s_off[kN4MaxGroups + 1];
  __shared__ int s_tile_start[kN4MaxGroups + 1];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_tiles = (p.N + kN4BN - 1) / kN4BN;
  const int stages = p.direct_store ? kN4StagesDirect : kN4Stages;

  for (int i = threadIdx.x; i <= p.e_local; i += blockDim.x) {
    const int v = p.expert_offsets[i];
    s_off[i] = v < p.max_rows ? v : p.max_rows;
  }
  if (threadIdx.x == 0) {
    abort_flag = 0;
    s_first_bad = kNoBadTile;
    for (int s = 0; s < kN4StagesDirect; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&tmem_full_bar, 1);
    mbar_init(&tmem_empty_bar, 8);
    mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int e = 0; e < p.e_local; ++e) {
      s_tile_start[e] = acc;
      const int rows = s_off[e + 1] - s_off[e];
      if ((s_off[e] & 127) != 0) set_status(p.status, kCapacityExceeded, -1, e, s_off[e]);  // rows must be 128-padded
      acc += ((rows + kN4BM - 1) / kN4BM) * n_tiles;
    }
    s_tile_start[p.e_local] = acc;
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_slot, kN4TmemCols);
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
      const uint8_t* sfa = p.sfa_base + (p.sfa_off ? *p.sfa_off : 0);
      const int col_blocks = (p.N + 127) >> 7;  // 128-wide blocks of the B side
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        const N4Tile t = n4_decode(tile, e, s_tile_start, s_off);
        const uint8_t* sfa_row = sfa + static_cast<int64_t>(t.row0 >> 7) * p.col_atoms * 512;
        const uint8_t* sfb_row0 = p.sfb + t.e * p.sfb_group_bytes + static_cast<int64_t>(t.n_blk * 2) * p.col_atoms * 512;
        const uint8_t* sfb_row1 = sfb_row0 + static_cast<int64_t>(p.col_atoms) * 512;
        const bool second = uniform(t.n_blk * 2 + 1 < col_blocks ? 1 : 0) != 0;  // the tile's upper 128 columns exist
        const int t_e = uniform(t.e), t_n = uniform(t.n_blk), t_row = uniform(t.row0);
#pragma unroll 1
        for (int kb = 0; kb < p.k_iters; ++kb) {
          ok = warp_mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_flag);
          if (!ok) break;
          uint8_t* sa = smem + stage * kN4Stage;
          uint8_t* sb = sa + kN4ABytes;
          uint8_t* ssa = sb + kN4BBytes;
          uint8_t* ssb = ssa + kN4SfBytes;
          if (elected) {
            mbar_arrive_expect_tx(&full_bar[stage], kN4ABytes + kN4BBytes + (second ? 3 : 2) * kN4SfBytes);
            tma_load_3d(sa, &p.tm_a, 0, a_line0 + kb, t_row, &full_bar[stage]);
            tma_load_2d(sb, &p.tm_b, kb * 128, t_e * p.N + t_n * kN4BN, &full_bar[stage]);
            bulk_load(ssa, sfa_row + static_cast<int64_t>(kb) * kN4SfBytes, kN4SfBytes, &full_bar[stage]);
            bulk_load(ssb, sfb_row0 + static_cast<int64_t>(kb) * kN4SfBytes, kN4SfBytes, &full_bar[stage]);
            if (second) bulk_load(ssb + kN4SfBytes, sfb_row1 + static_cast<int64_t>(kb) * kN4SfBytes, kN4SfBytes, &full_bar[stage]);
          }
          __syncwarp();
          if (++stage == stages) {
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
    // the MMAs issued before them occupy the pipe (twelve copies and four MMAs of N = 256: 512 cycles, as long as the
    // MMAs alone; from other warps a copy took 54 cycles).  Columns: A atom a (K step a) at +4a; B atoms of the tile's lower
    // and upper 128 columns side by side, 8 columns per K step.  The slot's previous MMAs are complete by then: the
    // producer refilled the stage only after their commit released it.
    {
      const bool elected = elect_one();
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO 1024, version 1, 128-byte swizzle
      constexpr uint32_t kStep = 32u >> 4, kLbo = (16u >> 4) << 16;
      constexpr uint32_t idesc = umma_idesc_blockscaled(kN4BN, 1, 0, 0);
      const uint32_t full0 = uniform(smem_u32(&full_bar[0])), empty0 = uniform(smem_u32(&empty_bar[0]));
      const uint32_t tfull = uniform(smem_u32(&tmem_full_bar));
      int stage = 0;
      uint32_t phase = 0, ready = 0;  // ready: the current stage is known to be there
      int it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++it) {
        ok = warp_mbar_wait(&tmem_empty_bar, (it & 1u) ^ 1u, &abort_flag);  // the epilogue has drained the accumulator
        if (!ok) break;
        tcgen05_fence_after();
#pragma unroll 1
        for (int kb = 0; kb < p.k_iters; ++kb) {
          if (!__all_sync(0xffffffffu, ready)) {
            ok = warp_mbar_wait(&full_bar[stage], phase, &abort_flag);
            if (!ok) break;
          }
          tcgen05_fence_after();
          const uint32_t a_addr = ring + stage * kN4Stage;
          const uint32_t a_lo = ((a_addr & 0x3ffffu) >> 4) | kLbo, b_lo = (((a_addr + kN4ABytes) & 0x3ffffu) >> 4) | kLbo;
          const uint32_t sf_lo = sf_desc_lo(a_addr + kN4ABytes + kN4BBytes);
          const uint32_t sfa_t = tmem_base + kN4SfTmemBase + stage * 64u;
          const uint32_t sfb_t = sfa_t + 16u;
          const uint32_t empty = empty0 + stage * 8;
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
          ready = mbar_test(full0 + stage * 8, phase);
          if (elected) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              tmem_cp_sf_lo(sfa_t + 4 * j, sf_lo + j * kSfAtomWords);
              tmem_cp_sf_lo(sfb_t + 8 * j, sf_lo + (4 + j) * kSfAtomWords);
              tmem_cp_sf_lo(sfb_t + 8 * j + 4, sf_lo + (8 + j) * kSfAtomWords);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
              umma_nvf4_lo(tmem_base, a_lo + j * kStep, b_lo + j * kStep, kDescHi, idesc, sfa_t + 4 * j, sfb_t + 8 * j,
                           (kb > 0 || j > 0) ? 1u : 0u);
            tcgen05_commit_addr(empty);
          }
          __syncwarp();
        }
        if (!ok) break;
        if (elected) tcgen05_commit_addr(tfull);
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
    // accumulator row; the warp transposes 32 x 32 blocks through its staging tile and stores 64-byte row segments.
    const int ew = warp - 2;
    const int quad = warp & 3;
    const int half = ew >> 2;
    const int row_in_tile = quad * 32 + lane;
    uint8_t* stg = smem + stages * kN4Stage + ew * kStaging64Bytes;
    int e = 0, it = 0;
    bool ok = true;
    const int64_t c_off = p.c_off ? *p.c_off : 0;
    const int64_t h2_off = p.h2_off ? *p.h2_off : 0;
    const float* row_inv =
        p.row_inv_base ? reinterpret_cast<const float*>(p.row_inv_base + (p.row_inv_off ? *p.row_inv_off : 0)) : nullptr;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++it) {
      const N4Tile t = n4_decode(tile, e, s_tile_start, s_off);
      asm volatile("bar.sync %0, %1;" ::"r"(handover_barrier(it)), "r"(8 * 32 + 32) : "memory");  // released by the watcher
      ok = handover_good(&s_first_bad, it);  // the same for every epilogue warp
      if (!ok) break;
      tcgen05_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
      const int row = t.row0 + row_in_tile;
      const bool row_ok = row < t.row_end;
      float scale = 1.0f;
      bool scaled = false;
      if (row_inv != nullptr && row_ok) {
        scale = row_inv[row];
        scaled = true;
      }
      const float escale = p.expert_inv ? p.expert_inv[t.e] : 1.0f;
      scaled = scaled || p.expert_inv != nullptr;
      if (p.swiglu) {
        // Columns come in groups of 16: 8 gate features then the matching 8 up features.
        const int F = p.N / 2;
        const uint64_t my_h2 =
            row_ok ? reinterpret_cast<uint64_t>(p.h2_base) + h2_off + static_cast<uint64_t>(row) * F * 2 : 0ull;
        const uint64_t my_h1 = (row_ok && p.c_base)
                                   ? reinterpret_cast<uint64_t>(p.c_base) + c_off + static_cast<uint64_t>(row) * p.N * 2
                                   : 0ull;
        // Drain this warp's 128 columns into registers and hand the accumulator back at once: the SwiGLU
        // arithmetic and the stores below then run while the next tile's MMAs fill the accumulator again.
        uint32_t ra[32], rb[32], rc[32], rd[32];
        tmem_ld_32x32(taddr + half * (kN4BN / 2), ra);
        tmem_ld_32x32(taddr + half * (kN4BN / 2) + 32, rb);
        tmem_ld_32x32(taddr + half * (kN4BN / 2) + 64, rc);
        tmem_ld_32x32(taddr + half * (kN4BN / 2) + 96, rd);
        tmem_ld_wait();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty_bar);
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
          const int c0 = half * (kN4BN / 2) + 64 * blk;
          uint32_t (&r0)[32] = blk == 0 ? ra : rc;
          uint32_t (&r1)[32] = blk == 0 ? rb : rd;
          uint4 zv[4], gv[4], uv[4];
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint32_t gw[4], uw[4];
            float gf[8], uf[8], zf[8];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int b = 16 * (g & 1) + 2 * q;
              float g0 = __uint_as_float(g < 2 ? r0[b] : r1[b]), g1 = __uint_as_float(g < 2 ? r0[b + 1] : r1[b + 1]);
              float u0 = __uint_as_float(g < 2 ? r0[b + 8] : r1[b + 8]), u1 = __uint_as_float(g < 2 ? r0[b + 9] : r1[b + 9]);
              if (scaled) {
                g0 = (g0 * scale) * escale; g1 = (g1 * scale) * escale;
                u0 = (u0 * scale) * escale; u1 = (u1 * scale) * escale;
              }
              gw[q] = pack_bf16x2(g0, g1);
              uw[q] = pack_bf16x2(u0, u1);
              gf[2 * q] = __uint_as_float(gw[q] << 16);
              gf[2 * q + 1] = __uint_as_float(gw[q] & 0xffff0000u);
              uf[2 * q] = __uint_as_float(uw[q] << 16);
              uf[2 * q + 1] = __uint_as_float(uw[q] & 0xffff0000u);
            }
            swiglu_f32(gf, uf, zf, p.act);
            zv[g] = make_uint4(pack_bf16x2(zf[0], zf[1]), pack_bf16x2(zf[2], zf[3]), pack_bf16x2(zf[4], zf[5]), pack_bf16x2(zf[6], zf[7]));
            gv[g] = make_uint4(gw[0], gw[1], gw[2], gw[3]);
            uv[g] = make_uint4(uw[0], uw[1], uw[2], uw[3]);
          }
          const int f0 = t.n_blk * (kN4BN / 2) + c0 / 2;  // first of the 32 features of this block
          if (p.direct_store) {
            if (my_h2 != 0) {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (f0 + 8 * j + 8 <= F) *reinterpret_cast<uint4*>(my_h2 + static_cast<uint64_t>(f0 + 8 * j) * 2) = zv[j];
            }
            continue;
          }
#pragma unroll
          for (int which = 0; which < 3; ++which) {
            if (which > 0 && p.c_base == nullptr) break;
#pragma unroll
            for (int j = 0; j < 4; ++j) stage64_put(stg, lane, j, which == 0 ? zv[j] : (which == 1 ? gv[j] : uv[j]));
            __syncwarp();
            const uint64_t base = which == 0 ? my_h2 : my_h1;
            const int col_out = which == 2 ? F + f0 : f0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int rr = i * 8 + (lane >> 2), j = lane & 3;
              const uint4 v = stage64_get(stg, rr, j);
              const uint64_t rp = __shfl_sync(0xffffffffu, base, rr);
              if (rp != 0 && f0 + 8 * j + 8 <= F)
                *reinterpret_cast<uint4*>(rp + static_cast<uint64_t>(col_out + 8 * j) * 2) = v;
            }
            __syncwarp();
          }
        }
      } else {
        uint64_t my_row = 0;
        if (row_ok) {
          if (p.scatter_ptrs != nullptr)
            my_row = static_cast<uint64_t>(p.scatter_ptrs[row]);
          else
            my_row = reinterpret_cast<uint64_t>(p.c_base) + c_off + static_cast<uint64_t>(row) * p.N * 2;
        }
        uint32_t ra[32], rb[32], rc[32], rd[32];
        tmem_ld_32x32(taddr + half * (kN4BN / 2), ra);
        tmem_ld_32x32(taddr + half * (kN4BN / 2) + 32, rb);
        tmem_ld_32x32(taddr + half * (kN4BN / 2) + 64, rc);
        tmem_ld_32x32(taddr + half * (kN4BN / 2) + 96, rd);
        tmem_ld_wait();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty_bar);  // accumulator handed back, see above
#pragma unroll
        for (int blk = 0; blk < 4; ++blk) {
          const int c0 = half * (kN4BN / 2) + 32 * blk;
          uint32_t (&r)[32] = blk == 0 ? ra : (blk == 1 ? rb : (blk == 2 ? rc : rd));
          if (scaled) {
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint((__uint_as_float(r[j]) * scale) * escale);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) stage64_put(stg, lane, j, pack8_bf16(r + 8 * j));
          __syncwarp();
          const int col = t.n_blk * kN4BN + c0;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int rr = i * 8 + (lane >> 2), j = lane & 3;
            const uint4 v = stage64_get(stg, rr, j);
            const uint64_t rp = __shfl_sync(0xffffffffu, my_row, rr);
            if (rp != 0 && col + 8 * j + 8 <= p.N)
              *reinterpret_cast<uint4*>(rp + static_cast<uint64_t>(col + 8 * j) * 2) = v;
          }
          __syncwarp();
        }
      }
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (abort_flag) {
    if (threadIdx.x == 0) {
      set_status(p.status, kPipelineTimeout, 4, blockIdx.x);
      const uint64_t deadline = globaltimer_ns() + kSettleNs;
      settle_ring(empty_bar, stages, s_stop[1], deadline);
      settle_ring(full_bar, stages, s_stop[0], deadline);
    }
    __syncthreads();
  }
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, kN4TmemCols);
  }
}

// 256 x 256 output tiles on CTA pairs (cta_group::2), for experts with hundreds of rows: each CTA has 128 rows on its M side
// and loads half of the tile's 256 weight columns, 38 KiB per stage where the kernel above loads 54 for the same MMAs (scales:
// its own rows' and all columns').  Five stages fit next to staging tiles for sixteen epilogue warps of 64 columns each:
// with eight of 128 the latency of their arithmetic held the SwiGLU form back (8 stages of K: 13 us a tile, now 6).  Rows past
// an expert's count are left out: a CTA without rows loads its peer's and stores nothing.
// One B200, 32 experts x 7168 x 2048, 2048 rows each: W13 with SwiGLU 807 -> 745 us; the plain form takes 569 us for W2 (K = 2048)
// where the kernel above takes 565, and wins from there on (K = 4096, 8 experts: 78 -> 66).  Bound: operand loads (W13 without the
// epilogue 684 us, without the loads of A and B 596) and the hand-over of the one accumulator, about 2000 cycles a tile; a second
// one does not fit next to the scales.  16 rows x 128 bytes per store instead of 32 x 64 cost W2 another 30 us.
constexpr int kN4PairEpilogue = 16;   // epilogue warps
constexpr int kN4PairThreads = (3 + kN4PairEpilogue) * 32;  // and TMA warp, MMA warp, accumulator watcher
constexpr uint32_t kN4PairBBytes = 128 * 128;  // a CTA loads half of the tile's weight columns
constexpr uint32_t kN4PairStage = kN4ABytes + kN4PairBBytes + 3 * kN4SfBytes;  // 38 KiB
constexpr int kN4PairStages = 5;
constexpr uint32_t kN4PairSfCols = 48;  // scale columns per stage slot after the accumulator: 16 of A, 32 of B
constexpr size_t kN4PairSmem = kN4PairStages * kN4PairStage + kN4PairEpilogue * kStaging64Bytes + 1024;
static_assert(kN4BN + kN4PairStages * kN4PairSfCols <= kN4TmemCols, "scale columns do not fit");

__device__ __forceinline__ N4Tile n4_pair_decode(int tile, int& e, const int* tile_start, const int* off, const int* rows) {
  while (tile >= tile_start[e + 1]) ++e;
  const int local = tile - tile_start[e];
  const int m_tiles = (rows[e] + 2 * kN4BM - 1) / (2 * kN4BM);
  N4Tile t;
  t.e = e;
  t.n_blk = local / m_tiles;
  t.row0 = off[e] + (local - t.n_blk * m_tiles) * 2 * kN4BM;
  t.row_end = off[e] + rows[e];
  return t;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kN4PairThreads, 1)
    nvfp4_pair_kernel(const __grid_constant__ N4Params p) {
  if (p.cond != nullptr && *p.cond == 0) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  __shared__ uint64_t full_bar[kN4PairStages];
  __shared__ uint64_t empty_bar[kN4PairStages];
  __shared__ uint64_t tmem_full_bar;
  __shared__ uint64_t tmem_empty_bar;
  __shared__ uint32_t tmem_base_slot;
  __shared__ uint32_t s_stop[2];  // where the producer and the issuer stopped
  __shared__ int abort_flag;
  __shared__ volatile int s_first_bad;  // first of this CTA's tiles whose accumulator never came
  __shared__ int s_off[kN4MaxGroups + 1];
  __shared__ int s_rows[kN4MaxGroups];  // rows of the group that are worked on
  __shared__ int s_tile_start[kN4MaxGroups + 1];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_tiles = (p.N + kN4BN - 1) / kN4BN;
  constexpr int stages = kN4PairStages;
  const uint32_t rank = cluster_ctarank();
  const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
  const int64_t a_off = p.a_off ? *p.a_off : 0, sfa_off = p.sfa_off ? *p.sfa_off : 0;  // on their way while the tables are built

  if (warp == 2) {
    if (lane < stages) {
      mbar_init(&full_bar[lane], 1);
      mbar_init(&empty_bar[lane], 1);
    }
    if (lane == 0) {
      mbar_init(&tmem_full_bar, 1);
      mbar_init(&tmem_empty_bar, 2 * kN4PairEpilogue);  // the leader's: the epilogue warps of both CTAs
      abort_flag = 0;
      s_first_bad = kNoBadTile;
    }
    mbar_fence_init();
    __syncwarp();
  }
  cluster_arrive();  // this CTA's barriers exist
  if (warp == 1) {
    tmem_alloc_pair(&tmem_base_slot, kN4TmemCols);
    tmem_relinquish_pair();
  }
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&p.tm_a);
      tma_prefetch_desc(&p.tm_b);
      tma_prefetch_desc(&p.tm_sfa);
      tma_prefetch_desc(&p.tm_sfb);
    }
    tile_tables(p.expert_offsets, p.expert_counts, p.e_local, p.max_rows, lane, s_off, s_tile_start,
                [&](int e, int lo, int hi, int count) {
      const int rows = bs_group_rows(lo, hi, count);
      s_rows[e] = rows;
      if (count > 0 && hi > lo && !bs_group_aligned(lo))
        set_status(p.status, kCapacityExceeded, -1, e, lo);  // groups must be 128-padded
      return ((rows + 2 * kN4BM - 1) / (2 * kN4BM)) * n_tiles;
    });
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_wait();  // both CTAs' barriers exist before either is signalled from the other
  tcgen05_fence_after();
  const uint32_t tmem_base = uniform(tmem_base_slot);
  const int total_tiles = uniform(s_tile_start[p.e_local]);
  const uint32_t ring = uniform(smem_u32(smem));

  if (warp == 0) {
    // ======================= producer =======================
    const bool elected = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    int e = 0;
    const int a_line0 = uniform(static_cast<int>(a_off >> 7)), sfa_line0 = uniform(static_cast<int>(sfa_off >> 7));
    const int sfa_x = uniform(static_cast<int>((sfa_off >> 4) & 7) * 4);  // word of its line that the scales start at
    const int col_blocks = (p.N + 127) >> 7;  // 128-wide blocks of the B side
    constexpr int kSfLines = kN4SfBytes / 128;
    const uint32_t lead_full = uniform(cluster_addr(smem_u32(&full_bar[0]), 0));
    bool ok = true;
    for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
      const N4Tile t = n4_pair_decode(tile, e, s_tile_start, s_off, s_rows);
      const bool second = uniform(t.n_blk * 2 + 1 < col_blocks ? 1 : 0) != 0;  // the tile's upper 128 columns exist
      // Groups end at multiples of 128: where the odd CTA has no rows it loads those of the even one.
      const int row = uniform(t.row0 + kN4BM * static_cast<int>(rank) < t.row_end ? t.row0 + kN4BM * static_cast<int>(rank) : t.row0);
      const int w_row = uniform(t.e * p.N + t.n_blk * kN4BN + 128 * static_cast<int>(rank));
      const int sfa_line = uniform(sfa_line0 + (row >> 7) * p.col_atoms * 4);
      const int sfb_line = uniform(static_cast<int>(t.e * (p.sfb_group_bytes >> 7)) + t.n_blk * 2 * p.col_atoms * 4);
#pragma unroll 1
      for (int kb = 0; kb < p.k_iters; ++kb) {
        ok = warp_mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_flag);
        if (!ok) break;
        uint8_t* sa = smem + stage * kN4PairStage;
        uint8_t* sb = sa + kN4ABytes;
        uint8_t* ssa = sb + kN4PairBBytes;
        uint8_t* ssb = ssa + kN4SfBytes;
        const uint32_t full = lead_full + stage * 8;
        if (elected) {
          if (rank == 0)
            mbar_arrive_expect_tx(&full_bar[stage], 2 * (kN4ABytes + kN4PairBBytes + (second ? 3 : 2) * kN4SfBytes));
          tma_load_3d_pair(sa, &p.tm_a, 0, a_line0 + kb, row, full);
          tma_load_2d_pair(sb, &p.tm_b, kb * 128, w_row, full);
          tma_load_2d_pair(ssa, &p.tm_sfa, sfa_x, sfa_line + kb * kSfLines, full);
          tma_load_2d_pair(ssb, &p.tm_sfb, 0, sfb_line + kb * kSfLines, full);
          if (second) tma_load_2d_pair(ssb + kN4SfBytes, &p.tm_sfb, 0, sfb_line + (p.col_atoms * 4 + kb * kSfLines), full);
        }
        __syncwarp();
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (lane == 0) s_stop[0] = ring_stop(stage, phase);
    __syncwarp();
  } else if (warp == 1) {
    // ======================= MMA issuer =======================
    // The warp that issues the MMAs copies a stage's scale atoms right before them, as in the kernel above.
    if (rank == 0) {
      const bool elected = elect_one();
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO 1024, version 1, 128-byte swizzle
      constexpr uint32_t kStep = 32u >> 4, kLbo = (16u >> 4) << 16;
      constexpr uint32_t idesc = umma_idesc_blockscaled(kN4BN, 1, 0, 0, 0, 0, 2 * kN4BM);
      const uint32_t full0 = uniform(smem_u32(&full_bar[0])), empty0 = uniform(smem_u32(&empty_bar[0]));
      const uint32_t tfull = uniform(smem_u32(&tmem_full_bar));
      int stage = 0;
      uint32_t phase = 0, ready = 0;  // ready: the current stage is known to be there
      int it = 0;
      bool ok = true;
      for (int tile = first_tile; tile < total_tiles; tile += tile_step, ++it) {
        ok = warp_mbar_wait(&tmem_empty_bar, (it & 1u) ^ 1u, &abort_flag);  // the epilogue has drained the accumulator
        if (!ok) break;
        tcgen05_fence_after();
#pragma unroll 1
        for (int kb = 0; kb < p.k_iters; ++kb) {
          if (!__all_sync(0xffffffffu, ready)) {
            ok = warp_mbar_wait(&full_bar[stage], phase, &abort_flag);
            if (!ok) break;
          }
          tcgen05_fence_after();
          const uint32_t a_addr = ring + stage * kN4PairStage;
          const uint32_t a_lo = ((a_addr & 0x3ffffu) >> 4) | kLbo, b_lo = (((a_addr + kN4ABytes) & 0x3ffffu) >> 4) | kLbo;
          const uint32_t sf_lo = sf_desc_lo(a_addr + kN4ABytes + kN4PairBBytes);
          const uint32_t sfa_t = tmem_base + kN4BN + stage * kN4PairSfCols;
          const uint32_t sfb_t = sfa_t + 16u;
          const uint32_t empty = empty0 + stage * 8;
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
          ready = mbar_test(full0 + stage * 8, phase);
          if (elected) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              tmem_cp_sf_lo_pair(sfa_t + 4 * j, sf_lo + j * kSfAtomWords);
              tmem_cp_sf_lo_pair(sfb_t + 8 * j, sf_lo + (4 + j) * kSfAtomWords);
              tmem_cp_sf_lo_pair(sfb_t + 8 * j + 4, sf_lo + (8 + j) * kSfAtomWords);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
              umma_nvf4_lo_pair(tmem_base, a_lo + j * kStep, b_lo + j * kStep, kDescHi, idesc, sfa_t + 4 * j, sfb_t + 8 * j,
                           (kb > 0 || j > 0) ? 1u : 0u);
            tcgen05_commit_pair(empty);
          }
          __syncwarp();
        }
        if (!ok) break;
        if (elected) tcgen05_commit_pair(tfull);
        __syncwarp();
      }
      if (lane == 0) s_stop[1] = ring_stop(stage, phase);
    }
    __syncwarp();
  } else if (warp == 2 + kN4PairEpilogue) {
    // ======================= accumulator watcher =======================
    // Polls the accumulator-ready barrier for the epilogue warps and releases them through a hardware named barrier;
    // after a timeout it releases them once more and stops.
    bool ok = true;
    int it = 0;
    for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step, ++it) {
      if (lane == 0) ok = handover_report(&s_first_bad, it, mbar_wait(&tmem_full_bar, it & 1u, &abort_flag));
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      asm volatile("bar.arrive %0, %1;" ::"r"(handover_barrier(it)), "r"(kN4PairEpilogue * 32 + 32) : "memory");
    }
  } else {
    // ======================= epilogue =======================
    // Four warps per TMEM lane quadrant, each owning 64 of the tile's 256 columns.  A lane reads its own accumulator row, the
    // warp hands the accumulator back at once, and 32 x 32 blocks are transposed through its staging tile and stored as
    // 64-byte row segments while the next tile's MMAs run.
    const int ew = warp - 2;
    const int quad = warp & 3;
    const int c0 = (ew >> 2) * 64;  // first of this warp's columns
    const int row_in_tile = static_cast<int>(rank) * kN4BM + quad * 32 + lane;
    const uint32_t lead_empty = cluster_addr(smem_u32(&tmem_empty_bar), 0);
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + c0;
    uint8_t* stg = smem + stages * kN4PairStage + ew * kStaging64Bytes;
    int e = 0, it = 0;
    bool ok = true;
    const int64_t c_off = p.c_off ? *p.c_off : 0;
    const int64_t h2_off = p.h2_off ? *p.h2_off : 0;
    const float* row_inv =
        p.row_inv_base ? reinterpret_cast<const float*>(p.row_inv_base + (p.row_inv_off ? *p.row_inv_off : 0)) : nullptr;
    const bool scaled = row_inv != nullptr || p.expert_inv != nullptr;
    for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step, ++it) {
      const N4Tile t = n4_pair_decode(tile, e, s_tile_start, s_off, s_rows);
      const int row = t.row0 + row_in_tile;
      const bool row_ok = row < t.row_end;
      const float scale = row_inv != nullptr && row_ok ? row_inv[row] : 1.0f;
      const float escale = p.expert_inv ? p.expert_inv[t.e] : 1.0f;
      // where this lane's row goes: h2 (and h1) with SwiGLU, C or the scatter destination otherwise
      uint64_t my_row = 0, my_h1 = 0;
      const int F = p.N / 2;
      if (row_ok) {
        if (p.swiglu) {
          my_row = reinterpret_cast<uint64_t>(p.h2_base) + h2_off + static_cast<uint64_t>(row) * F * 2;
          if (p.c_base) my_h1 = reinterpret_cast<uint64_t>(p.c_base) + c_off + static_cast<uint64_t>(row) * p.N * 2;
        } else if (p.scatter_ptrs != nullptr) {
          my_row = static_cast<uint64_t>(p.scatter_ptrs[row]);
        } else {
          my_row = reinterpret_cast<uint64_t>(p.c_base) + c_off + static_cast<uint64_t>(row) * p.N * 2;
        }
      }
      asm volatile("bar.sync %0, %1;" ::"r"(handover_barrier(it)), "r"(kN4PairEpilogue * 32 + 32) : "memory");  // released by the watcher
      ok = handover_good(&s_first_bad, it);  // the same for every epilogue warp
      if (!ok) break;
      tcgen05_fence_after();
      uint32_t ra[32], rb[32];
      tmem_ld_32x32(taddr, ra);
      tmem_ld_32x32(taddr + 32, rb);
      tmem_ld_wait();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(lead_empty);
      if (!__any_sync(0xffffffffu, row_ok)) continue;
      if (!row_ok) {  // whatever pads the group: keep it off the slow path of the sigmoid
#pragma unroll
        for (int j = 0; j < 32; ++j) ra[j] = rb[j] = 0u;
      }
      // sends what the staging tile holds (32 rows x 64 bytes) to byte `at` of the rows `base` names, if the 8 columns from `col` on exist
      auto store_block = [&](uint64_t base, int col, int limit, int64_t at) {
        __syncwarp();
        uint4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = stage64_get(stg, i * 8 + (lane >> 2), lane & 3);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint64_t rp = __shfl_sync(0xffffffffu, base, i * 8 + (lane >> 2));
          if (rp != 0 && col + 8 * (lane & 3) + 8 <= limit) store_global16(rp + at + 16 * (lane & 3), v[i]);
        }
      };
      if (p.swiglu) {
        // Columns come in groups of 16: 8 gate features then the matching 8 up features.
        uint4 zv[4], gv[4], uv[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t gw[4], uw[4];
          float gf[8], uf[8], zf[8];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int b = 16 * (g & 1) + 2 * q;
            float g0 = __uint_as_float(g < 2 ? ra[b] : rb[b]), g1 = __uint_as_float(g < 2 ? ra[b + 1] : rb[b + 1]);
            float u0 = __uint_as_float(g < 2 ? ra[b + 8] : rb[b + 8]), u1 = __uint_as_float(g < 2 ? ra[b + 9] : rb[b + 9]);
            if (scaled) {
              g0 = (g0 * scale) * escale; g1 = (g1 * scale) * escale;
              u0 = (u0 * scale) * escale; u1 = (u1 * scale) * escale;
            }
            gw[q] = pack_bf16x2(g0, g1);
            uw[q] = pack_bf16x2(u0, u1);
            gf[2 * q] = __uint_as_float(gw[q] << 16);
            gf[2 * q + 1] = __uint_as_float(gw[q] & 0xffff0000u);
            uf[2 * q] = __uint_as_float(uw[q] << 16);
            uf[2 * q + 1] = __uint_as_float(uw[q] & 0xffff0000u);
          }
          swiglu_f32(gf, uf, zf, p.act);
          zv[g] = make_uint4(pack_bf16x2(zf[0], zf[1]), pack_bf16x2(zf[2], zf[3]), pack_bf16x2(zf[4], zf[5]), pack_bf16x2(zf[6], zf[7]));
          gv[g] = make_uint4(gw[0], gw[1], gw[2], gw[3]);
          uv[g] = make_uint4(uw[0], uw[1], uw[2], uw[3]);
        }
        const int f0 = t.n_blk * (kN4BN / 2) + c0 / 2;  // first of this warp's 32 features
#pragma unroll
        for (int j = 0; j < 4; ++j) stage64_put(stg, lane, j, zv[j]);
        store_block(my_row, f0, F, f0 * 2);
        if (p.c_base != nullptr) {
#pragma unroll
          for (int j = 0; j < 4; ++j) stage64_put(stg, lane, j, gv[j]);
          store_block(my_h1, f0, F, f0 * 2);
#pragma unroll
          for (int j = 0; j < 4; ++j) stage64_put(stg, lane, j, uv[j]);
          store_block(my_h1, f0, F, (F + f0) * 2);
        }
      } else {
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
          uint32_t (&r)[32] = blk == 0 ? ra : rb;
          if (scaled) {
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint((__uint_as_float(r[j]) * scale) * escale);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) stage64_put(stg, lane, j, pack8_bf16(r + 8 * j));
          const int col = t.n_blk * kN4BN + c0 + 32 * blk;
          store_block(my_row, col, p.N, static_cast<int64_t>(col) * 2);
        }
      }
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (abort_flag && rank == 0 && threadIdx.x == 0) {  // the leader's barriers count both CTAs' loads and MMAs
    const uint64_t deadline = globaltimer_ns() + kSettleNs;
    settle_ring(empty_bar, stages, s_stop[1], deadline);
    settle_ring(full_bar, stages, s_stop[0], deadline);
  }
  __syncwarp();
  cluster_sync();  // neither CTA leaves while the other may still signal its barriers, or loads into either are in flight
  if (abort_flag && threadIdx.x == 0) set_status(p.status, kPipelineTimeout, 4, blockIdx.x);
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, kN4TmemCols);
  }
}

// What the two kernels share of the forward of dm_gemm_blockscaled (arguments checked by the entry points).
static int n4_setup(N4Params& p, const dm_operand& a, const dm_operand& sfa, const void* w, const void* sfb, const dm_operand& c,
                    const dm_operand& h2, const int64_t* scatter_ptrs, const dm_operand& row_scale_inv,
                    const float* expert_scale_inv, const int32_t* expert_offsets, int e_local, int64_t max_rows, int64_t N,
                    int64_t Kd, int swiglu_interleaved, const ActParams& act, const int* cond, int* status, int w_box_rows) {
  int rc = encode_arena_u8(&p.tm_a, a, Kd / 2, max_rows + 256, kN4BM);
  if (rc != kRcOk) return rc;
  rc = encode_2d_u8(&p.tm_b, w, static_cast<int64_t>(e_local) * N, Kd / 2, w_box_rows);
  if (rc != kRcOk) return rc;
  p.col_atoms = static_cast<int>((Kd / 16 + 3) / 4);
  p.sfb_group_bytes = (N + 127) / 128 * 128 * static_cast<int64_t>(p.col_atoms) * 4;
  p.a_off = a.offset;
  p.sfa_off = sfa.offset;
  p.sfa_base = static_cast<const uint8_t*>(sfa.base);
  p.sfb = static_cast<const uint8_t*>(sfb);
  p.c_off = c.offset;
  p.h2_off = h2.offset;
  p.c_base = static_cast<uint8_t*>(c.base);
  p.h2_base = static_cast<uint8_t*>(h2.base);
  p.row_inv_base = static_cast<const uint8_t*>(row_scale_inv.base);
  p.row_inv_off = row_scale_inv.offset;
  p.expert_inv = expert_scale_inv;
  p.scatter_ptrs = scatter_ptrs;
  p.expert_offsets = expert_offsets;
  p.cond = cond;
  p.status = status;
  p.e_local = e_local;
  p.max_rows = static_cast<int>(max_rows);
  p.N = static_cast<int>(N);
  p.k_iters = static_cast<int>(Kd / 256);
  p.swiglu = swiglu_interleaved ? 1 : 0;
  p.act = act;
  return kRcOk;
}

// The NVFP4 forward of dm_gemm_blockscaled (arguments checked there).
int nvfp4_forward(const dm_operand& a, const dm_operand& sfa, const void* w, const void* sfb, const dm_operand& c,
                  const dm_operand& h2, const int64_t* scatter_ptrs, const dm_operand& row_scale_inv,
                  const float* expert_scale_inv, const int32_t* expert_offsets, int e_local, int64_t max_rows, int64_t N,
                  int64_t Kd, int swiglu_interleaved, const ActParams& act, const int* cond, int num_sms, int* status,
                  cudaStream_t st) {
  N4Params p{};
  int rc = n4_setup(p, a, sfa, w, sfb, c, h2, scatter_ptrs, row_scale_inv, expert_scale_inv, expert_offsets, e_local, max_rows,
                    N, Kd, swiglu_interleaved, act, cond, status, kN4BN);
  if (rc != kRcOk) return rc;
  p.direct_store = (swiglu_interleaved && !c.base) ? 1 : 0;
  static PerDeviceOnce attr_set;
  rc = once_per_device(attr_set, [] {
    return static_cast<int>(cudaFuncSetAttribute(nvfp4_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(kN4SmemDirect)));
  });
  if (rc != 0) return rc;
  nvfp4_wide_kernel<<<persistent_grid(num_sms), kN4Threads, p.direct_store ? kN4SmemDirect : kN4Smem, st>>>(p);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace dm

using namespace dm;

// dm_gemm_blockscaled_counted for NVFP4 experts that received many rows.
extern "C" int dm_gemm_nvfp4_pairs(dm_operand a, dm_operand sfa, const void* w, const void* sfb, dm_operand c, dm_operand h2,
                                   const int64_t* scatter_ptrs, dm_operand row_scale_inv, const float* expert_scale_inv,
                                   const int32_t* expert_offsets, const int32_t* expert_counts, int e_local, int64_t max_rows,
                                   int64_t N, int64_t Kd, int swiglu_interleaved, int clamped, float alpha, float limit,
                                   const int* cond, int num_sms, int* status, void* stream) {
  if (!a.base || !sfa.base || !w || !sfb || !expert_offsets || e_local <= 0 || max_rows < 0 || N <= 0 || Kd <= 0)
    return kRcBadArg;
  if (!swiglu_interleaved && !c.base && !scatter_ptrs) return kRcBadArg;
  if (swiglu_interleaved && (!h2.base || scatter_ptrs)) return kRcBadArg;
  if (e_local > kN4MaxGroups || max_rows > (1 << 30)) return kRcTooLarge;
  if ((Kd % 256) != 0 || (N % 128) != 0 || (max_rows % 128) != 0) return kRcUnsupportedShape;
  if (max_rows == 0) return kRcOk;
  N4Params p{};
  int rc = n4_setup(p, a, sfa, w, sfb, c, h2, scatter_ptrs, row_scale_inv, expert_scale_inv, expert_offsets, e_local, max_rows,
                    N, Kd, swiglu_interleaved, ActParams{clamped, alpha, limit}, cond, status, 128);
  if (rc != kRcOk) return rc;
  p.expert_counts = scatter_ptrs || swiglu_interleaved ? expert_counts : nullptr;  // a dense C is written for whole groups
  // an extent that does not hold the layout was never told in earnest: the rows alone bound the loads then
  const int64_t layout_bytes = max_rows / 128 * static_cast<int64_t>(p.col_atoms) * 512;
  rc = encode_sf(&p.tm_sfa, sfa.base, sfa.bytes >= layout_bytes ? sfa.bytes : int64_t{1} << 37, true, 16);
  if (rc != kRcOk) return rc;
  rc = encode_sf(&p.tm_sfb, sfb, e_local * p.sfb_group_bytes, false, 16);
  if (rc != kRcOk) return rc;
  static PerDeviceOnce attr_set;
  rc = once_per_device(attr_set, [] {
    return static_cast<int>(cudaFuncSetAttribute(nvfp4_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(kN4PairSmem)));
  });
  if (rc != 0) return rc;
  nvfp4_pair_kernel<<<pair_grid(num_sms), kN4PairThreads, kN4PairSmem, static_cast<cudaStream_t>(stream)>>>(p);
  return static_cast<int>(cudaGetLastError());
}
