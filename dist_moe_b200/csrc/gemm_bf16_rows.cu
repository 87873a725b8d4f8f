// Persistent grouped BF16 GEMMs over routed rows on tcgen05 tensor cores (sm_100a): forward and input gradient.
//
//   fprop  C[r,n]  = sum_k A[r,k] W[e][n][k]     A, W K-major
//   dgrad  C[r,n]  = sum_k A[r,k] W[e][k][n]     A K-major, W N-major
//
// A pair of CTAs (cta_group::2) works on one tile: 256 output columns of the weights are the M side of the MMA (128 per
// CTA) and up to 256 routed rows its N side (each CTA loads half of them).  An expert's rows are split into
// ceil(rows / 256) equal tiles of a multiple of 32 rows, so hardly any tensor time goes into rows that the expert does not
// have; with rows on a 128-row M side an expert of 384 +- 20 rows needed a fourth tile half of the time (17 % of the
// issued MMAs at 64 experts x 384 rows, 27 % at 64 x 187).  The accumulator holds C transposed (TMEM lane = output column,
// TMEM column = routed row).
//
// Bound: with 128 x 256 tiles of single CTAs, operand loads from L2 (48 KiB per 512 tensor cycles and SM; every such launch
// ran at 12.5 to 13 TB/s); a pair loads 32 KiB for the same work.  With a few rows per expert, the weight stream from HBM.
// Launch loops on one power-capped B200 (SM clock near 1.4 GHz), D = 2048, F = 1408, single-CTA tiles with rows on the M side
// -> this kernel: 64 experts x 384 rows W13 281 -> 245 us, W13 input gradient 275 -> 242 us, W13 with SwiGLU 306 -> 283 us;
// 8 x 3072: 226 -> 198, 232 -> 198 (1430 TFLOP/s), 250 -> 232 us; 64 x 187: 180 -> 146, 170 -> 142, 200 -> 165 us; 64 x 3:
// 121 -> 119, 121 -> 120, 128 -> 122 us (the weights at 6.2 TB/s).
//
// One CTA per SM, warp-specialised:
//   warp 0       TMA producer of the weights: stages of 64 K elements, 16 KiB of weights and as many rows as the launch's
//                largest tile needs (16 to 128 per CTA; small tiles leave room for up to ten stages, which keeps enough of
//                the weight stream in flight when experts have few rows), no multicast.
//   warp 1       MMA issuer (of the leading CTA): 512 TMEM columns = two accumulators of up to 256 rows; the elected lane issues
//                tcgen05.mma (M256, N = rows of the tile, K16) and publishes with tcgen05.commit.
//   warps 2..9   epilogue (two per TMEM lane quadrant, each group of four owning half of the tile's rows): read 32 rows
//                x 32 columns, exchange pairs of columns between neighbouring lanes, and collect 32 rows x 128 columns
//                of the group in shared memory, which leave as 256-byte row pieces (128-byte pieces of gate, up and h2
//                with the fused SwiGLU) to local or peer memory.
//   warps 10..13 gather (fused dispatch): pull routed rows through the pointer table.
//   warp 14      accumulator watcher.
//   warp 15      TMA producer of the rows.
//
// Groups are the local experts; their row ranges come from device memory (expert_offsets), so the tile list is built
// by every CTA at kernel start and no host read is needed.  Activation operands are addressed as (arena base, device
// byte offset): the tensor map views the whole arena as [row][128-byte line][64 bf16] with overlapping strides, so a
// planner-chosen offset only changes a coordinate.
#include "gemm_common.cuh"
#include "row_tiles.cuh"

namespace dm {

constexpr int kRwBM = 128;    // output columns per CTA of a pair (weights, M side)
constexpr int kRwBK = 64;     // K of a stage (128 bytes per row)
constexpr int kRwMaxStages = 10;
constexpr int kRwThreads = 512;
constexpr int kRwGatherWarps = 4;
constexpr int kRwMaxGroups = 256;
constexpr uint32_t kRwWBytes = kRwBM * kRwBK * 2;  // 16 KiB
constexpr uint32_t kRwTmemCols = 512;
constexpr uint32_t kRwStagePlain = 32 * 256;        // per epilogue group: 32 rows x 128 columns
constexpr uint32_t kRwStageFused = 32 * 384;        // 32 rows x (64 gate, 64 up, 64 h2)
constexpr uint32_t kRwDynSmem = 227 * 1024 - 3072;  // the rest holds the tables and barriers
constexpr uint32_t kRwRingPlain = kRwDynSmem - 1024 - 2 * kRwStagePlain;
constexpr uint32_t kRwRingFused = kRwDynSmem - 1024 - 2 * kRwStageFused;
static_assert(kRwRingFused >= 6 * (kRwWBytes + kRwMaxN * 64), "six full stages");

struct RowsParams {
  CUtensorMap tm_w;            // weights: forward boxes of 128 rows x 64 K, input gradient 64 K rows x 64 columns
  CUtensorMap tm_x[kRwBoxes];  // routed rows, boxes of rw_box_rows(i) rows x 64 K
  const int64_t* a_off;        // device byte offsets (may be null = 0)
  const int64_t* c_off;
  const int64_t* h2_off;
  uint8_t* c_base;  // with the fused SwiGLU: h1, null where nothing reads it
  uint8_t* h2_base;
  const int64_t* scatter_ptrs;
  const int64_t* gather_ptrs;  // fused dispatch: row r of A is pulled from gather_ptrs[r] (may be peer memory)
  int* gather_flags;           // one counter per 128-row block of A, zero before the launch
  int* gather_ticket;          // next unit to pull, zero before the launch
  int* gather_done;            // not null: CTAs that need neither any more, zero before the launch; the last clears all three
  uint8_t* a_base;             // where the pulled rows land (the A operand itself)
  const int32_t* expert_offsets;
  const int* cond;
  int* status;
  int e_local;
  int max_rows;
  int N;   // output columns
  int Kd;  // contraction
  ActParams act;
};

// kRowsSwiglu: W13 forward with SwiGLU.  The values also name the kernel in a timeout status (2 is the weight gradient).
enum RowsMode : int { kRowsFprop = 0, kRowsDgrad = 1, kRowsSwiglu = 3 };

// Word of two neighbouring columns of one row from words of one column of two neighbouring rows: lanes 2p and 2p + 1
// hold columns 2p and 2p + 1 of the rows (t, t + 1); the even lane receives row t, the odd lane row t + 1.
__device__ __forceinline__ uint32_t rw_pair(uint32_t w, int odd) {
  const uint32_t o = __shfl_xor_sync(0xffffffffu, w, 1);
  return __byte_perm(w, o, odd ? 0x3276 : 0x5410);
}

// Pulls the `live` rows of a unit, kRows at a time (lane l holds row l's pointer, null: zeros), kLoads 16-byte pieces of each in
// flight per lane.
template <int kRows, int kLoads>
__device__ __forceinline__ void rw_pull(uint64_t my_ptr, int live, uint4* dst, int vec_per_row, int lane) {
  for (int rr = 0; rr < live; rr += kRows) {
    const uint4* src[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i) src[i] = reinterpret_cast<const uint4*>(__shfl_sync(0xffffffffu, my_ptr, (rr + i) & 31));
    for (int v0 = 0; v0 < vec_per_row; v0 += 32 * kLoads) {
      uint4 b[kRows][kLoads];
#pragma unroll
      for (int i = 0; i < kRows; ++i)
#pragma unroll
        for (int j = 0; j < kLoads; ++j) {
          const int v = v0 + j * 32 + lane;
          b[i][j] = (rr + i < live && src[i] != nullptr && v < vec_per_row) ? __ldcg(src[i] + v) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
      for (int i = 0; i < kRows; ++i)
#pragma unroll
        for (int j = 0; j < kLoads; ++j) {
          const int v = v0 + j * 32 + lane;
          if (rr + i < live && v < vec_per_row) dst[static_cast<int64_t>(rr + i) * vec_per_row + v] = b[i][j];
        }
    }
  }
}

// One part of this CTA, a gather warp or the row producer, needs the flags and the ticket no more.  The last part of the last
// CTA clears them for the next launch while the last tiles are computed: every part gets here, also after a timeout, and
// nothing waits.  A memset in front of the launch cost 1.3 to 1.7 us and the gap to the launch behind it, three times per
// training pass.
__device__ __forceinline__ void rw_gather_finished(const RowsParams& p, int* s_parts, int lane) {
  __syncwarp();
  int last = 0;
  if (lane == 0) {
    __threadfence();  // this warp's polls, draws and bumps come before
    if (atomicAdd(s_parts, 1) == kRwGatherWarps) {
      __threadfence();
      last = atomicAdd(p.gather_done, 1) == static_cast<int>(gridDim.x) - 1;
      __threadfence();
    }
  }
  if (uniform(last) == 0) return;
  const int blocks = (min(p.expert_offsets[p.e_local], p.max_rows) + kRwGatherBlock - 1) / kRwGatherBlock;
  for (int b = lane; b < blocks; b += 32) p.gather_flags[b] = 0;
  if (lane == 0) *p.gather_ticket = *p.gather_done = 0;
}

template <int kMode>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kRwThreads, 1) rows_gemm_kernel(const __grid_constant__ RowsParams p) {
  if (p.cond != nullptr && *p.cond == 0) return;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  __shared__ uint64_t full_bar[kRwMaxStages];
  __shared__ uint64_t empty_bar[kRwMaxStages];
  __shared__ uint64_t tmem_full_bar[2];
  __shared__ uint64_t tmem_empty_bar[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ volatile int s_first_bad;  // first of this CTA's tiles whose accumulator never came
  __shared__ uint32_t s_stop[3];  // where the weight producer, the row producer and the issuer stopped
  __shared__ int s_box;
  __shared__ int s_parts;  // gather warps and row producer that are finished with the flags
  __shared__ int s_off[kRwMaxGroups + 1];
  __shared__ int s_tile_start[kRwMaxGroups + 1];
  __shared__ uint16_t s_per[kRwMaxGroups];

  constexpr bool kSwiglu = kMode == kRowsSwiglu;
  constexpr int kTableBarrier = 1 + kHandoverBarriers + 2;  // after those of the hand-over and of the two epilogue groups
  constexpr uint32_t kRing = kSwiglu ? kRwRingFused : kRwRingPlain;
  constexpr uint32_t kStaging = kSwiglu ? kRwStageFused : kRwStagePlain;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();

  // The gather warps' first units: those of the first tiles go to the CTAs that start first.
  const bool gathers = warp >= 10 && warp < 10 + kRwGatherWarps && p.gather_flags != nullptr;
  int unit = 0;
  if (gathers && lane == 0) unit = atomicAdd(p.gather_ticket, 1);
  const int64_t a_off = p.a_off ? *p.a_off : 0;

  // ---- tile table -----------------------------------------------------------
  const int m_pairs = kSwiglu ? (p.N / 2) / 128 : (p.N + 2 * kRwBM - 1) / (2 * kRwBM);
  if (warp == 2) {
    if (lane < kRwMaxStages) {
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
      s_parts = 0;
    }
    mbar_fence_init();
    __syncwarp();
  }
  cluster_arrive();  // this CTA's barriers exist
  if (warp == 1) {
    tmem_alloc_pair(&tmem_base_slot, kRwTmemCols);
    tmem_relinquish_pair();
  }
  if (warp == 0) {
    if (lane == 0) tma_prefetch_desc(&p.tm_w);
    int box = 0;
    tile_tables(p.expert_offsets, nullptr, p.e_local, p.max_rows, lane, s_off, s_tile_start, [&](int e, int lo, int hi, int) {
      const int nt = rw_row_tiles(hi - lo), per = rw_rows_per_tile(hi - lo);
      s_per[e] = static_cast<uint16_t>(per);
      if (nt > 0) box = max(box, rw_box_index(per));
      return nt * m_pairs;
    });
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) box = max(box, __shfl_xor_sync(0xffffffffu, box, d));
    if (lane == 0) s_box = box;
  }
  tcgen05_fence_before();
  if (gathers) {
    // The gather warps need none of it and start at once, before the weights fill the memory system.  A barrier of its own: at
    // the one of __syncthreads they could arrive again, at the end of the kernel, before the tables are there.
    asm volatile("bar.arrive %0, %1;" ::"n"(kTableBarrier), "n"(kRwThreads) : "memory");
  } else {
    asm volatile("bar.sync %0, %1;" ::"n"(kTableBarrier), "n"(kRwThreads) : "memory");
    cluster_wait();  // both CTAs' barriers exist before either is signalled from the other
  }
  tcgen05_fence_after();
  const uint32_t tmem_base = uniform(tmem_base_slot);
  const int total_tiles = uniform(s_tile_start[p.e_local]);
  // One B200, 64 experts x 2048 x 1408, W13 / W2, rows per expert on average: 3 117.7 / 61.7 -> 117.2 / 61.6 us, 48 128.7 / 67.4 ->
  // 127.1 / 67.2, 64 131.1 / 66.1 -> 129.7 / 65.4, 96 136.6 / 68.4 -> 135.4 / 68.2; decode layer of 32 tokens 197.6 -> 195.3.  At
  // 187 rows on average, tiles of up to 256, nothing changes (312.2 and 312.8 us a layer).
  const int pair = blockIdx.x >> 1;
  const int tile_step = balanced_pairs(total_tiles, gridDim.x >> 1, 2 * rw_box_rows(uniform(s_box)), 128);
  const int first_tile = pair < tile_step ? pair : total_tiles;
  // ring: stages as large as the launch's largest tile needs
  const uint32_t stage_bytes = kRwWBytes + static_cast<uint32_t>(rw_box_rows(uniform(s_box))) * 128;
  const int fit = static_cast<int>(kRing / stage_bytes);
  const int stages = fit < kRwMaxStages ? fit : kRwMaxStages;

  if (warp == 0 || warp == 15) {
    // ======================= TMA producers: warp 0 the weights, warp 15 the rows =======================
    const bool rows_side = warp == 15;
    const bool elected = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    int e = 0;
    const int a_line0 = uniform(static_cast<int>(a_off >> 7));
    bool ok = true;
    const int total_rows = s_off[p.e_local];
    const int k_iters = p.Kd / kRwBK;
    const int ready = kRwGatherBlock / rw_gather_unit_rows(total_rows, static_cast<int>(gridDim.x) * kRwGatherWarps);
    if (rows_side && elected) tma_prefetch_desc(&p.tm_x[s_box]);
    const uint32_t lead_full = uniform(cluster_addr(smem_u32(&full_bar[0]), 0));
    for (int tile = first_tile; tile < total_tiles; tile += tile_step) {
      const RowsTile t = rw_decode(tile, e, s_tile_start, s_off, s_per);
      if (rows_side && p.gather_flags != nullptr) {
        // The tile's rows are pulled by the gather warps of some CTA: every one of its (at most three) 128-row blocks is
        // acquired, a lane each, before any of them is loaded, whatever earlier tiles have waited for.  One L2 read per tile,
        // hidden behind the ring: a training layer of 64 experts x 384 rows takes 1.907 ms, 1.911 ms without it.
        const RowsBlocks need = rw_tile_blocks(t, total_rows);
        const int b = need.first + lane;
        if (b <= need.last) {
          const uint64_t t0 = globaltimer_ns();
          uint32_t spins = 0;
          while (ld_acquire_gpu(p.gather_flags + b) < ready) {
            if ((++spins & 0xff) == 0 &&
                (*const_cast<volatile int*>(&abort_flag) || globaltimer_ns() - t0 > 2000000000ull)) {
              abort_flag = 1;
              ok = false;
              break;
            }
          }
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        __syncwarp();             // what the polling lanes acquired is ordered before the elected lane's loads
        fence_proxy_async_global();  // rows were written with ordinary stores, TMA reads them through the async proxy
      }
      const int box = uniform(rw_box_index(t.n));
      const CUtensorMap* tm_x = &p.tm_x[box];
      const uint32_t tx = 2 * (kRwWBytes + static_cast<uint32_t>(rw_box_rows(box)) * 128);  // both CTAs' loads
      const int m_blk = uniform(2 * t.pair + static_cast<int>(rank));
      const int x_row = uniform(t.row0 + static_cast<int>(rank) * (t.n >> 1));
      const int expert = uniform(t.e);
#pragma unroll 1
      for (int kb = 0; kb < k_iters; ++kb) {
        ok = warp_mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_flag);
        if (!ok) break;
        uint8_t* sw = smem + stage * stage_bytes;
        const uint32_t full = lead_full + stage * 8;
        if (elected) {
          if (rows_side) {
            tma_load_3d_pair(sw + kRwWBytes, tm_x, 0, a_line0 + kb, x_row, full);
          } else {
            if (rank == 0) mbar_arrive_expect_tx(&full_bar[stage], tx);
            if (kMode == kRowsFprop) {
              tma_load_2d_pair(sw, &p.tm_w, kb * kRwBK, expert * p.N + m_blk * kRwBM, full);
            } else if (kMode == kRowsSwiglu) {
              tma_load_5d_pair(sw, &p.tm_w, kb * kRwBK, 0, 0, m_blk * 4, expert, full);
            } else {
              tma_load_2d_pair(sw, &p.tm_w, m_blk * kRwBM, expert * p.Kd + kb * kRwBK, full);
              tma_load_2d_pair(sw + 8192, &p.tm_w, m_blk * kRwBM + 64, expert * p.Kd + kb * kRwBK, full);
            }
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
    if (rows_side && p.gather_done != nullptr) rw_gather_finished(p, &s_parts, lane);
  } else if (warp == 1) {
    // ======================= MMA issuer =======================
    // The loop around the four MMAs of a stage is kept to a few adds: running descriptor words, and the next stage's
    // barrier looked at while this stage's MMAs are on their way.
    constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO 1024, version 1, 128-byte swizzle
    constexpr uint32_t kLboK = (16u >> 4) << 16, kLboMN = (8192u >> 4) << 16;
    constexpr uint32_t w_step = kMode == kRowsDgrad ? (2048u >> 4) : (32u >> 4);
    constexpr uint32_t x_step = 32u >> 4;
    constexpr uint32_t kLboW = kMode == kRowsDgrad ? kLboMN : kLboK;
    constexpr uint32_t w_to_x = (kRwWBytes >> 4) + kLboK - kLboW;  // from a stage's weight word to its row word
    if (rank == 0) {
      const bool elected = elect_one();
      const uint32_t w_first = uniform(((smem_u32(smem) & 0x3ffffu) >> 4) | kLboW);
      const uint32_t stage_words = stage_bytes >> 4;
      const uint32_t full0 = uniform(smem_u32(&full_bar[0])), empty0 = uniform(smem_u32(&empty_bar[0]));
      const uint32_t tfull0 = uniform(smem_u32(&tmem_full_bar[0]));
      const uint32_t full_end = full0 + 8u * stages, to_empty = empty0 - full0;
      const int k_iters = p.Kd / kRwBK;
      uint32_t w = w_first, full = full0, phase = 0, ready = 0;  // ready: the current stage is known to be full
      int e = 0, it = 0;
      bool ok = true;
      for (int tile = first_tile; tile < total_tiles; tile += tile_step, ++it) {
        const RowsTile t = rw_decode(tile, e, s_tile_start, s_off, s_per);
        const uint32_t idesc = uniform(umma_idesc_bf16(2 * kRwBM, t.n, kMode == kRowsDgrad ? 1 : 0, 0));
        const int buf = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1u;
        const uint32_t d_tmem = tmem_base + buf * kRwMaxN;
        ok = warp_mbar_wait(&tmem_empty_bar[buf], acc_phase ^ 1u, &abort_flag);
        if (!ok) break;
        tcgen05_fence_after();
        uint32_t acc = 0;
#pragma unroll 1
        for (int kb = 0; kb < k_iters; ++kb) {
          if (!__all_sync(0xffffffffu, ready)) {
            ok = warp_mbar_wait(&full_bar[(full - full0) >> 3], phase, &abort_flag);
            if (!ok) break;
          }
          const uint32_t w_now = w, empty = full + to_empty;
          w += stage_words;
          full += 8;
          if (full == full_end) {
            full = full0;
            w = w_first;
            phase ^= 1u;
          }
          ready = mbar_test(full, phase);
          if (elected) {
            umma_bf16_lo_pair(d_tmem, w_now, w_now + w_to_x, kDescHi, idesc, acc);
            umma_bf16_lo_pair(d_tmem, w_now + w_step, w_now + (w_to_x + x_step), kDescHi, idesc, 1u);
            umma_bf16_lo_pair(d_tmem, w_now + 2 * w_step, w_now + (w_to_x + 2 * x_step), kDescHi, idesc, 1u);
            umma_bf16_lo_pair(d_tmem, w_now + 3 * w_step, w_now + (w_to_x + 3 * x_step), kDescHi, idesc, 1u);
            tcgen05_commit_pair(empty);
          }
          __syncwarp();
          acc = 1;
        }
        if (!ok) break;
        if (elected) tcgen05_commit_pair(tfull0 + buf * 8);
        __syncwarp();
      }
      if (lane == 0) s_stop[2] = ring_stop(static_cast<int>((full - full0) >> 3), phase);
    }
    __syncwarp();
  } else if (warp == 14) {
    // ======================= accumulator watcher =======================
    // One warp polls the accumulator-ready barriers on behalf of the eight epilogue warps and releases them
    // through a hardware named barrier: the epilogue warps then sleep without taking issue slots from the
    // MMA-issuing and TMA-issuing threads that share their schedulers.  After a timeout it releases them once more and stops.
    bool ok = true;
    int it = 0;
    for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step, ++it) {
      const int buf = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1u;
      if (lane == 0) ok = handover_report(&s_first_bad, it, mbar_wait(&tmem_full_bar[buf], acc_phase, &abort_flag));
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      asm volatile("bar.arrive %0, %1;" ::"r"(handover_barrier(it)), "r"(8 * 32 + 32) : "memory");
    }
  } else if (warp >= 10) {
    // ======================= gather (fused dispatch) =======================
    // Units of 1 to 8 rows go to the gather warps of the grid by ticket, in ascending row order, the order in which the tiles
    // consume them.  Each warp pulls its unit with 16-byte loads (peer memory allowed), sixteen in flight per lane, and then bumps
    // the counter of the unit's 128-row block; the TMA producer of whichever CTA needs a block waits for all of its units.
    // Gather warps wait on nothing, and a unit belongs only to a warp that is running: CTAs that come late, because kernels
    // of other streams hold their SMs, delay no row that the CTAs already there are waiting for (dealt out by CTA index,
    // such rows never came and the wait ran out).
    // The first tiles wait for the chain of one unit (pointer, rows, release, poll, proxy fence), so: units are as small as the
    // number of gather warps allows, the pointers of a unit are loaded at once, the warps start before the tile table is there and
    // with it before the weights fill the memory system, the CTAs that start first draw the first units, and the fence
    // between the proxies names global memory alone (for all spaces it waits for the weights on their way, up to 5700 cycles).
    // First row load after the start of the launch, cycles: 192 rows x 2048 22 900 -> 15 000, 4593 x 1088
    // 20 000 -> 15 000, 32 x 256 12 800 -> 8800.  One B200, launches: W13 of 192 rows, 64 experts 120.5 -> 115.4 us, W13 / its
    // repetition / W2 input gradient of 4593 rows 37.8 / 32.6 / 25.5 -> 30.1 / 28.6 / 18.2; layers 208.7 -> 204.9 and 330 -> 314.
    // A warp keeps 8 KiB in flight: over NVLink a 32-row unit took about 30 us before the first tiles could begin, an 8-row
    // unit a quarter of that.
    if (p.gather_flags != nullptr) {
      const int total_rows = min(p.expert_offsets[p.e_local], p.max_rows);  // the tables may not be there yet
      const int unit_rows = rw_gather_unit_rows(total_rows, static_cast<int>(gridDim.x) * kRwGatherWarps);
      const int per_block = kRwGatherBlock / unit_rows;
      const int units = (total_rows + kRwGatherBlock - 1) / kRwGatherBlock * per_block;
      const int vec_per_row = p.Kd / 8;
      uint4* dst_base = reinterpret_cast<uint4*>(p.a_base + a_off);
      int u = uniform(unit);
      while (u < units) {
        int next = 0;
        if (lane == 0) next = atomicAdd(p.gather_ticket, 1);  // on its way while this unit is pulled
        const int r_begin = u * unit_rows, left = total_rows - r_begin, live = left < unit_rows ? left : unit_rows;
        const uint64_t ptr = lane < live ? static_cast<uint64_t>(p.gather_ptrs[r_begin + lane]) : 0;
        uint4* dst = dst_base + static_cast<int64_t>(r_begin) * vec_per_row;
        if (vec_per_row > 128)
          rw_pull<2, 8>(ptr, live, dst, vec_per_row, lane);
        else
          rw_pull<4, 4>(ptr, live, dst, vec_per_row, lane);
        __syncwarp();  // all lanes' rows are stored before the release below
        if (lane == 0) red_release_gpu_add(p.gather_flags + u / per_block, 1);
        u = uniform(next);
      }
      __syncwarp();
      cluster_wait();  // the other half of the arrival above
      if (p.gather_done != nullptr) rw_gather_finished(p, &s_parts, lane);
    }
  } else {
    // ======================= epilogue =======================
    // Group `half` takes blocks of 32 rows (TMEM columns) of the tile: the first ceil(blocks / 2) or the rest.  Lane l of
    // quadrant q holds output column 32 q + l (fused: gate or up feature 16 q + l % 16).  The staging tile is laid out
    // row by row; the 16-byte chunks of a row are permuted so that the words the 32 lanes write (two rows, and gate and
    // up) fall into different banks, and the reads of whole rows stay conflict free.
    const int ew = warp - 2;    // 0..7
    const int quad = warp & 3;  // TMEM lanes [32*quad, 32*quad+32)
    const int half = ew >> 2;
    uint8_t* stg = smem + kRing + half * kStaging;
    const int bar_id = 1 + kHandoverBarriers + half;
    const uint32_t lead_empty = cluster_addr(smem_u32(&tmem_empty_bar[0]), 0);
    const int odd = lane & 1;
    int e = 0, it = 0;
    bool ok = true;
    const int64_t c_off = p.c_off ? *p.c_off : 0;
    const int64_t h2_off = p.h2_off ? *p.h2_off : 0;
    for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step, ++it) {
      const RowsTile t = rw_decode(tile, e, s_tile_start, s_off, s_per);
      const int buf = it & 1;
      const int blocks = t.n >> 5;
      const int m_blk = 2 * t.pair + static_cast<int>(rank);
      const int b_begin = half == 0 ? 0 : (blocks + 1) >> 1;
      const int b_end = half == 0 ? (blocks + 1) >> 1 : blocks;
      // row pointer of this lane's row of a block (the first one is loaded ahead of the accumulator)
      auto row_ptr = [&](int b) -> uint64_t {
        const int r = b * 32 + lane;
        if (r >= t.rows) return 0;
        if (!kSwiglu && p.scatter_ptrs != nullptr) return static_cast<uint64_t>(p.scatter_ptrs[t.row0 + r]);
        if (kSwiglu && p.c_base == nullptr) return 0;
        return reinterpret_cast<uint64_t>(p.c_base) + c_off + static_cast<uint64_t>(t.row0 + r) * p.N * 2;
      };
      uint64_t my_row = b_begin < b_end ? row_ptr(b_begin) : 0;
      asm volatile("bar.sync %0, %1;" ::"r"(handover_barrier(it)), "r"(8 * 32 + 32) : "memory");  // released by the watcher
      ok = handover_good(&s_first_bad, it);  // the same for every epilogue warp
      if (!ok) break;
      tcgen05_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + buf * kRwMaxN;
      for (int b = b_begin; b < b_end; ++b) {
        uint32_t v[32];
        tmem_ld_32x32(taddr + b * 32, v);
        const uint64_t next_row = b + 1 < b_end ? row_ptr(b + 1) : 0;
        tmem_ld_wait();
        if (b + 1 == b_end) {  // the group's last read: the accumulator is handed back before the stores
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(lead_empty + buf * 8);
        }
        uint32_t w[16];  // rows (2i, 2i + 1) of this lane's column
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = pack_bf16x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
        asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "r"(128) : "memory");  // the previous block has left the staging tile
        if (kSwiglu) {
          const int up = lane >> 4;  // lanes 0-15 hold gate features, lanes 16-31 the matching up features
          const int word = (lane & 15) >> 1;
          const int chunk = 2 * quad + (word >> 2);
          if (p.c_base != nullptr) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int r = 2 * i + odd;
              *reinterpret_cast<uint32_t*>(stg + r * 384 + up * 128 + ((chunk ^ (odd << 2) ^ (up << 1)) << 4) + (word & 3) * 4) =
                  rw_pair(w[i], odd);
            }
          }
          // Lane l < 16 takes rows 0-15 of its feature, lane l + 16 rows 16-31: each sends the half the other one needs.
          // Four rows of a lane at a time, in the staging tile before the next four: eight made the kernel spill.  Rows
          // past the tile's are neither stored nor worked on.  32 tokens over 6 of 64 experts each: layer 214 -> 211 us.
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            if (b * 32 + 4 * h >= t.rows) break;
            float gf[4], uf[4], zf[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const uint32_t lo = w[2 * h + i], hi = w[8 + 2 * h + i];
              const uint32_t o = __shfl_xor_sync(0xffffffffu, up ? lo : hi, 16);
              const uint32_t gw = up ? o : lo, uw = up ? hi : o;
              gf[2 * i] = __uint_as_float(gw << 16);
              gf[2 * i + 1] = __uint_as_float(gw & 0xffff0000u);
              uf[2 * i] = __uint_as_float(uw << 16);
              uf[2 * i + 1] = __uint_as_float(uw & 0xffff0000u);
            }
            swiglu_f32(gf, uf, zf, p.act);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int r = up * 16 + 4 * h + 2 * i + odd;
              *reinterpret_cast<uint32_t*>(stg + r * 384 + 256 + ((chunk ^ (odd << 2) ^ (up << 1)) << 4) + (word & 3) * 4) =
                  rw_pair(pack_bf16x2(zf[2 * i], zf[2 * i + 1]), odd);
            }
          }
        } else {
          const int word = lane >> 1;
          const int chunk = 4 * quad + (word >> 2);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int r = 2 * i + odd;
            *reinterpret_cast<uint32_t*>(stg + r * 256 + ((chunk ^ (odd << 2)) << 4) + (word & 3) * 4) = rw_pair(w[i], odd);
          }
        }
        asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "r"(128) : "memory");
        if (kSwiglu) {
          const int F = p.N / 2;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int r = quad * 8 + i * 4 + (lane >> 3), c = lane & 7;  // eight lanes per row and 128-byte piece
            const uint64_t h1 = __shfl_sync(0xffffffffu, my_row, r);
            const int col = m_blk * 64 + c * 8;
            if (b * 32 + r < t.rows && col + 8 <= F) {
              const uint8_t* src = stg + r * 384;
              const int sw = (r & 1) << 2;
              if (h1 != 0) {
                *reinterpret_cast<uint4*>(h1 + static_cast<uint64_t>(col) * 2) =
                    *reinterpret_cast<const uint4*>(src + ((c ^ sw) << 4));
                *reinterpret_cast<uint4*>(h1 + static_cast<uint64_t>(F + col) * 2) =
                    *reinterpret_cast<const uint4*>(src + 128 + ((c ^ sw ^ 2) << 4));
              }
              *reinterpret_cast<uint4*>(p.h2_base + h2_off + (static_cast<int64_t>(t.row0 + b * 32 + r) * F + col) * 2) =
                  *reinterpret_cast<const uint4*>(src + 256 + ((c ^ sw ^ ((r >> 4) << 1)) << 4));
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = quad * 8 + i * 2 + (lane >> 4), c = lane & 15;  // sixteen lanes per row
            const uint64_t rp = __shfl_sync(0xffffffffu, my_row, r);
            const int col = m_blk * kRwBM + c * 8;
            if (rp != 0 && col + 8 <= p.N)
              *reinterpret_cast<uint4*>(rp + static_cast<uint64_t>(col) * 2) =
                  *reinterpret_cast<const uint4*>(stg + r * 256 + ((c ^ ((r & 1) << 2)) << 4));
          }
        }
        my_row = next_row;
      }
      if (b_begin >= b_end) {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(lead_empty + buf * 8);
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
  if (abort_flag && threadIdx.x == 0) set_status(p.status, kPipelineTimeout, kMode, blockIdx.x);
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, kRwTmemCols);
  }
}

template <int kMode>
static int rows_launch(const RowsParams& p, int num_sms, cudaStream_t st) {
  static PerDeviceOnce attr_set;
  const int rc = once_per_device(attr_set, [] {
    return static_cast<int>(cudaFuncSetAttribute(rows_gemm_kernel<kMode>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(kRwDynSmem)));
  });
  if (rc != 0) return rc;
  const int grid = pair_grid(num_sms);
  rows_gemm_kernel<kMode><<<grid, kRwThreads, kRwDynSmem, st>>>(p);
  return static_cast<int>(cudaGetLastError());
}

// W13 = [expert][gate F | up F][K] as (K, 16 rows, gate/up, groups of 16, expert): one box of 64 K x 16 x 2 x 4 holds 64
// gate and the matching 64 up rows, alternating by 16.
static int encode_w13(CUtensorMap* tm, const void* w, int64_t experts, int64_t F, int64_t Kd) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return kRcNoDriver;
  const cuuint64_t pitch = static_cast<cuuint64_t>(Kd) * 2;
  cuuint64_t dims[5] = {static_cast<cuuint64_t>(Kd), 16, 2, static_cast<cuuint64_t>(F / 16), static_cast<cuuint64_t>(experts)};
  cuuint64_t strides[4] = {pitch, pitch * static_cast<cuuint64_t>(F), pitch * 16, pitch * 2 * static_cast<cuuint64_t>(F)};
  cuuint32_t box[5] = {64, 16, 2, 4, 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(w), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? kRcOk : 1000 + static_cast<int>(r);
}

}  // namespace dm

using namespace dm;

// gather_flags: a counter per 128-row block, then the ticket, then (kept clear) the CTAs that are finished.
static int64_t ticket_slot(int64_t max_rows) { return (max_rows + kRwGatherBlock - 1) / kRwGatherBlock; }

// What the forward and the input gradient share: row maps, row destinations, dispatch counters.
static int rows_setup(RowsParams& p, const dm_operand& a, const dm_operand& c, const int64_t* scatter_ptrs,
                      const int64_t* gather_ptrs, int32_t* gather_flags, const int32_t* expert_offsets, int e_local,
                      int64_t max_rows, int64_t N, int64_t Kd, const int* cond, int* status) {
  for (int i = 0; i < kRwBoxes; ++i) {
    const int rc = encode_arena(&p.tm_x[i], a, Kd * 2, max_rows + 256, rw_box_rows(i));
    if (rc != kRcOk) return rc;
  }
  p.a_off = a.offset;
  p.c_off = c.offset;
  p.c_base = static_cast<uint8_t*>(c.base);
  p.scatter_ptrs = scatter_ptrs;
  p.gather_ptrs = gather_ptrs;
  p.gather_flags = gather_ptrs ? gather_flags : nullptr;
  p.gather_ticket = gather_ptrs ? gather_flags + ticket_slot(max_rows) : nullptr;
  p.a_base = static_cast<uint8_t*>(a.base);
  p.expert_offsets = expert_offsets;
  p.cond = cond;
  p.status = status;
  p.e_local = e_local;
  p.max_rows = static_cast<int>(max_rows);
  p.N = static_cast<int>(N);
  p.Kd = static_cast<int>(Kd);
  return kRcOk;
}

// Takes DM_GATHER_FLAGS_KEPT_CLEAR out of num_sms; without it the flags are cleared in front of the launch.
static int clear_flags(RowsParams& p, int64_t max_rows, int& num_sms, cudaStream_t st) {
  if (p.gather_flags == nullptr) return kRcOk;
  static_assert(DM_GATHER_FLAGS_KEPT_CLEAR == kRwKeptClear, "the header's mark");
  if (rw_flags_kept_clear(num_sms)) {
    num_sms &= 0xffff;
    p.gather_done = p.gather_ticket + 1;
    return kRcOk;
  }
  return static_cast<int>(
      cudaMemsetAsync(p.gather_flags, 0, sizeof(int32_t) * static_cast<size_t>(ticket_slot(max_rows) + 1), st));
}

static int fprop_impl(dm_operand a, const void* w, dm_operand c, dm_operand h2, const int64_t* scatter_ptrs,
                      const int64_t* gather_ptrs, int32_t* gather_flags, const int32_t* expert_offsets, int e_local,
                      int64_t max_rows, int64_t N, int64_t Kd, int fuse_swiglu, int clamped, float alpha, float limit,
                      const int* cond, int num_sms, int* status, void* stream) {
  if (!a.base || !w || !expert_offsets || e_local <= 0 || max_rows < 0 || N <= 0 || Kd <= 0) return kRcBadArg;
  if (!c.base && !scatter_ptrs && !fuse_swiglu) return kRcBadArg;  // the fused forward may leave h1 out
  if (e_local > kRwMaxGroups || max_rows > (1 << 30)) return kRcTooLarge;
  if ((Kd % 64) != 0 || (N % 8) != 0) return kRcUnsupportedShape;
  if (fuse_swiglu && (((N / 2) % 128) != 0 || !h2.base || scatter_ptrs)) return kRcUnsupportedShape;
  if (max_rows == 0) return kRcOk;
  if (gather_ptrs != nullptr && gather_flags == nullptr) return kRcBadArg;
  RowsParams p{};
  int rc = rows_setup(p, a, c, scatter_ptrs, gather_ptrs, gather_flags, expert_offsets, e_local, max_rows, N, Kd, cond, status);
  if (rc != kRcOk) return rc;
  rc = fuse_swiglu ? encode_w13(&p.tm_w, w, e_local, N / 2, Kd)
                   : encode_2d(&p.tm_w, w, static_cast<int64_t>(e_local) * N, Kd, kRwBM);
  if (rc != kRcOk) return rc;
  p.h2_off = h2.offset;
  p.h2_base = static_cast<uint8_t*>(h2.base);
  p.act = ActParams{clamped, alpha, limit};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  rc = clear_flags(p, max_rows, num_sms, st);
  if (rc != kRcOk) return rc;
  return fuse_swiglu ? rows_launch<kRowsSwiglu>(p, num_sms, st) : rows_launch<kRowsFprop>(p, num_sms, st);
}

extern "C" int dm_gemm_fprop(dm_operand a, const void* w, dm_operand c, dm_operand h2, const int64_t* scatter_ptrs,
                             const int32_t* expert_offsets, int e_local, int64_t max_rows, int64_t N, int64_t Kd,
                             int fuse_swiglu, int clamped, float alpha, float limit, const int* cond, int num_sms,
                             int* status, void* stream) {
  return fprop_impl(a, w, c, h2, scatter_ptrs, nullptr, nullptr, expert_offsets, e_local, max_rows, N, Kd, fuse_swiglu,
                    clamped, alpha, limit, cond, num_sms, status, stream);
}

extern "C" int dm_gemm_fprop_dispatch(const int64_t* gather_ptrs, int32_t* gather_flags, dm_operand a, const void* w,
                                      dm_operand c, dm_operand h2, const int32_t* expert_offsets, int e_local,
                                      int64_t max_rows, int64_t N, int64_t Kd, int fuse_swiglu, int clamped,
                                      float alpha, float limit, const int* cond, int num_sms, int* status,
                                      void* stream) {
  if (!gather_ptrs || !gather_flags) return kRcBadArg;
  return fprop_impl(a, w, c, h2, nullptr, gather_ptrs, gather_flags, expert_offsets, e_local, max_rows, N, Kd,
                    fuse_swiglu, clamped, alpha, limit, cond, num_sms, status, stream);
}

static int dgrad_impl(dm_operand a, const void* w, dm_operand c, const int64_t* scatter_ptrs,
                      const int64_t* gather_ptrs, int32_t* gather_flags, const int32_t* expert_offsets, int e_local,
                      int64_t max_rows, int64_t N, int64_t Kd, const int* cond, int num_sms, int* status,
                      void* stream) {
  if (!a.base || !w || !expert_offsets || e_local <= 0 || max_rows < 0 || N <= 0 || Kd <= 0) return kRcBadArg;
  if (!c.base && !scatter_ptrs) return kRcBadArg;
  if (e_local > kRwMaxGroups || max_rows > (1 << 30)) return kRcTooLarge;
  if ((Kd % 64) != 0 || (N % 8) != 0) return kRcUnsupportedShape;
  if (max_rows == 0) return kRcOk;
  if (gather_ptrs != nullptr && gather_flags == nullptr) return kRcBadArg;
  RowsParams p{};
  int rc = rows_setup(p, a, c, scatter_ptrs, gather_ptrs, gather_flags, expert_offsets, e_local, max_rows, N, Kd, cond, status);
  if (rc != kRcOk) return rc;
  // W = [e_local * Kd][N], N contiguous; box = 64 k-rows x 64 columns.
  rc = encode_2d(&p.tm_w, w, static_cast<int64_t>(e_local) * Kd, N, 64);
  if (rc != kRcOk) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  rc = clear_flags(p, max_rows, num_sms, st);
  if (rc != kRcOk) return rc;
  return rows_launch<kRowsDgrad>(p, num_sms, st);
}

extern "C" int dm_gemm_dgrad(dm_operand a, const void* w, dm_operand c, const int64_t* scatter_ptrs,
                             const int32_t* expert_offsets, int e_local, int64_t max_rows, int64_t N, int64_t Kd,
                             const int* cond, int num_sms, int* status, void* stream) {
  return dgrad_impl(a, w, c, scatter_ptrs, nullptr, nullptr, expert_offsets, e_local, max_rows, N, Kd, cond, num_sms,
                    status, stream);
}

extern "C" int dm_gemm_dgrad_dispatch(const int64_t* gather_ptrs, int32_t* gather_flags, dm_operand a, const void* w,
                                      dm_operand c, const int32_t* expert_offsets, int e_local, int64_t max_rows,
                                      int64_t N, int64_t Kd, const int* cond, int num_sms, int* status, void* stream) {
  if (!gather_ptrs || !gather_flags) return kRcBadArg;
  return dgrad_impl(a, w, c, nullptr, gather_ptrs, gather_flags, expert_offsets, e_local, max_rows, N, Kd, cond,
                    num_sms, status, stream);
}
