// Persistent grouped BF16 weight-gradient GEMM on tcgen05 tensor cores (sm_100a).
//
//   wgrad  dW[e][n][k] (+)= sum_r dY[r,n] X[r,k] both operands MN-major; the ragged last
//          64-row chunk of an expert is zeroed in shared memory before the MMA reads it.
//
// One CTA per SM, warp-specialised:
//   warps 0, 10, 11  TMA producers: fill a 4-stage shared-memory ring (dY 64 rows x 128, X 64 rows x 256, boxes of 64 x
//               64, 128-byte swizzle) with cp.async.bulk.tensor loads, no multicast.
//   warp 1      MMA issuer: owns the TMEM allocation (512 columns = two 128x256 fp32
//               accumulators), stays converged around an elected lane's tcgen05.mma (M128 N256 K16)
//               and releases stages / publishes accumulators with tcgen05.commit.
//   warps 2..9  epilogue (two per TMEM lane quadrant): tcgen05.ld their 32 TMEM lanes, convert and store or add into dW
//               while the next tile's main loop already runs.
//   warp 14     accumulator watcher.
//
// Bound: operand loads from L2 (48 KiB per 64-row stage and 128x256 tile) and, with few rows per expert, dW itself.  The
// issuing warps stay converged (one lane in a divergent branch before): W13 8 experts x 3072 rows, D 2048, F 1408,
// accumulated in place, 265 -> 215 us (1312 TFLOP/s); 64 x 384 359 -> 351 us.
//
// Groups are the local experts; their row ranges come from device memory
// (expert_offsets), so the tile list is built by every CTA at kernel start and no
// host read is needed.  Operands are addressed as (arena base, device
// byte offset): the tensor map views the whole arena as [row][128-byte line][64 bf16]
// with overlapping strides, so a planner-chosen offset only changes a coordinate.
#include "gemm_common.cuh"

namespace dm {

constexpr int kBM = 128;
constexpr int kBN = 256;
constexpr int kBK = 64;
constexpr int kStages = 4;
constexpr int kGemmThreads = 480;  // TMA warp, MMA warp, eight epilogue warps, two more TMA warps, one accumulator watcher
constexpr int kMaxGroups = 256;
constexpr uint32_t kABytes = kBM * kBK * 2;  // 16 KiB
constexpr uint32_t kBBytes = kBN * kBK * 2;  // 32 KiB
constexpr uint32_t kStageBytes = kABytes + kBBytes;
constexpr uint32_t kTmemCols = 512;
constexpr size_t kGemmSmemBytes = kStages * kStageBytes + 8 * kStaging64Bytes + 1024;  // + slack for 1024-byte alignment

struct GemmParams {
  CUtensorMap tm_a;
  CUtensorMap tm_b;
  CUtensorMap tm_c;     // dW as [e_local][N][Kd], boxes of 16 rows x 128 bytes
  const int64_t* a_off;  // device byte offsets (may be null = 0)
  const int64_t* b_off;
  const int32_t* expert_offsets;
  int* status;
  int e_local;
  int max_rows;
  int N;   // dW rows
  int Kd;  // dW columns
  int out_fp32;
  int accumulate;
};

struct Tile {
  int e, m_blk, n_blk, row0, row_end, k_iters;
};

__device__ __forceinline__ Tile decode_tile(int tile, int& e, const int* tile_start, const int* off, int n_tiles) {
  while (tile >= tile_start[e + 1]) ++e;
  const int local = tile - tile_start[e];
  Tile t;
  t.e = e;
  t.n_blk = local % n_tiles;
  t.m_blk = local / n_tiles;
  t.row0 = off[e];
  t.row_end = off[e + 1];
  t.k_iters = (off[e + 1] - off[e] + kBK - 1) / kBK;
  return t;
}

__global__ void __launch_bounds__(kGemmThreads, 1) wgrad_gemm_kernel(const __grid_constant__ GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  __shared__ uint64_t full_bar[kStages];
  __shared__ uint64_t empty_bar[kStages];
  __shared__ uint64_t tmem_full_bar[2];
  __shared__ uint64_t tmem_empty_bar[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ uint32_t s_stop[4];  // where the three producers and the issuer stopped
  __shared__ int abort_flag;
  __shared__ volatile int s_first_bad;  // first of this CTA's tiles whose accumulator never came
  __shared__ int s_off[kMaxGroups + 1];
  __shared__ int s_tile_start[kMaxGroups + 1];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  const int64_t a_off = p.a_off ? *p.a_off : 0, b_off = p.b_off ? *p.b_off : 0;  // on their way while the tables are built

  // ---- tile table -----------------------------------------------------------
  const int n_tiles = (p.Kd + kBN - 1) / kBN;
  const int m_tiles = (p.N + kBM - 1) / kBM;
  for (int i = threadIdx.x; i <= p.e_local; i += blockDim.x) {
    int v = p.expert_offsets[i];
    s_off[i] = v < p.max_rows ? v : p.max_rows;
  }
  if (threadIdx.x == 0) {
    abort_flag = 0;
    s_first_bad = kNoBadTile;
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full_bar[b], 1);
      mbar_init(&tmem_empty_bar[b], 8);
    }
    mbar_fence_init();
  }
  for (int e = threadIdx.x; e <= p.e_local; e += blockDim.x) s_tile_start[e] = e * m_tiles * n_tiles;
  if (warp == 1) {
    tmem_alloc(&tmem_base_slot, kTmemCols);
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


  // Weight gradient: a stage is six 64 x 64 boxes, and one thread cannot issue six TMA loads in the time the
  // tensor cores need for the stage, so the (otherwise idle) warps 10 and 11 issue the boxes of the second
  // operand; warp 0 arms the stage's barrier and loads the first operand.
  const int wgrad_part = warp == 0 ? 0 : (warp == 10 ? 1 : (warp == 11 ? 2 : -1));
  if (warp == 0 || wgrad_part > 0) {
    // ======================= TMA producer =======================
    const bool elected = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    int e = 0;
    const int a_line0 = uniform(static_cast<int>(a_off >> 7));
    const int b_line0 = uniform(static_cast<int>(b_off >> 7));
    bool ok = true;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
      const Tile t = decode_tile(tile, e, s_tile_start, s_off, n_tiles);
      const int k_iters = uniform(t.k_iters), row0 = uniform(t.row0);
      const int line = wgrad_part == 0 ? a_line0 + uniform(t.m_blk) * (kBM / 64)
                                       : b_line0 + uniform(t.n_blk) * (kBN / 64) + (wgrad_part - 1) * 2;
      const uint32_t dst = wgrad_part == 0 ? 0u : kABytes + (wgrad_part - 1) * 16384u;
      const CUtensorMap* map = wgrad_part == 0 ? &p.tm_a : &p.tm_b;
#pragma unroll 1
      for (int kb = 0; kb < k_iters; ++kb) {
        ok = warp_mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_flag);
        if (!ok) break;
        uint8_t* box = smem + stage * kStageBytes + dst;
        if (elected) {
          if (wgrad_part == 0) mbar_arrive_expect_tx(&full_bar[stage], kStageBytes);
          tma_load_3d(box, map, 0, line, row0 + kb * kBK, &full_bar[stage]);
          tma_load_3d(box + 8192, map, 0, line + 1, row0 + kb * kBK, &full_bar[stage]);
        }
        __syncwarp();
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (lane == 0) s_stop[wgrad_part] = ring_stop(stage, phase);
  } else if (warp == 1) {
    // ======================= MMA issuer =======================
    // The warp stays converged around the elected lane's instructions (see "Issuing warps"); the next stage's barrier is
    // looked at while this stage's MMAs are on their way.  All lanes zero the tail rows of a ragged last chunk.
    constexpr uint32_t idesc = umma_idesc_bf16(kBM, kBN, 1, 1);
    constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO 1024, version 1, 128-byte swizzle
    constexpr uint32_t kLboMN = (8192u >> 4) << 16;
    constexpr uint32_t k_step = 2048u >> 4;  // 16 rows of both operands
    const bool elected = elect_one();
    const uint32_t a_lo0 = uniform(((smem_u32(smem) & 0x3ffffu) >> 4) | kLboMN);
    const uint32_t full0 = uniform(smem_u32(&full_bar[0])), empty0 = uniform(smem_u32(&empty_bar[0]));
    const uint32_t tfull0 = uniform(smem_u32(&tmem_full_bar[0]));
    int stage = 0;
    uint32_t phase = 0, ready = 0;  // ready: the current stage is known to be full
    int e = 0;
    int it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++it) {
      const Tile t = decode_tile(tile, e, s_tile_start, s_off, n_tiles);
      const int k_iters = uniform(t.k_iters);
      const int buf = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1u;
      const uint32_t d_tmem = tmem_base + buf * kBN;
      const int valid_last = uniform((t.row_end - t.row0) - (t.k_iters - 1) * kBK);  // rows of the last chunk
      ok = warp_mbar_wait(&tmem_empty_bar[buf], acc_phase ^ 1u, &abort_flag);
      if (!ok) break;
      tcgen05_fence_after();
      uint32_t acc = 0;
#pragma unroll 1
      for (int kb = 0; kb < k_iters; ++kb) {
        if (!__all_sync(0xffffffffu, ready)) {
          ok = warp_mbar_wait(&full_bar[stage], phase, &abort_flag);
          if (!ok) break;
        }
        int ksteps = kBK / 16;
        if (kb == k_iters - 1) {
          // Only the K = 16 steps that hold rows of this expert are issued, and the rows between the expert's end and the
          // end of its last step (at most 15) are zeroed.  Row r of every 64 x 64 box is one contiguous 128-byte line.
          ksteps = (valid_last + 15) >> 4;
          if ((valid_last & 15) != 0) {
            uint8_t* sa = smem + stage * kStageBytes;
            const int vec_per_box = (ksteps * 16 - valid_last) * 8;
            const int boxes = (kBM + kBN) / 64;
            for (int i = lane; i < boxes * vec_per_box; i += 32) {
              const int box = i / vec_per_box, v = i - box * vec_per_box;
              reinterpret_cast<uint4*>(sa + box * 8192 + valid_last * 128)[v] = make_uint4(0, 0, 0, 0);
            }
            fence_proxy_async_smem();
            __syncwarp();
          }
        }
        const uint32_t a_lo = a_lo0 + stage * (kStageBytes >> 4), b_lo = a_lo + (kABytes >> 4);
        const uint32_t empty = empty0 + stage * 8;
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
        ready = mbar_test(full0 + stage * 8, phase);
        if (elected) {
          umma_bf16_lo(d_tmem, a_lo, b_lo, kDescHi, idesc, acc);
          if (ksteps > 1) umma_bf16_lo(d_tmem, a_lo + k_step, b_lo + k_step, kDescHi, idesc, 1u);
          if (ksteps > 2) umma_bf16_lo(d_tmem, a_lo + 2 * k_step, b_lo + 2 * k_step, kDescHi, idesc, 1u);
          if (ksteps > 3) umma_bf16_lo(d_tmem, a_lo + 3 * k_step, b_lo + 3 * k_step, kDescHi, idesc, 1u);
          tcgen05_commit_addr(empty);
        }
        __syncwarp();
        acc = 1;
      }
      if (!ok) break;
      if (elected) {
        if (k_iters > 0)
          tcgen05_commit_addr(tfull0 + buf * 8);
        else
          mbar_arrive(&tmem_full_bar[buf]);
      }
      __syncwarp();
    }
    if (lane == 0) s_stop[3] = ring_stop(stage, phase);
  } else if (warp == 14) {
    // ======================= accumulator watcher =======================
    // One warp polls the accumulator-ready barriers on behalf of the eight epilogue warps and releases them
    // through a hardware named barrier: the epilogue warps then sleep without taking issue slots from the
    // MMA-issuing and TMA-issuing threads that share their schedulers.  After a timeout it releases them once more and stops.
    bool ok = true;
    int it = 0;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++it) {
      const int buf = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1u;
      if (lane == 0) ok = handover_report(&s_first_bad, it, mbar_wait(&tmem_full_bar[buf], acc_phase, &abort_flag));
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      asm volatile("bar.arrive %0, %1;" ::"r"(handover_barrier(it)), "r"(8 * 32 + 32) : "memory");
    }
  } else if (warp < 10) {
    // ======================= epilogue =======================
    // Eight warps: two per TMEM lane quadrant, each owning half of the tile's columns.
    const int ew = warp - 2;            // 0..7
    const int quad = warp & 3;          // TMEM lanes [32*quad, 32*quad+32)
    const int half = ew >> 2;           // column half of the tile
    uint8_t* stg = smem + kStages * kStageBytes + ew * kStaging64Bytes;
    int e = 0;
    int it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++it) {
      const Tile t = decode_tile(tile, e, s_tile_start, s_off, n_tiles);
      const int buf = it & 1;
      asm volatile("bar.sync %0, %1;" ::"r"(handover_barrier(it)), "r"(8 * 32 + 32) : "memory");  // released by the watcher
      ok = handover_good(&s_first_bad, it);  // the same for every epilogue warp
      if (!ok) break;
      tcgen05_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + buf * kBN;
      {
        // 128 bytes of output columns per trip (64 bf16 or 32 fp32).  The staging tile is laid out as a 16-row x
        // 128-byte box in the 128-byte swizzle, so the warp's 32 rows go in two passes; one thread hands each
        // box to the copy engine, which stores it or adds it to dW in L2 (accumulation rounds the fp32
        // accumulator to the stored type first, then L2 adds whole 128-byte lines: no read round trip through
        // the SM) and clips rows and columns past the matrix.
        const int cols_per_trip = p.out_fp32 ? 32 : 64;
        for (int c0 = half * (kBN / 2); c0 < (half + 1) * (kBN / 2); c0 += cols_per_trip) {
          uint32_t r0[32], r1[32];
          if (t.k_iters > 0) {
            tmem_ld_32x32(taddr + c0, r0);
            if (!p.out_fp32) tmem_ld_32x32(taddr + c0 + 32, r1);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) r0[j] = r1[j] = 0u;
          }
          const int cc = t.n_blk * kBN + c0;
#pragma unroll
          for (int pass = 0; pass < 2; ++pass) {
            if (lane == 0) bulk_wait_read();  // the engine has read the previous box out of the staging tile
            __syncwarp();
            if ((lane >> 4) == pass) {
              const int rr = lane & 15;
              if (p.out_fp32) {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  stage_put(stg, rr, j, make_uint4(r0[4 * j], r0[4 * j + 1], r0[4 * j + 2], r0[4 * j + 3]));
              } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  stage_put(stg, rr, j, pack8_bf16(r0 + 8 * j));
                  stage_put(stg, rr, j + 4, pack8_bf16(r1 + 8 * j));
                }
              }
            }
            fence_proxy_async_smem();
            __syncwarp();
            const int box_row = t.m_blk * kBM + quad * 32 + pass * 16;
            if (lane == 0 && box_row < p.N && cc < p.Kd) {
              if (p.accumulate)
                tma_reduce_add_3d(&p.tm_c, stg, cc, box_row, t.e);
              else
                tma_store_3d(&p.tm_c, stg, cc, box_row, t.e);
              bulk_commit();
            }
          }
        }
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty_bar[buf]);
    }
    if (lane == 0) bulk_wait_all();  // staged boxes are out of shared memory and written
  }

  // ---- teardown ---------------------------------------------------------------
  tcgen05_fence_before();
  __syncthreads();
  if (abort_flag) {
    if (threadIdx.x == 0) {
      set_status(p.status, kPipelineTimeout, 2, blockIdx.x);
      const uint64_t deadline = globaltimer_ns() + kSettleNs;
      settle_ring(empty_bar, kStages, s_stop[3], deadline);
      for (int i = 0; i < 3; ++i) settle_ring(full_bar, kStages, s_stop[i], deadline);
    }
    __syncthreads();
  }
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

static int launch(const GemmParams& p, int num_sms, cudaStream_t st) {
  static PerDeviceOnce attr_set;
  const int rc = once_per_device(attr_set, [] {
    return static_cast<int>(cudaFuncSetAttribute(wgrad_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(kGemmSmemBytes)));
  });
  if (rc != 0) return rc;
  const int grid = persistent_grid(num_sms);
  wgrad_gemm_kernel<<<grid, kGemmThreads, kGemmSmemBytes, st>>>(p);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace dm

using namespace dm;

extern "C" int dm_gemm_wgrad(dm_operand dy, dm_operand x, void* dw, int out_is_fp32, int accumulate,
                             const int32_t* expert_offsets, int e_local, int64_t max_rows, int64_t N, int64_t Kd,
                             int num_sms, int* status, void* stream) {
  if (!dy.base || !x.base || !dw || !expert_offsets || e_local <= 0 || max_rows < 0 || N <= 0 || Kd <= 0)
    return kRcBadArg;
  if (e_local > kMaxGroups || max_rows > (1 << 30)) return kRcTooLarge;
  if ((N % 64) != 0 || (Kd % 64) != 0) return kRcUnsupportedShape;
  if ((reinterpret_cast<uintptr_t>(dw) % 16) != 0) return kRcBadArg;
  GemmParams p{};
  int rc = encode_arena(&p.tm_a, dy, N * 2, max_rows + 256, kBK);
  if (rc != kRcOk) return rc;
  rc = encode_arena(&p.tm_b, x, Kd * 2, max_rows + 256, kBK);
  if (rc != kRcOk) return rc;
  p.a_off = dy.offset;
  p.b_off = x.offset;
  p.expert_offsets = expert_offsets;
  p.status = status;
  p.e_local = e_local;
  p.max_rows = static_cast<int>(max_rows);
  p.N = static_cast<int>(N);
  p.Kd = static_cast<int>(Kd);
  p.out_fp32 = out_is_fp32 ? 1 : 0;
  p.accumulate = accumulate ? 1 : 0;
  rc = encode_out_3d(&p.tm_c, dw, e_local, N, Kd, out_is_fp32 != 0);
  if (rc != kRcOk) return rc;
  return launch(p, num_sms, static_cast<cudaStream_t>(stream));
}
