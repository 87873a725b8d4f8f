// Helpers shared by the grouped GEMM kernels: issue loops, epilogue staging tile, L2 reductions and the
// host-side tensor-map encoding (through the driver entry point, no link-time libcuda).
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "tile_handover.cuh"
#include "../../include/dist_moe_b200.h"

namespace dm {

constexpr uint32_t kStaging64Bytes = 32 * 64;  // per epilogue warp: 32 rows x 64 bytes, or 16 rows x 128 bytes

// Staging tile of one epilogue warp: row r is 128 bytes, its 16-byte chunk j sits at j ^ (r & 7) (the 128-byte swizzle).
__device__ __forceinline__ void stage_put(uint8_t* stg, int row, int chunk, uint4 v) {
  reinterpret_cast<uint4*>(stg + row * 128)[chunk ^ (row & 7)] = v;
}
// 64-byte variant: row r is 64 bytes, its 16-byte chunk j sits at j ^ ((r >> 1) & 3).
__device__ __forceinline__ void stage64_put(uint8_t* stg, int row, int chunk, uint4 v) {
  reinterpret_cast<uint4*>(stg + row * 64)[chunk ^ ((row >> 1) & 3)] = v;
}
__device__ __forceinline__ uint4 stage64_get(const uint8_t* stg, int row, int chunk) {
  return reinterpret_cast<const uint4*>(stg + row * 64)[chunk ^ ((row >> 1) & 3)];
}
__device__ __forceinline__ uint4 pack8_bf16(const uint32_t* r) {
  return make_uint4(pack_bf16x2(__uint_as_float(r[0]), __uint_as_float(r[1])),
                    pack_bf16x2(__uint_as_float(r[2]), __uint_as_float(r[3])),
                    pack_bf16x2(__uint_as_float(r[4]), __uint_as_float(r[5])),
                    pack_bf16x2(__uint_as_float(r[6]), __uint_as_float(r[7])));
}

// 16 bytes to global memory (a peer's included).  Through a generic pointer the store might alias the staging tile, and the
// next read of the tile would wait for it.
__device__ __forceinline__ void store_global16(uint64_t addr, uint4 v) {
  asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w));
}

// ---------------------------------------------------------------------------
// Issuing warps.  tcgen05 and TMA instructions take their operands from uniform registers.  Code that only one lane runs
// (`if (lane == 0)`) keeps everything in per-lane registers and moves each operand over for each instruction: 85 to 93
// cycles per tcgen05.mma, measured.  The issuing warps here stay converged instead: all lanes walk the loop, values that
// come from memory are made uniform with a shuffle, and only the instruction itself is behind the elected lane's
// predicate: 39 cycles per tcgen05.mma of N <= 32 with its share of the loop, and N / 2 from N = 128 up (the pipe's rate).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }
// Bounded wait of a whole converged warp; every lane has seen the phase complete when it returns true.
__device__ __forceinline__ bool warp_mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

// One warp builds a launch's tables: the groups' offsets (bounded by max_rows) and the first tile of every expert.  `tiles(e, lo, hi,
// count)` tells how many tiles expert e's rows [lo, hi) make, `count` of them real (max_rows without counts).  All of its loads
// are on their way before the first is used, and nothing waits for another warp.  With the offsets loaded by all threads and a block
// barrier before the tables, a launch's first weight load came 4400 to 5200 cycles after its start (8 to 24 experts), so 3700 to
// 4600; MXFP8 decode (128 experts, two launches) 213.6 -> 208.6 us.
constexpr int kTableExperts = 256;
template <class Tiles>
__device__ __forceinline__ void tile_tables(const int32_t* offsets, const int32_t* counts, int e_local, int max_rows, int lane,
                                            int* s_off, int* s_tile_start, Tiles&& tiles) {
  int lo[kTableExperts / 32], hi[kTableExperts / 32], count[kTableExperts / 32];
#pragma unroll
  for (int c = 0; c < kTableExperts / 32; ++c) {
    const int e = 32 * c + lane;
    lo[c] = hi[c] = 0;
    count[c] = max_rows;
    if (e < e_local) {
      lo[c] = offsets[e];
      hi[c] = offsets[e + 1];
      if (counts != nullptr) count[c] = counts[e];
    }
  }
  int running = 0;
#pragma unroll
  for (int c = 0; c < kTableExperts / 32; ++c) {
    if (32 * c >= e_local) break;
    const int e = 32 * c + lane;
    const int l = min(lo[c], max_rows), h = min(hi[c], max_rows);
    const int own = e < e_local ? tiles(e, l, h, count[c]) : 0;
    int incl = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += t;
    }
    if (e < e_local) {
      s_off[e] = l;
      s_tile_start[e] = running + incl - own;
      if (e == e_local - 1) s_off[e_local] = h;
    }
    running += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) s_tile_start[e_local] = running;
}

// After a wait ran out: a role's copies or MMAs that are still in flight have to end before the block gives its shared
// memory and tensor memory back.  `bar` holds the barriers they complete, `stop` says where the role stopped.  Returns at
// the deadline where a stage never completes (it was left half filled; what was issued for it has landed by then).
__device__ __forceinline__ void settle_ring(uint64_t* bar, int stages, uint32_t stop, uint64_t deadline_ns) {
  for (int s = 0; s < stages; ++s)
    while (!mbar_try_wait(&bar[s], ring_last_parity(stop, s)))
      if (globaltimer_ns() > deadline_ns) return;
}
constexpr uint64_t kSettleNs = 1000000;  // a millisecond; loads take microseconds

// One look at a barrier that never suspends the thread: asked for the next stage before this stage's MMAs are issued, its
// latency hides behind them.
__device__ __forceinline__ uint32_t mbar_test(uint32_t bar_addr, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok) : "r"(bar_addr), "r"(parity) : "memory");
  return ok;
}

// MMAs and commits for the issue loops: barriers given by their shared-memory address, shared-memory matrix descriptors by
// their lower word (address >> 4 | LBO >> 4 << 16) and a constant upper word (SBO >> 4, version 1 in bit 14, 128-byte
// swizzle 2 in bits 29 to 31).  K-major operand: rows of 128 bytes, 8-row groups SBO = 1024 apart.  MN-major operand: lines
// of 128 bytes of M or N, one line per k, 8-k groups SBO = 1024 apart, the next 128 bytes of M or N LBO apart.
__device__ __forceinline__ void umma_bf16_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t"
      "}\n"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Block-scaled MMAs: scale factors live in TMEM (copied there by tcgen05.cp from shared memory).
__device__ __forceinline__ void umma_mxf8_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc,
                                             uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], da, db, %4, [%6], [%7], p;\n\t"
      "}\n"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)
      : "memory");
}
__device__ __forceinline__ void umma_nvf4_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc,
                                             uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], da, db, %4, [%6], [%7], p;\n\t"
      "}\n"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)
      : "memory");
}
// Scale atoms (512 bytes each) by the lower word of their no-swizzle descriptor: rows 16 bytes apart, 8-row groups 128.  An
// atom (32 rows x 16 bytes in shared memory) goes to 4 TMEM columns, replicated over the four 32-lane sub-partitions.
constexpr uint32_t kSfAtomWords = 512u >> 4;
__device__ __forceinline__ uint32_t sf_desc_lo(uint32_t smem_addr) { return ((smem_addr & 0x3ffffu) >> 4) | ((16u >> 4) << 16); }
__device__ __forceinline__ void tmem_cp_sf_lo(uint32_t taddr, uint32_t lo) {
  asm volatile(
      "{\n\t"
      ".reg .b64 d;\n\t"
      "mov.b64 d, {%1, %2};\n\t"
      "tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], d;\n\t"
      "}\n"
      ::"r"(taddr), "r"(lo), "n"((128 >> 4) | (1 << 14))
      : "memory");
}
__device__ __forceinline__ void tcgen05_commit_addr(uint32_t bar_addr) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_addr) : "memory");
}

// ---------------------------------------------------------------------------
// CTA pairs (clusters of two, tcgen05 cta_group::2).  The even CTA leads: it issues the MMAs of both, and its stage
// barriers count the bytes that both CTAs load, each into its own shared memory.  No load is multicast.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Address of the same shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t smem_addr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The two halves of it: what was done before a thread's arrival is seen by every thread that has waited.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Loads whose bytes count on the leader's barrier (`bar`: its shared::cluster address).
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const void* tmap, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const void* tmap, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_load_5d_pair(void* smem_dst, const void* tmap, int c0, int c1, int c2, int c3, int c4,
                                                 uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, "
      "%7}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}
__device__ __forceinline__ void umma_bf16_lo_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi,
                                                  uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p;\n\t"
      "}\n"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_mxf8_lo_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi,
                                                  uint32_t idesc, uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], da, db, %4, [%6], [%7], p;\n\t"
      "}\n"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)
      : "memory");
}
__device__ __forceinline__ void umma_nvf4_lo_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi,
                                                  uint32_t idesc, uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], da, db, %4, [%6], [%7], p;\n\t"
      "}\n"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)
      : "memory");
}
// Both CTAs copy the atom at this offset of their own shared memory to these columns of their own TMEM.
__device__ __forceinline__ void tmem_cp_sf_lo_pair(uint32_t taddr, uint32_t lo) {
  asm volatile(
      "{\n\t"
      ".reg .b64 d;\n\t"
      "mov.b64 d, {%1, %2};\n\t"
      "tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], d;\n\t"
      "}\n"
      ::"r"(taddr), "r"(lo), "n"((128 >> 4) | (1 << 14))
      : "memory");
}
// Arrive on the barrier at this shared-memory offset in both CTAs of the pair once the MMAs issued so far are complete.
__device__ __forceinline__ void tcgen05_commit_pair(uint32_t bar_addr) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar_addr),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}

// Bulk tensor store and reduce-add of one staged box (shared memory -> global), issued by one thread.  The
// staged bytes must have been made visible to the async proxy (fence_proxy_async_smem by every writer, then
// a barrier) and stay untouched until bulk_wait_read has returned.
__device__ __forceinline__ void tma_store_3d(const void* tmap, const void* smem_src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(tmap)),
               "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add_3d(const void* tmap, const void* smem_src, int c0, int c1, int c2) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(tmap)),
               "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---------------------------------------------------------------------------
// Host side: tensor-map encoding through the driver entry point (no link-time
// dependency on libcuda) and launch.
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static inline EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
  }
  return fn;
}

// Grid of a persistent kernel of CTA pairs, one CTA per SM: whole pairs within the caller's limit (one less for an odd
// limit), at least one pair.
static inline int pair_grid(int num_sms) {
  const int pairs = persistent_grid(num_sms) / 2;
  return 2 * (pairs > 0 ? pairs : 1);
}

// bf16 matrix [rows][cols], cols contiguous; box = box_rows x 64 columns.
static inline int encode_2d(CUtensorMap* tm, const void* base, int64_t rows, int64_t cols, int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return kRcNoDriver;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * 2};
  cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? kRcOk : 1000 + static_cast<int>(r);
}

// Arena view: element (c0, line, row) lives at base + 2*c0 + 128*line + pitch*row.
// `line` spans the whole allocation, so an operand at byte offset o is reached
// with line = o/128 + column/64; rows may run `guard` rows past the operand.
static inline int encode_arena(CUtensorMap* tm, const dm_operand& op, int64_t pitch_bytes, int64_t rows, int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return kRcNoDriver;
  const int64_t lines = op.bytes / 128;
  if (lines <= 0 || (pitch_bytes % 128) != 0 || (reinterpret_cast<uintptr_t>(op.base) % 128) != 0) return kRcBadArg;
  cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(lines), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[2] = {128, static_cast<cuuint64_t>(pitch_bytes)};
  cuuint32_t box[3] = {64, 1, static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, op.base, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? kRcOk : 1000 + static_cast<int>(r);
}

// Weight-gradient destination [groups][rows][cols] (bf16 or fp32), boxes of 16 rows x 128 bytes in the 128-byte swizzle:
// the layout of an epilogue warp's staging tile, and whole 128-byte lines of dW per store or reduce-add.
static inline int encode_out_3d(CUtensorMap* tm, void* base, int64_t groups, int64_t rows, int64_t cols, bool fp32) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return kRcNoDriver;
  const cuuint64_t esz = fp32 ? 4 : 2;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(groups)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(cols) * esz, static_cast<cuuint64_t>(cols) * rows * esz};
  cuuint32_t box[3] = {static_cast<cuuint32_t>(128 / esz), 16, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(tm, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides,
                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? kRcOk : 1000 + static_cast<int>(r);
}

// Byte-typed variants for quantised operands: rows of `row_bytes`, boxes of 128 bytes x box_rows.
static inline int encode_2d_u8(CUtensorMap* tm, const void* base, int64_t rows, int64_t row_bytes, int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return kRcNoDriver;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(row_bytes), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_bytes)};
  cuuint32_t box[2] = {128, static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? kRcOk : 1000 + static_cast<int>(r);
}

static inline int encode_arena_u8(CUtensorMap* tm, const dm_operand& op, int64_t pitch_bytes, int64_t rows,
                                  int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return kRcNoDriver;
  const int64_t lines = op.bytes / 128;
  if (lines <= 0 || (pitch_bytes % 128) != 0 || (reinterpret_cast<uintptr_t>(op.base) % 128) != 0) return kRcBadArg;
  cuuint64_t dims[3] = {128, static_cast<cuuint64_t>(lines), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[2] = {128, static_cast<cuuint64_t>(pitch_bytes)};
  cuuint32_t box[3] = {128, 1, static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, op.base, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? kRcOk : 1000 + static_cast<int>(r);
}

// Scales as lines that start every 128 bytes, boxes of `lines` lines (an atom has four); base 16-byte aligned.  The rows' lines
// are 256 bytes long and overlap: an atom that starts at word x < 32 of line l is the box at (x, l), contiguous as stored.
// (Two maps, chosen in the kernel by the offset, cost 2 of 220 us: 16 tokens, 128 experts x 2816 x 2816.)
static inline int encode_sf(CUtensorMap* tm, const void* base, int64_t bytes, bool overlap, int lines = 4) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return kRcNoDriver;
  if (bytes < 128) return kRcBadArg;
  cuuint64_t dims[2] = {overlap ? 64u : 32u, static_cast<cuuint64_t>(bytes / 128)};
  cuuint64_t strides[1] = {128};
  cuuint32_t box[2] = {32, static_cast<cuuint32_t>(lines)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? kRcOk : 1000 + static_cast<int>(r);
}

}  // namespace dm
