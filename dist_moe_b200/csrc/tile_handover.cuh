// What the roles of a persistent GEMM tell one another when a wait has run out.  Plain code, for the kernels and for host
// code.
//
// The watcher waits (bounded) for the accumulators of the CTA's tiles in turn and arrives at the tile's named barrier, where
// the epilogue warps wait for it.  Where an accumulator never comes it records the tile, arrives once more, so that the
// epilogue warps get past that barrier, and stops: another arrival could stand in for an epilogue warp that is still busy
// with the tile before, which would then wait alone.  The epilogue warps decide by the record, which is written before the
// arrival that releases them, and so take the same decision; a flag that other roles may raise at any moment would let some
// of them leave while the others wait for all of them at the next tile.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define DM_HANDOVER __host__ __device__ __forceinline__
#else
#define DM_HANDOVER inline
#endif

namespace dm {

constexpr int kNoBadTile = 0x7fffffff;

// Named barriers 1 to 3 take turns.  An accumulator comes only after the epilogue warps have handed back the one of two tiles
// before, so when the watcher arrives for a tile, all of them are past the barrier of three tiles before, but one may still
// be on its way to that of two tiles before, however long the watcher has waited.
constexpr int kHandoverBarriers = 3;
DM_HANDOVER int handover_barrier(int it) { return 1 + it % kHandoverBarriers; }

// Watcher, before its arrival for tile `it`: returns whether it goes on with the next tile.
DM_HANDOVER bool handover_report(volatile int* first_bad, int it, bool came) {
  if (!came) *first_bad = it;
  return came;
}

// Epilogue warps, after the barrier of tile `it`.
DM_HANDOVER bool handover_good(const volatile int* first_bad, int it) { return it < *first_bad; }

// Where a role stopped in the ring of stages: the stage it would have used next, and the parity of that use.
DM_HANDOVER uint32_t ring_stop(int stage, uint32_t phase) { return static_cast<uint32_t>(stage) | phase << 8; }

// Parity of the last use that a role stopped at `stop` has made of stage `s`; of a stage it has not used, the parity that a
// fresh barrier reports as complete.
DM_HANDOVER uint32_t ring_last_parity(uint32_t stop, int s) {
  const uint32_t phase = stop >> 8;
  return s < static_cast<int>(stop & 0xffu) ? phase : phase ^ 1u;
}

}  // namespace dm
