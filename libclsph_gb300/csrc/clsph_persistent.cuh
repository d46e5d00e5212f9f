// The whole substep loop as one persistent, cooperative launch (for batched
// scenes of uneven sizes; no counterpart in the reference).
//
// One block of 256 threads per resident slot on every SM (all co-resident,
// which the cooperative launch guarantees) runs every phase of a substep in
// turn, S substeps per launch, with a grid-wide barrier between phases:
//   grid set-up (block 0) | keys, digit counts, cell-index clear |
//   radix passes (tiles by ticket, decoupled look-back) | gather |
//   density (two warps per occupied cell, 4 teams a block) | forces | advection
// Each phase is the block-level body of the corresponding kernel of
// clsph_kernels.cuh, so the results are those of the launched substeps bit
// for bit. The barrier is a counter and a generation word in device memory;
// every wait on it is bounded (a wait that runs out sets kFlagBarrierStall,
// its block leaves the kernel, and clsph_gpu_sync reports the error and
// resets the words).
#pragma once

#include "clsph_kernels.cuh"

namespace clsph {

constexpr uint32_t kFlagBarrierStall = 1u << 17;  // internal: a grid barrier wait ran out
constexpr uint32_t kPersistThreads = 256;
constexpr uint32_t kBarrierSpins = 1u << 22;  // ~ seconds: longer than any phase
constexpr uint32_t kNoBlock = 0xFFFFFFFFu;

struct PersistArgs {
  uint32_t n, nscenes, ntiles, slots, nlist_cap, max_iters;
  uint32_t* bbox;
  DevGrid* grids;
  const float* scene_h;
  uint32_t* status;
  uint32_t* digit_total;
  uint32_t* step_counters;
  uint32_t* ctl;
  const uint16_t* scene_of;
  uint32_t* keys;
  uint32_t* vals;
  uint32_t* lookback;
  State st[2];
  uint32_t* ids[2];
  CellIndex ci;
  uint2* cell_list;
  uint32_t* planes;
  const Consts* consts;
  float4* aux;
  uint16_t* nlist;
  uint32_t* ncount;
  float4* frec;
  uint32_t* nb_start;
  float4* acc;
  const DevMesh* meshes;
  unsigned long long* capped;
  uint32_t* barrier;  // [0] arrivals, [1] generation
  uint32_t spin_limit, withheld_tile;  // radix look-back bound and test hook
  uint32_t barrier_limit, withheld_block;  // grid barrier bound and test hook
};

using PersistTeam = CellTeamSmem<2, 128, 14>;

union PersistSmem {
  RadixSmem<kPersistThreads> radix;
  KeysSmem keys;
  PersistTeam dens[kPersistThreads / 64];  // one team of two warps for each 64 threads
  GatherSmem gather;
  BboxSmem bbox;
  uint32_t word;
};
// dynamic shared memory: three resident blocks of the SM's 227 KB
static_assert(sizeof(PersistSmem) <= 74 * 1024, "shared memory of the persistent kernel");

// Grid-wide barrier; false (for the whole block) when this block's wait ran
// out or when it is the test hook's withheld block (which leaves at once,
// as a block that never arrives).
__device__ __forceinline__ bool grid_barrier(const PersistArgs& a, uint32_t& ok_s) {
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t good = 1u;
    if (blockIdx.x == a.withheld_block) {
      good = 0u;
    } else {
      const uint32_t gen = ld_acquire_gpu(&a.barrier[1]);
      __threadfence();  // the block's writes (ordered by the barrier above) before the arrival
      if (atomicAdd(&a.barrier[0], 1u) == gridDim.x - 1u) {
        atomicExch(&a.barrier[0], 0u);
        __threadfence();
        atomicAdd(&a.barrier[1], 1u);
      } else {
        uint32_t spins = 0;
        while (ld_acquire_gpu(&a.barrier[1]) == gen) {
          if (++spins > a.barrier_limit) {
            atomicOr(a.status, kFlagBarrierStall);
            good = 0u;
            break;
          }
          __nanosleep(64);
        }
      }
      __threadfence();
    }
    ok_s = good;
  }
  __syncthreads();
  return ok_s != 0u;
}

// three resident blocks per SM (24 warps): at most 85 registers per thread
static __global__ void __launch_bounds__(kPersistThreads, 3)
    k_substeps_persistent(PersistArgs a, uint32_t substeps, uint32_t ids_sel0) {
  extern __shared__ __align__(16) unsigned char persist_smem[];
  PersistSmem& sm = *reinterpret_cast<PersistSmem*>(persist_smem);
  __shared__ uint32_t ok_s;
  const uint32_t n = a.n;
  const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t gstride = gridDim.x * blockDim.x;
  const uint32_t nblk = (n + kPersistThreads - 1) / kPersistThreads;
  for (uint32_t s = 0; s < substeps; ++s) {
    const uint32_t src_ids = (ids_sel0 + s) & 1u;
    // grid set-up of every scene
    if (blockIdx.x == 0)
      grid_setup_block(a.bbox, a.grids, a.scene_h, a.nscenes, a.status, a.digit_total, a.step_counters, a.ctl,
                       sm.word);
    if (!grid_barrier(a, ok_s)) return;
    keys_blocks(blockIdx.x, gridDim.x, a.st[0].pos, n, a.grids, a.scene_of, a.ctl, a.keys, a.digit_total,
                reinterpret_cast<uint4*>(a.lookback), a.ntiles, reinterpret_cast<uint4*>(a.ci.keys), a.slots / 4u,
                sm.keys);
    if (!grid_barrier(a, ok_s)) return;
    radix_sort_blocks<kPersistThreads>(substep_buffers(a.keys, a.vals, n), n, radix_passes(a.ctl[kCtlMaxKey]),
                                       a.digit_total, a.lookback, a.ntiles, a.step_counters + kCntRadix, a.status,
                                       a.spin_limit, a.withheld_tile, sm.radix);
    if (!grid_barrier(a, ok_s)) return;
    for (uint32_t vb = blockIdx.x; vb < nblk; vb += gridDim.x)
      gather_block(vb, n, a.grids, a.scene_of, a.ctl, a.keys, a.vals, a.st[0], a.st[1], a.ids[src_ids],
                   a.ids[src_ids ^ 1u], a.ci, a.cell_list, a.step_counters + kCntCells, a.planes, sm.gather);
    if (!grid_barrier(a, ok_s)) return;
    density_cells_team<true>(n, a.grids, a.ctl, a.scene_of, a.keys, a.st[1].pos, a.planes, a.ci, a.consts, a.aux,
                             a.nlist, a.ncount, a.nlist_cap, a.st[1].vel, a.frec, a.cell_list, a.step_counters,
                             a.nb_start, sm.dens[threadIdx.x >> 6], (threadIdx.x >> 5) & 1u,
                             blockIdx.x * (kPersistThreads / 64u) + (threadIdx.x >> 6),
                             gridDim.x * (kPersistThreads / 64u), 1u + (threadIdx.x >> 6));
    if (!grid_barrier(a, ok_s)) return;
    for (uint32_t i = gtid; (i & ~31u) < n; i += gstride)
      forces_particle<true>(i < n, i, n, a.grids, a.scene_of, a.ctl, a.keys, a.st[1], a.aux, a.ci, a.consts, a.nlist,
                            a.ncount, a.nlist_cap, a.acc, NoForceHook{}, a.frec, a.nb_start);
    if (!grid_barrier(a, ok_s)) return;
    advect_blocks<false>(blockIdx.x, gridDim.x, n, a.st[1], a.acc, a.st[0], a.meshes, a.consts, a.scene_of,
                         a.max_iters, a.bbox, a.status, a.capped, nullptr, 1.f, 1.f, nullptr, nullptr, sm.bbox);
    if (!grid_barrier(a, ok_s)) return;
  }
}

}  // namespace clsph
