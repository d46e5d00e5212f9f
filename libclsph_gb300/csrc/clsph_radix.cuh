// Stable LSD radix sort of 32-bit keys and their slots (libclsph/kernels/sort.cl:1-59,
// sph_simulation.cpp:107-156), 8-bit digits, one launch for all passes.
//
// The digit counts of every pass are known before the sort (they do not depend
// on the order). Blocks take tiles of 4,096 keys by a ticket that runs over the
// tiles of all passes; a tile ranks its keys in shared memory, publishes its
// digit counts, finds the counts of all earlier tiles by decoupled look-back
// (each digit's thread walks back over the published words until it meets an
// inclusive prefix) and scatters. A tile of a later pass first waits until
// every tile of the pass before is done. As many passes as the largest key
// needs.
//
// Look-back words (one per tile and digit, per pass): bits 30-31 the state
// (0 not yet published, 1 the tile's own count, 2 the inclusive prefix of all
// tiles up to it), bits 0-29 the value (n < 2^28). Tickets are taken in the
// order blocks ask, so every tile that a block waits for belongs to a block
// that is already running and whose own waits are for earlier tickets; every
// wait is bounded all the same (spin_limit, by default kRadixLookbackSpins),
// and one that runs out raises kFlagSortStall, which clsph_gpu_sync reports as
// an error (the stand-alone sort, which has no later call to report it, sorts
// again in one block). After a stall the offsets of the tiles behind it are
// wrong, but every store stays in bounds (destinations >= n are skipped, and the
// slots a pass leaves unwritten keep earlier in-range values), so the context
// stays usable.
//
// Bound: latency of a pass (key loads, ranking, look-back), then L2 for large
// n. One launch with tiles of 4,096 keys and 512 threads, against a histogram
// launch and four pass launches (those past the key width returned at once)
// with tiles of 2,048: 1,048,576 keys of 22 bits 0.056 -> 0.025 ms, 32,768 0.038
// -> 0.015, 4,096 0.032 -> 0.014, 4,194,304 0.122 -> 0.088. Half the tiles halve
// the look-back; the tile's counts come from the ranking instead of an atomic
// per key, which equal digits of neighbouring keys serialise. Tiles of 2,048 /
// 8,192 0.029 / 0.024 (32,768: 0.015 / 0.018); ranks by eight ballots instead of
// match 0.030; look-back windows of 4 / 16 tiles 0.025 / 0.033; three blocks an
// SM (40 registers) 0.031.
//
// withheld_tile (a test hook of clsph_gpu_set_wait_limits; kNoTile in normal
// use): that tile of every pass never publishes its words, so the tile after
// it waits on a word that nothing sets until its spin limit runs out.
#pragma once

#include "clsph_common.cuh"

namespace clsph {

constexpr uint32_t kFlagSortStall = 1u << 16;  // internal: a wait of the radix sort ran out
constexpr uint32_t kRadixLookbackSpins = 1u << 20;
constexpr uint32_t kNoTile = 0xFFFFFFFFu;
constexpr uint32_t kLbAggregate = 1u << 30, kLbInclusive = 2u << 30, kLbValue = (1u << 30) - 1u;
constexpr uint32_t kRadixTile = 4096;
constexpr uint32_t kRadixThreads = 512;
constexpr uint32_t kRadixMaxPasses = 4;

// 8-bit radix passes that cover every key of the substep.
__host__ __device__ __forceinline__ uint32_t radix_passes(uint32_t maxkey) {
  uint32_t k = maxkey | 1u, bits = 0;
  while (k) { ++bits; k >>= 1; }
  return (bits + 7u) / 8u;
}
// Ping-pong buffer that holds the sorted keys and slots after all passes.
__host__ __device__ __forceinline__ uint32_t sorted_sel(uint32_t maxkey) {
  return radix_passes(maxkey) & 1u;
}

__device__ __forceinline__ uint32_t ld_relaxed_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_gpu(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

// Adds a warp's keys to a block's digit counts; `valid` lanes come first. Keys
// of neighbouring slots are mostly equal (a cell's particles lie together), so
// each run of equal keys adds its length once.
__device__ __forceinline__ void radix_count(uint32_t key, bool valid, uint32_t passes,
                                            uint32_t (&hist)[kRadixMaxPasses][256]) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, key, 1);
  const uint32_t count = __popc(__ballot_sync(0xFFFFFFFFu, valid));
  const bool head = valid && (lane == 0u || prev != key);
  const uint32_t later = __ballot_sync(0xFFFFFFFFu, head) & (0xFFFFFFFEu << lane);
  if (head) {
    const uint32_t run = (later ? __ffs(later) - 1u : count) - lane;
    for (uint32_t p = 0; p < passes; ++p) atomicAdd(&hist[p][(key >> (8u * p)) & 0xFFu], run);
  }
}
// The block's counts into the totals (all threads, after a barrier).
__device__ __forceinline__ void radix_count_flush(const uint32_t (&hist)[kRadixMaxPasses][256], uint32_t passes,
                                                  uint32_t* __restrict__ digit_total) {
  for (uint32_t i = threadIdx.x; i < 256u * passes; i += blockDim.x) {
    const uint32_t c = hist[i >> 8][i & 255u];
    if (c) atomicAdd(&digit_total[i], c);
  }
}

// Pass p reads `in` (p = 0) or buffer (p + flip) & 1 and writes buffer
// (p + 1 + flip) & 1; the slots of pass 0 are the keys' positions.
struct RadixBuffers {
  const uint32_t* in;
  uint32_t *keys0, *keys1, *vals0, *vals1;
  uint32_t flip;
};

template <uint32_t THREADS>
struct RadixSmem {
  uint32_t cnt[THREADS / 32][256];
  uint32_t tile_off[256];
  uint32_t warp_sums[8];
  uint32_t ticket;
};

// Every pass, by all blocks of the grid: `counters` are the ticket and the
// tiles done of each pass (zero at the start, as the look-back words). kAlone:
// by the calling block alone, tile after tile, with the digits' counts of the
// tiles before carried from tile to tile and no waits.
template <uint32_t THREADS, bool kAlone = false>
__device__ __forceinline__ void radix_sort_blocks(const RadixBuffers& buf, uint32_t n, uint32_t passes,
                                                  const uint32_t* __restrict__ digit_total,
                                                  uint32_t* __restrict__ lookback, uint32_t ntiles,
                                                  uint32_t* __restrict__ counters, uint32_t* __restrict__ status,
                                                  uint32_t spin_limit, uint32_t withheld_tile,
                                                  RadixSmem<THREADS>& sm) {
  constexpr uint32_t kWarps = THREADS / 32, kItems = kRadixTile / THREADS, kSpan = 32 * kItems;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, d = threadIdx.x;
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint32_t turn = 0, carry = 0;
  for (;;) {
    __syncthreads();  // the block's previous tile is done with the shared arrays
    if (kAlone) {
      if (threadIdx.x == 0) sm.ticket = turn++;
    } else if (threadIdx.x == 0) {
      const uint32_t t = atomicAdd(&counters[0], 1u);
      const uint32_t p = t / ntiles;
      if (p > 0u && p < passes) {
        uint32_t spins = 0;
        while (ld_acquire_gpu(&counters[p]) < ntiles) {  // [p]: tiles of pass p - 1 that are done
          if (++spins > spin_limit) {
            atomicOr(status, kFlagSortStall);
            break;
          }
          __nanosleep(32);
        }
      }
      sm.ticket = t;
    }
    for (uint32_t w = threadIdx.x; w < kWarps * 256u; w += THREADS) sm.cnt[w >> 8][w & 255u] = 0u;
    __syncthreads();
    const uint32_t pass = sm.ticket / ntiles, tile = sm.ticket - pass * ntiles;
    if (pass >= passes) return;
    const bool odd = (pass + buf.flip) & 1u;
    const uint32_t* keys_in = pass == 0u ? buf.in : odd ? buf.keys1 : buf.keys0;
    const uint32_t* vals_in = odd ? buf.vals1 : buf.vals0;
    uint32_t* keys_out = odd ? buf.keys0 : buf.keys1;
    uint32_t* vals_out = odd ? buf.vals0 : buf.vals1;
    const uint32_t shift = 8u * pass;
    const uint32_t base = tile * kRadixTile + warp * kSpan;
    uint32_t key[kItems], val[kItems], rank[kItems];
#pragma unroll
    for (uint32_t r = 0; r < kItems; ++r) {
      const uint32_t idx = base + r * 32u + lane;
      key[r] = idx < n ? keys_in[idx] : 0u;
      val[r] = idx < n && pass ? vals_in[idx] : idx;
    }
    // ranks within the tile: per warp in key order (rows of 32), then warps in order
#pragma unroll
    for (uint32_t r = 0; r < kItems; ++r) {
      const bool valid = base + r * 32u + lane < n;
      const uint32_t dr = (key[r] >> shift) & 0xFFu;
      const uint32_t peers = __match_any_sync(0xFFFFFFFFu, valid ? dr : 256u);
      uint32_t rk = 0;
      if (valid) rk = sm.cnt[warp][dr] + __popc(peers & lt_mask);
      __syncwarp();
      if (valid && (peers & lt_mask) == 0u) sm.cnt[warp][dr] += __popc(peers);
      __syncwarp();
      rank[r] = (rk << 8) | dr;
    }
    __syncthreads();
    uint32_t below = 0, total = 0, excl = 0;
    if (d < 256u) {
      // the tile's count of digit d, its exclusive prefix over the warps; published for the later tiles
      uint32_t local = 0;
#pragma unroll
      for (uint32_t w = 0; w < kWarps; ++w) {
        const uint32_t c = sm.cnt[w][d];
        sm.cnt[w][d] = local;
        local += c;
      }
      uint32_t* lb = lookback + (size_t)pass * ntiles * 256u + d;
      const bool publish = !kAlone && tile != withheld_tile;
      if (publish) st_relaxed_gpu(&lb[(size_t)tile * 256u], (tile == 0 ? kLbInclusive : kLbAggregate) | local);
      // keys with a smaller digit: exclusive scan of the pass's digit totals
      total = digit_total[pass * 256u + d];
      below = total;
#pragma unroll
      for (uint32_t off = 1; off < 32u; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, below, off);
        if (lane >= off) below += y;
      }
      if (lane == 31u) sm.warp_sums[warp] = below;
      if (kAlone) {
        excl = tile ? carry : 0u;
        carry = excl + local;
      } else if (tile > 0) {
        // walk back kWindow tiles per round (independent loads), adding published counts until an inclusive
        // prefix (tile 0 always has one)
        constexpr int kWindow = 8;
        int64_t t = (int64_t)tile - 1;
        uint32_t spins = 0;
        bool done = false;
        while (!done) {
          uint32_t w[kWindow];
#pragma unroll
          for (int k = 0; k < kWindow; ++k)
            w[k] = t - k >= 0 ? ld_relaxed_gpu(&lb[(size_t)(t - k) * 256u]) : kLbInclusive;
          int used = 0;
#pragma unroll
          for (int k = 0; k < kWindow; ++k) {
            if (done || used < k) break;          // stopped at an earlier word of this round
            if ((w[k] & ~kLbValue) == 0u) break;  // not published yet: load it again
            excl += w[k] & kLbValue;
            ++used;
            if (w[k] & kLbInclusive) done = true;
          }
          t -= used;
          if (!done && used == 0) {
            if (++spins > spin_limit) {
              atomicOr(status, kFlagSortStall);
              break;
            }
            __nanosleep(32);
          }
        }
        if (publish) st_relaxed_gpu(&lb[(size_t)tile * 256u], kLbInclusive | (excl + local));
      }
    }
    __syncthreads();
    if (d < 256u) {
      for (uint32_t w = 0; w < warp; ++w) below += sm.warp_sums[w];
      sm.tile_off[d] = below - total + excl;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t r = 0; r < kItems; ++r) {
      if (base + r * 32u + lane >= n) continue;
      const uint32_t dd = rank[r] & 0xFFu;
      const uint32_t dst = sm.tile_off[dd] + sm.cnt[warp][dd] + (rank[r] >> 8);
      if (dst >= n) continue;  // only after a wait ran out (flagged)
      keys_out[dst] = key[r];
      vals_out[dst] = val[r];
    }
    __syncthreads();
    if (!kAlone && threadIdx.x == 0 && pass + 1u < passes) {
      __threadfence();  // the block's stores (ordered by the barrier above) before the count
      atomicAdd(&counters[pass + 1u], 1u);
    }
  }
}

}  // namespace clsph
