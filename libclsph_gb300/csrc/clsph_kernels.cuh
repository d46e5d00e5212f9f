// Device kernels of one SPH substep (sm_103a).
//
// Data layout in HBM (SoA, sorted order, 16-byte float4 rows):
//   pos[n], vel[n], ivel[n]   position, velocity, intermediate (half-step) velocity
//   aux[n]                    (rho, p, own cell's first slot (bits), p/rho^2) of the substep
//   nlist[cap][n], ncount[n]  contributing neighbours of each particle, in visiting order,
//                             as 16-bit tags (neighbour cell k of 27 << 11 | offset in it)
//   nb_start[n][27]           first slot of each of the 27 cells around a cell, in the
//                             row of the cell's first slot (resolves the tags)
//   acc[n]                    acceleration (forces -> advection)
//   keys[2][n], vals[2][n]    radix-sort ping-pong (Morton key, source slot)
//   ids[2][n]                 persistent particle ids (the reference has none)
//   hkeys[S], hstart[S], hend[S]  cell index: Morton key -> [start, end)
// A handle holds S independent scenes (S = 1 for a single simulation): the
// particles of scene s occupy one contiguous slot range, scene_of[slot] = s.
// The sort key is (s << scene_shift) | Morton key, so the one stable sort
// keeps every scene in its range and orders it exactly like a sort of that
// scene alone. Per-scene grids (bounding box, cell size, dense cell count),
// constants and meshes live in device arrays; the sort control (largest key,
// hence the number of radix passes) is shared. Nothing needs a host round
// trip between kernels.
#pragma once

#include <cuda_fp16.h>

#include <type_traits>

#include "clsph_common.cuh"
#include "clsph_mesh.cuh"
#include "clsph_radix.cuh"

namespace clsph {

constexpr int kBlock = 256;
// per-substep counters, zeroed by k_grid_setup
constexpr int kStepCounters = 8;
// [kCntCells] occupied cells listed by k_gather, [kCntWorkDensity] cells
// taken by the cell-warp density search, [kCntRadix] the radix sort's ticket
// and the tiles done of its passes (kRadixMaxPasses words)
enum : int { kCntCells = 0, kCntWorkDensity = 1, kCntRadix = 4 };

enum : uint32_t {
  kFlagGridOverflow = 1u,
  kFlagCollisionCap = 2u,
  kFlagNonFinite = 4u,
};

struct DevGrid {         // one scene's grid of the current substep
  float lo[3];
  float hi[3];
  float cell;           // 2h
  int32_t size[3];      // grid_size_x/y/z
  uint32_t cells;       // grid_cell_count (dense Morton range)
  float half_margin;    // rounding margin of the half-cell tests, in cells
  uint32_t pad_[4];
};

// Sort control block of a substep (device memory): [0] largest key,
// [1] Morton bits (widest grid of all scenes), [2] scene bits, [3] nonzero when
// some coordinate is nonzero but below kTinyCoordinate (k_gather).
enum : int { kCtlMaxKey = 0, kCtlShift = 1, kCtlSceneBits = 2, kCtlTiny = 3, kCtlWords = 8 };

// Differences of coordinates of at least this size are 0 or at least 2^-99,
// as div_rn_normal needs.
constexpr float kTinyCoordinate = 0x1p-76f;

// Scene bits of a sort key and its Morton part.
struct KeySplit {
  uint32_t shift;  // Morton keys use bits [0, shift)
  __host__ __device__ __forceinline__ uint32_t morton(uint32_t key) const {
    return shift >= 32u ? key : (key & ((1u << shift) - 1u));
  }
  __host__ __device__ __forceinline__ uint32_t scene_bits(uint32_t scene) const {
    return shift >= 32u ? 0u : (scene << shift);
  }
};

// Per-substep constants (kernel argument).
struct Consts {
  uint32_t n;
  float h, mass, rho0, K, mu, sigma, sigma_threshold, restitution;
  float time_delta, scale, vmax;
  float gx, gy, gz;
  float poly6, grad6, lap6, spiky, visc, spiky_zero;
  float cull_r2;  // conservative h^2 for the FMA cull test
  uint32_t plain_h;  // h in [2^-20, 2^20]: near_norm and the short quotients are exact
};

struct State {
  float4* pos;
  float4* vel;
  float4* ivel;
};

struct CellIndex {
  uint32_t* keys;   // key + 1, 0 = empty
  uint32_t* start;
  uint32_t* end;
  uint32_t mask;    // slots - 1 (power of two)
  uint32_t shift;   // 32 - log2(slots)
};

struct DevMesh {
  const float4* packed;  // kFaceRows per face (k_pack_faces, clsph_mesh.cuh)
  uint32_t faces;
  // per-cell triangle lists (CSR over a uniform grid covering the mesh)
  const uint32_t* cell_start;  // dims product + 1
  const uint32_t* cell_faces;
  float lo[3];
  float inv_cell;
  int32_t dims[3];
  float reach;  // longest segment a cell list covers
};

// Loads of what a substep's own phases write (positions, cell index, neighbour
// starts and records, ...): read-only loads where each phase is a kernel of its
// own; plain ones (kLive) in the persistent kernel, which writes these arrays
// in the launch that reads them.
template <bool kLive, typename T>
__device__ __forceinline__ T ld_step(const T* p) {
  if constexpr (kLive) return *p;
  else return __ldg(p);
}

// ------------------------------------------------------------ cell index
__device__ __forceinline__ uint32_t cell_slot_insert(const CellIndex& ci, uint32_t key) {
  const uint32_t tag = key + 1u;
  uint32_t slot = cell_hash(key) >> ci.shift;
  for (uint32_t probe = 0; probe <= ci.mask; ++probe) {
    uint32_t prev = atomicCAS(&ci.keys[slot], 0u, tag);
    if (prev == 0u || prev == tag) return slot;
    slot = (slot + 1u) & ci.mask;
  }
  return 0xFFFFFFFFu;  // unreachable: at most n keys in >= 2n slots
}

template <bool kLive = false>
__device__ __forceinline__ uint2 cell_lookup(const CellIndex& ci, uint32_t key) {
  const uint32_t tag = key + 1u;
  uint32_t slot = cell_hash(key) >> ci.shift;
  for (uint32_t probe = 0; probe <= ci.mask; ++probe) {
    uint32_t k = ld_step<kLive>(&ci.keys[slot]);
    if (k == tag) return make_uint2(ld_step<kLive>(&ci.start[slot]), ld_step<kLive>(&ci.end[slot]));
    if (k == 0u) break;
    slot = (slot + 1u) & ci.mask;
  }
  return make_uint2(0u, 0u);
}

// ---------------------------------------------------- neighbour cell window
// The support radius is h but cells are 2h wide (grid.cl:56-61 vs
// smoothing.cl:2). Each particle carries, per axis, whether it may lie in the
// lower half of its cell (bit 2a) and whether it may lie in the upper half
// (bit 2a+1), decided with a rounding margin so that a particle near the
// middle has both bits. A particle with only the lower bit cannot be within
// h of anything in the next cell up (the distance is > half a cell = h), and
// symmetrically; cells and particles so excluded contribute exact zeros in
// the reference, so skipping them keeps the reference's summation sequence.
// The code is computed after the sort and kept in pos.w of the sorted state.
__device__ __forceinline__ uint32_t half_code(float4 p, uint32_t key, const DevGrid& g) {
  const uint32_t c[3] = {compact_bits3(key), compact_bits3(key >> 1), compact_bits3(key >> 2)};
  const float pc[3] = {p.x, p.y, p.z};
  uint32_t code = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float frac = XDIV(XSUB(pc[a], g.lo[a]), g.cell) - (float)c[a];
    code |= (frac < 0.5f + g.half_margin ? 1u : 0u) << (2 * a);
    code |= (frac > 0.5f - g.half_margin ? 1u : 0u) << (2 * a + 1);
  }
  return code;
}

struct Window {
  uint32_t lo[3], hi[3];
};

__device__ __forceinline__ Window neighbour_window(float4 p, uint32_t key, const DevGrid& g) {
  const uint32_t c[3] = {compact_bits3(key), compact_bits3(key >> 1), compact_bits3(key >> 2)};
  const uint32_t code = __float_as_uint(p.w);
  Window w;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    w.lo[a] = ((code >> (2 * a)) & 1u) ? c[a] - 1u : c[a];
    w.hi[a] = ((code >> (2 * a + 1)) & 1u) ? c[a] + 1u : c[a];
  }
  return w;
}

// --------------------------------------------------------------- kernels

// Grid set-up of every scene (sph_simulation.cpp:199-252), one thread per
// scene, from the bounding boxes accumulated by the previous kernel; resets
// the boxes, the radix digit totals and the sort control for this substep.
// (The kernels of this file are thin wrappers around block-level bodies with
// their shared memory passed in, so the persistent substep kernel of
// clsph_persistent.cuh runs the same code on its own blocks.)
__device__ __forceinline__ void grid_setup_block(uint32_t* __restrict__ bbox_all, DevGrid* __restrict__ grids,
                                                 const float* __restrict__ scene_h, uint32_t nscenes,
                                                 uint32_t* __restrict__ status, uint32_t* __restrict__ digit_total,
                                                 uint32_t* __restrict__ step_counters, uint32_t* __restrict__ ctl,
                                                 uint32_t& shift_s) {
  for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) digit_total[i] = 0u;
  if (threadIdx.x < kStepCounters) step_counters[threadIdx.x] = 0u;
  if (threadIdx.x == 0) shift_s = 1u;
  __syncthreads();
  for (uint32_t sc = threadIdx.x; sc < nscenes; sc += blockDim.x) {
  uint32_t* bbox = bbox_all + 6 * (size_t)sc;
  DevGrid* grid = grids + sc;
  const float cell = XMUL(scene_h[sc], 2.f);
  DevGrid g;
  bool overflow = false;
  for (int a = 0; a < 3; ++a) {
    float mn = ord2f(bbox[a]);
    float mx = ord2f(bbox[3 + a]);
    mn = XSUB(mn, XMUL(cell, 2.f));
    mx = XADD(mx, XMUL(cell, 2.f));
    g.lo[a] = mn;
    g.hi[a] = mx;
    uint32_t sz = __float2uint_rz(XDIV(XSUB(mx, mn), cell));
    g.size[a] = (int32_t)sz;
    if (g.size[a] < 0 || g.size[a] >= 1024) overflow = true;
  }
  g.cell = cell;
  g.cells = morton3((uint32_t)g.size[0], (uint32_t)g.size[1], (uint32_t)g.size[2]);
  atomicMax(&shift_s, 32u - __clz(g.cells | 1u));  // keys of this scene are < cells
  // The cell coordinate t = fl(fl(p - lo) / 2h) is within ~2^-22 * t of the
  // exact value and t < grid size G, so 2^-20 * (G + 2) covers its rounding
  // and that of the distance test twice over.
  const int gmax = max(g.size[0], max(g.size[1], g.size[2]));
  g.half_margin = (float)(gmax + 2) * 0x1p-20f;
  for (int i = 0; i < 4; ++i) g.pad_[i] = 0u;
  *grid = g;
  if (overflow) {  // cells holds the wrapped sizes, while coordinates wrap at ten bits: take all the bits there are
    atomicOr(status, kFlagGridOverflow);
    atomicMax(&shift_s, min(30u, 32u - ctl[kCtlSceneBits]));
  }
  // sentinels of sph_simulation.cpp:204-205 for the next accumulation
  for (int a = 0; a < 3; ++a) {
    bbox[a] = f2ord(2147483648.0f);
    bbox[3 + a] = f2ord(-2147483648.0f);
  }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ctl[kCtlMaxKey] = 0u;
    ctl[kCtlTiny] = 0u;
    ctl[kCtlShift] = shift_s;
    // scene bits above the Morton bits must fit in 32 (batched scenes)
    if (shift_s + ctl[kCtlSceneBits] > 32u) atomicOr(status, kFlagGridOverflow);
  }
}

static __global__ void k_grid_setup(uint32_t* __restrict__ bbox_all, DevGrid* __restrict__ grids,
                                    const float* __restrict__ scene_h, uint32_t nscenes,
                                    uint32_t* __restrict__ status, uint32_t* __restrict__ digit_total,
                                    uint32_t* __restrict__ step_counters, uint32_t* __restrict__ ctl) {
  if (never_after_previous()) return;
  __shared__ uint32_t shift_s;
  grid_setup_block(bbox_all, grids, scene_h, nscenes, status, digit_total, step_counters, ctl, shift_s);
}

static __global__ void k_bbox_reset(uint32_t* __restrict__ bbox, uint32_t nscenes) {
  if (never_after_previous()) return;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < 6 * nscenes; k += gridDim.x * blockDim.x)
    bbox[k] = (k % 6) < 3 ? f2ord(2147483648.0f) : f2ord(-2147483648.0f);
}

// Per-scene min/max of positions: a block whose threads all saw one scene
// reduces to one atomic per axis; otherwise every warp (or, across a scene
// boundary, every thread) adds its own. NaN coordinates are ignored, as the
// reference's `<` / `>` tests do. A thread with no particle passes scene = -1.
__device__ __forceinline__ void bbox_atomics(const float v[6], uint32_t* bbox) {
  if (v[0] == v[0]) atomicMin(&bbox[0], f2ord(v[0]));
  if (v[1] == v[1]) atomicMin(&bbox[1], f2ord(v[1]));
  if (v[2] == v[2]) atomicMin(&bbox[2], f2ord(v[2]));
  if (v[3] == v[3]) atomicMax(&bbox[3], f2ord(v[3]));
  if (v[4] == v[4]) atomicMax(&bbox[4], f2ord(v[4]));
  if (v[5] == v[5]) atomicMax(&bbox[5], f2ord(v[5]));
}

struct BboxSmem {
  int block_scene;
  float red[6][kBlock / 32];
};

__device__ __forceinline__ void bbox_accumulate(float3 lo, float3 hi, int scene, uint32_t* bbox_all,
                                                BboxSmem& sm) {
  int& block_scene = sm.block_scene;
  auto& red = sm.red;
  if (threadIdx.x == 0) block_scene = -2;
  __syncthreads();
  if (scene >= 0) atomicCAS(&block_scene, -2, scene);
  __syncthreads();
  const int s0 = block_scene;
  const bool uniform = __syncthreads_and(scene < 0 || scene == s0);
  if (!uniform) {
    const float v[6] = {lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
    if (scene >= 0) bbox_atomics(v, bbox_all + 6 * (size_t)scene);
    return;
  }
  if (s0 < 0) return;
  uint32_t* bbox = bbox_all + 6 * (size_t)s0;
  float v[6] = {lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
#pragma unroll
  for (int k = 0; k < 6; ++k) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      float o = __shfl_xor_sync(0xFFFFFFFFu, v[k], off);
      v[k] = k < 3 ? fminf(v[k], o) : fmaxf(v[k], o);
    }
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0)
    for (int k = 0; k < 6; ++k) red[k][warp] = v[k];
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      float x = lane < nw ? red[k][lane] : __int_as_float(0x7FC00000);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        float o = __shfl_xor_sync(0xFFFFFFFFu, x, off);
        x = k < 3 ? fminf(x, o) : fmaxf(x, o);
      }
      if (lane == 0 && x == x) {
        if (k < 3)
          atomicMin(&bbox[k], f2ord(x));
        else
          atomicMax(&bbox[k], f2ord(x));
      }
    }
  }
}

__device__ __forceinline__ void bbox_accumulate(float3 lo, float3 hi, int scene, uint32_t* bbox_all) {
  __shared__ BboxSmem sm;
  bbox_accumulate(lo, hi, scene, bbox_all, sm);
}

// Host AoS (80-byte particle records, 5 float4 each) -> SoA state, with
// bounding box. One thread per float4 of the record array, so a warp reads
// 512 contiguous bytes: `aos` is the device staging copy or, for pinned host
// memory, the caller's records themselves, read over the host link.
static __global__ void k_unpack_aos(const float4* __restrict__ aos, uint32_t n, State st,
                             const uint16_t* __restrict__ scene_of, uint32_t* __restrict__ bbox,
                             uint32_t* __restrict__ status) {
  if (never_after_previous()) return;
  const float qnan = __int_as_float(0x7FC00000);
  const size_t words = (size_t)n * 5;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t base = (size_t)blockIdx.x * blockDim.x; base < words; base += stride) {
    const size_t q = base + threadIdx.x;
    float3 lo = make_float3(qnan, qnan, qnan), hi = lo;
    int scene = -1;
    if (q < words) {
      const uint32_t i = (uint32_t)(q / 5), f = (uint32_t)(q - (size_t)i * 5);
      if (f < 3) {  // position, velocity, intermediate velocity; the rest is output only
        float4 v = aos[q];
        v.w = 0.f;
        if (f == 0) {
          st.pos[i] = v;
          lo = make_float3(v.x, v.y, v.z);
          hi = lo;
          scene = scene_of[i];
          if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z))) atomicOr(status, kFlagNonFinite);
        } else if (f == 1) {
          st.vel[i] = v;
        } else {
          st.ivel[i] = v;
        }
      }
    }
    bbox_accumulate(lo, hi, scene, bbox);
  }
}

// SoA -> host AoS: acceleration is 0 after the advection loop (sph.cl:97-99).
// One thread per float4 of the record array (contiguous stores), into the
// staging copy or straight into pinned host memory.
static __global__ void k_pack_aos(float4* __restrict__ aos, uint32_t n, State st,
                           const float4* __restrict__ aux, const uint32_t* __restrict__ keys_base,
                           const uint32_t* __restrict__ ctl, int have_fields) {
  if (never_after_previous()) return;
  const KeySplit split{ctl[kCtlShift]};
  const uint32_t sel = have_fields ? sorted_sel(ctl[kCtlMaxKey]) : 0u;
  const uint32_t* keys = keys_base + (size_t)sel * n;
  const size_t words = (size_t)n * 5;
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < words; q += (size_t)gridDim.x * blockDim.x) {
    const uint32_t i = (uint32_t)(q / 5), f = (uint32_t)(q - (size_t)i * 5);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (f == 0) {
      v = st.pos[i];
    } else if (f == 1) {
      v = st.vel[i];
    } else if (f == 2) {
      v = st.ivel[i];
    } else if (f == 4 && have_fields) {  // density, pressure, grid cell code, 0
      const float4 a = aux[i];
      v.x = a.x;
      v.y = a.y;
      v.z = __uint_as_float(split.morton(keys[i]));
    }
    aos[q] = v;
  }
}

// Morton key per particle (grid.cl:56-66), the largest key and the digit
// counts of the sort's passes. Also clears the sort's look-back words and the
// cell index for this substep's k_gather (16 bytes a thread), which no kernel
// between reads.
struct KeysSmem {
  uint32_t hist[kRadixMaxPasses][256];
  uint32_t block_max;
};

__device__ __forceinline__ void keys_blocks(uint32_t blk, uint32_t nblk, const float4* __restrict__ pos, uint32_t n,
                                            const DevGrid* __restrict__ grids, const uint16_t* __restrict__ scene_of,
                                            uint32_t* __restrict__ ctl, uint32_t* __restrict__ keys,
                                            uint32_t* __restrict__ digit_total, uint4* __restrict__ lookback,
                                            uint32_t ntiles, uint4* __restrict__ index_keys, uint32_t index_quads,
                                            KeysSmem& sm) {
  const KeySplit split{ctl[kCtlShift]};
  // no key has more bits than the widest grid's keys and the scenes (the Morton part is masked: on an overflowed
  // grid it can hold more)
  const uint32_t passes = (min(split.shift + ctl[kCtlSceneBits], 32u) + 7u) / 8u;
  const uint32_t first = blk * blockDim.x + threadIdx.x, stride = nblk * blockDim.x;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (uint32_t q = first; q < index_quads; q += stride) index_keys[q] = zero;
  for (uint32_t q = first; q < passes * ntiles * 64u; q += stride) lookback[q] = zero;
  for (uint32_t q = threadIdx.x; q < kRadixMaxPasses * 256u; q += blockDim.x) sm.hist[q >> 8][q & 255u] = 0u;
  if (threadIdx.x == 0) sm.block_max = 0u;
  __syncthreads();
  uint32_t top = 0u;
  for (uint32_t i = first; (i & ~31u) < n; i += stride) {
    uint32_t key = 0u;
    if (i < n) {
      const uint32_t sc = scene_of[i];
      const DevGrid& g = grids[sc];
      const float4 p = pos[i];
      const uint32_t cx = __float2uint_rz(XDIV(XSUB(p.x, g.lo[0]), g.cell));
      const uint32_t cy = __float2uint_rz(XDIV(XSUB(p.y, g.lo[1]), g.cell));
      const uint32_t cz = __float2uint_rz(XDIV(XSUB(p.z, g.lo[2]), g.cell));
      key = split.morton(morton3(cx, cy, cz)) | split.scene_bits(sc);
      keys[i] = key;
      top = max(top, key);
    }
    radix_count(key, i < n, passes, sm.hist);
  }
  top = __reduce_max_sync(0xFFFFFFFFu, top);
  if ((threadIdx.x & 31) == 0) atomicMax(&sm.block_max, top);
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(&ctl[kCtlMaxKey], sm.block_max);
  radix_count_flush(sm.hist, passes, digit_total);
}

static __global__ void __launch_bounds__(kBlock)
    k_keys(const float4* __restrict__ pos, uint32_t n, const DevGrid* __restrict__ grids,
           const uint16_t* __restrict__ scene_of, uint32_t* __restrict__ ctl, uint32_t* __restrict__ keys,
           uint32_t* __restrict__ digit_total, uint4* __restrict__ lookback, uint32_t ntiles,
           uint4* __restrict__ index_keys, uint32_t index_quads) {
  if (never_after_previous()) return;
  __shared__ KeysSmem sm;
  keys_blocks(blockIdx.x, gridDim.x, pos, n, grids, scene_of, ctl, keys, digit_total, lookback, ntiles, index_keys,
              index_quads, sm);
}

// The sort of the substep's keys (clsph_radix.cuh): pass p reads buffer p & 1
// and writes the other.
__device__ __forceinline__ RadixBuffers substep_buffers(uint32_t* keys, uint32_t* vals, uint32_t n) {
  return RadixBuffers{keys, keys, keys + n, vals, vals + n, 0u};
}

static __global__ void __launch_bounds__(kRadixThreads)
    k_radix_sort(uint32_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t n,
                 const uint32_t* __restrict__ ctl, const uint32_t* __restrict__ digit_total,
                 uint32_t* __restrict__ lookback, uint32_t ntiles, uint32_t* __restrict__ counters,
                 uint32_t* __restrict__ status, uint32_t spin_limit, uint32_t withheld_tile) {
  if (never_after_previous()) return;
  __shared__ RadixSmem<kRadixThreads> sm;
  radix_sort_blocks<kRadixThreads>(substep_buffers(keys, vals, n), n, radix_passes(ctl[kCtlMaxKey]), digit_total,
                                   lookback, ntiles, counters, status, spin_limit, withheld_tile, sm);
}

// Half codes as bit planes: word [g * kHalfPlanes + b] holds bit b of the half
// codes of the 32 sorted slots of group g (written by k_gather, read by the
// cell search).
constexpr uint32_t kHalfPlanes = 6;

// Gathers the state into sorted order (the stable scatter of sort.cl:41-59)
// and records every cell's [start, end) in the cell index (the dense cell
// table of sph_simulation.cpp:162-170 in compact form).
// Cell starts join the cell list with one atomic per block (slot order is
// kept within the block, so the list stays close to sorted order).
struct GatherSmem {
  uint32_t warp_base[kBlock / 32];
  uint32_t block_base;
};

__device__ __forceinline__ void gather_block(uint32_t vb, uint32_t n, const DevGrid* __restrict__ grids,
                                             const uint16_t* __restrict__ scene_of,
                                             uint32_t* __restrict__ ctl,
                                             const uint32_t* __restrict__ keys_base,
                                             const uint32_t* __restrict__ vals_base, State src, State dst,
                                             const uint32_t* __restrict__ ids_src, uint32_t* __restrict__ ids_dst,
                                             CellIndex ci, uint2* __restrict__ cell_list,
                                             uint32_t* __restrict__ cell_count, uint32_t* __restrict__ planes,
                                             GatherSmem& sm) {
  auto& warp_base = sm.warp_base;
  uint32_t& block_base = sm.block_base;
  const uint32_t s = vb * blockDim.x + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const KeySplit split{ctl[kCtlShift]};
  const uint32_t sel = sorted_sel(ctl[kCtlMaxKey]);
  const uint32_t* keys = keys_base + (size_t)sel * n;
  const uint32_t* perm = vals_base + (size_t)sel * n;
  bool first = false, tiny = false;
  uint32_t key = 0u, code = 0u;
  if (s < n) {
    const uint32_t from = min(perm[s], n - 1u);  // in range even after a flagged sort stall
    key = keys[s];
    float4 p = src.pos[from];
    auto below = [](float x) { return x != 0.f && fabsf(x) < kTinyCoordinate; };
    tiny = below(p.x) || below(p.y) || below(p.z);
    code = half_code(p, split.morton(key), grids[scene_of[s]]);
    p.w = __uint_as_float(code);
    dst.pos[s] = p;
    dst.vel[s] = src.vel[from];
    dst.ivel[s] = src.ivel[from];
    ids_dst[s] = ids_src[from];
    first = s == 0 || keys[s - 1] != key;
    if (first) {
      uint32_t slot = cell_slot_insert(ci, key);
      if (slot != 0xFFFFFFFFu) ci.start[slot] = s;
    }
    if (s + 1 == n || keys[s + 1] != key) {
      uint32_t slot = cell_slot_insert(ci, key);
      if (slot != 0xFFFFFFFFu) ci.end[slot] = s + 1;
    }
  }
  uint32_t plane = 0u;  // the half codes of the warp's 32 slots as bit planes, for the cell search
#pragma unroll
  for (uint32_t b = 0; b < kHalfPlanes; ++b) {
    const uint32_t v = __ballot_sync(0xFFFFFFFFu, (code >> b) & 1u);
    if (lane == b) plane = v;
  }
  if (lane < kHalfPlanes && (s & ~31u) < n) planes[(size_t)(s >> 5) * kHalfPlanes + lane] = plane;
  if (tiny) ctl[kCtlTiny] = 1u;
  const uint32_t bal = __ballot_sync(0xFFFFFFFFu, first);
  if (lane == 0) warp_base[warp] = __popc(bal);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t run = 0;
    for (int w = 0; w < kBlock / 32; ++w) {
      const uint32_t c = warp_base[w];
      warp_base[w] = run;
      run += c;
    }
    block_base = run ? atomicAdd(cell_count, run) : 0u;
  }
  __syncthreads();
  if (first) cell_list[block_base + warp_base[warp] + __popc(bal & ((1u << lane) - 1u))] = make_uint2(s, key);
  __syncthreads();  // the shared counts are read before the block's next use
}

static __global__ void __launch_bounds__(kBlock)
    k_gather(uint32_t n, const DevGrid* __restrict__ grids,
             const uint16_t* __restrict__ scene_of, uint32_t* __restrict__ ctl,
             const uint32_t* __restrict__ keys_base,
             const uint32_t* __restrict__ vals_base, State src, State dst,
             const uint32_t* __restrict__ ids_src, uint32_t* __restrict__ ids_dst,
             CellIndex ci, uint2* __restrict__ cell_list,
             uint32_t* __restrict__ cell_count, uint32_t* __restrict__ planes) {
  if (never_after_previous()) return;
  __shared__ GatherSmem sm;
  gather_block(blockIdx.x, n, grids, scene_of, ctl, keys_base, vals_base, src, dst, ids_src, ids_dst, ci,
               cell_list, cell_count, planes, sm);
}

// ------------------------------------------------- density and forces
// Both gathers visit neighbours in the reference's order (27 cells in z, y, x
// order, each cell's particles in sorted order; only the window cells can
// contribute, the others add exact zeros) and evaluate every contributing
// pair with IEEE round-to-nearest operations in the reference's expression
// order, so the sums are bit-identical to the reference's.
//
// A candidate j contributes iff fl(r/h) < 1 (the (1 - clamp(floor(r/h),0,1))
// factor of smoothing.cl). For floats r >= 0 and h > 0 that is exactly r < h:
// fl(r/h) < 1 iff r/h < 1 - 2^-25, i.e. r < h(1 - 2^-25), and no float lies in
// [h(1 - 2^-25), h) because the float below h is at most h(1 - 2^-24).
//
// Per particle the density kernel also stores (rho, p, m/rho, p/rho^2) -- the
// same IEEE quotients the reference forms per pair -- and the list of its
// contributing neighbours in visiting order (column-major, nlist[k*n + i]),
// which the forces kernel walks without a second search. The list is stored
// and read with evict-first (streaming) hints: it is read once, and at 1M
// particles it is larger than L2, where the neighbour records should stay.

// Tait pressure (sph.cl:36-39): K * (pown(rho / rho0, 7) - 1).
__device__ __forceinline__ float tait_pressure(float rho, const Consts& c) {
  const float x = XDIV(rho, c.rho0);
  float p7 = x;
#pragma unroll
  for (int k = 1; k < 7; ++k) p7 = XMUL(p7, x);
  return XMUL(c.K, XSUB(p7, 1.f));
}

__device__ __forceinline__ float4 density_aux(float rho, const Consts& c) {
  const float p = tait_pressure(rho, c);
  return make_float4(rho, p, XDIV(c.mass, rho), XDIV(p, XMUL(rho, rho)));
}

// m * W_poly6(r) for a contributing pair (forces.cl:33-36, smoothing.cl:1-4).
__device__ __forceinline__ float poly6_term(float rr, float hh, const Consts& c) {
  const float q = XSUB(hh, XMUL(rr, rr));
  return XMUL(c.mass, XMUL(c.poly6, XMUL(XMUL(q, q), q)));
}

struct ForceSums {
  V3 P, Vs, Nm;
  float lap;
};

// One contributing pair of forces.cl:67-97; mj = m/rho_j, qj = p_j/rho_j^2.
// kShort: the quotients share one reciprocal.
template <bool kShort>
__device__ __forceinline__ void force_pair(ForceSums& f, bool self, V3 d, float rr, float4 vi, float4 vj, float mj,
                                           float qj, float own, float hh, float lap_b, const Consts& c) {
  if (!self) {
    const float coef = XMUL(XADD(qj, own), c.mass);
    V3 sg;
    if (XSUB(rr, 0.0000001f) < 0.f) {  // smoothing.cl:23-25
      sg = {c.spiky_zero, c.spiky_zero, c.spiky_zero};
    } else {
      const float q = XSUB(c.h, rr);
      const float q2 = XMUL(q, q);
      const float y = kShort ? rcp_rn_normal(rr) : 0.f;
      auto over_r = [&](float x) { return kShort ? div_rn_normal(x, rr, y) : XDIV(x, rr); };
      sg = {XMUL(XMUL(c.spiky, over_r(d.x)), q2), XMUL(XMUL(c.spiky, over_r(d.y)), q2),
            XMUL(XMUL(c.spiky, over_r(d.z)), q2)};
    }
    f.P.x = XADD(f.P.x, XMUL(coef, sg.x));
    f.P.y = XADD(f.P.y, XMUL(coef, sg.y));
    f.P.z = XADD(f.P.z, XMUL(coef, sg.z));
    const float vl = XMUL(c.visc, XSUB(c.h, rr));
    f.Vs.x = XADD(f.Vs.x, XMUL(XMUL(XSUB(vj.x, vi.x), mj), vl));
    f.Vs.y = XADD(f.Vs.y, XMUL(XMUL(XSUB(vj.y, vi.y), mj), vl));
    f.Vs.z = XADD(f.Vs.z, XMUL(XMUL(XSUB(vj.z, vi.z), mj), vl));
  }
  const float q = XSUB(hh, XMUL(rr, rr));
  const float q2 = XMUL(q, q);
  f.Nm.x = XADD(f.Nm.x, XMUL(mj, XMUL(XMUL(c.grad6, d.x), q2)));
  f.Nm.y = XADD(f.Nm.y, XMUL(mj, XMUL(XMUL(c.grad6, d.y), q2)));
  f.Nm.z = XADD(f.Nm.z, XMUL(mj, XMUL(XMUL(c.grad6, d.z), q2)));
  f.lap = XADD(f.lap, XMUL(mj, XMUL(XMUL(c.lap6, q), XSUB(lap_b, XMUL(7.f, XMUL(rr, rr))))));
}

// forces.cl:103-109 then sph.cl:53-58.
__device__ __forceinline__ float4 finish_accel(const ForceSums& f, float rho_i, const Consts& c) {
  const float nr = -rho_i;
  V3 sum = {XADD(XMUL(nr, f.P.x), XMUL(f.Vs.x, c.mu)), XADD(XMUL(nr, f.P.y), XMUL(f.Vs.y, c.mu)),
            XADD(XMUL(nr, f.P.z), XMUL(f.Vs.z, c.mu))};
  const float nl = xnorm(f.Nm);
  if (nl > c.sigma_threshold) {
    const float s = XMUL(-c.sigma, f.lap);
    sum.x = XADD(sum.x, XDIV(XMUL(s, f.Nm.x), nl));
    sum.y = XADD(sum.y, XDIV(XMUL(s, f.Nm.y), nl));
    sum.z = XADD(sum.z, XDIV(XMUL(s, f.Nm.z), nl));
  }
  return make_float4(XADD(XDIV(sum.x, rho_i), c.gx), XADD(XDIV(sum.y, rho_i), c.gy),
                     XADD(XDIV(sum.z, rho_i), c.gz), 0.f);
}

// Calls f(j) for every candidate of particle i's window in the reference's order.
template <class F>
__device__ __forceinline__ void for_each_candidate(const Window& w, uint32_t sbits,
                                                   const CellIndex& ci, F&& f) {
  for (uint32_t z = w.lo[2]; z <= w.hi[2]; ++z)
    for (uint32_t y = w.lo[1]; y <= w.hi[1]; ++y)
      for (uint32_t x = w.lo[0]; x <= w.hi[0]; ++x) {
        const uint2 r = cell_lookup(ci, morton3(x, y, z) | sbits);
        for (uint32_t j = r.x; j < r.y; ++j) f(j);
      }
}

// Density (forces.cl:15-43) + Tait pressure (sph.cl:36-39) + neighbour list.
// One thread per particle, two phases:
//  1. walk the window cells (z, y, x order; each cell's particles in sorted
//     order). A particle in a neighbour cell that lies in the half facing
//     away from this particle's cell (per its half code in pos.w) is more
//     than h away: skipped with one bit test. The others get an FMA distance
//     cull; survivors are buffered per thread in shared memory;
//  2. evaluate the survivors with exact arithmetic, in the same order, in
//     lock-step across the warp (the expensive part is no longer divergent).
// A thread with more survivors than its buffer repeats phase 1 inline.
constexpr int kScanCap = 48;

// Bits of a neighbour's half code that must be set for it to face cell
// offset (ox, oy, oz): its upper half when it is below, lower half when above.
__device__ __forceinline__ uint32_t facing_mask(int ox, int oy, int oz) {
  uint32_t m = 0;
  if (ox < 0) m |= 2u;
  if (ox > 0) m |= 1u;
  if (oy < 0) m |= 8u;
  if (oy > 0) m |= 4u;
  if (oz < 0) m |= 32u;
  if (oz > 0) m |= 16u;
  return m;
}

// Neighbour-list tags: the neighbour's cell as its index k < 27 among the 27
// cells around the particle's own cell (z, y, x order, 13 = own) in bits
// 11-15 and its offset in that cell in bits 0-10; a cell of 2048 or more
// particles cannot be tagged (kNoTag) and sends its particles to the rescan.
constexpr uint32_t kTagOffBits = 11;
constexpr uint32_t kNoTag = 0xFFFFu;
__device__ __forceinline__ uint32_t nb_tag(uint32_t k, uint32_t off) {
  return off < (1u << kTagOffBits) ? (k << kTagOffBits) | off : kNoTag;
}

// Calls f(j, pj, tag) for every candidate of the window that faces the
// particle's cell, in the reference's order, and g(k, start) once per window
// cell before its candidates.
template <class F, class G>
__device__ __forceinline__ void for_each_facing_candidate(const Window& w, uint32_t key,
                                                          uint32_t sbits, const CellIndex& ci,
                                                          const float4* __restrict__ pos, F&& f,
                                                          G&& g) {
  const int c[3] = {(int)compact_bits3(key), (int)compact_bits3(key >> 1), (int)compact_bits3(key >> 2)};
  for (uint32_t z = w.lo[2]; z <= w.hi[2]; ++z)
    for (uint32_t y = w.lo[1]; y <= w.hi[1]; ++y)
      for (uint32_t x = w.lo[0]; x <= w.hi[0]; ++x) {
        const int ox = (int)x - c[0], oy = (int)y - c[1], oz = (int)z - c[2];
        const uint32_t need = facing_mask(ox, oy, oz);
        const uint32_t k = (uint32_t)((oz + 1) * 9 + (oy + 1) * 3 + (ox + 1));
        const uint2 r = cell_lookup(ci, morton3(x, y, z) | sbits);
        g(k, r.x);
        for (uint32_t j = r.x; j < r.y; ++j) {
          const float4 pj = __ldg(&pos[j]);
          if ((__float_as_uint(pj.w) & need) == need) f(j, pj, nb_tag(k, j - r.x));
        }
      }
}
template <class F>
__device__ __forceinline__ void for_each_facing_candidate(const Window& w, uint32_t key,
                                                          uint32_t sbits, const CellIndex& ci,
                                                          const float4* __restrict__ pos, F&& f) {
  for_each_facing_candidate(w, key, sbits, ci, pos, f, [](uint32_t, uint32_t) {});
}

// Per-particle outputs of the density pass: aux = (rho, p, first slot of the
// particle's own cell as bits, p/rho^2) (the forces kernel resolves the
// neighbour tags through that cell's nb_start row), the forces kernel's two
// 16-byte neighbour records (position, m/rho) and (velocity, p/rho^2), and the
// neighbour count (> nlist_cap: the list is incomplete or holds an untaggable
// neighbour, so the forces kernel searches again).
__device__ __forceinline__ void density_outputs(uint32_t i, uint32_t n, float rho, const Consts& c,
                                                uint32_t own_start, float4 pi, const float4* __restrict__ vel,
                                                float4* __restrict__ aux_out, float4* __restrict__ frec,
                                                uint32_t* __restrict__ ncount, uint32_t count) {
  const float4 a = density_aux(rho, c);
  aux_out[i] = make_float4(a.x, a.y, __uint_as_float(own_start), a.w);
  const float4 v = vel[i];
  frec[i] = make_float4(pi.x, pi.y, pi.z, a.z);
  frec[(size_t)n + i] = make_float4(v.x, v.y, v.z, a.w);
  ncount[i] = count;
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK)
    k_density(uint32_t n, const DevGrid* __restrict__ grids, const uint16_t* __restrict__ scene_of,
              const uint32_t* __restrict__ ctl,
              const uint32_t* __restrict__ keys_base, const float4* __restrict__ pos, CellIndex ci,
              const Consts* __restrict__ consts, float4* __restrict__ aux_out,
              uint16_t* __restrict__ nlist, uint32_t* __restrict__ ncount, uint32_t nlist_cap,
              const float4* __restrict__ vel, float4* __restrict__ frec, uint32_t* __restrict__ nb_start) {
  if (never_after_previous()) return;
  __shared__ uint16_t cand[kScanCap][BLOCK];  // tags of the cull's survivors
  __shared__ uint32_t cstart[27][BLOCK];      // first slot of each window cell
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const KeySplit split{ctl[kCtlShift]};
  const uint32_t sc = scene_of[i];
  const Consts c = consts[sc];
  const uint32_t sbits = split.scene_bits(sc);
  const uint32_t* keys = keys_base + (size_t)sorted_sel(ctl[kCtlMaxKey]) * n;
  const uint32_t key = split.morton(keys[i]);
  const float4 pi = pos[i];
  const Window w = neighbour_window(pi, key, grids[sc]);
  const float hh = XMUL(c.h, c.h);
  uint32_t found = 0;
  for_each_facing_candidate(
      w, key, sbits, ci, pos,
      [&](uint32_t, float4 pj, uint32_t tag) {
        const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        if (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= c.cull_r2) {
          if (found < kScanCap) cand[found][threadIdx.x] = (uint16_t)tag;
          found = tag == kNoTag ? kScanCap + 1u : found + 1u;  // untaggable: rescan
        }
      },
      [&](uint32_t k, uint32_t start) { cstart[k][threadIdx.x] = start; });
  const uint32_t own_start = cstart[13][threadIdx.x];
  float rho = 0.f;
  uint32_t kept = 0;
  bool untagged = false;
  auto visit = [&](uint32_t j, float4 pj, uint32_t tag) {
    const V3 d = {XSUB(pi.x, pj.x), XSUB(pi.y, pj.y), XSUB(pi.z, pj.z)};
    const float rr = xnorm(d);
    if (rr < c.h) {
      rho = XADD(rho, poly6_term(rr, hh, c));
      if (tag == kNoTag) untagged = true;
      else if (kept < nlist_cap) __stcs(&nlist[(size_t)kept * n + i], (uint16_t)tag);
      ++kept;
    }
  };
  if (found <= (uint32_t)kScanCap) {
    for (uint32_t k = 0; k < found; ++k) {
      const uint32_t tag = cand[k][threadIdx.x];
      const uint32_t j = cstart[tag >> kTagOffBits][threadIdx.x] + (tag & ((1u << kTagOffBits) - 1u));
      visit(j, __ldg(&pos[j]), tag);
    }
  } else {
    for_each_facing_candidate(w, key, sbits, ci, pos, [&](uint32_t j, float4 pj, uint32_t tag) {
      const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
      if (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= c.cull_r2) visit(j, pj, tag);
    });
  }
  // the own cell's row of the neighbour-start table (every particle of the
  // cell writes the same values for the cells of its window)
  const int cc[3] = {(int)compact_bits3(key), (int)compact_bits3(key >> 1), (int)compact_bits3(key >> 2)};
  for (uint32_t z = w.lo[2]; z <= w.hi[2]; ++z)
    for (uint32_t y = w.lo[1]; y <= w.hi[1]; ++y)
      for (uint32_t x = w.lo[0]; x <= w.hi[0]; ++x) {
        const uint32_t k = (uint32_t)(((int)z - cc[2] + 1) * 9 + ((int)y - cc[1] + 1) * 3 + ((int)x - cc[0] + 1));
        nb_start[(size_t)own_start * 27u + k] = cstart[k][threadIdx.x];
      }
  density_outputs(i, n, rho, c, own_start, pi, vel, aux_out, frec, ncount,
                  untagged ? max(kept, nlist_cap + 1u) : kept);
}

// ------------------------------------------------- density, one particle by a warp
// The warp walks the particle's window cells in the reference's order, 32
// candidates at a time (far halves skipped by half code, FMA cull), every
// lane evaluates its candidate exactly, and the contributing terms are added
// to the density one after another in lane order (ballot + shuffle), which is
// the reference's visiting order; survivors append to the neighbour list in
// the same order.
__device__ __forceinline__ bool near_cull(const float4& p, const float4& q, float r2) {
  const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
  return fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= r2;
}

template <bool kLive = false>
__device__ __forceinline__ void density_particle_warp(
    uint32_t i, uint32_t n, const DevGrid* __restrict__ grids, const uint16_t* __restrict__ scene_of,
    const KeySplit& split, const uint32_t* __restrict__ keys, const float4* __restrict__ pos, const CellIndex& ci,
    const Consts* __restrict__ consts, float4* __restrict__ aux_out, uint16_t* __restrict__ nlist,
    uint32_t* __restrict__ ncount, uint32_t nlist_cap, const float4* __restrict__ vel, float4* __restrict__ frec,
    uint32_t* __restrict__ nb_start) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t sc = scene_of[i];
  const Consts& c = consts[sc];
  const uint32_t sbits = split.scene_bits(sc);
  const uint32_t key = split.morton(keys[i]);
  const float4 pi = pos[i];
  const Window w = neighbour_window(pi, key, grids[sc]);
  const int cc[3] = {(int)compact_bits3(key), (int)compact_bits3(key >> 1), (int)compact_bits3(key >> 2)};
  const float hh = XMUL(c.h, c.h);
  const float h = c.h, cull_r2 = c.cull_r2;
  float rho = 0.f;
  uint32_t kept = 0;
  bool untagged = false;
  // lane k < 27 looks up window cell k (z, y, x order) in parallel
  uint32_t cs = 0, ce = 0;
  bool inw = false;
  if (lane < 27u) {
    const uint32_t x = (uint32_t)cc[0] + lane % 3u - 1u, y = (uint32_t)cc[1] + (lane / 3u) % 3u - 1u,
                   z = (uint32_t)cc[2] + lane / 9u - 1u;
    inw = x >= w.lo[0] && x <= w.hi[0] && y >= w.lo[1] && y <= w.hi[1] && z >= w.lo[2] && z <= w.hi[2];
    if (inw) {
      const uint2 r = cell_lookup<kLive>(ci, morton3(x, y, z) | sbits);
      cs = r.x;
      ce = r.y;
    }
  }
  const uint32_t own_start = __shfl_sync(0xFFFFFFFFu, cs, 13);
  if (inw) nb_start[(size_t)own_start * 27u + lane] = cs;  // the same values from every particle of the cell
  uint32_t cells = __ballot_sync(0xFFFFFFFFu, inw && ce > cs);
  while (cells) {
    const uint32_t k = __ffs(cells) - 1u;
    cells &= cells - 1u;
    const uint32_t need = facing_mask((int)(k % 3u) - 1, (int)((k / 3u) % 3u) - 1, (int)(k / 9u) - 1);
    const uint2 r = make_uint2(__shfl_sync(0xFFFFFFFFu, cs, k), __shfl_sync(0xFFFFFFFFu, ce, k));
    for (uint32_t cb = r.x; cb < r.y; cb += 32u) {
      const uint32_t j = cb + lane;
      bool hit = false;
      float term = 0.f;
      if (j < r.y) {
        const float4 pj = ld_step<kLive>(&pos[j]);
        if ((__float_as_uint(pj.w) & need) == need && near_cull(pi, pj, cull_r2)) {
          const V3 d = {XSUB(pi.x, pj.x), XSUB(pi.y, pj.y), XSUB(pi.z, pj.z)};
          const float rr = xnorm(d);
          if (rr < h) {
            hit = true;
            term = poly6_term(rr, hh, c);
          }
        }
      }
      uint32_t bal = __ballot_sync(0xFFFFFFFFu, hit);
      const uint32_t tag = nb_tag(k, j - r.x);
      untagged |= __any_sync(0xFFFFFFFFu, hit && tag == kNoTag);
      const uint32_t at = kept + __popc(bal & lt);
      if (hit && at < nlist_cap) __stcs(&nlist[(size_t)at * n + i], (uint16_t)tag);
      kept += __popc(bal);
      while (bal) {  // in lane order: the reference's summation sequence
        const int l = __ffs(bal) - 1;
        rho = XADD(rho, __shfl_sync(0xFFFFFFFFu, term, l));
        bal &= bal - 1u;
      }
    }
  }
  if (lane == 0)
    density_outputs(i, n, rho, c, own_start, pi, vel, aux_out, frec, ncount,
                    untagged ? max(kept, nlist_cap + 1u) : kept);
}

// Density + pressure + neighbour list with one warp per particle, for scenes
// too small to fill the GPU with one thread per particle or one team per cell.
constexpr int kParticleWarps = 8;

static __global__ void __launch_bounds__(kParticleWarps * 32)
    k_density_pwarp(uint32_t n, const DevGrid* __restrict__ grids, const uint16_t* __restrict__ scene_of,
                    const uint32_t* __restrict__ ctl, const uint32_t* __restrict__ keys_base,
                    const float4* __restrict__ pos, CellIndex ci, const Consts* __restrict__ consts,
                    float4* __restrict__ aux_out, uint16_t* __restrict__ nlist,
                    uint32_t* __restrict__ ncount, uint32_t nlist_cap, const float4* __restrict__ vel,
                    float4* __restrict__ frec, uint32_t* __restrict__ nb_start) {
  if (never_after_previous()) return;
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= n) return;  // whole warps
  const KeySplit split{ctl[kCtlShift]};
  const uint32_t* keys = keys_base + (size_t)sorted_sel(ctl[kCtlMaxKey]) * n;
  density_particle_warp(i, n, grids, scene_of, split, keys, pos, ci, consts, aux_out, nlist, ncount, nlist_cap, vel,
                        frec, nb_start);
}

// ------------------------------------------------- density, one team of warps per cell
// A team of warps takes one occupied cell at a time (dynamic work counter):
//  1. one warp looks up the 27 cells around it (lane k < 27: offset k in the
//     reference's z, y, x loop order; also stored as the cell's nb_start row)
//     and reads, from the half codes' bit planes, which of their particles
//     face the own cell (the far half is skipped, as in k_density): the
//     cell's candidates, whose tags it writes in visiting order;
//  2. a particle in one octant of the cell needs 8 of the 27 lists (its 2 x 2
//     x 2 window), 4 runs of consecutive candidates: the warp writes the
//     numbers of each octant's chunks of eight candidates;
//  3. all warps load the candidates' positions into the chunks: relative to
//     the own cell's centre in units of h, in half precision, with the
//     negated squared norm, candidate e beside candidate e + 4 so that one
//     packed operation tests both;
//  4. one lane per particle walks its octant's chunks: three packed FMAs and a
//     packed compare test two candidates, 2 p'.q' - |q'|^2 >= |p'|^2 - R^2,
//     and 32 candidates make one word of hit bits in shared memory, first
//     candidate in the top bit;
//  5. the lane walks its hit bits, which is the reference's visiting order,
//     and evaluates each survivor exactly, as in k_density, with the next
//     one's position in flight.
// The first warp prepares the next cell (1, 2) before it waits for the
// others. A chunk can hold candidates of a neighbouring list that the octant
// doesn't need (they lie more than h away: the exact test drops them), and
// one that two runs share is walked once. Particles that the lists don't
// serve are done by a whole warp each (density_particle_warp): those on a
// mid-plane of the cell, so in two octants; cells of up to kSparseCell
// particles, for which the lists cost more than they save; lists longer than
// the team's shared memory; and neighbours of a cell of 2048 or more particles,
// which tags can't address. Every scene's h lies in near_norm's range (handles
// with another take a search of their own).
//
// Bound: instruction issue, half of it the exact evaluation. 1,048,576
// particles spread over a floor (29,552 cells, a quarter of them of one or
// two particles): 212 M warp instructions, 60 % of the issue slots, 0.303 ms,
// against 313 M and 0.454 ms for the form before, one warp per cell that
// tested each of its 64 particles against all 512 candidates in FP32; the
// same on the h/2 lattice: 0.230 ms against 0.359. Of the 212 M: the cell's
// look-up and the outputs 38 M, candidates 24 M, culls 38 M (an octant's 216
// candidates instead of 512, two per operation), exact evaluation 112 M.
// Staging with FP32 positions streamed per neighbour list and compacted by
// ballot took 104 M (each list's far half is read and dropped, and a list
// rarely fills its warps); planes cost one bit per particle and axis half.
//
// Rounding of the cull, in units of h, for a particle whose coordinates are at
// most g = 1 + 1/64 (kCellGate; others, in cells whose centre is rounded far
// from the origin, are not served) and a candidate within 1 of it:
// |p'| < 1.76, |q'| < 2.76, |q'|^2 < 7.62.
//  2 p' (below 4) is off by 2^-10 a component: 2^-10 sqrt(3) 2.76 = 4.7e-3 in
//   the product; q' by 2^-11 a component below 2: 2 g 3 * 2^-11 = 3.0e-3, or
//   2^-10 for one above 2 (then p' and q' lie close together in the other two,
//   and the sums are 4.2e-3 and 4.0e-3): 8.2e-3 in all;
//  |q'|^2 and the first FMA are below 8, 2^-9 each; the second below 4, 2^-10
//   (if not, p' is near an axis and the product's share below 5.6e-3); the last,
//   |p'|^2 - |p' - q'|^2, below 4, 2^-10: 5.9e-3.
// 1.41e-2 in all (1.40e-2 is the largest of 10^7 draws; at 1.25 it would be
// 1.76e-2), and |p'|^2 - R^2 is rounded down. So every candidate within h
// passes with R^2 = 1.015; the exact evaluation decides.
constexpr float kCellCullR2 = 1.015f;
constexpr float kCellGate = 1.015625f;
constexpr uint32_t kCellOffBits = kTagOffBits;

// Per neighbour offset k (z, y, x order): the half-code bits a candidate of
// that cell needs to face the own cell, facing_mask(o).
struct OffsetMasks {
  uint8_t m[27];
};
constexpr OffsetMasks make_offset_masks() {
  OffsetMasks t{};
  for (int k = 0; k < 27; ++k) {
    const int o[3] = {k % 3 - 1, (k / 3) % 3 - 1, k / 9 - 1};
    uint32_t cand = 0;
    for (int a = 0; a < 3; ++a) {
      if (o[a] < 0) cand |= 2u << (2 * a);
      if (o[a] > 0) cand |= 1u << (2 * a);
    }
    t.m[k] = (uint8_t)cand;
  }
  return t;
}
__constant__ OffsetMasks kOffsetMasks = make_offset_masks();

// The cells of a particle's window as bits k < 27 (z, y, x order): on every
// axis offset 0, and -1 / +1 where its half code has the lower / upper bit.
// Bit k is set exactly when (code & facing_mask(-o)) == facing_mask(-o) for
// the cell's offset o.
__device__ __forceinline__ uint32_t window_cells(uint32_t code) {
  const uint32_t ax = 2u | (code & 1u) | ((code << 1) & 4u);
  const uint32_t ay = 2u | ((code >> 2) & 1u) | ((code >> 1) & 4u);
  const uint32_t az = 2u | ((code >> 4) & 1u) | ((code >> 3) & 4u);
  const uint32_t yx = ((ay & 1u) ? ax : 0u) | (ax << 3) | ((ay & 4u) ? ax << 6 : 0u);
  return ((az & 1u) ? yx : 0u) | (yx << 9) | ((az & 4u) ? yx << 18 : 0u);
}

// A cell of at most this many particles is done by a warp per particle.
constexpr uint32_t kSparseCell = 4;

// Shared memory of one team of WARPS warps: CHUNKS chunks for a cell's
// candidates (512, 64 chunks, on the h/2 lattice), WORDS mask words for an
// octant's (216, 7 words, and up to a chunk more per window row).
template <int WARPS, int CHUNKS, int WORDS>
struct CellTeamSmem {
  static constexpr int kWarps = WARPS;
  static constexpr uint32_t kChunks = CHUNKS, kWords = WORDS;
  static_assert(CHUNKS <= 256, "chunk numbers are bytes");
  uint4 chunk[CHUNKS][5];  // four pairs of four halves; eight 16-bit tags
  uint4 no_chunk[4];       // a chunk that never hits
  uint32_t mask[WARPS][WORDS][32];
  uint16_t pend[8 * CHUNKS];  // the next cell's candidates: their tags in visiting order
  // two sets of what is known of a cell: one is made while the other is read
  struct Cell {
    float4 origin;           // its centre and 1 / h
    uint32_t slot_of[32];    // slot minus tag of neighbour k's particles
    uint32_t seq[8][WORDS];  // an octant's chunk numbers, four to a word, first in the top byte
    uint32_t chunks[8];      // and their count
    uint32_t scene, first, count;  // its particles
    uint32_t candidates;     // kNoLists: the lists don't serve it; kNoCell: no cell left
  } cell[2];
};
constexpr uint32_t kNoLists = 0xFFFFFFFEu, kNoCell = 0xFFFFFFFFu;

// The slots of word `w` of the planes in [s, e) that have all of `need`.
template <bool kLive>
__device__ __forceinline__ uint32_t facing_slots(const uint32_t* __restrict__ planes, uint32_t w, uint32_t s,
                                                 uint32_t e, uint32_t need) {
  const uint32_t* p = planes + (size_t)w * kHalfPlanes;
  uint32_t m = 0xFFFFFFFFu;
#pragma unroll
  for (uint32_t b = 0; b < kHalfPlanes; b += 2) {  // an axis needs at most one of its two bits
    const uint32_t both = (need >> b) & 3u;
    const uint32_t v = ld_step<kLive>(&p[b + (both >> 1)]);  // (loaded in any case: the loads don't wait for one another)
    m &= both ? v : 0xFFFFFFFFu;
  }
  const uint32_t w0 = 32u * w;
  if (s > w0) m &= 0xFFFFFFFFu << (s - w0);
  if (e < w0 + 32u) m &= (1u << (e - w0)) - 1u;
  return m;
}

template <bool kLive = false, class Team>
__device__ __forceinline__ void density_cells_team(
    uint32_t n, const DevGrid* __restrict__ grids, const uint32_t* __restrict__ ctl,
    const uint16_t* __restrict__ scene_of, const uint32_t* __restrict__ keys_base, const float4* __restrict__ pos,
    const uint32_t* __restrict__ planes, const CellIndex& ci, const Consts* __restrict__ consts,
    float4* __restrict__ aux_out, uint16_t* __restrict__ nlist, uint32_t* __restrict__ ncount, uint32_t nlist_cap,
    const float4* __restrict__ vel, float4* __restrict__ frec, const uint2* __restrict__ cell_list,
    uint32_t* __restrict__ counters, uint32_t* __restrict__ nb_start, Team& sm, uint32_t wid, uint32_t team,
    uint32_t teams, uint32_t barrier_id) {
  constexpr uint32_t kWarps = Team::kWarps, kWords = Team::kWords;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt = (1u << lane) - 1u;
  auto team_sync = [&]() {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(barrier_id), "n"(kWarps * 32) : "memory");
  };
  constexpr uint32_t kNever = 0xFC00u;  // -infinity in half precision: a squared norm that no test accepts
  if (wid == 0 && lane < 4u) sm.no_chunk[lane] = make_uint4(0u, 0u, 0u, kNever * 0x10001u);
  const uint32_t ncells = counters[kCntCells];
  const KeySplit split{ctl[kCtlShift]};
  const bool whole_keys = split.shift + ctl[kCtlSceneBits] <= 32u;  // (if not, flagged, keys lose upper scene bits)
  auto by_warp = [&](uint32_t i) {
    density_particle_warp<kLive>(i, n, grids, scene_of, split, keys_base + (size_t)sorted_sel(ctl[kCtlMaxKey]) * n,
                                 pos, ci, consts, aux_out, nlist, ncount, nlist_cap, vel, frec, nb_start);
  };
  // the last warp, which has the fewest particles, looks the next cell up; the first two cells have fixed
  // numbers, the others come from the work counter, and both are loaded a cell ahead
  const bool fetcher = wid == kWarps - 1u;
  uint32_t ticket = team;
  uint2 entry = make_uint2(0u, 0u);
  bool have = false;
  auto load_entry = [&]() {
    have = ticket < ncells;
    if (have) entry = ld_step<kLive>(&cell_list[ticket]);
  };
  if (fetcher) {
    load_entry();
    ticket += teams;
  }
  for (uint32_t par = 0;; par ^= 1u) {
    typename Team::Cell& cell = sm.cell[par];
    if (fetcher && !have) {
      if (lane == 0) cell.candidates = kNoCell;
    } else if (fetcher) {
      const uint2 own = entry;
      const uint32_t key = split.morton(own.y);
      uint32_t s = 0, e = 0;
      if (lane < 27u) {
        const uint32_t x = compact_bits3(key) + lane % 3u - 1u, y = compact_bits3(key >> 1) + (lane / 3u) % 3u - 1u,
                       z = compact_bits3(key >> 2) + lane / 9u - 1u;
        const uint2 r = cell_lookup<kLive>(ci, morton3(x, y, z) | (own.y ^ key));
        s = lane == 13u ? own.x : r.x;  // (a flagged sort stall can leave the index with another start)
        e = r.y;
        nb_start[(size_t)own.x * 27u + lane] = s;
      }
      load_entry();
      uint32_t next = 0;
      if (lane == 0) next = atomicAdd(&counters[kCntWorkDensity], 1u);
      ticket = __shfl_sync(0xFFFFFFFFu, next, 0) + 2u * teams;
      const uint32_t own_e = __shfl_sync(0xFFFFFFFFu, e, 13);
      const uint32_t count = own_e > own.x ? own_e - own.x : 0u;
      uint32_t candidates = kNoLists;
      const uint32_t sc = whole_keys ? (split.shift >= 32u ? 0u : own.y >> split.shift) : scene_of[own.x];
      if (!__any_sync(0xFFFFFFFFu, e - s >= (1u << kCellOffBits)) && count > kSparseCell) {
        // the candidates of list k as bits, in up to three words of the planes (more are counted and read again)
        const uint32_t need = kOffsetMasks.m[min(lane, 26u)];
        const uint32_t w0 = s >> 5, words = e > s && lane != 13u ? ((e - 1u) >> 5) - w0 + 1u : 0u;
        uint32_t m[3];
#pragma unroll
        for (uint32_t w = 0; w < 3u; ++w) {
          const bool on = w < words;
          m[w] = facing_slots<kLive>(planes, on ? w0 + w : 0u, on ? s : 0u, on ? e : 1u, need) & (on ? 0xFFFFFFFFu : 0u);
        }
        if (count <= 32u) {  // only the neighbour cells in its particles' windows
          uint32_t any = 0;
          if (lane < kHalfPlanes)
            for (uint32_t w = own.x >> 5; w <= (own_e - 1u) >> 5; ++w)
              any |= facing_slots<kLive>(planes, w, own.x, own_e, 1u << lane);
          if (!((window_cells(__ballot_sync(0xFFFFFFFFu, any != 0u)) >> lane) & 1u)) m[0] = m[1] = m[2] = 0u;
        }
        uint32_t size = lane == 13u ? count : __popc(m[0]) + __popc(m[1]) + __popc(m[2]);
        for (uint32_t w = 3; w < words; ++w) size += __popc(facing_slots<kLive>(planes, w0 + w, s, e, need));
        uint32_t end = size;
#pragma unroll
        for (uint32_t d = 1; d < 32u; d <<= 1) {
          const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, end, d);
          if (lane >= d) end += y;
        }
        const uint32_t begin = end - size;
        const uint32_t all = __shfl_sync(0xFFFFFFFFu, end, 26);
        if (all <= 8u * Team::kChunks) {
          candidates = all;
          const uint32_t own_at = __shfl_sync(0xFFFFFFFFu, begin, 13);
          for (uint32_t j = lane; j < count; j += 32u) sm.pend[own_at + j] = (uint16_t)((13u << kCellOffBits) + j);
          uint32_t tag = (lane << kCellOffBits) + 32u * w0 - s;  // of the first word's first slot
          uint32_t at = begin;
          for (uint32_t w = 2u; at < end && lane != 13u;) {
            while (m[0] == 0u) {
              m[0] = m[1];
              m[1] = m[2];
              ++w;
              m[2] = w < words ? facing_slots<kLive>(planes, w0 + w, s, e, need) : 0u;
              tag += 32u;
            }
            sm.pend[at++] = (uint16_t)(tag + __ffs(m[0]) - 1u);
            m[0] &= m[0] - 1u;
          }
          // octant o's chunks in visiting order: lane (o, r) appends those of window row r, two lists side by
          // side, without a chunk that an earlier row shares
          const uint32_t o = lane >> 2, r = lane & 3u;
          const uint32_t k = (o & 1u) + 3u * (((o >> 1) & 1u) + (r & 1u)) + 9u * ((o >> 2) + (r >> 1));
          const uint32_t a = __shfl_sync(0xFFFFFFFFu, begin, k), b = __shfl_sync(0xFFFFFFFFu, end, k + 1u);
          uint32_t c0 = a >> 3;
          const uint32_t c1 = b > a ? (b + 7u) >> 3 : 0u;  // chunks [c0, c1)
          uint32_t seen = c1;
#pragma unroll
          for (uint32_t d = 1; d < 4u; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, seen, d, 4);
            if (r >= d) seen = max(seen, y);
          }
          const uint32_t before = __shfl_up_sync(0xFFFFFFFFu, seen, 1, 4);
          if (r) c0 = max(c0, before);
          const uint32_t cnt = c1 > c0 ? c1 - c0 : 0u;
          uint32_t last = cnt;
#pragma unroll
          for (uint32_t d = 1; d < 4u; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, last, d, 4);
            if (r >= d) last += y;
          }
          uint8_t* out = reinterpret_cast<uint8_t*>(cell.seq[o]);
          uint32_t i = last - cnt;
          for (uint32_t c = c0; c < c1 && i < 4u * kWords; ++c, ++i) out[i ^ 3u] = (uint8_t)c;
          if (r == 3u) cell.chunks[o] = last;
        }
      }
      cell.slot_of[lane] = s - (lane << kCellOffBits);
      if (lane == 0) {
        const DevGrid& g = grids[sc];
        cell.origin = make_float4(g.lo[0] + ((float)compact_bits3(key) + 0.5f) * g.cell,
                                  g.lo[1] + ((float)compact_bits3(key >> 1) + 0.5f) * g.cell,
                                  g.lo[2] + ((float)compact_bits3(key >> 2) + 0.5f) * g.cell, 1.f / consts[sc].h);
        cell.scene = sc;
        cell.first = own.x;
        cell.count = count;
        cell.candidates = candidates;
      }
    }
    team_sync();
    const uint32_t candidates = cell.candidates, first = cell.first, count = cell.count;
    if (candidates == kNoCell) break;
    if (candidates == kNoLists) {
      for (uint32_t q = wid; q < count; q += kWarps) by_warp(first + q);
      continue;
    }
    const float4 org = cell.origin;
    constexpr uint32_t kAhead = 4;  // candidates in flight per thread
    for (uint32_t e0 = 32u * wid + lane; e0 < candidates; e0 += 32u * kWarps * kAhead) {
      uint32_t tag[kAhead];
      float4 q[kAhead];
#pragma unroll
      for (uint32_t u = 0; u < kAhead; ++u) {
        const uint32_t e = min(e0 + 32u * kWarps * u, candidates - 1u);
        tag[u] = sm.pend[e];
        q[u] = ld_step<kLive>(&pos[cell.slot_of[tag[u] >> kCellOffBits] + tag[u]]);
      }
#pragma unroll
      for (uint32_t u = 0; u < kAhead; ++u) {
        const uint32_t e = e0 + 32u * kWarps * u;
        if (e >= candidates) break;
        const float x = (q[u].x - org.x) * org.w, y = (q[u].y - org.y) * org.w, z = (q[u].z - org.z) * org.w;
        uint4* c = sm.chunk[e >> 3];
        __half* h = reinterpret_cast<__half*>(&c[e & 3u]) + ((e >> 2) & 1u);
        h[0] = __float2half_rn(x);
        h[2] = __float2half_rn(y);
        h[4] = __float2half_rn(z);
        h[6] = __float2half_rn(-fmaf(x, x, fmaf(y, y, z * z)));
        reinterpret_cast<uint16_t*>(&c[4])[~e & 7u] = (uint16_t)tag[u];
      }
    }
    if (wid == 0 && lane < (0u - candidates & 7u)) {  // the last chunk's free places
      const uint32_t e = candidates + lane;
      reinterpret_cast<uint16_t*>(&sm.chunk[e >> 3][e & 3u])[6u + ((e >> 2) & 1u)] = (uint16_t)kNever;
    }
    team_sync();
    const Consts& c = consts[cell.scene];
    for (uint32_t base = 32u * wid; base < count; base += 32u * kWarps) {
      const bool valid = base + lane < count;
      const uint32_t i = first + (valid ? base + lane : 0u);
      const float4 pi = pos[i];
      const uint32_t code = __float_as_uint(pi.w);
      const float x = (pi.x - org.x) * org.w, y = (pi.y - org.y) * org.w, z = (pi.z - org.z) * org.w;
      // the particle's octant, from its upper-half bits when each axis has exactly one
      const uint32_t up = (code >> 1) & 0x15u;
      const uint32_t o = (up & 1u) | ((up >> 1) & 2u) | ((up >> 2) & 4u);
      uint32_t nc = cell.chunks[o];
      const bool served = valid && ((code ^ up) & 0x15u) == 0x15u &&
                          fmaxf(fmaxf(fabsf(x), fabsf(y)), fabsf(z)) <= kCellGate && nc <= 4u * kWords;
      if (!served) nc = 0u;
      const uint32_t nw = (__reduce_max_sync(0xFFFFFFFFu, nc) + 3u) >> 2;
      const __half2 px = __float2half2_rn(2.f * x), py = __float2half2_rn(2.f * y), pz = __float2half2_rn(2.f * z);
      const __half2 pt = __half2half2(__float2half_rd(fmaf(x, x, fmaf(y, y, z * z)) - kCellCullR2));
      const uint32_t* seq = cell.seq[o];
      uint32_t* mask = &sm.mask[wid][0][lane];
      uint32_t found = 0;
      for (uint32_t w = 0; w < nw; ++w) {
        const uint32_t ids = seq[w];
        uint32_t acc = 0;
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
          const uint4* ch = 4u * w + q < nc ? sm.chunk[(ids >> (24u - 8u * q)) & 255u] : sm.no_chunk;
#pragma unroll
          for (uint32_t u = 0; u < 4u; ++u) {
            const uint4 v = ch[u];
            auto h2 = [](uint32_t b) { return *reinterpret_cast<const __half2*>(&b); };
            const __half2 t = __hfma2(px, h2(v.x), __hfma2(py, h2(v.y), __hfma2(pz, h2(v.z), h2(v.w))));
            acc |= __hge2_mask(t, pt) & (0x80008000u >> (4u * q + u));
          }
        }
        // halves to candidate order: the upper half's nibble of each chunk after the lower half's
        uint32_t m = __byte_perm(acc, 0u, 0x1302);
        m ^= ((m ^ (m >> 4)) & 0x00F000F0u) * 17u;
        mask[32u * w] = m;
        found += __popc(m);
      }
      const float hh = XMUL(c.h, c.h);
      float rho = 0.f;
      uint32_t kept = 0;
      uint16_t* list = nlist + i;
      uint32_t m = 0, ids = 0, w = 0;
      auto next = [&](uint32_t& tag) {  // the next survivor's tag and position
        while (m == 0u) {
          m = mask[32u * w];
          ids = seq[w];
          ++w;
        }
        const uint32_t b = 31u - __clz(m);
        m ^= 1u << b;
        tag = reinterpret_cast<const uint16_t*>(&sm.chunk[(ids >> (b & 24u)) & 255u][4])[b & 7u];
        return ld_step<kLive>(&pos[cell.slot_of[tag >> kCellOffBits] + tag]);
      };
      uint32_t tag = 0;
      float4 pj = make_float4(0.f, 0.f, 0.f, 0.f);
      if (found) pj = next(tag);
      const float ch = c.h, cm = c.mass, c6 = c.poly6;
      for (uint32_t k = 0; k < found;) {
        uint32_t tagn = 0;
        float4 pn = pj;
        if (++k < found) pn = next(tagn);
        const V3 d = {XSUB(pi.x, pj.x), XSUB(pi.y, pj.y), XSUB(pi.z, pj.z)};
        const float rr = near_norm(d);
        const bool hit = rr < ch;
        const float qq = XSUB(hh, XMUL(rr, rr));
        const float sum = XADD(rho, XMUL(cm, XMUL(c6, XMUL(XMUL(qq, qq), qq))));
        rho = hit ? sum : rho;
        if (hit && kept < nlist_cap) __stcs(list + (uint64_t)kept * n, (uint16_t)tag);
        kept += hit ? 1u : 0u;
        tag = tagn;
        pj = pn;
      }
      if (served) density_outputs(i, n, rho, c, first, pi, vel, aux_out, frec, ncount, kept);
      uint32_t rest = __ballot_sync(0xFFFFFFFFu, valid && !served);
      while (rest) {
        by_warp(first + base + __ffs(rest) - 1u);
        rest &= rest - 1u;
      }
    }
  }
}

template <class Team, int BLOCKS>
__global__ void __launch_bounds__(Team::kWarps * 32, BLOCKS)
    k_density_cells(uint32_t n, const DevGrid* __restrict__ grids,
                    const uint16_t* __restrict__ scene_of, const uint32_t* __restrict__ ctl,
                    const uint32_t* __restrict__ keys_base, const float4* __restrict__ pos,
                    const uint32_t* __restrict__ planes, CellIndex ci, const Consts* __restrict__ consts,
                    float4* __restrict__ aux_out, uint16_t* __restrict__ nlist, uint32_t* __restrict__ ncount,
                    uint32_t nlist_cap, const float4* __restrict__ vel,
                    float4* __restrict__ frec, const uint2* __restrict__ cell_list,
                    uint32_t* __restrict__ counters, uint32_t* __restrict__ nb_start) {
  if (never_after_previous()) return;
  __shared__ Team sm;
  density_cells_team(n, grids, ctl, scene_of, keys_base, pos, planes, ci, consts, aux_out, nlist, ncount, nlist_cap, vel,
                     frec, cell_list, counters, nb_start, sm, threadIdx.x >> 5, blockIdx.x, gridDim.x, 1u);
}

// Per-pair hook of k_forces (the learned stepper gathers its neighbour
// features in the same walk); the plain substep uses this empty one.
struct NoForceHook {
  static constexpr bool kPairs = false;  // needs no visit of every pair by the particle's own lane
  struct Acc {};
  __device__ __forceinline__ Acc begin(uint32_t) const { return {}; }
  __device__ __forceinline__ void pair(Acc&, uint32_t, uint32_t, const V3&, const V3&) const {}
  __device__ __forceinline__ void end(Acc&, uint32_t, const float4&) const {}
};

// Forces of one particle by a whole warp, for particles without a complete
// neighbour list: the window's cells in the reference's order, 32 candidates
// at a time; each lane evaluates its candidate and the contributing terms are
// added one after another in lane order, which is the reference's sequence.
// (One lane alone walks its 500 to 1,000 candidates in about 150 us, which a
// single such particle adds to the kernel; the warp takes a few us.)
template <bool kLive = false>
__device__ __forceinline__ void forces_particle_warp(uint32_t i, uint32_t n, const DevGrid* grids,
                                                     const uint16_t* scene_of, const uint32_t* ctl,
                                                     const uint32_t* keys_base, const State& st, const float4* aux,
                                                     const CellIndex& ci, const Consts* consts, float4* acc_out,
                                                     const float4* frec) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t sc = scene_of[i];
  const Consts& c = consts[sc];
  const KeySplit split{ctl[kCtlShift]};
  const float4 pi = st.pos[i], vi = st.vel[i], ai = aux[i];
  const float hh = XMUL(c.h, c.h), lap_b = XMUL(3.f, hh);
  const Window w = neighbour_window(pi, split.morton(keys_base[(size_t)sorted_sel(ctl[kCtlMaxKey]) * n + i]), grids[sc]);
  ForceSums f = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, 0.f};
  for (uint32_t z = w.lo[2]; z <= w.hi[2]; ++z)
    for (uint32_t y = w.lo[1]; y <= w.hi[1]; ++y)
      for (uint32_t x = w.lo[0]; x <= w.hi[0]; ++x) {
        const uint2 r = cell_lookup<kLive>(ci, morton3(x, y, z) | split.scene_bits(sc));
        for (uint32_t base = r.x; base < r.y; base += 32u) {
          const uint32_t j = base + lane;
          bool hit = false;
          ForceSums t{};
          if (j < r.y) {
            const float4 pj = frec[j];
            const V3 d = {XSUB(pi.x, pj.x), XSUB(pi.y, pj.y), XSUB(pi.z, pj.z)};
            const float rr = xnorm(d);
            hit = near_cull(pi, pj, c.cull_r2) && rr < c.h;
            if (hit) {
              const float4 vj = frec[(size_t)n + j];
              force_pair<false>(t, j == i, d, rr, vi, vj, pj.w, vj.w, ai.w, hh, lap_b, c);
            }
          }
          for (uint32_t bal = __ballot_sync(0xFFFFFFFFu, hit); bal; bal &= bal - 1u) {
            const int l = __ffs(bal) - 1;
            // (a sum that starts at +0 is never -0, so adding the +0 of a term that doesn't count changes nothing)
            auto add = [&](float& sum, float term) { sum = XADD(sum, __shfl_sync(0xFFFFFFFFu, term, l)); };
            auto add3 = [&](V3& sum, const V3& term) { add(sum.x, term.x), add(sum.y, term.y), add(sum.z, term.z); };
            add3(f.P, t.P), add3(f.Vs, t.Vs), add3(f.Nm, t.Nm), add(f.lap, t.lap);
          }
        }
      }
  if (lane == 0) acc_out[i] = finish_accel(f, ai.x, c);
}

// The same by the particle's own lane, for hooks that visit every pair.
template <class Hook>
__device__ __forceinline__ void forces_particle_alone(uint32_t i, uint32_t n, const DevGrid* grids,
                                                      const uint16_t* scene_of, const uint32_t* ctl,
                                                      const uint32_t* keys_base, const State& st, const float4* aux,
                                                      const CellIndex& ci, const Consts* consts, float4* acc_out,
                                                      const Hook& hook, const float4* frec) {
  typename Hook::Acc ha = hook.begin(i);
  const uint32_t sc = scene_of[i];
  const Consts& c = consts[sc];
  const KeySplit split{ctl[kCtlShift]};
  const float4 pi = st.pos[i], vi = st.vel[i], ai = aux[i];
  const float hh = XMUL(c.h, c.h), lap_b = XMUL(3.f, hh);
  const Window w = neighbour_window(pi, split.morton(keys_base[(size_t)sorted_sel(ctl[kCtlMaxKey]) * n + i]), grids[sc]);
  ForceSums f = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, 0.f};
  for_each_candidate(w, split.scene_bits(sc), ci, [&](uint32_t j) {
    const float4 pj = frec[j];
    if (!near_cull(pi, pj, c.cull_r2)) return;
    const V3 d = {XSUB(pi.x, pj.x), XSUB(pi.y, pj.y), XSUB(pi.z, pj.z)};
    const float rr = xnorm(d);
    if (!(rr < c.h)) return;
    const float4 vj = frec[(size_t)n + j];
    force_pair<false>(f, j == i, d, rr, vi, vj, pj.w, vj.w, ai.w, hh, lap_b, c);
    hook.pair(ha, i, j, d, V3{XSUB(vj.x, vi.x), XSUB(vj.y, vi.y), XSUB(vj.z, vi.z)});
  });
  const float4 a = finish_accel(f, ai.x, c);
  acc_out[i] = a;
  hook.end(ha, i, a);
}

// Forces from the particle's list with the general quotients and square root,
// where a coordinate or h lies outside the short ones' range: one coordinate of
// (0, 2^-76) in any scene of the handle. (Rescanning the window by a warp each,
// 1,048,576 particles took 3.12 ms; the list takes 0.213, with the short
// quotients 0.156.)
template <bool kLive, class Hook>
__device__ __forceinline__ void forces_particle_general(uint32_t i, uint32_t n, uint32_t cnt, const uint16_t* scene_of,
                                                        const State& st, const float4* aux, const Consts* consts,
                                                        const uint16_t* nlist, float4* acc_out, const Hook& hook,
                                                        const float4* frec, const uint32_t* nb_start) {
  typename Hook::Acc ha = hook.begin(i);
  const Consts& c = consts[scene_of[i]];
  const float4 pi = st.pos[i], vi = st.vel[i], ai = aux[i];
  const float hh = XMUL(c.h, c.h), lap_b = XMUL(3.f, hh);
  const uint32_t* nbs = nb_start + (size_t)__float_as_uint(ai.z) * 27u;
  ForceSums f = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, 0.f};
  auto slot_at = [&](uint32_t k) {
    const uint32_t tag = __ldcs(&nlist[(size_t)k * n + i]);
    return ld_step<kLive>(&nbs[tag >> kTagOffBits]) + (tag & ((1u << kTagOffBits) - 1u));
  };
  uint32_t next = cnt ? slot_at(0) : 0u;
  for (uint32_t k = 0; k < cnt; ++k) {  // (the next record's slot is looked up a pair ahead)
    const uint32_t j = next;
    const float4 pj = ld_step<kLive>(&frec[j]), vj = ld_step<kLive>(&frec[(size_t)n + j]);
    if (k + 1u < cnt) next = slot_at(k + 1u);
    const V3 d = {XSUB(pi.x, pj.x), XSUB(pi.y, pj.y), XSUB(pi.z, pj.z)};
    force_pair<false>(f, j == i, d, xnorm(d), vi, vj, pj.w, vj.w, ai.w, hh, lap_b, c);
    hook.pair(ha, i, j, d, V3{XSUB(vj.x, vi.x), XSUB(vj.y, vi.y), XSUB(vj.z, vi.z)});
  }
  const float4 a = finish_accel(f, ai.x, c);
  acc_out[i] = a;
  hook.end(ha, i, a);
}

// Internal forces (forces.cl:45-112) -> acceleration (sph.cl:53-58), walking
// the neighbour list of the density kernel (or the window, for particles
// without a complete list).
// Whole warps call it; `valid`: the lane has a particle.
//
// Bound: latency of the record gathers and FP32 issue. The quotients of a pair
// share one reciprocal and the square root has no slow path: 64 registers, 32
// warps an SM, instead of 72 and 28; 1,048,576 particles (25 neighbours on
// average) 0.186 -> 0.155 ms, with the learned step's features 0.361 -> 0.256
// (at most 102 registers: the features' 22 sums; unbounded, the compiler took
// 113 and 0.310 ms).
template <bool kLive = false, class Hook>
__device__ __forceinline__ void forces_particle(
    bool valid, uint32_t i, uint32_t n, const DevGrid* __restrict__ grids, const uint16_t* __restrict__ scene_of,
    const uint32_t* __restrict__ ctl, const uint32_t* __restrict__ keys_base, const State& st,
    const float4* __restrict__ aux, const CellIndex& ci, const Consts* __restrict__ consts,
    const uint16_t* __restrict__ nlist, const uint32_t* __restrict__ ncount, uint32_t nlist_cap,
    float4* __restrict__ acc_out, const Hook& hook, const float4* __restrict__ frec,
    const uint32_t* __restrict__ nb_start) {
  if (!valid) i = 0;
  // (every load of the prologue is issued before the first is used)
  auto tag_at = [&](uint32_t k) { return (uint32_t)__ldcs(&nlist[(size_t)k * n + i]); };
  const uint32_t t0 = tag_at(0), t1 = tag_at(1), t2 = tag_at(2);
  const uint32_t cnt = ncount[i];
  const float4 pi = st.pos[i];
  const float4 vi = st.vel[i];
  const float4 ai = aux[i];
  const Consts c = consts[scene_of[i]];
  const bool listed = valid && cnt <= nlist_cap;
  if (__any_sync(0xFFFFFFFFu, !c.plain_h || ctl[kCtlTiny])) {
    if (listed)
      forces_particle_general<kLive>(i, n, cnt, scene_of, st, aux, consts, nlist, acc_out, hook, frec, nb_start);
  } else if (listed) {
    typename Hook::Acc ha = hook.begin(i);
    const float own = ai.w;
    const float hh = XMUL(c.h, c.h);
    const float lap_b = XMUL(3.f, hh);
    ForceSums f = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, 0.f};
    // a tag names the neighbour's cell among the 27 around the own cell and
    // its offset there; the own cell's nb_start row holds their first slots
    const uint32_t* nbs = nb_start + (size_t)__float_as_uint(ai.z) * 27u;
    auto slot = [&](uint32_t tag) {
      return ld_step<kLive>(&nbs[tag >> kTagOffBits]) + (tag & ((1u << kTagOffBits) - 1u));
    };
    // software pipeline: while a pair is evaluated, the tag three pairs
    // ahead is loaded, the tag two ahead is resolved to its slot and the
    // records of the next pair (the density kernel's 32 bytes) are loaded
    if (cnt > 0) {
      uint32_t tnn = cnt > 2 ? t2 : cnt > 1 ? t1 : t0;
      uint32_t j = slot(t0);
      uint32_t jn = slot(cnt > 1 ? t1 : t0);
      float4 pj = ld_step<kLive>(&frec[j]), vj = ld_step<kLive>(&frec[(size_t)n + j]);
      for (uint32_t k = 0; k < cnt; ++k) {
        const uint32_t t3 = k + 3 < cnt ? tag_at(k + 3) : tnn;
        const uint32_t jnn = slot(tnn);
        const float4 pn = ld_step<kLive>(&frec[jn]), vn = ld_step<kLive>(&frec[(size_t)n + jn]);
        const V3 d = {XSUB(pi.x, pj.x), XSUB(pi.y, pj.y), XSUB(pi.z, pj.z)};
        force_pair<true>(f, j == i, d, near_norm(d), vi, vj, pj.w, vj.w, own, hh, lap_b, c);
        // the same differences the terms use (the compiler shares them); dead
        // code for the plain substep's empty hook
        const V3 dv = {XSUB(vj.x, vi.x), XSUB(vj.y, vi.y), XSUB(vj.z, vi.z)};
        hook.pair(ha, i, j, d, dv);
        j = jn;
        jn = jnn;
        pj = pn;
        vj = vn;
        tnn = t3;
      }
    }
    const float4 a = finish_accel(f, ai.x, c);
    acc_out[i] = a;
    hook.end(ha, i, a);
  }
  if constexpr (!Hook::kPairs) {
    for (uint32_t rest = __ballot_sync(0xFFFFFFFFu, valid && !listed); rest; rest &= rest - 1u)
      forces_particle_warp<kLive>(__shfl_sync(0xFFFFFFFFu, i, __ffs(rest) - 1), n, grids, scene_of, ctl, keys_base, st,
                                  aux, ci, consts, acc_out, frec);
  } else if (valid && !listed) {
    forces_particle_alone(i, n, grids, scene_of, ctl, keys_base, st, aux, ci, consts, acc_out, hook, frec);
  }
}

template <int BLOCK, class Hook = NoForceHook>
__global__ void __launch_bounds__(BLOCK, Hook::kPairs ? 640 / BLOCK : 1024 / BLOCK)
    k_forces(uint32_t n, const DevGrid* __restrict__ grids, const uint16_t* __restrict__ scene_of,
             const uint32_t* __restrict__ ctl,
             const uint32_t* __restrict__ keys_base, State st, const float4* __restrict__ aux,
             CellIndex ci, const Consts* __restrict__ consts, const uint16_t* __restrict__ nlist,
             const uint32_t* __restrict__ ncount, uint32_t nlist_cap,
             float4* __restrict__ acc_out, Hook hook, const float4* __restrict__ frec,
             const uint32_t* __restrict__ nb_start) {
  if (never_after_previous()) return;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if ((i & ~31u) >= n) return;  // whole warps
  forces_particle(i < n, i, n, grids, scene_of, ctl, keys_base, st, aux, ci, consts, nlist, ncount, nlist_cap,
                  acc_out, hook, frec, nb_start);
}

// The same with LANES lanes per particle, for scenes too small to hide a list's
// latencies behind other particles: the group evaluates LANES neighbours at
// once, lane l the neighbours l, l + LANES, ..., writes their terms to shared
// memory, and lane l adds terms l, l + LANES, ... of each in the list's order.
// One lane per particle walks its 25 to 40 neighbours one after another, about
// 18 us however few particles there are; eight lanes take 10 us for 4,096 and
// 14,000 particles.
constexpr uint32_t kWideTerms = 10, kWideThreads = 128;
template <uint32_t LANES>
static __global__ void __launch_bounds__(kWideThreads)
    k_forces_wide(uint32_t n, const DevGrid* __restrict__ grids, const uint16_t* __restrict__ scene_of,
                  const uint32_t* __restrict__ ctl, const uint32_t* __restrict__ keys_base, State st,
                  const float4* __restrict__ aux, CellIndex ci, const Consts* __restrict__ consts,
                  const uint16_t* __restrict__ nlist, const uint32_t* __restrict__ ncount, uint32_t nlist_cap,
                  float4* __restrict__ acc_out, const float4* __restrict__ frec,
                  const uint32_t* __restrict__ nb_start) {
  if (never_after_previous()) return;
  __shared__ float terms[kWideThreads][kWideTerms + 1];
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u, l = lane & (LANES - 1u);
  if (((t & ~31u) / LANES) >= n) return;  // whole warps
  const bool valid = t / LANES < n;
  const uint32_t i = valid ? t / LANES : 0u;
  const uint32_t cnt = ncount[i];
  const float4 pi = st.pos[i], vi = st.vel[i], ai = aux[i];
  const Consts c = consts[scene_of[i]];
  const bool listed = valid && cnt <= nlist_cap, plain = c.plain_h && !ctl[kCtlTiny];
  const float hh = XMUL(c.h, c.h), lap_b = XMUL(3.f, hh);
  const uint32_t* nbs = nb_start + (size_t)__float_as_uint(ai.z) * 27u;
  const uint32_t last = __reduce_max_sync(0xFFFFFFFFu, listed ? cnt : 0u);
  float* mine = terms[threadIdx.x];
  const float(*group)[kWideTerms + 1] = &terms[threadIdx.x & ~(LANES - 1u)];
  constexpr uint32_t kSums = (kWideTerms + LANES - 1u) / LANES;
  float sum[kSums] = {};
  float4 pj = make_float4(0.f, 0.f, 0.f, 0.f), vj = pj;
  uint32_t j = 0;
  auto load = [&](uint32_t k) {
    if (listed && k < cnt) {
      const uint32_t tag = __ldcs(&nlist[(size_t)k * n + i]);
      j = __ldg(&nbs[tag >> kTagOffBits]) + (tag & ((1u << kTagOffBits) - 1u));
      pj = __ldg(&frec[j]);
      vj = __ldg(&frec[(size_t)n + j]);
    }
  };
  load(l);
  for (uint32_t k = l; k < last + l; k += LANES) {
    ForceSums f = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, 0.f};
    if (listed && k < cnt) {
      const V3 d = {XSUB(pi.x, pj.x), XSUB(pi.y, pj.y), XSUB(pi.z, pj.z)};
      if (plain) force_pair<true>(f, j == i, d, near_norm(d), vi, vj, pj.w, vj.w, ai.w, hh, lap_b, c);
      else force_pair<false>(f, j == i, d, xnorm(d), vi, vj, pj.w, vj.w, ai.w, hh, lap_b, c);
    }
    load(k + LANES);
    // (0 + x is x, and adding the +0 of a term that doesn't count changes no sum, which is never -0)
    const float v[kWideTerms] = {f.P.x, f.P.y, f.P.z, f.Vs.x, f.Vs.y, f.Vs.z, f.Nm.x, f.Nm.y, f.Nm.z, f.lap};
#pragma unroll
    for (uint32_t a = 0; a < kWideTerms; ++a) mine[a] = v[a];
    __syncwarp();
#pragma unroll
    for (uint32_t q = 0; q < LANES; ++q) {
#pragma unroll
      for (uint32_t a = 0; a < kSums; ++a)
        sum[a] = XADD(sum[a], group[q][min(l + a * LANES, kWideTerms - 1u)]);
    }
    __syncwarp();
  }
  auto term = [&](uint32_t a) { return __shfl_sync(0xFFFFFFFFu, sum[a / LANES], a % LANES, LANES); };
  const ForceSums f = {{term(0), term(1), term(2)}, {term(3), term(4), term(5)}, {term(6), term(7), term(8)}, term(9)};
  if (listed && l == 0u) acc_out[i] = finish_accel(f, ai.x, c);
  for (uint32_t rest = __ballot_sync(0xFFFFFFFFu, valid && !listed && l == 0u); rest; rest &= rest - 1u)
    forces_particle_warp(__shfl_sync(0xFFFFFFFFu, i, __ffs(rest) - 1), n, grids, scene_of, ctl, keys_base, st, aux, ci,
                         consts, acc_out, frec);
}

// ------------------------------------------------------- mesh collision
struct Hit {
  V3 point, normal;
  float depth;
  bool any;
};

// One face of collisions.cl:21-87 (nearest hit; an equal distance replaces),
// from its packed rows (normal, |normal|), (v0, u.v), (u = v1 - v0, u.u),
// (v = v2 - v0, v.v), which hold the reference's own intermediate values.
// Most faces of a list lie out of the segment's reach: the first two rows
// decide, without the divisions (dot(n, d) / (|n| |d|) <= 0 has the sign of
// its numerator unless the quotient underflows; r = num / den outside [0, 1]
// shows by comparing the two). The lists of the 131,072-triangle heightfield
// hold about 26 faces near the surface; reading 15 words and dividing three
// times for each took most of the advection there: 4,194,304 particles landing
// on it, the first substep, 210 M -> 92 M warp instructions.
__device__ __forceinline__ void test_face(const float4* __restrict__ face, V3 p0, V3 p1, V3 d, float dlen, Hit& h) {
  const float4 fn = __ldg(&face[0]), f0 = __ldg(&face[1]);
  V3 nrm = v3(fn);
  const V3 v0 = v3(f0);
  float den = xdot(nrm, d), num = xdot(nrm, xsub3(v0, p0));
  const float nd = XMUL(fn.w, dlen);
  const bool clear = fabsf(den) >= nd * 0x1p-100f && nd <= 3.402823466e38f;
  if (clear ? den <= 0.f : XDIV(den, nd) <= 0.f) {  // the reference turns the normal: every product changes sign
    nrm = {-nrm.x, -nrm.y, -nrm.z};
    den = -den;
    num = -num;
  }
  if (den == 0.f) return;
  if (fabsf(num) > fabsf(den) * 1.000001f) return;                                           // r > 1 or r < -1
  if ((num < 0.f) != (den < 0.f) && fabsf(num) > fabsf(den) * 0x1p-100f) return;             // r < 0
  const float r = XDIV(num, den);
  if (!(0.f <= r && r <= 1.f)) return;
  const V3 at = {XADD(p0.x, XMUL(r, d.x)), XADD(p0.y, XMUL(r, d.y)), XADD(p0.z, XMUL(r, d.z))};
  const float4 fu = __ldg(&face[2]), fv = __ldg(&face[3]);
  const V3 w = xsub3(at, v0);
  const float uv = f0.w, uu = fu.w, vv = fv.w, wv = xdot(w, v3(fv)), wu = xdot(w, v3(fu));
  const float den2 = XSUB(XMUL(uv, uv), XMUL(uu, vv));
  const float s = XDIV(XSUB(XMUL(uv, wv), XMUL(vv, wu)), den2);
  const float t = XDIV(XSUB(XMUL(uv, wu), XMUL(uu, wv)), den2);
  if (s >= 0.f && t >= 0.f && XADD(s, t) <= 1.f) {
    if (h.any && xnorm(xsub3(p0, at)) > xnorm(xsub3(p0, h.point))) return;
    h.normal = nrm;
    h.point = at;
    h.depth = xnorm(xsub3(p1, at));
    h.any = true;
  }
}

// Faces that can meet the segment, in ascending face order: the list of
// the cell holding p0 when the segment is short enough for that list, no
// face when p0 lies outside the list grid (nothing within reach), else all.
__device__ __forceinline__ bool nearest_hit(const DevMesh& m, V3 p0, V3 p1, Hit& h) {
  h.any = false;
  if (m.faces == 0) return false;
  const V3 d = xsub3(p1, p0);
  const float dlen = xnorm(d);
  uint32_t first = 0, last = m.faces;
  const uint32_t* list = nullptr;
  if (m.cell_start != nullptr && dlen <= m.reach) {
    const float t[3] = {(p0.x - m.lo[0]) * m.inv_cell, (p0.y - m.lo[1]) * m.inv_cell,
                        (p0.z - m.lo[2]) * m.inv_cell};
    bool inside = true;
    int ci[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      inside = inside && (t[a] >= 0.f) && (t[a] < (float)m.dims[a]);
      ci[a] = inside ? (int)t[a] : 0;
      if (ci[a] >= m.dims[a]) ci[a] = m.dims[a] - 1;
    }
    if (!inside) return false;
    const uint32_t cell = ((uint32_t)ci[2] * (uint32_t)m.dims[1] + (uint32_t)ci[1]) * (uint32_t)m.dims[0] + (uint32_t)ci[0];
    first = __ldg(&m.cell_start[cell]);
    last = __ldg(&m.cell_start[cell + 1]);
    list = m.cell_faces;
  }
  for (uint32_t k = first; k < last; ++k) {
    const uint32_t f = list ? __ldg(&list[k]) : k;
    test_face(m.packed + (size_t)f * kFaceRows, p0, p1, d, dlen, h);
  }
  return h.any;
}

// Leapfrog + collision loop of sph.cl:64-112 (advection.cl:6-23,
// collisions.cl:91-129), capped at max_iters passes; writes the new state
// into `out` (same slots) and accumulates the next bounding box.
// kLearned (the learned stepper, no counterpart in the reference): the step
// spans dt_mult plain time steps, corr[i].xyz is added to the acceleration,
// corr[i].w (the predicted density) is stored in out.vel.w, and positions
// advance with (1 - pos_w) v + pos_w v' instead of v' (pos_w = (m + 1) / 2m
// for m = dt_mult reproduces m leapfrog substeps exactly under constant
// acceleration; m = 1 is the plain update).
// (4 resident blocks of 256 threads, 64 registers: 1,048,576 particles on a
// floor 0.038 ms; 3 blocks 0.043, 5 blocks 0.042. Blocks take consecutive
// particles and reduce their bounding box once, instead of at every 256: with
// a barrier per 256 particles the lanes without collisions waited for those
// with. Both changes: on a floor 0.049 -> 0.038 ms, 256 batched scenes 0.206 ->
// 0.126, 4,194,304 particles on the heightfield 0.681 -> 0.295. Bound: load
// latency.)
// With y_stats (the network's output means and standard deviations, 4 + 4),
// corr holds the MLP's de-standardised outputs and learned_correction turns
// them into the correction here.

// Each output clamped to its training mean +- kLearnedOutputClamp standard
// deviations (which bounds the correction one step can apply); outputs 0..2
// are accelerations in units of h / dt^2, output 3 the relative density
// change: (correction xyz, predicted density).
constexpr float kLearnedOutputClamp = 4.f;
__device__ __forceinline__ float4 learned_correction(float4 y, const float* y_stats, const Consts& c,
                                                     float rho) {
  auto clamp_out = [&](float v, int k) {
    const float mu = y_stats[k], sigma = y_stats[4 + k];
    return fminf(fmaxf(v, mu - kLearnedOutputClamp * sigma), mu + kLearnedOutputClamp * sigma);
  };
  const float dt = c.time_delta * c.scale;
  const float s = c.h / (dt * dt);
  return make_float4(clamp_out(y.x, 0) * s, clamp_out(y.y, 1) * s, clamp_out(y.z, 2) * s,
                     rho * (1.f + clamp_out(y.w, 3)));
}

template <bool kLearned>
__device__ __forceinline__ void advect_blocks(
    uint32_t blk, uint32_t nblk, uint32_t n, State in, const float4* __restrict__ acc, State out,
    const DevMesh* __restrict__ meshes, const Consts* __restrict__ consts,
    const uint16_t* __restrict__ scene_of, uint32_t max_iters, uint32_t* __restrict__ bbox,
    uint32_t* __restrict__ status, unsigned long long* __restrict__ capped_count,
    const float4* __restrict__ corr, float dt_mult, float pos_w, const float4* __restrict__ aux,
    const float* __restrict__ y_stats, BboxSmem& bsm) {
  const float qnan = __int_as_float(0x7FC00000);
  // a block takes consecutive particles and keeps their bounding box in
  // registers until the scene changes or its particles end
  const uint32_t chunks = (n + blockDim.x - 1) / blockDim.x, per = (chunks + nblk - 1) / nblk;
  const uint32_t first = min(blk * per, chunks) * blockDim.x, end = min((uint64_t)n, (uint64_t)first + per * blockDim.x);
  float3 lo = make_float3(qnan, qnan, qnan), hi = lo;
  int scene = -1;
  for (uint32_t i = first + threadIdx.x; i < end; i += blockDim.x) {
    const int sc = scene_of[i];
    if (sc != scene) {
      if (scene >= 0) {
        const float v[6] = {lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
        bbox_atomics(v, bbox + 6 * (size_t)scene);
      }
      lo = hi = make_float3(qnan, qnan, qnan);
      scene = sc;
    }
    const Consts& c = consts[scene];
    const DevMesh& m = meshes[scene];
    float remaining = XMUL(c.time_delta, c.scale);
    V3 pos = v3(in.pos[i]);
    const V3 vh_old = v3(in.ivel[i]);
    V3 v = vh_old;
    V3 a = v3(acc[i]);
    float predicted_rho = 0.f;
    if constexpr (kLearned) {
      remaining = XMUL(remaining, dt_mult);
      float4 d = corr[i];
      if (y_stats) d = learned_correction(d, y_stats, c, aux[i].x);
      a = {XADD(a.x, d.x), XADD(a.y, d.y), XADD(a.z, d.z)};
      predicted_rho = d.w;
    }
    bool capped = false;
    for (uint32_t it = 0;; ++it) {
      V3 nv = {XADD(v.x, XMUL(a.x, remaining)), XADD(v.y, XMUL(a.y, remaining)),
               XADD(v.z, XMUL(a.z, remaining))};
      const float sp = xnorm(nv);
      if (sp > c.vmax)
        nv = {XMUL(XDIV(nv.x, sp), c.vmax), XMUL(XDIV(nv.y, sp), c.vmax), XMUL(XDIV(nv.z, sp), c.vmax)};
      V3 vp = nv;
      if constexpr (kLearned) {
        const float w0 = XSUB(1.f, pos_w);
        vp = {XADD(XMUL(v.x, w0), XMUL(nv.x, pos_w)), XADD(XMUL(v.y, w0), XMUL(nv.y, pos_w)),
              XADD(XMUL(v.z, w0), XMUL(nv.z, pos_w))};
      }
      const V3 np = {XADD(pos.x, XMUL(vp.x, remaining)), XADD(pos.y, XMUL(vp.y, remaining)),
                     XADD(pos.z, XMUL(vp.z, remaining))};
      Hit h;
      const bool hit = nearest_hit(m, pos, np, h);
      float elapsed = remaining;
      V3 opos = np, ov = nv;
      if (hit) {
        opos = {XSUB(h.point.x, XMUL(h.normal.x, 0.001f)), XSUB(h.point.y, XMUL(h.normal.y, 0.001f)),
                XSUB(h.point.z, XMUL(h.normal.z, 0.001f))};
        const float k = XMUL(XADD(1.f, XDIV(XMUL(c.restitution, h.depth), XMUL(remaining, xnorm(nv)))),
                             xdot(nv, h.normal));
        ov = {XSUB(nv.x, XMUL(k, h.normal.x)), XSUB(nv.y, XMUL(k, h.normal.y)),
              XSUB(nv.z, XMUL(k, h.normal.z))};
        elapsed = XMUL(remaining, XDIV(xnorm(xsub3(opos, pos)), xnorm(xsub3(np, pos))));
      }
      pos = opos;
      v = ov;
      remaining = XSUB(remaining, elapsed);
      a = {0.f, 0.f, 0.f};
      if (!hit) break;
      if (it + 1 >= max_iters) {
        capped = true;
        break;
      }
    }
    if (capped) {
      atomicOr(status, kFlagCollisionCap);
      atomicAdd(capped_count, 1ull);
    }
    out.pos[i] = make_float4(pos.x, pos.y, pos.z, 0.f);
    out.ivel[i] = make_float4(v.x, v.y, v.z, 0.f);
    out.vel[i] = make_float4(XDIV(XADD(vh_old.x, v.x), 2.f), XDIV(XADD(vh_old.y, v.y), 2.f),
                             XDIV(XADD(vh_old.z, v.z), 2.f), predicted_rho);
    if (!(isfinite(pos.x) && isfinite(pos.y) && isfinite(pos.z))) atomicOr(status, kFlagNonFinite);
    lo = make_float3(fminf(lo.x, pos.x), fminf(lo.y, pos.y), fminf(lo.z, pos.z));
    hi = make_float3(fmaxf(hi.x, pos.x), fmaxf(hi.y, pos.y), fmaxf(hi.z, pos.z));
  }
  bbox_accumulate(lo, hi, scene, bbox, bsm);
  __syncthreads();  // the shared reduction is read before the block's next use
}

template <bool kLearned>
__global__ void __launch_bounds__(kBlock, 4)
    k_advect(uint32_t n, State in, const float4* __restrict__ acc, State out,
             const DevMesh* __restrict__ meshes, const Consts* __restrict__ consts,
             const uint16_t* __restrict__ scene_of, uint32_t max_iters, uint32_t* __restrict__ bbox,
             uint32_t* __restrict__ status, unsigned long long* __restrict__ capped_count,
             const float4* __restrict__ corr, float dt_mult, float pos_w, const float4* __restrict__ aux,
             const float* __restrict__ y_stats) {
  if (never_after_previous()) return;
  __shared__ BboxSmem bsm;
  advect_blocks<kLearned>(blockIdx.x, gridDim.x, n, in, acc, out, meshes, consts, scene_of, max_iters, bbox,
                          status, capped_count, corr, dt_mult, pos_w, aux, y_stats, bsm);
}

// Dense reference cell table of one scene from the sorted keys of its slot
// range [first, last): table[c] = lower_bound(c) - first, c < cells.
static __global__ void k_dense_table(const uint32_t* __restrict__ keys_base, uint32_t n,
                              const uint32_t* __restrict__ ctl, const DevGrid* __restrict__ grid,
                              uint32_t scene, uint32_t first, uint32_t last,
                              uint32_t* __restrict__ table) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t cells = grid->cells;
  if (c >= cells) return;
  const KeySplit split{ctl[kCtlShift]};
  const uint32_t* keys = keys_base + (size_t)sorted_sel(ctl[kCtlMaxKey]) * n;
  const uint32_t want = c | split.scene_bits(scene);
  uint32_t lo = first, hi = last;
  while (lo < hi) {
    uint32_t mid = lo + (hi - lo) / 2;
    if (keys[mid] < want) lo = mid + 1; else hi = mid;
  }
  table[c] = lo - first;
}

}  // namespace clsph
