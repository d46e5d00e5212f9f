// Allocation-free stable key sort: clsph_gpu_sort_keys_noalloc.
//
// Some callers cannot allocate device memory themselves: a host application
// or framework that owns every device allocation through its own allocator
// and forbids raw cudaMalloc/cudaFree (whose implicit device-wide
// synchronisation would stall its other work), or a fixed-budget real-time
// loop that must not allocate after start-up. This entry point runs the
// substep's stable sort (the 4 x 8-bit LSD radix sort of
// libclsph/sph_simulation.cpp:107-156 + kernels/sort.cl, with 32-bit offsets)
// on caller-provided device buffers and takes its scratch space from one
// file-scope __device__ array instead of cudaMalloc.
//
// Limits and rules:
//  * at most kNoAllocMaxKeys (1,048,576) keys per call; larger n is rejected
//    with CLSPH_ERR_TOO_LARGE before any GPU work;
//  * the scratch array (9.4 MB) is part of the library's device image: every
//    GPU that loads the library holds it until the process exits;
//  * all calls share that one array and it keeps the last call's contents;
//    each call clears what must start at zero itself. Calls whose GPU work
//    overlaps (other streams, other host threads on the same device) race on
//    it, so the caller must serialise them;
//  * the first call on each device looks up the array's device address with
//    cudaGetSymbolAddress (with that device current); make that first call
//    before any stream capture.
// It makes no cudaMalloc, cudaFree or other allocating call.
//
// Bound: the sort's own latencies (clsph_radix.cuh). Four launches, all but the
// first with their blocks placed while the one before still runs: 1,048,576
// keys of 22 bits 39 us, against 91 with a launch per pass and step. With the
// first launch placed early too 37; without the last one, which is there for a
// wait that ran out, 35; without it, all launched in the plain way behind a
// memset node, 46.

#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>

#include "clsph_gpu.h"
#include "clsph_radix.cuh"

void clsph_set_last_error(const std::string& msg);

namespace {

using namespace clsph;

constexpr uint32_t kNoAllocMaxKeys = 1u << 20;
constexpr uint32_t kMaxTiles = kNoAllocMaxKeys / kRadixTile;
constexpr int kThreads = 256;

// scratch layout, in 32-bit words; the control words are cleared by every call
constexpr size_t kOffKeys = 0;                                      // ping-pong keys
constexpr size_t kOffVals = kOffKeys + kNoAllocMaxKeys;             // ping-pong slots
constexpr size_t kOffLookback = kOffVals + kNoAllocMaxKeys;         // [4 passes][tiles][256]
constexpr size_t kOffTotals = kOffLookback + kRadixMaxPasses * 256 * (size_t)kMaxTiles;  // [4][256]
constexpr size_t kOffCtl = kOffTotals + kRadixMaxPasses * 256;
enum : int { kMaxKey = 0, kStatus = 1, kCounters = 4 };             // control words
constexpr size_t kScratchWords = kOffCtl + 64;

static __device__ __align__(256) uint32_t g_sort_scratch[kScratchWords];

// Clears the digit totals and the control words, which lie side by side.
__global__ void __launch_bounds__(kThreads) k_na_clear(uint32_t* __restrict__ scratch) {
  if (never_after_previous()) return;
  for (size_t q = kOffTotals + threadIdx.x; q < kScratchWords; q += kThreads) scratch[q] = 0u;
}

// Largest key and the digit counts of every pass; clears the look-back words.
__global__ void __launch_bounds__(kThreads) k_na_count(const uint32_t* __restrict__ keys, uint32_t n, uint32_t ntiles,
                                                       uint32_t* __restrict__ scratch) {
  if (never_after_previous()) return;
  __shared__ uint32_t hist[kRadixMaxPasses][256];
  __shared__ uint32_t block_max;
  const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  uint4* lookback = reinterpret_cast<uint4*>(scratch + kOffLookback);
  for (uint32_t q = first; q < kRadixMaxPasses * 64u * ntiles; q += stride) lookback[q] = make_uint4(0u, 0u, 0u, 0u);
  for (uint32_t q = threadIdx.x; q < kRadixMaxPasses * 256u; q += blockDim.x) hist[q >> 8][q & 255u] = 0u;
  if (threadIdx.x == 0) block_max = 0u;
  __syncthreads();
  uint32_t top = 0u;
  for (uint32_t i = first; (i & ~31u) < n; i += stride) {
    const uint32_t key = i < n ? __ldg(&keys[i]) : 0u;
    top = max(top, key);
    radix_count(key, i < n, kRadixMaxPasses, hist);
  }
  top = __reduce_max_sync(0xFFFFFFFFu, top);
  if ((threadIdx.x & 31) == 0) atomicMax(&block_max, top);
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(&scratch[kOffCtl + kMaxKey], block_max);
  radix_count_flush(hist, kRadixMaxPasses, scratch + kOffTotals);
}

// The last pass always lands in the caller's output.
__device__ __forceinline__ RadixBuffers caller_buffers(const uint32_t* keys, uint32_t* keys_out, uint32_t* vals_out,
                                                       uint32_t passes, uint32_t* scratch) {
  return RadixBuffers{keys, scratch + kOffKeys, keys_out, scratch + kOffVals, vals_out, (passes + 1u) & 1u};
}

__global__ void __launch_bounds__(kRadixThreads)
    k_na_sort(const uint32_t* __restrict__ keys, uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
              uint32_t n, uint32_t ntiles, uint32_t* __restrict__ scratch, uint32_t spin_limit,
              uint32_t withheld_tile) {
  if (never_after_previous()) return;
  __shared__ RadixSmem<kRadixThreads> sm;
  uint32_t* ctl = scratch + kOffCtl;
  const uint32_t passes = radix_passes(ctl[kMaxKey]);
  const RadixBuffers buf = caller_buffers(keys, keys_out, vals_out, passes, scratch);
  radix_sort_blocks<kRadixThreads>(buf, n, passes, scratch + kOffTotals, scratch + kOffLookback, ntiles,
                                   ctl + kCounters, ctl + kStatus, spin_limit, withheld_tile, sm);
}

// The call has returned by now, so a wait that ran out cannot be reported: one
// block sorts everything again without waits (the input is untouched, and the
// digit counts do not depend on the order). 6.7 ms for 1,048,576 keys of 22
// bits; without a stall the launch adds 1.4 us. (In the sort kernel itself,
// by its last block to finish, the count of blocks alone took 2 us.)
__global__ void __launch_bounds__(kRadixThreads)
    k_na_again(const uint32_t* __restrict__ keys, uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
               uint32_t n, uint32_t ntiles, uint32_t* __restrict__ scratch) {
  if (never_after_previous()) return;
  uint32_t* ctl = scratch + kOffCtl;
  if (ctl[kStatus] == 0u) return;
  __shared__ RadixSmem<kRadixThreads> sm;
  const uint32_t passes = radix_passes(ctl[kMaxKey]);
  const RadixBuffers buf = caller_buffers(keys, keys_out, vals_out, passes, scratch);
  radix_sort_blocks<kRadixThreads, true>(buf, n, passes, scratch + kOffTotals, scratch + kOffLookback, ntiles,
                                         ctl + kCounters, ctl + kStatus, 0u, kNoTile, sm);
}

// Device address of g_sort_scratch, looked up once per device and kept for
// the life of the process (a cudaDeviceReset reloads the device code and
// makes it stale; the header tells callers not to use the entry point on a
// device after resetting it).
constexpr int kMaxDevices = 64;
std::mutex g_setup_mutex;
uint32_t* g_scratch_addr[kMaxDevices] = {};

int scratch_for_current_device(uint32_t** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    clsph_set_last_error(std::string("sort_keys_noalloc: cudaGetDevice: ") + cudaGetErrorString(e));
    return CLSPH_ERR_CUDA;
  }
  if (dev < 0 || dev >= kMaxDevices) {
    clsph_set_last_error("sort_keys_noalloc: device ordinal out of range");
    return CLSPH_ERR_ARGUMENT;
  }
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (!g_scratch_addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_sort_scratch);
    if (e != cudaSuccess || p == nullptr) {
      clsph_set_last_error(std::string("sort_keys_noalloc: cudaGetSymbolAddress: ") +
                           cudaGetErrorString(e));
      return CLSPH_ERR_CUDA;
    }
    g_scratch_addr[dev] = static_cast<uint32_t*>(p);
  }
  *out = g_scratch_addr[dev];
  return CLSPH_OK;
}

}  // namespace

extern "C" int clsph_gpu_sort_keys_noalloc_limited(const uint32_t* keys_in, uint32_t* keys_out, uint32_t* perm_out,
                                                   uint32_t n, void* stream, uint32_t spin_limit,
                                                   uint32_t withheld_tile) {
  if (n > kNoAllocMaxKeys) {
    clsph_set_last_error("sort_keys_noalloc: n = " + std::to_string(n) +
                         " exceeds the maximum of 1048576 keys");
    return CLSPH_ERR_TOO_LARGE;
  }
  if (n == 0) return CLSPH_OK;
  if (!keys_in || !keys_out || !perm_out) {
    clsph_set_last_error("sort_keys_noalloc: null buffer");
    return CLSPH_ERR_ARGUMENT;
  }
  uint32_t* scratch = nullptr;
  int rc = scratch_for_current_device(&scratch);
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const uint32_t ntiles = (n + kRadixTile - 1) / kRadixTile;
  const uint32_t blocks = (n + kThreads - 1) / kThreads;
  // the first launch is a plain one: it waits for all earlier work of the caller's stream, also where the kernel just
  // before was itself placed early and ends without having waited for its own predecessors
  launch_early(k_na_clear, dim3(1), dim3(kThreads), 0, s, false, scratch);
  launch_early(k_na_count, dim3(blocks < 608u ? blocks : 608u), dim3(kThreads), 0, s, true, keys_in, n, ntiles,
               scratch);
  launch_early(k_na_sort, dim3(ntiles), dim3(kRadixThreads), 0, s, true, keys_in, keys_out, perm_out, n, ntiles,
               scratch, spin_limit, withheld_tile);
  launch_early(k_na_again, dim3(1), dim3(kRadixThreads), 0, s, true, keys_in, keys_out, perm_out, n, ntiles, scratch);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    clsph_set_last_error(std::string("sort_keys_noalloc: launch: ") + cudaGetErrorString(e));
    return CLSPH_ERR_CUDA;
  }
  return CLSPH_OK;
}

extern "C" int clsph_gpu_sort_keys_noalloc(const uint32_t* keys_in, uint32_t* keys_out,
                                           uint32_t* perm_out, uint32_t n, void* stream) {
  return clsph_gpu_sort_keys_noalloc_limited(keys_in, keys_out, perm_out, n, stream, kRadixLookbackSpins, kNoTile);
}
