// Host dispatch of the batch kernel (batch_kernel.cuh), the small kernels of a run's launch chain and the batch run without
// device allocation.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <mutex>

#include "batch_kernel.cuh"

namespace ssb {

namespace {

// Calls f with the kernel's instantiation for teams of W warps; f returns a cudaError_t.
template <bool MIXED, bool FLEET, class F>
cudaError_t with_kernel(int W, F f) {
  switch (W) {
    case 1: return f(BatchKernel<MIXED, 1, FLEET>{});
    case 2: return f(BatchKernel<MIXED, 2, FLEET>{});
    case 4: return f(BatchKernel<MIXED, 4, FLEET>{});
    case 8: return f(BatchKernel<MIXED, 8, FLEET>{});
    case 16: return f(BatchKernel<MIXED, 16, FLEET>{});
  }
  return cudaErrorInvalidValue;
}

template <class F>
cudaError_t with_kernel(bool mixed, bool fleet, int W, F f) {
  if (fleet) return mixed ? with_kernel<true, true>(W, f) : with_kernel<false, true>(W, f);
  return mixed ? with_kernel<true, false>(W, f) : with_kernel<false, false>(W, f);
}

}  // namespace

bool valid_team_size(int W) { return W == 1 || W == 2 || W == 4 || W == 8 || W == 16; }

std::size_t column_stage_bytes(bool mixed, int ncol) {
  // the table, then its 8-byte mbarrier (kept at a 16-byte boundary)
  return (mixed ? staged_columns<float>(ncol).bytes : staged_columns<double>(ncol).bytes) + 16;
}

cudaError_t configure_batch_kernel(bool mixed, int teamWarps, std::size_t smemBytes, bool fleet) {
  return with_kernel(mixed, fleet, teamWarps, [&](auto k) { return decltype(k)::set_smem(smemBytes); });
}

cudaError_t launch_batch_kernel(bool mixed, int teamWarps, const DevModel& M, const DevBatch& B, const SlotLayout& L, int grid,
                                int teamsPerBlock, cudaStream_t stream) {
  if (!valid_team_size(teamWarps) || teamsPerBlock * teamWarps > kMaxWarpsPerBlock) return cudaErrorInvalidValue;
  const bool fleet = B.models != nullptr;
  const std::size_t smem = static_cast<std::size_t>(teamsPerBlock) * L.bytes + (B.stageColumns && !fleet ? column_stage_bytes(mixed, M.ncol) : 0);
  const int threads = teamsPerBlock * teamWarps * 32;
  const cudaError_t e = with_kernel(mixed, fleet, teamWarps, [&](auto k) {
    decltype(k)::launch(M, B, L, grid, threads, smem, stream);
    return cudaSuccess;
  });
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

namespace {
__global__ void start_run(std::int32_t* remaining, std::int32_t count, unsigned long long* phaseSteps, int phases) {
  if (threadIdx.x == 0) *remaining = count;
  for (int k = static_cast<int>(threadIdx.x); k < phases; k += blockDim.x) phaseSteps[k] = 0;
}
}  // namespace

cudaError_t launch_start_run(std::int32_t* remaining, std::int32_t count, unsigned long long* phaseSteps, int phases, cudaStream_t stream) {
  start_run<<<1, 32, 0, stream>>>(remaining, count, phaseSteps, phases);
  return cudaGetLastError();
}

// Claim order of a launch phase after the first. The phase before paused its instances; the one with the most work
// left should get a larger team first, or it waits behind others for a free one and ends last. The work left is not
// known, but a run's length is bounded (tMax, and in practice the founder/settle times), so the fewer steps an
// instance has done, the more it has left: the order is by steps done, ascending, ties by index.
namespace {
constexpr int kOrderThreads = 256;

__global__ void compact_unfinished(const std::int32_t* stop, std::int32_t count, std::int32_t* list, std::int32_t* n) {
  for (std::int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    if (stop[i] == kRunning) list[atomicAdd(n, 1)] = i;
}

// order[rank of (steps[i], i) among the listed instances] = i: ranks of distinct keys, so a permutation of 0 .. n-1
// whatever order the compaction listed them in.
__global__ void __launch_bounds__(kOrderThreads) rank_unfinished(const long long* steps, const std::int32_t* list, const std::int32_t* n,
                                                                 std::int32_t* order) {
  __shared__ long long keyS[kOrderThreads];
  __shared__ std::int32_t keyI[kOrderThreads];
  const std::int32_t R = *n;
  for (std::int32_t base = blockIdx.x * kOrderThreads; base < R; base += gridDim.x * kOrderThreads) {
    const std::int32_t k = base + static_cast<std::int32_t>(threadIdx.x);
    const bool mine = k < R;
    const std::int32_t me = mine ? list[k] : 0;
    const long long ms = mine ? steps[me] : 0;
    std::int32_t rank = 0;
    for (std::int32_t t0 = 0; t0 < R; t0 += kOrderThreads) {
      __syncthreads();
      const std::int32_t m = t0 + static_cast<std::int32_t>(threadIdx.x);
      if (m < R) {
        const std::int32_t j = list[m];
        keyI[threadIdx.x] = j;
        keyS[threadIdx.x] = steps[j];
      }
      __syncthreads();
      const std::int32_t lim = min(kOrderThreads, R - t0);
      if (mine)
        for (std::int32_t j = 0; j < lim; ++j) rank += (keyS[j] < ms || (keyS[j] == ms && keyI[j] < me)) ? 1 : 0;
    }
    if (mine) order[rank] = me;
  }
}
}  // namespace

cudaError_t launch_order_unfinished(const std::int32_t* stop, const long long* steps, std::int32_t count, std::int32_t bound,
                                    std::int32_t* list, std::int32_t* order, std::int32_t* n, cudaStream_t stream) {
  if (count < 1 || bound < 1) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(n, 0, sizeof(std::int32_t), stream);
  if (e != cudaSuccess) return e;
  const int compactBlocks = static_cast<int>(std::min<std::int64_t>((static_cast<std::int64_t>(count) + 255) / 256, 1024));
  compact_unfinished<<<compactBlocks, 256, 0, stream>>>(stop, count, list, n);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  const int rankBlocks = static_cast<int>(std::min<std::int64_t>((static_cast<std::int64_t>(std::min(bound, count)) + kOrderThreads - 1) / kOrderThreads, 1024));
  rank_unfinished<<<rankBlocks, kOrderThreads, 0, stream>>>(steps, list, n, order);
  return cudaGetLastError();
}

cudaError_t batch_kernel_occupancy(bool mixed, int teamWarps, int teamsPerBlock, std::size_t smemBytes, int* blocksPerSM, bool fleet) {
  const int threads = teamsPerBlock * teamWarps * 32;
  return with_kernel(mixed, fleet, teamWarps, [&](auto k) { return decltype(k)::occupancy(threads, smemBytes, blocksPerSM); });
}

// ----------------------------------------------------------------------------- the batch run without device allocation
// Some callers cannot call cudaMalloc when they run a batch: a host application that owns every device allocation
// through its own pool (a calibration or control loop embedded in a larger program), or code that must not allocate
// once it is running. For them the batch kernel's scratch, the memory it needs beyond the caller's inputs and outputs
// (the work-queue head, the count of unfinished instances, and each instance's outputs, event log, overflow and mark
// times), lives in this fixed array instead of in buffers the engine allocates. Every GPU that loads the library
// holds it until the process exits. All calls share it and it keeps the last call's contents, so each call clears
// what must start at zero; two calls that overlap on the GPU (on different streams) would race on it.

namespace {

constexpr std::size_t kNoAllocScratchBytes = std::size_t(4) << 20;
__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
void* g_scratch_address[kMaxDevices] = {};

// The device address of g_noalloc_scratch on the current device. The array's name in host code is a host-side stand-in,
// not a device address, so the first call on a device looks the address up (cudaGetSymbolAddress, with that device
// current). Later calls look it up again and replace the cached value if it moved: the query is cheap and allocates
// nothing, and a cudaDeviceReset between calls reloads the module at a possibly different address. The mutex keeps host
// threads that call at the same time from racing on the cache.
cudaError_t scratch_address(int device, void** out) {
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  void* p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess) return e;
  g_scratch_address[device] = p;
  *out = p;
  return cudaSuccess;
}

// The per-instance fields the batch kernel expects to find set before its first launch.
__global__ void clear_noalloc_scratch(DevBatch B, int nmon, int nmark) {
  const std::int32_t stride = gridDim.x * blockDim.x;
  for (std::int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < B.count; i += stride) {
    for (int k = 0; k < 7; ++k) B.out[static_cast<std::size_t>(i) * 7 + k] = 0;
    B.evCount[i] = 0;
    B.foundered[i] = 0;
    B.founderT[i] = -1;
    B.steps[i] = 0;
    B.stop[i] = kRunning;
    for (int m = 0; m < nmon; ++m) B.overT[static_cast<std::size_t>(i) * nmon + m] = -1;
    for (int m = 0; m < nmark; ++m) B.markT[static_cast<std::size_t>(i) * nmark + m] = -1;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *B.queue = 0;
    *B.remaining = B.count;
    *B.error = 0;
  }
}

std::size_t align256(std::size_t x) { return (x + 255) & ~static_cast<std::size_t>(255); }

}  // namespace

std::size_t noalloc_scratch_capacity() { return kNoAllocScratchBytes; }

std::size_t noalloc_scratch_bytes(const DevModel& M, int count) {
  const auto c = static_cast<std::size_t>(count);
  std::size_t b = align256(3 * sizeof(std::int32_t));                         // queue, remaining, error
  b += align256(c * 7 * sizeof(double));                                        // outputs
  b += 2 * align256(c * sizeof(std::int32_t)) + align256(c * sizeof(double));   // evCount, foundered, founderT
  b += align256(c * M.evCap * sizeof(double)) + 2 * align256(c * M.evCap * sizeof(std::int32_t));  // event log
  b += align256(c * std::max(M.nmon, 1) * sizeof(double)) + align256(c * std::max(M.nmark, 1) * sizeof(double));
  return b;
}

cudaError_t run_batch_noalloc(bool mixed, const DevModel& M, const SlotLayout& L, const NoAllocRun& r, cudaStream_t stream) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  if (noalloc_scratch_bytes(M, r.count) > kNoAllocScratchBytes) return cudaErrorMemoryAllocation;
  void* address = nullptr;
  e = scratch_address(device, &address);
  if (e != cudaSuccess) return e;
  auto* base = static_cast<unsigned char*>(address);
  std::size_t off = 0;
  auto carve = [&](std::size_t bytes) { unsigned char* p = base + off; off += align256(bytes); return p; };
  const auto c = static_cast<std::size_t>(r.count);
  DevBatch B{};
  B.count = r.count;
  B.queue = reinterpret_cast<std::int32_t*>(carve(3 * sizeof(std::int32_t)));
  B.remaining = B.queue + 1;
  B.error = B.queue + 2;
  B.out = reinterpret_cast<double*>(carve(c * 7 * sizeof(double)));
  B.evCount = reinterpret_cast<std::int32_t*>(carve(c * sizeof(std::int32_t)));
  B.foundered = reinterpret_cast<std::int32_t*>(carve(c * sizeof(std::int32_t)));
  B.founderT = reinterpret_cast<double*>(carve(c * sizeof(double)));
  B.evT = reinterpret_cast<double*>(carve(c * M.evCap * sizeof(double)));
  B.evId = reinterpret_cast<std::int32_t*>(carve(c * M.evCap * sizeof(std::int32_t)));
  B.evKind = reinterpret_cast<std::int32_t*>(carve(c * M.evCap * sizeof(std::int32_t)));
  B.overT = reinterpret_cast<double*>(carve(c * std::max(M.nmon, 1) * sizeof(double)));
  B.markT = reinterpret_cast<double*>(carve(c * std::max(M.nmark, 1) * sizeof(double)));
  // the caller's inputs and outputs
  B.en = r.en; B.area = r.area; B.tOn = r.tOn;
  B.st = r.state; B.vol = r.vol; B.level = r.level; B.cx = r.cx; B.cy = r.cy; B.cz = r.cz;
  B.finalRec = r.finalRec; B.steps = r.steps; B.stop = r.stop;
  B.curveEvery = 0; B.traced = 0;
  B.tMax = r.tMax;
  B.maxSteps = LLONG_MAX;
  B.firstLaunch = 1;
  B.rule = r.rule;
  B.stopWhenStable = r.stopWhenStable ? 1 : 0;
  B.yieldBelow = 0;
  clear_noalloc_scratch<<<64, 256, 0, stream>>>(B, M.nmon, M.nmark);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return launch_batch_kernel(mixed, r.teamWarps, M, B, L, r.blocks, r.teamsPerBlock, stream);
}

}  // namespace ssb
