// Shared definitions for the B200 coupled-channel kernels.
//
// Layout conventions used by every kernel in this library:
//  * matrices are row-major doubles; a "batch" of matrices is a base pointer plus a
//    batch stride in elements;
//  * matrices that go through the blocked symmetric sweep are padded to a multiple
//    of kBlock (128) rows and columns; padding carries the identity on the diagonal
//    and zeros elsewhere, so sweeping it leaves -1 on the padded diagonal and never
//    couples it to the logical channels;
//  * complex symmetric matrices A = X + iZ are swept through the real symmetric
//    embedding with 2x2 blocks [[X, Z], [Z, -X]] interleaved per channel, which is
//    invertible exactly when A is and keeps every 2x2 diagonal block nonsingular.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <cstdint>

namespace ticc {

constexpr int kBlock = 128;          // sweep pivot block = GEMM output tile edge
constexpr int kChunk = 32;           // K rows staged per shared-memory stage
constexpr int kPad = 4;              // shared-memory row padding (doubles)
constexpr int kStride = kBlock + kPad;  // 132: conflict-free DMMA fragment loads
constexpr int kGemmThreads = 256;    // 8 warps: 2 (rows of 64) x 4 (cols of 32)
constexpr int kPivotThreads = 256;

// Device status codes written into the caller's status word (first error wins).
enum DeviceStatus : int {
  kDeviceOk = 0,
  kDeviceSingularPivot = 1,   // a pivot block of the sweep was singular or non-finite
  kDeviceNonFinite = 2,       // a non-finite value reached an output
  kDeviceBesselFailed = 3,    // a Bessel continued fraction did not converge
  kDeviceThreshold = 4,       // a total energy sits exactly on a channel threshold
  kDeviceStalled = 6,         // a fused sweep step gave up waiting for a row-panel tile (bounded wait)
};

// Host-side count of kernels this library has enqueued (process lifetime).
inline std::atomic<long long>& launch_counter() {
  static std::atomic<long long> count{0};
  return count;
}
inline void note_launch(long long n = 1) { launch_counter().fetch_add(n, std::memory_order_relaxed); }

// Launch `kernel` so that its CTAs may come up while the kernel before it in the stream drains: the CTAs of a kernel launched so
// call previous_kernel_done() before they touch anything that the call's earlier kernels write.  A kernel that starts
// behind such a one and waits is ordered behind everything before it too, because the other finished only after its own wait.
// Between the passes and sweeps of a propagation this hides the launch and the first loads (only the passes call
// next_kernel_may_start(), so nothing runs beside a sweep's thinning tail):
// measured, N = 231, 16 energies, 8 sectors 1865 -> 1808 us, a rigid-rotor solve of 24 sectors 7.96 -> 7.69 ms, mixed windows of N = 1860 24.7 -> 24.5 ms.
template <typename... Params, typename... Args>
inline cudaError_t launch_overlapped(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchAttribute attribute{};
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = dim3((unsigned)threads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  config.attrs = &attribute;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}
__device__ __forceinline__ void previous_kernel_done() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The next kernel's CTAs may come up as soon as every CTA of this one has said so.
__device__ __forceinline__ void next_kernel_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

inline __host__ __device__ long long round_up(long long x, long long m) { return (x + m - 1) / m * m; }

// Record the first device-side error: status[0] = code, status[1] = batch item,
// status[2] = detail (block or channel index).  Later errors are dropped.
__device__ inline void report_status(int* status, int code, int item, int detail) {
  if (status == nullptr) return;
  if (atomicCAS(status, 0, code) == 0) {
    status[1] = item;
    status[2] = detail;
  }
}

}  // namespace ticc
