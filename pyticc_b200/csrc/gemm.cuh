// Batched FP64 GEMM C = alpha * A^T B on the DMMA tile core, for padded operands
// (M, N multiples of 128, K a multiple of 32).  A and B are k-major (row k holds
// A^T[k][:] and B[k][:]).  The result is stored as is or transposed.
#pragma once

#include "dmma_tile.cuh"
#include "ticc_common.cuh"

namespace ticc {

struct GemmBatch {
  const double* A;
  long long lda, strideA;
  const double* B;
  long long ldb, strideB;
  double* C;
  long long ldc, strideC;
  int K;
  double alpha;
  int transpose_store;
  const int* chunks;  // per 128-column tile of A its chunk count and chunk numbers (row stride K / kChunk + 1), or null: all
  int* nonfinite;     // set to 1 when a stored value is not finite, or null
};

// The chunks (kChunk rows) of each 128-column tile of A (k-major, K x M, the same for the whole batch) that hold anything but zeros.
// A BF -> SF matrix is block diagonal with ladders of at most 2 J + 1 channels, so 5 or 6 of the 62 chunks of a 1984-channel
// product have anything to add.  With *nonfinite set (an infinity or NaN in the other operand, which zeros
// would turn into NaN) every chunk is listed.  A warp looks through a chunk; grid: M / 128; kListThreads threads.
constexpr int kListThreads = 1024;
__global__ void __launch_bounds__(kListThreads) chunk_list_kernel(const double* __restrict__ A, long long lda, int K, const int* __restrict__ nonfinite, int* __restrict__ lists) {
  const int nchunk = K / kChunk, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* list = lists + (long long)blockIdx.x * (nchunk + 1);
  const bool all = *nonfinite != 0;
  __shared__ unsigned has;  // of the kListThreads / 32 chunks in hand
  int count = 0;
  for (int c0 = 0; c0 < nchunk; c0 += kListThreads / 32) {
    if (threadIdx.x == 0) has = 0u;
    __syncthreads();
    if (c0 + warp < nchunk) {
      const double2* a = reinterpret_cast<const double2*>(A + (long long)(c0 + warp) * kChunk * lda + (long long)blockIdx.x * kBlock);
      bool mine = all;
#pragma unroll 8
      for (int e = lane; e < kChunk * kBlock / 2; e += 32) {
        const double2 x = a[(long long)(e / (kBlock / 2)) * (lda / 2) + e % (kBlock / 2)];
        mine |= x.x != 0.0 || x.y != 0.0;
      }
      if (__any_sync(0xffffffffu, mine) && lane == 0) atomicOr(&has, 1u << warp);
    }
    __syncthreads();
    const unsigned m = has;
    if (threadIdx.x < 32 && ((m >> lane) & 1u)) list[1 + count + __popc(m & ((1u << lane) - 1u))] = c0 + lane;
    count += __popc(m);
    __syncthreads();
  }
  if (threadIdx.x == 0) list[0] = count;
}

__global__ void __launch_bounds__(kGemmThreads) gemm_tn_kernel(GemmBatch g) {
  extern __shared__ double smem[];
  const int m0 = blockIdx.x * kBlock, n0 = blockIdx.y * kBlock, b = blockIdx.z;
  TileAcc acc;
  const int* list = g.chunks != nullptr ? g.chunks + (long long)blockIdx.x * (g.K / kChunk + 1) : nullptr;
  tile_gemm_tn(acc, g.A + b * g.strideA + m0, g.lda, g.B + b * g.strideB + n0, g.ldb, g.K, smem, list != nullptr ? list + 1 : nullptr, list != nullptr ? list[0] : 0);
  if (g.nonfinite != nullptr) {
    bool bad = false;
#pragma unroll
    for (int mt = 0; mt < 8; ++mt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) bad |= !isfinite(acc.v[mt][nt][0]) || !isfinite(acc.v[mt][nt][1]);
    if (bad) *g.nonfinite = 1;
  }
  acc_to_smem(acc, smem, g.alpha);
  __syncthreads();
  double* C = g.C + b * g.strideC;
  for (int piece = threadIdx.x; piece < kBlock * 64; piece += kGemmThreads) {
    const int r = piece >> 6, c = (piece & 63) * 2;
    double2 v;
    if (g.transpose_store) {
      // destination row n0 + r, columns m0 + c, m0 + c + 1
      v.x = smem[c * kStride + r];
      v.y = smem[(c + 1) * kStride + r];
      *reinterpret_cast<double2*>(C + (long long)(n0 + r) * g.ldc + m0 + c) = v;
    } else {
      v.x = smem[r * kStride + c];
      v.y = smem[r * kStride + c + 1];
      *reinterpret_cast<double2*>(C + (long long)(m0 + r) * g.ldc + n0 + c) = v;
    }
  }
}

inline cudaError_t gemm_tn(const GemmBatch& g, int M, int N, int batch, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(gemm_tn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmemBytes);
  if (e != cudaSuccess) return e;
  gemm_tn_kernel<<<dim3(M / kBlock, N / kBlock, batch), kGemmThreads, kTileSmemBytes, stream>>>(g);
  note_launch();
  return cudaGetLastError();
}

// Copy a batch of n x n matrices (complex interleaved when is_complex: `part` 0 = real,
// 1 = imaginary plane) into zero-padded np x np planes; *nonfinite (optional) is set when one holds an infinity or NaN.
__global__ void pad_plane_kernel(const double* src, int n, int is_complex, int part, double* dst, int np, int* nonfinite = nullptr) {
  const int b = blockIdx.y;
  const double* s = src + (long long)b * n * n * (is_complex ? 2 : 1);
  double* d = dst + (long long)b * np * np;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < (long long)np * np; idx += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(idx / np), j = (int)(idx % np);
    double v = 0.0;
    if (i < n && j < n) v = is_complex ? s[2 * ((long long)i * n + j) + part] : s[(long long)i * n + j];
    if (nonfinite != nullptr && !isfinite(v)) *nonfinite = 1;
    d[idx] = v;
  }
}

__global__ void unpad_plane_kernel(const double* src, int np, double* dst, int n, int is_complex, int part) {
  const int b = blockIdx.y;
  const double* s = src + (long long)b * np * np;
  double* d = dst + (long long)b * n * n * (is_complex ? 2 : 1);
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < (long long)n * n; idx += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(idx / n), j = (int)(idx % n);
    const double v = s[(long long)i * np + j];
    if (is_complex) {
      d[2 * idx + part] = v;
    } else {
      d[idx] = v;
    }
  }
}

}  // namespace ticc
