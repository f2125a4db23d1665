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
  const int* has;     // [M / 128][K / kChunk]: whether that chunk of A (kChunk rows x 128 columns) holds anything but zeros, or null: all do
  const int* wide;    // n_wide (1 or 2) flags: with one set every chunk counts (an infinity or NaN in B, which zeros would turn into NaN)
  int n_wide;
  int* nonfinite;     // set to 1 when a stored value is not finite, or null
};

// A BF -> SF matrix is block diagonal with ladders of at most 2 J + 1 channels, so 5 or 6 of the 62 chunks of a 1984-channel
// product have anything to add.  A CTA lists its chunks from `has`, which the kernel that pads A fills on the way: lists made by a
// kernel of their own before each product cost a dense B 20 us a call (N = 128, 16 matrices: 84 -> 104 us).
__global__ void __launch_bounds__(kGemmThreads) gemm_tn_kernel(GemmBatch g) {
  extern __shared__ double smem[];
  const int m0 = blockIdx.x * kBlock, n0 = blockIdx.y * kBlock, b = blockIdx.z;
  TileAcc acc;
  int* list = nullptr;
  int listed = 0;
  if (g.has != nullptr) {
    list = reinterpret_cast<int*>(smem + kTileSmemBytes / sizeof(double));
    if (threadIdx.x < 32) {
      const int nchunk = g.K / kChunk, lane = threadIdx.x;
      const int* has = g.has + (long long)blockIdx.x * nchunk;
      const int first = g.wide[0], last = g.wide[g.n_wide - 1];
      int next = lane < nchunk ? has[lane] : 0;  // with the flags in flight
      int count = 0;
      for (int c0 = 0; c0 < nchunk; c0 += 32) {
        const bool mine = c0 + lane < nchunk && (first | last | next) != 0;
        next = c0 + 32 + lane < nchunk ? has[c0 + 32 + lane] : 0;
        const unsigned m = __ballot_sync(0xffffffffu, mine);
        if (mine) list[1 + count + __popc(m & ((1u << lane) - 1u))] = c0 + lane;
        count += __popc(m);
      }
      if (lane == 0) list[0] = count;
    }
    __syncthreads();
    listed = *list++;
  }
  tile_gemm_tn(acc, g.A + b * g.strideA + m0, g.lda, g.B + b * g.strideB + n0, g.ldb, g.K, smem, list, listed);
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
  const size_t bytes = kTileSmemBytes + (g.has != nullptr ? (1 + g.K / kChunk) * sizeof(int) : 0);
  cudaError_t e = cudaFuncSetAttribute(gemm_tn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  gemm_tn_kernel<<<dim3(M / kBlock, N / kBlock, batch), kGemmThreads, bytes, stream>>>(g);
  note_launch();
  return cudaGetLastError();
}

// Copy a batch of n x n matrices (complex interleaved when is_complex: `part` 0 = real,
// 1 = imaginary plane) into zero-padded np x np planes; *nonfinite is set when one holds an infinity or NaN.
__global__ void pad_plane_kernel(const double* src, int n, int is_complex, int part, double* dst, int np, int* nonfinite) {
  const int b = blockIdx.y;
  const double* s = src + (long long)b * n * n * (is_complex ? 2 : 1);
  double* d = dst + (long long)b * np * np;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < (long long)np * np; idx += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(idx / np), j = (int)(idx % np);
    double v = 0.0;
    if (i < n && j < n) v = is_complex ? s[2 * ((long long)i * n + j) + part] : s[(long long)i * n + j];
    if (!isfinite(v)) *nonfinite = 1;
    d[idx] = v;
  }
}

// The same for the n x n matrix that the product is taken with, a CTA a chunk of a 128-column tile, and has (as GemmBatch's) of
// each; clears `flags` ints for the kernels behind it.
constexpr int kPadThreads = 1024;
__global__ void __launch_bounds__(kPadThreads) pad_chunks_kernel(const double* __restrict__ src, int n, double* __restrict__ dst, int np, int* has, int* flags, int n_flags) {
  constexpr int kPer = kChunk * kBlock / kPadThreads;
  const int nchunk = np / kChunk, i0 = ((int)blockIdx.x % nchunk) * kChunk + threadIdx.x / kBlock, j = ((int)blockIdx.x / nchunk) * kBlock + (threadIdx.x & (kBlock - 1));
  double v[kPer];
  bool any = false;
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int i = i0 + u * (kPadThreads / kBlock);
    v[u] = i < n && j < n ? src[(long long)i * n + j] : 0.0;
  }
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    any |= v[u] != 0.0;  // a NaN too
    dst[(long long)(i0 + u * (kPadThreads / kBlock)) * np + j] = v[u];
  }
  const bool mine = __syncthreads_or(any);
  if (threadIdx.x == 0) has[blockIdx.x] = mine ? 1 : 0;
  if (blockIdx.x == 0 && (int)threadIdx.x < n_flags) flags[threadIdx.x] = 0;
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
