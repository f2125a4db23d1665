// PotentialGrid -> V(R) contraction with the W_base assembly fused in.
//
// For one K group with weighted rows B (n_K x n_grid) and PES values v(R) on the
// quadrature grid, V_K(R)[a][b] = norm sum_q (Br[a][q] Br[b][q] + Bi[a][q] Bi[b][q]) v[q].
// One launch covers every group: each CTA computes a 32x32 lower-triangular tile of one group
// at one R on the FP64 tensor pipe and writes both (a, b) and (b, a), so V is exactly symmetric
// (the reference symmetrises explicitly).  The init kernel writes U/R^2 + 2 mu diag(E_int) (or
// zeros when only V is wanted) and the group kernel adds 2 mu V (or V) at the rows' output
// channel positions.
#pragma once

#include "dmma_tile.cuh"
#include "ticc_common.cuh"

namespace ticc {

__global__ void contract_init_kernel(double* out, int n, int n_R, const double* radial_points, const double* U, const double* E_int, double mu) {
  const long long total = (long long)n_R * n * n;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total; idx += (long long)gridDim.x * blockDim.x) {
    double v = 0.0;
    if (U != nullptr) {
      const long long r = idx / ((long long)n * n);
      const long long ij = idx % ((long long)n * n);
      const int i = (int)(ij / n), j = (int)(ij % n);
      const double R = radial_points[r];
      v = U[ij] / (R * R);
      if (i == j) v += 2.0 * mu * E_int[i];
    }
    out[idx] = v;
  }
}

// ---- the weighted-product tile on the FP64 tensor pipe ------------------------------------------
// A CTA computes one kVTile x kVTile tile X[i][j] = sum_q A[i][q] w[q] B[j][q] (plus the same over a second pair A2, B2: the
// imaginary rows of a complex basis) with mma.sync m8n8k4 f64 (DMMA), FP64 accumulation.  The rows are read as stored
// (row-major, q contiguous, any n_grid and any row offset) in chunks of 32 grid points: each warp loads whole 256-byte row
// segments, the weight is applied to A on the way into shared memory, and rows past the operand's end read as zeros.
// Shared tiles are [row][q] with a row stride of 36 doubles, so the fragment loads of a half-warp (rows mr = 0..3, k =
// 0..3) hit 16 distinct bank pairs.  Chunk c + 1 is copied asynchronously while chunk c is multiplied from the other shared buffer
// (one barrier per chunk).  kR radial points share a CTA where that leaves enough CTAs: the rows are the same at every one of them, so they are fetched
// once and the weight is applied to the A fragments.
// kVTile = 32, 4 warps of 16 x 16 (2 x 2 DMMA accumulators), six CTAs an SM.  K groups have 4 to a few hundred rows: a 64-tile
// (8 warps, three CTAs an SM) multiplies up to half of its work for nothing on ragged groups and the upper halves of diagonal
// tiles, and leaves small jobs with too few CTAs, while the operand bytes it saves come from L2 either way.  Measured, us,
// 64 / 32: AB+CD pair, 5 groups of 140-224 rows x 2700 complex points, 33 radii 2281 / 1758; 3 radii 394 / 284; 7 groups of
// 285-480 rows 4722 / 4732; vibrating A+BC, 31 groups of 4-124 rows x 1024 points, 33 radii 903 / 677; 9 groups of 20-52
// rows, 21 radii 114 / 76 (one radial point a CTA, rows staged through registers; as it stands the first takes 1480, the
// vibrating one 605).
constexpr int kVTile = 32;
constexpr int kVThreads = 128;
constexpr int kVChunk = 32;
constexpr int kVLd = kVChunk + 4;
constexpr int kVMaxGroups = 128;

constexpr int kVPart = 16;  // rows and columns of a warp's part of the tile
constexpr int kVLoad = kVTile / (kVThreads / 32);  // rows of a chunk that a warp loads
template <int kR>
constexpr int kVStage = 2 * kVTile * kVLd + kR * kVChunk;  // doubles of a chunk: A, B, weights
template <int kR>
constexpr size_t kVSmemBytes = size_t(2) * kVStage<kR> * sizeof(double);

// Element [r][mt][nt][h] of a warp's accumulator: radial point r, row vtile_row() + 8 mt + lane / 4, column vtile_col() + 8 nt + 2 (lane % 4) + h.
template <int kR>
struct VTileAcc {
  double v[kR][2][2][2];
};
__device__ __forceinline__ int vtile_row() { return (threadIdx.x >> 6) * kVPart; }
__device__ __forceinline__ int vtile_col() { return ((threadIdx.x >> 5) & 1) * kVPart; }

// 8 bytes, zero where !valid (the source is then not read).
__device__ __forceinline__ void cp_async8_or_zero(double* smem, const double* gmem, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem))), "l"(gmem), "r"(valid ? 8 : 0));
}

// A, B (and A2, B2) point at the tile's first row; rows at or beyond na (nb) read as zero.  w: kR rows of
// weights, w_stride apart.  A warp whose part of the tile is not `wanted` loads with the others but does not multiply.
template <int kR>
__device__ inline void vtile_product(VTileAcc<kR>& acc, const double* __restrict__ A, int na, const double* __restrict__ B, int nb, const double* __restrict__ A2,
                                     const double* __restrict__ B2, int n_grid, const double* __restrict__ w, long long w_stride, double* smem, bool wanted = true) {
  constexpr int kWarps = kVThreads / 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = vtile_row(), wn = vtile_col(), kr = lane & 3, mr = lane >> 2;
#pragma unroll
  for (int r = 0; r < kR; ++r)
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) acc.v[r][mt][nt][0] = acc.v[r][mt][nt][1] = 0.0;
  const int nq = (n_grid + kVChunk - 1) / kVChunk;
  const int nc = A2 != nullptr ? 2 * nq : nq;
  auto fetch = [&](int c) {
    const bool second = c >= nq;
    const int q = (second ? c - nq : c) * kVChunk + lane;  // loader: this grid point of rows warp + kWarps i
    const bool in = q < n_grid;
    const double* sa = (second ? A2 : A) + (in ? q : 0);
    const double* sb = (second ? B2 : B) + (in ? q : 0);
    double* buf = smem + (c & 1) * kVStage<kR> + lane;
#pragma unroll
    for (int i = 0; i < kVLoad; ++i) {
      const int row = warp + kWarps * i;
      const bool va = in && row < na, vb = in && row < nb;
      cp_async8_or_zero(buf + row * kVLd, va ? sa + (long long)row * n_grid : sa, va);
      cp_async8_or_zero(buf + (kVTile + row) * kVLd, vb ? sb + (long long)row * n_grid : sb, vb);
    }
    if (warp < kR) cp_async8_or_zero(buf + 2 * kVTile * kVLd + warp * kVChunk, w + warp * w_stride + (in ? q : 0), in);
    cp_async_commit();
  };
  static_assert(kR <= kWarps, "a warp loads the weights of one radial point");
  fetch(0);
  for (int c = 0; c < nc; ++c) {
    cp_async_wait<0>();
    __syncthreads();  // chunk c is in; the other buffer has been read
    if (c + 1 < nc) fetch(c + 1);
    const double* As = smem + (c & 1) * kVStage<kR>;
    const double* Bs = As + kVTile * kVLd;
    const double* ws = As + 2 * kVTile * kVLd + kr;
    if (wanted) {
#pragma unroll
      for (int kk = 0; kk < kVChunk; kk += 4) {
        double a[2], b[2];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) a[mt] = As[(wm + mt * 8 + mr) * kVLd + kk + kr];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) b[nt] = Bs[(wn + nt * 8 + mr) * kVLd + kk + kr];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          const double x = ws[r * kVChunk + kk];
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            const double ax = a[mt] * x;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) dmma_8x8x4(acc.v[r][mt][nt], ax, b[nt]);
          }
        }
      }
    }
  }
}

// Lower kVTile-tiles of every K group in one launch: tile t belongs to the group g with
// tile_start[g] <= t < tile_start[g + 1] (only groups with rows are listed).
struct ContractTiles {
  int n_groups;
  int tile_start[kVMaxGroups + 1];
  int row0[kVMaxGroups];
  int rows[kVMaxGroups];
};

// grid: (the table's tiles, groups of kR of the n_r radial points from r_first on).
template <int kR>
__global__ void __launch_bounds__(kVThreads, kR <= 2 ? 6 : 5) contract_group_kernel(const __grid_constant__ ContractTiles tiles, const double* __restrict__ Br,
                                                                                               const double* __restrict__ Bi, const int* __restrict__ row_out, int n_grid, double scale,
                                                                                               const double* __restrict__ potential, long long pot_stride, int r_first, int n_r, int n,
                                                                                               double* __restrict__ out) {
  extern __shared__ __align__(16) double vsmem[];
  const int t = blockIdx.x;
  int g = 0, hi = tiles.n_groups - 1;
  while (g < hi) {  // the last group whose first tile is at or before t
    const int mid = (g + hi + 1) >> 1;
    if (tiles.tile_start[mid] <= t) g = mid;
    else hi = mid - 1;
  }
  const int local = t - tiles.tile_start[g];
  int ta = (int)((sqrt(8.0 * local + 1.0) - 1.0) * 0.5);
  while ((ta + 1) * (ta + 2) / 2 <= local) ++ta;
  while (ta * (ta + 1) / 2 > local) --ta;
  const int tb = local - ta * (ta + 1) / 2;
  const int row0 = tiles.row0[g], rows = tiles.rows[g];
  const int first = blockIdx.y * kR, nr = min(kR, n_r - first), r0 = r_first + first;
  const long long ia = (long long)(row0 + ta * kVTile) * n_grid, ib = (long long)(row0 + tb * kVTile) * n_grid;
  const int wm = vtile_row(), wn = vtile_col(), lane = threadIdx.x & 31;
  // a warp's part below the last row, or strictly above the diagonal, adds nothing
  const bool wanted = ta * kVTile + wm < rows && tb * kVTile + wn < rows && (ta != tb || wm + kVPart > wn);
  const auto radii = [&](auto& acc, int at, int count) {  // `count` radial points from r0 + at on
    const double* w = potential + (long long)(r0 + at) * pot_stride;
    vtile_product(acc, Br + ia, rows - ta * kVTile, Br + ib, rows - tb * kVTile, Bi != nullptr ? Bi + ia : nullptr, Bi != nullptr ? Bi + ib : nullptr, n_grid, w, pot_stride, vsmem, wanted);
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int a = ta * kVTile + wm + mt * 8 + (lane >> 2);
          const int b = tb * kVTile + wn + nt * 8 + 2 * (lane & 3) + h;
          if (a >= rows || b >= rows || b > a) continue;
          const int pa = row_out[row0 + a], pb = row_out[row0 + b];
#pragma unroll
          for (int r = 0; r < count; ++r) {
            double* o = out + (long long)(r0 + at + r) * n * n;
            const double val = scale * acc.v[r][mt][nt][h];
            o[(long long)pa * n + pb] += val;
            if (a != b) o[(long long)pb * n + pa] += val;
          }
        }
  };
  if (nr == kR) {
    VTileAcc<kR> acc;
    radii(acc, 0, kR);
  } else {  // the last few radial points, one by one
    for (int r = 0; r < nr; ++r) {
      VTileAcc<1> acc;
      radii(acc, r, 1);
      __syncthreads();  // the next point's chunks go where the last one was read
    }
  }
}

template <int kR>
inline cudaError_t contract_groups_by(const ContractTiles& tiles, const double* Br, const double* Bi, const int* row_out, int n_grid, double scale, const double* potential, long long pot_stride, int n_R,
                                      int n, double* out, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(contract_group_kernel<kR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kVSmemBytes<kR>);
  constexpr int kMost = 65535 / kR * kR;  // radial points of a launch
  for (int r0 = 0; r0 < n_R && e == cudaSuccess; r0 += kMost) {
    const int n_r = n_R - r0 < kMost ? n_R - r0 : kMost;
    contract_group_kernel<kR><<<dim3(tiles.tile_start[tiles.n_groups], (n_r + kR - 1) / kR), kVThreads, kVSmemBytes<kR>, stream>>>(tiles, Br, Bi, row_out, n_grid, scale, potential, pot_stride, r0, n_r, n, out);
    note_launch();
    e = cudaGetLastError();
  }
  return e;
}
// How many radial points share a CTA.  Sharing saves the rows' copies and costs CTAs, which long grids bear better than short
// ones, so the lines lie between the two systems measured: two points from 2200 units (tiles x radial points) on, 1100
// CTAs for the 888 places of 148 SMs (six each), four from 4600 on, 1150 CTAs for 740 places (five each).
// Measured, us a call, 1 / 2 / 4 points: AB+CD pair (2 x 2700 grid points), 579 tiles, 2316 units 1205 / 1066 / 1011,
// 4632 2287 / 1949 / 1867, 13896 6613 / 5573 / 5301; vibrating A+BC (1024), 150 tiles, 1350 units 238 / 273 / 289, 2550 353 / 358 /
// 374, 4950 628 / 605 / 606, 13500 1608 / 1483 / 1387.
inline cudaError_t contract_groups(const ContractTiles& tiles, const double* Br, const double* Bi, const int* row_out, int n_grid, double scale, const double* potential, long long pot_stride, int n_R,
                                   int n, double* out, cudaStream_t stream) {
  const long long units = (long long)tiles.tile_start[tiles.n_groups] * n_R;
  const int pick = units >= 4600 ? 4 : units >= 2200 ? 2 : 1;
  return (pick == 4 ? contract_groups_by<4> : pick == 2 ? contract_groups_by<2> : contract_groups_by<1>)(tiles, Br, Bi, row_out, n_grid, scale, potential, pot_stride, n_R, n, out, stream);
}

// One block of a state-resolved (diabatic) contraction at every R:
//     X(R)[i][j] = sum_q A[i][q] w(R)[q] B[j][q],   A: n_a x n_grid, B: n_b x n_grid (row strides n_grid)
// written to out(R)[pos_a[i]][pos_b[j]] and, with `mirror`, also to out(R)[pos_b[j]][pos_a[i]].
// A symmetric block (`symmetric`: B is A and pos_b is pos_a) computes only i >= j and writes
// both (i, j) and (j, i), so the block is exactly symmetric.  grid: (tiles of A, tiles of B,
// radial points r_first ..); kVThreads threads; kVSmemBytes<1> dynamic shared memory.
__global__ void __launch_bounds__(kVThreads) weighted_block_kernel(const double* __restrict__ A, int n_a, const double* __restrict__ B, int n_b, int n_grid, const double* __restrict__ w,
                                                             long long w_stride, int r_first, const int* __restrict__ pos_a, const int* __restrict__ pos_b, int symmetric,
                                                             int mirror, int n, double* __restrict__ out) {
  extern __shared__ __align__(16) double vsmem[];
  const int ti = blockIdx.x, tj = blockIdx.y, R = r_first + blockIdx.z;
  if (symmetric && tj > ti) return;
  const int i0 = ti * kVTile, j0 = tj * kVTile;
  VTileAcc<1> acc;
  vtile_product(acc, A + (long long)i0 * n_grid, n_a - i0, B + (long long)j0 * n_grid, n_b - j0, nullptr, nullptr, n_grid, w + (long long)R * w_stride, w_stride, vsmem);
  double* o = out + (long long)R * n * n;
  const int lane = threadIdx.x & 31, wm = vtile_row(), wn = vtile_col();
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = i0 + wm + mt * 8 + (lane >> 2), j = j0 + wn + nt * 8 + 2 * (lane & 3) + h;
        if (i >= n_a || j >= n_b || (symmetric && j > i)) continue;
        const int pa = pos_a[i], pb = pos_b[j];
        o[(long long)pa * n + pb] = acc.v[0][mt][nt][h];
        if (mirror || (symmetric && i != j)) o[(long long)pb * n + pa] = acc.v[0][mt][nt][h];
      }
}


// Packed lower-triangle channel pairs of a fine-structure contraction into matrices: for every R
// and pair p = (i, j) = (pair_rows[p], pair_cols[p]), i >= j, with value v = src(R, p):
//   real (scalar FS):   out[i][j] = out[j][i] = v;
//   complex (spin FS):  v is conjugated where reversed[p]; out[i][j] = v, out[j][i] = conj(v),
//                       a diagonal element keeps the real part.
// src: n_R rows of src_stride elements (doubles, or interleaved complex doubles); out: n_R x n x n.
__global__ void __launch_bounds__(256) pairs_to_matrix_kernel(const double* __restrict__ src, int is_complex, long long src_stride, int n_pairs, const int* __restrict__ pair_rows,
                                                              const int* __restrict__ pair_cols, const unsigned char* __restrict__ reversed, int n, int n_R,
                                                              double* __restrict__ out) {
  const long long total = (long long)n_R * n_pairs;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int R = (int)(e / n_pairs), p = (int)(e % n_pairs);
    const int i = pair_rows[p], j = pair_cols[p];
    if (is_complex) {
      const double re = src[(long long)R * src_stride + 2 * p];
      double im = src[(long long)R * src_stride + 2 * p + 1];
      if (reversed != nullptr && reversed[p]) im = -im;
      double* o = out + 2 * (long long)R * n * n;
      if (i == j) {
        o[2 * ((long long)i * n + i)] = re;
        o[2 * ((long long)i * n + i) + 1] = 0.0;
      } else {
        o[2 * ((long long)i * n + j)] = re;
        o[2 * ((long long)i * n + j) + 1] = im;
        o[2 * ((long long)j * n + i)] = re;
        o[2 * ((long long)j * n + i) + 1] = -im;
      }
    } else {
      const double v = src[(long long)R * src_stride + p];
      double* o = out + (long long)R * n * n;
      o[(long long)i * n + j] = v;
      o[(long long)j * n + i] = v;
    }
  }
}

}  // namespace ticc
