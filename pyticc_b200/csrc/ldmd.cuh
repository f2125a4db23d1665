// LDMD log-derivative propagation (two half-steps per sector, diagonal reference
// potential at the sector midpoint), batched over energies, driven sector by sector.
//
// Per sector s with half-step h, ref = diag(W_mid), p^2 = ref - 2 mu E:
//   y1 = p coth(ph) | |p| cot(|p|h),  y2 = p csch(ph) | |p| csc(|p|h)   (series if |ph| < 1e-5)
//   Q_start = h (W_start - diag ref)/3,  Q_end = h (W_end - diag ref)/3,
//   Q_mid = (4/h) [(I - h^2 (W_mid - diag ref)/6)^{-1} - I]        (energy independent)
//   Y_mid = Q_mid + y1 - y2 (Y + Q_start + y1)^{-1} y2
//   Y_end = Q_end + y1 - y2 (Y_mid + Q_mid + y1)^{-1} y2
// The sweep returns S = -A^{-1}, so "- y2 A^{-1} y2" is "+ y2 S y2": every step
// between two inversions is one fused elementwise pass over the work matrices.
//
// Several channel blocks of one size (the K blocks of a coupled-states or NNCC system,
// padded to a common n) propagate together: the batch is (block g, energy e) with
// b = g * n_energy + e, block g reads its W at offset g * wb_stride, and Q_mid is one
// energy-shared matrix per (sector, block).
#pragma once

#include "sweep_fine.cuh"
#include "ticc_common.cuh"

namespace ticc {

struct LdmdSectors {
  const double* h;        // [n_sector] half-steps (device)
  const double* Ws;       // W_base at sector starts, sector stride ws_stride, row stride n
  const double* Wm;
  const double* We;
  long long ws_stride, wm_stride, we_stride;
  int n_sector;
  long long wb_stride;    // offset between the W of consecutive channel blocks (0: one block)
};

struct LdmdLayout {
  int n;          // logical channels
  int n_energy;
  int n_block;    // channel blocks; the batch of work matrices is n_block * n_energy
  int is_complex;
  int np;         // padded sweep size of the per-energy work matrix
  int npr;        // padded sweep size of the real, energy-shared Q_mid matrix
  double* M;      // [n_block * n_energy][np][np]
  double* Qm;     // [n_sector][n_block][npr][npr]
  double* y1;     // [n_sector][n_block * n_energy][n]
  double* y2;
  double* scratch;
  size_t scratch_doubles;
  int* reduced;   // [n_sector] leading sweep blocks taken in TF32x3 (mixed mode), else null
  double* fine;   // 64-tile sweeps' panels and flags (FP64 work matrices where they fit), else null
  double* fine_q; // the same region for the Q_mid sweeps, else null
  bool joint_q;   // the region holds the first work matrices and all Q_mid matrices together
  float* split;   // FP32 operand panels of the reduced steps' tcgen05 update (mixed mode), else null
};

// Mixed precision: a channel whose local wavenumber at the sector midpoint exceeds this
// (for the highest energy of the batch, p^2 = W_mid,ii - 2 mu E_max > kappa^2) is closed
// strongly enough that the FP32-level error of its block's trailing update decays before
// it reaches the open channels.  30 bohr^-1 keeps max|dS| ~1e-8 in the tested systems.
constexpr double kMixedKappa = 30.0;

inline int ldmd_np(int n, int is_complex) { return (int)round_up((long long)(is_complex ? 2 * n : n), kBlock); }

__device__ __forceinline__ void reference_pair(double h, double p2, double& y1, double& y2) {
  const double mag = sqrt(fabs(p2));
  const double arg = mag * h;
  if (fabs(arg) < 1.0e-5) {
    y1 = 1.0 / h + p2 * h / 3.0 - p2 * p2 * h * h * h / 45.0;
    y2 = 1.0 / h - p2 * h / 6.0 + 7.0 * p2 * p2 * h * h * h / 360.0;
  } else if (p2 >= 0.0) {
    y1 = mag / tanh(arg);
    y2 = mag / sinh(arg);
  } else {
    y1 = mag / tan(arg);
    y2 = mag / sin(arg);
  }
}

// y1/y2 for every (sector, block, energy, channel).
__global__ void ldmd_reference_kernel(LdmdSectors sec, const double* energies, double mu, int n, int n_energy, int n_block, double* y1, double* y2) {
  const long long total = (long long)sec.n_sector * n_block * n_energy * n;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total; idx += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(idx % n);
    const long long sb = idx / n;
    const int e = (int)(sb % n_energy);
    const long long sg = sb / n_energy;
    const int g = (int)(sg % n_block);
    const int s = (int)(sg / n_block);
    const double ref = sec.Wm[s * sec.wm_stride + g * sec.wb_stride + (long long)i * n + i];
    double a, b;
    reference_pair(sec.h[s], ref - 2.0 * mu * energies[e], a, b);
    y1[idx] = a;
    y2[idx] = b;
  }
}

__device__ __forceinline__ double sym(const double* W, int n, int i, int j) { return 0.5 * (W[(long long)i * n + j] + W[(long long)j * n + i]); }

// Number of leading 128-blocks of the (closed-first ordered) work matrix whose channels
// are all closed beyond kMixedKappa at the highest energy, in every channel block; one CTA
// per sector.
__global__ void ldmd_reduced_blocks_kernel(LdmdSectors sec, const double* energies, double mu, int n, int n_energy, int n_block, int np, int is_complex, int* reduced) {
  __shared__ double e_max;
  __shared__ int first_open;
  const int s = blockIdx.x;
  if (threadIdx.x == 0) {
    double m = energies[0];
    for (int e = 1; e < n_energy; ++e) m = fmax(m, energies[e]);
    e_max = m;
    first_open = n;
  }
  __syncthreads();
  for (int g = 0; g < n_block; ++g) {
    const double* Wm = sec.Wm + s * sec.wm_stride + g * sec.wb_stride;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const double p2 = Wm[(long long)i * n + i] - 2.0 * mu * e_max;
      if (!(p2 > kMixedKappa * kMixedKappa)) atomicMin(&first_open, i);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int rows = (first_open == n) ? np : first_open * (is_complex ? 2 : 1);
    reduced[s] = rows / kBlock;
  }
}

// Mq = I - h^2 (W_mid - diag ref)/6 (padded identity), batched over (sector, block):
// blockIdx.y = s * n_block + g.
__global__ void ldmd_qmid_build_kernel(LdmdSectors sec, int n, int n_block, int npr, double* Qm) {
  const int sg = blockIdx.y;
  const int s = sg / n_block, g = sg % n_block;
  const double h = sec.h[s];
  const double* Wm = sec.Wm + s * sec.wm_stride + g * sec.wb_stride;
  double* Q = Qm + (long long)sg * npr * npr;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < (long long)npr * npr; idx += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(idx / npr), j = (int)(idx % npr);
    double v;
    if (i < n && j < n) {
      v = (i == j) ? 1.0 : -h * h * sym(Wm, n, i, j) / 6.0;
    } else {
      v = (i == j) ? 1.0 : 0.0;
    }
    Q[idx] = v;
  }
}

// Q_mid = (4/h)(X - I) from the swept matrix -X.
__global__ void ldmd_qmid_finish_kernel(LdmdSectors sec, int n, int n_block, int npr, double* Qm) {
  const int sg = blockIdx.y;
  const double h = sec.h[sg / n_block];
  double* Q = Qm + (long long)sg * npr * npr;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < (long long)npr * npr; idx += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(idx / npr), j = (int)(idx % npr);
    Q[idx] = (i < n && j < n) ? 4.0 / h * (-Q[idx] - (i == j ? 1.0 : 0.0)) : 0.0;
  }
}

// Store one logical element (X + iZ) of a work matrix, or padding.
__device__ __forceinline__ void put_element(double* Mb, int np, int i, int j, double x, double z, int is_complex) {
  if (is_complex) {
    Mb[(long long)(2 * i) * np + 2 * j] = x;
    Mb[(long long)(2 * i) * np + 2 * j + 1] = z;
    Mb[(long long)(2 * i + 1) * np + 2 * j] = z;
    Mb[(long long)(2 * i + 1) * np + 2 * j + 1] = -x;
  } else {
    Mb[(long long)i * np + j] = x;
  }
}

// Read the swept value S = -A^{-1} at logical (i, j): real part S00 and the imaginary
// companion -S01 (so that -A^{-1} = s_re + i s_im).  The symmetric sweep keeps only the
// lower and diagonal 128-tiles current, so an element of an upper tile is read at (j, i).
__device__ __forceinline__ void get_swept(const double* Mb, int np, int i, int j, int is_complex, double& s_re, double& s_im) {
  const int mi = is_complex ? 2 * i : i, mj = is_complex ? 2 * j : j;
  if ((mi >> 7) < (mj >> 7)) {
    const int x = i;
    i = j;
    j = x;
  }
  if (is_complex) {
    s_re = Mb[(long long)(2 * i) * np + 2 * j];
    s_im = -Mb[(long long)(2 * i) * np + 2 * j + 1];
  } else {
    s_re = Mb[(long long)i * np + j];
    s_im = 0.0;
  }
}

// Work-matrix padding: identity on the padded diagonal of the real sweep matrix.
__device__ __forceinline__ void put_padding(double* Mb, int np, long long r, long long c) { Mb[r * np + c] = (r == c) ? 1.0 : 0.0; }

// One complex element of the caller's Y, which need not be 16-byte aligned.
__device__ __forceinline__ void put_pair(double* y, double re, double im) {
  y[0] = re;
  y[1] = im;
}

// W_base must be exactly symmetric (the contraction writes both halves from one value), so the per-energy passes read
// W[i][j] only, row-contiguous across the lanes of a warp.
// phase 0: A = Y_in + Q_start + y1          (first sector of the call)
// phase 1: A = [Q_end' + y1' + y2' S y2'] + Q_start + y1   (S from the previous sector)
// phase 2: B = 2 Q_mid + 2 y1 + y2 S y2
// phase 3: Y_out = Q_end + y1 + y2 S y2     (last sector of the call)
// Every quantity is symmetric and the sweep reads only the lower and diagonal 128-tiles, so only those are passed over: bound by
// reading and writing them once.  A CTA covers 16 logical rows of one 128-tile (a warp two rows, a lane two double2
// of each: two columns of a real matrix, one element X + iZ of a complex one) for a group of energies; the
// energy-independent part of its elements stays in registers over the group, and two energies' loads are in flight at a
// time.  The groups are cut so that few or small matrices still fill the chip (one CTA a row over all energies took
// 15 us for 16 matrices of 231 channels and 350 us for 16 of 1984 in phase 2: here 7 and 97, 5.9 TB/s).  Y_in and Y_out are dense
// n x n; their transposed halves pass through shared memory in 16-column strips.
constexpr int kElemRows = 16;
constexpr int kElemThreads = 256;

template <int kPhase, bool kCplx>
__global__ void __launch_bounds__(kElemThreads) ldmd_elementwise_kernel(int s, int e_per, LdmdSectors sec, LdmdLayout L, const double* Yin, double* Yout) {
  constexpr int kCols = kCplx ? kBlock / 2 : kBlock;     // logical columns (and rows) of a 128-tile
  constexpr int kGroups = kCols / kElemRows;             // row groups of a tile
  constexpr int kEach = kCplx ? 1 : 2;                   // logical columns of a double2
  constexpr bool kDense = kPhase == 0 || kPhase == 3;    // reads or writes Y
  // [logical column of the tile][row of the group]: the transposed half of Y, one plane for each part of a complex element
  __shared__ double strip[kDense ? (kCplx ? 2 : 1) * kCols * (kElemRows + 1) : 1];
  int ta, tb;
  lower_pair(blockIdx.x / kGroups, ta, tb);
  const int g = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = L.n, np = L.np, ne = L.n_energy, batch = L.n_block * ne;
  const int i0 = ta * kCols + (blockIdx.x % kGroups) * kElemRows, j0 = tb * kCols;
  const int e0 = blockIdx.y * e_per, e1 = min(ne, e0 + e_per);
  // The W matrices and (but for the first sector) Q_mid were complete before the sweep ahead of this pass began: their part is
  // read ahead of the wait.  A sweep does not let its successor start before its last CTA has left, so for a pass that is
  // its launch and these loads; the sweep behind a pass comes up with the pass's last wave.
  next_kernel_may_start();
  if (s == 0) previous_kernel_done();
  if (kPhase == 3 && i0 >= n) return;
  const double h = sec.h[s];
  const long long wb = g * sec.wb_stride;
  const double* Wm = sec.Wm + s * sec.wm_stride + wb;
  const int i[2] = {i0 + 2 * warp, i0 + 2 * warp + 1};
  // energy-independent part of each element: [row][chunk][column of the double2]
  double base[2][2][kEach];
  const double* Wrow = (kPhase == 3 ? sec.We + s * sec.we_stride : sec.Ws + s * sec.ws_stride) + wb;
  const double* Wprev = kPhase == 1 ? sec.We + (s - 1) * sec.we_stride + wb : nullptr;
  const double* Q = L.Qm + ((long long)s * L.n_block + g) * L.npr * L.npr;
  const double h3 = h / 3.0, hp3 = kPhase == 1 ? sec.h[s - 1] / 3.0 : 0.0;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    double ref = 0.0, ref_p = 0.0;  // taken off the diagonal before anything is multiplied: W_ii - ref_i cancels
    if (kPhase != 2 && i[r] < n) {
      ref = Wm[(long long)i[r] * n + i[r]];
      if (kPhase == 1) ref_p = sec.Wm[(s - 1) * sec.wm_stride + wb + (long long)i[r] * n + i[r]];
    }
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int c = 0; c < kEach; ++c) {
        const int j = j0 + (q * 32 + lane) * kEach + c;
        double v = 0.0;
        if (i[r] < n && j < n) {
          if (kPhase == 2) {
            v = 2.0 * Q[(long long)i[r] * L.npr + j];
          } else {
            v = h3 * (Wrow[(long long)i[r] * n + j] - (i[r] == j ? ref : 0.0));
            if (kPhase == 1) v = fma(hp3, Wprev[(long long)i[r] * n + j] - (i[r] == j ? ref_p : 0.0), v);
          }
        }
        base[r][q][c] = v;
      }
  }
  previous_kernel_done();
  const int sy = kPhase == 1 ? s - 1 : s;  // the sector whose y1, y2 fold the swept matrix
  for (int e = e0; e < e1; e += 2) {
    const int cnt = min(2, e1 - e);
    double2 m[2][2][2];  // [energy][row][chunk]: swept values in, new values out
    double yj[2][2][kEach];
    if (kPhase != 0) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int b = g * ne + e + (u < cnt ? u : 0);
        const double* Mb = L.M + (long long)b * np * np + (long long)j0 * (kCplx ? 2 : 1);
        const double* y2 = L.y2 + ((long long)sy * batch + b) * n;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
#pragma unroll
          for (int r = 0; r < 2; ++r) m[u][r][q] = *reinterpret_cast<const double2*>(Mb + (long long)(kCplx ? 2 * i[r] : i[r]) * np + (q * 32 + lane) * 2);
#pragma unroll
          for (int c = 0; c < kEach; ++c) {
            const int j = j0 + (q * 32 + lane) * kEach + c;
            yj[u][q][c] = j < n ? y2[j] : 0.0;
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (u >= cnt) break;
      const int b = g * ne + e + u;
      const double* Yb = Yin + (long long)b * n * n * (kCplx ? 2 : 1);
      if (kPhase == 0) {  // Y[j][i] of the group's rows, 16 contiguous columns a row
        __syncthreads();
        for (int t = threadIdx.x; t < kCols * kElemRows; t += kElemThreads) {
          const int jj = t / kElemRows, ii = t % kElemRows;
          const bool in = j0 + jj < n && i0 + ii < n;
          const long long at = (long long)(j0 + jj) * n + i0 + ii;
          if (kCplx) {
            strip[jj * (kElemRows + 1) + ii] = in ? Yb[2 * at] : 0.0;
            strip[(kCols + jj) * (kElemRows + 1) + ii] = in ? Yb[2 * at + 1] : 0.0;
          } else {
            strip[jj * (kElemRows + 1) + ii] = in ? Yb[at] : 0.0;
          }
        }
        __syncthreads();
      }
      if (kPhase == 3) __syncthreads();  // the previous energy's strip has been written out
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const bool row_in = i[r] < n;
        const double* y1 = L.y1 + ((long long)s * batch + b) * n;
        const double y1i = row_in ? y1[i[r]] : 0.0;
        const double y2i = row_in && kPhase != 0 ? L.y2[((long long)sy * batch + b) * n + i[r]] : 0.0;
        const double d = kPhase == 2 ? 2.0 * y1i : kPhase == 1 ? y1i + (row_in ? L.y1[((long long)sy * batch + b) * n + i[r]] : 0.0) : y1i;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int j = j0 + (q * 32 + lane) * kEach, jj = j - j0, ii = i[r] - i0;
          double2 x;
          if (kCplx) {
            const bool in = row_in && j < n;
            x = make_double2(base[r][q][0] + (i[r] == j ? d : 0.0), 0.0);
            if (kPhase == 0) {
              const long long at = (long long)i[r] * n + j;
              if (in) {
                x.x += 0.5 * (Yb[2 * at] + strip[jj * (kElemRows + 1) + ii]);
                x.y = 0.5 * (Yb[2 * at + 1] + strip[(kCols + jj) * (kElemRows + 1) + ii]);
              }
            } else {
              x.x += y2i * m[u][r][q].x * yj[u][q][0];
              x.y = -(y2i * m[u][r][q].y * yj[u][q][0]);  // the embedding holds -S on its imaginary places
            }
            if (!in) x = make_double2(i[r] == j ? 1.0 : 0.0, 0.0);
          } else {
            x = make_double2(base[r][q][0] + (i[r] == j ? d : 0.0), base[r][q][kEach - 1] + (i[r] == j + 1 ? d : 0.0));
            if (kPhase == 0) {
              const long long at = (long long)i[r] * n + j;
              if (row_in && j < n) x.x += 0.5 * (Yb[at] + strip[jj * (kElemRows + 1) + ii]);
              if (row_in && j + 1 < n) x.y += 0.5 * (Yb[at + 1] + strip[(jj + 1) * (kElemRows + 1) + ii]);
            } else {
              x.x += y2i * m[u][r][q].x * yj[u][q][0];
              x.y += y2i * m[u][r][q].y * yj[u][q][kEach - 1];
            }
            if (!row_in || j >= n) x.x = (i[r] == j) ? 1.0 : 0.0;
            if (!row_in || j + 1 >= n) x.y = (i[r] == j + 1) ? 1.0 : 0.0;
          }
          if (kPhase != 3) {
            double* Mb = L.M + (long long)b * np * np + (long long)j0 * (kCplx ? 2 : 1) + (q * 32 + lane) * 2;
            if (kCplx) {
              const bool pad = !row_in || j >= n;
              *reinterpret_cast<double2*>(Mb + (long long)(2 * i[r]) * np) = x;
              *reinterpret_cast<double2*>(Mb + (long long)(2 * i[r] + 1) * np) = pad ? make_double2(0.0, x.x) : make_double2(x.y, -x.x);
            } else {
              *reinterpret_cast<double2*>(Mb + (long long)i[r] * np) = x;
            }
          } else {
            double* Yo = Yout + (long long)b * n * n * (kCplx ? 2 : 1);
            const long long at = (long long)i[r] * n + j;
            if (kCplx) {
              if (row_in && j < n) put_pair(Yo + 2 * at, x.x, x.y);
              strip[jj * (kElemRows + 1) + ii] = x.x;
              strip[(kCols + jj) * (kElemRows + 1) + ii] = x.y;
            } else {
              if (row_in && j < n) Yo[at] = x.x;
              if (row_in && j + 1 < n) Yo[at + 1] = x.y;
              strip[jj * (kElemRows + 1) + ii] = x.x;
              strip[(jj + 1) * (kElemRows + 1) + ii] = x.y;
            }
          }
        }
      }
      if (kPhase == 3 && ta != tb) {  // the upper half as the transpose of the lower tiles
        __syncthreads();
        double* Yo = Yout + (long long)b * n * n * (kCplx ? 2 : 1);
        for (int t = threadIdx.x; t < kCols * kElemRows; t += kElemThreads) {
          const int jj = t / kElemRows, ii = t % kElemRows;
          if (j0 + jj >= n || i0 + ii >= n) continue;
          const long long at = (long long)(j0 + jj) * n + i0 + ii;
          if (kCplx) put_pair(Yo + 2 * at, strip[jj * (kElemRows + 1) + ii], strip[(kCols + jj) * (kElemRows + 1) + ii]);
          else Yo[at] = strip[jj * (kElemRows + 1) + ii];
        }
      }
    }
  }
}

inline cudaError_t ldmd_elementwise(int phase, int s, const LdmdSectors& sec, const LdmdLayout& L, const double* Yin, double* Yout, cudaStream_t stream) {
  const int nt = L.np / kBlock, groups = (L.is_complex ? kBlock / 2 : kBlock) / kElemRows;
  const long long tiles = (long long)nt * (nt + 1) / 2 * groups;
  // energies of a CTA: all of them where that still gives some six CTAs an SM
  const long long per_energy = tiles * L.n_block, target = 900;
  long long e_per = per_energy * L.n_energy / target;
  e_per = e_per < 1 ? 1 : e_per > L.n_energy ? L.n_energy : e_per;
  const dim3 grid((unsigned)tiles, (unsigned)((L.n_energy + e_per - 1) / e_per), (unsigned)L.n_block);
  const auto launch = [&](auto* real, auto* complex) { return launch_overlapped(L.is_complex ? complex : real, grid, kElemThreads, 0, stream, s, (int)e_per, sec, L, Yin, Yout); };
  note_launch();
  switch (phase) {
    case 0: return launch(ldmd_elementwise_kernel<0, false>, ldmd_elementwise_kernel<0, true>);
    case 1: return launch(ldmd_elementwise_kernel<1, false>, ldmd_elementwise_kernel<1, true>);
    case 2: return launch(ldmd_elementwise_kernel<2, false>, ldmd_elementwise_kernel<2, true>);
    default: return launch(ldmd_elementwise_kernel<3, false>, ldmd_elementwise_kernel<3, true>);
  }
}

// ---- matrices of at most 128 rows: the whole call in one launch ----------------------------------------
// A sweep of so small a matrix is one CTA's work, and launched pass by pass it is mostly launches, fills of idle SMs and
// traffic of padding (a 24-row matrix was padded to 128 rows in memory): 27 us per half-step of 21 channels.  Here
// one CTA keeps its (block, energy) matrix in shared memory through every sector of the call: the elementwise passes
// run between inversions on the tile itself, and only W, Q_mid, y1 and y2 are read.  D = 32 or 64: Gauss-Jordan
// exchange, whose permuted result the next pass reads in place; D = 128: the two-level sweep_block.
// Measured (B200), propagate_logD of N = 21, 1 energy, 16 sectors: 898 -> 363 us a call; coupled-states blocks of 1 to 21
// channels, 16 energies, 12 sectors: 5.7 -> 4.1 ms a call (the rest was the host's per-block work: 1.7 ms since that is shared).
template <int D>
struct SmallShape {
  static constexpr int kThreads = D == 32 ? 128 : 256;
  static constexpr int kLd = D + 4;
  static constexpr size_t kAux = D == 128 ? kPivotAuxBytes / sizeof(double) : kGJAuxDoubles + size_t(D) * kLd;
  static constexpr size_t kSmemBytes = (size_t(D) * kLd + kAux + 6 * D) * sizeof(double);
  static constexpr int kPer = D == 128 ? 1 : D * D / kThreads;
  static constexpr int kPerSM = D == 32 ? 4 : D == 64 ? 2 : 1;
};

// Invert the matrix in S (used rows: `used`) and call f(r, c, v, w) for every c <= r < used with the swept value v = -A^{-1}(r, c),
// symmetrised, and w = pre(r, c): what f needs from global memory, fetched before the inversion where registers hold it.
template <int D, class P, class F>
__device__ inline bool small_sweep_then(double* S, double* aux, int used, P&& pre, F&& f) {
  using Sh = SmallShape<D>;
  const int n_act = (int)round_up(used, kGJPanel);
  if constexpr (D == 128) {
    const bool singular = sweep_block<true>(S, aux, n_act);
    // pairs (r, c), (c, r) belong to one thread: in place
    for (int e = threadIdx.x; e < used * D; e += Sh::kThreads) {
      const int r = e / D, c = e % D;
      if (c > r) continue;
      const double v = 0.5 * (S[r * Sh::kLd + c] + S[c * Sh::kLd + r]);
      f(r, c, v, pre(r, c));
    }
    __syncthreads();
    return singular;
  } else {
    double w[Sh::kPer], x[Sh::kPer];
#pragma unroll
    for (int u = 0; u < Sh::kPer; ++u) {
      const int e = threadIdx.x + u * Sh::kThreads, r = e / D, c = e % D;
      w[u] = (D == 32 && r < used && c <= r) ? pre(r, c) : 0.0;  // (64 rows: the registers are the exchange's)
    }
    GJOrder order;
    const bool singular = gauss_jordan_exchange<Sh::kLd, Sh::kThreads, D>(S, aux, order, n_act, GJFromCopy<Sh::kLd, Sh::kThreads, D>{aux + kGJAuxDoubles});
#pragma unroll
    for (int u = 0; u < Sh::kPer; ++u) {
      const int e = threadIdx.x + u * Sh::kThreads, r = e / D, c = e % D;
      x[u] = 0.0;
      if (r < used && c <= r) x[u] = -0.5 * (S[order.perm[r] * Sh::kLd + order.iperm[c]] + S[order.perm[c] * Sh::kLd + order.iperm[r]]);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < Sh::kPer; ++u) {
      const int e = threadIdx.x + u * Sh::kThreads, r = e / D, c = e % D;
      if (r < used && c <= r) f(r, c, x[u], D == 32 ? w[u] : pre(r, c));
    }
    __syncthreads();
    return singular;
  }
}

// Both elements of a pair; the identity (once: sweeping leaves +-1 there, decoupled) on the rows from `used` to the edge.
template <int D>
__device__ __forceinline__ void small_put(double* S, int r, int c, double v) {
  S[r * SmallShape<D>::kLd + c] = v;
  S[c * SmallShape<D>::kLd + r] = v;
}
template <int D>
__device__ __forceinline__ void small_pad(double* S, int used) {
  const int n_act = D == 128 ? D : (int)round_up(used, kGJPanel);
  for (int e = threadIdx.x; e < n_act * n_act; e += SmallShape<D>::kThreads) {
    const int r = e / n_act, c = e % n_act;
    if (r >= used || c >= used) S[r * SmallShape<D>::kLd + c] = (r == c) ? 1.0 : 0.0;
  }
}

// Q_mid of every (sector, block): one CTA each.
template <int D>
__global__ void __launch_bounds__(SmallShape<D>::kThreads, SmallShape<D>::kPerSM) ldmd_small_qmid_kernel(LdmdSectors sec, int n, int n_block, int npr, double* Qm, int* status) {
  extern __shared__ __align__(16) double smem[];
  using Sh = SmallShape<D>;
  double* S = smem;
  double* aux = smem + D * Sh::kLd;
  const int sg = blockIdx.x, s = sg / n_block, g = sg % n_block;
  const double h = sec.h[s];
  const double* Wm = sec.Wm + s * sec.wm_stride + g * sec.wb_stride;
  double* Q = Qm + (long long)sg * npr * npr;
  small_pad<D>(S, n);
  for (int e = threadIdx.x; e < n * n; e += Sh::kThreads) {
    const int i = e / n, j = e % n;
    S[i * Sh::kLd + j] = (i == j) ? 1.0 : -h * h * sym(Wm, n, i, j) / 6.0;
  }
  __syncthreads();
  const bool singular = small_sweep_then<D>(S, aux, n, [](int, int) { return 0.0; }, [&](int i, int j, double v, double) {
    const double q = 4.0 / h * (-v - (i == j ? 1.0 : 0.0));
    Q[(long long)i * npr + j] = q;
    Q[(long long)j * npr + i] = q;
  });
  if (singular && threadIdx.x == 0) report_status(status, kDeviceSingularPivot, sg, 0);
}

template <int D>
__global__ void __launch_bounds__(SmallShape<D>::kThreads, SmallShape<D>::kPerSM) ldmd_small_kernel(LdmdSectors sec, LdmdLayout L, double* Y, int* status) {
  extern __shared__ __align__(16) double smem[];
  using Sh = SmallShape<D>;
  double* S = smem;
  double* aux = smem + D * Sh::kLd;
  double* vec = aux + Sh::kAux;  // ref, y1, y2 of this sector and the one before
  const int b = blockIdx.x, g = b / L.n_energy, n = L.n, batch = L.n_block * L.n_energy;
  const bool cplx = L.is_complex != 0;
  const int used = cplx ? 2 * n : n;
  bool singular = false;
  small_pad<D>(S, used);
  double* Yb = Y + (long long)b * n * n * (cplx ? 2 : 1);
  const long long wb = g * sec.wb_stride;
  double h_next = sec.h[0], h = 0.0, hp = 0.0, ref_next = 0.0, y1_next = 0.0, y2_next = 0.0;
  const auto fetch = [&](int s) {  // a sector's channel values, a channel a thread, ahead of the sector
    h_next = sec.h[s];
    const int i = threadIdx.x;
    if (i < n) {
      ref_next = sec.Wm[s * sec.wm_stride + wb + (long long)i * n + i];
      y1_next = L.y1[((long long)s * batch + b) * n + i];
      y2_next = L.y2[((long long)s * batch + b) * n + i];
    }
  };
  fetch(0);
  for (int s = 0; s < sec.n_sector; ++s) {
    double *ref = vec + 3 * D * (s & 1), *y1 = ref + D, *y2 = y1 + D;
    const double *refp = vec + 3 * D * ((s + 1) & 1), *y1p = refp + D, *y2p = y1p + D;
    hp = h;
    h = h_next;
    const double* Ws = sec.Ws + s * sec.ws_stride + wb;
    const double *We = sec.We + s * sec.we_stride + wb, *Wep = s > 0 ? sec.We + (s - 1) * sec.we_stride + wb : We;
    const double* Q = L.Qm + ((long long)s * L.n_block + g) * L.npr * L.npr;
    if ((int)threadIdx.x < n) {
      ref[threadIdx.x] = ref_next;
      y1[threadIdx.x] = y1_next;
      y2[threadIdx.x] = y2_next;
    }
    __syncthreads();
    if (s + 1 < sec.n_sector) fetch(s + 1);
    // element (r, c) of the work matrix: the real part of logical (i, j), or in a complex call the part that its
    // place in the 2x2 block [[X, Z], [Z, -X]] asks for
    const double h3 = h / 3.0, hp3 = hp / 3.0;
    const auto imaginary = [&](int r, int c) { return cplx && ((r ^ c) & 1); };
    const auto start_w = [&](int r, int c) {  // the part of phases 0 and 1 that comes from W
      const int i = cplx ? r >> 1 : r, j = cplx ? c >> 1 : c;
      if (imaginary(r, c)) return 0.0;
      double x = h3 * (Ws[(long long)i * n + j] - (i == j ? ref[i] : 0.0));
      if (s > 0) x += hp3 * (Wep[(long long)i * n + j] - (i == j ? refp[i] : 0.0));
      return x;
    };
    const auto start = [&](int r, int c, double before, double w) {  // `before` is Y, or y2 S y2 of the last sector
      const int i = cplx ? r >> 1 : r, j = cplx ? c >> 1 : c;
      const bool imag = imaginary(r, c);
      double x = before + w;
      if (!imag && i == j) x += s > 0 ? y1[i] + y1p[i] : y1[i];
      small_put<D>(S, r, c, (cplx && !imag && (r & 1)) ? -x : x);
    };
    // y2_i S_ij y2_j from the swept element of the same place (in a complex call -S on the imaginary places and on the
    // lower right one of each block)
    const auto folded = [&](int r, int c, double v, const double* w) {
      if (!cplx) return w[r] * v * w[c];
      const bool imag = (r ^ c) & 1, lower = !imag && (r & 1);
      return w[r >> 1] * (imag || lower ? -v : v) * w[c >> 1];
    };
    if (s == 0) {
      for (int e = threadIdx.x; e < used * used; e += Sh::kThreads) {
        const int r = e / used, c = e % used;
        if (c > r) continue;
        double v;
        if (cplx) {
          const int i = r >> 1, j = c >> 1, im = (r ^ c) & 1;
          v = 0.5 * (Yb[2 * ((long long)i * n + j) + im] + Yb[2 * ((long long)j * n + i) + im]);
        } else {
          v = 0.5 * (Yb[(long long)r * n + c] + Yb[(long long)c * n + r]);
        }
        start(r, c, v, start_w(r, c));
      }
      __syncthreads();
    } else {
      singular |= small_sweep_then<D>(S, aux, used, start_w, [&](int r, int c, double v, double w) { start(r, c, folded(r, c, v, y2p), w); });
    }
    singular |= small_sweep_then<D>(
        S, aux, used, [&](int r, int c) { return imaginary(r, c) ? 0.0 : 2.0 * Q[(long long)(cplx ? r >> 1 : r) * L.npr + (cplx ? c >> 1 : c)]; },
        [&](int r, int c, double v, double w) {
          const int i = cplx ? r >> 1 : r, j = cplx ? c >> 1 : c;
          const bool imag = imaginary(r, c);
          double x = folded(r, c, v, y2) + w;
          if (!imag && i == j) x += 2.0 * y1[i];
          small_put<D>(S, r, c, (cplx && !imag && (r & 1)) ? -x : x);
        });
    if (s + 1 == sec.n_sector) {
      singular |= small_sweep_then<D>(
          S, aux, used,
          [&](int r, int c) {
            const int i = cplx ? r >> 1 : r, j = cplx ? c >> 1 : c;
            return imaginary(r, c) ? 0.0 : h3 * (We[(long long)i * n + j] - (i == j ? ref[i] : 0.0));
          },
          [&](int r, int c, double v, double w) {
            const int i = cplx ? r >> 1 : r, j = cplx ? c >> 1 : c;
            const bool imag = imaginary(r, c);
            // the first row of each 2x2 block holds both parts (on the diagonal its imaginary part is visited in the second)
            if (cplx && (r & 1) && !(imag && i == j)) return;
            double x = folded(r, c, v, y2) + w;
            if (!imag && i == j) x += y1[i];
            if (cplx) {
              Yb[2 * ((long long)i * n + j) + (imag ? 1 : 0)] = x;
              Yb[2 * ((long long)j * n + i) + (imag ? 1 : 0)] = x;
            } else {
              Yb[(long long)i * n + j] = x;
              Yb[(long long)j * n + i] = x;
            }
          });
    }
  }
  if (singular && threadIdx.x == 0) report_status(status, kDeviceSingularPivot, b, 0);
}

inline unsigned grid_for(long long work, int threads, unsigned cap = 1u << 16) {
  long long blocks = (work + threads - 1) / threads;
  if (blocks < 1) blocks = 1;
  return (unsigned)(blocks > cap ? cap : blocks);
}

// Q_mid for every (sector, block) of the call: build, sweep (batched, chunked to fit scratch) and finish.
inline void ldmd_qmid_build(const LdmdSectors& sec, const LdmdLayout& L, cudaStream_t stream) {
  ldmd_qmid_build_kernel<<<dim3(grid_for((long long)L.npr * L.npr, 256, 4096), sec.n_sector * L.n_block), 256, 0, stream>>>(sec, L.n, L.n_block, L.npr, L.Qm);
  note_launch();
}
inline cudaError_t ldmd_qmid_sweep(const LdmdSectors& sec, const LdmdLayout& L, int* status, cudaStream_t stream) {
  const long long per = (long long)L.npr * L.npr;
  const int count = sec.n_sector * L.n_block;
  const int chunk = (int)(L.scratch_doubles / sweep_scratch_doubles(L.npr));
  FineState fine{L.fine_q};
  for (int s0 = 0; s0 < count; s0 += chunk) {
    const int cnt = (count - s0 < chunk) ? count - s0 : chunk;
    cudaError_t e = sweep_any(fine, L.Qm + (long long)s0 * per, per, L.npr, cnt, L.scratch, status, stream, nullptr, L.n, nullptr);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
inline cudaError_t ldmd_qmid_finish(const LdmdSectors& sec, const LdmdLayout& L, cudaStream_t stream) {
  ldmd_qmid_finish_kernel<<<dim3(grid_for((long long)L.npr * L.npr, 256, 4096), sec.n_sector * L.n_block), 256, 0, stream>>>(sec, L.n, L.n_block, L.npr, L.Qm);
  note_launch();
  return cudaGetLastError();
}

// Whether the Q_mid matrices of a call are swept beside its first work matrices, in one launch: they have the same size
// in a real call, and the 64-tile sweep is bound by its chain, which more matrices do not lengthen.
inline bool ldmd_joint_qmid(int n, size_t batch, size_t q_count, int is_complex, bool fp64) { return fp64 && !is_complex && q_count <= 64 && use_fine(n, batch) && use_fine(n, batch + q_count); }

template <int D>
inline cudaError_t ldmd_small_qmid(const LdmdSectors& sec, const LdmdLayout& L, int* status, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(ldmd_small_qmid_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SmallShape<D>::kSmemBytes);
  if (e != cudaSuccess) return e;
  ldmd_small_qmid_kernel<D><<<sec.n_sector * L.n_block, SmallShape<D>::kThreads, SmallShape<D>::kSmemBytes, stream>>>(sec, L.n, L.n_block, L.npr, L.Qm, status);
  note_launch();
  return cudaGetLastError();
}
template <int D>
inline cudaError_t ldmd_small(double* Y, const LdmdSectors& sec, const LdmdLayout& L, int* status, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(ldmd_small_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SmallShape<D>::kSmemBytes);
  if (e != cudaSuccess) return e;
  ldmd_small_kernel<D><<<L.n_block * L.n_energy, SmallShape<D>::kThreads, SmallShape<D>::kSmemBytes, stream>>>(sec, L, Y, status);
  note_launch();
  return cudaGetLastError();
}

// Propagate every (block, energy) through every sector of the call.  Y (device,
// n_block x n_energy x n x n, complex interleaved when is_complex) is read at the first
// sector start and overwritten with the log-derivative at the last sector end.
inline cudaError_t ldmd_propagate(double* Y, const double* energies, double mu, const LdmdSectors& sec, LdmdLayout& L, int* status, cudaStream_t stream) {
  const int batch = L.n_block * L.n_energy;
  ldmd_reference_kernel<<<grid_for((long long)sec.n_sector * batch * L.n, 256), 256, 0, stream>>>(sec, energies, mu, L.n, L.n_energy, L.n_block, L.y1, L.y2);
  note_launch();
  if (L.reduced != nullptr) {
    ldmd_reduced_blocks_kernel<<<sec.n_sector, 256, 0, stream>>>(sec, energies, mu, L.n, L.n_energy, L.n_block, L.np, L.is_complex, L.reduced);
    note_launch();
  }
  const int rows = L.is_complex ? 2 * L.n : L.n;
  if (rows <= kBlock) {
    cudaError_t e = L.n <= 32 ? ldmd_small_qmid<32>(sec, L, status, stream) : L.n <= 64 ? ldmd_small_qmid<64>(sec, L, status, stream) : ldmd_small_qmid<128>(sec, L, status, stream);
    if (e != cudaSuccess) return e;
    return rows <= 32 ? ldmd_small<32>(Y, sec, L, status, stream) : rows <= 64 ? ldmd_small<64>(Y, sec, L, status, stream) : ldmd_small<128>(Y, sec, L, status, stream);
  }
  // one launch sweeps the first sector's work matrices and every Q_mid where the layout has room for both
  const bool joint = L.joint_q;
  ldmd_qmid_build(sec, L, stream);
  cudaError_t err = joint ? cudaSuccess : ldmd_qmid_sweep(sec, L, status, stream);
  if (err == cudaSuccess && !joint) err = ldmd_qmid_finish(sec, L, stream);
  if (err != cudaSuccess) return err;
  const long long mstride = (long long)L.np * L.np;
  const int used = L.is_complex ? 2 * L.n : L.n;  // rows of the work matrix beyond these are identity padding
  FineState fine{L.fine};
  for (int s = 0; s < sec.n_sector; ++s) {
    err = ldmd_elementwise(s == 0 ? 0 : 1, s, sec, L, Y, Y, stream);
    if (err != cudaSuccess) return err;
    if (s == 0 && joint) {
      err = fine_sweep(fine, L.M, mstride, L.np, used, batch, status, stream, L.Qm, (long long)L.npr * L.npr, sec.n_sector * L.n_block);
      if (err == cudaSuccess) err = ldmd_qmid_finish(sec, L, stream);
    } else {
      err = sweep_any(fine, L.M, mstride, L.np, batch, L.scratch, status, stream, L.reduced ? L.reduced + s : nullptr, used, L.split);
    }
    if (err != cudaSuccess) return err;
    err = ldmd_elementwise(2, s, sec, L, Y, Y, stream);
    if (err != cudaSuccess) return err;
    err = sweep_any(fine, L.M, mstride, L.np, batch, L.scratch, status, stream, L.reduced ? L.reduced + s : nullptr, used, L.split);
    if (err != cudaSuccess) return err;
  }
  return ldmd_elementwise(3, sec.n_sector - 1, sec, L, Y, Y, stream);
}

}  // namespace ticc
