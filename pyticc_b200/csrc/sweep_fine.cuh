// The symmetric sweep M <- -M^{-1} for matrices that are too few or too small to fill the chip with
// 128-tiles: 64-wide steps on 64x64 tiles, the whole sweep in one persistent launch.
//
// Such a sweep is bound by its critical chain (invert a pivot block, form the next block column's panel, update
// the next pivot block, invert it ...), not by flops or bytes: with one launch per 128-step each link of the chain also
// paid a launch, and its 128x128 products ran on one SM each (17 us on the FP64 pipe; 64x64x64: 2.4 us).  Here
// work units come from one queue, in an order in which every unit depends on earlier units only, so that waiting
// for flags cannot deadlock (an earlier unit belongs to a CTA that is already running).  Per step k:
//   chain unit (one per matrix): panel of block column k + 1, update of the pivot block k + 1 and its inverse,
//     all in one CTA's shared memory: the critical chain leaves the SM only to publish P^{-1};
//   panel units: for every other block row j the old tile X of (j, k) and R = its product with P^{-1}, both
//     into the step's panel slot as they stand (row-major, X[k][c] for j < k, X[c][k] for j > k: the
//     consumer's fragment strides absorb the orientation, so no tile is transposed), and R into M;
//   update units: M(i, j) -= cold_i^T U_j for the lower tiles outside row and column k, those of block
//     column k + 1 first (the next step's panels), then k + 2.
// Flags (per matrix, monotonic over the sweeps of one call, so that only the first one clears them): per lower tile the number
// of steps applied, per block row the last panel, the last inverted pivot, per step the finished updates (a
// panel slot is rewritten kFineSlots steps later, once its readers are done).
// A step of the chain takes 22-23 us: 13 for the block's inversion, 2.3 and 1.3 for its two products (one SM's FP64 pipe),
// 2 for publishing P^{-1}, the rest the flag's way to the next CTA, its load of P^{-1} and the stores in between.  The last
// block is inverted to its last used panel of columns only: N = 231 (40 of 64), 16 energies, 8 sectors 1807 -> 1747 us;
// N = 660 (24 of 64) 2420 -> 2390.
#pragma once

#include <algorithm>

#include "sweep.cuh"

namespace ticc {

constexpr int kFineThreads = 256;
constexpr int kFineSlots = 2;                         // panel slots of a matrix, by step
constexpr int kFinePinv = kFineSlots + 1;             // P^{-1} slots: step k's readers are done once step k's updates are, which the chain of step k + 2 waits for
constexpr int kFineTile = kSub * kSub;                // doubles of a tile
constexpr int kFineMaxTiles = 64;                     // block rows (N <= 4096)
constexpr int kFineTransLd = kSub + 1;
constexpr size_t kFineSmemBytes = (size_t(3) * kSub * kSmallLd + kGJAuxDoubles + 2) * sizeof(double);

inline int fine_tiles(int n_used) { return (n_used + kSub - 1) / kSub; }
// Integers of one matrix's flags: panels, finished updates per step, pivot, tile versions.
__host__ __device__ inline int fine_flag_ints(int nt) { return 2 * nt + 2 + nt * (nt + 1) / 2; }
// Doubles of scratch per matrix, and of the control block before them (queue, abort flag).
constexpr int kFineControlDoubles = 32;
inline size_t fine_scratch_doubles(int nt) { return size_t(kFineSlots) * 2 * nt * kFineTile + size_t(kFinePinv) * kFineTile + (fine_flag_ints(nt) + 1) / 2; }
inline size_t fine_total_doubles(int nt, size_t batch) { return kFineControlDoubles + batch * fine_scratch_doubles(nt); }

struct FineSweep {
  double* M;
  long long mstride;
  int ld, nt, batch;
  double* M2;      // matrices `split` .. batch - 1 (same size and row stride) lie here
  long long mstride2;
  int split;
  double* slots;   // [batch][kFineSlots][2 (X, R)][nt][64][64]
  double* pinv;    // [batch][kFinePinv][64][64]
  int* flags;      // [batch][fine_flag_ints(nt)]
  int* control;    // queue, abort flag
  int* status;
  int base;        // value that the flags of this sweep start from: sweep number * nt
  int sweep;       // number of this sweep in the call (the finished-update counters grow by one sweep's worth each)
  int queue_base;  // queue value at which this launch starts
  int last;        // columns of the last block to invert (a multiple of kGJPanel): the rest of it is decoupled identity
};

__device__ __forceinline__ double* fine_matrix(const FineSweep& w, int b) { return b < w.split ? w.M + (long long)b * w.mstride : w.M2 + (long long)(b - w.split) * w.mstride2; }

// Batch item of matrix b in the device status: its place among its own kind.
__device__ __forceinline__ int fine_item(const FineSweep& w, int b) { return b < w.split ? b : b - w.split; }

// Positions 0 .. nt - 2 of the block rows other than k, from k + 1 on, cyclic.
__device__ __forceinline__ int fine_row_at(int k, int nt, int pos) {
  const int j = k + 1 + pos;
  return j < nt ? j : j - nt;
}
__device__ __forceinline__ int fine_lower(int a, int b) { return a >= b ? a * (a + 1) / 2 + b : b * (b + 1) / 2 + a; }

// Thread 0 polls until every flag reaches its target (all flags' loads in flight together: one after the other they cost the
// chain 2000 cycles a step); all threads return whether that happened before the poll limit and without an abort by
// another CTA.  Ends with a __syncthreads().
struct FineNeed {
  const int* flag[4];
  int target[4];
};
__device__ __forceinline__ FineNeed fine_need(const int* f0, int t0, const int* f1, int t1, const int* f2, int t2, const int* f3, int t3) { return FineNeed{{f0, f1, f2, f3}, {t0, t1, t2, t3}}; }
__device__ inline bool fine_wait(const FineSweep& w, const FineNeed& need, int b, int* shared_ok) {
  if (threadIdx.x == 0) {
    int ok = 1;
    const long long limit = g_step_poll_limit;
    for (long long it = 0;; ++it) {
      if (it >= limit) {
        if (atomicExch(w.control + 1, 1) == 0) report_status(w.status, kDeviceStalled, fine_item(w, b), -1);
        ok = 0;
        break;
      }
      const int abort = load_relaxed(w.control + 1);
      const int f0 = load_relaxed(need.flag[0]), f1 = load_relaxed(need.flag[1]), f2 = load_relaxed(need.flag[2]), f3 = load_relaxed(need.flag[3]);
      if (abort != 0) {
        ok = 0;
        break;
      }
      if (f0 >= need.target[0] && f1 >= need.target[1] && f2 >= need.target[2] && f3 >= need.target[3]) {
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        break;
      }
      if (it > 64) __nanosleep(64);
    }
    *shared_ok = ok;
  }
  __syncthreads();
  return *shared_ok != 0;
}

// 64x64 tile (row stride ld, 16-byte aligned rows) into shared rows of kSmallLd, in two cp.async groups' worth of
// halves: rows [32 half, +32).
__device__ __forceinline__ void fine_stage(double* S, const double* src, long long ld, int half) {
#pragma unroll
  for (int u = 0; u < kFineTile / 4 / kFineThreads; ++u) {
    const int piece = threadIdx.x + u * kFineThreads, r = 32 * half + (piece >> 5), c = (piece & 31) * 2;
    cp_async16(S + r * kSmallLd + c, src + (long long)r * ld + c);
  }
}

struct FineAcc {
  double v[2][4][2];  // rows 16 (warp / 2) + 8 u + lane / 4, columns 32 (warp % 2) + 8 w + 2 (lane % 4) + h
};
// acc += sum_k A[m][k] B[k][n] over k0 .. k0 + K - 1 with element strides (am, ak), (bk, bn), one of each pair 1 and the other
// kSmallLd (4 mod 16: conflict-free fragments either way).
__device__ __forceinline__ void fine_product(FineAcc& acc, const double* A, int am, int ak, const double* B, int bk, int bn, int k0, int K) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, mr = lane >> 2, kr = lane & 3;
  const double* a0 = A + (16 * (warp >> 1) + mr) * am + (k0 + kr) * ak;
  const double* b0 = B + (k0 + kr) * bk + (32 * (warp & 1) + mr) * bn;
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    double a[2], b[4];
#pragma unroll
    for (int u = 0; u < 2; ++u) a[u] = a0[8 * u * am + k * ak];
#pragma unroll
    for (int w = 0; w < 4; ++w) b[w] = b0[8 * w * bn + k * bk];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int w = 0; w < 4; ++w) dmma_8x8x4(acc.v[u][w], a[u], b[w]);
  }
}
// S[r][c] = S[c][r] = old - (A B^T)[r][c] for the lower triangle, A, B and S 64 x 64 with row stride kSmallLd.  Of the 36 lower 8 x 8
// tiles warp s < 4 multiplies tile row s and warp 4 + s tile row 7 - s: nine for every SM sub-partition, where the whole
// square takes sixteen.  A template of the tile row, since predicated-off multiplications cost as much as real ones.
// old: the row's tiles from C (row stride ld).
template <int kRow>
__device__ __forceinline__ void fine_lower_row(const double* A, const double* B, double* S, const double* C, long long ld) {
  const int lane = threadIdx.x & 31, mr = lane >> 2, kr = lane & 3, r = 8 * kRow + mr;
  double2 old[kRow + 1];
  double acc[kRow + 1][2];
#pragma unroll
  for (int i = 0; i <= kRow; ++i) {
    old[i] = __ldcg(reinterpret_cast<const double2*>(C + (long long)r * ld + 8 * i + 2 * kr));
    acc[i][0] = acc[i][1] = 0.0;
  }
  const double *a = A + r * kSmallLd + kr, *b = B + mr * kSmallLd + kr;
#pragma unroll 2
  for (int k = 0; k < kSub; k += 4) {
    const double x = a[k];
#pragma unroll
    for (int i = 0; i <= kRow; ++i) dmma_8x8x4(acc[i], x, b[8 * i * kSmallLd + k]);
  }
  __syncthreads();  // S may be A
#pragma unroll
  for (int i = 0; i <= kRow; ++i) {
    const int c = 8 * i + 2 * kr;
    const double x = old[i].x - acc[i][0], y = old[i].y - acc[i][1];
    if (i < kRow || r >= c) S[r * kSmallLd + c] = S[c * kSmallLd + r] = x;
    if (i < kRow || r >= c + 1) S[r * kSmallLd + c + 1] = S[(c + 1) * kSmallLd + r] = y;
  }
}
__device__ __forceinline__ void fine_lower_update(const double* A, const double* B, double* S, const double* C, long long ld) {
  switch (threadIdx.x >> 5) {
    case 0: fine_lower_row<0>(A, B, S, C, ld); break;
    case 1: fine_lower_row<1>(A, B, S, C, ld); break;
    case 2: fine_lower_row<2>(A, B, S, C, ld); break;
    case 3: fine_lower_row<3>(A, B, S, C, ld); break;
    case 4: fine_lower_row<7>(A, B, S, C, ld); break;
    case 5: fine_lower_row<6>(A, B, S, C, ld); break;
    case 6: fine_lower_row<5>(A, B, S, C, ld); break;
    default: fine_lower_row<4>(A, B, S, C, ld); break;
  }
}
__device__ __forceinline__ void fine_zero(FineAcc& acc) {
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int w = 0; w < 4; ++w) acc.v[u][w][0] = acc.v[u][w][1] = 0.0;
}
__device__ __forceinline__ void fine_sub(FineAcc& c, const FineAcc& d) {
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      c.v[u][w][0] -= d.v[u][w][0];
      c.v[u][w][1] -= d.v[u][w][1];
    }
}
// By one thread behind a __syncthreads(): count a finished update of this step.  The fence orders the reads of its panel tiles (the
// whole CTA's, through the barrier) before the count, on which the chain waits before it has the slots written again; with
// `version` it publishes the updated tile too, so that the two cost one fence.
__device__ __forceinline__ void fine_count_update(int* done, int* version = nullptr, int value = 0) {
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  if (version != nullptr) asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(version), "r"(value) : "memory");
  asm volatile("red.relaxed.gpu.global.add.s32 [%0], 1;" ::"l"(done) : "memory");
}
// Call f(row, column, double2 of the accumulator) for every pair this lane holds.
template <class F>
__device__ __forceinline__ void fine_each(FineAcc& acc, F&& f) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int w = 0; w < 4; ++w) f(16 * (warp >> 1) + 8 * u + (lane >> 2), 32 * (warp & 1) + 8 * w + 2 * (lane & 3), acc.v[u][w]);
}

// The upper 64-tile of a diagonal 128-tile is read by the passes after the sweep: whoever writes its lower partner last also
// writes the transpose.
__device__ __forceinline__ bool fine_mirrors(int ta, int tb, bool last) { return last && ta == tb + 1 && (tb & 1) == 0; }

// A pivot block once more, for gauss_jordan_any_range, from what it was made of: M's diagonal tile, which is written after the
// inversion only, less X R^T behind a panel (X in its slot, which no step after the next writes before this
// block's pivot is out, and R in shared memory).  Nothing to keep, and no pointer of its own: the kernel with two CTAs an
// SM has no register for one (2 % of a sweep).
struct FineAgain {
  const FineSweep& w;
  int b, k;
  const double* R;
  __device__ __forceinline__ void keep(const GJStrip<kSub>&) const {}
  __device__ __forceinline__ void restore(double* S) const {
    const double* C = fine_matrix(w, b) + (long long)k * kSub * w.ld + k * kSub;
    const double* X = w.slots + (((long long)b * kFineSlots + (k - 1) % kFineSlots) * 2 * w.nt + k) * kFineTile;
#pragma unroll 1
    for (int e = threadIdx.x; e < kFineTile; e += kFineThreads) {  // the lower half to both places
      const int r = e / kSub, c = e % kSub, i = max(r, c), j = min(r, c);
      double v = __ldcg(C + (long long)i * w.ld + j);
      if (k > 0) {
#pragma unroll 1
        for (int q = 0; q < kSub; ++q) v = fma(-__ldcg(X + i * kSub + q), R[j * kSmallLd + q], v);
      }
      S[r * kSmallLd + c] = v;
    }
    __syncthreads();
  }
};

// Invert the symmetric block in S; publish P^{-1} first (`pivot_flag`, on which the chain waits), then write -P^{-1} into
// M's diagonal tile and set its version.  T: 64 x kFineTransLd scratch, written after the inversion
// (behind a panel it comes with R, row stride kSmallLd).
__device__ inline void fine_invert(const FineSweep& w, int b, int k, double* S, double* T, double* aux, double* Mb, int* pivot_flag, int* version, int value) {
  GJOrder order;
  const int n_act = k == w.nt - 1 ? w.last : kSub;
  const bool singular = gauss_jordan_exchange<kSmallLd, kFineThreads>(S, aux, order, n_act, FineAgain{w, b, k, T});
  if (singular && threadIdx.x == 0) report_status(w.status, kDeviceSingularPivot, fine_item(w, b), k * kSub / kBlock);  // detail: the 128-block, as on the other paths
  double* P = w.pinv + ((long long)b * kFinePinv + k % kFinePinv) * kFineTile;
  double* D = Mb + (long long)k * kSub * w.ld + k * kSub;
  // the inverse out of its exchange order into T (odd row stride: conflict-free columns), then symmetrised on the way out
  for (int e = threadIdx.x; e < kFineTile; e += kFineThreads) {
    const int r = e / kSub, c = e % kSub;
    T[r * kFineTransLd + c] = S[order.perm[r] * kSmallLd + order.iperm[c]];
  }
  __syncthreads();
  constexpr int kPer = kFineTile / kFineThreads;
  double p[kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int e = threadIdx.x + u * kFineThreads, r = e / kSub, c = e % kSub;
    p[u] = 0.5 * (T[r * kFineTransLd + c] + T[c * kFineTransLd + r]);
    P[e] = p[u];
  }
  __syncthreads();
  if (threadIdx.x == 0) store_release(pivot_flag, value);
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int e = threadIdx.x + u * kFineThreads;
    D[(long long)(e / kSub) * w.ld + e % kSub] = -p[u];
  }
  __syncthreads();
  if (threadIdx.x == 0) store_release(version, value);
}

template <int kPerSM>
__global__ void __launch_bounds__(kFineThreads, kPerSM) sweep_fine_kernel(const FineSweep w) {
  extern __shared__ __align__(16) double smem[];
  double* SA = smem;
  double* SB = smem + kSub * kSmallLd;
  double* SC = smem + 2 * kSub * kSmallLd;
  double* aux = smem + 3 * kSub * kSmallLd;
  int* slot = reinterpret_cast<int*>(aux + kGJAuxDoubles);
  const int nt = w.nt, t = nt - 1, fints = fine_flag_ints(nt), batch = w.batch;
  const int per_step = batch * (t + t * (t + 1) / 2 - 1);  // the last step has `batch` more
  const int total = batch + per_step * nt + batch;
  const int tid = threadIdx.x;
  previous_kernel_done();
  for (;;) {
    if (tid == 0) slot[0] = atomicAdd(w.control, 1) - w.queue_base;
    __syncthreads();
    const int u = slot[0];
    __syncthreads();  // also: the previous unit's shared memory is free
    if (u < 0 || u >= total) return;
    if (u < batch) {  // the first pivot
      double* Mb = fine_matrix(w, u);
      for (int half = 0; half < 2; ++half) fine_stage(SA, Mb, w.ld, half);
      cp_async_commit();
      cp_async_wait<0>();
      __syncthreads();
      int* f = w.flags + (long long)u * fints;
      fine_invert(w, u, 0, SA, SC, aux, Mb, f + 2 * nt, f + 2 * nt + 2, w.base + 1);
      continue;
    }
    int v = u - batch;
    const int k = v / per_step < t ? v / per_step : t;
    v -= k * per_step;
    const bool last = k == t;
    int b, pos = -1, px = -1, py = -1;  // panel position, or the positions of an update's tile
    bool chain = false;
    if (!last && v < batch) {
      b = v;
      pos = 0;
      chain = true;
    } else {
      if (!last) v -= batch;
      const int first = last ? 0 : 1, panels = t - first;
      b = v % batch;
      v /= batch;
      if (v < panels) {
        pos = v + first;
      } else {
        v -= panels;
        // block column k + 1 (position 0) first, then the others as a triangle; its own (0, 0) is the chain's
        const int column = t - first;
        if (v < column) {
          px = v + first;
          py = 0;
        } else {
          lower_pair(v - column, px, py);
          ++px;
          ++py;
        }
      }
    }
    double* Mb = fine_matrix(w, b);
    int* f = w.flags + (long long)b * fints;
    int* done = f + nt;
    const int* ver = f + 2 * nt + 2;
    double* X = w.slots + ((long long)b * kFineSlots + k % kFineSlots) * 2 * nt * kFineTile;
    double* R = X + (long long)nt * kFineTile;
    const int now = w.base + k;  // version of a tile that has been through steps 0 .. k - 1
    const int per_update = t * (t + 1) / 2;
    if (pos >= 0) {
      // ---- panel of block row j (and, in a chain unit, the next pivot)
      const int j = fine_row_at(k, nt, pos);
      const bool below = j > k;  // the lower tile is (j, k), X[c][k]; else (k, j), X[k][c]
      double* T = Mb + (long long)(below ? j : k) * kSub * w.ld + (below ? k : j) * kSub;
      const int* mine = ver + fine_lower(j, k);
      const int* pivot = f + 2 * nt;
      const int* diagonal = chain ? ver + fine_lower(j, j) : mine;
      const int* readers = k >= kFineSlots ? done + k - kFineSlots : mine;  // the slot's readers kFineSlots steps ago
      const int readers_target = k >= kFineSlots ? (w.sweep + 1) * per_update : now;
      double* Xj = X + (long long)j * kFineTile;
      double* Rj = R + (long long)j * kFineTile;
      // everything but P^{-1} first: the chain's next link is then only P^{-1} away
      if (!fine_wait(w, fine_need(mine, now, diagonal, now, readers, readers_target, mine, now), b, slot + 1)) return;
      for (int half = 0; half < 2; ++half) fine_stage(SA, T, w.ld, half);
      cp_async_commit();
      cp_async_wait<0>();
      __syncthreads();
#pragma unroll 4
      for (int e = tid; e < kFineTile / 2; e += kFineThreads) {
        const int r = e / (kSub / 2), c = 2 * (e % (kSub / 2));
        *reinterpret_cast<double2*>(Xj + r * kSub + c) = *reinterpret_cast<const double2*>(SA + r * kSmallLd + c);
      }
      if (!fine_wait(w, fine_need(pivot, now + 1, pivot, now + 1, pivot, now + 1, pivot, now + 1), b, slot + 1)) return;
      const double* P = w.pinv + ((long long)b * kFinePinv + k % kFinePinv) * kFineTile;
      for (int half = 0; half < 2; ++half) fine_stage(SB, P, kSub, half);
      cp_async_commit();
      cp_async_wait<0>();
      __syncthreads();
      FineAcc acc;
      fine_zero(acc);
      // P is symmetric: X P for a tile below the diagonal block (rows of X are its channels), P X for one before it
      if (below) fine_product(acc, SA, kSmallLd, 1, SB, kSmallLd, 1, 0, kSub);
      else fine_product(acc, SB, kSmallLd, 1, SA, kSmallLd, 1, 0, kSub);
      const bool mirror = fine_mirrors(below ? j : k, below ? k : j, last);
      double* Mt = Mb + (long long)(below ? k : j) * kSub * w.ld + (below ? j : k) * kSub;
      fine_each(acc, [&](int r, int c, double(&d)[2]) {
        const double2 x = make_double2(d[0], d[1]);
        *reinterpret_cast<double2*>(T + (long long)r * w.ld + c) = x;
        *reinterpret_cast<double2*>(Rj + r * kSub + c) = x;
        if (mirror) {
          Mt[(long long)c * w.ld + r] = d[0];
          Mt[(long long)(c + 1) * w.ld + r] = d[1];
        }
      });
      if (chain) fine_each(acc, [&](int r, int c, double(&d)[2]) { *reinterpret_cast<double2*>(SC + r * kSmallLd + c) = make_double2(d[0], d[1]); });
      __syncthreads();
      // published by a warp that the inversion needs last
      if (tid == kFineThreads - 32) {
        store_release(f + j, now + 1);
        store_release(const_cast<int*>(ver) + fine_lower(j, k), now + 1);
      }
      if (!chain) continue;
      // M(j, j) - X R^T (here j = k + 1 > k: X[c][k], R[c][k]), lower half, mirrored
      fine_lower_update(SA, SC, SA, Mb + (long long)j * kSub * w.ld + j * kSub, w.ld);
      __syncthreads();
      if (tid == kFineThreads - 64) fine_count_update(done + k);
      fine_invert(w, b, j, SA, SC, aux, Mb, f + 2 * nt, const_cast<int*>(ver) + fine_lower(j, j), now + 2);
      continue;
    }
    // ---- trailing update of one lower tile
    const int jx = fine_row_at(k, nt, px), jy = fine_row_at(k, nt, py);
    const int ta = max(jx, jy), tb = min(jx, jy);
    const int* mine = ver + fine_lower(ta, tb);
    if (!fine_wait(w, fine_need(f + ta, now + 1, f + tb, now + 1, mine, now, mine, now), b, slot + 1)) return;
    const double* Xa = X + (long long)ta * kFineTile;
    const double* Rb = R + (long long)tb * kFineTile;
    for (int half = 0; half < 2; ++half) {
      fine_stage(SA, Xa, kSub, half);
      fine_stage(SB, Rb, kSub, half);
    }
    cp_async_commit();
    double* C = Mb + (long long)ta * kSub * w.ld + tb * kSub;
    FineAcc old, acc;
    fine_each(old, [&](int r, int c, double(&d)[2]) {
      const double2 x = __ldcg(reinterpret_cast<const double2*>(C + (long long)r * w.ld + c));
      d[0] = x.x;
      d[1] = x.y;
    });
    fine_zero(acc);
    cp_async_wait<0>();
    __syncthreads();
    fine_product(acc, SA, ta > k ? kSmallLd : 1, ta > k ? 1 : kSmallLd, SB, tb > k ? 1 : kSmallLd, tb > k ? kSmallLd : 1, 0, kSub);
    const bool diagonal = ta == tb, mirror = fine_mirrors(ta, tb, last);
    double* Ct = Mb + (long long)tb * kSub * w.ld + ta * kSub;
    fine_sub(old, acc);
    fine_each(old, [&](int r, int c, double(&d)[2]) {
      if (!diagonal) {
        *reinterpret_cast<double2*>(C + (long long)r * w.ld + c) = make_double2(d[0], d[1]);
        if (mirror) {
          Ct[(long long)c * w.ld + r] = d[0];
          Ct[(long long)(c + 1) * w.ld + r] = d[1];
        }
      } else {  // the lower half to both places: the tile stays exactly symmetric
        if (r >= c) {
          C[(long long)r * w.ld + c] = d[0];
          if (r > c) C[(long long)c * w.ld + r] = d[0];
        }
        if (r >= c + 1) {
          C[(long long)r * w.ld + c + 1] = d[1];
          if (r > c + 1) C[(long long)(c + 1) * w.ld + r] = d[1];
        }
      }
    });
    __syncthreads();
    if (tid == 0) fine_count_update(done + k, const_cast<int*>(ver) + fine_lower(ta, tb), now + 1);
  }
}

// The sweeps of one call share `scratch` (fine_total_doubles(nt, batch) doubles) and are numbered: the first one clears the
// flags, a later one starts from the values that the one before left.
struct FineState {
  double* scratch = nullptr;  // null: the path is not available
  int nt = 0, batch = 0, sweeps = 0, queue = 0;
};

// M2 (optional): `batch2` more matrices of the same size, swept in the same launch.
inline cudaError_t fine_sweep(FineState& state, double* M, long long mstride, int ld, int n_used, int batch, int* status, cudaStream_t stream, double* M2 = nullptr, long long mstride2 = 0,
                              int batch2 = 0) {
  cudaError_t e = cudaFuncSetAttribute(sweep_fine_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFineSmemBytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(sweep_fine_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFineSmemBytes);
  if (e != cudaSuccess) return e;
  const int nt = fine_tiles(n_used), t = nt - 1;
  int dev = 0, sms = 0;
  e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  FineSweep w{};
  w.M = M;
  w.mstride = mstride;
  w.M2 = M2;
  w.mstride2 = mstride2;
  w.split = batch;
  batch += batch2;
  w.ld = ld;
  w.nt = nt;
  w.last = (int)round_up(n_used - t * kSub, kGJPanel);
  w.batch = batch;
  w.control = reinterpret_cast<int*>(state.scratch);
  w.slots = state.scratch + kFineControlDoubles;
  w.pinv = w.slots + (size_t)batch * kFineSlots * 2 * nt * kFineTile;
  w.flags = reinterpret_cast<int*>(w.pinv + (size_t)batch * kFinePinv * kFineTile);
  w.status = status;
  const long long total = (long long)batch + (long long)batch * (t + t * (t + 1) / 2 - 1) * nt + batch;
  // flag values and queue counts stay far below 2^31; another shape, or a long run of sweeps, starts afresh
  const bool fresh = state.sweeps == 0 || state.nt != nt || state.batch != batch || state.sweeps > 4096 || state.queue > (1 << 30);
  if (fresh) {
    e = cudaMemsetAsync(w.control, 0, kFineControlDoubles * sizeof(double), stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(w.flags, 0, sizeof(int) * (size_t)batch * fine_flag_ints(nt), stream);
    if (e != cudaSuccess) return e;
    state.nt = nt;
    state.batch = batch;
    state.sweeps = 0;
    state.queue = 0;
  }
  w.sweep = state.sweeps;
  w.base = state.sweeps * nt;
  w.queue_base = state.queue;
  // One CTA per SM leaves the chain its SM (and twice the registers); two where a step has more units than four waves of
  // that.  Measured, us an inversion call (its loads and stores included), one / two per SM: N = 231, batch 32 (288 units a
  // step) 139 / 156, batch 64 (576) 205 / 188; N = 512, batch 16 (560) 306 / 306; N = 660, batch 8 (520) 370 / 375, batch 16
  // (1040) 650 / 519; N = 1984, batch 1 (495) 894 / 944, batch 2 (990) 1487 / 1150; N = 2610, batch 1 (860) 1779 / 1482.
  const bool dense = (long long)batch * (t + t * (t + 1) / 2) > 4LL * sms;
  const long long slots = dense ? 2LL * sms : sms;
  const int grid = (int)(total < slots ? total : slots);
  auto* kernel = dense ? sweep_fine_kernel<2> : sweep_fine_kernel<1>;
  note_launch();
  ++state.sweeps;
  state.queue += (int)total + grid;
  if (!fresh) return launch_overlapped(kernel, grid, kFineThreads, kFineSmemBytes, stream, w);
  kernel<<<grid, kFineThreads, kFineSmemBytes, stream>>>(w);  // behind the clearing of its flags
  return cudaGetLastError();
}

// The symmetric sweep on whichever path fits; n_used: the leading rows and columns that differ from the identity.
inline cudaError_t sweep_any(FineState& fine, double* M, long long mstride, int np, int batch, double* scratch, int* status, cudaStream_t stream, const int* reduced_blocks, int n_used, float* split) {
  if (fine.scratch != nullptr && reduced_blocks == nullptr) return fine_sweep(fine, M, mstride, np, n_used, batch, status, stream);
  return sweep_sym(M, mstride, np, batch, scratch, status, stream, reduced_blocks, n_used, split);
}

// Whether a batch of FP64 sweeps of n_used rows takes the 64-tile path: where its estimated time is below that of the
// 128-tile steps, both the larger of a latency (per step of the chain) and a throughput (per cubed tile count) term, in
// us.  (The chain's 28 us a link is a large matrix's, 23 at N = 660; it never decides, a 128-step costing four times as
// much.)  An odd tile count saves the steps' padding, so that up to nine tiles every batch comes here.
// Measured, us an inversion call (its loads and stores included), 128-tile steps / here: N = 192, batch 16 229 / 101, 128 321 / 199,
// 1000 2081 / 1302; N = 231, 16 232 / 120, 128 334 / 304, 200 534 / 460 (left to the steps); N = 320, 128 771 / 562, 1000
// 5315 / 4230; N = 396, 8 442 / 195, 64 766 / 616; N = 448, 1000 10722 / 9574; N = 512, 32 573 / 436, 64 809 / 871; N = 576,
// 128 2527 / 2411, 1000 18829 / 18847; N = 660, 4 649 / 286, 16 772 / 519, 64 2062 / 2035 (left); N = 1024, 8 977 / 700, 16
// 1327 / 1403; N = 1984, 1 1685 / 896, 2 1772 / 1148, 4 2330 / 2174 (left), 8 3744 / 4514; N = 2610, 1 2256 / 1482, 2 2468 /
// 2364 (left).
inline bool use_fine(int n_used, size_t batch) {
  const int nt = fine_tiles(n_used), steps = (n_used + kBlock - 1) / kBlock;
  if (steps < 2 || nt > kFineMaxTiles) return false;
  const double cubed = (double)nt * nt * nt * (double)batch, steps_cubed = (double)steps * steps * steps * (double)batch;
  return std::max(28.0 * nt, 0.0205 * cubed) < std::max(110.0 * steps, 0.125 * steps_cubed);
}

}  // namespace ticc
