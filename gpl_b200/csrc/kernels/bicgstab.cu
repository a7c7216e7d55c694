// The initial placement's solver (`bicgstab`, src/bicgstab.rs:615-669) on the device: CSR
// SpMV with each row summed in column order (the reference's `Csr::mul` order), float vectors,
// and the inner products and residual norms in double (deterministic partials). The whole loop
// is one persistent cooperative kernel (k_solve): the scalars (rho, alpha, omega) and the
// loop's tests (the residual bound, the iteration cap, the restart) stay on the device, the
// steps of an iteration are separated by barriers among the system's blocks, and the host
// reads the loop's state once per launch and runs a restart itself when the device asks for one.
#include "bicgstab.h"

#include <algorithm>
#include <cstring>

#include "common.cuh"

namespace gpl {

namespace {

enum Scal { S_RHO = 0, S_RHO_OLD, S_ALPHA, S_W, S_RR, S_R0R, S_R0SQ, S_BB, S_COUNT };
// The loop's state, after the three sums k_scalar's case 0 writes from S_R0SQ: the iteration
// count, the state (0 iterate, 1 waiting for a restart, 2 ended), and the bounds the tests
// compare with. Small integers, exact in double.
enum Loop { S_I = 10, S_STATE, S_TOL2, S_EPS2, S_MAXIT, S_END };
// The persistent loop's words (unsigned ints, each in a 128-byte line of its own past the
// scalars): the blocks' arrivals at its barriers, and whether a wait ran out.
constexpr int S_ARRIVE = 16, S_ERROR = 32;
constexpr double kIterate = 0.0, kRestart = 1.0, kEnded = 2.0;
// The loop's tests (`while rr > tol2 && i < max_iters`, then the restart test
// |rho| < eps^2 |r0|^2 at the head of the next iteration), in the reference's order.
__device__ __forceinline__ double loop_state(const double *S) {
  if (!(S[S_RR] > S[S_TOL2] && S[S_I] < S[S_MAXIT])) return kEnded;
  return fabs(S[S_RHO]) < S[S_EPS2] * S[S_R0SQ] ? kRestart : kIterate;
}

// y = A x, then `0 + 1 * tmp` as the library writes it, each row's products summed in
// column order (the reference's order). Three forms with the same results (SpmvForm):
//  rows:  a thread per row straight from memory;
//  tiled: a block's rows are contiguous in the CSR arrays, so the block first forms every
//         product vals[k] * x[cols[k]] of its rows with coalesced loads into shared memory
//         (eight entries per thread in flight), then each thread sums its row's products; a
//         block whose rows hold more than kSpmvTile entries sums straight from memory.
constexpr int kSpmvTile = 6144;
constexpr int kSpmvUnroll = 8;

__device__ __forceinline__ int64_t row_end(const int64_t *__restrict__ rs, const int64_t *__restrict__ cnt, int64_t i) { return cnt ? rs[i] + cnt[i] : rs[i + 1]; }

// Each form hands every row it forms to emit(row, value), at most one row per thread, and
// returns nowhere early, so a block-wide step may follow.
template <class Emit>
__device__ __forceinline__ void spmv_rows_rows(int64_t n, const int64_t *__restrict__ rs, const int32_t *__restrict__ cols, const float *__restrict__ vals, const float *__restrict__ x, Emit emit) {
  const int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x;
  if (i < n) {
    float tmp = 0.0f;
    const int64_t b = rs[i], e = rs[i + 1];
    for (int64_t k = b; k < e; k++) tmp = __fadd_rn(tmp, __fmul_rn(vals[k], x[cols[k]]));
    emit(i, __fadd_rn(0.0f, __fmul_rn(1.0f, tmp)));
  }
}
__global__ void __launch_bounds__(kThreads) k_spmv_rows(int64_t n, const int64_t *__restrict__ rs, const int32_t *__restrict__ cols, const float *__restrict__ vals, const float *__restrict__ x, float *__restrict__ y) {
  spmv_rows_rows(n, rs, cols, vals, x, [&](int64_t r, float v) { y[r] = v; });
}

template <class Emit>
__device__ __forceinline__ void spmv_tiled_rows(int64_t n, const int64_t *__restrict__ rs, const int32_t *__restrict__ cols, const float *__restrict__ vals, const float *__restrict__ x, Emit emit) {
  __shared__ float prod[kSpmvTile];
  const int64_t r0 = blockIdx.x * (int64_t)kThreads;
  const int64_t r1 = min(n, r0 + (int64_t)kThreads);
  const int64_t k0 = rs[r0], k1 = rs[r1];
  const int64_t i = r0 + threadIdx.x;
  int64_t b = 0, e = 0;
  if (i < n) {
    b = rs[i];
    e = rs[i + 1];
  }
  const bool tiled = k1 - k0 <= kSpmvTile;
  const bool inside = tiled && b >= k0 && e <= k1;  // not so where the starts do not ascend
  if (tiled) {
    const int cnt = (int)(k1 - k0);
    const int32_t *c = cols + k0;
    const float *v = vals + k0;
    for (int j = threadIdx.x; j < cnt; j += kSpmvUnroll * kThreads) {
      int cc[kSpmvUnroll];
      float vv[kSpmvUnroll], xv[kSpmvUnroll];
#pragma unroll
      for (int u = 0; u < kSpmvUnroll; u++) {
        int q = j + u * kThreads;
        cc[u] = q < cnt ? __ldg(c + q) : 0;
        vv[u] = q < cnt ? __ldg(v + q) : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < kSpmvUnroll; u++) xv[u] = j + u * kThreads < cnt ? __ldg(x + cc[u]) : 0.0f;
#pragma unroll
      for (int u = 0; u < kSpmvUnroll; u++) {
        int q = j + u * kThreads;
        if (q < cnt) prod[q] = __fmul_rn(vv[u], xv[u]);
      }
    }
  }
  __syncthreads();
  if (i < n) {
    float tmp = 0.0f;
    if (inside) {
      const int lb = (int)(b - k0), le = (int)(e - k0);
      for (int k = lb; k < le; k++) tmp = __fadd_rn(tmp, prod[k]);
    } else {
      for (int64_t k = b; k < e; k++) tmp = __fadd_rn(tmp, __fmul_rn(vals[k], x[cols[k]]));
    }
    emit(i, __fadd_rn(0.0f, __fmul_rn(1.0f, tmp)));
  }
}
__global__ void __launch_bounds__(kThreads) k_spmv_tiled(int64_t n, const int64_t *__restrict__ rs, const int32_t *__restrict__ cols, const float *__restrict__ vals, const float *__restrict__ x, float *__restrict__ y) {
  spmv_tiled_rows(n, rs, cols, vals, x, [&](int64_t r, float v) { y[r] = v; });
}

//  sliced: over the sliced copy (rows in order of length). The long rows first, a warp per
//         row (long_row). Then
//         a thread per short row: at step k a warp's rows read one coalesced run of entries
//         (the slice's column k), each row summed in column order and stopping at its own
//         length. y is written at the row's own index. Blocks [0, long_blocks) take the long
//         rows, kThreads / 32 rows each.
// A long row by a warp: the lanes form kLongChunk products at a time from the CSR arrays into
// buf (that many floats of the warp's own, 16-byte aligned), from where every lane adds them in
// column order, four a load; the next chunk's x and the entries of the one after are in flight
// meanwhile. The longest row bounds a product (a bound pin's cell ties to all its nets' pins:
// 2500 entries at 400k cells): adding through shuffles took 20 ns an entry, this 4.
constexpr int kLongPer = 4, kLongChunk = 32 * kLongPer;
template <class Load>
__device__ __forceinline__ float long_row(int64_t b, int64_t e, const int32_t *__restrict__ cols, const float *__restrict__ vals, float *buf, Load x) {
  const int lane = threadIdx.x & 31;
  int32_t c[kLongPer];
  float v[kLongPer], xv[kLongPer], vx[kLongPer];
  auto entries = [&](int64_t m) {
#pragma unroll
    for (int u = 0; u < kLongPer; u++) {
      const int64_t k = m + 32 * u + lane;
      c[u] = k < e ? __ldg(cols + k) : -1;
      v[u] = k < e ? __ldg(vals + k) : 0.0f;
    }
  };
  auto gather = [&]() {
#pragma unroll
    for (int u = 0; u < kLongPer; u++) {
      xv[u] = c[u] >= 0 ? x(c[u]) : 0.0f;
      vx[u] = v[u];
    }
  };
  entries(b);
  gather();
  entries(b + kLongChunk);
  float sum = 0.0f;
  for (int64_t m = b; m < e; m += kLongChunk) {
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kLongPer; u++) buf[32 * u + lane] = __fmul_rn(vx[u], xv[u]);
    __syncwarp();
    gather();
    entries(m + 2 * kLongChunk);
    const float4 *q = reinterpret_cast<const float4 *>(buf);
    if (e - m >= kLongChunk) {
#pragma unroll
      for (int t = 0; t < kLongChunk / 4; t++) {
        const float4 z = q[t];
        sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, z.x), z.y), z.z), z.w);
      }
    } else {
      const int cnt = (int)(e - m);
      int t = 0;
#pragma unroll 4
      for (; t + 4 <= cnt; t += 4) {
        const float4 z = q[t / 4];
        sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, z.x), z.y), z.z), z.w);
      }
      for (; t < cnt; t++) sum = __fadd_rn(sum, buf[t]);
    }
  }
  __syncwarp();
  return __fadd_rn(0.0f, __fmul_rn(1.0f, sum));
}
__host__ __device__ __forceinline__ int64_t sliced_long_blocks(int64_t n_long) { return (n_long + kThreads / 32 - 1) / (kThreads / 32); }
__host__ __device__ __forceinline__ int64_t sliced_blocks(int64_t n, int64_t n_long) { return sliced_long_blocks(n_long) + (n - n_long + kThreads - 1) / kThreads; }
template <class Emit>
__device__ __forceinline__ void spmv_sliced_rows(int64_t n, int64_t n_long, const int64_t *__restrict__ rs, const int64_t *__restrict__ cnt, const int32_t *__restrict__ cols, const float *__restrict__ vals, const int32_t *__restrict__ sl_row, const int32_t *__restrict__ sl_len, const int64_t *__restrict__ sl_start, const int2 *__restrict__ sl_ent, const float *__restrict__ x, Emit emit) {
  __shared__ __align__(16) float buf[kThreads / 32][kLongChunk];
  const int64_t lb = sliced_long_blocks(n_long);
  if (blockIdx.x < lb) {
    const int64_t w = blockIdx.x * (int64_t)(kThreads / 32) + (threadIdx.x >> 5);
    if (w >= n_long) return;  // the whole warp; such a warp forms no row
    const int32_t row = sl_row[w];
    const float v = long_row(rs[row], row_end(rs, cnt, row), cols, vals, buf[threadIdx.x >> 5], [&](int32_t c) { return __ldg(x + c); });
    if ((threadIdx.x & 31) == 0) emit(row, v);
    return;
  }
  const int64_t i = (blockIdx.x - lb) * (int64_t)kThreads + threadIdx.x;  // short position
  const int64_t j = n_long + i;
  if (j >= n) return;
  const int32_t len = sl_len[j];
  const int32_t row = sl_row[j];
  const int64_t base = sl_start[i / kSliceRows] + (i % kSliceRows);
  const int2 *ent = sl_ent + base;
  // kSpmvUnroll entries at a time, the last group's loads predicated, so every group costs
  // two dependent round trips (its entries, then their x) whatever the row's length; the
  // products still add in column order
  float tmp = 0.0f;
  for (int32_t k = 0; k < len; k += kSpmvUnroll) {
    int2 cv[kSpmvUnroll];
    float xv[kSpmvUnroll];
#pragma unroll
    for (int u = 0; u < kSpmvUnroll; u++) cv[u] = k + u < len ? __ldg(ent + (int64_t)(k + u) * kSliceRows) : make_int2(0, 0);
#pragma unroll
    for (int u = 0; u < kSpmvUnroll; u++) xv[u] = k + u < len ? __ldg(x + cv[u].x) : 0.0f;
#pragma unroll
    for (int u = 0; u < kSpmvUnroll; u++)
      if (k + u < len) tmp = __fadd_rn(tmp, __fmul_rn(__int_as_float(cv[u].y), xv[u]));
  }
  emit(row, __fadd_rn(0.0f, __fmul_rn(1.0f, tmp)));
}
__global__ void __launch_bounds__(kThreads) k_spmv_sliced(int64_t n, int64_t n_long, const int64_t *__restrict__ rs, const int64_t *__restrict__ cnt, const int32_t *__restrict__ cols, const float *__restrict__ vals, const int32_t *__restrict__ sl_row, const int32_t *__restrict__ sl_len, const int64_t *__restrict__ sl_start, const int2 *__restrict__ sl_ent, const float *__restrict__ x, float *__restrict__ y) {
  spmv_sliced_rows(n, n_long, rs, cnt, cols, vals, sl_row, sl_len, sl_start, sl_ent, x, [&](int64_t r, float v) { y[r] = v; });
}

// The order by length: a histogram of the (capped) lengths per block in shared memory, the
// buckets' starts longest first, then each row's position from its bucket's cursor (a warp's
// rows of one bucket take one atomic between them).
__global__ void __launch_bounds__(kThreads) k_len_hist(int64_t n, const int64_t *__restrict__ rs, const int64_t *__restrict__ cnt, int32_t *__restrict__ count) {
  __shared__ int32_t h[kSliceLenCap + 1];
  for (int b = threadIdx.x; b <= kSliceLenCap; b += kThreads) h[b] = 0;
  __syncthreads();
  const int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x;
  if (i < n) atomicAdd(&h[(int)min(row_end(rs, cnt, i) - rs[i], (int64_t)kSliceLenCap)], 1);
  __syncthreads();
  for (int b = threadIdx.x; b <= kSliceLenCap; b += kThreads)
    if (h[b]) atomicAdd(&count[b], h[b]);
}
// The counts to starts, longest first: one warp, each lane a run of classes (its loads in
// flight together), the runs' totals scanned across the warp.
constexpr int kLenPerLane = (kSliceLenCap + 1 + 31) / 32;
__global__ void k_len_starts(int32_t *count) {
  const int lane = threadIdx.x;
  int32_t c[kLenPerLane];
  int32_t sum = 0;
#pragma unroll
  for (int q = 0; q < kLenPerLane; q++) {
    const int b = kSliceLenCap - (lane * kLenPerLane + q);  // descending
    c[q] = b >= 0 ? count[b] : 0;
    sum += c[q];
  }
  int32_t run = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t y = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += y;
  }
  run -= sum;  // exclusive
#pragma unroll
  for (int q = 0; q < kLenPerLane; q++) {
    const int b = kSliceLenCap - (lane * kLenPerLane + q);
    if (b >= 0) count[b] = run;
    run += c[q];
  }
}
__global__ void __launch_bounds__(kThreads) k_len_scatter(int64_t n, const int64_t *__restrict__ rs, const int64_t *__restrict__ cnt, int32_t *__restrict__ cursor, int32_t *__restrict__ row, int32_t *__restrict__ len) {
  const int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x;
  const bool live = i < n;
  const int64_t l = live ? row_end(rs, cnt, i) - rs[i] : 0;
  const int b = live ? (int)min(l, (int64_t)kSliceLenCap) : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, b);
  const int leader = __ffs(peers) - 1, lane = threadIdx.x & 31;
  int32_t at = 0;
  if (live && lane == leader) at = atomicAdd(&cursor[b], __popc(peers));
  at = __shfl_sync(0xffffffffu, at, leader);
  if (!live) return;
  at += __popc(peers & ((1u << lane) - 1u));
  row[at] = (int32_t)i;
  len[at] = (int32_t)l;
}
// kSliceRows times each slice's longest row (a warp's short positions are one slice).
__global__ void __launch_bounds__(kThreads) k_slice_widths(int64_t n, int64_t n_long, const int32_t *__restrict__ len, int64_t *__restrict__ widths) {
  static_assert(kSliceRows == 32 && kThreads % 32 == 0, "a slice is a warp's rows");
  const int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x, ns = n - n_long;
  if (i - (threadIdx.x & 31) >= ns) return;  // the warp's slice starts past the end
  const unsigned l = i < ns ? (unsigned)len[n_long + i] : 0u;
  const unsigned m = __reduce_max_sync(0xffffffffu, l);
  if ((threadIdx.x & 31) == 0) widths[i / kSliceRows] = (int64_t)m * kSliceRows;
}
__global__ void __launch_bounds__(kThreads) k_slice_fill(int64_t n, int64_t n_long, const int64_t *__restrict__ rs, const int32_t *__restrict__ cols, const float *__restrict__ vals, const int32_t *__restrict__ sl_row, const int32_t *__restrict__ sl_len, const int64_t *__restrict__ sl_start, int2 *__restrict__ sl_ent) {
  const int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x, j = n_long + i;
  if (j >= n) return;
  const int64_t b = rs[sl_row[j]];
  const int32_t len = sl_len[j];
  const int64_t base = sl_start[i / kSliceRows] + (i % kSliceRows);
  for (int32_t k = 0; k < len; k++) sl_ent[base + (int64_t)k * kSliceRows] = make_int2(cols[b + k], __float_as_int(vals[b + k]));
}

static void spmv_launch(int form, cudaStream_t st, const CsrDev &A, const float *in, float *o) {
  if (A.n <= 0) return;
  const unsigned eb = (unsigned)((A.n + kThreads - 1) / kThreads);
  if (form == kSpmvSliced)
    k_spmv_sliced<<<(unsigned)std::max<int64_t>(sliced_blocks(A.n, A.sl_long), 1), kThreads, 0, st>>>(A.n, A.sl_long, A.rs, A.cnt, A.cols, A.vals, A.sl_row, A.sl_len, A.sl_start, A.sl_ent, in, o);
  else if (form == kSpmvTiled)
    k_spmv_tiled<<<eb, kThreads, 0, st>>>(A.n, A.rs, A.cols, A.vals, in, o);
  else
    k_spmv_rows<<<eb, kThreads, 0, st>>>(A.n, A.rs, A.cols, A.vals, in, o);
}

// ---- the start: residual and inner products, in launches of their own
// Up to three dot products at once; partials[blk * 3 + j].
__global__ void k_dots(int64_t n, const float *__restrict__ a0, const float *__restrict__ b0, const float *__restrict__ a1, const float *__restrict__ b1, const float *__restrict__ a2, const float *__restrict__ b2, double *__restrict__ part) {
  __shared__ double sh[kThreads / 32];
  double s0 = 0, s1 = 0, s2 = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    s0 += (double)a0[i] * (double)b0[i];
    if (a1) s1 += (double)a1[i] * (double)b1[i];
    if (a2) s2 += (double)a2[i] * (double)b2[i];
  }
  double t0 = block_sum<kThreads>(s0, sh);
  double t1 = block_sum<kThreads>(s1, sh);
  double t2 = block_sum<kThreads>(s2, sh);
  if (threadIdx.x == 0) {
    part[3 * blockIdx.x] = t0;
    part[3 * blockIdx.x + 1] = t1;
    part[3 * blockIdx.x + 2] = t2;
  }
}

// The partials' sums (the block's threads over the blocks' partials, in a fixed order):
//  which 0 (start): S[S_R0SQ..] = the three sums
//  which 4 (restart): S_R0SQ = S_RHO = S_RR = sum0
__global__ void k_scalar(const double *__restrict__ part, int nblk, double *__restrict__ S, int which) {
  __shared__ double sh[kThreads / 32];
  double v[3];
  for (int j = 0; j < 3; j++) {
    double s = 0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) s += part[3 * b + j];
    v[j] = block_sum<kThreads>(s, sh);
  }
  if (threadIdx.x != 0) return;
  if (which == 0) {
    S[S_R0SQ] = v[0];
    S[S_R0SQ + 1] = v[1];
    S[S_R0SQ + 2] = v[2];
  } else {
    S[S_R0SQ] = v[0];
    S[S_RHO] = v[0];
    S[S_RR] = v[0];
  }
}

// After a restart (which 4 above): the first one sets the iteration count back to zero.
__global__ void k_restart_done(double *S, int first) {
  if (first) S[S_I] = 0.0;
  S[S_STATE] = kIterate;
}

__global__ void k_loop_init(double *S, double tol2, double eps2, int max_iters) {
  S[S_RHO] = S[S_COUNT];  // dot(r0, r) of the start point
  S[S_RR] = S[S_R0SQ];
  S[S_RHO_OLD] = 1.0;
  S[S_ALPHA] = 1.0;
  S[S_W] = 1.0;
  S[S_I] = 0.0;
  S[S_TOL2] = tol2;
  S[S_EPS2] = eps2;
  S[S_MAXIT] = (double)max_iters;
  S[S_STATE] = loop_state(S);
}

__global__ void k_residual(int64_t n, const float *__restrict__ b, const float *__restrict__ ax, float *__restrict__ r, float *__restrict__ r0) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float v = __fsub_rn(b[i], ax[i]);
  r[i] = v;
  r0[i] = v;
}
__global__ void k_set_ended(double *S) { S[S_STATE] = kEnded; }
__global__ void k_fill(int64_t n, float *a, float v) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) a[i] = v;
}

// ---- the loop: one persistent cooperative kernel for one or two systems
//
// An iteration is seven steps that each need the whole of the one before: p, A p, r0.v, s,
// A s, (t.t, t.s), and x, r with their two inner products. As launches (seven an iteration,
// chained) they cost 65 us an iteration for two systems of 100k rows, most of it launch and
// drain latency; here each system's blocks stay resident and meet at barriers in global memory
// (1.4 us among 148 blocks), and every block takes the scalar steps itself from the partials
// instead of waiting for one to publish them. Measured, the initial placement's pair: 38 us an
// iteration at 100k rows (65 before), 107 us at 400k (165), 10 us at 300 (45); one system of
// 300k rows 81 us (310, a thread per row). What is left at 100k: two products of 11 us each,
// bound by their gathers of x, seven barriers, five vector steps of 1.2 to 2.3 us. Two blocks of
// 512 threads an SM (64 registers); the two systems' barriers are their own, so each takes exactly
// the steps it would take alone.
constexpr int kSolveThreads = 512;
// A block's products of the tiled form at once (40 KB); longer runs go in pieces.
constexpr int kSolveTile = 10240;
// Iterations a launch may run before the host looks at the loop's state again.
constexpr int kSolveBudget = 128;

struct SysDev {
  int64_t n;
  const int64_t *rs, *cnt;
  const int32_t *cols;
  const float *vals;
  int64_t sl_long;
  const int32_t *sl_row, *sl_len;
  const int64_t *sl_start;
  const int2 *sl_ent;
  float *x, *r, *r0, *v, *p, *s, *t;
  double *part, *S;
};
struct SysPair {
  SysDev a[2];
};

__device__ __forceinline__ unsigned int load_acquire(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// Waits until *p has reached `target` (counts that wrap); false once the wait has run out
// here or in another block.
__device__ __forceinline__ bool wait_for(const unsigned int *p, unsigned int target, unsigned int *err, unsigned long long limit) {
  unsigned long long t0 = 0;
  for (unsigned int k = 1;; k++) {
    if ((int)(load_acquire(p) - target) >= 0) return true;
    if ((k & 255u) == 0) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
      if (!t0) t0 = t;
      if (t - t0 > limit || load_acquire(err)) {
        atomicExch(err, 1u);
        return false;
      }
    }
  }
}

// The system's blocks meeting: what any of them wrote before is visible to all after (one
// thread's release of the block's writes, its acquire of everyone's; the block's other threads
// through the block barriers). About 1.5 us among 148 blocks; nothing but the block barrier in
// a system of one block. False once a wait has run out.
struct Meet {
  unsigned int *arrive, *err;
  unsigned int blocks;   // the system's blocks
  unsigned int gen;      // barriers passed since the launch
  unsigned long long limit;  // a wait gives up after this many ns (a block of the system is gone)
};
__device__ __forceinline__ bool meet(Meet &m) {
  if (m.blocks == 1) {
    __syncthreads();
    return true;
  }
  bool good = true;
  m.gen++;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(m.arrive) : "memory");
    good = wait_for(m.arrive, m.gen * m.blocks, m.err, m.limit);
  }
  return __syncthreads_and(good);
}

// Two sums, each of 256 threads' values (a half of the block), in block_sum's order, in each
// half's thread 0. sh: 32 doubles, not used again before the next block barrier.
__device__ __forceinline__ void half_sums(double &a, double &b, double *sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = a, sh[16 + w] = b;
  __syncthreads();
  if ((w & 7) == 0) {
    a = l < 8 ? sh[w + l] : 0.0;
    b = l < 8 ? sh[16 + w + l] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, o);
      b += __shfl_down_sync(0xffffffffu, b, o);
    }
  }
}

// The scalars: thread 0 of every block holds them all and takes every scalar step itself from
// the partials (the same sums in the same order in each block), the steps' factors as floats
// in shared memory.
struct Scalars {
  double rho, rho_old, alpha, w, rr, i;
};
struct Factors {
  float alpha, w, beta;
  int live;  // the loop goes on
};
__device__ __forceinline__ float beta_of(const Scalars &s) { return (float)((s.rho / s.rho_old) * (s.alpha / s.w)); }

// Columns [col, col + 2) of the partials summed (`live` parts of 256 threads; the others'
// partials are zero), after a barrier; in thread 0.
__device__ __forceinline__ void sum_parts(const double *part, int col, int live, double *sh, double &s0, double &s1) {
  s0 = s1 = 0;
  if (threadIdx.x < kThreads)
    for (int b = threadIdx.x; b < live; b += kThreads) {
      s0 += __ldcg(part + kBicgParts * b + col);
      s1 += __ldcg(part + kBicgParts * b + col + 1);
    }
  half_sums(s0, s1, sh);
}

__device__ __forceinline__ bool aligned16(const void *a, const void *b) { return (((uintptr_t)a | (uintptr_t)b) & 15) == 0; }
__device__ __forceinline__ double dot4(float4 a, float4 b, double s) {
  s += (double)a.x * (double)b.x;
  s += (double)a.y * (double)b.y;
  s += (double)a.z * (double)b.z;
  s += (double)a.w * (double)b.w;
  return s;
}
// How many of the kBicgBlocks blocks of 256 threads have a term of an inner product: their
// threads take runs of four (n4 of them, then the tail one element a thread), or, off 16-byte
// boundaries, one element each.
__device__ __forceinline__ int live_parts(int64_t n, int64_t n4) {
  const int64_t a = (n4 + kThreads - 1) / kThreads, b = (n - 4 * n4 + kThreads - 1) / kThreads;
  return (int)min((int64_t)kBicgBlocks, max(max(a, b), (int64_t)1));
}
constexpr int64_t kPartStride = (int64_t)kBicgBlocks * kThreads;

// The loop's two inner-product steps: TWO 0 is a.b (r0.v), TWO 1 is a.a and a.b (t.t and t.s).
// The sums are those of kBicgBlocks blocks of 256 threads, each thread over runs of four
// elements in index order; a block here takes one such block a half (parts c and blocks + c),
// so the partials and their order do not depend on the launch's shape.
template <int TWO>
__device__ __forceinline__ int loop_dots(int64_t n, const float *a, const float *b, double *part, int col, int c, int blocks, double *sh) {
  const int h = threadIdx.x / kThreads, t = threadIdx.x % kThreads;
  const int64_t n4 = aligned16(a, b) ? n / 4 : 0;
  const int live = live_parts(n, n4);
  for (int base = 0; base < live; base += 2 * blocks) {
    const int vb = base + h * blocks + c;
    double s0 = 0, s1 = 0;
    if (vb < live) {
      const int64_t tid = (int64_t)vb * kThreads + t;
      const float4 *A = (const float4 *)a, *B = (const float4 *)b;
      for (int64_t i = tid; i < n4; i += 2 * kPartStride) {
        const int64_t j = i + kPartStride;
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 x0 = A[i], y0 = B[i], x1 = j < n4 ? A[j] : z, y1 = j < n4 ? B[j] : z;
        if (TWO) s0 = dot4(x0, x0, s0);
        (TWO ? s1 : s0) = dot4(x0, y0, TWO ? s1 : s0);
        if (j < n4) {
          if (TWO) s0 = dot4(x1, x1, s0);
          (TWO ? s1 : s0) = dot4(x1, y1, TWO ? s1 : s0);
        }
      }
      for (int64_t i = 4 * n4 + tid; i < n; i += kPartStride) {
        if (TWO) {
          s0 += (double)a[i] * (double)a[i];
          s1 += (double)a[i] * (double)b[i];
        } else {
          s0 += (double)a[i] * (double)b[i];
        }
      }
    }
    if (base) __syncthreads();  // the sums' shared words again
    half_sums(s0, s1, sh);
    if (t == 0 && vb < live) {
      part[kBicgParts * vb + col] = s0;
      part[kBicgParts * vb + col + 1] = s1;
    }
  }
  return live;
}

// x += alpha p + w s; r = s - w t; partials of |r|^2 and r0.r, in the same parts.
__device__ __forceinline__ int update_xr(const SysDev &q, float al, float w, int col, int c, int blocks, double *sh) {
  const int h = threadIdx.x / kThreads, t = threadIdx.x % kThreads;
  auto fx = [&](float xi, float pi, float si) { return __fadd_rn(xi, __fadd_rn(__fmul_rn(al, pi), __fmul_rn(w, si))); };
  auto fr = [&](float si, float ti) { return __fsub_rn(si, __fmul_rn(w, ti)); };
  const int64_t n4 = aligned16(q.x, q.r) ? q.n / 4 : 0;  // the scratch's vectors lie alike
  const int live = live_parts(q.n, n4);
  for (int base = 0; base < live; base += 2 * blocks) {
    const int vb = base + h * blocks + c;
    double rr = 0, r0r = 0;
    if (vb < live) {
      const int64_t tid = (int64_t)vb * kThreads + t;
      for (int64_t k = tid; k < n4; k += kPartStride) {
        const float4 X = ((const float4 *)q.x)[k], P = ((const float4 *)q.p)[k], Sv = ((const float4 *)q.s)[k], T = ((const float4 *)q.t)[k], R0 = ((const float4 *)q.r0)[k];
        ((float4 *)q.x)[k] = make_float4(fx(X.x, P.x, Sv.x), fx(X.y, P.y, Sv.y), fx(X.z, P.z, Sv.z), fx(X.w, P.w, Sv.w));
        const float4 R = make_float4(fr(Sv.x, T.x), fr(Sv.y, T.y), fr(Sv.z, T.z), fr(Sv.w, T.w));
        ((float4 *)q.r)[k] = R;
        rr = dot4(R, R, rr);
        r0r = dot4(R0, R, r0r);
      }
      for (int64_t i = 4 * n4 + tid; i < q.n; i += kPartStride) {
        q.x[i] = fx(q.x[i], q.p[i], q.s[i]);
        const float rv = fr(q.s[i], q.t[i]);
        q.r[i] = rv;
        rr += (double)rv * (double)rv;
        r0r += (double)q.r0[i] * (double)rv;
      }
    }
    if (base) __syncthreads();  // the sums' shared words again
    half_sums(rr, r0r, sh);
    if (t == 0 && vb < live) {
      q.part[kBicgParts * vb + col] = rr;
      q.part[kBicgParts * vb + col + 1] = r0r;
    }
  }
  return live;
}

// out[i] = f(i, a run of four or one element) over the system's threads.
template <class F>
__device__ __forceinline__ void each4(int64_t n, bool aligned, int c, int blocks, F f) {
  const int64_t tid = (int64_t)c * kSolveThreads + threadIdx.x, stride = (int64_t)blocks * kSolveThreads;
  const int64_t n4 = aligned ? n / 4 : 0;
  for (int64_t i = tid; i < n4; i += stride) f(4 * i, true);
  for (int64_t i = 4 * n4 + tid; i < n; i += stride) f(i, false);
}

// The sliced form's items taken in the block so far; a product's first is left_base, the fetches
// of the ones before it (a barrier apart).
struct Left {
  int taken;
};

// y = A x over the system's blocks, each row's products summed in column order (the forms of
// SpmvForm, bit for bit the same y). x and y are written in this kernel: plain loads.
//  rows:   a thread per row straight from memory;
//  tiled:  a block's run of rows, its entries' products formed by all its threads into shared
//          memory (coalesced, eight gathers a thread in flight), then a thread per row;
//  sliced: a warp per long row, then per slice of 32 rows. The gathers bound it: 0.8 a cycle
//          and SM at 400k rows, near the one L1 looks up a cycle (the same loads without them
//          took a third of the time).
template <int FORM>
__device__ __forceinline__ void solve_spmv(const SysDev &q, const float *x, float *y, int c, int blocks, float *prod, Left &left, int &left_base) {
  const int64_t n = q.n;
  if (FORM == kSpmvRows) {
    for (int64_t i = (int64_t)c * kSolveThreads + threadIdx.x; i < n; i += (int64_t)blocks * kSolveThreads) {
      float tmp = 0.0f;
      const int64_t b = __ldg(q.rs + i), e = __ldg(q.rs + i + 1);
      for (int64_t k = b; k < e; k++) tmp = __fadd_rn(tmp, __fmul_rn(__ldg(q.vals + k), x[__ldg(q.cols + k)]));
      y[i] = __fadd_rn(0.0f, __fmul_rn(1.0f, tmp));
    }
  } else if (FORM == kSpmvTiled) {
    // runs of at most kSolveThreads rows, as many a block as fill them evenly
    const int64_t per = (n + (int64_t)blocks * kSolveThreads - 1) / ((int64_t)blocks * kSolveThreads);
    const int64_t run = min((int64_t)kSolveThreads, ((n + blocks * per - 1) / (blocks * per) + 31) / 32 * 32);
    for (int64_t r0 = c * run; r0 < n; r0 += blocks * run) {
      const int64_t r1 = min(n, r0 + run), i = r0 + threadIdx.x;
      const int64_t k0 = __ldg(q.rs + r0), k1 = __ldg(q.rs + r1);
      int64_t at = 0, e = 0;
      if (i < r1) {
        at = __ldg(q.rs + i);
        e = __ldg(q.rs + i + 1);
      }
      float tmp = 0.0f;
      if (at < k0 || e > k1) {  // starts that do not ascend: the row is no part of the run
        for (int64_t k = at; k < e; k++) tmp = __fadd_rn(tmp, __fmul_rn(__ldg(q.vals + k), x[__ldg(q.cols + k)]));
        at = e = k1;
      }
      for (int64_t m0 = k0; m0 < k1; m0 += kSolveTile) {
        const int cnt = (int)min((int64_t)kSolveTile, k1 - m0);
        const int32_t *cc = q.cols + m0;
        const float *vv = q.vals + m0;
        for (int j = threadIdx.x; j < cnt; j += kSpmvUnroll * kSolveThreads) {
          int ci[kSpmvUnroll];
          float va[kSpmvUnroll], xv[kSpmvUnroll];
#pragma unroll
          for (int u = 0; u < kSpmvUnroll; u++) {
            const int w = j + u * kSolveThreads;
            ci[u] = w < cnt ? __ldg(cc + w) : 0;
            va[u] = w < cnt ? __ldg(vv + w) : 0.0f;
          }
#pragma unroll
          for (int u = 0; u < kSpmvUnroll; u++) xv[u] = j + u * kSolveThreads < cnt ? x[ci[u]] : 0.0f;
#pragma unroll
          for (int u = 0; u < kSpmvUnroll; u++) {
            const int w = j + u * kSolveThreads;
            if (w < cnt) prod[w] = __fmul_rn(va[u], xv[u]);
          }
        }
        __syncthreads();
        const int64_t m1 = m0 + cnt;
        const int lb = (int)(min(at, m1) - m0), le = (int)(min(e, m1) - m0);
        int k = lb;
        if (le - lb >= 4 * kSpmvUnroll) {
          // a long row: 16-byte loads, the next eight products beside the eight dependent adds
          for (; k & 3; k++) tmp = __fadd_rn(tmp, prod[k]);
          const float4 *p4 = reinterpret_cast<const float4 *>(prod + k);
          float4 c0 = p4[0], c1 = p4[1];
          for (; k + 16 <= le; k += 8) {
            p4 += 2;
            const float4 n0 = p4[0], n1 = p4[1];
            tmp = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(tmp, c0.x), c0.y), c0.z), c0.w);
            tmp = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(tmp, c1.x), c1.y), c1.z), c1.w);
            c0 = n0;
            c1 = n1;
          }
          tmp = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(tmp, c0.x), c0.y), c0.z), c0.w);
          tmp = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(tmp, c1.x), c1.y), c1.z), c1.w);
          k += 8;
        }
        for (; k < le; k++) tmp = __fadd_rn(tmp, prod[k]);
        if (le > lb) at = m0 + le;
        __syncthreads();
      }
      if (i < r1) y[i] = __fadd_rn(0.0f, __fmul_rn(1.0f, tmp));
    }
  } else {
    const int lane = threadIdx.x & 31, warps = kSolveThreads / 32;
    const int64_t ns = (n - q.sl_long + kSliceRows - 1) / kSliceRows, items = q.sl_long + ns;
    // the block's items are c, c + blocks, ...: neighbours lie on different blocks, so the
    // longest rows spread over the SMs. With more of them than warps each warp takes the next
    // one left when it is done: a fetch an item and one a warp past the end. 400k rows, two
    // systems, an iteration: 149 us with fixed items and shuffled sums, 130 with the long rows'
    // sums from shared memory, 107 with items taken too (112 to 117 taken one ahead, with or
    // without the next one's loads in flight); 100k: 38 for all.
    const int mine = (int)((items - c + blocks - 1) / blocks);
    const bool shared = mine > warps;
    int it = threadIdx.x >> 5;
    auto next = [&](int now) {
      if (!shared) return now + warps;
      int z = 0;
      if (lane == 0) z = atomicAdd(&left.taken, 1);
      return __shfl_sync(0xffffffffu, z, 0) - left_base;
    };
    if (shared) it = next(it);
    for (; it >= 0 && it < mine; it = next(it)) {
      const int64_t w = (int64_t)it * blocks + c;
      if (w < q.sl_long) {
        const int32_t row = __ldg(q.sl_row + w);
        const float v = long_row(__ldg(q.rs + row), row_end(q.rs, q.cnt, row), q.cols, q.vals, prod + (threadIdx.x >> 5) * kLongChunk, [&](int32_t i) { return x[i]; });
        if (lane == 0) y[row] = v;
      } else {
        const int64_t slice = w - q.sl_long, j = q.sl_long + slice * kSliceRows + lane;
        const bool has = j < n;
        const int32_t len = has ? __ldg(q.sl_len + j) : 0, row = has ? __ldg(q.sl_row + j) : 0;
        const int2 *e = q.sl_ent + __ldg(q.sl_start + slice) + lane;
        float tmp = 0.0f;
        for (int32_t k = 0; k < len; k += kSpmvUnroll) {
          int2 cv[kSpmvUnroll];
          float xv[kSpmvUnroll];
#pragma unroll
          for (int u = 0; u < kSpmvUnroll; u++) cv[u] = k + u < len ? __ldg(e + (int64_t)(k + u) * kSliceRows) : make_int2(0, 0);
#pragma unroll
          for (int u = 0; u < kSpmvUnroll; u++) xv[u] = k + u < len ? x[cv[u].x] : 0.0f;
#pragma unroll
          for (int u = 0; u < kSpmvUnroll; u++)
            if (k + u < len) tmp = __fadd_rn(tmp, __fmul_rn(__int_as_float(cv[u].y), xv[u]));
        }
        if (has) y[row] = __fadd_rn(0.0f, __fmul_rn(1.0f, tmp));
      }
      __syncwarp();
    }
    if (shared) left_base += mine + warps;
  }
}

// blocks: a system's blocks; block b belongs to system b % nsys (with an even count of SMs and
// two blocks an SM, both of an SM's are one system's, so they share its vectors in L1).
template <int FORM>
__global__ void __launch_bounds__(kSolveThreads, 2) k_solve(SysPair P, int nsys, int blocks, SolveWait wait) {
  __shared__ double shp[32], shs[32];  // the partials' sums, the scalar steps' sums
  __shared__ __align__(16) float prod[FORM == kSpmvTiled ? kSolveTile : FORM == kSpmvSliced ? kSolveThreads / 32 * kLongChunk : 4];
  __shared__ Factors f;
  __shared__ Left left;
  int left_base = 0;
  if (threadIdx.x == 0) left.taken = 0;
  const int sys = (int)(blockIdx.x % nsys), c = (int)(blockIdx.x / nsys);
  const SysDev q = sys ? P.a[1] : P.a[0];
  const int64_t n = q.n;
  double *S = q.S;
  Meet m{reinterpret_cast<unsigned int *>(S + S_ARRIVE), reinterpret_cast<unsigned int *>(S + S_ERROR), (unsigned int)blocks, 0u, wait.ns + wait.entry_ns * (unsigned long long)q.rs[n]};
  const bool al = aligned16(q.r, q.r);
  Scalars k{};
  double s0, s1;
  if (threadIdx.x == 0) {
    k = Scalars{S[S_RHO], S[S_RHO_OLD], S[S_ALPHA], S[S_W], S[S_RR], S[S_I]};
    f.live = S[S_STATE] == kIterate;
    f.beta = beta_of(k);
    f.w = (float)k.w;
  }
  const double tol2 = S[S_TOL2], eps2r = S[S_EPS2] * S[S_R0SQ], maxit = S[S_MAXIT];
  double state = S[S_STATE];  // thread 0's follows the loop
  __syncthreads();
  if (!f.live) return;
  for (int it = 0; it < kSolveBudget && f.live; it++) {
    // p = r + beta (p - w v), beta = (rho / rho_old) (alpha / w)
    {
      const float beta = f.beta, w = f.w;
      auto g = [&](float ri, float pi, float vi) { return __fadd_rn(ri, __fmul_rn(beta, __fsub_rn(pi, __fmul_rn(w, vi)))); };
      each4(n, al, c, blocks, [&](int64_t i, bool four) {
        if (four) {
          const float4 R = *(const float4 *)(q.r + i), V = *(const float4 *)(q.v + i), Pv = *(const float4 *)(q.p + i);
          *(float4 *)(q.p + i) = make_float4(g(R.x, Pv.x, V.x), g(R.y, Pv.y, V.y), g(R.z, Pv.z, V.z), g(R.w, Pv.w, V.w));
        } else {
          q.p[i] = g(q.r[i], q.p[i], q.v[i]);
        }
      });
    }
    if (!meet(m)) return;
    solve_spmv<FORM>(q, q.p, q.v, c, blocks, prod, left, left_base);
    if (!meet(m)) return;
    int live = loop_dots<0>(n, q.r0, q.v, q.part, 0, c, blocks, shp);
    if (!meet(m)) return;
    sum_parts(q.part, 0, live, shs, s0, s1);
    if (threadIdx.x == 0) {
      k.alpha = k.rho / s0;
      f.alpha = (float)k.alpha;
    }
    __syncthreads();
    const float alpha = f.alpha;
    // s = r - alpha v
    {
      auto g = [&](float ri, float vi) { return __fsub_rn(ri, __fmul_rn(alpha, vi)); };
      each4(n, al, c, blocks, [&](int64_t i, bool four) {
        if (four) {
          const float4 R = *(const float4 *)(q.r + i), V = *(const float4 *)(q.v + i);
          *(float4 *)(q.s + i) = make_float4(g(R.x, V.x), g(R.y, V.y), g(R.z, V.z), g(R.w, V.w));
        } else {
          q.s[i] = g(q.r[i], q.v[i]);
        }
      });
    }
    if (!meet(m)) return;
    solve_spmv<FORM>(q, q.s, q.t, c, blocks, prod, left, left_base);
    if (!meet(m)) return;
    live = loop_dots<1>(n, q.t, q.s, q.part, 0, c, blocks, shp);
    if (!meet(m)) return;
    sum_parts(q.part, 0, live, shs, s0, s1);
    if (threadIdx.x == 0) {
      k.w = s0 > 0.0 ? s1 / s0 : 0.0;
      f.w = (float)k.w;
    }
    __syncthreads();
    // the third pair's columns are its own: a block may still read the second's
    live = update_xr(q, alpha, f.w, 2, c, blocks, shp);
    if (!meet(m)) return;
    sum_parts(q.part, 2, live, shs, s0, s1);
    if (threadIdx.x == 0) {
      // the iteration's end and the loop's tests (`while rr > tol2 && i < max_iters`, then the
      // restart test |rho| < eps^2 |r0|^2 at the head of the next iteration), in that order
      k.rr = s0;
      k.rho_old = k.rho;
      k.rho = s1;
      k.i += 1.0;
      state = !(k.rr > tol2 && k.i < maxit) ? kEnded : fabs(k.rho) < eps2r ? kRestart : kIterate;
      f.live = state == kIterate;
      f.beta = beta_of(k);
    }
    __syncthreads();
  }
  if (c == 0 && threadIdx.x == 0) {
    S[S_RHO] = k.rho;
    S[S_RHO_OLD] = k.rho_old;
    S[S_ALPHA] = k.alpha;
    S[S_W] = k.w;
    S[S_RR] = k.rr;
    S[S_I] = k.i;
    S[S_STATE] = state;
  }
}

}  // namespace

size_t bicgstab_scratch_bytes(int64_t n) {
  size_t vec = (size_t)n * sizeof(float);
  vec = (vec + 255) / 256 * 256;
  return 7 * vec + (size_t)kBicgBlocks * kBicgParts * sizeof(double) + 64 * sizeof(double);
}

size_t bicgstab_pair_scratch_bytes(int64_t n) { return bicgstab_scratch_bytes(n); }

cudaError_t csr_slice_order(const CsrDev &A, int32_t *row, int32_t *len, int32_t *count, cudaStream_t st) {
  if (A.n <= 0) return cudaSuccess;
  const unsigned g = (unsigned)((A.n + kThreads - 1) / kThreads);
  cudaError_t e = cudaMemsetAsync(count, 0, (kSliceLenCap + 1) * sizeof(int32_t), st);
  if (e != cudaSuccess) return e;
  k_len_hist<<<g, kThreads, 0, st>>>(A.n, A.rs, A.cnt, count);
  k_len_starts<<<1, 32, 0, st>>>(count);
  k_len_scatter<<<g, kThreads, 0, st>>>(A.n, A.rs, A.cnt, count, row, len);
  return cudaGetLastError();
}

cudaError_t csr_slice_widths(int64_t n, int64_t n_long, const int32_t *len, int64_t *widths, cudaStream_t st) {
  if (n - n_long <= 0) return cudaSuccess;
  k_slice_widths<<<(unsigned)((n - n_long + kThreads - 1) / kThreads), kThreads, 0, st>>>(n, n_long, len, widths);
  return cudaGetLastError();
}

cudaError_t csr_slice_fill(const CsrDev &A, int2 *sl_ent, cudaStream_t st) {
  if (A.n - A.sl_long <= 0) return cudaSuccess;
  k_slice_fill<<<(unsigned)((A.n - A.sl_long + kThreads - 1) / kThreads), kThreads, 0, st>>>(A.n, A.sl_long, A.rs, A.cols, A.vals, A.sl_row, A.sl_len, A.sl_start, sl_ent);
  return cudaGetLastError();
}

cudaError_t spmv(const CsrDev &A, const float *x, float *y, int form, cudaStream_t st) {
  if (form != kSpmvRows && form != kSpmvTiled && form != kSpmvSliced) return cudaErrorInvalidValue;
  if (form == kSpmvSliced ? !A.sl_start || !A.sl_row || !A.sl_len : A.cnt != nullptr) return cudaErrorInvalidValue;
  if (A.n <= 0) return cudaSuccess;
  spmv_launch(form, st, A, x, y);
  return cudaGetLastError();
}

// One launch of the loop: its blocks are all resident at once (a cooperative launch), at most
// two an SM. A system of up to kSolveThreads rows runs in one block, where a barrier is the
// block's own (300 rows: 10 us an iteration against 17 in three blocks). Beyond that the
// tiled form, whose threads share a run's entries, takes a block for every 128 rows (3000 rows:
// 19.5 us against 22.4 with 512), the others a thread per row (10k rows, sliced, two systems:
// 24 us against 25 with 128).
static cudaError_t solve_launch(int form, SysPair P, int nsys, SolveWait wait, cudaStream_t st) {
  const void *fn = form == kSpmvSliced ? (const void *)k_solve<kSpmvSliced> : form == kSpmvTiled ? (const void *)k_solve<kSpmvTiled> : (const void *)k_solve<kSpmvRows>;
  int dev = 0, sms = 0, per = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, kSolveThreads, 0);
  if (e != cudaSuccess) return e;
  const int most = std::max(1, sms * std::min(per, 2) / nsys);
  const int64_t rows = form == kSpmvTiled && P.a[0].n > kSolveThreads ? kSolveThreads / 4 : kSolveThreads;
  int blocks = (int)std::min<int64_t>(most, std::max<int64_t>(1, (P.a[0].n + rows - 1) / rows));
  for (int a = 0; a < nsys; a++)
    if ((e = cudaMemsetAsync(P.a[a].S + S_ARRIVE, 0, (64 - S_ARRIVE) * sizeof(double), st)) != cudaSuccess) return e;
  void *args[] = {&P, &nsys, &blocks, &wait};
  return cudaLaunchCooperativeKernel(fn, dim3((unsigned)(blocks * nsys)), dim3(kSolveThreads), args, 0, st);
}

// One or two systems of the same size, each with its own scalars and state.
static cudaError_t solve_systems(int nsys, const CsrDev *A, const float *const *b, float *const *x, int max_iters, void *const *scratch, cudaStream_t st, BicgResult *out, int form, SolveWait wait) {
  static_assert(S_END <= S_ARRIVE && S_ERROR < 64, "the scalars fit the scratch's 64 doubles");
  const int64_t n = A[0].n;
  const size_t vec = ((size_t)n * sizeof(float) + 255) / 256 * 256;
  SysPair P{};
  for (int a = 0; a < nsys; a++) {
    if (A[a].n != n) return cudaErrorInvalidValue;
    if (form == kSpmvSliced ? !A[a].sl_start || !A[a].sl_row || !A[a].sl_len : A[a].cnt != nullptr) return cudaErrorInvalidValue;
    char *base = (char *)scratch[a];
    SysDev &q = P.a[a];
    q.n = n;
    q.rs = A[a].rs;
    q.cnt = A[a].cnt;
    q.cols = A[a].cols;
    q.vals = A[a].vals;
    q.sl_long = A[a].sl_long;
    q.sl_row = A[a].sl_row;
    q.sl_len = A[a].sl_len;
    q.sl_start = A[a].sl_start;
    q.sl_ent = A[a].sl_ent;
    q.x = x[a];
    q.r = (float *)base;
    q.r0 = (float *)(base + vec);
    q.v = (float *)(base + 2 * vec);
    q.p = (float *)(base + 3 * vec);
    q.s = (float *)(base + 4 * vec);
    q.t = (float *)(base + 5 * vec);
    q.part = (double *)(base + 7 * vec);
    q.S = q.part + (size_t)kBicgBlocks * kBicgParts;
  }
  auto ax_of = [&](int a) { return (float *)((char *)scratch[a] + 6 * vec); };
  const int eb = (int)std::max<int64_t>((n + kThreads - 1) / kThreads, 1);
  const int rb = kBicgBlocks;
  const float tol = 1.1920929e-07f;
  double hs[2][64];
  auto pull = [&]() -> cudaError_t {
    for (int a = 0; a < nsys; a++) {
      cudaError_t e = cudaMemcpyAsync(hs[a], P.a[a].S, sizeof hs[a], cudaMemcpyDeviceToHost, st);
      if (e != cudaSuccess) return e;
    }
    return cudaStreamSynchronize(st);
  };
  cudaError_t e;
  for (int a = 0; a < nsys; a++) {
    const SysDev &q = P.a[a];
    spmv_launch(form, st, A[a], q.x, ax_of(a));
    k_residual<<<eb, kThreads, 0, st>>>(n, b[a], ax_of(a), q.r, q.r0);
    k_dots<<<rb, kThreads, 0, st>>>(n, q.r0, q.r0, b[a], b[a], q.r0, q.r, q.part);
    k_scalar<<<1, kThreads, 0, st>>>(q.part, rb, q.S, 0);  // S_R0SQ, S_BB, then dot(r0, r) in S[S_COUNT]
  }
  if ((e = pull()) != cudaSuccess) return e;
  double rhs_sqnorm[2];
  bool live[2] = {false, false};
  for (int a = 0; a < nsys; a++) {
    const SysDev &q = P.a[a];
    rhs_sqnorm[a] = hs[a][S_BB];
    live[a] = rhs_sqnorm[a] != 0.0;
    if (!live[a]) {
      k_fill<<<eb, kThreads, 0, st>>>(n, q.x, 0.0f);
      k_set_ended<<<1, 1, 0, st>>>(q.S);
      out[a].iterations = max_iters;
      out[a].error = tol;
      out[a].converged = true;
      continue;
    }
    if ((e = cudaMemsetAsync(q.v, 0, (size_t)n * sizeof(float), st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(q.p, 0, (size_t)n * sizeof(float), st)) != cudaSuccess) return e;
    double tol2 = (double)tol * (double)tol * rhs_sqnorm[a];
    double eps2 = (double)tol * (double)tol;
    k_loop_init<<<1, 1, 0, st>>>(q.S, tol2, eps2, max_iters);
  }
  if (!live[0] && !live[1]) return cudaGetLastError();
  // Every iteration counts one and only the first restart sets the count back, so a system
  // ends within 2 max_iters + 1 iterations; a launch whose systems wait for a restart holds
  // until the host has run it, and every launch but the last runs at least one iteration.
  const int64_t max_launches = 2 * (2 * (int64_t)max_iters + 3);
  int64_t n_launches = 0;
  int restarts[2] = {0, 0};
  for (;;) {
    if ((e = solve_launch(form, P, nsys, wait, st)) != cudaSuccess) return e;
    if ((e = pull()) != cudaSuccess) return e;
    bool ended = true;
    for (int a = 0; a < nsys; a++) {
      // a barrier's wait ran out: the word's bits, since as a double it is a denormal, which a
      // thread that takes those for zero would not tell from one
      unsigned int timed_out;
      std::memcpy(&timed_out, &hs[a][S_ERROR], sizeof timed_out);
      if (timed_out) return cudaErrorLaunchTimeout;
      ended = ended && hs[a][S_STATE] == kEnded;
    }
    if (ended) break;
    if (++n_launches > max_launches) return cudaErrorUnknown;  // cannot happen: the count above
    for (int a = 0; a < nsys; a++) {
      if (hs[a][S_STATE] != kRestart) continue;
      // too orthogonal to r0: restart from the current residual (that system alone)
      const SysDev &q = P.a[a];
      spmv_launch(form, st, A[a], q.x, ax_of(a));
      k_residual<<<eb, kThreads, 0, st>>>(n, b[a], ax_of(a), q.r, q.r0);
      k_dots<<<rb, kThreads, 0, st>>>(n, q.r, q.r, nullptr, nullptr, nullptr, nullptr, q.part);
      k_scalar<<<1, kThreads, 0, st>>>(q.part, rb, q.S, 4);
      k_restart_done<<<1, 1, 0, st>>>(q.S, restarts[a] == 0 ? 1 : 0);
      restarts[a]++;
    }
  }
  for (int a = 0; a < nsys; a++) {
    if (!live[a]) continue;
    out[a].iterations = (int)hs[a][S_I];
    out[a].error = (float)std::sqrt(hs[a][S_RR] / rhs_sqnorm[a]);
    out[a].converged = out[a].error <= tol;
  }
  return cudaGetLastError();
}

cudaError_t bicgstab_solve(const CsrDev &A, const float *b, float *x, int max_iters, void *scratch, cudaStream_t st, BicgResult *out, SolveWait wait) { return solve_systems(1, &A, &b, &x, max_iters, &scratch, st, out, kSpmvTiled, wait); }

cudaError_t bicgstab_solve_pair(const CsrDev A[2], const float *const b[2], float *const x[2], int max_iters, void *const scratch[2], cudaStream_t st, BicgResult out[2], int form) { return solve_systems(2, A, b, x, max_iters, scratch, st, out, form, SolveWait{}); }

// Loads this file's module (the driver loads a module at its first launch otherwise).
void load_module_bicgstab() {
  cudaFuncAttributes a;
  cudaFuncGetAttributes(&a, k_solve<kSpmvSliced>);
}

}  // namespace gpl
