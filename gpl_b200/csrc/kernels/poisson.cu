// The density solver (`Fft::solve`, src/nesterov.rs:412-444) as dense transforms: each 2-D
// cosine/sine transform of Ooura's package (src/ooura.rs:71-98) is a product with basis
// matrices on both sides, B_x^T * A * B_y, so the solve is six GEMMs and one spectral step:
//
//   T1t[v][x] = sum_y CyTs[v][y] rho[x][y]        forward along y (scale and halving folded in)
//   Ah[u][v]  = sum_x CxTs[u][x] T1t[v][x]        forward along x
//   Exh = Ah wx/(wx^2+wy^2), Eyh = Ah wy/(wx^2+wy^2), 0 at (0,0)
//   T2t[y][u] = sum_v Cy[y][v] Exh[u][v]   ;  Ex[x][y] = sum_u Sx[x][u] T2t[y][u]   (ddsct2d)
//   T3t[y][u] = sum_v Sy[y][v] Eyh[u][v]   ;  Ey[x][y] = sum_u Cx[x][u] T3t[y][u]   (ddcst2d)
//
// Every GEMM is D[m][n] = sum_k A[m][k] B[n][k] with both operands K-contiguous. The forward
// halving of row and column 0 and the 4/(nx*ny) scale are separable (h_u h_v (2/nx)(2/ny);
// the (0,0) term they disagree on is zeroed by the solve). Ooura's sine inverse keeps A[n] in
// a[0]; its basis column 0 is therefore (-1)^x. The potential is not computed: nothing but
// the reference's probes reads it.
//
// Mode 0 (this file): FP32 SIMT GEMMs. Mode 1: split-BF16 tcgen05 GEMMs (poisson_tc.cu).
// Mode 2 (this file): the FP32 form's sequence in double, the precision yardstick.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "engine_kernels.h"
#include "poisson_internal.h"
#include "parallel.h"
#include "scratch.h"

namespace gpl {

// ---------------------------------------------------------------- FP32, spread over the SMs
// BM x BN output tile per block, K in chunks of 32 through two shared buffers (the next chunk's
// loads in flight beside the current one's products), TM x 4 outputs a thread, pairs of rows in
// one packed FMA. Each output is one chain of fused multiply-adds over k in order, whatever the
// tile, so every shape gives the same bits.
constexpr int FG_BK = 32;

// The second GEMM's output taken through the spectral step (src/nesterov.rs:425-440) where it
// is formed: phi = Ah / (wx2 + wy2), Ex = phi wx, Ey = phi wy, zero at (0, 0). wx NULL: none.
struct GemmEpi {
  const float *wx, *wx2, *wy, *wy2;
  float *exh, *eyh;
};

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }

// One operand's chunk: `rows` of 32 k values, four at a time; element (r, k) sits at
// [k][(r / 4 ^ k / 4) * 4 + r % 4], so the transposing stores of a warp and the 16-byte reads
// along r meet no bank conflict.
template <int R, int NT>
struct Chunk {
  static constexpr int V = R * FG_BK / 4 / NT;
  float4 v[V];
  __device__ __forceinline__ void load(const float *__restrict__ A, int lda, int r0, int rows, int k0, int K, bool vec) {
#pragma unroll
    for (int i = 0; i < V; i++) {
      const int e = threadIdx.x + i * NT, r = r0 + e / (FG_BK / 4), k = k0 + e % (FG_BK / 4) * 4;
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r >= rows) continue;
      const float *p = A + (size_t)r * lda + k;
      if (vec) {
        if (k < K) v[i] = *reinterpret_cast<const float4 *>(p);
      } else {
        if (k < K) v[i].x = p[0];
        if (k + 1 < K) v[i].y = p[1];
        if (k + 2 < K) v[i].z = p[2];
        if (k + 3 < K) v[i].w = p[3];
      }
    }
  }
  __device__ __forceinline__ void store(float *s) const {
#pragma unroll
    for (int i = 0; i < V; i++) {
      const int e = threadIdx.x + i * NT, r = e / (FG_BK / 4), k4 = e % (FG_BK / 4);
      float *p = s + k4 * 4 * R + ((r >> 2) ^ k4) * 4 + (r & 3);
      p[0] = v[i].x;
      p[R] = v[i].y;
      p[2 * R] = v[i].z;
      p[3 * R] = v[i].w;
    }
  }
};

template <int BM, int BN, int TM>
__device__ __forceinline__ void gemm_tile_f32(const GemmProblem &P, const GemmEpi &E, const int m0, const int n0) {
  static_assert(BM % 32 == 0 && BN % 32 == 0 && TM % 4 == 0, "the chunks' layout");
  constexpr int NT = (BM / TM) * (BN / 4);
  __shared__ __align__(16) float As[2][FG_BK * BM];
  __shared__ __align__(16) float Bs[2][FG_BK * BN];
  const int tx = threadIdx.x % (BN / 4), ty = threadIdx.x / (BN / 4);
  const bool vec = ((P.K | P.lda | P.ldb) & 3) == 0 && (((uintptr_t)P.A | (uintptr_t)P.B) & 15) == 0;
  unsigned long long acc[TM / 2][4];
#pragma unroll
  for (int i = 0; i < TM / 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0ull;
  Chunk<BM, NT> ca;
  Chunk<BN, NT> cb;
  ca.load(P.A, P.lda, m0, P.M, 0, P.K, vec);
  cb.load(P.B, P.ldb, n0, P.N, 0, P.K, vec);
  int buf = 0;
  for (int k0 = 0; k0 < P.K; k0 += FG_BK) {
    ca.store(As[buf]);
    cb.store(Bs[buf]);
    __syncthreads();
    if (k0 + FG_BK < P.K) {
      ca.load(P.A, P.lda, m0, P.M, k0 + FG_BK, P.K, vec);
      cb.load(P.B, P.ldb, n0, P.N, k0 + FG_BK, P.K, vec);
    }
    const float *as = As[buf], *bs = Bs[buf];
#pragma unroll
    for (int kk = 0; kk < FG_BK; kk++) {
      unsigned long long a[TM / 2], b[4];
#pragma unroll
      for (int g = 0; g < TM / 4; g++) {
        const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(as + kk * BM + (((ty * TM / 4 + g) ^ (kk >> 2)) * 4));
        a[2 * g] = q.x;
        a[2 * g + 1] = q.y;
      }
      const float4 bv = *reinterpret_cast<const float4 *>(bs + kk * BN + ((tx ^ (kk >> 2)) * 4));
      b[0] = pack2(bv.x, bv.x);
      b[1] = pack2(bv.y, bv.y);
      b[2] = pack2(bv.z, bv.z);
      b[3] = pack2(bv.w, bv.w);
#pragma unroll
      for (int i = 0; i < TM / 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fma2(a[i], b[j], acc[i][j]);
    }
    buf ^= 1;
  }
  const int n = n0 + tx * 4;
  if (n >= P.N) return;
  const bool vs = n + 4 <= P.N && (P.ldd & 3) == 0 && (((uintptr_t)P.D | (uintptr_t)E.exh | (uintptr_t)E.eyh) & 15) == 0;
  auto put = [&](float *D, int m, const float *v) {
    float *p = D + (size_t)m * P.ldd + n;
    if (vs) {
      *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (n + j < P.N) p[j] = v[j];
    }
  };
#pragma unroll
  for (int i = 0; i < TM; i++) {
    const int m = m0 + ty * TM + i;
    if (m >= P.M) break;
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      float lo, hi;
      unpack2(acc[i >> 1][j], lo, hi);
      v[j] = (i & 1) ? hi : lo;
    }
    if (!E.wx) {
      put(P.D, m, v);
      continue;
    }
    const float wx = E.wx[m], wx2 = E.wx2[m];
    float ex[4], ey[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      ex[j] = ey[j] = 0.0f;
      if (n + j < P.N && (m != 0 || n + j != 0)) {
        const float p = __fdiv_rn(v[j], __fadd_rn(wx2, E.wy2[n + j]));
        ex[j] = __fmul_rn(p, wx);
        ey[j] = __fmul_rn(p, E.wy[n + j]);
      }
    }
    put(E.exh, m, ex);
    put(E.eyh, m, ey);
  }
}

template <int BM, int BN, int TM>
__global__ void __launch_bounds__((BM / TM) * (BN / 4)) k_gemm_f32(GemmBatch gb, GemmEpi E) {
  chain_enter();
  const GemmProblem P = gb.p[blockIdx.z];
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  if (m0 >= P.M || n0 >= P.N) return;
  gemm_tile_f32<BM, BN, TM>(P, E, m0, n0);
}

// Many problems in one launch: block b takes tile b - first[k] of problem k (the last with
// first[k] <= b), tiles row-major over the problem's grid; epis NULL: no spectral step.
template <int BM, int BN, int TM>
__global__ void __launch_bounds__((BM / TM) * (BN / 4)) k_gemm_grouped(const GemmProblem *__restrict__ probs, const GemmEpi *__restrict__ epis, const int *__restrict__ first, int n) {
  chain_enter();
  __shared__ int s_k;
  if (threadIdx.x == 0) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (first[mid] <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    s_k = lo;
  }
  __syncthreads();
  const GemmProblem P = probs[s_k];
  const GemmEpi E = epis ? epis[s_k] : GemmEpi{};
  const int t = (int)blockIdx.x - first[s_k];
  const int tn = (P.N + BN - 1) / BN;
  gemm_tile_f32<BM, BN, TM>(P, E, (t / tn) * BM, (t % tn) * BN);
}

// ---------------------------------------------------------------- FP64
// The same in double (the check paths: the FP64 solve, the density objective) on the double
// tensor path (mma m8n8k4), whose result is the chain of fused multiply-adds over k in order bit
// for bit: 64 x 32 tiles, a warp 32 x 16 of it, K in chunks of 16 through a ring of three
// asynchronous copies (two chunks in flight cover the round trip to L2). Rows are padded to 20
// values, so a fragment's 8 x 4 reads meet no bank conflict.
// 512 x 512 x 512: 21 us (94 in 32 tiles of 128 x 64 with eight-wide steps; 30 with these
// tiles in scalar multiply-adds); the chip's double rate bounds it at 7.
constexpr int DG_BM = 64, DG_BN = 32, DG_BK = 16, DG_NT = 128, DG_LD = DG_BK + 4, DG_STAGES = 3;

// One chunk of an operand into shared memory: asynchronously in pairs, or (an odd K or a base
// off 16 bytes) value by value.
template <int R>
__device__ __forceinline__ void dg_fetch(double *s, const double *__restrict__ A, int lda, int r0, int rows, int k0, int K, bool vec) {
  constexpr int PAIRS = R * DG_BK / 2;
#pragma unroll
  for (int i = 0; i < (PAIRS + DG_NT - 1) / DG_NT; i++) {
    const int e = threadIdx.x + i * DG_NT, r = e / (DG_BK / 2), k = e % (DG_BK / 2) * 2;
    if (PAIRS % DG_NT != 0 && e >= PAIRS) break;
    double *d = s + r * DG_LD + k;
    const bool in = r0 + r < rows;
    const double *p = A + (size_t)(in ? r0 + r : 0) * lda + k0 + k;
    if (vec) {
      const int bytes = in && k0 + k < K ? 16 : 0;  // the rest of the 16 is zero-filled
      if (!bytes) p = A;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(d)), "l"(p), "r"(bytes) : "memory");
    } else {
      d[0] = in && k0 + k < K ? p[0] : 0.0;
      d[1] = in && k0 + k + 1 < K ? p[1] : 0.0;
    }
  }
}

__global__ void __launch_bounds__(DG_NT) k_dgemm_tn(GemmBatchT<double> gb) {
  __shared__ __align__(16) double As[DG_STAGES][DG_BM * DG_LD];
  __shared__ __align__(16) double Bs[DG_STAGES][DG_BN * DG_LD];
  const GemmProblemT<double> P = gb.p[blockIdx.z];
  const int m0 = blockIdx.y * DG_BM, n0 = blockIdx.x * DG_BN;
  if (m0 >= P.M || n0 >= P.N) return;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int wm = (warp / 2) * 32, wn = (warp % 2) * 16;  // the warp's part of the tile
  const bool vec = ((P.K | P.lda | P.ldb) & 1) == 0 && (((uintptr_t)P.A | (uintptr_t)P.B) & 15) == 0;
  double acc[4][2][2] = {};
  const int chunks = (P.K + DG_BK - 1) / DG_BK;
  auto fetch = [&](int q) {
    if (q < chunks) {
      dg_fetch<DG_BM>(As[q % DG_STAGES], P.A, P.lda, m0, P.M, q * DG_BK, P.K, vec);
      dg_fetch<DG_BN>(Bs[q % DG_STAGES], P.B, P.ldb, n0, P.N, q * DG_BK, P.K, vec);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0);
  fetch(1);
  for (int q = 0; q < chunks; q++) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // chunk q is there for every thread, and chunk q - 1's buffer is free
    fetch(q + 2);
    const double *as = As[q % DG_STAGES] + (wm + lane / 4) * DG_LD + lane % 4, *bs = Bs[q % DG_STAGES] + (wn + lane / 4) * DG_LD + lane % 4;
#pragma unroll
    for (int k = 0; k < DG_BK; k += 4) {
      double a[4], b[2];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = as[i * 8 * DG_LD + k];
#pragma unroll
      for (int j = 0; j < 2; j++) b[j] = bs[j * 8 * DG_LD + k];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 2; j++)
          asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(acc[i][j][0]), "+d"(acc[i][j][1]) : "d"(a[i]), "d"(b[j]));
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int m = m0 + wm + i * 8 + lane / 4;
    if (m >= P.M) continue;
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int n = n0 + wn + j * 8 + 2 * (lane % 4) + h;
        if (n < P.N) P.D[(size_t)m * P.ldd + n] = acc[i][j][h];
      }
  }
}

cudaError_t dgemm_tn(const GemmBatchT<double> &gb, int count, cudaStream_t s) {
  int M = 0, N = 0;
  for (int i = 0; i < count; i++) {
    M = std::max(M, gb.p[i].M);
    N = std::max(N, gb.p[i].N);
  }
  k_dgemm_tn<<<dim3((N + DG_BN - 1) / DG_BN, (M + DG_BM - 1) / DG_BM, count), DG_NT, 0, s>>>(gb);
  return cudaGetLastError();
}

// One stage of the FP32 solve.
template <int BM, int BN, int TM>
static cudaError_t gemm_f32_launch(const GemmBatch &gb, int count, const GemmEpi &E, cudaStream_t s) {
  int M = 0, N = 0;
  for (int i = 0; i < count; i++) {
    M = std::max(M, gb.p[i].M);
    N = std::max(N, gb.p[i].N);
  }
  return launch_chained(k_gemm_f32<BM, BN, TM>, dim3((N + BN - 1) / BN, (M + BM - 1) / BM, count), dim3((BM / TM) * (BN / 4)), 0, s, gb, E);
}
// 128 x 64 tiles once they give nearly every one of the 148 SMs one (a 1024 x 1024 solve 334 us, 388 with
// 64 x 32, 640 with the unpacked 128 x 64 tile before); below that 64 x 32 tiles, so a small
// grid's products spread over the chip (512 x 512 80 us, 126 with 128 x 64; 64 x 64 8 blocks
// instead of one).
static cudaError_t gemm_f32(const GemmBatch &gb, int count, const GemmEpi &E, cudaStream_t s) {
  const GemmProblem &P = gb.p[0];
  if ((int64_t)((P.M + 127) / 128) * ((P.N + 63) / 64) >= 128) return gemm_f32_launch<128, 64, 8>(gb, count, E, s);
  return gemm_f32_launch<64, 32, 4>(gb, count, E, s);
}

// The FP64 yardstick's spectral step: the same in double (wavenumbers widened from float).
__global__ void k_spectral_d(int nx, int ny, const double *__restrict__ ah, const float *__restrict__ wx, const float *__restrict__ wy, double *__restrict__ exh, double *__restrict__ eyh) {
  int64_t n = (int64_t)nx * ny;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    int u = (int)(k / ny), v = (int)(k % ny);
    double ex = 0.0, ey = 0.0;
    if (u != 0 || v != 0) {
      const double a = (double)wx[u], b = (double)wy[v];
      const double p = ah[k] / (a * a + b * b);
      ex = p * a;
      ey = p * b;
    }
    exh[k] = ex;
    eyh[k] = ey;
  }
}
template <typename A, typename B>
__global__ void k_convert(int64_t n, const A *__restrict__ in, B *__restrict__ out) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) out[k] = (B)in[k];
}

// ---------------------------------------------------------------- basis matrices
// The host library's cosine and sine in double, the arguments exact products of the reference's
// order, rounded once to the form's type.
static double cos_entry(int k, int j, int n) { return std::cos(M_PI * (double)k * ((double)j + 0.5) / (double)n); }
static double sin_entry(int k, int j, int n) { return k == 0 ? ((j & 1) ? -1.0 : 1.0) : std::sin(M_PI * (double)k * ((double)j + 0.5) / (double)n); }
// Entry (r, c) of a basis matrix of side n.
static double basis_entry(int which, int r, int c, int n) {
  if (which == B_CYTS || which == B_CXTS) {
    const double h = (r == 0 ? 0.5 : 1.0) * 2.0 / (double)n;
    return h * cos_entry(r, c, n);
  }
  return which == B_SY || which == B_SX ? sin_entry(c, r, n) : cos_entry(c, r, n);
}

void build_basis(int nx, int ny, BasisHost &b) {
  for (int w = 0; w < B_COUNT; w++) {
    const int n = basis_of_x(w) ? nx : ny;
    b.m[w].assign((size_t)n * n, 0);
    parallel_for((size_t)n, [&](size_t r0, size_t r1) {
      for (int r = (int)r0; r < (int)r1; r++)
        for (int c = 0; c < n; c++) b.m[w][(size_t)r * n + c] = basis_entry(w, r, c, n);
    }, 16);
  }
}

// The float forms' matrices on the device. An entry's argument is the host's bit for bit (IEEE
// products and quotient), and the device's cosine and sine are within a few ulp of it, as the
// host library's are; where every double that near rounds to one float, that float is the
// host's. The few entries left (one in 10^7) are listed and taken from the host library. On
// the host the six matrices of a 1024 x 1024 grid took 12 ms on its threads and 4 ms to upload
// 25 MB; here 0.1 ms.
constexpr int kMaxUnsure = 1 << 16;
struct Unsure {
  unsigned int count, pad[3];
  int4 at[kMaxUnsure];  // matrix, row, column
};
__device__ __forceinline__ void basis_store(const BasisOut &out, int w, int n, int r, int c, float x) {
  if (out.f32[w]) out.f32[w][(size_t)r * n + c] = x;
  if (out.split[w]) {
    const __nv_bfloat16 hi = __float2bfloat16_rn(x);
    out.split[w][(size_t)r * 2 * n + c] = hi;
    out.split[w][(size_t)r * 2 * n + n + c] = __float2bfloat16_rn(x - __bfloat162float(hi));
  }
}
__global__ void __launch_bounds__(256) k_basis(int nx, int ny, BasisOut out, Unsure *unsure) {
  const int w = blockIdx.z;
  const bool x_side = w == B_CXTS || w == B_SX || w == B_CX;
  const int n = x_side ? nx : ny;
  for (int r = blockIdx.y; r < n; r += gridDim.y)
    for (int c = blockIdx.x * 256 + threadIdx.x; c < n; c += gridDim.x * 256) {
      const bool fwd = w == B_CYTS || w == B_CXTS;
      const int k = fwd ? r : c, j = fwd ? c : r;
      const double a = __ddiv_rn(__dmul_rn(__dmul_rn(M_PI, (double)k), __dadd_rn((double)j, 0.5)), (double)n);
      double v;
      if (w == B_SY || w == B_SX)
        v = k == 0 ? ((j & 1) ? -1.0 : 1.0) : sin(a);
      else
        v = cos(a);
      if (fwd) v = __dmul_rn(__ddiv_rn(__dmul_rn(r == 0 ? 0.5 : 1.0, 2.0), (double)n), v);
      const double e = fabs(v) * 0x1p-49;
      const float x = __double2float_rn(v);
      if (__double2float_rn(v - e) != x || __double2float_rn(v + e) != x) {
        const unsigned q = atomicAdd(&unsure->count, 1u);
        if (q < kMaxUnsure) unsure->at[q] = make_int4(w, r, c, 0);
      }
      basis_store(out, w, n, r, c, x);
    }
}
__global__ void k_basis_patch(int nx, int ny, BasisOut out, const Unsure *unsure, const float *x, unsigned count) {
  const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= count) return;
  const int4 at = unsure->at[q];
  const bool x_side = at.x == B_CXTS || at.x == B_SX || at.x == B_CX;
  basis_store(out, at.x, x_side ? nx : ny, at.y, at.z, x[q]);
}

constexpr int kMaxGridY = 65535;  // a row of blocks a matrix row, the rest of a longer side's in turn
cudaError_t device_basis(int nx, int ny, const BasisOut &out, cudaStream_t s) {
  Scratch buf(sizeof(Unsure), s);
  cudaError_t e = buf.error();
  if (e != cudaSuccess) return e;
  Unsure *u = static_cast<Unsure *>(buf.get());
  if ((e = cudaMemsetAsync(u, 0, sizeof(unsigned), s)) != cudaSuccess) return e;
  const int n = std::max(nx, ny);
  k_basis<<<dim3((unsigned)std::min((n + 255) / 256, 8), (unsigned)std::min(n, kMaxGridY), B_COUNT), 256, 0, s>>>(nx, ny, out, u);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  unsigned count = 0;
  if ((e = cudaMemcpyAsync(&count, u, sizeof count, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return e;
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
  if (count == 0) return cudaSuccess;
  if (count > (unsigned)kMaxUnsure) return cudaErrorUnknown;  // cannot happen: one entry in 10^7
  std::vector<int4> at(count);
  if ((e = cudaMemcpyAsync(at.data(), u->at, count * sizeof(int4), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return e;
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
  std::vector<float> x(count);
  for (unsigned q = 0; q < count; q++) x[q] = (float)basis_entry(at[q].x, at[q].y, at[q].z, basis_of_x(at[q].x) ? nx : ny);
  Scratch dx(count * sizeof(float), s);
  if ((e = dx.error()) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(dx.get(), x.data(), count * sizeof(float), cudaMemcpyHostToDevice, s)) != cudaSuccess) return e;
  k_basis_patch<<<(count + 255) / 256, 256, 0, s>>>(nx, ny, out, u, static_cast<const float *>(dx.get()), count);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  return cudaStreamSynchronize(s);  // the host values have been read
}

// One arena holds the plan: from the device's default pool (an engine's plans: kept warm by its
// release threshold), ordered on the legacy stream and complete when the create returns; or
// (scratch) from the entry points' own pool, ordered on the call's stream.
PoissonPlan *poisson_plan_create(int nx, int ny, const float *wx_host, const float *wy_host, int mode, cudaError_t *err, bool scratch, cudaStream_t s) {
  PoissonPlan *p = new PoissonPlan();
  p->nx = nx;
  p->ny = ny;
  // the tensor-core tiles are 128 rows by up to 128 columns, with K-blocks of 64: a grid whose
  // sides are not multiples of 128 (small or odd -bin_grid_count grids) is solved with the FP32
  // GEMMs
  if (mode == 1 && (nx % 128 != 0 || ny % 128 != 0)) mode = 0;
  p->mode = mode;
  p->scratch = scratch;
  p->stream = s;
  *err = cudaSuccess;
  const size_t n = (size_t)nx * ny, xx = (size_t)nx * nx, yy = (size_t)ny * ny;
  auto side2 = [&](int w) { return basis_of_x(w) ? xx : yy; };
  // the arena's layout, twice: its size, then the pointers
  char *base = nullptr;
  size_t at = 0;
  auto take = [&](auto **ptr, size_t count) {
    using E = typename std::remove_pointer<typename std::remove_reference<decltype(*ptr)>::type>::type;
    if (base) *ptr = reinterpret_cast<E *>(base + at);
    at += (count * sizeof(E) + 255) / 256 * 256;
  };
  float *w_all = nullptr;
  BasisOut out{};
  auto layout = [&]() {
    at = 0;
    take(&w_all, 2 * (size_t)(nx + ny));
    if (mode == 2) {
      for (int k = 0; k < B_COUNT; k++) take(&p->d_basis[k], side2(k));
      for (int k = 0; k < 8; k++) take(&p->d_buf[k], n);
    } else if (mode == 0) {
      for (int k = 0; k < B_COUNT; k++) take(&out.f32[k], side2(k));
      for (float **b : {&p->t1, &p->exh, &p->eyh, &p->t2, &p->t3}) take(b, n);
    } else {
      char *tc = nullptr;
      take(&tc, tc_plan_bytes(nx, ny));
      if (tc) *err = tc_plan_init(p, tc, out);
    }
  };
  auto fail = [&]() -> PoissonPlan * {
    poisson_plan_destroy(p);
    return nullptr;
  };
  layout();
  *err = scratch ? scratch_alloc(&p->arena, at, s) : cudaMallocAsync(&p->arena, at, s);
  if (*err != cudaSuccess) return fail();
  base = static_cast<char *>(p->arena);
  layout();
  if (*err != cudaSuccess) return fail();
  p->wx = w_all;
  p->wx2 = w_all + nx;
  p->wy = w_all + 2 * (size_t)nx;
  p->wy2 = p->wy + ny;
  std::vector<float> w((size_t)2 * (nx + ny));
  for (int i = 0; i < nx; i++) w[i] = wx_host[i], w[nx + i] = wx_host[i] * wx_host[i];
  for (int i = 0; i < ny; i++) w[2 * nx + i] = wy_host[i], w[2 * nx + ny + i] = wy_host[i] * wy_host[i];
  *err = cudaMemcpyAsync(w_all, w.data(), w.size() * sizeof(float), cudaMemcpyHostToDevice, s);
  if (*err == cudaSuccess && mode == 2) {
    BasisHost b;
    build_basis(nx, ny, b);
    for (int k = 0; k < B_COUNT && *err == cudaSuccess; k++) *err = cudaMemcpyAsync(p->d_basis[k], b.m[k].data(), b.m[k].size() * sizeof(double), cudaMemcpyHostToDevice, s);
    if (*err == cudaSuccess) *err = cudaStreamSynchronize(s);
  } else if (*err == cudaSuccess) {
    *err = device_basis(nx, ny, out, s);  // synchronises: the copies above have been read
  }
  if (*err != cudaSuccess) return fail();
  p->CyTs = out.f32[B_CYTS];
  p->CxTs = out.f32[B_CXTS];
  p->Cy = out.f32[B_CY];
  p->Sy = out.f32[B_SY];
  p->Sx = out.f32[B_SX];
  p->Cx = out.f32[B_CX];
  return p;
}

void poisson_plan_destroy(PoissonPlan *p) {
  if (!p) return;
  if (p->arena) {
    // an engine's plan may have been used on any of its streams
    if (!p->scratch) cudaDeviceSynchronize();
    cudaFreeAsync(p->arena, p->stream);
  }
  tc_plan_free(p);
  delete p;
}

__nv_bfloat16 *poisson_split_input(PoissonPlan *p, int *ld) {
  if (p->mode != 1) return nullptr;
  *ld = 2 * p->ny;
  return p->tc_dens;
}

__global__ void k_split_density(int nx, int ny, const float *__restrict__ d, __nv_bfloat16 *__restrict__ out, int ld) {
  int64_t n = (int64_t)nx * ny;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    int64_t x = k / ny, y = k % ny;
    float v = d[k];
    __nv_bfloat16 hi = __float2bfloat16_rn(v);
    out[x * ld + y] = hi;
    out[x * ld + ny + y] = __float2bfloat16_rn(v - __bfloat162float(hi));
  }
}

cudaError_t poisson_split_density(PoissonPlan *p, const float *density, cudaStream_t s) {
  if (p->mode != 1) return cudaSuccess;
  int64_t n = (int64_t)p->nx * p->ny;
  int blocks = (int)std::min<int64_t>((n + 255) / 256, 148 * 8);
  k_split_density<<<blocks, 256, 0, s>>>(p->nx, p->ny, density, p->tc_dens, 2 * p->ny);
  return cudaGetLastError();
}

int poisson_plan_mode(const PoissonPlan *p) { return p->mode; }

int poisson_launches(const PoissonPlan *p) { return p->mode == 0 ? 4 : p->mode == 2 ? 9 : tc_launches(p); }

// The FP64 form: the density widened to double, the FP32 form's six GEMMs and spectral step
// in double throughout, the fields rounded to float once at the end. The yardstick the
// other forms' placements are compared with; not a speed path.
static cudaError_t solve_fp64(PoissonPlan *p, const float *density, float *field_x, float *field_y, cudaStream_t s) {
  const int nx = p->nx, ny = p->ny;
  const int64_t n = (int64_t)nx * ny;
  const int blocks = (int)std::min<int64_t>((n + 255) / 256, 148 * 8);
  double *const *B = p->d_basis;
  double *rho = p->d_buf[0], *t1 = p->d_buf[1], *ah = p->d_buf[2], *exh = p->d_buf[3], *eyh = p->d_buf[4], *t2 = p->d_buf[5], *t3 = p->d_buf[6], *f = p->d_buf[7];
  k_convert<float, double><<<blocks, 256, 0, s>>>(n, density, rho);
  GemmBatchT<double> g{};
  g.p[0] = GemmProblemT<double>{ny, nx, ny, B[0], ny, rho, ny, t1, nx};
  cudaError_t e = dgemm_tn(g, 1, s);
  if (e != cudaSuccess) return e;
  g.p[0] = GemmProblemT<double>{nx, ny, nx, B[1], nx, t1, nx, ah, ny};
  if ((e = dgemm_tn(g, 1, s)) != cudaSuccess) return e;
  k_spectral_d<<<blocks, 256, 0, s>>>(nx, ny, ah, p->wx, p->wy, exh, eyh);
  g.p[0] = GemmProblemT<double>{ny, nx, ny, B[2], ny, exh, ny, t2, nx};
  g.p[1] = GemmProblemT<double>{ny, nx, ny, B[3], ny, eyh, ny, t3, nx};
  if ((e = dgemm_tn(g, 2, s)) != cudaSuccess) return e;
  g.p[0] = GemmProblemT<double>{nx, ny, nx, B[4], nx, t2, nx, f, ny};
  if ((e = dgemm_tn(g, 1, s)) != cudaSuccess) return e;
  k_convert<double, float><<<blocks, 256, 0, s>>>(n, f, field_x);
  g.p[0] = GemmProblemT<double>{nx, ny, nx, B[5], nx, t3, nx, f, ny};
  if ((e = dgemm_tn(g, 1, s)) != cudaSuccess) return e;
  k_convert<double, float><<<blocks, 256, 0, s>>>(n, f, field_y);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- many FP32 solves at once
// The FP32 solves of several regions (each its own grid) as four launches, each GEMM stage
// over every region's problems; every field is poisson_solve's bit for bit.
// 32 x 32 tiles: the groups' grids are mostly 16 to 64 points a side, which wider tiles would fill
// with padding. 48 groups of 2000 cells: the whole command level with 64 x 32 tiles (0.296 / 0.294
// s, runs 2 % apart).
constexpr int kGroupTile = 32;
struct PoissonGroup {
  // per stage: problems and each one's first tile; the second stage's spectral steps
  GemmProblem *probs[4] = {};
  int *first[4] = {};
  int count[4] = {}, tiles[4] = {};
  GemmEpi *epis = nullptr;
  int regions = 0;
};

PoissonGroup *poisson_group_create(PoissonPlan *const *plans, const float *const *density, float *const *field_x, float *const *field_y, int n, cudaError_t *err) {
  *err = cudaSuccess;
  PoissonGroup *g = new PoissonGroup();
  std::vector<GemmProblem> st[4];
  std::vector<GemmEpi> epis;
  for (int k = 0; k < n; k++) {
    PoissonPlan *p = plans[k];
    if (p->mode != 0) {
      *err = cudaErrorInvalidValue;  // the FP32 form's plans only
      poisson_group_destroy(g);
      return nullptr;
    }
    const int nx = p->nx, ny = p->ny;
    st[0].push_back(GemmProblem{ny, nx, ny, p->CyTs, ny, density[k], ny, p->t1, nx});
    st[1].push_back(GemmProblem{nx, ny, nx, p->CxTs, nx, p->t1, nx, nullptr, ny});
    st[2].push_back(GemmProblem{ny, nx, ny, p->Cy, ny, p->exh, ny, p->t2, nx});
    st[2].push_back(GemmProblem{ny, nx, ny, p->Sy, ny, p->eyh, ny, p->t3, nx});
    st[3].push_back(GemmProblem{nx, ny, nx, p->Sx, nx, p->t2, nx, field_x[k], ny});
    st[3].push_back(GemmProblem{nx, ny, nx, p->Cx, nx, p->t3, nx, field_y[k], ny});
    epis.push_back(GemmEpi{p->wx, p->wx2, p->wy, p->wy2, p->exh, p->eyh});
  }
  auto put = [&](auto **d, const auto &v) {
    if (*err != cudaSuccess || v.empty()) return;
    using E = typename std::remove_reference<decltype(v)>::type::value_type;
    *err = pool_alloc((void **)d, v.size() * sizeof(E));
    if (*err == cudaSuccess) *err = pool_upload(*d, v.data(), v.size() * sizeof(E));
  };
  for (int q = 0; q < 4; q++) {
    std::vector<int> first;
    int t = 0;
    for (const GemmProblem &P : st[q]) {
      first.push_back(t);
      t += ((P.M + kGroupTile - 1) / kGroupTile) * ((P.N + kGroupTile - 1) / kGroupTile);
    }
    g->count[q] = (int)st[q].size();
    g->tiles[q] = t;
    put(&g->probs[q], st[q]);
    put(&g->first[q], first);
  }
  g->regions = n;
  put(&g->epis, epis);
  if (*err == cudaSuccess) *err = cudaStreamSynchronize(0);
  if (*err != cudaSuccess) {
    poisson_group_destroy(g);
    return nullptr;
  }
  return g;
}

void poisson_group_destroy(PoissonGroup *g) {
  if (!g) return;
  cudaDeviceSynchronize();
  for (int q = 0; q < 4; q++) {
    pool_free(g->probs[q]);
    pool_free(g->first[q]);
  }
  pool_free(g->epis);
  delete g;
}

cudaError_t poisson_group_solve(const PoissonGroup *g, cudaStream_t s) {
  if (!g || g->regions == 0) return cudaSuccess;
  cudaError_t e = cudaSuccess;
  for (int q = 0; q < 4 && e == cudaSuccess; q++)
    e = launch_chained(k_gemm_grouped<kGroupTile, kGroupTile, 4>, dim3(g->tiles[q]), dim3(kGroupTile * kGroupTile / 16), 0, s, (const GemmProblem *)g->probs[q],
                       (const GemmEpi *)(q == 1 ? g->epis : nullptr), (const int *)g->first[q], g->count[q]);
  return e;
}

int poisson_group_launches(const PoissonGroup *g) { return g && g->regions ? 4 : 0; }

cudaError_t poisson_solve(PoissonPlan *p, const float *density, float *field_x, float *field_y, cudaStream_t s) {
  if (p->mode == 2) return solve_fp64(p, density, field_x, field_y, s);
  if (p->mode != 0) return tc_solve(p, field_x, field_y, s);
  int nx = p->nx, ny = p->ny;
  const GemmEpi none{}, spectral{p->wx, p->wx2, p->wy, p->wy2, p->exh, p->eyh};
  GemmBatch g{};
  g.p[0] = GemmProblem{ny, nx, ny, p->CyTs, ny, density, ny, p->t1, nx};
  cudaError_t e = gemm_f32(g, 1, none, s);
  if (e != cudaSuccess) return e;
  g.p[0] = GemmProblem{nx, ny, nx, p->CxTs, nx, p->t1, nx, nullptr, ny};
  if ((e = gemm_f32(g, 1, spectral, s)) != cudaSuccess) return e;
  g.p[0] = GemmProblem{ny, nx, ny, p->Cy, ny, p->exh, ny, p->t2, nx};
  g.p[1] = GemmProblem{ny, nx, ny, p->Sy, ny, p->eyh, ny, p->t3, nx};
  if ((e = gemm_f32(g, 2, none, s)) != cudaSuccess) return e;
  g.p[0] = GemmProblem{nx, ny, nx, p->Sx, nx, p->t2, nx, field_x, ny};
  g.p[1] = GemmProblem{nx, ny, nx, p->Cx, nx, p->t3, nx, field_y, ny};
  return gemm_f32(g, 2, none, s);
}


// Loads this file's module (the driver loads a module at its first launch otherwise).
void load_module_poisson() {
  cudaFuncAttributes a;
  cudaFuncGetAttributes(&a, k_gemm_grouped<kGroupTile, kGroupTile, 4>);
}

}  // namespace gpl

// Test-only: the double GEMM, D[M][N] = A[M][K] B[N][K]^T on device arrays.
extern "C" int gpl_rules_dgemm(int32_t M, int32_t N, int32_t K, const double *A, int32_t lda, const double *B, int32_t ldb, double *D, int32_t ldd, void *stream) {
  gpl::GemmBatchT<double> g{};
  g.p[0] = gpl::GemmProblemT<double>{M, N, K, A, lda, B, ldb, D, ldd};
  return (int)gpl::dgemm_tn(g, 1, (cudaStream_t)stream);
}

// Test-only: the six matrices the device makes, in float, one after the other into host memory
// (sides ny, nx, ny, ny, nx, nx).
extern "C" int gpl_rules_basis(int32_t nx, int32_t ny, float *out) {
  using namespace gpl;
  if (nx <= 0 || ny <= 0) return (int)cudaErrorInvalidValue;
  const size_t xx = (size_t)nx * nx, yy = (size_t)ny * ny;
  Scratch buf(3 * (xx + yy) * sizeof(float), 0);
  cudaError_t e = buf.error();
  if (e != cudaSuccess) return (int)e;
  BasisOut o{};
  size_t at = 0;
  for (int k = 0; k < B_COUNT; k++) {
    o.f32[k] = static_cast<float *>(buf.get()) + at;
    at += basis_of_x(k) ? xx : yy;
  }
  e = device_basis(nx, ny, o, 0);
  if (e == cudaSuccess) e = cudaMemcpy(out, buf.get(), at * sizeof(float), cudaMemcpyDeviceToHost);
  return (int)e;
}
