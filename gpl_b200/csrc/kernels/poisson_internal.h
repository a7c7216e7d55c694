// The density solver's internals: GEMM problem descriptors, the plan, the basis matrices.
#pragma once
#include <cstdint>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace gpl {

// D[m][n] = sum_k A[m][k] * B[n][k], row-major, leading dimensions in elements.
template <typename T>
struct GemmProblemT {
  int M, N, K;
  const T *A;
  int lda;
  const T *B;
  int ldb;
  T *D;
  int ldd;
};
template <typename T>
struct GemmBatchT {
  GemmProblemT<T> p[2];
};
using GemmProblem = GemmProblemT<float>;
using GemmBatch = GemmBatchT<float>;
cudaError_t dgemm_tn(const GemmBatchT<double> &gb, int count, cudaStream_t s);

// The six basis matrices (see poisson.cu): CyTs[v][y], CxTs[u][x] (forward, scaled and
// halved), Cy[y][v], Sy[y][v], Sx[x][u], Cx[x][u] (inverses).
enum Basis { B_CYTS = 0, B_CXTS, B_CY, B_SY, B_SX, B_CX, B_COUNT };
inline bool basis_of_x(int b) { return b == B_CXTS || b == B_SX || b == B_CX; }
struct BasisHost {
  std::vector<double> m[B_COUNT];  // in double (the FP64 form)
};
void build_basis(int nx, int ny, BasisHost &b);
// Where the device writes one of them: FP32 [n][n], or split BF16 [n][2 n] (hi | lo).
struct BasisOut {
  float *f32[B_COUNT];
  __nv_bfloat16 *split[B_COUNT];
};
// The matrices in float, rounded from the host library's double cosines and sines bit for bit
// (poisson.cu), on stream s, which it synchronises.
cudaError_t device_basis(int nx, int ny, const BasisOut &out, cudaStream_t s);

// A group's tables come from the device's stream-ordered pool (kept warm), ordered on the
// legacy stream: a group is complete once its create has synchronised that stream, and its
// destroy synchronises the device before it returns the memory, as cudaFree would.
inline cudaError_t pool_alloc(void **p, size_t bytes) { return cudaMallocAsync(p, bytes, 0); }
inline cudaError_t pool_upload(void *d, const void *h, size_t bytes) { return cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, 0); }
inline void pool_free(void *p) {
  if (p) cudaFreeAsync(p, 0);
}

struct TcState;  // the split-BF16 tensor-core path's buffers (poisson_tc.cu)

struct PoissonPlan {
  int nx = 0, ny = 0, mode = 0;
  void *arena = nullptr;       // every buffer below
  bool scratch = false;        // the arena is the entry points' scratch, ordered on `stream`
  cudaStream_t stream = nullptr;
  float *wx = nullptr, *wx2 = nullptr, *wy = nullptr, *wy2 = nullptr;
  // FP32 path
  float *CyTs = nullptr, *CxTs = nullptr, *Cy = nullptr, *Sy = nullptr, *Sx = nullptr, *Cx = nullptr;
  float *t1 = nullptr, *exh = nullptr, *eyh = nullptr, *t2 = nullptr, *t3 = nullptr;
  // tensor-core path
  __nv_bfloat16 *tc_dens = nullptr;  // density as [nx][2*ny] bf16 (hi | lo)
  TcState *tc = nullptr;
  // FP64 path (the yardstick): the FP32 path's matrices and sequence in double
  double *d_basis[6] = {};           // CyTs, CxTs, Cy, Sy, Sx, Cx
  double *d_buf[8] = {};             // rho, t1, ah, exh, eyh, t2, t3, and the fields' staging
};

// The tensor-core form's buffers and tensor maps: its size, then (the arena allocated) its
// layout from `base` and the basis matrices' places.
size_t tc_plan_bytes(int nx, int ny);
cudaError_t tc_plan_init(PoissonPlan *p, char *base, BasisOut &out);
void tc_plan_free(PoissonPlan *p);
cudaError_t tc_solve(PoissonPlan *p, float *field_x, float *field_y, cudaStream_t s);
int tc_launches(const PoissonPlan *p);

}  // namespace gpl
