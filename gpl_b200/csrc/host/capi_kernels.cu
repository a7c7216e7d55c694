// The per-kernel C entry points (include/gpl.h) and the synthetic router.
#include <algorithm>
#include <climits>
#include <cstring>
#include <cstdlib>
#include <memory>
#include <string>
#include <vector>

#include "../../../include/gpl.h"
#include "../kernels/b2b.h"
#include "../kernels/bicgstab.h"
#include "../kernels/engine_kernels.h"
#include "../kernels/rudy.h"
#include "../kernels/scratch.h"
#include "parallel.h"

using namespace gpl;

// A grid of the caller's bins as the trial kernels read it; its upper corner and the scatter's
// 32-bit test are taken from the edges on the device, into `corner` (NULL: not needed), so the
// call waits for nothing.
static void region_args(RegionArgs &r, int4 *corner, int32_t nx, int32_t ny, int32_t grid_lx, int32_t grid_ly, const int32_t *bx, const int32_t *by, double size_x, double size_y, float target_density, cudaStream_t s) {
  r.nx = nx;
  r.ny = ny;
  r.lx = grid_lx;
  r.ly = grid_ly;
  r.size_x = size_x;
  r.size_y = size_y;
  r.inv_size_x = 1.0 / size_x;
  r.inv_size_y = 1.0 / size_y;
  r.target_density = target_density;
  // GPL_SCATTER=global|pooled: the scatter's other forms (the engine's tuner picks per region)
  if (const char *f = std::getenv("GPL_SCATTER")) r.scatter_form = std::string(f) == "global" ? 1 : std::string(f) == "pooled" ? 2 : 0;
  r.bx = bx;
  r.by = by;
  r.corner = corner;
  if (corner) k_grid_corner<<<1, kThreadsPerBlock, 0, s>>>(nx, ny, bx, by, corner);
}

static bool counts_fit(int64_t n_cells, int32_t nx, int32_t ny) { return n_cells >= 0 && n_cells < ((int64_t)1 << 31) && nx > 0 && ny > 0; }

extern "C" {

int gpl_kernel_density_scatter(int64_t n_cells, const int32_t *cx, const int32_t *cy, const int32_t *hx, const int32_t *hy, const float *scale, const uint8_t *kind, int32_t nx, int32_t ny, int32_t grid_lx, int32_t grid_ly, const int32_t *bx, const int32_t *by, double size_x, double size_y, float target_density, int64_t *inst, int64_t *filler, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  size_t nb = (size_t)nx * ny;
  cudaError_t e = cudaMemsetAsync(inst, 0, nb * sizeof(int64_t), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(filler, 0, nb * sizeof(int64_t), s);
  if (e != cudaSuccess) return (int)e;
  if (n_cells <= 0) return 0;
  RegionArgs r{};
  r.n_cells = (int32_t)n_cells;
  // the engine keeps a cell's centre as one int2: pack the caller's two arrays
  Scratch buf(sizeof(int4) + (size_t)n_cells * sizeof(int2), s);
  if ((e = buf.error()) != cudaSuccess) return (int)e;
  region_args(r, static_cast<int4 *>(buf.get()), nx, ny, grid_lx, grid_ly, bx, by, size_x, size_y, target_density, s);
  r.acc_inst = inst;
  r.acc_fill = filler;
  int2 *dc = reinterpret_cast<int2 *>(static_cast<int4 *>(buf.get()) + 1);
  unsigned blocks = (unsigned)((n_cells + kThreadsPerBlock - 1) / kThreadsPerBlock);
  k_pack_centres<<<blocks, kThreadsPerBlock, 0, s>>>(n_cells, cx, cy, dc);
  CellArgs c{};
  c.dc = dc;
  c.hx = hx;
  c.hy = hy;
  c.dscale = scale;
  c.kind = kind;
  k_place_cells<<<blocks, kThreadsPerBlock, 0, s>>>(r, c, PLACE_GIVEN, 0.0f, 0.0f, nullptr);
  return (int)cudaGetLastError();
}

static bool aligned8(const void *p) { return ((uintptr_t)p & 7u) == 0; }

int gpl_kernel_nesterov_step(int64_t n_cells, const float *cur_slp, const float *cur_slp_sum, const float *cur, const int32_t *hx, const int32_t *hy, const float *scale, const uint8_t *kind, const uint8_t *locked, int32_t nx, int32_t ny, int32_t grid_lx, int32_t grid_ly, const int32_t *bx, const int32_t *by, double size_x, double size_y, float target_density, float step, float coeff, float *next, float *next_slp, int32_t *centre, int64_t *inst, int64_t *filler, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (!counts_fit(n_cells, nx, ny)) return (int)cudaErrorInvalidValue;
  for (const void *p : {(const void *)cur_slp, (const void *)cur_slp_sum, (const void *)cur, (const void *)next, (const void *)next_slp, (const void *)centre})
    if (!aligned8(p)) return (int)cudaErrorMisalignedAddress;  // read and written as pairs
  size_t nb = (size_t)nx * ny;
  cudaError_t e = cudaMemsetAsync(inst, 0, nb * sizeof(int64_t), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(filler, 0, nb * sizeof(int64_t), s);
  if (e != cudaSuccess || n_cells == 0) return (int)e;
  Scratch buf(sizeof(int4), s);
  if ((e = buf.error()) != cudaSuccess) return (int)e;
  RegionArgs r{};
  r.n_cells = (int32_t)n_cells;
  region_args(r, static_cast<int4 *>(buf.get()), nx, ny, grid_lx, grid_ly, bx, by, size_x, size_y, target_density, s);
  r.acc_inst = inst;
  r.acc_fill = filler;
  CellArgs c{};
  c.dc = reinterpret_cast<int2 *>(centre);
  c.hx = hx;
  c.hy = hy;
  c.dscale = scale;
  c.kind = kind;
  c.locked = locked;
  // the kernel reads cur_slp, cur_slp_sum and cur and writes next and next_slp only
  c.cur_slp = reinterpret_cast<float2 *>(const_cast<float *>(cur_slp));
  c.cur_slp_sum = reinterpret_cast<float2 *>(const_cast<float *>(cur_slp_sum));
  c.cur = reinterpret_cast<float2 *>(const_cast<float *>(cur));
  c.next = reinterpret_cast<float2 *>(next);
  c.next_slp = reinterpret_cast<float2 *>(next_slp);
  unsigned blocks = (unsigned)((n_cells + kThreadsPerBlock - 1) / kThreadsPerBlock);
  k_place_cells<<<blocks, kThreadsPerBlock, 0, s>>>(r, c, PLACE_NESTEROV, step, coeff, nullptr);
  return (int)cudaGetLastError();
}

int gpl_kernel_gradients(int64_t n_cells, const int32_t *centre, const int32_t *hx, const int32_t *hy, const float *scale, const float *area, const int64_t *cell_pin_start, const float *pin_force, int32_t nx, int32_t ny, int32_t grid_lx, int32_t grid_ly, const int32_t *bx, const int32_t *by, double size_x, double size_y, const float *field_x, const float *field_y, float penalty, float *sum, const float *a1, const float *b1, const float *b2, double *sums, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  for (int k = 0; k < 4; k++) sums[k] = 0.0;
  if (!counts_fit(n_cells, nx, ny)) return (int)cudaErrorInvalidValue;
  for (const void *p : {(const void *)centre, (const void *)pin_force, (const void *)sum, (const void *)a1, (const void *)b1, (const void *)b2})
    if (!aligned8(p)) return (int)cudaErrorMisalignedAddress;
  if ((a1 == nullptr) != (b1 == nullptr)) return (int)cudaErrorInvalidValue;
  if (n_cells == 0) return 0;
  RegionArgs r{};
  r.n_cells = (int32_t)n_cells;
  region_args(r, nullptr, nx, ny, grid_lx, grid_ly, bx, by, size_x, size_y, 1.0f, s);  // the update reads no corner
  r.field_x = const_cast<float *>(field_x);
  r.field_y = const_cast<float *>(field_y);
  CellArgs c{};
  c.dc = reinterpret_cast<int2 *>(const_cast<int32_t *>(centre));
  c.hx = hx;
  c.hy = hy;
  c.dscale = scale;
  c.area = area;
  c.pin_start = cell_pin_start;
  const int blocks = (int)((n_cells + kThreadsPerBlock - 1) / kThreadsPerBlock);
  // the block partials, the arrival ticket and the four sums, in one scratch block
  const size_t bytes = (size_t)(4 * blocks + 4) * sizeof(double) + 256;
  Scratch buf(bytes, s);
  cudaError_t e = buf.error();
  if (e != cudaSuccess) return (int)e;
  double *partials = static_cast<double *>(buf.get()), *out = partials + 4 * blocks;
  unsigned int *ticket = reinterpret_cast<unsigned int *>(out + 4);
  e = cudaMemsetAsync(ticket, 0, sizeof(unsigned int), s);
  if (e == cudaSuccess) {
    k_gradients<<<blocks, kThreadsPerBlock, 0, s>>>(r, c, reinterpret_cast<const float2 *>(pin_force), penalty, reinterpret_cast<float2 *>(sum), reinterpret_cast<const float2 *>(a1),
                                                    reinterpret_cast<const float2 *>(b1), reinterpret_cast<const float2 *>(b2), partials, ticket, out, Publish{});
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(sums, out, 4 * sizeof(double), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  return (int)e;
}

int gpl_kernel_poisson(int32_t nx, int32_t ny, const float *wx, const float *wy, const float *density, float *field_x, float *field_y, int mode, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaSuccess;
  PoissonPlan *p = poisson_plan_create(nx, ny, wx, wy, mode, &e, true, s);
  if (!p) return (int)e;
  int ld = 0;
  __nv_bfloat16 *split = poisson_split_input(p, &ld);
  if (split) {
    // the tensor-core path reads the density as split bf16: convert it
    e = poisson_split_density(p, density, s);
  }
  if (e == cudaSuccess) e = poisson_solve(p, density, field_x, field_y, s);
  cudaError_t e2 = cudaStreamSynchronize(s);
  poisson_plan_destroy(p);
  return (int)(e != cudaSuccess ? e : e2);
}

// The caller's nets as the engine's kernels take them, grouped by degree on the device: a class
// a degree up to kWaTilePins (its nets' pins then lie at a fixed stride, so no scan is needed)
// and one for the larger nets, which stay where they are. A net's place within its class is
// free: every force goes back to its pin's own slot and the HPWL is an integer sum. The host
// sees the classes' counts only (it sorted and copied the nets and pins before: a call of 105k nets
// took 5.2 ms, now 0.09).
constexpr int kClasses = kWaTilePins + 2;  // degrees 0 .. kWaTilePins, larger

__device__ __forceinline__ int net_class(const int64_t *start, int64_t n) {
  const int64_t d = start[n + 1] - start[n];
  return d < 0 ? 0 : d > kWaTilePins ? kWaTilePins + 1 : (int)d;
}
// The classes' counts, and the pins the windows reach to (past the last start, where the starts do
// not ascend).
struct NetCounts {
  long long reach;
  int32_t count[kClasses];
};
static __global__ void __launch_bounds__(256) k_net_classes(int64_t n, const int64_t *__restrict__ start, NetCounts *__restrict__ out) {
  __shared__ int32_t h[kClasses];
  __shared__ long long reach;
  int32_t *count = out->count;
  for (int k = threadIdx.x; k < kClasses; k += 256) h[k] = 0;
  if (threadIdx.x == 0) reach = 0;
  __syncthreads();
  long long top = 0;
  for (int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
    const int c = net_class(start, i);
    if (c > 0) top = max(top, (long long)start[i + 1]);
    atomicAdd(&h[c], 1);
  }
  if (top > 0) atomicMax(&reach, top);
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(&out->reach, reach);
  for (int k = threadIdx.x; k < kClasses; k += 256)
    if (h[k]) atomicAdd(&count[k], h[k]);
}
// cursor[c]: the class's next net; first, pin0: its first net and pin. The larger nets' indices
// go to `big`.
static __global__ void __launch_bounds__(256) k_net_place(int64_t n, const int64_t *__restrict__ start, const int32_t *__restrict__ xy, const float *__restrict__ weight, int32_t *__restrict__ cursor, const int32_t *__restrict__ first,
                                                           const int64_t *__restrict__ pin0, int64_t *__restrict__ ns, int2 *__restrict__ xy2, int32_t *__restrict__ slot, float *__restrict__ weight2, int32_t *__restrict__ big) {
  const int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x;
  const int c = i < n ? net_class(start, i) : -1;
  // one atomic for a warp's nets of a class
  const unsigned peers = __match_any_sync(0xffffffffu, c);
  const int lead = __ffs(peers) - 1, lane = threadIdx.x & 31;
  int32_t at = 0;
  if (c >= 0 && lane == lead) at = atomicAdd(&cursor[c], __popc(peers));
  at = __shfl_sync(0xffffffffu, at, lead) + __popc(peers & ((1u << lane) - 1u));
  if (c < 0) return;
  if (c > kWaTilePins) {
    big[at] = (int32_t)i;
    return;
  }
  const int64_t p = pin0[c] + (int64_t)(at - first[c]) * c, q = start[i];
  ns[at + 1] = p + c;
  if (weight) weight2[at] = weight[i];
  for (int k = 0; k < c; k++) {
    xy2[p + k] = make_int2(xy[2 * (q + k)], xy[2 * (q + k) + 1]);  // 4-byte aligned, as the caller may have it
    slot[p + k] = (int32_t)(q + k);
  }
}

struct DeviceNets {
  cudaStream_t s;
  WaArgs w{};     // the grouped nets
  WaArgs big{};   // the larger nets, in the caller's arrays
  int64_t n_pins = 0;
  std::unique_ptr<Scratch> buf;
  explicit DeviceNets(cudaStream_t st) : s(st) {}
  cudaError_t build(int64_t n_nets, const int64_t *net_start, const int32_t *pin_xy, const float *net_weight) {
    if (n_nets >= ((int64_t)1 << 31)) return cudaErrorInvalidValue;  // net numbers are 32-bit
    Scratch hist(sizeof(NetCounts), s);
    cudaError_t e = hist.error();
    NetCounts *d_count = static_cast<NetCounts *>(hist.get()), got;
    if (e == cudaSuccess) e = cudaMemsetAsync(d_count, 0, sizeof got, s);
    if (e != cudaSuccess) return e;
    k_net_classes<<<(unsigned)std::min<int64_t>((n_nets + 255) / 256, 148 * 8), 256, 0, s>>>(n_nets, net_start, d_count);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    e = cudaMemcpyAsync(&got, d_count, sizeof got, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    const int32_t *count = got.count;
    const int64_t np = n_pins = got.reach;
    if (np >= ((int64_t)1 << 31)) return cudaErrorInvalidValue;  // pin numbers are 32-bit
    // the classes' places, the tiles of the degrees outside 2..4
    std::vector<int32_t> first(kClasses);
    std::vector<int64_t> pin0(kClasses);
    std::vector<int4> tiles;
    int32_t net = 0;
    int64_t pin = 0;
    for (int c = 0; c <= kWaTilePins; c++) {
      first[c] = net;
      pin0[c] = pin;
      if (c >= 2 && c <= 4) {
        w.small.first[c - 2] = net;
        w.small.count[c - 2] = count[c];
        w.small.pin0[c - 2] = pin;
      } else if (c > 0) {
        const int32_t per = std::min(kWaTileNets, kWaTilePins / c);
        for (int32_t k = 0; k < count[c]; k += per) {
          const int32_t m = std::min(per, count[c] - k);
          tiles.push_back(make_int4(net + k, net + k + m, (int32_t)(pin + (int64_t)k * c), m * c));
        }
      }
      net += count[c];
      pin += (int64_t)count[c] * c;
    }
    if (pin >= ((int64_t)1 << 31)) return cudaErrorInvalidValue;  // the same of the copies, where windows share pins
    first[kWaTilePins + 1] = 0;  // the larger nets' list
    const int32_t n_big = count[kWaTilePins + 1];
    // one block of scratch: the tables (uploaded together), then what the placement writes
    size_t at = 0;
    auto take = [&](size_t bytes) {
      const size_t o = at;
      at += (bytes + 255) / 256 * 256;
      return o;
    };
    const size_t o_cur = take(kClasses * sizeof(int32_t)), o_first = take(kClasses * sizeof(int32_t)), o_pin0 = take(kClasses * sizeof(int64_t)), o_tiles = take(tiles.size() * sizeof(int4)), tables = at;
    const size_t o_ns = take(((size_t)net + 1) * sizeof(int64_t)), o_xy = take((size_t)pin * sizeof(int2)), o_slot = take((size_t)pin * sizeof(int32_t)), o_big = take((size_t)n_big * sizeof(int32_t)),
                 o_w = take(net_weight ? (size_t)net * sizeof(float) : 0);
    // the larger nets' kernels read positions as pairs
    const bool pairs = n_big == 0 || ((uintptr_t)pin_xy & 7) == 0;
    const size_t o_copy = take(pairs ? 0 : (size_t)np * sizeof(int2));
    buf = std::make_unique<Scratch>(at, s);
    if ((e = buf->error()) != cudaSuccess) return e;
    char *d = static_cast<char *>(buf->get());
    std::vector<char> host(tables, 0);
    std::memcpy(host.data() + o_cur, first.data(), kClasses * sizeof(int32_t));
    std::memcpy(host.data() + o_first, first.data(), kClasses * sizeof(int32_t));
    std::memcpy(host.data() + o_pin0, pin0.data(), kClasses * sizeof(int64_t));
    if (!tiles.empty()) std::memcpy(host.data() + o_tiles, tiles.data(), tiles.size() * sizeof(int4));
    if ((e = cudaMemcpyAsync(d, host.data(), tables, cudaMemcpyHostToDevice, s)) != cudaSuccess) return e;
    int64_t *ns = reinterpret_cast<int64_t *>(d + o_ns);
    if ((e = cudaMemsetAsync(ns, 0, sizeof(int64_t), s)) != cudaSuccess) return e;
    float *weight2 = net_weight ? reinterpret_cast<float *>(d + o_w) : nullptr;
    int32_t *slot = reinterpret_cast<int32_t *>(d + o_slot), *big_list = reinterpret_cast<int32_t *>(d + o_big);
    int2 *xy2 = reinterpret_cast<int2 *>(d + o_xy);
    k_net_place<<<(unsigned)((n_nets + 255) / 256), 256, 0, s>>>(n_nets, net_start, pin_xy, net_weight, reinterpret_cast<int32_t *>(d + o_cur), reinterpret_cast<const int32_t *>(d + o_first),
                                                               reinterpret_cast<const int64_t *>(d + o_pin0), ns, xy2, slot, weight2, big_list);
    w.net_start = ns;
    w.net_weight = weight2;
    w.pin_base = xy2;
    w.pin_slot = slot;
    w.n_tiles = (int32_t)tiles.size();
    w.tiles = reinterpret_cast<const int4 *>(d + o_tiles);
    big.n_nets = n_big;
    big.net_start = net_start;
    big.net_order = big_list;
    big.net_weight = net_weight;
    big.pin_base = reinterpret_cast<const int2 *>(pairs ? reinterpret_cast<const char *>(pin_xy) : d + o_copy);
    e = cudaGetLastError();
    if (e == cudaSuccess && !pairs) e = cudaMemcpyAsync(d + o_copy, pin_xy, (size_t)np * sizeof(int2), cudaMemcpyDeviceToDevice, s);
    return e;
  }
  // The two argument blocks with the forces' array and the HPWL sum.
  void out(float *grad, unsigned long long *hpwl) {
    w.pin_grad = big.pin_grad = reinterpret_cast<float2 *>(grad);
    w.hpwl_out = big.hpwl_out = hpwl;
  }
};

static void launch_net_forces(const DeviceNets &d, float cx, float cy, cudaStream_t s) {
  // in the engine's launches: joint for few nets
  if (wa_joint_fits(d.w.small, d.w.n_tiles) && !std::getenv("GPL_WA_SMALL")) {
    launch_wa_joint(d.w, cx, cy, s);
  } else {
    launch_wa_small(d.w, cx, cy, 1, s);
    if (d.w.n_tiles) launch_wa_tiles(d.w, cx, cy, s);
  }
  if (d.big.n_nets) k_wa<<<(unsigned)((d.big.n_nets + kThreadsPerBlock - 1) / kThreadsPerBlock), kThreadsPerBlock, 0, s>>>(d.big, cx, cy);
}

int gpl_kernel_wa(int64_t n_nets, const int64_t *net_start, const int32_t *pin_xy, const float *net_weight, float coef_x, float coef_y, float *grad, void *stream) {
  if (n_nets <= 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e;
  {
    DeviceNets d(s);
    e = d.build(n_nets, net_start, pin_xy, net_weight);
    if (e == cudaSuccess) {
      d.out(grad, nullptr);
      launch_net_forces(d, coef_x, coef_y, s);
      e = cudaGetLastError();
    }
  }
  cudaError_t e2 = cudaStreamSynchronize(s);
  return (int)(e != cudaSuccess ? e : e2);
}

int gpl_kernel_hpwl(int64_t n_nets, const int64_t *net_start, const int32_t *pin_xy, int32_t fused, int64_t *hpwl, void *stream) {
  *hpwl = 0;
  if (n_nets <= 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e;
  unsigned long long h = 0;
  {
    DeviceNets d(s);
    e = d.build(n_nets, net_start, pin_xy, nullptr);
    const size_t force_bytes = fused ? (size_t)std::max<int64_t>(d.n_pins, 1) * 2 * sizeof(float) : 0;
    std::unique_ptr<Scratch> buf;
    if (e == cudaSuccess) {
      buf = std::make_unique<Scratch>(256 + force_bytes, s);
      e = buf->error();
    }
    unsigned long long *acc = buf ? static_cast<unsigned long long *>(buf->get()) : nullptr;
    if (e == cudaSuccess) e = cudaMemsetAsync(acc, 0, sizeof(unsigned long long), s);
    if (e == cudaSuccess) {
      d.out(fused ? reinterpret_cast<float *>(reinterpret_cast<char *>(acc) + 256) : nullptr, acc);
      if (fused) {
        // the HPWL the WA kernels add up beside the forces (the trial's read-back)
        const float c = 1e-4f;  // any coefficient: the HPWL is the pins' boxes
        launch_net_forces(d, c, c, s);
      } else {
        // the HPWL kernels of an iteration without a WA pass
        launch_wa_small(d.w, 0.0f, 0.0f, 0, s);
        if (d.w.n_tiles) k_hpwl_tiles<<<(unsigned)d.w.n_tiles, kThreadsPerBlock, 0, s>>>(d.w, acc);
        if (d.big.n_nets) k_hpwl<<<(unsigned)((d.big.n_nets + kThreadsPerBlock - 1) / kThreadsPerBlock), kThreadsPerBlock, 0, s>>>(d.big, acc);
      }
      e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaMemcpyAsync(&h, acc, sizeof h, cudaMemcpyDeviceToHost, s);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  cudaError_t e2 = cudaStreamSynchronize(s);
  if (e == cudaSuccess && e2 == cudaSuccess) *hpwl = (int64_t)h;
  return (int)(e != cudaSuccess ? e : e2);
}

int gpl_kernel_csr_from_triplets(int64_t n, int64_t nt, const int32_t *rows, const int32_t *cols, const float *vals, int64_t *row_start, int32_t *out_cols, float *out_vals, int64_t *nnz, void *stream) {
  if (n < 0 || nt < 0 || nt >= ((int64_t)1 << 32)) return (int)cudaErrorInvalidValue;  // positions are 32-bit
  IpDevice dev((cudaStream_t)stream);
  return (int)dev.csr_from_triplets(n, nt, rows, cols, vals, row_start, out_cols, out_vals, nnz);
}

// Test-only (not in include/gpl.h): both axes' assembled matrix and right-hand side for given
// instances and pins (host arrays); per axis row_start[n + 1], rhs[n] and at most cap entries.
int gpl_rules_b2b(int64_t n, const int32_t *box, const uint8_t *locked, const int64_t n_pins, const int32_t *pin_e, const int32_t *pin_inst, const uint8_t *pin_mio, const int32_t *pin_xy, int32_t n_nets, const int64_t *net_start, int32_t max_fanout, int32_t min_diff,
                  float weight_scale, int64_t cap, int64_t *row_start, int32_t *cols, float *vals, float *rhs, void *stream) {
  IpSetup s;
  s.box.assign(reinterpret_cast<const int4 *>(box), reinterpret_cast<const int4 *>(box) + n);
  s.locked.assign(locked, locked + n);
  s.clamp.assign(n, int4{});
  s.grouped.assign(n, 0);
  s.db_box.assign(n, int4{});
  s.db_size.assign(n, int2{});
  s.pin_e.assign(pin_e, pin_e + n_pins);
  s.pin_inst.assign(pin_inst, pin_inst + n_pins);
  s.pin_mio.assign(pin_mio, pin_mio + n_pins);
  s.pin_off.assign(n_pins, int2{});
  s.pin_xy.assign(reinterpret_cast<const int2 *>(pin_xy), reinterpret_cast<const int2 *>(pin_xy) + n_pins);
  s.pin_hp.assign(n_pins, 2);
  s.pin_static.assign(n_pins, int4{});
  s.net_start.assign(net_start, net_start + n_nets + 1);
  s.max_fanout = max_fanout;
  s.min_diff = min_diff;
  s.weight_scale = weight_scale;
  IpDevice dev((cudaStream_t)stream);
  IpAxisResult r[2];
  cudaError_t e = dev.upload(s);
  if (e == cudaSuccess) e = dev.assemble(r);
  for (int a = 0; a < 2 && e == cudaSuccess; a++) {
    std::vector<int64_t> st;
    std::vector<int32_t> c;
    std::vector<float> v, b;
    if ((e = dev.rows(a, st, c, v, b)) != cudaSuccess) break;
    if ((int64_t)c.size() > cap) return (int)cudaErrorInvalidValue;
    std::copy(st.begin(), st.end(), row_start + a * (n + 1));
    std::copy(c.begin(), c.end(), cols + a * cap);
    std::copy(v.begin(), v.end(), vals + a * cap);
    std::copy(b.begin(), b.end(), rhs + a * n);
  }
  return (int)e;
}

static_assert(GPL_SPMV_ROWS == kSpmvRows && GPL_SPMV_TILED == kSpmvTiled, "the C ABI's SpMV forms");

// A matrix's sliced copy: the order by length and the slice widths on the device, their
// exclusive scan here, the entries.
struct SlicedCopy {
  int64_t *starts = nullptr;
  int32_t *row = nullptr, *len = nullptr, *count = nullptr;
  int2 *ent = nullptr;
  ~SlicedCopy() {
    for (void *p : {(void *)starts, (void *)row, (void *)len, (void *)count, (void *)ent}) cudaFree(p);
  }
  cudaError_t make(CsrDev &A, cudaStream_t s) {
    const int64_t n = A.n;
    int32_t n_long = 0;
    cudaError_t e = cudaMalloc(&row, (size_t)n * sizeof(int32_t));
    if (e == cudaSuccess) e = cudaMalloc(&len, (size_t)n * sizeof(int32_t));
    if (e == cudaSuccess) e = cudaMalloc(&count, (size_t)(kSliceLenCap + 1) * sizeof(int32_t));
    if (e == cudaSuccess) e = csr_slice_order(A, row, len, count, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&n_long, count + kSliceLongRow + 1, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    const int64_t ns = (n - n_long + kSliceRows - 1) / kSliceRows;
    std::vector<int64_t> h((size_t)ns + 1, 0);
    if (e == cudaSuccess) e = cudaMalloc(&starts, (size_t)(ns + 1) * sizeof(int64_t));
    if (e == cudaSuccess) e = csr_slice_widths(n, n_long, len, starts, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), starts, (size_t)ns * sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    int64_t run = 0;
    for (int64_t k = 0; k < ns; k++) {
      const int64_t w = h[(size_t)k];
      h[(size_t)k] = run;
      run += w;
    }
    h[(size_t)ns] = run;
    e = cudaMemcpyAsync(starts, h.data(), (size_t)(ns + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMalloc(&ent, (size_t)std::max<int64_t>(run, 1) * sizeof(int2));
    if (e != cudaSuccess) return e;
    A.sl_long = n_long;
    A.sl_row = row;
    A.sl_len = len;
    A.sl_start = starts;
    e = csr_slice_fill(A, ent, s);
    A.sl_ent = ent;
    // the host's starts have been read
    cudaError_t e2 = cudaStreamSynchronize(s);
    return e != cudaSuccess ? e : e2;
  }
};

int gpl_kernel_spmv(int64_t n, const int64_t *row_start, const int32_t *cols, const float *vals, const float *x, float *y, int32_t form, void *stream) {
  CsrDev A{n, row_start, cols, vals};
  cudaStream_t s = (cudaStream_t)stream;
  if (form != kSpmvSliced || n <= 0) return (int)spmv(A, x, y, form, s);
  SlicedCopy copy;
  cudaError_t e = copy.make(A, s);
  if (e == cudaSuccess) e = spmv(A, x, y, form, s);
  cudaError_t e2 = cudaStreamSynchronize(s);
  return (int)(e != cudaSuccess ? e : e2);
}

// Test-only (not in include/gpl.h): the initial placement's pair solve in one of the SpMV's
// forms, the same matrix and right-hand side on both axes, each with its own start point and
// solution; iterations and error of each.
int gpl_rules_bicgstab_pair(int64_t n, const int64_t *row_start, const int32_t *cols, const float *vals, const float *rhs, float *x0, float *x1, int32_t max_iters, int32_t form, int32_t *iterations, float *error, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (n <= 0) return (int)cudaErrorInvalidValue;
  CsrDev A{n, row_start, cols, vals};
  SlicedCopy copy;
  cudaError_t e = form == kSpmvSliced ? copy.make(A, s) : cudaSuccess;
  if (e != cudaSuccess) return (int)e;
  const size_t bytes = (bicgstab_pair_scratch_bytes(n) + 255) / 256 * 256;
  char *mem = nullptr;
  if ((e = cudaMalloc((void **)&mem, 2 * bytes)) != cudaSuccess) return (int)e;
  const CsrDev m[2] = {A, A};
  const float *b[2] = {rhs, rhs};
  float *x[2] = {x0, x1};
  void *scratch[2] = {mem, mem + bytes};
  BicgResult r[2]{};
  e = bicgstab_solve_pair(m, b, x, max_iters, scratch, s, r, form);
  cudaError_t e2 = cudaStreamSynchronize(s);
  cudaFree(mem);
  for (int a = 0; a < 2; a++) iterations[a] = r[a].iterations, error[a] = r[a].error;
  return (int)(e != cudaSuccess ? e : e2);
}

static int bicgstab_call(int64_t n, const int64_t *row_start, const int32_t *cols, const float *vals, const float *rhs, float *x, int32_t max_iters, int32_t *iterations, float *error, SolveWait wait, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  void *scratch = nullptr;
  cudaError_t e = cudaMalloc(&scratch, bicgstab_scratch_bytes(n));
  if (e != cudaSuccess) return (int)e;
  CsrDev A{n, row_start, cols, vals};
  BicgResult r{};
  e = bicgstab_solve(A, rhs, x, max_iters, scratch, s, &r, wait);
  cudaError_t e2 = cudaStreamSynchronize(s);
  cudaFree(scratch);
  *iterations = r.iterations;
  *error = r.error;
  return (int)(e != cudaSuccess ? e : e2);
}

int gpl_kernel_bicgstab(int64_t n, const int64_t *row_start, const int32_t *cols, const float *vals, const float *rhs, float *x, int32_t max_iters, int32_t *iterations, float *error, void *stream) {
  return bicgstab_call(n, row_start, cols, vals, rhs, x, max_iters, iterations, error, SolveWait{}, stream);
}

// Test-only (not in include/gpl.h): the same with the limit of the solver's waits given.
int gpl_rules_bicgstab_wait(int64_t n, const int64_t *row_start, const int32_t *cols, const float *vals, const float *rhs, float *x, int32_t max_iters, int32_t *iterations, float *error, uint64_t wait_ns, uint64_t entry_ns, void *stream) {
  return bicgstab_call(n, row_start, cols, vals, rhs, x, max_iters, iterations, error, SolveWait{wait_ns, entry_ns}, stream);
}

int gpl_kernel_rudy(int64_t n_nets, const int32_t *boxes, int32_t die_lx, int32_t die_ly, int32_t die_ux, int32_t die_uy, int32_t cnt_x, int32_t cnt_y, int32_t tile_size, int32_t wire_width, float *demand, void *stream) {
  RudyGrid g{die_lx, die_ly, die_ux, die_uy, cnt_x, cnt_y, tile_size, wire_width};
  return (int)rudy_demand(g, n_nets, reinterpret_cast<const int4 *>(boxes), demand, (cudaStream_t)stream);
}

// ---------------------------------------------------------------- the synthetic router
struct SynthRouter {
  gpl_router_t r;
  int32_t die[4];
  int32_t tile;
  std::vector<int32_t> pitches;
  uint8_t capacity;
  std::vector<int32_t> inst_xy;   // lower-left per design instance
  std::vector<int64_t> net_iterm_start, net_bterm_start;
  std::vector<int32_t> iterm_inst, iterm_shape, bterm_box;
  std::vector<uint8_t> bterm_placed;
};

static int sr_write(void *u, int64_t n, const int32_t *loc) {
  SynthRouter *s = (SynthRouter *)u;
  for (int64_t k = 0; k < n; k++) {
    int32_t di = loc[3 * k];
    if (di < 0 || (size_t)di * 2 + 1 >= s->inst_xy.size()) return 1;
    s->inst_xy[2 * di] = loc[3 * k + 1];
    s->inst_xy[2 * di + 1] = loc[3 * k + 2];
  }
  return 0;
}
static int sr_inputs(void *u, int32_t die[4], int32_t *xg, int32_t *yg, int32_t *ts, int32_t *np, int32_t p[32]) {
  SynthRouter *s = (SynthRouter *)u;
  std::memcpy(die, s->die, sizeof s->die);
  *xg = std::max(1, (s->die[2] - s->die[0]) / s->tile);
  *yg = std::max(1, (s->die[3] - s->die[1]) / s->tile);
  *ts = s->tile;
  *np = (int32_t)std::min<size_t>(32, s->pitches.size());
  for (int i = 0; i < *np; i++) p[i] = s->pitches[i];
  return 0;
}
static int sr_cap(void *u, uint8_t *cr, int64_t n) {
  SynthRouter *s = (SynthRouter *)u;
  for (int64_t i = 0; i < n; i++) {
    cr[2 * i] = s->capacity;
    cr[2 * i + 1] = 0;
  }
  return 0;
}
static int64_t sr_boxes(void *u, int32_t *idx, int32_t *boxes, int64_t cap) {
  SynthRouter *s = (SynthRouter *)u;
  int64_t nn = (int64_t)s->net_iterm_start.size() - 1;
  if (!boxes) return nn;
  // each net's box from its own terminals: the nets in parallel
  parallel_for((size_t)std::min(nn, cap), [&](size_t n0, size_t n1) {
  for (int64_t n = (int64_t)n0; n < (int64_t)n1; n++) {
    int32_t lx = INT32_MAX, ly = INT32_MAX, ux = INT32_MIN, uy = INT32_MIN;
    for (int64_t t = s->net_iterm_start[n]; t < s->net_iterm_start[n + 1]; t++) {
      int32_t i = s->iterm_inst[t];
      const int32_t *sh = &s->iterm_shape[4 * t];
      int32_t x = s->inst_xy[2 * i], y = s->inst_xy[2 * i + 1];
      lx = std::min(lx, x + sh[0]);
      ly = std::min(ly, y + sh[1]);
      ux = std::max(ux, x + sh[2]);
      uy = std::max(uy, y + sh[3]);
    }
    for (int64_t t = s->net_bterm_start[n]; t < s->net_bterm_start[n + 1]; t++) {
      if (!s->bterm_placed[t]) continue;
      const int32_t *b = &s->bterm_box[4 * t];
      lx = std::min(lx, b[0]);
      ly = std::min(ly, b[1]);
      ux = std::max(ux, b[2]);
      uy = std::max(uy, b[3]);
    }
    idx[n] = (int32_t)n;
    boxes[4 * n] = lx;
    boxes[4 * n + 1] = ly;
    boxes[4 * n + 2] = ux;
    boxes[4 * n + 3] = uy;
  }
  });
  return std::min(nn, cap);
}

gpl_router_t *gpl_synthetic_router_create(const gpl_design_t *d, int32_t tile_size, int32_t n_pitches, const int32_t *pitches, uint8_t capacity) {
  if (tile_size <= 0) return nullptr;
  SynthRouter *s = new SynthRouter();
  std::memcpy(s->die, d->die, sizeof s->die);
  s->tile = tile_size;
  s->pitches.assign(pitches, pitches + std::max(0, n_pitches));
  s->capacity = capacity;
  s->inst_xy.resize(2 * (size_t)d->n_insts);
  for (int32_t i = 0; i < d->n_insts; i++) {
    s->inst_xy[2 * i] = d->inst_box[4 * i];
    s->inst_xy[2 * i + 1] = d->inst_box[4 * i + 1];
  }
  s->net_iterm_start.assign(d->net_iterm_start, d->net_iterm_start + d->n_nets + 1);
  s->net_bterm_start.assign(d->net_bterm_start, d->net_bterm_start + d->n_nets + 1);
  int64_t nt = s->net_iterm_start.back(), nb = s->net_bterm_start.back();
  s->iterm_inst.assign(d->iterm_inst, d->iterm_inst + nt);
  s->iterm_shape.assign(d->iterm_shape, d->iterm_shape + 4 * nt);
  s->bterm_box.assign(d->bterm_box, d->bterm_box + 4 * nb);
  s->bterm_placed.resize(nb);
  for (int64_t t = 0; t < nb; t++) s->bterm_placed[t] = d->bterm_flags[t] & GPL_BTERM_PLACED;
  s->r.user = s;
  s->r.write_locations = sr_write;
  s->r.rudy_inputs = sr_inputs;
  s->r.capacity_reduction = sr_cap;
  s->r.net_term_boxes = sr_boxes;
  return &s->r;
}

void gpl_synthetic_router_destroy(gpl_router_t *r) {
  if (r) delete (SynthRouter *)r->user;
}

}  // extern "C"
