// bsam_noalloc.cu -- residual norm of one patch without any device allocation.
//
// Some callers cannot allocate device memory when they need this number: a
// host whose device memory is already handed to its own pool (for example a
// Fortran code with one preallocated arena, or PyTorch's caching allocator
// holding the free memory), or a time-step loop that must not pay the
// implicit device-wide synchronisation of cudaMalloc/cudaFree.  For them,
// bsam_gpu_resid_norm_noalloc computes the ErrorAFAS residual norm
// (errortype 1, lib/afasroutines.f90:108-221) of fields that live in the
// caller's own device memory, using a fixed scratch array compiled into the
// library instead of allocated storage.
//
// Scratch: g_noalloc_scratch below, a file-scope __device__ array.  Every GPU
// that loads this library holds it (512 KiB) until the process
// exits.  All calls share it, so calls whose kernels overlap on the GPU (two
// host threads, or two streams without ordering between them) race on it and
// give wrong results; order such calls on one stream.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "../../include/bsam_gpu.h"
#include "bsam_types.h"
#include "kernels.cuh"

using namespace bsam;

namespace {

// Partial sums, one per tile of 64 x 4 x 1 cells.  Nothing
// in it is carried from one call to the next: a call whose kernels overlapped
// another's spoils no later one.
constexpr int NOALLOC_MAX_TILES = BSAM_NOALLOC_MAX_TILES;

static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_MAX_TILES];
static_assert(sizeof(g_noalloc_scratch) <= 512 * 1024,
              "the scratch array is meant to stay at 512 KiB");

// Device address of g_noalloc_scratch per device.  In host code the symbol
// name is only a host-side stand-in, never a device address, so the address
// is looked up once per device with cudaGetSymbolAddress.
constexpr int kMaxDevices = 64;
std::mutex g_setup_mutex;
double* g_scratch_addr[kMaxDevices] = {nullptr};

int scratch_for_device(int device, double** out) {
  if (device < 0 || device >= kMaxDevices) return BSAM_ERR_NODEVICE;
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (!g_scratch_addr[device]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p)
      return BSAM_ERR_CUDA;
    g_scratch_addr[device] = static_cast<double*>(p);
  }
  *out = g_scratch_addr[device];
  return BSAM_OK;
}

// ErrorAFAS's norm over the caller's Fortran-layout arrays, reduced through the
// static scratch in the solver's order (resid_rows, kernels.cuh), so that the norm
// is the solver's bit for bit: per row of a tile each lane's two cells, a tree over
// the lanes, then the rows; the tiles' sums by k_norm_total.
//
// A warp takes the 64 columns of a tile and marches down `rows` rows (whole tiles),
// so that a row of q is loaded once as the next row's centre and reused as south
// neighbour; two CTAs per SM stay for the whole patch and take such pieces in turn.
// Lane l holds columns l and l + 32, which keeps every load whole lines; the tree's
// pairs (columns 2m, 2m + 1) then meet across neighbouring lanes, its lanes m and
// m + 16 within one.  Bound by HBM latency: a tile's four rows of two columns
// unrolled keep their loads in flight, for which a thread needs 128 registers (4096^2,
// 537 MB: 100 us = 5.3 TB/s with two CTAs per SM; 120 with three of 80
// registers or four of 64.  128^3 18.6 against 25, 256^3 120 against 252.  Warps of
// 32 columns with sums in an order of their own took 113, 23 and 167.)
constexpr int NORM_WARPS = 8;
constexpr int NORM_CTAS_PER_SM = 2;
template <int D>
__global__ void __launch_bounds__(32 * NORM_WARPS, NORM_CTAS_PER_SM)
    k_resid_norm_noalloc(DevPatch P, const double* __restrict__ fbase, int64_t fsy,
                         int64_t fsz, int64_t fcomp, int nseg, int nchunk, int rows,
                         int64_t pieces, int tiles_y, double* __restrict__ scratch) {
  next_may_launch();
  const int lane = threadIdx.x & 31;
  constexpr unsigned FULL = 0xffffffffu;
  for (int64_t w = (int64_t)blockIdx.x * NORM_WARPS + (threadIdx.x >> 5); w < pieces;
       w += (int64_t)gridDim.x * NORM_WARPS) {
    const int64_t chunks = w / nseg;
    const int seg = (int)(w - chunks * nseg);
    const int plane = (int)(chunks / nchunk);
    const int j0 = (int)(chunks - (int64_t)plane * nchunk) * rows + 1;
    const int j1 = min(j0 + rows - 1, P.n[1]);
    const int k = D == 3 ? plane + 1 : 0;
    const int i = seg * TILE_X + lane + 1;
    const bool on[2] = {i <= P.n[0], i + 32 <= P.n[0]};
    const double* q0 = static_cast<const double*>(P.q[0]) + cidx(P, i, j0, k);
    const double* q1 = static_cast<const double*>(P.q[1]) + cidx(P, i, j0, k);
    const double* f = fbase + (int64_t)(i - 1) + (int64_t)(j0 - 1) * fsy +
                      (int64_t)(D == 3 ? plane : 0) * fsz;
    // Lanes beyond the row load nothing and add nothing.
    auto ld = [&](const double* p, int h) { return on[h] ? p[32 * h] : 0.0; };
    double ps[2], pc[2], ms[2], mc[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      ps[h] = ld(q0 - P.sy, h);
      pc[h] = ld(q0, h);
      ms[h] = ld(q1 - P.sy, h);
      mc[h] = ld(q1, h);
    }
    int64_t tile = ((int64_t)plane * tiles_y + (j0 - 1) / TILE_Y) * nseg + seg;
    // The squares of row r of the current tile; the pointers move on.
    auto row = [&](double (&v)[2]) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        Problem::Stencil<double, D> s;
        s.pc = pc[h];
        s.mc = mc[h];
        s.pm[0] = ld(q0 - 1, h);
        s.pp[0] = ld(q0 + 1, h);
        s.mm[0] = ld(q1 - 1, h);
        s.mp[0] = ld(q1 + 1, h);
        s.pm[1] = ps[h];
        s.pp[1] = ld(q0 + P.sy, h);
        s.mm[1] = ms[h];
        s.mp[1] = ld(q1 + P.sy, h);
        if (D == 3) {
          s.pm[D - 1] = ld(q0 - P.sz, h);
          s.pp[D - 1] = ld(q0 + P.sz, h);
          s.mm[D - 1] = ld(q1 - P.sz, h);
          s.mp[D - 1] = ld(q1 + P.sz, h);
        }
        double o0, o1;
        Problem::OperatorCell<double, D>(s, P.tmp1, P.tmp2, P.alpha, o0, o1);
        const double r0 = ld(f, h) - o0, r1 = ld(f + fcomp, h) - o1;
        v[h] = on[h] ? r0 * r0 + r1 * r1 : 0.0;
        ps[h] = pc[h];
        ms[h] = mc[h];
        pc[h] = s.pp[1];
        mc[h] = s.mp[1];
      }
      q0 += P.sy;
      q1 += P.sy;
      f += fsy;
    };
    for (int jt = j0; jt <= j1; jt += TILE_Y, tile += nseg) {
      double v[TILE_Y][2] = {};
      if (jt + TILE_Y - 1 <= j1) {  // without conditions between the rows' loads
#pragma unroll
        for (int r = 0; r < TILE_Y; ++r) row(v[r]);
      } else {
#pragma unroll
        for (int r = 0; r < TILE_Y - 1; ++r)
          if (jt + r <= j1) row(v[r]);
      }
      double sum = 0.0;
#pragma unroll
      for (int r = 0; r < TILE_Y; ++r) {
        // Lane 2m: the sums of pairs m and m + 16, then the tree's further levels.
        const double a = v[r][0] + __shfl_xor_sync(FULL, v[r][0], 1);
        const double b = v[r][1] + __shfl_xor_sync(FULL, v[r][1], 1);
        double s = a + b;
#pragma unroll
        for (int o = 16; o > 1; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
        sum += s;
      }
      if (lane == 0) scratch[tile] = sum;
    }
  }
}

// The sum of the tiles' sums in the solver's order (last_block_sum, kernels.cuh:
// BLOCK_THREADS strided sums in index order, then block_sum), and the norm.  A
// launch of its own, which overlaps the one before it: a ticket that the last CTA
// to finish recognises itself by would have to outlive the call or be cleared by
// every one.  Up to TOTAL_FEW tiles by one CTA whose threads load all they add at
// once (256^2: 6.4 us a call against 6.9 with the cluster below).
constexpr int TOTAL_FEW = 16 * BLOCK_THREADS;
__global__ void __launch_bounds__(BLOCK_THREADS)
    k_norm_total_few(const double* scratch, int count, double denom, double* __restrict__ out) {
  after_previous();
  double v[TOTAL_FEW / BLOCK_THREADS], s = 0.0;
#pragma unroll
  for (int u = 0; u < TOTAL_FEW / BLOCK_THREADS; ++u) {
    const int at = threadIdx.x + u * BLOCK_THREADS;
    v[u] = at < count ? __ldcg(scratch + at) : 0.0;
  }
#pragma unroll
  for (int u = 0; u < TOTAL_FEW / BLOCK_THREADS; ++u) s += v[u];
  const double total = block_sum(s);
  if (threadIdx.x == 0) {
    out[0] = sqrt(total / denom);
    out[1] = total;
  }
}

// More tiles by a cluster: each CTA loads all that its TOTAL_SUMS strided sums need
// at once and adds it from shared memory.
constexpr int TOTAL_CTAS = 8, TOTAL_SUMS = BLOCK_THREADS / TOTAL_CTAS;
constexpr int TOTAL_THREADS = 512, TOTAL_ROWS = TOTAL_THREADS / TOTAL_SUMS;
constexpr int TOTAL_LOADS = NOALLOC_MAX_TILES / BLOCK_THREADS / TOTAL_ROWS;  // a thread
constexpr int TOTAL_ROUNDS = 2;                                              // of shared memory
__global__ void __cluster_dims__(TOTAL_CTAS, 1, 1) __launch_bounds__(TOTAL_THREADS)
    k_norm_total(const double* scratch, int count, double denom, double* __restrict__ out) {
  __shared__ double part[TOTAL_LOADS / TOTAL_ROUNDS * TOTAL_ROWS][TOTAL_SUMS];
  __shared__ double sums[BLOCK_THREADS];
  const int lane = threadIdx.x % TOTAL_SUMS, row = threadIdx.x / TOTAL_SUMS;
  const int first = blockIdx.x * TOTAL_SUMS + lane;
  after_previous();
  double v[TOTAL_LOADS];
#pragma unroll
  for (int u = 0; u < TOTAL_LOADS; ++u) {
    const int at = first + (u * TOTAL_ROWS + row) * BLOCK_THREADS;
    v[u] = at < count ? __ldcg(scratch + at) : 0.0;
  }
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < TOTAL_ROUNDS; ++k) {
    constexpr int U = TOTAL_LOADS / TOTAL_ROUNDS;
    if (k > 0) __syncthreads();
#pragma unroll
    for (int u = 0; u < U; ++u) part[u * TOTAL_ROWS + row][lane] = v[k * U + u];
    __syncthreads();
    const int left = (count + BLOCK_THREADS - 1) / BLOCK_THREADS - k * U * TOTAL_ROWS;
    const int n = min(left, U * TOTAL_ROWS);
    if (row == 0)
#pragma unroll 16
      for (int r = 0; r < n; ++r) s += part[r][lane];
  }
  if (row == 0) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(&sums[first]);
    uint32_t at;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(at) : "r"(a));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(s) : "memory");
  }
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
  if (blockIdx.x != 0) return;
  // block_sum of BLOCK_THREADS threads.
  __shared__ double red[BLOCK_THREADS / 32];
  if (threadIdx.x < BLOCK_THREADS) {
    double x = sums[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double total = 0.0;
    for (int w = 0; w < BLOCK_THREADS / 32; ++w) total += red[w];
    out[0] = sqrt(total / denom);
    out[1] = total;
  }
}

template <int D, class... A>
cudaError_t launch_norm(unsigned ctas, int tiles, cudaStream_t s, double* scratch, double denom, double* out,
                        A... args) {
  k_resid_norm_noalloc<D><<<ctas, 32 * NORM_WARPS, 0, s>>>(args..., scratch);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  const bool few = tiles <= TOTAL_FEW;
  cfg.gridDim = dim3(few ? 1 : TOTAL_CTAS);
  cfg.blockDim = dim3(few ? BLOCK_THREADS : TOTAL_THREADS);
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, few ? k_norm_total_few : k_norm_total, (const double*)scratch, tiles, denom, out);
  return cudaGetLastError();
}

}  // namespace

extern "C" int bsam_gpu_resid_norm_noalloc(int device, int ndims, const int32_t* mx, double dx,
                                           double dt, double eps, double alpha, const double* q,
                                           const double* f, double* out, void* stream) {
  if ((ndims != 2 && ndims != 3) || !mx || !q || !f || !out || !(dx > 0.0))
    return BSAM_ERR_ARG;
  int64_t n[3] = {1, 1, 1};
  for (int d = 0; d < ndims; ++d) {
    if (mx[d] <= 0) return BSAM_ERR_ARG;
    n[d] = mx[d];
  }
  const int64_t tiles_x = (n[0] + TILE_X - 1) / TILE_X;
  const int64_t tiles_y = (n[1] + TILE_Y - 1) / TILE_Y;
  const int64_t tiles = tiles_x * tiles_y * n[2];
  if (tiles > NOALLOC_MAX_TILES) return BSAM_ERR_TOO_LARGE;

  int prev = -1;
  if (cudaGetDevice(&prev) != cudaSuccess) return BSAM_ERR_NODEVICE;
  if (cudaSetDevice(device) != cudaSuccess) return BSAM_ERR_NODEVICE;
  double* scratch = nullptr;
  int rc = scratch_for_device(device, &scratch);
  if (rc == BSAM_OK) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    DevPatch P{};
    P.ndims = ndims;
    for (int d = 0; d < 3; ++d) P.n[d] = (int32_t)n[d];
    P.sy = n[0] + 2;
    P.sz = ndims == 3 ? (n[0] + 2) * (n[1] + 2) : 0;
    const int64_t qcomp = (n[0] + 2) * (n[1] + 2) * (ndims == 3 ? n[2] + 2 : 1);
    P.q[0] = const_cast<double*>(q);
    P.q[1] = const_cast<double*>(q) + qcomp;
    // Operator constants computed as in problem.f90:246-248.
    const double h2 = dx * dx;
    P.h = dx;
    P.alpha = alpha;
    P.tmp1 = dt / h2;
    P.tmp2 = eps * eps / h2;
    const double denom = (double)(2 * n[0] * n[1] * n[2]);
    const int64_t fsy = n[0], fsz = n[0] * n[1], fcomp = n[0] * n[1] * n[2];
    const int64_t nseg = tiles_x;
    // Rows per piece, whole tiles: those for which the warps, each at its share of
    // the pieces, take the fewest rows (the row above a piece is loaded again).
    const int64_t kCtas = B200_SMS * NORM_CTAS_PER_SM;
    int64_t rows = TILE_Y, least = INT64_MAX;
    for (int64_t r = TILE_Y; r <= 32 * TILE_Y; r += TILE_Y) {
      const int64_t all = nseg * ((n[1] + r - 1) / r) * n[2];
      const int64_t cost = (all + kCtas * NORM_WARPS - 1) / (kCtas * NORM_WARPS) * (r + 1);
      if (cost < least) {
        least = cost;
        rows = r;
      }
    }
    const int64_t nchunk = (n[1] + rows - 1) / rows;
    const int64_t pieces = nseg * nchunk * n[2];
    const int64_t ctas = std::min<int64_t>(kCtas, (pieces + NORM_WARPS - 1) / NORM_WARPS);
    auto launch = [&](auto dim) {
      return launch_norm<decltype(dim)::value>((unsigned)ctas, (int)tiles, s, scratch, denom, out, P, f, fsy,
                                               fsz, fcomp, (int)nseg, (int)nchunk, (int)rows,
                                               pieces, (int)tiles_y);
    };
    const cudaError_t e = ndims == 2 ? launch(std::integral_constant<int, 2>{})
                                     : launch(std::integral_constant<int, 3>{});
    if (e != cudaSuccess) rc = BSAM_ERR_CUDA;
  }
  cudaSetDevice(prev);
  return rc;
}
