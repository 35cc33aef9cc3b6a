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
// unrolled keep their loads in flight, for which a thread needs 128 registers
// (4096^2, 537 MB: 92 us = 5.8 TB/s; with pieces of 16 rows 100, and then with three
// CTAs per SM of 80 registers or four of 64 120.  128^3 17.9, 256^3 128.  Warps of 32
// columns with sums in an order of their own took 113, 23 and 167.)
constexpr int NORM_WARPS = 8;
constexpr int NORM_CTAS_PER_SM = 2;

struct NormArgs {
  const double *q0, *q1, *f;  // element (0, 0, 0) of q's components, (1, 1, 1) of f's first
  int64_t sy, sz, fsy, fsz, fcomp;
  double tmp1, tmp2, alpha;
  int64_t pieces;
  int n0, n1, nseg, nchunk, rows, tiles_y;
};

// Piece w: its tiles' sums go to out(tile, sum), by lane 0.
template <int D, class Out>
__device__ __forceinline__ void norm_piece(const NormArgs& P, int64_t w, Out&& out) {
  const int lane = threadIdx.x & 31;
  constexpr unsigned FULL = 0xffffffffu;
  const int64_t chunks = w / P.nseg;
  const int seg = (int)(w - chunks * P.nseg);
  const int plane = (int)(chunks / P.nchunk);
  const int j0 = (int)(chunks - (int64_t)plane * P.nchunk) * P.rows + 1;
  const int j1 = min(j0 + P.rows - 1, P.n1);
  const int k = D == 3 ? plane + 1 : 0;
  const int i = seg * TILE_X + lane + 1;
  const bool on[2] = {i <= P.n0, i + 32 <= P.n0};
  const int64_t c = i + j0 * P.sy + (D == 3 ? k * P.sz : 0);
  const double *q0 = P.q0 + c, *q1 = P.q1 + c;
  const double* f = P.f + (i - 1) + (j0 - 1) * P.fsy + (D == 3 ? plane * P.fsz : 0);
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
  int64_t tile = ((int64_t)plane * P.tiles_y + (j0 - 1) / TILE_Y) * P.nseg + seg;
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
      const double r0 = ld(f, h) - o0, r1 = ld(f + P.fcomp, h) - o1;
      v[h] = on[h] ? r0 * r0 + r1 * r1 : 0.0;
      ps[h] = pc[h];
      ms[h] = mc[h];
      pc[h] = s.pp[1];
      mc[h] = s.mp[1];
    }
    q0 += P.sy;
    q1 += P.sy;
    f += P.fsy;
  };
  for (int jt = j0; jt <= j1; jt += TILE_Y, tile += P.nseg) {
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
    if (lane == 0) out(tile, sum);
  }
}

template <int D>
__global__ void __launch_bounds__(32 * NORM_WARPS, NORM_CTAS_PER_SM)
    k_resid_norm_noalloc(const NormArgs P, double* __restrict__ scratch) {
  next_may_launch();
  for (int64_t w = (int64_t)blockIdx.x * NORM_WARPS + (threadIdx.x >> 5); w < P.pieces;
       w += (int64_t)gridDim.x * NORM_WARPS)
    norm_piece<D>(P, w, [&](int64_t tile, double sum) { scratch[tile] = sum; });
}

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}
// Stores into the cluster's first CTA, at the place of this CTA's own `p`.
__device__ __forceinline__ void store_first(double* p, double v) {
  uint32_t at;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(p)));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}

// block_sum of BLOCK_THREADS threads by the first of a larger CTA, then the norm.
__device__ __forceinline__ void norm_out(double x, double denom, double* out) {
  __shared__ double red[BLOCK_THREADS / 32];
  if (threadIdx.x < BLOCK_THREADS) {
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

// Patches of at most a tile per warp by one cluster in one launch, the tiles' sums in
// its first CTA's shared memory: such a call is bound by the host, where a second
// launch costs 2 us (101 x 200 from Python 9.7 us a call against 11.6; 309 x 105, 135
// tiles, takes 8.3 us on the device this way and 6.8 by two launches).
constexpr int SMALL_CTAS = 8, SMALL_THREADS = 512, SMALL_WARPS = SMALL_CTAS * SMALL_THREADS / 32;
constexpr int SMALL_TILES = 128;
template <int D>
__global__ void __cluster_dims__(SMALL_CTAS, 1, 1) __launch_bounds__(SMALL_THREADS, 1)
    k_norm_small(const NormArgs P, int tiles, double denom, double* __restrict__ out) {
  __shared__ double part[SMALL_TILES];
  cluster_arrive();
  cluster_wait();  // every CTA of the cluster runs: its memory may be written
  for (int64_t w = (int64_t)blockIdx.x * (SMALL_THREADS / 32) + (threadIdx.x >> 5); w < P.pieces;
       w += SMALL_WARPS)
    norm_piece<D>(P, w, [&](int64_t tile, double sum) { store_first(part + tile, sum); });
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  if (blockIdx.x != 0) return;
  double s = 0.0;
  if (threadIdx.x < BLOCK_THREADS)
    for (int b = threadIdx.x; b < tiles; b += BLOCK_THREADS) s += part[b];
  norm_out(s, denom, out);
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
  cluster_arrive();
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
  cluster_wait();  // every CTA of the cluster runs: its memory may be written
  if (row == 0) store_first(sums + first, s);
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  if (blockIdx.x == 0) norm_out(threadIdx.x < BLOCK_THREADS ? sums[threadIdx.x] : 0.0, denom, out);
}

template <int D>
cudaError_t launch_norm(const NormArgs& P, unsigned ctas, int tiles, cudaStream_t s,
                        double* scratch, double denom, double* out) {
  if (tiles <= SMALL_TILES) {
    k_norm_small<D><<<SMALL_CTAS, SMALL_THREADS, 0, s>>>(P, tiles, denom, out);
    return cudaGetLastError();
  }
  k_resid_norm_noalloc<D><<<ctas, 32 * NORM_WARPS, 0, s>>>(P, scratch);
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
  (void)cudaLaunchKernelEx(&cfg, few ? k_norm_total_few : k_norm_total, (const double*)scratch,
                           tiles, denom, out);
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
  if (prev != device && cudaSetDevice(device) != cudaSuccess) return BSAM_ERR_NODEVICE;
  double* scratch = nullptr;
  int rc = scratch_for_device(device, &scratch);
  if (rc == BSAM_OK) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    NormArgs P{};
    P.n0 = (int)n[0];
    P.n1 = (int)n[1];
    P.sy = n[0] + 2;
    P.sz = ndims == 3 ? (n[0] + 2) * (n[1] + 2) : 0;
    const int64_t qcomp = (n[0] + 2) * (n[1] + 2) * (ndims == 3 ? n[2] + 2 : 1);
    P.q0 = q;
    P.q1 = q + qcomp;
    P.f = f;
    P.fsy = n[0];
    P.fsz = n[0] * n[1];
    P.fcomp = n[0] * n[1] * n[2];
    // Operator constants computed as in problem.f90:246-248.
    const double h2 = dx * dx;
    P.alpha = alpha;
    P.tmp1 = dt / h2;
    P.tmp2 = eps * eps / h2;
    const double denom = (double)(2 * n[0] * n[1] * n[2]);
    P.nseg = (int)tiles_x;
    P.tiles_y = (int)tiles_y;
    // Rows per piece, whole tiles: as many as let the warps finish in one to four
    // pieces each, whichever takes the fewest rows (the row above a piece is loaded
    // again), at most 128.  (In 32-bit arithmetic and few steps: trying every size took
    // the host a microsecond.)
    constexpr int kCtas = B200_SMS * NORM_CTAS_PER_SM;
    const int warps = tiles <= SMALL_TILES ? SMALL_WARPS : kCtas * NORM_WARPS;
    const int columns = (int)(tiles_x * n[2]);
    int least = 0;
    for (int turns = 1; turns <= 4; ++turns) {
      const int chunks = std::max(1, turns * warps / columns);
      const int r = std::min(32, ((int)tiles_y + chunks - 1) / chunks) * TILE_Y;
      const int at = ((int)n[1] + r - 1) / r * columns;
      const int cost = (at + warps - 1) / warps * (r + 1);
      if (turns > 1 && cost >= least) continue;
      least = cost;
      P.rows = r;
      P.pieces = at;
    }
    P.nchunk = (int)(P.pieces / columns);
    const unsigned ctas =
        (unsigned)std::min<int64_t>(kCtas, (P.pieces + NORM_WARPS - 1) / NORM_WARPS);
    const cudaError_t e =
        ndims == 2 ? launch_norm<2>(P, ctas, (int)tiles, s, scratch, denom, out)
                   : launch_norm<3>(P, ctas, (int)tiles, s, scratch, denom, out);
    if (e != cudaSuccess) rc = BSAM_ERR_CUDA;
  }
  if (prev != device) cudaSetDevice(prev);
  return rc;
}
