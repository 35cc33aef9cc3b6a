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

// Partial sums, one per CTA (at most one per tile of 64 x 4 x 1 cells).  Nothing
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
// static scratch.  A warp takes 32 columns and marches down `rows` rows, so that
// a row of q is loaded once as the next row's centre and reused as south
// neighbour; three CTAs per SM stay for the whole patch and take such pieces in
// turn.  Bound by HBM latency: eight rows unrolled put the loads of eight rows
// in flight, which pays more than warps (4096^2, 537 MB: 106 us = 5.1 TB/s with
// eight rows and three CTAs; 126 with four rows and four CTAs, 156 with two and
// eight; a CTA per 64 x 4 tile with its own reduction and ticket took 210).
constexpr int NORM_WARPS = 8;
constexpr int NORM_CTAS_PER_SM = 3;
template <int D>
__global__ void __launch_bounds__(32 * NORM_WARPS, NORM_CTAS_PER_SM)
    k_resid_norm_noalloc(DevPatch P, const double* __restrict__ fbase, int64_t fsy,
                         int64_t fsz, int64_t fcomp, int nseg, int nchunk, int rows,
                         int64_t pieces, double* __restrict__ scratch) {
  next_may_launch();
  const int lane = threadIdx.x & 31;
  double acc = 0.0;
  for (int64_t w = (int64_t)blockIdx.x * NORM_WARPS + (threadIdx.x >> 5); w < pieces;
       w += (int64_t)gridDim.x * NORM_WARPS) {
    const int64_t chunks = w / nseg;
    const int seg = (int)(w - chunks * nseg);
    const int plane = (int)(chunks / nchunk);
    const int j0 = (int)(chunks - (int64_t)plane * nchunk) * rows + 1;
    const int j1 = min(j0 + rows - 1, P.n[1]);
    const int i = seg * 32 + lane + 1, k = D == 3 ? plane + 1 : 0;
    const int ii = min(i, P.n[0]);  // lanes beyond the row add nothing
    const double* q0 = static_cast<const double*>(P.q[0]) + cidx(P, ii, j0, k);
    const double* q1 = static_cast<const double*>(P.q[1]) + cidx(P, ii, j0, k);
    const double* f = fbase + (int64_t)(ii - 1) + (int64_t)(j0 - 1) * fsy +
                      (int64_t)(D == 3 ? plane : 0) * fsz;
    double sum = 0.0;
    double ps = q0[-P.sy], pc = q0[0], ms = q1[-P.sy], mc = q1[0];
#pragma unroll 8
    for (int j = j0; j <= j1; ++j) {
      Problem::Stencil<double, D> s;
      s.pc = pc;
      s.mc = mc;
      s.pm[0] = q0[-1];
      s.pp[0] = q0[1];
      s.mm[0] = q1[-1];
      s.mp[0] = q1[1];
      s.pm[1] = ps;
      s.pp[1] = q0[P.sy];
      s.mm[1] = ms;
      s.mp[1] = q1[P.sy];
      if (D == 3) {
        s.pm[D - 1] = q0[-P.sz];
        s.pp[D - 1] = q0[P.sz];
        s.mm[D - 1] = q1[-P.sz];
        s.mp[D - 1] = q1[P.sz];
      }
      double o0, o1;
      Problem::OperatorCell<double, D>(s, P.tmp1, P.tmp2, P.alpha, o0, o1);
      const double r0 = f[0] - o0, r1 = f[fcomp] - o1;
      sum += r0 * r0 + r1 * r1;
      ps = pc;
      ms = mc;
      pc = s.pp[1];
      mc = s.mp[1];
      q0 += P.sy;
      q1 += P.sy;
      f += fsy;
    }
    if (i <= P.n[0]) acc += sum;
  }
  const double bs = block_sum(acc);
  if (threadIdx.x == 0) scratch[blockIdx.x] = bs;
}

// The sum of the partials, in index order by BLOCK_THREADS strided sums, and the
// norm.  A launch of its own, which overlaps the one before it: a ticket that
// the last CTA to finish recognises itself by would have to outlive the call or be
// cleared by every one.
__global__ void __launch_bounds__(BLOCK_THREADS)
    k_norm_total(const double* scratch, int count, double denom, double* __restrict__ out) {
  after_previous();
  double s = 0.0;
  for (int b = threadIdx.x; b < count; b += BLOCK_THREADS) s += __ldcg(scratch + b);
  const double total = block_sum(s);
  if (threadIdx.x == 0) {
    out[0] = sqrt(total / denom);
    out[1] = total;
  }
}

template <int D, class... A>
cudaError_t launch_norm(unsigned ctas, cudaStream_t s, double* scratch, double denom, double* out,
                        A... args) {
  k_resid_norm_noalloc<D><<<ctas, 32 * NORM_WARPS, 0, s>>>(args..., scratch);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(1);
  cfg.blockDim = dim3(BLOCK_THREADS);
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, k_norm_total, (const double*)scratch, (int)ctas, denom, out);
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
    const int64_t nseg = (n[0] + 31) / 32;
    // Rows per piece: 16 where that still gives every resident warp one, fewer
    // (down to a tile's 4) on small patches.
    constexpr int64_t kCtas = 148 * NORM_CTAS_PER_SM;
    const int64_t rows = std::max<int64_t>(
        4, std::min<int64_t>(16, nseg * n[1] * n[2] / (kCtas * NORM_WARPS)));
    const int64_t nchunk = (n[1] + rows - 1) / rows;
    const int64_t pieces = nseg * nchunk * n[2];
    const int64_t ctas = std::min<int64_t>(kCtas, (pieces + NORM_WARPS - 1) / NORM_WARPS);
    auto launch = [&](auto dim) {
      return launch_norm<decltype(dim)::value>((unsigned)ctas, s, scratch, denom, out, P, f, fsy,
                                               fsz, fcomp, (int)nseg, (int)nchunk, (int)rows,
                                               pieces);
    };
    const cudaError_t e = ndims == 2 ? launch(std::integral_constant<int, 2>{})
                                     : launch(std::integral_constant<int, 3>{});
    if (e != cudaSuccess) rc = BSAM_ERR_CUDA;
  }
  cudaSetDevice(prev);
  return rc;
}
