// bsam_gpu.cu -- C ABI of the B200 FAS V-cycle (include/bsam_gpu.h).
//
// Host orchestration of the reference's MultigridIterations / AFASVcycle
// (lib/afasroutines.f90:38-106, 488-547) over the device patch table.  All
// field storage lives in one device arena per handle and stays resident
// across time steps; host arrays cross the bus only in put/get calls.
//
// Device layout of a field (one component of one patch): element (i,j,k),
// i in [0, mx1+1] etc., lives at base + i + j*sy + k*sz.  The allocation
// starts `lead` elements before element (0,0,0) so that every interior row
// (i = 1) begins on a 128-byte boundary; sy is a multiple of 128 bytes.
//
// Patch records: the caller's patches keep their indices.  The FP64 form
// runs the V-cycle on them directly.  The mixed form (mixed.cuh) appends one
// working "twin" per finest-level patch: the caller's finest patch stays the
// FP64 master state (put/get/mass/source/residual), the twin carries the
// FP32 V-cycle; levels above 4096 cells are FP32, smaller ones FP64.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <exception>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "../../include/bsam_gpu.h"
#include "bsam_types.h"
#include "kernels.cuh"
#include "smooth_fused.cuh"
#include "stage2.cuh"
#include "chain.cuh"
#include "mixed.cuh"
#include "amr.cuh"
#include "regrid.cuh"
#include "rows.cuh"
#include "stats.cuh"
#include "engine_view.h"

using namespace bsam;

namespace {

// Levels with at most this many cells per patch stay FP64 in the mixed form.
constexpr int64_t MIXED_FP64_CELLS = 4096;
// Largest level of the bottom chain where the caller asks for fused stages
// (levels above it may run them), per dimensionality.
constexpr int FUSED_BOTTOM_CELLS_2D = 1024;
constexpr int FUSED_BOTTOM_CELLS_3D = 512;
// Largest level of the bottom chain where other levels run above it.
constexpr int64_t CHAIN_TOP_CELLS_2D = 128 * 128;
constexpr int64_t CHAIN_TOP_CELLS_3D = 16384;

constexpr int MAX_GRID_Y = 65535;

struct LevelPlan {
  int level = 0;
  std::vector<int> patches;  // records the V-cycle runs on (ApplyOnLevel order)
  Item* d_fine = nullptr;    // tiles over each patch's interior
  int nfine = 0;
  Item* d_coarse = nullptr;  // tiles over each patch's footprint in its parent
  Item* d_corr = nullptr;    // tiles over each patch's blocks for the correction
  int ncoarse = 0;
  int ncorr = 0;
  Item* d_fused = nullptr;   // fused-stage tiles (tile x, tile y, z chunk)
  int nfused = 0;
  bool fused = false;
  int prec = PREC_F64;
  // AMR levels (above the root): SetGhost is coarse-fine interpolation +
  // sibling exchange + SetBC, over the level's patch list.
  bool amr = false;
  int* d_plist = nullptr;       // the level's patches
  int nplist = 0;
  OverlapCopy* d_ovl = nullptr; // GhostOverlap transfers (ApplyOnLevelPairs order)
  int novl = 0;
  // The same transfers grouped by destination, and per entry of d_plist the
  // {first, count} of its group (the one-launch SetGhost of 2D levels).
  OverlapCopy* d_ovl_by_dst = nullptr;
  int2* d_ovl_range = nullptr;
  // Parent of a refined level: its children do not cover it, so the
  // snapshot qs is a full copy of q taken after restriction + SetGhost.
  bool snap = false;
  CopySpan* d_snap = nullptr;  // the copies of its parent patches
  int nsnap = 0;
  int64_t snap_max = 0;
};

}  // namespace

struct bsam_gpu {
  int device = 0;
  cudaStream_t stream = nullptr;
  bsam_run_params rp{};
  bool have_hierarchy = false;
  bool mixed = false;
  int minlevel = 0, finestlevel = 0;
  int nuser = 0;                     // caller's patches: records [0, nuser)
  std::vector<bsam_patch_desc> desc;
  std::vector<DevPatch> hp;
  std::vector<int64_t> field_elems;  // elements per field allocation, per record
  DevPatch* d_patches = nullptr;
  char* d_arena = nullptr;
  size_t arena_bytes = 0;
  // The stash: copies of the q of every refined patch, taken by
  // bsam_gpu_stash (old grids as TransferValues reads them), with records
  // whose q pointers point into it.
  char* d_stash = nullptr;
  size_t stash_cap = 0;
  // The hierarchy's tables (records, work lists, patch lists, overlap copies,
  // copy spans, tensor maps, partial sums) in one device buffer, grown and
  // never shrunk, filled by one copy from a host image per set_hierarchy.
  char* d_meta = nullptr;
  size_t meta_cap = 0;
  std::vector<unsigned char> meta_host;
  // The arena a regrid released, kept for the next hierarchy of no larger
  // size (regridding every step alternates between two arenas).
  char* spare_arena = nullptr;
  size_t spare_bytes = 0;
  bool regridding = false;  // set_hierarchy called by bsam_gpu_regrid
  // Task lists of bsam_gpu_regrid and bsam_gpu_errflags_level (grown, never
  // shrunk; both synchronise before returning, so one buffer serves both).
  char* d_regrid = nullptr;
  size_t regrid_cap = 0;
  std::vector<unsigned char> regrid_host;
  // Page-locked bounce buffer (grown, never shrunk) for the handle's copies
  // from and to pageable host memory; every user synchronises the stream
  // before the buffer is written again.
  void* h_pin = nullptr;
  size_t pin_cap = 0;
  bool pin_busy = false;       // queued work still reads it (a put_field)
  // put / get of large fields: a piece's slot is free / full; streams of host threads.
  cudaEvent_t slot_ev[8] = {};
  cudaStream_t copy_streams[3] = {};
  bool attrs_set = false;      // the fused kernels' shared-memory attributes
  uint8_t* d_flags = nullptr;  // bsam_gpu_errflags_level's device flags
  int32_t* d_sat = nullptr;    // bsam_gpu_tag_level's summed-area tables
  size_t sat_cap = 0;
  CopySpan* d_qold_spans = nullptr;  // CopyQToQold: q -> qold of every patch that has qold
  int nqold_spans = 0;
  int64_t qold_span_max = 0;
  // SetBC at and below the root: the FP64 state patches, by level (entry l -
  // minlevel of setbc_first: where level l starts), and the largest one's cells.
  int* d_setbc = nullptr;
  std::vector<int> setbc_first;
  int64_t setbc_cells = 1;
  CopySpan* d_stash_spans = nullptr;
  size_t stash_spans_cap = 0;
  size_t flags_cap = 0;
  std::vector<DevPatch> stash_hp;
  std::vector<bsam_patch_desc> stash_desc;
  std::vector<LevelPlan> levels;     // index level - minlevel
  std::vector<int> masters;          // finest-level state patches
  Item* d_master = nullptr;          // tiles over the masters
  Item* d_state = nullptr;           // tiles over every state patch on levels >= 0
  int nstate = 0;
  Item* d_root = nullptr;            // tiles over the root patch (mass)
  int nroot = 0;
  bool amr = false;                  // levels above the root exist
  int* d_plist = nullptr;            // patch lists of the refined levels
  OverlapCopy* d_ovl = nullptr;      // their GhostOverlap transfers
  // Host copies of the refined levels' patch lists and transfers grouped by
  // destination, with per level the span of each (engine_view).
  std::vector<int> h_plist;
  std::vector<OverlapCopy> h_ovl_by_dst;
  std::vector<int2> h_ovl_range;
  std::vector<std::pair<int, int>> h_span_plist, h_span_ovl;
  int nmaster = 0;
  Item* d_items = nullptr;
  CUtensorMap* d_tmaps = nullptr;    // TMA maps of the fused levels' fields
  double* d_partials = nullptr;
  int max_items = 0;
  int* d_err = nullptr;  // kernel error flag (bounded waits that gave up)
  // Fused stages off by default: at L2-resident sizes the per-pass kernels
  // are faster; tests and tuning switch them on.
  bsam_tuning tuning{0, 64, 0, 0, 0, {0, 0, 0}};
  int bottom_level = -1000;  // levels <= this run inside k_chain
  ChainPlan* d_chains = nullptr;  // one plan per patch of that level
  int nchains = 0, chain_ctas = 1;
  size_t chain_smem = 0;
  bool chain_loop = false;   // the chain is the whole solve: V-cycle loop in the kernel
  int max_cluster = 0;       // CTAs of the largest cluster the device runs, 0: not asked yet
  double denom = 1.0;        // nrvars * cells of the finest level (ErrorAFAS)
  cudaGraphExec_t step_exec = nullptr;  // V-cycle loop graph (built lazily)
  int graph_kernels_per_vcycle = 0;
  // The status and, behind it, the residual of every V-cycle (one copy brings
  // both back).
  DevStatus* d_status = nullptr;
  DevStatus* h_status = nullptr;  // pinned
  double* d_trace = nullptr;
  double* h_trace = nullptr;
  std::vector<double> trace;
  std::string err;
  // instrumentation
  bool profiling = false;
  bsam_gpu_stats stats{};
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ev_pool;
  size_t ev_used = 0;
  int64_t ev_cells = 0;   // cells of the finest V-cycle level
  int ev_bytes = 8;       // bytes per value on that level
};

namespace {

int fail(bsam_gpu* h, int code, const std::string& msg) {
  if (h) h->err = msg;
  return code;
}

#define CU(call)                                                                  \
  do {                                                                            \
    cudaError_t e_ = (call);                                                      \
    if (e_ != cudaSuccess)                                                        \
      return fail(h, BSAM_ERR_CUDA, std::string(__func__) + ":" + std::to_string(__LINE__) + \
                                        ": " #call ": " + cudaGetErrorString(e_));         \
  } while (0)

int64_t roundup(int64_t x, int64_t a) { return (x + a - 1) / a * a; }

size_t status_bytes(int maxvcycles) { return sizeof(DevStatus) + sizeof(double) * maxvcycles; }
static_assert(sizeof(DevStatus) % sizeof(double) == 0, "the trace follows the status");

LevelPlan& plan(bsam_gpu* h, int level) { return h->levels[level - h->minlevel]; }

// The bounce buffer with room for `bytes`.  Copies through it are DMA
// copies queued on the stream; copies from pageable memory instead pass
// through the driver's staging, which handles regridding side by side on
// several host threads contend for.
void* pin_reserve(bsam_gpu* h, size_t bytes) {
  if (h->pin_busy) {
    cudaStreamSynchronize(h->stream);
    h->pin_busy = false;
  }
  if (bytes > h->pin_cap) {
    if (h->h_pin) cudaFreeHost(h->h_pin);
    h->h_pin = nullptr;
    h->pin_cap = 0;
    const size_t want = std::max<size_t>(bytes + bytes / 2, (size_t)1 << 16);
    if (cudaMallocHost(&h->h_pin, want) != cudaSuccess) return nullptr;
    h->pin_cap = want;
  }
  return h->h_pin;
}

// Queues a host -> device copy of pageable `src` through the bounce buffer
// (the caller synchronises the stream before the buffer's next use).
int h2d_bounce(bsam_gpu* h, void* dst, const void* src, size_t bytes) {
  if (!bytes) return BSAM_OK;
  void* p = pin_reserve(h, bytes);
  if (!p) return fail(h, BSAM_ERR_NOMEM, "page-locked staging allocation failed");
  std::memcpy(p, src, bytes);
  CU(cudaMemcpyAsync(dst, p, bytes, cudaMemcpyHostToDevice, h->stream));
  return BSAM_OK;
}

// Device -> pageable host through the bounce buffer; waits for the stream.
int d2h_bounce(bsam_gpu* h, void* dst, const void* src, size_t bytes) {
  if (!bytes) return BSAM_OK;
  void* p = pin_reserve(h, bytes);
  if (!p) return fail(h, BSAM_ERR_NOMEM, "page-locked staging allocation failed");
  CU(cudaMemcpyAsync(p, src, bytes, cudaMemcpyDeviceToHost, h->stream));
  CU(cudaStreamSynchronize(h->stream));
  std::memcpy(dst, p, bytes);
  return BSAM_OK;
}

void tiles_for(int patch, const int* n, int ndims, std::vector<Item>& out) {
  const int tx = (n[0] + TILE_X - 1) / TILE_X;
  const int ty = (n[1] + TILE_Y - 1) / TILE_Y;
  const int tz = ndims == 3 ? n[2] : 1;
  for (int z = 0; z < tz; ++z)
    for (int y = 0; y < ty; ++y)
      for (int x = 0; x < tx; ++x) out.push_back(Item{patch, x, y, z});
}

dim3 block_dim() { return dim3(32, TILE_Y, 1); }

int elem_bytes(int prec) { return prec == PREC_F32 ? 4 : 8; }

// Timed finest-level smoothing stages: events are pooled and read back at
// the next host synchronisation (drain_events).
void stage_begin(bsam_gpu* h, int level) {
  if (!h->profiling || level != h->finestlevel) return;
  if (h->ev_used == h->ev_pool.size()) {
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    h->ev_pool.push_back({a, b});
  }
  cudaEventRecord(h->ev_pool[h->ev_used].first, h->stream);
}

void stage_end(bsam_gpu* h, int level) {
  if (!h->profiling || level != h->finestlevel) return;
  cudaEventRecord(h->ev_pool[h->ev_used].second, h->stream);
  ++h->ev_used;
}

void drain_events(bsam_gpu* h) {
  for (size_t e = 0; e < h->ev_used; ++e) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, h->ev_pool[e].first, h->ev_pool[e].second) == cudaSuccess) {
      h->stats.smooth_ms += ms;
      h->stats.smooth_stages += 1;
      h->stats.smooth_cells += h->ev_cells;
      h->stats.smooth_bytes += 6.0 * h->ev_bytes * (double)h->ev_cells;
    }
  }
  h->ev_used = 0;
}

// ---- typed launches -----------------------------------------------------------

// Launches a kernel that starts with after_previous(): its launch overlaps the
// kernel before it, one to two microseconds of the five that a small level's
// kernel takes.  Solves: 320 x 200 2.67 -> 2.55 ms, 512^2 mixed 4.8 -> 4.54, 96 x
// 64 x 80 mixed 8.72 -> 8.47, 128^3 16.8 -> 16.5.
template <class... P, class... A>
void launch_after(bsam_gpu* h, void (*k)(P...), dim3 grid, dim3 block, size_t smem, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = h->stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

template <class T, int D>
void launch_relax_t(bsam_gpu* h, const LevelPlan& L, int color) {
  launch_after(h, k_relax<T, D>, L.nfine, block_dim(), 0, h->d_patches, L.d_fine, color);
}

// what: 0 = RestrictSolution, 2 = CoarseLoadingFunction, 1 = CorrectFine.
template <class TC, class TP, int D>
void launch_transfer_t(bsam_gpu* h, const LevelPlan& L, int what) {
  if (what == 0)
    launch_after(h, k_restrict<TC, TP, D>, L.ncoarse, block_dim(), 0, h->d_patches, L.d_coarse);
  else if (what == 2)
    launch_after(h, k_coarse_load<TC, TP, D>, L.ncoarse, block_dim(), 0, h->d_patches, L.d_coarse);
  else
    launch_after(h, k_correct<TC, TP, D>, L.ncorr, block_dim(), 0, h->d_patches, L.d_corr);
}

// SetGhost(level, ipass) of a refined level (boundary.f90:58-89): coarse-fine
// interpolation, sibling exchange, physical faces -- one launch (a CTA per
// patch runs the three in order).
// Levels at and below the root keep their ghosts by write-through.
void amr_ghost(bsam_gpu* h, int level, int ipass) {
  if (level < h->minlevel || level > h->finestlevel) return;
  const LevelPlan& L = plan(h, level);
  if (!L.amr) return;
  if (h->rp.ndims == 2) {
    launch_after(h, k_ghost2, L.nplist, 128, 0, h->d_patches, L.d_plist, L.d_ovl_by_dst,
                 L.d_ovl_range, ipass);
  } else {
    launch_after(h, k_ghost3, L.nplist, 256, 0, h->d_patches, L.d_plist, L.d_ovl_by_dst,
                 L.d_ovl_range, ipass);
  }
  ++h->stats.launches;
}

// GetCoarseGhostPoints for the children of a partly covered level: the
// snapshot qs of every parent patch becomes a full copy of q (taken after
// restriction and SetGhost), all of them in one launch (a level of the AMR
// workload has about 40 such patches: as two copies each they were 80 graph
// nodes in a row).
void snapshot(bsam_gpu* h, int level) {
  const LevelPlan& L = plan(h, level);
  if (!L.snap) return;
  for (int first = 0; first < L.nsnap; first += MAX_GRID_Y) {
    const int n = std::min(MAX_GRID_Y, L.nsnap - first);
    launch_after(h, k_copy_spans, copy_spans_grid(L.snap_max, n), 256, 0, L.d_snap + first);
    ++h->stats.launches;
  }
}

// FillDown(solutionfield) over the refined levels (afas:223-239): each
// level's q restricted into its parent, then the parent level's SetGhost.
// Below the root the same restriction is overwritten by RestrictSolution
// before any read, so it is not issued.
void filldown(bsam_gpu* h) {
  for (int level = h->finestlevel; level >= 1; --level) {
    const LevelPlan& L = plan(h, level);
    if (h->rp.ndims == 2)
      launch_after(h, k_filldown<2>, L.ncoarse, block_dim(), 0, h->d_patches, L.d_coarse);
    else
      launch_after(h, k_filldown<3>, L.ncoarse, block_dim(), 0, h->d_patches, L.d_coarse);
    ++h->stats.launches;
    amr_ghost(h, level - 1, 0);
  }
}

template <int D>
void launch_transfer_d(bsam_gpu* h, const LevelPlan& L, int pc, int pp, int what) {
  if (pc == PREC_F32 && pp == PREC_F32) launch_transfer_t<float, float, D>(h, L, what);
  else if (pc == PREC_F32) launch_transfer_t<float, double, D>(h, L, what);
  else launch_transfer_t<double, double, D>(h, L, what);
}

// A 2D level's stage with its transfer (stage2.cuh).  Tiles of 32 x 16 where
// they give every SM two (V-cycle of 512^2 FP64 137 us against 140 with 32 x 8,
// of 1024^2 280 against 302), of 32 x 8 on smaller levels (160^2 78 against 82,
// 256^2 100 against 102).
template <class T, bool DELTA>
void launch_stage2_t(bsam_gpu* h, const LevelPlan& L, int dir) {
  const int p = L.patches[0];
  const DevPatch& P = h->hp[p];
  const unsigned tx = (unsigned)(P.n[0] + 31) / 32;
  const int upd = dir == 1 && P.master >= 0, nu = h->rp.nsmoothingpasses;
  auto tiles = [&](auto ty) {
    using S = Stage2<T, DELTA, decltype(ty)::value>;
    launch_after(h, k_stage2<T, DELTA, decltype(ty)::value>,
                 dim3(tx, (unsigned)(P.n[1] + S::TY - 1) / S::TY), S::THREADS, S::SMEM,
                 h->d_patches, p, dir, nu, upd);
  };
  if (tx * ((unsigned)(P.n[1] + 15) / 16) >= 2 * B200_SMS)
    tiles(std::integral_constant<int, 16>{});
  else tiles(std::integral_constant<int, 8>{});
  ++h->stats.launches;
}

void launch_stage2(bsam_gpu* h, const LevelPlan& L, int dir) {
  if (!h->mixed) launch_stage2_t<double, false>(h, L, dir);
  else if (L.prec == PREC_F32) launch_stage2_t<float, true>(h, L, dir);
  else launch_stage2_t<double, true>(h, L, dir);
}

// LevelRelax (afas:523-547).  dir selects the buffers of a fused level:
// 0 = pre-smoothing (q -> qb), 1 = post-smoothing (qb -> q).
void relax_level(bsam_gpu* h, int level, int dir) {
  const LevelPlan& L = plan(h, level);
  stage_begin(h, level);
  if (L.fused && h->rp.ndims == 2) {
    launch_stage2(h, L, dir);
  } else if (L.fused) {
    if (L.prec == PREC_F32)
      k_smooth3_fused<float><<<L.nfused, Fused3<float>::THREADS, Fused3<float>::SMEM, h->stream>>>(
          h->d_patches, L.d_fused, dir, 0, h->d_err);
    else
      k_smooth3_fused<double><<<L.nfused, Fused3<double>::THREADS, Fused3<double>::SMEM,
                                h->stream>>>(h->d_patches, L.d_fused, dir, 0, h->d_err);
    ++h->stats.launches;
  } else {
    for (int pass = 0; pass < h->rp.nsmoothingpasses; ++pass)
      for (int color = 0; color < 2; ++color) {
        if (h->rp.ndims == 2) {
          if (L.prec == PREC_F32) launch_relax_t<float, 2>(h, L, color);
          else launch_relax_t<double, 2>(h, L, color);
        } else {
          if (L.prec == PREC_F32) launch_relax_t<float, 3>(h, L, color);
          else launch_relax_t<double, 3>(h, L, color);
        }
        ++h->stats.launches;
        amr_ghost(h, level, color + 1);  // SetGhost(level, ipass) (afas:542)
      }
  }
  stage_end(h, level);
}

// what 0: RestrictSolution, parent SetGhost(level-1, 0), GetCoarseGhostPoints
// and CoarseLoadingFunction (afas:503-509); what 1: CorrectFine and
// SetGhost(level, 0) (afas:513-515).
void transfer(bsam_gpu* h, int level, int what) {
  const LevelPlan& L = plan(h, level);
  const int pp = plan(h, level - 1).prec;
  auto launch = [&](int w) {
    if (h->rp.ndims == 2) launch_transfer_d<2>(h, L, L.prec, pp, w);
    else launch_transfer_d<3>(h, L, L.prec, pp, w);
    ++h->stats.launches;
  };
  // A 2D fused level's stages restrict and correct it themselves.
  const bool in_stage = L.fused && h->rp.ndims == 2;
  if (what == 0) {
    if (!in_stage) launch(0);
    amr_ghost(h, level - 1, 0);
    snapshot(h, level - 1);
    launch(2);
  } else {
    if (!in_stage) launch(1);
    amr_ghost(h, level, 0);
  }
}

// The chain kernel of a handle's dimension and form.
auto chain_kernel(const bsam_gpu* h) {
  return h->rp.ndims == 2 ? (h->mixed ? k_chain<2, true> : k_chain<2, false>)
                          : (h->mixed ? k_chain<3, true> : k_chain<3, false>);
}

// The chains below and including bottom_level (chain.cuh): one V-cycle, or
// with loop.maxv > 0 MultigridIterations' whole loop.
void launch_chain(bsam_gpu* h, const ChainLoop& loop) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(h->nchains * h->chain_ctas));
  cfg.blockDim = dim3(CHAIN_THREADS);
  cfg.dynamicSmemBytes = h->chain_smem;
  cfg.stream = h->stream;
  cudaLaunchAttribute at[2]{};
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)h->chain_ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  (void)cudaLaunchKernelEx(&cfg, chain_kernel(h), (const DevPatch*)h->d_patches,
                           (const ChainPlan*)h->d_chains, loop);
  ++h->stats.launches;
}

// AFASVcycle (afas:488-521).
void vcycle(bsam_gpu* h, int level) {
  // A finest level in the chain is run as launches while its stages are timed (the
  // same bits), and with it the levels below.
  if (level == h->bottom_level && !(h->profiling && level == h->finestlevel)) {
    launch_chain(h, ChainLoop{});  // AFASVcycle(level) down to the coarsest level
    return;
  }
  relax_level(h, level, 0);  // LevelRelax (afas:499)
  if (level > h->minlevel) {
    transfer(h, level, 0);   // RestrictSolution + CoarseLoadingFunction (afas:503-509)
    vcycle(h, level - 1);    // afas:511
    transfer(h, level, 1);   // CorrectFine (afas:513)
    relax_level(h, level, 1);  // afas:517
  }
}

// ErrorAFAS on the finest level (afas:94, 108-221) into d_status.  In the
// mixed form the same FP64 norm is taken by k_defect, which also prepares
// the twins for the next FP32 V-cycle.
void launch_resid(bsam_gpu* h) {
  const int nd = h->rp.ndims;
  const dim3 b = block_dim();
  const unsigned g = (unsigned)(h->nmaster + TILE_Y - 1) / TILE_Y;
  if (!h->mixed) {
    if (nd == 2)
      launch_after(h, k_resid_norm<2>, g, b, 0, h->d_patches, h->d_master, h->d_partials,
                   h->d_status, h->nmaster, h->denom, h->rp.qerrortol);
    else
      launch_after(h, k_resid_norm<3>, g, b, 0, h->d_patches, h->d_master, h->d_partials,
                   h->d_status, h->nmaster, h->denom, h->rp.qerrortol);
  } else {
    const bool f32 = plan(h, h->finestlevel).prec == PREC_F32;
#define DEFECT(TW, D)                                                                     \
  launch_after(h, k_defect<TW, D>, g, b, 0, h->d_patches, h->d_master, h->d_partials, \
               h->d_status, h->nmaster, h->denom, h->rp.qerrortol)
    if (nd == 2) {
      if (f32) DEFECT(float, 2);
      else DEFECT(double, 2);
    } else {
      if (f32) DEFECT(float, 3);
      else DEFECT(double, 3);
    }
#undef DEFECT
  }
  ++h->stats.launches;
}

// Mixed form: q64 += q32 - fl32(q64) after the FP32 V-cycle.
void launch_update(bsam_gpu* h) {
  const int nd = h->rp.ndims;
  const LevelPlan& L = plan(h, h->finestlevel);  // the twins' tiles
  const bool f32 = L.prec == PREC_F32;
  const dim3 b = block_dim();
  if (nd == 2) {
    if (f32) launch_after(h, k_update<float, 2>, L.nfine, b, 0, h->d_patches, L.d_fine);
    else launch_after(h, k_update<double, 2>, L.nfine, b, 0, h->d_patches, L.d_fine);
  } else {
    if (f32) launch_after(h, k_update<float, 3>, L.nfine, b, 0, h->d_patches, L.d_fine);
    else launch_after(h, k_update<double, 3>, L.nfine, b, 0, h->d_patches, L.d_fine);
  }
  ++h->stats.launches;
}

// One outer iteration of MultigridIterations: V-cycle, then ErrorAFAS.
void iteration(bsam_gpu* h) {
  vcycle(h, h->finestlevel);
  // A 2D fused finest level has updated its master in its last stage.
  if (h->mixed && !(h->rp.ndims == 2 && plan(h, h->finestlevel).fused)) launch_update(h);
  if (h->amr) filldown(h);  // FillDown(solutionfield) after the V-cycle (afas:73)
  launch_resid(h);
}

// Captures the V-cycle loop of MultigridIterations (afas:69-104) as a graph
// with one conditional WHILE node whose body is one iteration + k_mg_loop;
// k_mg_loop sets the condition.  The default value 1 makes the body run at
// least once per launch, as the reference's loop does.
int build_step_graph(bsam_gpu* h) {
  cudaGraph_t g = nullptr;
  CU(cudaGraphCreate(&g, 0));
  cudaGraphConditionalHandle handle;
  cudaError_t e = cudaGraphConditionalHandleCreate(&handle, g, 1, cudaGraphCondAssignDefault);
  cudaGraphNodeParams np{};
  cudaGraphNode_t node;
  if (e == cudaSuccess) {
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = handle;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    e = cudaGraphAddNode(&node, g, nullptr, 0, &np);
  }
  if (e == cudaSuccess) {
    cudaGraph_t body = np.conditional.phGraph_out[0];
    e = cudaStreamBeginCaptureToGraph(h->stream, body, nullptr, nullptr, 0,
                                      cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      const int64_t before = h->stats.launches;
      iteration(h);
      launch_after(h, k_mg_loop, 1, 1, 0, h->d_status, h->d_trace, h->rp.maxvcycles,
                   h->rp.qerrortol, handle);
      h->graph_kernels_per_vcycle = (int)(h->stats.launches - before) + 1;
      h->stats.launches = before;
      cudaGraph_t captured = nullptr;
      e = cudaStreamEndCapture(h->stream, &captured);
    }
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&h->step_exec, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) {
    h->step_exec = nullptr;
    cudaGetLastError();
    return fail(h, BSAM_ERR_CUDA, std::string("step graph: ") + cudaGetErrorString(e));
  }
  return BSAM_OK;
}

// SetBC on the FP64 state patches of the levels from `lo` to `hi` at and below
// the root, in one launch (each reads and writes only itself) per MAX_GRID_Y of them.
void ghost_levels(bsam_gpu* h, int lo, int hi) {
  const int first = h->setbc_first[std::max(lo, h->minlevel) - h->minlevel];
  const int last = h->setbc_first[std::min(hi, 0) - h->minlevel + 1];
  for (int p = first; p < last; p += MAX_GRID_Y) {
    const dim3 g(setbc_blocks(h->rp.ndims, h->setbc_cells),
                 (unsigned)std::min(MAX_GRID_Y, last - p));
    const int* list = h->d_setbc + p;
    if (h->rp.ndims == 2)
      k_setbc_list<double, 2><<<g, SETBC_THREADS, 0, h->stream>>>(h->d_patches, list);
    else
      k_setbc_list<double, 3><<<g, SETBC_THREADS, 0, h->stream>>>(h->d_patches, list);
    ++h->stats.launches;
  }
}

int face_rule(int ndims, int face, int code, int* rule) {
  if (code == 1) {
    *rule = BC_COPY;
  } else if (code >= 10 && code <= 99) {
    // UserBC2D: faces 1,2 -> 2 - q (all vars); faces 3,4 -> copy of vars 1,2.
    // UserBC3D: every face -> 2 - q (problem.f90:646-756).
    *rule = (ndims == 2 && face >= 2) ? BC_COPY : BC_REFLECT;
  } else if (code == 999) {
    *rule = BC_NONE;
  } else if (code == 2) {
    *rule = BC_PERIODIC;  // both faces of the dimension (checked by the caller)
  } else {
    return -1;
  }
  return 0;
}

int64_t cells_of(const int* mx, int nd) {
  int64_t c = 1;
  for (int n = 0; n < nd; ++n) c *= mx[n];
  return c;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// dependency on libcuda).
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// 3D map of one field of patch P: the array from its allocation start
// (`lead` elements before element (0,0,0)), dims (sy, n1+2, n2+2), box
// (hx, hy, 1).  Returns false if the driver rejects it.
bool encode_field_map(CUtensorMap* m, const DevPatch& P, const void* field, int hx, int hy) {
  auto enc = tensor_map_encoder();
  if (!enc) return false;
  const int es = elem_bytes(P.prec);
  const int64_t lead = 128 / es - 1;
  void* base = (char*)field - lead * es;
  const cuuint64_t dims[3] = {(cuuint64_t)P.sy, (cuuint64_t)(P.n[1] + 2),
                              (cuuint64_t)(P.n[2] + 2)};
  const cuuint64_t strides[2] = {(cuuint64_t)(P.sy * es), (cuuint64_t)(P.sz * es)};
  const cuuint32_t box[3] = {(cuuint32_t)hx, (cuuint32_t)hy, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r =
      enc(m, P.prec == PREC_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
          3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

}  // namespace

namespace bsam {

int engine_view(bsam_gpu* h, EngineView& v) {
  if (!h || !h->have_hierarchy) return BSAM_ERR_STATE;
  v.ndims = h->rp.ndims;
  v.minlevel = h->minlevel;
  v.finestlevel = h->finestlevel;
  v.nsmoothingpasses = h->rp.nsmoothingpasses;
  v.maxvcycles = h->rp.maxvcycles;
  v.mixed = h->mixed;
  v.qerrortol = h->rp.qerrortol;
  v.denom = h->denom;
  v.recs = h->hp;
  v.masters = h->masters;
  v.levels.assign(h->levels.size(), EngineLevelView{});
  for (size_t li = 0; li < h->levels.size(); ++li) {
    const LevelPlan& L = h->levels[li];
    EngineLevelView& E = v.levels[li];
    E.level = L.level;
    E.amr = L.amr;
    E.snap = L.snap;
    E.patches = L.patches;
    if (!L.amr || li >= h->h_span_plist.size()) continue;
    const auto sp = h->h_span_plist[li], so = h->h_span_ovl[li];
    E.ovl.assign(h->h_ovl_by_dst.begin() + so.first,
                 h->h_ovl_by_dst.begin() + so.first + so.second);
    E.range.assign(h->h_ovl_range.begin() + sp.first,
                   h->h_ovl_range.begin() + sp.first + sp.second);
  }
  return BSAM_OK;
}

int engine_prologue(bsam_gpu* h) {
  if (!h || !h->have_hierarchy) return BSAM_ERR_STATE;
  if (h->mixed) return fail(h, BSAM_ERR_UNSUPPORTED, "the batch runs refined hierarchies in FP64");
  CU(cudaSetDevice(h->device));
  if (h->amr) filldown(h);
  if (h->rp.ndims == 2)
    k_source<double, 2><<<h->nstate, block_dim(), 0, h->stream>>>(h->d_patches, h->d_state);
  else
    k_source<double, 3><<<h->nstate, block_dim(), 0, h->stream>>>(h->d_patches, h->d_state);
  ++h->stats.launches;
  CU(cudaGetLastError());
  return BSAM_OK;
}

cudaStream_t engine_stream(bsam_gpu* h) { return h ? h->stream : nullptr; }

int engine_device(bsam_gpu* h) { return h ? h->device : -1; }

}  // namespace bsam

namespace {

// put_field / get_field of q or qold (both components, ghost ring included)
// between the caller's pageable array and the pitched fields, through page-locked
// memory: a kernel spreads the rows from it, or packs them into it, over the bus; a
// host copy does the rest.  For small fields, in the bounce buffer, that is one
// launch instead of two staged pitched copies (a 16 KB field: put 28 -> 12 us, get
// 27 -> 19).  Large fields go in pieces that a few host threads copy side by side,
// each through two slots and on a stream of its own, so that host copies, launches
// and the bus overlap.  Between the two limits the driver's pitched copies are as
// good and need no page-locked memory, which costs 1 to 2 ms per MB to allocate:
// hence as little of it as keeps the bus busy.  Against the driver's copies, in ms
// (put, get, and a whole one-shot solve: create, a step, get, destroy): 96 x 64 x 80
// (8.3 MB) 1.4 -> 0.55, 0.7 -> 0.65, 8.1 -> 7.3; 128^3 (35 MB) 4.0 -> 1.7, 1.8 to 2.6
// -> 1.7, 14 -> 14; 192^3 13 -> 5.1, 5.8 to 7.6 -> 5.1, 33 -> 27.  Long rows suit the
// driver: 1024 x 512 (8.4 MB) 0.54 -> 0.64, 0.70 -> 0.67; 2048^2 (67 MB) 6.0 -> 3.0,
// 3.3 to 3.9 -> 3.0.
constexpr size_t kBounceBytes = (size_t)128 << 10;
constexpr int kCopyThreads = 4;

// Bytes of a slot for a field of `bytes` in rows of `row`, 0: not in pieces.
size_t piece_bytes(size_t bytes, size_t row) {
  const size_t least = (size_t)(row < 4096 ? 8 : 32) << 20;
  const size_t piece = (size_t)(bytes < ((size_t)24 << 20) ? 128 : 256) << 10;
  return bytes >= least && row <= piece ? piece : 0;
}

// The page-locked blocks of large copies, for all handles of the process: a
// copy takes one and gives it back when it is done with it; up to two wait for
// the next copies, until the last handle is destroyed.
struct PieceBlocks {
  struct Block {
    void* p = nullptr;
    size_t bytes = 0;
  };
  std::mutex mutex;
  Block idle[2];
  int handles = 0;
  static PieceBlocks& get() {
    static PieceBlocks* p = new PieceBlocks;  // outlives every handle
    return *p;
  }
  Block take(size_t bytes) {
    {
      std::lock_guard<std::mutex> lock(mutex);
      for (Block& b : idle)
        if (b.bytes >= bytes) {
          const Block t = b;
          b = Block{};
          return t;
        }
    }
    Block t;
    if (cudaHostAlloc(&t.p, bytes, cudaHostAllocPortable) != cudaSuccess) return Block{};
    t.bytes = bytes;
    return t;
  }
  void give(Block t) {
    {
      std::lock_guard<std::mutex> lock(mutex);
      Block& least = idle[0].bytes <= idle[1].bytes ? idle[0] : idle[1];
      if (handles > 0 && t.bytes > least.bytes) std::swap(t, least);
    }
    if (t.p) cudaFreeHost(t.p);
  }
  void count(int d) {
    Block drop[2];
    {
      std::lock_guard<std::mutex> lock(mutex);
      handles += d;
      if (handles == 0) std::swap(drop, idle);
    }
    for (const Block& b : drop)
      if (b.p) cudaFreeHost(b.p);
  }
};

}  // namespace

extern "C" {

const char* bsam_gpu_strerror(int code) {
  switch (code) {
    case BSAM_OK: return "ok";
    case BSAM_ERR_ARG: return "invalid argument";
    case BSAM_ERR_CUDA: return "CUDA runtime error";
    case BSAM_ERR_NOMEM: return "device memory allocation failed";
    case BSAM_ERR_STATE: return "call out of order";
    case BSAM_ERR_UNSUPPORTED: return "configuration not supported";
    case BSAM_ERR_NODEVICE: return "no usable CUDA device";
    case BSAM_ERR_DIVERGED: return "non-finite residual";
    case BSAM_ERR_TOO_LARGE: return "patch exceeds the static scratch limit of the no-alloc entry point";
    default: return "unknown status";
  }
}

const char* bsam_gpu_last_error(bsam_gpu* h) { return h ? h->err.c_str() : "null handle"; }

int bsam_gpu_create(bsam_gpu** out, int device, const bsam_run_params* p) {
  bsam_gpu* h = nullptr;
  if (!out || !p) return BSAM_ERR_ARG;
  *out = nullptr;
  if (p->ndims < 2 || p->ndims > 3 || p->nrvars != 2 || p->mbc != 1 || p->maux != 0 ||
      p->errortype != 1 || p->nsmoothingpasses < 1 || p->maxvcycles < 1)
    return BSAM_ERR_UNSUPPORTED;
  if (p->precision != BSAM_PREC_FP64 && p->precision != BSAM_PREC_MIXED)
    return BSAM_ERR_UNSUPPORTED;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= device || device < 0)
    return BSAM_ERR_NODEVICE;
  h = new bsam_gpu();
  h->device = device;
  h->rp = *p;
  h->mixed = p->precision == BSAM_PREC_MIXED;
  if (cudaSetDevice(device) != cudaSuccess) {
    delete h;
    return BSAM_ERR_NODEVICE;
  }
  if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaMalloc(&h->d_status, status_bytes(p->maxvcycles)) != cudaSuccess ||
      cudaMallocHost(&h->h_status, status_bytes(p->maxvcycles)) != cudaSuccess) {
    delete h;
    return BSAM_ERR_CUDA;
  }
  cudaMemset(h->d_status, 0, sizeof(DevStatus));
  h->d_trace = reinterpret_cast<double*>(h->d_status + 1);
  h->h_trace = reinterpret_cast<double*>(h->h_status + 1);
  h->d_err = &h->d_status->kerr;
  PieceBlocks::get().count(1);
  *out = h;
  return BSAM_OK;
}

static void free_hierarchy(bsam_gpu* h) {
  // d_items, d_tmaps, d_chains, d_patches, d_partials, d_qold_spans, d_plist
  // and d_ovl point into d_meta, which the handle keeps.
  h->d_tmaps = nullptr;
  if (h->step_exec) cudaGraphExecDestroy(h->step_exec);
  if (h->d_arena) cudaFree(h->d_arena);
  h->d_qold_spans = nullptr;
  h->nqold_spans = 0;
  h->qold_span_max = 0;
  h->d_items = nullptr;
  h->d_chains = nullptr;
  h->nchains = 0;
  h->step_exec = nullptr;
  h->d_arena = nullptr;
  h->d_patches = nullptr;
  h->d_partials = nullptr;
  h->d_master = nullptr;
  h->nmaster = 0;
  h->d_state = h->d_root = nullptr;
  h->nstate = h->nroot = 0;
  h->d_plist = nullptr;
  h->d_ovl = nullptr;
  h->amr = false;
  h->levels.clear();
  h->masters.clear();
  h->hp.clear();
  h->desc.clear();
  h->field_elems.clear();
  h->have_hierarchy = false;
}

// Sets the attributes of the handle's chain kernel and returns the CTAs of the
// largest cluster of it that the device can hold (16 need a GPC with 16 free SMs,
// 8 always fit; negative: a CUDA error).  The attributes belong to the device's
// context, which a reset replaces: every handle sets its own.  The answer is the
// device's and is asked for once: the query takes milliseconds.
static int chain_cluster(const bsam_gpu* h) {
  constexpr int DEVICES = 64;
  static std::atomic<int> known[DEVICES][4];
  const auto k = chain_kernel(h);
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)CHAIN_SMEM_MAX) != cudaSuccess ||
      cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return -1;
  const int form = (h->rp.ndims == 3 ? 2 : 0) + (h->mixed ? 1 : 0);
  int most = h->device < DEVICES ? known[h->device][form].load() : 0;
  if (most != 0) return most;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(CHAIN_MAX_CTAS);
  cfg.blockDim = dim3(CHAIN_THREADS);
  cfg.dynamicSmemBytes = CHAIN_SMEM_MAX;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = CHAIN_MAX_CTAS;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int n = 0;
  most = CHAIN_MAX_CTAS;
  if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    most = 8;
  }
  if (h->device < DEVICES) known[h->device][form].store(most);
  return most;
}

// The chains whose tops are the patches of `level`, each following parent
// links to the coarsest level, laid out in shared memory.  False when one
// does not fit, when a top exceeds bmax cells, or when two chains meet.
static bool find_chains(bsam_gpu* h, int npatch, const bsam_patch_desc* patches, int level,
                        int64_t bmax, int64_t fp64_cells, bool loop,
                        std::vector<std::vector<int>>& chains, std::vector<ChainPlan>& plans) {
  const int nd = h->rp.ndims;
  chains.clear();
  plans.clear();
  std::vector<char> seen(npatch, 0);
  for (int p = 0; p < npatch; ++p) {
    if (patches[p].level != level) continue;
    std::vector<int> chain, prec;
    std::vector<std::array<int, 3>> n;
    for (int r = p; r >= 0; r = patches[r].parent) {
      if (r >= npatch || seen[r] || (int)chain.size() == CHAIN_MAX_LEVELS) {
        chains.clear();
        plans.clear();
        return false;
      }
      seen[r] = 1;
      chain.push_back(r);
      std::array<int, 3> e{1, 1, 1};
      for (int d = 0; d < nd; ++d) e[d] = patches[r].mx[d];
      const int64_t cells = (int64_t)e[0] * e[1] * e[2];
      n.push_back(e);
      prec.push_back(!h->mixed || cells <= fp64_cells ? PREC_F64 : PREC_F32);
    }
    ChainPlan C;
    bool ok = cells_of(n[0].data(), nd) <= bmax;
    for (auto& e : n) ok = ok && e[0] > 0 && e[1] > 0 && e[2] > 0;
    if (!ok || !chain_layout(nd, n, prec, h->mixed, h->rp.nsmoothingpasses, h->max_cluster, loop,
                             C)) {
      chains.clear();
      plans.clear();
      return false;
    }
    chains.push_back(chain);
    plans.push_back(C);
  }
  return !plans.empty();
}

// stages2: 2D levels above the chain may run as stages (stage2.cuh), which need a
// second state.
static int set_hierarchy(bsam_gpu* h, int npatch, const bsam_patch_desc* patches, int finestlevel,
                         bool stages2) {
  CU(cudaSetDevice(h->device));
  free_hierarchy(h);
  const int nd = h->rp.ndims;
  int minlevel = patches[0].level;
  for (int p = 0; p < npatch; ++p) minlevel = std::min(minlevel, patches[p].level);
  if (finestlevel < 0 || minlevel > 0) return fail(h, BSAM_ERR_ARG, "levels out of range");
  if (finestlevel > 0 && h->mixed)
    return fail(h, BSAM_ERR_UNSUPPORTED,
                "levels above the root are built for the FP64 form (no mixed-precision AMR)");
  h->amr = finestlevel > 0;
  h->minlevel = minlevel;
  h->finestlevel = finestlevel;
  h->nuser = npatch;
  h->levels.assign(finestlevel - minlevel + 1, LevelPlan{});
  for (int l = minlevel; l <= finestlevel; ++l) plan(h, l).level = l;
  h->desc.assign(patches, patches + npatch);

  // Mixed form: levels at or below this size stay FP64: 4096 cells, or the
  // size the caller gives for the bottom chain.
  const bool dflt = h->tuning.bottom_cells == 0;
  const int64_t fp64_cells = h->tuning.bottom_cells > 0 ? h->tuning.bottom_cells
                                                        : MIXED_FP64_CELLS;
  // Bottom level: the finest level from which every chain of levels down to
  // the coarsest fits in the shared memory of one cluster (chain.cuh) and pays
  // there.  A whole FP64 problem that fits does: its V-cycle loop runs in the
  // one launch (192^2 V-cycle 70 us, against 85 with its finest level as
  // stages).  Below other levels a chain's top level has 16 SMs against all of
  // them.  In 2D a level of 128^2 still costs less in the chain (256^2 FP64 97
  // against 102 us a V-cycle, 256^2 mixed 107 against 113), one of 144^2, 160 x 128
  // or 160^2 the same or more (a step of four V-cycles of 288^2 FP64 417 against 408
  // us, of 320 x 256 mixed 487 against 472) and one of 192^2 or 256^2 more (512^2
  // mixed 140 against 160 us a V-cycle).  In 3D a level of 20 x 20 x 24, 20 x 24 x 28
  // or 24^3 costs less in the chain (a step of 40 x 40 x 48 FP64 505 against 604 us,
  // of 40 x 48 x 56 545 against 628, of 48^3 605 against 656; mixed 556 against 640,
  // 580 against 645, 651 against 695), one of 28^3 about the same (56^3 FP64 643
  // against 663, mixed 690 against 692) and one of 32^3 more (64^3 FP64 191 against
  // 181 us a V-cycle, 128^3 505 against 491).  A caller's bottom_cells stands as given.
  const int64_t chain_top = nd == 3 ? CHAIN_TOP_CELLS_3D : CHAIN_TOP_CELLS_2D;
  int64_t bmax = dflt ? INT64_MAX : h->tuning.bottom_cells;
  if (dflt && h->tuning.fuse_smoother != 0)
    bmax = nd == 3 ? FUSED_BOTTOM_CELLS_3D : FUSED_BOTTOM_CELLS_2D;
  if (h->max_cluster == 0 && (h->max_cluster = chain_cluster(h)) < 0) {
    h->max_cluster = 0;
    return fail(h, BSAM_ERR_CUDA, "the chain kernel's attributes were rejected");
  }
  h->bottom_level = -1000;
  h->chain_loop = false;
  std::vector<std::vector<int>> chains;  // per chain its patches, top first
  std::vector<ChainPlan> plans;
  for (int l = std::min(finestlevel, 0); bmax > 0 && l >= minlevel; --l) {
    const bool loop = l == finestlevel && !h->mixed && finestlevel == 0;
    const int64_t cells = loop || !dflt ? bmax : std::min(bmax, chain_top);
    if (find_chains(h, npatch, patches, l, cells, fp64_cells, loop, chains, plans)) {
      h->bottom_level = l;
      h->chain_loop = loop && chains.size() == 1;
      break;
    }
  }

  // Records: the caller's patches, then one twin per finest-level patch in
  // the mixed form.
  std::vector<int> twin_of(npatch, -1);
  int nrec = npatch;
  for (int p = 0; p < npatch; ++p)
    if (patches[p].level == finestlevel) {
      h->masters.push_back(p);
      if (h->mixed) twin_of[p] = nrec++;
    }
  h->hp.assign(nrec, DevPatch{});
  h->field_elems.assign(nrec, 0);
  // rec_src[r]: the caller's patch whose geometry record r has.
  std::vector<int> rec_src(nrec);
  for (int p = 0; p < npatch; ++p) {
    rec_src[p] = p;
    if (twin_of[p] >= 0) rec_src[twin_of[p]] = p;
  }

  // Levels of a single patch.
  std::vector<char> alone(finestlevel - minlevel + 1, 0);
  for (int p = 0; p < npatch; ++p)
    if (patches[p].level >= minlevel && patches[p].level <= finestlevel) {
      char& n = alone[patches[p].level - minlevel];
      n = n == 0 ? 1 : 2;
    }
  for (char& n : alone) n = n == 1;
  std::vector<char> has_child(npatch, 0);
  for (int p = 0; p < npatch; ++p)
    if (patches[p].parent >= 0 && patches[p].parent < npatch) has_child[patches[p].parent] = 1;
  const double eps2 = h->rp.eps * h->rp.eps;
  size_t total = 0;
  std::vector<size_t> offs(nrec);
  std::vector<int> nfields(nrec, 0);
  std::vector<char> want_qold(nrec, 0), want_qs(nrec, 0);
  for (int r = 0; r < nrec; ++r) {
    const int p = rec_src[r];
    const bool is_twin = r >= npatch;
    const bsam_patch_desc& d = patches[p];
    if (d.level < minlevel || d.level > finestlevel)
      return fail(h, BSAM_ERR_ARG, "patch level out of range");
    DevPatch& P = h->hp[r];
    P.ndims = nd;
    for (int n = 0; n < 3; ++n) {
      P.n[n] = n < nd ? d.mx[n] : 1;
      if (P.n[n] <= 0) return fail(h, BSAM_ERR_ARG, "mx must be positive");
    }
    P.parent = d.parent;
    P.level = d.level;
    P.problem = 0;
    P.active = 1;
    P.newstep = 0;
    P.twin = is_twin ? -1 : twin_of[p];
    P.master = is_twin ? p : -1;
    // Precision of the record.
    const int64_t ncell = cells_of(P.n, nd);
    if (!h->mixed || (!is_twin && d.level == finestlevel) || ncell <= fp64_cells)
      P.prec = PREC_F64;
    else
      P.prec = PREC_F32;
    if (d.parent >= 0) {
      if (d.parent >= npatch || patches[d.parent].level != d.level - 1)
        return fail(h, BSAM_ERR_ARG, "parent must be a patch on the next coarser level");
      for (int n = 0; n < nd; ++n) {
        if (P.n[n] % 2) return fail(h, BSAM_ERR_ARG, "a patch with a parent needs even mx");
        P.cn[n] = P.n[n] / 2;
        P.off[n] = d.mbounds[n][0] - 1;
        if (d.mbounds[n][1] - d.mbounds[n][0] + 1 != P.cn[n] || P.off[n] < 0 ||
            d.mbounds[n][1] > patches[d.parent].mx[n])
          return fail(h, BSAM_ERR_ARG, "mbounds inconsistent with mx / parent");
      }
    } else if (d.level != minlevel) {
      return fail(h, BSAM_ERR_ARG, "only the coarsest level may lack a parent");
    }
    for (int n = nd; n < 3; ++n) {
      P.cn[n] = 1;
      P.off[n] = 0;
    }
    P.wt = 1;
    for (int f = 0; f < 6; ++f) {
      if (f >= 2 * nd) {
        P.bc[f] = BC_NONE;
        continue;
      }
      int rule;
      if (face_rule(nd, f, d.mthbc[f], &rule))
        return fail(h, BSAM_ERR_UNSUPPORTED, "boundary code not supported");
      P.bc[f] = rule;
      P.code[f] = d.mthbc[f];
      if (rule == BC_NONE) P.wt = 0;
    }
    if (!P.wt && d.level < 1)
      return fail(h, BSAM_ERR_UNSUPPORTED, "internal faces occur only on refined levels");
    // Periodic faces (PeriodicSetup, boundary.f90:893-963): in pairs (the
    // reference stops otherwise, bsamroutines.f90:307-316), on hierarchies
    // without refined levels (TransferPeriodicBC between refined grids has no
    // device form here), and on dimensions whose extent is even or 1: with an
    // odd extent above 1 the first and last cells of the dimension have the
    // same colour, and a colour pass would read the periodic ghost that its
    // opposite cell writes through in the same pass.
    for (int n = 0; n < nd; ++n) {
      const bool lo = P.bc[2 * n] == BC_PERIODIC, hi = P.bc[2 * n + 1] == BC_PERIODIC;
      if (lo != hi) return fail(h, BSAM_ERR_ARG, "periodic faces come in pairs");
      if (lo && finestlevel > 0)
        return fail(h, BSAM_ERR_UNSUPPORTED, "periodic faces with refined levels");
      if (lo && P.n[n] > 1 && P.n[n] % 2)
        return fail(h, BSAM_ERR_UNSUPPORTED, "periodic dimension with an odd extent above 1");
    }
    // Does the V-cycle run on this record?  (Not on the masters of the mixed form.)
    const bool in_vcycle = !(h->mixed && !is_twin && d.level == finestlevel);
    // Mixed form: the V-cycle levels carry a correction of the master state
    // (mixed.cuh); a reflecting face maps a correction to its negative.
    P.delta = (h->mixed && in_vcycle) ? 1 : 0;
    if (P.delta)
      for (int f = 0; f < 2 * nd; ++f)
        if (P.bc[f] == BC_REFLECT) P.bc[f] = BC_NEGATE;
    // Fused stages: V-cycle levels of uniform hierarchies (in 2D also the root
    // of a refined one and the levels below it) with a parent, above the bottom
    // chain.  3D, on request: all faces physical (the stage derives face ghosts
    // from the tile itself).  2D, unless the caller wants every level as launches
    // (bottom_cells -1): one patch, at most two sweeps (the tile's halo of 4).
    const int fmin = std::max(8, h->tuning.fuse_min_n);
    bool periodic = false;
    for (int f = 0; f < 2 * nd; ++f) periodic |= P.bc[f] == BC_PERIODIC;
    const bool fuse3 = h->tuning.fuse_smoother != 0 && nd == 3 && finestlevel == 0 && !periodic &&
                       !(P.delta && P.prec == PREC_F64) && P.n[0] >= fmin && P.n[1] >= fmin &&
                       P.n[2] >= fmin;
    // (Levels with more rows of tiles than a grid holds, above 1048560 rows of cells,
    // run a launch per pass.)
    const bool fuse2 = stages2 && nd == 2 && h->tuning.bottom_cells >= 0 && d.level <= 0 &&
                       h->rp.nsmoothingpasses <= 2 && alone[d.level - minlevel] &&
                       P.n[1] <= 16 * MAX_GRID_Y;
    P.fused = (fuse3 || fuse2) && in_vcycle && d.parent >= 0 && d.level > h->bottom_level ? 1 : 0;
    if (P.fused && nd == 3) {
      const int ftx = P.prec == PREC_F32 ? Fused3<float>::TX : Fused3<double>::TX;
      const int fty = P.prec == PREC_F32 ? Fused3<float>::TY : Fused3<double>::TY;
      const int tiles = ((P.n[0] + ftx - 1) / ftx) * ((P.n[1] + fty - 1) / fty);
      int chunk = h->tuning.chunk;
      if (chunk <= 0) {
        // About one CTA per SM, chunks of at least 16 planes.
        const int nchunk = std::max(1, std::min(B200_SMS / std::max(tiles, 1), P.n[2] / 16));
        chunk = (P.n[2] + nchunk - 1) / nchunk;
      }
      P.zchunk = std::max(1, std::min(chunk, P.n[2]));
    }
    // Layout: rows aligned to 128 bytes; the slack after the last row keeps
    // the fused kernel's halo'd row copies inside the allocation.
    const int es = elem_bytes(P.prec);
    const int64_t A = 128 / es, lead = A - 1;
    P.sy = roundup(lead + P.n[0] + 2, A);
    P.sz = nd == 3 ? P.sy * (P.n[1] + 2) : 0;
    const int64_t vol = nd == 3 ? P.sz * (P.n[2] + 2) : P.sy * (P.n[1] + 2);
    h->field_elems[r] = roundup(lead + vol + 64, 256 / es);
    offs[r] = total;
    const bool parent_of_any = in_vcycle && has_child[p];
    const bool has_qold = !is_twin && d.level >= 0 && P.prec == PREC_F64 &&
                          (!h->mixed || d.level == finestlevel);
    nfields[r] = 2 /*q*/ + 2 /*f*/ + (has_qold ? 2 : 0) + (parent_of_any ? 2 : 0) +
                 (P.fused ? 2 : 0) + (P.delta ? 1 : 0);
    total += (size_t)h->field_elems[r] * nfields[r] * es;
    // Problem constants (problem.f90:183-187): h2 = h*h; dt/h2; eps2/h2; 2d*eps2/h2.
    P.h = d.dx;
    const double h2 = d.dx * d.dx;
    P.dt = h->rp.dt;
    P.eps2 = eps2;
    P.alpha = h->rp.alpha;
    P.tmp1 = h->rp.dt / h2;
    P.tmp2 = eps2 / h2;
    P.tmp3 = (2.0 * nd) * eps2 / h2;
    if (in_vcycle) plan(h, d.level).patches.push_back(r);
    want_qold[r] = has_qold;
    want_qs[r] = parent_of_any;
  }
  if (h->spare_arena && h->spare_bytes >= total) {
    h->d_arena = h->spare_arena;
    total = h->spare_bytes;
    h->spare_arena = nullptr;
    h->spare_bytes = 0;
  } else {
    // Under regridding the arena alternates with the spare: a quarter more
    // than this table needs lets the next tables of similar size reuse it.
    if (h->regridding) total += total / 4;
    if (cudaMalloc(&h->d_arena, total) != cudaSuccess) {
      cudaGetLastError();
      h->d_arena = nullptr;
      return fail(h, BSAM_ERR_NOMEM, "arena allocation failed");
    }
  }
  h->arena_bytes = total;
  CU(cudaMemsetAsync(h->d_arena, 0, total, h->stream));
  for (int r = 0; r < nrec; ++r) {
    DevPatch& P = h->hp[r];
    const int es = elem_bytes(P.prec);
    char* base = h->d_arena + offs[r];
    const int64_t fe = h->field_elems[r], lead = 128 / es - 1;
    int slot = 0;
    auto next = [&]() { return (void*)(base + (fe * (slot++) + lead) * es); };
    const bool has_qold = want_qold[r], has_qs = want_qs[r];
    P.q[0] = next();
    P.q[1] = next();
    P.f[0] = next();
    P.f[1] = next();
    P.qo[0] = P.qo[1] = nullptr;
    P.qs[0] = P.qs[1] = nullptr;
    if (has_qold) {
      P.qo[0] = next();
      P.qo[1] = next();
    }
    if (has_qs) {
      P.qs[0] = next();
      P.qs[1] = next();
    }
    if (P.fused) {
      P.qb[0] = next();
      P.qb[1] = next();
    }
    P.bs = P.delta ? next() : nullptr;
  }
  // CopyQToQold as one launch: the whole field allocation of q onto qold's.
  std::vector<CopySpan> qold_spans;
  {
    std::vector<CopySpan>& spans = qold_spans;
    for (int r = 0; r < npatch; ++r) {
      const DevPatch& P = h->hp[r];
      if (!P.qo[0]) continue;
      const int64_t lead = 128 / sizeof(double) - 1;
      for (int c = 0; c < 2; ++c)
        spans.push_back(CopySpan{static_cast<const double*>(P.q[c]) - lead,
                                 static_cast<double*>(P.qo[c]) - lead, h->field_elems[r]});
      h->qold_span_max = std::max(h->qold_span_max, h->field_elems[r]);
    }
    h->nqold_spans = (int)spans.size();
  }
  // SetBC's patches at and below the root, and the snapshots of partly covered
  // parents (levels >= root below the finest).
  std::vector<int> setbc_list;
  h->setbc_first.assign(1, 0);
  h->setbc_cells = 1;
  for (int l = minlevel; l <= 0; ++l) {
    for (int p = 0; p < npatch; ++p) {
      const DevPatch& P = h->hp[p];
      if (P.level != l || P.prec != PREC_F64 || P.delta) continue;
      setbc_list.push_back(p);
      h->setbc_cells = std::max(h->setbc_cells, cells_of(P.n, nd));
    }
    h->setbc_first.push_back((int)setbc_list.size());
  }
  std::vector<CopySpan> snap_spans;
  std::vector<int> snap_first(h->levels.size() + 1, 0);
  for (size_t li = 0; li < h->levels.size(); ++li) {
    LevelPlan& L = h->levels[li];
    snap_first[li] = (int)snap_spans.size();
    L.snap_max = 0;
    if (L.level >= 0 && L.level < finestlevel)
      for (int p : L.patches) {
        const DevPatch& P = h->hp[p];
        if (!P.qs[0]) continue;  // not a parent: no child reads a snapshot of it
        const int64_t lead = 128 / sizeof(double) - 1;
        for (int c = 0; c < 2; ++c)
          snap_spans.push_back(CopySpan{static_cast<const double*>(P.q[c]) - lead,
                                        static_cast<double*>(P.qs[c]) - lead,
                                        h->field_elems[p]});
        L.snap_max = std::max(L.snap_max, h->field_elems[p]);
      }
    L.nsnap = (int)snap_spans.size() - snap_first[li];
  }
  // Parents of the twins are the masters' parents.
  for (int r = npatch; r < nrec; ++r) h->hp[r].parent = h->hp[rec_src[r]].parent;
  for (int r = 0; r < nrec; ++r)
    h->hp[r].pprec = h->hp[r].parent >= 0 ? h->hp[h->hp[r].parent].prec : h->hp[r].prec;
  // TMA tensor maps of the fused records (q0, q1, qb0, qb1, f0, f1, bs).
  std::vector<int> fused_recs;
  std::vector<CUtensorMap> maps;
  {
    for (int r = 0; r < nrec; ++r)
      if (h->hp[r].fused && nd == 3) fused_recs.push_back(r);
    if (!fused_recs.empty()) {
      maps.resize(7 * fused_recs.size());
      for (size_t k = 0; k < fused_recs.size(); ++k) {
        const DevPatch& P = h->hp[fused_recs[k]];
        const int hx = P.prec == PREC_F32 ? Fused3<float>::HX : Fused3<double>::HX;
        const int hy = P.prec == PREC_F32 ? Fused3<float>::HY : Fused3<double>::HY;
        const void* fields[7] = {P.q[0], P.q[1], P.qb[0], P.qb[1],
                                 P.f[0], P.f[1], P.bs ? P.bs : P.q[0]};
        for (int m = 0; m < 7; ++m)
          if (!encode_field_map(&maps[7 * k + m], P, fields[m], hx, hy))
            return fail(h, BSAM_ERR_CUDA, "cuTensorMapEncodeTiled rejected a field map");
      }

    }
  }

  // Level precisions and work lists.
  std::vector<Item> all;
  const size_t nl = h->levels.size();
  std::vector<std::pair<int, int>> spans_fine(nl), spans_coarse(nl), spans_corr(nl), spans_fused(nl);
  for (size_t li = 0; li < nl; ++li) {
    LevelPlan& L = h->levels[li];
    if (L.patches.empty()) return fail(h, BSAM_ERR_ARG, "a level between minlevel and finest is empty");
    L.prec = h->hp[L.patches[0]].prec;
    for (int p : L.patches)
      if (h->hp[p].prec != L.prec) return fail(h, BSAM_ERR_ARG, "mixed precisions on one level");
    int s = (int)all.size();
    for (int p : L.patches) work_tiles(p, h->hp[p].n, nd, all);
    spans_fine[li] = {s, (int)all.size() - s};
    s = (int)all.size();
    for (int p : L.patches)
      if (h->hp[p].parent >= 0) work_tiles(p, h->hp[p].cn, nd, all);
    spans_coarse[li] = {s, (int)all.size() - s};
    s = (int)all.size();
    for (int p : L.patches)
      if (h->hp[p].parent >= 0) block_tiles(p, h->hp[p].cn, nd, all);
    spans_corr[li] = {s, (int)all.size() - s};
    // A level runs fused stages only when every patch on it does.
    L.fused = true;
    for (int p : L.patches) L.fused = L.fused && h->hp[p].fused;
    if (!L.fused)
      for (int p : L.patches) h->hp[p].fused = 0;
    s = (int)all.size();
    if (L.fused && nd == 3)
      for (int p : L.patches) {
        const DevPatch& P = h->hp[p];
        const int ftx = P.prec == PREC_F32 ? Fused3<float>::TX : Fused3<double>::TX;
        const int fty = P.prec == PREC_F32 ? Fused3<float>::TY : Fused3<double>::TY;
        const int tx = (P.n[0] + ftx - 1) / ftx;
        const int ty = (P.n[1] + fty - 1) / fty;
        const int tz = (P.n[2] + P.zchunk - 1) / P.zchunk;
        for (int z = 0; z < tz; ++z)
          for (int y = 0; y < ty; ++y)
            for (int x = 0; x < tx; ++x) all.push_back(Item{p, x, y, z});
      }
    spans_fused[li] = {s, (int)all.size() - s};
  }
  const int s_master = (int)all.size();
  for (int p : h->masters) tiles_for(p, h->hp[p].n, nd, all);
  h->nmaster = (int)all.size() - s_master;
  // State patches (levels >= root, the caller's records) and the root.
  const int s_state = (int)all.size();
  for (int p = 0; p < npatch; ++p)
    if (patches[p].level >= 0) tiles_for(p, h->hp[p].n, nd, all);
  h->nstate = (int)all.size() - s_state;
  const int s_root = (int)all.size();
  for (int p = 0; p < npatch; ++p)
    if (patches[p].level == 0) tiles_for(p, h->hp[p].n, nd, all);
  h->nroot = (int)all.size() - s_root;
  // Refined levels: patch lists and GhostOverlap transfers
  // (ApplyOnLevelPairs order: each patch with every later one).
  std::vector<int> plist_all;
  std::vector<OverlapCopy> ovl_all;
  std::vector<std::pair<int, int>> span_plist(nl), span_ovl(nl);
  for (size_t li = 0; li < nl; ++li) {
    LevelPlan& L = h->levels[li];
    L.amr = L.level >= 1;
    L.snap = L.level >= 0 && L.level < finestlevel;
    span_plist[li] = {(int)plist_all.size(), 0};
    span_ovl[li] = {(int)ovl_all.size(), 0};
    if (!L.amr) continue;
    for (int p : L.patches) plist_all.push_back(p);
    for (size_t a = 0; a < L.patches.size(); ++a)
      for (size_t bi = a + 1; bi < L.patches.size(); ++bi) {
        const bsam_patch_desc& g1 = patches[L.patches[a]];
        const bsam_patch_desc& g2 = patches[L.patches[bi]];
        int ov[3][2] = {{1, 1}, {1, 1}, {1, 1}};
        bool empty = false;
        for (int n = 0; n < nd; ++n) {
          ov[n][0] = std::max(g1.mglobal[n][0] - 1, g2.mglobal[n][0] - 1);
          ov[n][1] = std::min(g1.mglobal[n][1] + 1, g2.mglobal[n][1] + 1);
          empty |= ov[n][1] < ov[n][0];
        }
        if (empty) continue;
        // dst takes the other grid's interior inside the overlap.
        auto emit = [&](int dst, const bsam_patch_desc& gd, int src, const bsam_patch_desc& gs) {
          int box[3][2] = {{1, 1}, {1, 1}, {1, 1}};
          for (int n = 0; n < nd; ++n) {
            box[n][0] = std::max(ov[n][0], gs.mglobal[n][0]);
            box[n][1] = std::min(ov[n][1], gs.mglobal[n][1]);
            if (box[n][1] < box[n][0]) return;
          }
          OverlapCopy o;
          o.dst = dst;
          o.src = src;
          o.i0 = box[0][0] - gd.mglobal[0][0] + 1;
          o.i1 = box[0][1] - gd.mglobal[0][0] + 1;
          o.j0 = box[1][0] - gd.mglobal[1][0] + 1;
          o.j1 = box[1][1] - gd.mglobal[1][0] + 1;
          o.di = gd.mglobal[0][0] - gs.mglobal[0][0];
          o.dj = gd.mglobal[1][0] - gs.mglobal[1][0];
          if (nd == 3) {
            o.k0 = box[2][0] - gd.mglobal[2][0] + 1;
            o.k1 = box[2][1] - gd.mglobal[2][0] + 1;
            o.dk = gd.mglobal[2][0] - gs.mglobal[2][0];
          } else {
            o.k0 = o.k1 = 0;
            o.dk = 0;
          }
          ovl_all.push_back(o);
        };
        emit(L.patches[a], g1, L.patches[bi], g2);
        emit(L.patches[bi], g2, L.patches[a], g1);
      }
    span_plist[li].second = (int)plist_all.size() - span_plist[li].first;
    span_ovl[li].second = (int)ovl_all.size() - span_ovl[li].first;
  }
  // Per level: the overlap transfers grouped by destination (stable), with
  // each patch-list entry's {first, count} relative to the level's group.
  std::vector<OverlapCopy> ovl_by_dst(ovl_all.size());
  std::vector<int2> ovl_range(plist_all.size(), make_int2(0, 0));
  for (size_t li = 0; li < nl; ++li) {
    const int p0 = span_plist[li].first, np = span_plist[li].second;
    const int o0 = span_ovl[li].first, no = span_ovl[li].second;
    int at = o0;
    for (int k = 0; k < np; ++k) {
      const int dst = plist_all[p0 + k];
      const int first = at;
      for (int c = o0; c < o0 + no; ++c)
        if (ovl_all[c].dst == dst) ovl_by_dst[at++] = ovl_all[c];
      ovl_range[p0 + k] = make_int2(first - o0, at - first);
    }
    if (at != o0 + no) return fail(h, BSAM_ERR_ARG, "an overlap names no patch of its level");
  }
  h->h_plist = plist_all;
  h->h_ovl_by_dst = ovl_by_dst;
  h->h_ovl_range = ovl_range;
  h->h_span_plist = span_plist;
  h->h_span_ovl = span_ovl;
  h->max_items = std::max(1, h->nmaster);
  for (size_t li = 0; li < nl; ++li) {
    LevelPlan& L = h->levels[li];
    L.nplist = span_plist[li].second;
    L.novl = span_ovl[li].second;
    L.nfine = spans_fine[li].second;
    L.ncoarse = spans_coarse[li].second;
    L.ncorr = spans_corr[li].second;
    L.nfused = spans_fused[li].second;
    h->max_items = std::max(h->max_items, L.nfine);
  }
  h->max_items = std::max(h->max_items, h->nroot);
  if (!h->attrs_set) {
    CU(cudaFuncSetAttribute(k_smooth3_fused<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)Fused3<double>::SMEM));
    CU(cudaFuncSetAttribute(k_smooth3_fused<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)Fused3<float>::SMEM));
    h->attrs_set = true;
  }
  {
    int64_t ncells = 0;
    for (int p : h->masters) ncells += cells_of(h->hp[p].n, nd);
    h->denom = (double)(h->rp.nrvars * ncells);  // L2Error's integralresult(2)
  }
  h->nchains = (int)plans.size();
  h->chain_ctas = 1;
  h->chain_smem = 0;
  for (size_t c = 0; c < plans.size(); ++c) {
    ChainPlan& C = plans[c];
    h->chain_ctas = std::max(h->chain_ctas, C.ctas);
    h->chain_smem = std::max(h->chain_smem, (size_t)C.smem);
    for (int l = 0; l < C.nlev; ++l) {
      const int p = chains[c][l];
      const int r = twin_of[p] >= 0 ? twin_of[p] : p;
      const DevPatch& P = h->hp[r];
      if (P.prec != C.L[l].prec || P.delta != C.L[l].delta)
        return fail(h, BSAM_ERR_ARG, "a chain level's form differs from its record's");
      chain_faces(C, l, r, P);
    }
  }
  for (ChainPlan& C : plans) C.ctas = h->chain_ctas;
  // The tables' layout in d_meta (256-byte aligned pieces), the buffer grown
  // when too small, then the pointers, and one copy of the host image.
  {
    size_t off = 0;
    auto place = [&](size_t bytes) {
      const size_t at = (size_t)roundup((int64_t)off, 256);
      off = at + bytes;
      return at;
    };
    const size_t o_patches = place(sizeof(DevPatch) * nrec);
    const size_t o_items = place(sizeof(Item) * all.size());
    const size_t o_plist = place(sizeof(int) * plist_all.size());
    const size_t o_ovl = place(sizeof(OverlapCopy) * ovl_all.size());
    const size_t o_ovl_dst = place(sizeof(OverlapCopy) * ovl_by_dst.size());
    const size_t o_ovl_rng = place(sizeof(int2) * ovl_range.size());
    const size_t o_qold = place(sizeof(CopySpan) * qold_spans.size());
    const size_t o_snap = place(sizeof(CopySpan) * snap_spans.size());
    const size_t o_setbc = place(sizeof(int) * setbc_list.size());
    const size_t o_maps = place(sizeof(CUtensorMap) * maps.size());
    const size_t o_chains = place(sizeof(ChainPlan) * plans.size());
    const size_t o_part = place(sizeof(double) * h->max_items);
    const size_t total_meta = off;
    if (total_meta > h->meta_cap) {
      if (h->d_meta) cudaFree(h->d_meta);
      h->d_meta = nullptr;
      h->meta_cap = 0;
      const size_t want = total_meta + total_meta / 2;  // headroom for the next regrid
      if (cudaMalloc(&h->d_meta, want) != cudaSuccess)
        return fail(h, BSAM_ERR_NOMEM, "table allocation failed");
      h->meta_cap = want;
    }
    char* base = h->d_meta;
    h->d_items = reinterpret_cast<Item*>(base + o_items);
    h->d_plist = plist_all.empty() ? nullptr : reinterpret_cast<int*>(base + o_plist);
    h->d_ovl = ovl_all.empty() ? nullptr : reinterpret_cast<OverlapCopy*>(base + o_ovl);
    h->d_qold_spans = qold_spans.empty() ? nullptr : reinterpret_cast<CopySpan*>(base + o_qold);
    h->d_setbc = reinterpret_cast<int*>(base + o_setbc);
    h->d_tmaps = maps.empty() ? nullptr : reinterpret_cast<CUtensorMap*>(base + o_maps);
    h->d_chains = plans.empty() ? nullptr : reinterpret_cast<ChainPlan*>(base + o_chains);
    h->d_partials = reinterpret_cast<double*>(base + o_part);
    h->d_patches = reinterpret_cast<DevPatch*>(base + o_patches);
    for (size_t k = 0; k < fused_recs.size(); ++k) h->hp[fused_recs[k]].tmaps = h->d_tmaps + 7 * k;
    for (size_t li = 0; li < nl; ++li) {
      LevelPlan& L = h->levels[li];
      L.d_plist = h->d_plist ? h->d_plist + span_plist[li].first : nullptr;
      L.d_ovl = h->d_ovl ? h->d_ovl + span_ovl[li].first : nullptr;
      L.d_snap = reinterpret_cast<CopySpan*>(base + o_snap) + snap_first[li];
      L.d_ovl_by_dst = ovl_by_dst.empty()
                           ? nullptr
                           : reinterpret_cast<OverlapCopy*>(base + o_ovl_dst) + span_ovl[li].first;
      L.d_ovl_range = ovl_range.empty()
                          ? nullptr
                          : reinterpret_cast<int2*>(base + o_ovl_rng) + span_plist[li].first;
      L.d_fine = h->d_items + spans_fine[li].first;
      L.d_coarse = h->d_items + spans_coarse[li].first;
      L.d_corr = h->d_items + spans_corr[li].first;
      L.d_fused = h->d_items + spans_fused[li].first;
    }
    h->d_master = h->d_items + s_master;
    h->d_state = h->d_items + s_state;
    h->d_root = h->d_items + s_root;
    std::vector<unsigned char>& img = h->meta_host;
    img.assign(o_part, 0);  // the partial sums need no initial contents
    auto put = [&](size_t at, const void* src, size_t bytes) {
      if (bytes) std::memcpy(img.data() + at, src, bytes);
    };
    put(o_patches, h->hp.data(), sizeof(DevPatch) * nrec);
    put(o_items, all.data(), sizeof(Item) * all.size());
    put(o_plist, plist_all.data(), sizeof(int) * plist_all.size());
    put(o_ovl, ovl_all.data(), sizeof(OverlapCopy) * ovl_all.size());
    put(o_ovl_dst, ovl_by_dst.data(), sizeof(OverlapCopy) * ovl_by_dst.size());
    put(o_ovl_rng, ovl_range.data(), sizeof(int2) * ovl_range.size());
    put(o_qold, qold_spans.data(), sizeof(CopySpan) * qold_spans.size());
    put(o_snap, snap_spans.data(), sizeof(CopySpan) * snap_spans.size());
    put(o_setbc, setbc_list.data(), sizeof(int) * setbc_list.size());
    put(o_maps, maps.data(), sizeof(CUtensorMap) * maps.size());
    put(o_chains, plans.data(), sizeof(ChainPlan) * plans.size());
    const int urc = h2d_bounce(h, h->d_meta, img.data(), img.size());
    if (urc) return urc;
  }
  CU(cudaMemsetAsync(h->d_status, 0, sizeof(DevStatus), h->stream));
  CU(cudaStreamSynchronize(h->stream));
  h->have_hierarchy = true;
  return BSAM_OK;
}

int bsam_gpu_set_hierarchy(bsam_gpu* h, int npatch, const bsam_patch_desc* patches,
                           int finestlevel) {
  if (!h || npatch <= 0 || !patches) return BSAM_ERR_ARG;
  const int rc = set_hierarchy(h, npatch, patches, finestlevel, true);
  // Where the second states of the 2D stages do not fit beside the rest, every pass
  // is a launch of its own (the same bits).
  if (rc == BSAM_ERR_NOMEM && h->rp.ndims == 2)
    return set_hierarchy(h, npatch, patches, finestlevel, false);
  return rc;
}

static int field_ptr(bsam_gpu* h, int patch, int field, int comp, double** ptr, bool* interior) {
  const DevPatch& P = h->hp[patch];
  void* p = nullptr;
  *interior = false;
  switch (field) {
    case BSAM_FIELD_Q: p = P.q[comp]; break;
    case BSAM_FIELD_QOLD: p = P.qo[comp]; break;
    case BSAM_FIELD_F: p = P.f[comp]; *interior = true; break;
    default: return BSAM_ERR_ARG;
  }
  if (!p) return BSAM_ERR_UNSUPPORTED;
  *ptr = static_cast<double*>(p);
  return BSAM_OK;
}

// taken = false: no page-locked memory was to be had and nothing was done.
static int copy_state(bsam_gpu* h, RowsTask task, double* host, int dir, bool& taken) {
  taken = true;
  auto none = [&] {
    cudaGetLastError();
    taken = false;
    return BSAM_OK;
  };
  const int64_t rows = 2 * task.rows;
  const size_t row_bytes = sizeof(double) * task.e0;
  auto launch = [&](cudaStream_t st, double* packed, int64_t r0, int64_t r1) {
    RowsTask t = task;
    t.packed = packed - r0 * task.e0;  // so that row r0 lies at `packed`
    const int64_t warps = (r1 - r0) * ((task.e0 + ROW_PART - 1) / ROW_PART);
    const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((warps + 7) / 8, 592));
    if (dir == 0) k_rows<true><<<g, 256, 0, st>>>(t, r0, r1);
    else k_rows<false><<<g, 256, 0, st>>>(t, r0, r1);
    return cudaGetLastError();
  };
  if (row_bytes * rows <= kBounceBytes) {
    double* pin = static_cast<double*>(pin_reserve(h, row_bytes * rows));
    if (!pin) return none();
    if (dir == 0) std::memcpy(pin, host, row_bytes * rows);
    CU(launch(h->stream, pin, 0, rows));
    ++h->stats.launches;
    if (dir == 0) {
      h->pin_busy = true;
    } else {
      CU(cudaStreamSynchronize(h->stream));
      std::memcpy(host, pin, row_bytes * rows);
    }
    return BSAM_OK;
  }
  const size_t piece = piece_bytes(row_bytes * rows, row_bytes);
  const int64_t per = (int64_t)(piece / row_bytes);
  const int64_t pieces = (rows + per - 1) / per;
  for (cudaEvent_t& e : h->slot_ev)
    if (!e) CU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  for (cudaStream_t& st : h->copy_streams)
    if (!st && cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess)
      return none();
  const PieceBlocks::Block block = PieceBlocks::get().take(2 * kCopyThreads * piece);
  if (!block.p) return none();
  char* pin = static_cast<char*>(block.p);
  const int nt = (int)std::max(1u, std::min((unsigned)kCopyThreads,
                                            std::thread::hardware_concurrency()));
  // Thread 0 copies on the handle's stream, the others on their own, which take up
  // where the handle's stands and are waited for before the call returns.
  auto stream = [&](int t) { return t == 0 ? h->stream : h->copy_streams[t - 1]; };
  std::atomic<int> failed{(int)cudaEventRecord(h->slot_ev[0], h->stream)};
  for (int t = 1; t < nt; ++t)
    if (failed.load() == (int)cudaSuccess)
      failed.store((int)cudaStreamWaitEvent(stream(t), h->slot_ev[0], 0));
  // Thread t takes pieces t, t + nt, ..., the k-th of them in its slot k % 2.
  auto work = [&](int t) {
    cudaError_t e = (cudaError_t)failed.load();
    if (e == cudaSuccess) e = cudaSetDevice(h->device);
    auto first = [&](int64_t k) { return (t + k * nt) * per; };
    auto last = [&](int64_t k) { return std::min(rows, first(k) + per); };
    auto buf = [&](int64_t k) {
      return reinterpret_cast<double*>(pin + (2 * t + (int)(k & 1)) * piece);
    };
    auto ev = [&](int64_t k) { return h->slot_ev[2 * t + (int)(k & 1)]; };
    const int64_t n = (pieces - t + nt - 1) / nt;
    auto issue = [&](int64_t k) {
      if (e == cudaSuccess) e = launch(stream(t), buf(k), first(k), last(k));
      if (e == cudaSuccess) e = cudaEventRecord(ev(k), stream(t));
    };
    if (dir != 0)
      for (int64_t k = 0; k < std::min<int64_t>(2, n); ++k) issue(k);
    for (int64_t k = 0; k < n && e == cudaSuccess; ++k) {
      double* user = host + first(k) * task.e0;
      const size_t bytes = row_bytes * (size_t)(last(k) - first(k));
      if (dir == 0) {
        if (k >= 2) e = cudaEventSynchronize(ev(k));
        if (e != cudaSuccess) break;
        std::memcpy(buf(k), user, bytes);
        issue(k);
      } else {
        e = cudaEventSynchronize(ev(k));
        if (e != cudaSuccess) break;
        std::memcpy(user, buf(k), bytes);
        if (k + 2 < n) issue(k + 2);
      }
    }
    const cudaError_t done = cudaStreamSynchronize(stream(t));
    if (e == cudaSuccess) e = done;
    if (e != cudaSuccess) failed.store((int)e);
  };
  // The shares of threads that cannot be had are done by this one.
  std::vector<std::thread> pool;
  int started = 1;
  try {
    for (; started < nt; ++started) pool.emplace_back(work, started);
  } catch (const std::exception&) {
  }
  work(0);
  for (int t = started; t < nt; ++t) work(t);
  for (auto& t : pool) t.join();
  h->stats.launches += pieces;
  PieceBlocks::get().give(block);
  if (failed.load() != (int)cudaSuccess)
    return fail(h, BSAM_ERR_CUDA,
                std::string("field copy: ") + cudaGetErrorString((cudaError_t)failed.load()));
  return BSAM_OK;
}

// Copy between a Fortran array and the pitched device field; dir 0 = H2D.
static int copy_field(bsam_gpu* h, int patch, int field, double* host, int dir) {
  if (!h || !h->have_hierarchy) return BSAM_ERR_STATE;
  if (patch < 0 || patch >= h->nuser || !host) return BSAM_ERR_ARG;
  CU(cudaSetDevice(h->device));
  const DevPatch& P = h->hp[patch];
  if (P.prec != PREC_F64 || P.delta)
    return fail(h, BSAM_ERR_UNSUPPORTED, "the fields of mixed-precision working levels are internal");
  const int nd = h->rp.ndims;
  for (int comp = 0; comp < 2; ++comp) {
    double* dev;
    bool interior;
    const int rc = field_ptr(h, patch, field, comp, &dev, &interior);
    if (rc) return fail(h, rc, "field not held for this patch");
    const int g = interior ? 0 : 1;  // ghost layers present in the host array
    const int e0 = P.n[0] + 2 * g, e1 = P.n[1] + 2 * g, e2 = nd == 3 ? P.n[2] + 2 * g : 1;
    const size_t hcomp = (size_t)e0 * e1 * e2;
    double* hbase = host + comp * hcomp;
    if (g == 1) {
      // With the ghost ring every row of every plane sits at stride sy on the
      // device (sz = sy * (n1 + 2)).
      const size_t bytes = 2 * hcomp * sizeof(double);
      if (bytes <= kBounceBytes || piece_bytes(bytes, e0 * sizeof(double)) > 0) {
        double* dev1;
        const int rc1 = field_ptr(h, patch, field, 1, &dev1, &interior);
        if (rc1) return fail(h, rc1, "field not held for this patch");
        bool taken;
        const RowsTask task{nullptr, {dev, dev1}, (int64_t)e1 * e2, P.sy, e0, 0};
        const int src = copy_state(h, task, host, dir, taken);
        if (taken) return src;
      }
      if (dir == 0)
        CU(cudaMemcpy2DAsync(dev, P.sy * sizeof(double), hbase, e0 * sizeof(double),
                             e0 * sizeof(double), (size_t)e1 * e2, cudaMemcpyHostToDevice,
                             h->stream));
      else
        CU(cudaMemcpy2DAsync(hbase, e0 * sizeof(double), dev, P.sy * sizeof(double),
                             e0 * sizeof(double), (size_t)e1 * e2, cudaMemcpyDeviceToHost,
                             h->stream));
      continue;
    }
    for (int kz = 0; kz < e2; ++kz) {
      const int k = nd == 3 ? kz + 1 : 0;
      double* d = dev + 1 + P.sy + (int64_t)k * P.sz;
      double* hs = hbase + (size_t)kz * e0 * e1;
      if (dir == 0)
        CU(cudaMemcpy2DAsync(d, P.sy * sizeof(double), hs, e0 * sizeof(double),
                             e0 * sizeof(double), e1, cudaMemcpyHostToDevice, h->stream));
      else
        CU(cudaMemcpy2DAsync(hs, e0 * sizeof(double), d, P.sy * sizeof(double),
                             e0 * sizeof(double), e1, cudaMemcpyDeviceToHost, h->stream));
    }
  }
  CU(cudaStreamSynchronize(h->stream));
  return BSAM_OK;
}

int bsam_gpu_put_field(bsam_gpu* h, int patch, int field, const double* a) {
  return copy_field(h, patch, field, const_cast<double*>(a), 0);
}

int bsam_gpu_get_field(bsam_gpu* h, int patch, int field, double* out) {
  return copy_field(h, patch, field, out, 1);
}

int bsam_gpu_set_ghost(bsam_gpu* h) {
  if (!h || !h->have_hierarchy) return BSAM_ERR_STATE;
  CU(cudaSetDevice(h->device));
  // Coarse levels first: a refined level's interpolation reads its parent.
  ghost_levels(h, h->minlevel, 0);
  for (int l = 1; l <= h->finestlevel; ++l) amr_ghost(h, l, 0);
  CU(cudaGetLastError());
  return BSAM_OK;
}

int bsam_gpu_set_ghost_level(bsam_gpu* h, int level) {
  if (!h || !h->have_hierarchy) return BSAM_ERR_STATE;
  if (level < h->minlevel || level > h->finestlevel)
    return fail(h, BSAM_ERR_ARG, "set_ghost_level: level out of range");
  CU(cudaSetDevice(h->device));
  if (plan(h, level).amr) amr_ghost(h, level, 0);
  else ghost_levels(h, level, level);
  CU(cudaGetLastError());
  return BSAM_OK;
}

int bsam_gpu_fill_down(bsam_gpu* h) {
  if (!h || !h->have_hierarchy) return BSAM_ERR_STATE;
  CU(cudaSetDevice(h->device));
  if (h->amr) filldown(h);
  CU(cudaGetLastError());
  return BSAM_OK;
}

int bsam_gpu_restrict_level(bsam_gpu* h, int level) {
  if (!h || !h->have_hierarchy) return BSAM_ERR_STATE;
  if (level < 1 || level > h->finestlevel)
    return fail(h, BSAM_ERR_ARG, "restrict_level needs a refined level");
  CU(cudaSetDevice(h->device));
  const LevelPlan& L = plan(h, level);
  if (h->rp.ndims == 2)
    launch_after(h, k_filldown<2>, L.ncoarse, block_dim(), 0, h->d_patches, L.d_coarse);
  else
    launch_after(h, k_filldown<3>, L.ncoarse, block_dim(), 0, h->d_patches, L.d_coarse);
  ++h->stats.launches;
  amr_ghost(h, level - 1, 0);
  CU(cudaGetLastError());
  return BSAM_OK;
}

int bsam_gpu_copy_q_to_qold(bsam_gpu* h) {
  if (!h || !h->have_hierarchy) return BSAM_ERR_STATE;
  CU(cudaSetDevice(h->device));
  // qold exists on levels >= root only (Source reads it there).
  if (h->nqold_spans == 0) return BSAM_OK;
  k_copy_spans<<<copy_spans_grid(h->qold_span_max, h->nqold_spans), 256, 0, h->stream>>>(
      h->d_qold_spans);
  ++h->stats.launches;
  CU(cudaGetLastError());
  return BSAM_OK;
}

int bsam_gpu_multigrid_iterations(bsam_gpu* h, int* nvcycles, double* residual, int* converged) {
  if (!h || !h->have_hierarchy) return BSAM_ERR_STATE;
  CU(cudaSetDevice(h->device));
  const int nd = h->rp.ndims;
  const dim3 b = block_dim();
  // FillDown(solution) (afas:47) over the refined levels; below the root it
  // and FillDown(source) (afas:66, 90) only write regions that
  // RestrictSolution / CoarseLoadingFunction overwrite before any read, so
  // they are not issued.  Then GetSourceFunction + UpdateSourceFunction on
  // the state patches of levels >= root (afas:57-64).
  if (h->amr) filldown(h);
  if (nd == 2) k_source<double, 2><<<h->nstate, b, 0, h->stream>>>(h->d_patches, h->d_state);
  else k_source<double, 3><<<h->nstate, b, 0, h->stream>>>(h->d_patches, h->d_state);
  ++h->stats.launches;
  // Mixed form: the FP32 working copy and its right-hand side for the first
  // V-cycle (the norm computed here is not a convergence test).
  if (h->mixed) launch_resid(h);
  h->trace.clear();
  int it = 0, conv = 0;
  double res = 0.0;
  if (h->tuning.graph == 0 && !h->profiling) {
    if (h->chain_loop) {
      // Every level in one cluster's shared memory: the loop is one launch.
      launch_chain(h, ChainLoop{h->rp.maxvcycles, 0, h->rp.qerrortol, h->denom, h->d_status,
                                h->d_trace});
      CU(cudaGetLastError());
      h->graph_kernels_per_vcycle = 0;
    } else {
      // The whole V-cycle loop as one graph launch (device-side WHILE node).
      if (!h->step_exec) {
        const int rc = build_step_graph(h);
        if (rc) return rc;
      }
      k_mg_begin<<<1, 1, 0, h->stream>>>(h->d_status);
      CU(cudaGetLastError());
      CU(cudaGraphLaunch(h->step_exec, h->stream));
      ++h->stats.launches;
    }
    CU(cudaMemcpyAsync(h->h_status, h->d_status, status_bytes(h->rp.maxvcycles),
                       cudaMemcpyDeviceToHost, h->stream));
    CU(cudaStreamSynchronize(h->stream));
    it = std::max(1, std::min(h->h_status->iters, h->rp.maxvcycles));
    h->stats.launches += (int64_t)h->graph_kernels_per_vcycle * h->h_status->iters;
    res = h->h_status->residual;
    h->trace.assign(h->h_trace, h->h_trace + it);
    if (nvcycles) *nvcycles = it;
    if (residual) *residual = res;
    if (converged) *converged = 0;
    if (h->h_status->kerr)
      return fail(h, BSAM_ERR_CUDA, "a fused smoothing stage timed out waiting for its copies");
    if (!std::isfinite(res)) return fail(h, BSAM_ERR_DIVERGED, "residual is not finite");
    if (converged) *converged = h->h_status->converged;
    return BSAM_OK;
  }
  for (it = 1; it <= h->rp.maxvcycles; ++it) {
    iteration(h);
    CU(cudaGetLastError());
    CU(cudaMemcpyAsync(h->h_status, h->d_status, sizeof(DevStatus), cudaMemcpyDeviceToHost,
                       h->stream));
    CU(cudaStreamSynchronize(h->stream));
    drain_events(h);
    res = h->h_status->residual;
    if (h->h_status->kerr) {
      if (nvcycles) *nvcycles = it;
      if (residual) *residual = res;
      if (converged) *converged = 0;
      return fail(h, BSAM_ERR_CUDA, "a fused smoothing stage timed out waiting for its copies");
    }
    h->trace.push_back(res);
    if (!std::isfinite(res)) {
      if (nvcycles) *nvcycles = it;
      if (residual) *residual = res;
      if (converged) *converged = 0;
      return fail(h, BSAM_ERR_DIVERGED, "residual is not finite");
    }
    if (res < h->rp.qerrortol) {
      conv = 1;
      break;
    }
  }
  if (it > h->rp.maxvcycles) it = h->rp.maxvcycles;
  if (nvcycles) *nvcycles = it;
  if (residual) *residual = res;
  if (converged) *converged = conv;
  return BSAM_OK;
}

int bsam_gpu_residual_trace(bsam_gpu* h, double* out, int maxn) {
  if (!h) return BSAM_ERR_ARG;
  const int n = std::min<int>(maxn, (int)h->trace.size());
  for (int i = 0; i < n; ++i) out[i] = h->trace[i];
  return (int)h->trace.size();
}

int bsam_gpu_mass(bsam_gpu* h, double* mass) {
  if (!h || !h->have_hierarchy || !mass) return BSAM_ERR_STATE;
  if (h->nroot == 0) return fail(h, BSAM_ERR_UNSUPPORTED, "no root-level patch");
  CU(cudaSetDevice(h->device));
  // AfterStep2D/3D integral(1) on the root level (problem.f90:102-134).
  int root = 0;
  for (int p = 0; p < h->nuser; ++p)
    if (h->desc[p].level == 0) root = p;
  const double hh = h->hp[root].h;
  const double hd = h->rp.ndims == 2 ? hh * hh : hh * hh * hh;
  if (h->rp.ndims == 2)
    k_mass<double, 2><<<h->nroot, block_dim(), 0, h->stream>>>(
        h->d_patches, h->d_root, h->d_partials, h->d_status, h->nroot, hd);
  else
    k_mass<double, 3><<<h->nroot, block_dim(), 0, h->stream>>>(
        h->d_patches, h->d_root, h->d_partials, h->d_status, h->nroot, hd);
  ++h->stats.launches;
  CU(cudaGetLastError());
  CU(cudaMemcpyAsync(h->h_status, h->d_status, sizeof(DevStatus), cudaMemcpyDeviceToHost,
                     h->stream));
  CU(cudaStreamSynchronize(h->stream));
  *mass = h->h_status->mass;
  return BSAM_OK;
}

int bsam_gpu_errflags(bsam_gpu* h, int patch, double tol, uint8_t* flags) {
  if (!h || !h->have_hierarchy || !flags) return BSAM_ERR_ARG;
  if (patch < 0 || patch >= h->nuser || h->desc[patch].level < 0)
    return fail(h, BSAM_ERR_ARG, "errflags needs a patch on a level >= 0");
  CU(cudaSetDevice(h->device));
  const DevPatch& P = h->hp[patch];
  const int nd = h->rp.ndims;
  const size_t ncell = (size_t)P.n[0] * P.n[1] * (nd == 3 ? P.n[2] : 1);
  uint8_t* d_flags = nullptr;
  CU(cudaMalloc(&d_flags, ncell));
  const int blocks = (int)std::min<size_t>((ncell + 255) / 256, 4096);
  if (nd == 2) k_errflags<2><<<blocks, 256, 0, h->stream>>>(h->d_patches, patch, tol, d_flags);
  else k_errflags<3><<<blocks, 256, 0, h->stream>>>(h->d_patches, patch, tol, d_flags);
  ++h->stats.launches;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(flags, d_flags, ncell, cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  cudaFree(d_flags);
  if (e != cudaSuccess) return fail(h, BSAM_ERR_CUDA, cudaGetErrorString(e));
  return BSAM_OK;
}

// Copies a host task list into the handle's task buffer (grown, never
// shrunk) on the stream; the caller synchronises before the next upload.
static int upload_tasks(bsam_gpu* h, const void* src, size_t bytes) {
  if (bytes > h->regrid_cap) {
    if (h->d_regrid) cudaFree(h->d_regrid);
    h->d_regrid = nullptr;
    h->regrid_cap = 0;
    const size_t want = bytes + bytes / 2;
    if (cudaMalloc(&h->d_regrid, want) != cudaSuccess)
      return fail(h, BSAM_ERR_NOMEM, "task buffer allocation failed");
    h->regrid_cap = want;
  }
  return h2d_bounce(h, h->d_regrid, src, bytes);
}

int bsam_gpu_errflags_level(bsam_gpu* h, int level, double tol, uint8_t* flags) {
  if (!h || !h->have_hierarchy || !flags) return BSAM_ERR_ARG;
  if (level < 0 || level > h->finestlevel)
    return fail(h, BSAM_ERR_ARG, "errflags_level needs a level >= 0");
  CU(cudaSetDevice(h->device));
  const int nd = h->rp.ndims;
  size_t total = 0;
  for (int p = 0; p < h->nuser; ++p)
    if (h->desc[p].level == level) total += (size_t)cells_of(h->hp[p].n, nd);
  if (total == 0) return BSAM_OK;
  if (total > h->flags_cap) {
    if (h->d_flags) cudaFree(h->d_flags);
    h->d_flags = nullptr;
    h->flags_cap = 0;
    if (cudaMalloc(&h->d_flags, total) != cudaSuccess)
      return fail(h, BSAM_ERR_NOMEM, "flag buffer allocation failed");
    h->flags_cap = total;
  }
  // One launch over the level: a task per patch (offset into the flags).
  std::vector<FlagTask> tasks;
  size_t off = 0, ncell_max = 0;
  for (int p = 0; p < h->nuser; ++p) {
    if (h->desc[p].level != level) continue;
    const size_t ncell = (size_t)cells_of(h->hp[p].n, nd);
    tasks.push_back(FlagTask{(int64_t)off, p, 0});
    ncell_max = std::max(ncell_max, ncell);
    off += ncell;
  }
  if (tasks.size() > 65535) return fail(h, BSAM_ERR_ARG, "errflags_level: too many patches");
  const int rc = upload_tasks(h, tasks.data(), sizeof(FlagTask) * tasks.size());
  if (rc) return rc;
  const dim3 g((unsigned)std::min<size_t>((ncell_max + 255) / 256, 1024), (unsigned)tasks.size());
  const FlagTask* d_tasks = reinterpret_cast<const FlagTask*>(h->d_regrid);
  if (nd == 2) k_errflags_list<2><<<g, 256, 0, h->stream>>>(h->d_patches, d_tasks, tol, h->d_flags);
  else k_errflags_list<3><<<g, 256, 0, h->stream>>>(h->d_patches, d_tasks, tol, h->d_flags);
  ++h->stats.launches;
  CU(cudaGetLastError());
  {
    const int drc = d2h_bounce(h, flags, h->d_flags, total);
    if (drc) return drc;
  }
  return BSAM_OK;
}

int bsam_gpu_tag_level(bsam_gpu* h, int level, double tol, int ibuffer, int32_t* sat) {
  if (!h || !h->have_hierarchy || !sat || ibuffer < 0) return BSAM_ERR_ARG;
  if (level < 0 || level > h->finestlevel)
    return fail(h, BSAM_ERR_ARG, "tag_level needs a level >= 0");
  CU(cudaSetDevice(h->device));
  const int nd = h->rp.ndims;
  // The level's patches in table order, their cells concatenated.
  std::vector<FlagTask> tasks;
  std::vector<LevelPatch> lp;
  size_t total = 0, ncell_max = 0;
  for (int p = 0; p < h->nuser; ++p) {
    if (h->desc[p].level != level) continue;
    const size_t ncell = (size_t)cells_of(h->hp[p].n, nd);
    tasks.push_back(FlagTask{(int64_t)total, p, 0});
    LevelPatch L{};
    L.off = (int64_t)total;
    for (int n = 0; n < 3; ++n) {
      L.n[n] = n < nd ? h->hp[p].n[n] : 1;
      L.g0[n] = n < nd ? h->desc[p].mglobal[n][0] : 1;
    }
    lp.push_back(L);
    ncell_max = std::max(ncell_max, ncell);
    total += ncell;
  }
  if (total == 0) return BSAM_OK;
  const int np = (int)tasks.size();
  if (np > 65535) return fail(h, BSAM_ERR_ARG, "tag_level: too many patches");
  if (2 * total > h->flags_cap) {
    if (h->d_flags) cudaFree(h->d_flags);
    h->d_flags = nullptr;
    h->flags_cap = 0;
    if (cudaMalloc(&h->d_flags, 2 * total) != cudaSuccess)
      return fail(h, BSAM_ERR_NOMEM, "flag buffer allocation failed");
    h->flags_cap = 2 * total;
  }
  if (total > h->sat_cap) {
    if (h->d_sat) cudaFree(h->d_sat);
    h->d_sat = nullptr;
    h->sat_cap = 0;
    if (cudaMalloc(&h->d_sat, sizeof(int32_t) * total) != cudaSuccess)
      return fail(h, BSAM_ERR_NOMEM, "summed-area table allocation failed");
    h->sat_cap = total;
  }
  // One upload: the tagging tasks, then the level's patches.
  std::vector<unsigned char> buf(sizeof(FlagTask) * np + sizeof(LevelPatch) * np);
  std::memcpy(buf.data(), tasks.data(), sizeof(FlagTask) * np);
  std::memcpy(buf.data() + sizeof(FlagTask) * np, lp.data(), sizeof(LevelPatch) * np);
  int rc = upload_tasks(h, buf.data(), buf.size());
  if (rc) return rc;
  const FlagTask* d_tasks = reinterpret_cast<const FlagTask*>(h->d_regrid);
  const LevelPatch* d_lp = reinterpret_cast<const LevelPatch*>(h->d_regrid + sizeof(FlagTask) * np);
  uint8_t* raw = h->d_flags;
  uint8_t* buffered = h->d_flags + total;
  const dim3 g((unsigned)std::min<size_t>((ncell_max + 255) / 256, 1024), (unsigned)np);
  if (nd == 2) {
    k_errflags_list<2><<<g, 256, 0, h->stream>>>(h->d_patches, d_tasks, tol, raw);
    k_buffer_list<2><<<g, 256, 0, h->stream>>>(d_lp, np, ibuffer, raw, buffered);
    k_sat_list<2><<<np, 256, 0, h->stream>>>(d_lp, buffered, h->d_sat);
  } else {
    k_errflags_list<3><<<g, 256, 0, h->stream>>>(h->d_patches, d_tasks, tol, raw);
    k_buffer_list<3><<<g, 256, 0, h->stream>>>(d_lp, np, ibuffer, raw, buffered);
    k_sat_list<3><<<np, 256, 0, h->stream>>>(d_lp, buffered, h->d_sat);
  }
  h->stats.launches += 3;
  CU(cudaGetLastError());
  return d2h_bounce(h, sat, h->d_sat, sizeof(int32_t) * total);
}

int bsam_gpu_init_patch(bsam_gpu* h, int patch) {
  if (!h || !h->have_hierarchy) return BSAM_ERR_ARG;
  if (patch < 0 || patch >= h->nuser || h->desc[patch].level < 1)
    return fail(h, BSAM_ERR_ARG, "init_patch needs a refined patch (level >= 1)");
  const DevPatch& P = h->hp[patch];
  if (!P.qo[0] || h->mixed) return fail(h, BSAM_ERR_UNSUPPORTED, "init_patch: FP64 form only");
  CU(cudaSetDevice(h->device));
  const int nd = h->rp.ndims;
  const size_t ncoarse = (size_t)(P.cn[0] + 2) * (P.cn[1] + 2) * (nd == 3 ? P.cn[2] + 2 : 1);
  const int blocks = (int)std::min<size_t>((ncoarse + 255) / 256, 4096);
  if (nd == 2) k_init_mc<2><<<blocks, 256, 0, h->stream>>>(h->d_patches, patch);
  else k_init_mc<3><<<blocks, 256, 0, h->stream>>>(h->d_patches, patch);
  ++h->stats.launches;
  CU(cudaGetLastError());
  return BSAM_OK;
}

int bsam_gpu_energy(bsam_gpu* h, double* energy) {
  if (!h || !h->have_hierarchy || !energy) return BSAM_ERR_STATE;
  if (h->rp.ndims != 2 || h->amr || h->nroot == 0)
    return fail(h, BSAM_ERR_UNSUPPORTED,
                "the energy is defined for a 2D hierarchy without refined levels (AfterStep2D "
                "at level 0)");
  CU(cudaSetDevice(h->device));
  int root = 0;
  for (int p = 0; p < h->nuser; ++p)
    if (h->desc[p].level == 0) root = p;
  const double hh = h->hp[root].h, h2 = hh * hh;
  const double tmp = h->rp.eps * h->rp.eps / h2 / 4.0;  // eps2/h2/4.0 (problem.f90:355)
  double s[2];
  for (int which = 0; which < 2; ++which) {
    k_energy2<double><<<h->nroot, block_dim(), 0, h->stream>>>(
        h->d_patches, h->d_root, h->d_partials, h->d_status, h->nroot, which);
    ++h->stats.launches;
    CU(cudaGetLastError());
    CU(cudaMemcpyAsync(h->h_status, h->d_status, sizeof(DevStatus), cudaMemcpyDeviceToHost,
                       h->stream));
    CU(cudaStreamSynchronize(h->stream));
    s[which] = h->h_status->esum;
  }
  *energy = h2 * (s[0] + tmp * s[1]);
  return BSAM_OK;
}

int bsam_gpu_after_step_stats(bsam_gpu* h, double* integral) {
  if (!h || !h->have_hierarchy || !integral) return BSAM_ERR_ARG;
  const int nd = h->rp.ndims;
  // The terms, in the order AfterStepStatistics adds them: levels finest to
  // root, ApplyOnLevel (table) order within a level.  Per patch: sum(c), then
  // (2D) Ff and squared-difference sums; on a refined patch the same over its
  // parent's footprint.
  struct Term {
    int patch, kind, lo[3], hi[3];
  };
  std::vector<Term> terms;
  std::vector<int> order;
  for (int level = h->finestlevel; level >= 0; --level)
    for (int p = 0; p < h->nuser; ++p)
      if (h->desc[p].level == level) order.push_back(p);
  for (int p : order) {
    const bsam_patch_desc& d = h->desc[p];
    if (h->hp[p].prec != PREC_F64) return fail(h, BSAM_ERR_UNSUPPORTED, "stats need FP64 patches");
    const int nk = nd == 2 ? 3 : 1;  // 2D adds the two energy sums
    for (int side = 0; side < (d.level > 0 ? 2 : 1); ++side) {
      Term t{};
      t.patch = side == 0 ? p : d.parent;
      if (side == 1 && h->hp[t.patch].prec != PREC_F64)
        return fail(h, BSAM_ERR_UNSUPPORTED, "stats need FP64 patches");
      for (int n = 0; n < 3; ++n) {
        if (n >= nd) {
          t.lo[n] = t.hi[n] = 0;
        } else if (side == 0) {
          t.lo[n] = 1;
          t.hi[n] = d.mx[n];
        } else {
          t.lo[n] = d.mbounds[n][0];
          t.hi[n] = d.mbounds[n][1];
        }
      }
      for (int kind = 0; kind < nk; ++kind) {
        t.kind = kind;
        terms.push_back(t);
      }
    }
  }
  // Split each term's rows over CTAs (about 16k cells a CTA).
  std::vector<StatBlock> blocks;
  std::vector<int> first(terms.size() + 1, 0);
  for (size_t ti = 0; ti < terms.size(); ++ti) {
    const Term& t = terms[ti];
    const int nx = t.hi[0] - t.lo[0] + 1, ny = t.hi[1] - t.lo[1] + 1;
    const int nz = nd == 3 ? t.hi[2] - t.lo[2] + 1 : 1;
    const int rows = ny * nz;
    const int per = std::max(1, 16384 / std::max(1, nx));
    first[ti] = (int)blocks.size();
    for (int r0 = 0; r0 < rows; r0 += per) {
      StatBlock b{};
      b.patch = t.patch;
      b.kind = t.kind;
      for (int n = 0; n < 3; ++n) {
        b.lo[n] = t.lo[n];
        b.hi[n] = t.hi[n];
      }
      b.row0 = r0;
      b.row1 = std::min(rows, r0 + per);
      blocks.push_back(b);
    }
  }
  first[terms.size()] = (int)blocks.size();
  const int nb = (int)blocks.size();
  CU(cudaSetDevice(h->device));
  StatBlock* d_blocks = nullptr;
  double* d_part = nullptr;
  std::vector<double> part(nb);
  cudaError_t e = cudaMalloc(&d_blocks, sizeof(StatBlock) * nb);
  if (e == cudaSuccess) e = cudaMalloc(&d_part, sizeof(double) * nb);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_blocks, blocks.data(), sizeof(StatBlock) * nb, cudaMemcpyHostToDevice,
                        h->stream);
  if (e == cudaSuccess) {
    if (nd == 2) k_stats<2><<<nb, 256, 0, h->stream>>>(h->d_patches, d_blocks, d_part);
    else k_stats<3><<<nb, 256, 0, h->stream>>>(h->d_patches, d_blocks, d_part);
    ++h->stats.launches;
    e = cudaGetLastError();
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(part.data(), d_part, sizeof(double) * nb, cudaMemcpyDeviceToHost,
                        h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  if (d_blocks) cudaFree(d_blocks);
  if (d_part) cudaFree(d_part);
  if (e != cudaSuccess) return fail(h, BSAM_ERR_CUDA, cudaGetErrorString(e));
  auto term_sum = [&](size_t ti) {
    double s = 0.0;
    for (int b = first[ti]; b < first[ti + 1]; ++b) s += part[b];
    return s;
  };
  // Combine as AfterStep2D/3D do.
  const double eps2 = h->rp.eps * h->rp.eps;
  double r1 = 0.0, r2 = 0.0;
  size_t ti = 0;
  auto energy = [&](double hh, double sF, double sG) {
    const double h2 = hh * hh;
    return h2 * (sF + eps2 / h2 / 4.0 * sG);
  };
  for (int p : order) {
    const bsam_patch_desc& d = h->desc[p];
    const double hh = h->hp[p].h, ch = hh * 2.0;
    const double hd = nd == 2 ? hh * hh : hh * hh * hh;
    const double chd = nd == 2 ? ch * ch : ch * ch * ch;
    if (nd == 2) {
      const double s = term_sum(ti), sF = term_sum(ti + 1), sG = term_sum(ti + 2);
      ti += 3;
      if (d.level == 0) {
        r1 = r1 + hd * s;
        r2 = r2 + energy(hh, sF, sG);
      } else {
        const double cs = term_sum(ti), cF = term_sum(ti + 1), cG = term_sum(ti + 2);
        ti += 3;
        r1 = r1 + hd * s - chd * cs;
        r2 = r2 + energy(hh, sF, sG) - energy(ch, cF, cG);
      }
    } else {
      const double s = term_sum(ti);
      ti += 1;
      if (d.level == 0) {
        r1 = r1 + hd * s;
      } else {
        const double cs = term_sum(ti);
        ti += 1;
        r1 = r1 + hd * s - chd * cs;
      }
    }
  }
  integral[0] = r1;
  integral[1] = r2;
  return BSAM_OK;
}

int bsam_gpu_stash(bsam_gpu* h) {
  if (!h || !h->have_hierarchy) return BSAM_ERR_STATE;
  if (h->mixed) return fail(h, BSAM_ERR_UNSUPPORTED, "regridding: FP64 form only");
  CU(cudaSetDevice(h->device));
  h->stash_hp.assign(h->nuser, DevPatch{});
  h->stash_desc = h->desc;
  size_t total = 0;
  std::vector<size_t> off(h->nuser, 0);
  for (int p = 0; p < h->nuser; ++p)
    if (h->desc[p].level >= 1) {
      off[p] = total;
      total += 2 * (size_t)h->field_elems[p] * sizeof(double);
    }
  if (total == 0) return BSAM_OK;
  if (total > h->stash_cap) {
    if (h->d_stash) cudaFree(h->d_stash);
    h->d_stash = nullptr;
    h->stash_cap = 0;
    const size_t want = total + total / 2;  // headroom for the next steps
    if (cudaMalloc(&h->d_stash, want) != cudaSuccess)
      return fail(h, BSAM_ERR_NOMEM, "stash allocation failed");
    h->stash_cap = want;
  }
  const int64_t lead = 128 / sizeof(double) - 1;
  std::vector<CopySpan> spans;
  int64_t span_max = 0;
  for (int p = 0; p < h->nuser; ++p) {
    if (h->desc[p].level < 1) continue;
    DevPatch S = h->hp[p];
    for (int c = 0; c < 2; ++c) {
      double* dst = reinterpret_cast<double*>(h->d_stash + off[p]) + c * h->field_elems[p];
      spans.push_back(CopySpan{static_cast<const double*>(S.q[c]) - lead, dst, h->field_elems[p]});
      S.q[c] = dst + lead;
    }
    span_max = std::max(span_max, h->field_elems[p]);
    h->stash_hp[p] = S;
  }
  if (spans.size() > h->stash_spans_cap) {
    if (h->d_stash_spans) cudaFree(h->d_stash_spans);
    h->d_stash_spans = nullptr;
    h->stash_spans_cap = 0;
    const size_t want = spans.size() + spans.size() / 2;
    if (cudaMalloc(&h->d_stash_spans, sizeof(CopySpan) * want) != cudaSuccess)
      return fail(h, BSAM_ERR_NOMEM, "stash allocation failed");
    h->stash_spans_cap = want;
  }
  {
    const int urc = h2d_bounce(h, h->d_stash_spans, spans.data(), sizeof(CopySpan) * spans.size());
    if (urc) return urc;
  }
  k_copy_spans<<<copy_spans_grid(span_max, (int64_t)spans.size()), 256, 0, h->stream>>>(
      h->d_stash_spans);
  ++h->stats.launches;
  CU(cudaGetLastError());
  // The span list is host memory: wait until it has been read.
  CU(cudaStreamSynchronize(h->stream));
  return BSAM_OK;
}

int bsam_gpu_regrid(bsam_gpu* h, int npatch, const bsam_patch_desc* patches, int finestlevel,
                    const int* carry, int ntransfer, const int* transfer) {
  if (!h || !h->have_hierarchy || npatch <= 0 || !patches || !carry || ntransfer < 0 ||
      (ntransfer > 0 && !transfer))
    return BSAM_ERR_ARG;
  if (h->mixed) return fail(h, BSAM_ERR_UNSUPPORTED, "regridding: FP64 form only");
  const int nd = h->rp.ndims;
  const int nold = h->nuser;
  for (int i = 0; i < npatch; ++i) {
    const int o = carry[i];
    if (o < -1 || o >= nold) return fail(h, BSAM_ERR_ARG, "regrid: carry index out of range");
    if (o >= 0) {
      if (h->desc[o].level != patches[i].level)
        return fail(h, BSAM_ERR_ARG, "regrid: a carried patch changes level");
      for (int n = 0; n < nd; ++n)
        if (h->desc[o].mx[n] != patches[i].mx[n])
          return fail(h, BSAM_ERR_ARG, "regrid: a carried patch changes size");
    } else if (patches[i].level < 1) {
      return fail(h, BSAM_ERR_ARG, "regrid: only refined patches may be new");
    }
  }
  for (int t = 0; t < ntransfer; ++t) {
    const int c = transfer[2 * t], s = transfer[2 * t + 1];
    if (c < 0 || c >= npatch || carry[c] >= 0 || s < 0 || s >= (int)h->stash_hp.size() ||
        h->stash_desc[s].level != patches[c].level)
      return fail(h, BSAM_ERR_ARG, "regrid: a transfer names no new grid and stashed grid");
  }
  CU(cudaSetDevice(h->device));
  CU(cudaStreamSynchronize(h->stream));
  // Keep the old arena (the carried q and qold) until the copies are done.
  char* old_arena = h->d_arena;
  const size_t old_bytes = h->arena_bytes;
  h->d_arena = nullptr;
  const std::vector<DevPatch> old_hp = h->hp;
  const std::vector<int64_t> old_fe = h->field_elems;
  h->regridding = true;
  int rc = bsam_gpu_set_hierarchy(h, npatch, patches, finestlevel);
  h->regridding = false;
  if (rc != BSAM_OK) {
    cudaFree(old_arena);
    return rc;
  }
  // The device work as three launches from one uploaded task list: the
  // carried patches' q and qold (whole field allocations), InitFields of every
  // new grid from its carried parent, then the transfers from the stash.
  const int64_t lead = 128 / sizeof(double) - 1;
  cudaError_t e = cudaSuccess;
  std::vector<CopySpan> spans;
  std::vector<int> children;
  std::vector<TransferTask> tasks;
  int64_t span_max = 0, child_max = 0, task_max = 0;
  for (int i = 0; i < npatch; ++i) {
    const int o = carry[i];
    if (o < 0) {
      const DevPatch& P = h->hp[i];
      children.push_back(i);
      child_max = std::max<int64_t>(
          child_max, (int64_t)(P.cn[0] + 2) * (P.cn[1] + 2) * (nd == 3 ? P.cn[2] + 2 : 1));
      continue;
    }
    const DevPatch& A = old_hp[o];
    const DevPatch& B = h->hp[i];
    if (old_fe[o] != h->field_elems[i]) {
      e = cudaErrorInvalidValue;
      break;
    }
    for (int c = 0; c < 2; ++c) {
      spans.push_back(CopySpan{static_cast<const double*>(A.q[c]) - lead,
                               static_cast<double*>(B.q[c]) - lead, old_fe[o]});
      if (A.qo[c] && B.qo[c])
        spans.push_back(CopySpan{static_cast<const double*>(A.qo[c]) - lead,
                                 static_cast<double*>(B.qo[c]) - lead, old_fe[o]});
    }
    span_max = std::max(span_max, old_fe[o]);
  }
  for (int t = 0; t < ntransfer && e == cudaSuccess; ++t) {
    const int c = transfer[2 * t], s = transfer[2 * t + 1];
    const bsam_patch_desc& T = patches[c];
    const bsam_patch_desc& S = h->stash_desc[s];
    TransferTask tk{};
    tk.S = h->stash_hp[s];
    tk.target = c;
    bool empty = false;
    int64_t cells = 1;
    for (int n = 0; n < 3; ++n) {
      if (n >= nd) {
        tk.n[n] = 1;
        continue;
      }
      const int lo = std::max(T.mglobal[n][0], S.mglobal[n][0]);
      const int hi = std::min(T.mglobal[n][1], S.mglobal[n][1]);
      empty |= hi < lo;
      tk.n[n] = hi - lo + 1;
      tk.si[n] = lo - S.mglobal[n][0] + 1;
      tk.ti[n] = lo - T.mglobal[n][0] + 1;
      cells *= tk.n[n];
    }
    if (empty) continue;
    tasks.push_back(tk);
    task_max = std::max(task_max, cells);
  }
  if (e == cudaSuccess && (spans.size() > 65535 || children.size() > 65535 || tasks.size() > 65535))
    e = cudaErrorInvalidValue;  // one grid row per item: at most 65535 of each
  if (e == cudaSuccess && (!spans.empty() || !children.empty() || !tasks.empty())) {
    // Layout: spans, children, tasks; 256-byte aligned pieces.
    const size_t o_sp = 0;
    const size_t o_ch = (size_t)roundup((int64_t)(sizeof(CopySpan) * spans.size()), 256);
    const size_t o_tk = o_ch + (size_t)roundup((int64_t)(sizeof(int) * children.size()), 256);
    const size_t bytes = o_tk + sizeof(TransferTask) * tasks.size();
    h->regrid_host.assign(bytes, 0);
    unsigned char* img = h->regrid_host.data();
    if (!spans.empty()) std::memcpy(img + o_sp, spans.data(), sizeof(CopySpan) * spans.size());
    if (!children.empty()) std::memcpy(img + o_ch, children.data(), sizeof(int) * children.size());
    if (!tasks.empty()) std::memcpy(img + o_tk, tasks.data(), sizeof(TransferTask) * tasks.size());
    const int urc = upload_tasks(h, img, bytes);
    if (urc != BSAM_OK) {
      cudaFree(old_arena);
      return urc;
    }
    const auto grid_x = [](int64_t n) { return (unsigned)std::min<int64_t>((n + 255) / 256, 64); };
    if (e == cudaSuccess && !spans.empty()) {
      k_copy_spans<<<copy_spans_grid(span_max, (int64_t)spans.size()), 256, 0, h->stream>>>(
          reinterpret_cast<const CopySpan*>(h->d_regrid + o_sp));
      ++h->stats.launches;
      e = cudaGetLastError();
    }
    if (e == cudaSuccess && !children.empty()) {
      const dim3 g(grid_x(child_max), (unsigned)children.size());
      const int* d_ch = reinterpret_cast<const int*>(h->d_regrid + o_ch);
      if (nd == 2) k_init_mc_list<2><<<g, 256, 0, h->stream>>>(h->d_patches, d_ch);
      else k_init_mc_list<3><<<g, 256, 0, h->stream>>>(h->d_patches, d_ch);
      ++h->stats.launches;
      e = cudaGetLastError();
    }
    if (e == cudaSuccess && !tasks.empty()) {
      const dim3 g(grid_x(task_max), (unsigned)tasks.size());
      const TransferTask* d_tk = reinterpret_cast<const TransferTask*>(h->d_regrid + o_tk);
      if (nd == 2) k_transfer_list<2><<<g, 256, 0, h->stream>>>(h->d_patches, d_tk);
      else k_transfer_list<3><<<g, 256, 0, h->stream>>>(h->d_patches, d_tk);
      ++h->stats.launches;
      e = cudaGetLastError();
    }
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  // The old arena becomes the spare (the larger of it and the current spare).
  if (h->spare_arena && h->spare_bytes >= old_bytes) {
    cudaFree(old_arena);
  } else {
    if (h->spare_arena) cudaFree(h->spare_arena);
    h->spare_arena = old_arena;
    h->spare_bytes = old_bytes;
  }
  if (e != cudaSuccess) return fail(h, BSAM_ERR_CUDA, cudaGetErrorString(e));
  return BSAM_OK;
}

int bsam_gpu_set_tuning(bsam_gpu* h, const bsam_tuning* t) {
  if (!h || !t) return BSAM_ERR_ARG;
  if (t->fuse_smoother < -1 || t->fuse_smoother > 1 || t->chunk < 0 || t->graph < -1 ||
      t->graph > 0)
    return BSAM_ERR_ARG;
  h->tuning = *t;
  if (h->step_exec) {
    cudaGraphExecDestroy(h->step_exec);
    h->step_exec = nullptr;
  }
  return BSAM_OK;
}

int bsam_gpu_get_stream(bsam_gpu* h, void** stream) {
  if (!h || !stream) return BSAM_ERR_ARG;
  *stream = (void*)h->stream;
  return BSAM_OK;
}

int bsam_gpu_profile(bsam_gpu* h, int enable) {
  if (!h) return BSAM_ERR_ARG;
  if (enable) {
    h->stats = bsam_gpu_stats{};
    h->ev_used = 0;
    if (h->have_hierarchy) {
      h->ev_cells = 0;
      const LevelPlan& F = plan(h, h->finestlevel);
      for (int p : F.patches) h->ev_cells += cells_of(h->hp[p].n, h->rp.ndims);
      h->ev_bytes = elem_bytes(F.prec);
    }
  }
  h->profiling = enable != 0;
  return BSAM_OK;
}

int bsam_gpu_get_stats(bsam_gpu* h, bsam_gpu_stats* out) {
  if (!h || !out) return BSAM_ERR_ARG;
  if (h->ev_used) {
    cudaStreamSynchronize(h->stream);
    drain_events(h);
  }
  *out = h->stats;
  return BSAM_OK;
}

int bsam_gpu_destroy(bsam_gpu* h) {
  if (!h) return BSAM_ERR_ARG;
  cudaSetDevice(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (auto& e : h->ev_pool) {
    cudaEventDestroy(e.first);
    cudaEventDestroy(e.second);
  }
  free_hierarchy(h);
  if (h->h_pin) cudaFreeHost(h->h_pin);
  for (cudaEvent_t e : h->slot_ev)
    if (e) cudaEventDestroy(e);
  for (cudaStream_t st : h->copy_streams)
    if (st) cudaStreamDestroy(st);
  if (h->spare_arena) cudaFree(h->spare_arena);
  if (h->d_stash) cudaFree(h->d_stash);
  if (h->d_stash_spans) cudaFree(h->d_stash_spans);
  if (h->d_meta) cudaFree(h->d_meta);
  if (h->d_regrid) cudaFree(h->d_regrid);
  if (h->d_flags) cudaFree(h->d_flags);
  if (h->d_sat) cudaFree(h->d_sat);
  if (h->d_status) cudaFree(h->d_status);
  if (h->h_status) cudaFreeHost(h->h_status);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
  PieceBlocks::get().count(-1);
  return BSAM_OK;
}

}  // extern "C"
