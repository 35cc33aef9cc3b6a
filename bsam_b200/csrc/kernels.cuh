// kernels.cuh -- FAS V-cycle kernels over the device patch table.
//
// One per-cell device function per reference routine on the hot path, and
// two ways of mapping cells to threads:
//  * grid kernels (k_*) take a work list of Items (patch, tile) so that one
//    launch covers every patch of a level.  A CTA is 32 x TILE_Y threads;
//    every thread owns a pair of adjacent cells in x (one red, one black),
//    which keeps warps on 64 contiguous cells of a row;
//  * block loops (bottom.cuh) walk all cells of a small patch with one CTA.
//
// Ghost cells: for patches whose faces are all physical (DevPatch::wt), the
// code that changes a boundary cell also writes the ghost cells SetBC would
// derive from it (write-through).  This reproduces SetGhost's result exactly:
// SetBC2D/3D (boundary.f90:661-885) processes the faces in order and copies
// whole rows including the ghost rows, so a ghost outside in the set S of
// dimensions ends up as the map of each face in S (ascending dimension)
// applied to the interior cell reflected across all of S.
#pragma once
#include <vector>

#include <algorithm>

#include "bsam_types.h"
#include "problem.cuh"

namespace bsam {

// SMs of a B200: sizes of grids and shares of work; no result depends on it.
constexpr int B200_SMS = 148;

template <class T> __device__ __forceinline__ T* fld(void* p) { return static_cast<T*>(p); }

// Programmatic dependent launch: a kernel that starts with this may be launched
// (launch_after, bsam_gpu.cu) while the one before it still runs; here it waits
// until that one has completed and its results are visible, and lets the next
// one be launched in its turn.
__device__ __forceinline__ void next_may_launch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  next_may_launch();
}

// The entries of an n-long work list a CTA takes: runs of `chunk`
// consecutive entries, run r going to CTA r mod gridDim.x (chunk 1 is the
// plain grid-stride order).  A list holds each problem's tiles in a row, so
// the tiles of a run mostly share their patch records, which after the
// run's first tile come from L1 instead of a chain of L2 round trips; the
// order in which a CTA visits tiles changes no result.  A list too short to
// give every CTA a run is taken tile by tile (fit): in runs of two the coarse
// levels' lists kept half as many CTAs busy.  The ticks of 24 problems of 32^3 and
// 64^3: runs of two throughout 20.8 ms, single tiles throughout 19.4; later, other
// kernels having become faster, single tiles 16.8 and by this rule 16.4.
struct TileRuns {
  int chunk;
  __device__ __forceinline__ TileRuns fit(int n, int takers) const {
    return TileRuns{n >= takers * chunk ? chunk : 1};
  }
  __device__ __forceinline__ TileRuns fit(int n) const { return fit(n, (int)gridDim.x); }
  __device__ __forceinline__ int first() const { return (int)blockIdx.x * chunk; }
  __device__ __forceinline__ int next(int x) const {
    ++x;
    return (x % chunk) != 0 ? x : x + (int)(gridDim.x - 1) * chunk;
  }
};

// The same for kernels whose warps take a tile each.
struct WarpRuns {
  int chunk, skip, at;
  __device__ __forceinline__ WarpRuns(const TileRuns& R, int n) {
    const int w = (threadIdx.x + blockDim.x * threadIdx.y) / 32;
    const int warps = blockDim.x * blockDim.y / 32;
    chunk = R.fit(n, (int)gridDim.x * warps).chunk;
    skip = ((int)gridDim.x * warps - 1) * chunk;
    at = ((int)blockIdx.x * warps + w) * chunk;
  }
  __device__ __forceinline__ int next(int x) const {
    ++x;
    return (x % chunk) != 0 ? x : x + skip;
  }
};

// The pre-smoothed state of a level: the second buffer when the level's
// stages run the fused kernel (q -> qb -> q), else q itself.
__device__ __forceinline__ void* const* mid_state(const DevPatch& P) {
  return P.fused ? P.qb : P.q;
}

__device__ __forceinline__ int64_t cidx(const DevPatch& P, int i, int j, int k) {
  return (int64_t)i + (int64_t)j * P.sy + (int64_t)k * P.sz;
}

// Two neighbouring cells of a row, the first of odd index: rows start so that
// cell 1 is 128-byte aligned, so the pair is one aligned load.
template <class T> struct PairOf;
template <> struct PairOf<float> { using V = float2; };
template <> struct PairOf<double> { using V = double2; };
template <class T>
__device__ __forceinline__ typename PairOf<T>::V load_pair(const T* p) {
  return *reinterpret_cast<const typename PairOf<T>::V*>(p);
}

// ---- work tiles --------------------------------------------------------------
//
// Tiles of the kernels whose result does not depend on which thread takes which
// cell (all but the sums, whose tiles are TILE_X x TILE_Y): W lanes a row, two
// cells a lane, BLOCK_THREADS / W rows of one plane.  W is the least power of
// two that covers a row, up to a warp: on rows of 24 cells the fixed 32 lanes
// left 20 of them idle.
__host__ __device__ inline int work_lanes(int n0) {
  return n0 <= 8 ? 4 : n0 <= 16 ? 8 : n0 <= 32 ? 16 : 32;
}

inline void work_tiles(int patch, const int* n, int nd, std::vector<Item>& out) {
  const int W = work_lanes(n[0]), rows = BLOCK_THREADS / W;
  for (int z = 0; z < (nd == 3 ? n[2] : 1); ++z)
    for (int y = 0; y < (n[1] + rows - 1) / rows; ++y)
      for (int x = 0; x < (n[0] + 2 * W - 1) / (2 * W); ++x) out.push_back(Item{patch, x, y, z});
}

// A thread's place in a work tile: its pair of cells starts at i0; as two
// strided cells it takes a0 and a0 + W.
template <int D>
struct WorkPlace {
  int W, i0, a0, j, k;
  __device__ __forceinline__ WorkPlace(const Item& it, int n0) {
    W = work_lanes(n0);
    const int t = threadIdx.x + 32 * threadIdx.y, lane = t & (W - 1);
    j = it.ty * (BLOCK_THREADS / W) + t / W + 1;
    k = D == 3 ? it.tz + 1 : 0;
    i0 = 2 * (it.tx * W + lane) + 1;
    a0 = 2 * it.tx * W + lane + 1;
  }
};

template <class T> __device__ __forceinline__ T bc_map(int code, T v) {
  return code == BC_REFLECT ? T(2) - v : (code == BC_NEGATE ? -v : v);
}

// Choice s of one dimension for a ghost combination: 0 = the cell's own
// coordinate, 1 = the low ghost (fed by coordinate 1 on a physical low face,
// by coordinate n on a periodic one), 2 = the high ghost (fed by coordinate n
// on a physical high face, by coordinate 1 on a periodic one).
__device__ __forceinline__ bool ghost_choice(int s, int co, int n, int lo_code, int hi_code,
                                             int& g, int& code) {
  if (s == 0) {
    g = co;
    code = BC_NONE;
    return true;
  }
  if (s == 1) {
    g = 0;
    code = lo_code;
    if (lo_code == BC_PERIODIC) return co == n;
    return co == 1 && lo_code != BC_NONE;
  }
  g = n + 1;
  code = hi_code;
  if (hi_code == BC_PERIODIC) return co == 1;
  return co == n && hi_code != BC_NONE;
}

// The one ghost of a dimension that coordinate co feeds, as its distance in that
// dimension (0: none; 2 n + 1, which is none: two) and its face's code.
__device__ __forceinline__ int ghost_step(int co, int n, int lo_code, int hi_code, int& code) {
  const bool lo = lo_code == BC_PERIODIC ? co == n : co == 1 && lo_code != BC_NONE;
  const bool hi = hi_code == BC_PERIODIC ? co == 1 : co == n && hi_code != BC_NONE;
  code = lo ? lo_code : hi_code;
  return lo && hi ? 2 * n + 1 : lo ? -co : hi ? n + 1 - co : 0;
}

// Ghost write-through for the cell (i,j,k) of patch P whose new values are
// (v0, v1): every combination of the dimensions' choices.
template <class T, int D>
__device__ __forceinline__ void write_through_all(const DevPatch& P, T* q0, T* q1, int i, int j,
                                                  int k, T v0, T v1) {
#pragma unroll
  for (int sz = 0; sz < (D == 3 ? 3 : 1); ++sz) {
    int gz = k, cz = BC_NONE;
    if (D == 3 && !ghost_choice(sz, k, P.n[2], P.bc[4], P.bc[5], gz, cz)) continue;
#pragma unroll
    for (int sy = 0; sy < 3; ++sy) {
      int gy, cy;
      if (!ghost_choice(sy, j, P.n[1], P.bc[2], P.bc[3], gy, cy)) continue;
#pragma unroll
      for (int sx = 0; sx < 3; ++sx) {
        if (sx == 0 && sy == 0 && sz == 0) continue;
        int gx, cx;
        if (!ghost_choice(sx, i, P.n[0], P.bc[0], P.bc[1], gx, cx)) continue;
        // Face maps applied in ascending dimension (SetBC's face order).
        T a = v0, b = v1;
        if (sx) {
          a = bc_map<T>(cx, a);
          b = bc_map<T>(cx, b);
        }
        if (sy) {
          a = bc_map<T>(cy, a);
          b = bc_map<T>(cy, b);
        }
        if (sz) {
          a = bc_map<T>(cz, a);
          b = bc_map<T>(cz, b);
        }
        const int64_t c = cidx(P, gx, gy, D == 3 ? gz : 0);
        q0[c] = a;
        q1[c] = b;
      }
    }
  }
}

// The same, a cell that feeds one ghost through one face first: most of those that
// feed any; cells at edges and corners go through all combinations.  (All through
// the combinations: a colour pass of 128^3 23 us, now 20.9, of 48 x 32 x 40 FP32
// 5.5, now 4.7.  As a loop over the ghosts a cell feeds, one by one: restriction of
// 16^3 13.5 us against 9.7 and 8.2.  The 2D fused stages, which write few ghosts
// and have no registers to spare, are 5 % slower this way: write_through_all.)
template <class T, int D>
__device__ __forceinline__ void write_through(const DevPatch& P, T* q0, T* q1, int i, int j,
                                              int k, T v0, T v1) {
  int cx, cy, cz = BC_NONE;
  const int dx = ghost_step(i, P.n[0], P.bc[0], P.bc[1], cx);
  const int dy = ghost_step(j, P.n[1], P.bc[2], P.bc[3], cy);
  const int dz = D == 3 ? ghost_step(k, P.n[2], P.bc[4], P.bc[5], cz) : 0;
  const int faces = (dx != 0) + (dy != 0) + (dz != 0);
  if (faces == 0) return;
  if (faces > 1 || dx > P.n[0] || dy > P.n[1] || (D == 3 && dz > P.n[2])) {
    write_through_all<T, D>(P, q0, q1, i, j, k, v0, v1);
    return;
  }
  const int code = dx ? cx : dy ? cy : cz;
  const int64_t c = cidx(P, i + dx, j + dy, D == 3 ? k + dz : 0);
  q0[c] = bc_map<T>(code, v0);
  q1[c] = bc_map<T>(code, v1);
}

template <class T, int D>
__device__ __forceinline__ void load_stencil(const DevPatch& P, const T* __restrict__ q0,
                                             const T* __restrict__ q1, int64_t c,
                                             Problem::Stencil<T, D>& s) {
  const int64_t st[3] = {1, P.sy, P.sz};
  s.pc = q0[c];
  s.mc = q1[c];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    s.pm[d] = q0[c - st[d]];
    s.pp[d] = q0[c + st[d]];
    s.mm[d] = q1[c - st[d]];
    s.mp[d] = q1[c + st[d]];
  }
}

__device__ __forceinline__ bool near_boundary(const DevPatch& P, int i, int j, int k, int D) {
  bool b = (i == 1) | (i == P.n[0]) | (j == 1) | (j == P.n[1]);
  if (D == 3) b = b | (k == 1) | (k == P.n[2]);
  return b;
}

// ---- per-cell bodies ---------------------------------------------------------

// One cell of RelaxGrid (problem.f90:192-213 / 485-516), in place on q, with
// SetGhost(level, ipass) for physical faces.
template <class T, int D>
__device__ __forceinline__ void relax_cell(const DevPatch& P, int i, int j, int k) {
  T* q0 = fld<T>(P.q[0]);
  T* q1 = fld<T>(P.q[1]);
  const T* f0 = fld<T>(P.f[0]);
  const T* f1 = fld<T>(P.f[1]);
  const int64_t c = cidx(P, i, j, k);
  Problem::Stencil<T, D> s;
  load_stencil<T, D>(P, q0, q1, c, s);
  T phi, mu;
  if (P.delta)
    Problem::RelaxCell<T, D, true>(s, f0[c], f1[c], T(P.tmp1), T(P.tmp2), T(P.tmp3), T(P.alpha),
                                   phi, mu, fld<T>(P.bs)[c]);
  else
    Problem::RelaxCell<T, D>(s, f0[c], f1[c], T(P.tmp1), T(P.tmp2), T(P.tmp3), T(P.alpha), phi,
                             mu);
  q0[c] = phi;
  q1[c] = mu;
  if (P.wt && near_boundary(P, i, j, k, D)) write_through<T, D>(P, q0, q1, i, j, k, phi, mu);
}

// Operator at one cell from its stencil, in the patch's form.
template <class T, int D>
__device__ __forceinline__ void operator_at(const DevPatch& P, const Problem::Stencil<T, D>& s,
                                            int64_t c, T& o0, T& o1) {
  if (P.delta)
    Problem::OperatorCell<T, D, true>(s, T(P.tmp1), T(P.tmp2), T(P.alpha), o0, o1,
                                      fld<T>(P.bs)[c]);
  else
    Problem::OperatorCell<T, D>(s, T(P.tmp1), T(P.tmp2), T(P.alpha), o0, o1);
}

// The same with the base state's value given (correction form only).
template <class T, int D>
__device__ __forceinline__ void operator_with(const DevPatch& P, const Problem::Stencil<T, D>& s,
                                              T base, T& o0, T& o1) {
  if (P.delta)
    Problem::OperatorCell<T, D, true>(s, T(P.tmp1), T(P.tmp2), T(P.alpha), o0, o1, base);
  else
    Problem::OperatorCell<T, D>(s, T(P.tmp1), T(P.tmp2), T(P.alpha), o0, o1);
}

// RestrictSolution (afas:600-644) of the coarse cell (ic,jc,kc) of child C
// into parent P, + the parent's SetGhost(level-1, 0) for physical faces +
// GetCoarseGhostPoints (boundary.f90:1203-1269): the parent solution and its
// snapshot qs (the children's qc) are both written.
// TC / TP: value types of the child and the parent (equal in the FP64 path;
// in the mixed path the child may be FP32 over an FP64 parent).  Restriction
// runs in the child's precision; the stored value converts exactly upward.
template <class TC, class TP, int D>
__device__ __forceinline__ void restrict_cell(const DevPatch& C, const DevPatch& P, int ic, int jc,
                                              int kc) {
  // The block's cells, row by row from the high end, high cell first: the
  // order of the sum.
  const int64_t c0 = cidx(C, 2 * ic - 1, 2 * jc - 1, D == 3 ? 2 * kc - 1 : 0);
  auto average = [&](const TC* a) {
    TC s = TC(0);
#pragma unroll
    for (int r = (D == 3 ? 3 : 1); r >= 0; --r) {
      const auto v = load_pair<TC>(a + c0 + (r & 1) * C.sy + (r >> 1) * C.sz);
      s = r == (D == 3 ? 3 : 1) ? v.y : s + v.y;
      s = s + v.x;
    }
    return TP((D == 3 ? TC(0.125) : TC(0.25)) * s);
  };
  const TP val[2] = {average(fld<TC>(mid_state(C)[0])), average(fld<TC>(mid_state(C)[1]))};
  const int pi = C.off[0] + ic, pj = C.off[1] + jc, pk = (D == 3) ? C.off[2] + kc : 0;
  const int64_t pc = cidx(P, pi, pj, pk);
  TP* pq0 = fld<TP>(P.q[0]);
  TP* pq1 = fld<TP>(P.q[1]);
  TP* ps0 = fld<TP>(P.qs[0]);
  TP* ps1 = fld<TP>(P.qs[1]);
  pq0[pc] = val[0];
  pq1[pc] = val[1];
  ps0[pc] = val[0];
  ps1[pc] = val[1];
  if (P.wt && near_boundary(P, pi, pj, pk, D)) {
    write_through<TP, D>(P, pq0, pq1, pi, pj, pk, val[0], val[1]);
    write_through<TP, D>(P, ps0, ps1, pi, pj, pk, val[0], val[1]);
  }
  if (P.delta) {
    // Correction form: the coarse base is the restriction of the fine base.
    fld<TP>(P.bs)[pc] = average(fld<TC>(C.bs));
  }
}

// The 2^D block of fine cells whose low corner is element c, with its face
// neighbours: a[z][y][x], the block at indices 1 and 2 (2D: z = 0).  The rows
// through the block come as aligned pairs, and each value is loaded once.
template <class T, int D>
__device__ __forceinline__ void load_block(const DevPatch& C, const T* __restrict__ q, int64_t c,
                                           T (&a)[D == 3 ? 4 : 1][4][4]) {
#pragma unroll
  for (int z = 0; z < (D == 3 ? 4 : 1); ++z)
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const bool zin = D == 2 || z == 1 || z == 2, yin = y == 1 || y == 2;
      if (!zin && !yin) continue;
      const T* p = q + c + (y - 1) * C.sy + (D == 3 ? (z - 1) * C.sz : 0);
      const auto v = load_pair<T>(p);
      a[z][y][1] = v.x;
      a[z][y][2] = v.y;
      if (zin && yin) {
        a[z][y][0] = p[-1];
        a[z][y][3] = p[2];
      }
    }
}

// CoarseLoadingFunction (afas:646-714) at one coarse cell:
//   parent%f(mb) = Restriction(f - Operator(q)) + Operator(qc, h = parent%dx)
// A thread holds its block of children with the neighbours in registers
// (load_block).  Loaded cell by cell, with every second element of a row per
// warp and 13 (2D) or 17 loads a child, the pass ran at 78 % of L1's rate and a
// third of the memory's.  From a 128^3 FP64 level 41 -> 35 us, all levels of 24
// problems of 32^3 and 64^3 (FP32) 130 -> 77, of 512 of 64^2 to 256^2 190 -> 175,
// of 96 in FP64 100 -> 66; now the latency of the loads bounds it.
template <class TC, class TP, int D>
__device__ __forceinline__ void coarse_load_cell(const DevPatch& C, const DevPatch& P, int ic,
                                                 int jc, int kc) {
  const int64_t c0 = cidx(C, 2 * ic - 1, 2 * jc - 1, D == 3 ? 2 * kc - 1 : 0);
  TC a[2][D == 3 ? 4 : 1][4][4];
  load_block<TC, D>(C, fld<TC>(mid_state(C)[0]), c0, a[0]);
  load_block<TC, D>(C, fld<TC>(mid_state(C)[1]), c0, a[1]);
  // Restriction of rf: children in the reference's summation order, from the
  // high end of each dimension.
  TC s0 = TC(0), s1 = TC(0);
#pragma unroll
  for (int r = (D == 3 ? 3 : 1); r >= 0; --r) {
    const int y = 1 + (r & 1), z = D == 3 ? 1 + (r >> 1) : 0;
    const int64_t c = c0 + (r & 1) * C.sy + (r >> 1) * C.sz;
    const auto f0 = load_pair<TC>(fld<TC>(C.f[0]) + c), f1 = load_pair<TC>(fld<TC>(C.f[1]) + c);
    typename PairOf<TC>::V base{};
    if (C.delta) base = load_pair<TC>(fld<TC>(C.bs) + c);
#pragma unroll
    for (int x = 2; x >= 1; --x) {
      Problem::Stencil<TC, D> s;
      s.pc = a[0][z][y][x];
      s.mc = a[1][z][y][x];
      s.pm[0] = a[0][z][y][x - 1];
      s.pp[0] = a[0][z][y][x + 1];
      s.mm[0] = a[1][z][y][x - 1];
      s.mp[0] = a[1][z][y][x + 1];
      s.pm[1] = a[0][z][y - 1][x];
      s.pp[1] = a[0][z][y + 1][x];
      s.mm[1] = a[1][z][y - 1][x];
      s.mp[1] = a[1][z][y + 1][x];
      if (D == 3) {
        s.pm[D - 1] = a[0][D == 3 ? z - 1 : 0][y][x];
        s.pp[D - 1] = a[0][D == 3 ? z + 1 : 0][y][x];
        s.mm[D - 1] = a[1][D == 3 ? z - 1 : 0][y][x];
        s.mp[D - 1] = a[1][D == 3 ? z + 1 : 0][y][x];
      }
      TC o0, o1;
      operator_with<TC, D>(C, s, x == 2 ? base.y : base.x, o0, o1);
      const TC r0 = (x == 2 ? f0.y : f0.x) - o0, r1 = (x == 2 ? f1.y : f1.x) - o1;
      const bool first = x == 2 && r == (D == 3 ? 3 : 1);
      s0 = first ? r0 : s0 + r0;
      s1 = first ? r1 : s1 + r1;
    }
  }
  const TC w = (D == 2) ? TC(0.25) : TC(0.125);
  const TP R0 = TP(w * s0), R1 = TP(w * s1);
  const int pi = C.off[0] + ic, pj = C.off[1] + jc, pk = (D == 3) ? C.off[2] + kc : 0;
  const int64_t pc = cidx(P, pi, pj, pk);
  Problem::Stencil<TP, D> s;
  load_stencil<TP, D>(P, fld<TP>(P.qs[0]), fld<TP>(P.qs[1]), pc, s);
  TP o0, o1;
  operator_at<TP, D>(P, s, pc, o0, o1);
  fld<TP>(P.f[0])[pc] = R0 + o0;
  fld<TP>(P.f[1])[pc] = R1 + o1;
}

template <class T>
__device__ __forceinline__ T lin_x(bool even, T a, T b) {
  return even ? T(3) * a + b : a + T(3) * b;
}

// CorrectFine with BiLin/TriLinProlongationP1 (afas:842-963,
// gridutilities.f90:137-175, 474-529) at the fine cell (I,J,K):
// q += P(parent%q - qc); the ghost ring is refreshed by write-through (the
// reference's SetGhost(level, 0) overwrites the prolongated ring, afas:515).
// The correction e = parent%q - qc is formed and prolongated in the parent's
// precision and added in the child's.
template <class TC, class TP, int D>
__device__ __forceinline__ void correct_cell(const DevPatch& C, const DevPatch& P, int I, int J,
                                             int K) {
  const TP* pq0 = fld<TP>(P.q[0]);
  const TP* pq1 = fld<TP>(P.q[1]);
  const TP* ps0 = fld<TP>(P.qs[0]);
  const TP* ps1 = fld<TP>(P.qs[1]);
  TC* q0 = fld<TC>(mid_state(C)[0]);
  TC* q1 = fld<TC>(mid_state(C)[1]);
  const int m = I >> 1, n = J >> 1, p = K >> 1;
  const bool ex = (I & 1) == 0, ey = (J & 1) == 0, ez = (K & 1) == 0;
  TP corr[2];
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    const TP* pq = v ? pq1 : pq0;
    const TP* ps = v ? ps1 : ps0;
    auto e = [&](int a, int b, int c) -> TP {
      const int64_t x = cidx(P, C.off[0] + a, C.off[1] + b, D == 3 ? C.off[2] + c : 0);
      return pq[x] - ps[x];
    };
    if (D == 2) {
      const TP b0 = lin_x<TP>(ex, e(m, n, 0), e(m + 1, n, 0));
      const TP b1 = lin_x<TP>(ex, e(m, n + 1, 0), e(m + 1, n + 1, 0));
      corr[v] = lin_x<TP>(ey, b0, b1) / TP(16);
    } else {
      const TP b00 = lin_x<TP>(ex, e(m, n, p), e(m + 1, n, p));
      const TP b10 = lin_x<TP>(ex, e(m, n + 1, p), e(m + 1, n + 1, p));
      const TP b01 = lin_x<TP>(ex, e(m, n, p + 1), e(m + 1, n, p + 1));
      const TP b11 = lin_x<TP>(ex, e(m, n + 1, p + 1), e(m + 1, n + 1, p + 1));
      const TP c0 = lin_x<TP>(ey, b00, b10);
      const TP c1 = lin_x<TP>(ey, b01, b11);
      corr[v] = lin_x<TP>(ez, c0, c1) / TP(64);
    }
  }
  const int64_t c = cidx(C, I, J, K);
  const TC a0 = q0[c] + TC(corr[0]);
  const TC a1 = q1[c] + TC(corr[1]);
  q0[c] = a0;
  q1[c] = a1;
  if (C.wt && near_boundary(C, I, J, K, D)) write_through<TC, D>(C, q0, q1, I, J, K, a0, a1);
}

// CorrectFine by 2^D blocks of fine cells: the fine cells 2m, 2m+1 of each
// dimension read the same 2^D parent corrections, formed once here; each cell
// then takes correct_cell's expression on them, so the values are
// correct_cell's bit for bit.  Block (m, n, p) from 0 to cn of each dimension
// covers the fine cells 1 to n exactly once.  Cell by cell a fine cell took 16
// (2D) or 32 parent loads: 128^3 FP64 46 us, now 28; three levels of 24 problems
// of 32^3 and 64^3 130 and 101 us.
template <class TC, class TP, int D>
__device__ __forceinline__ void correct_block(const DevPatch& C, const DevPatch& P, int m, int n,
                                              int p) {
  TC* q0 = fld<TC>(mid_state(C)[0]);
  TC* q1 = fld<TC>(mid_state(C)[1]);
  constexpr int NZ = D == 3 ? 2 : 1;
  TP e[2][NZ][2][2];  // [component][p + c][n + b][m + a]
  const int64_t x0 = cidx(P, C.off[0] + m, C.off[1] + n, D == 3 ? C.off[2] + p : 0);
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    const TP* pq = fld<TP>(P.q[v]) + x0;
    const TP* ps = fld<TP>(P.qs[v]) + x0;
#pragma unroll
    for (int c = 0; c < NZ; ++c)
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int a = 0; a < 2; ++a) {
          const int64_t x = a + b * P.sy + c * P.sz;
          e[v][c][b][a] = pq[x] - ps[x];
        }
  }
#pragma unroll 1
  for (int r = 0; r < 2 * NZ; ++r) {
    const int dy = r & 1, dz = r >> 1;
    const int J = 2 * n + dy, K = D == 3 ? 2 * p + dz : 0;
    if (J < 1 || J > C.n[1] || (D == 3 && (K < 1 || K > C.n[2]))) continue;
    // lin_x with the choice at run time; its two terms commute.
    auto lin = [](bool even, TP a, TP b) { return TP(3) * (even ? a : b) + (even ? b : a); };
#pragma unroll
    for (int dx = 0; dx < 2; ++dx) {
      const int I = 2 * m + dx;
      if (I < 1 || I > C.n[0]) continue;
      TP corr[2];
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        TP cz[NZ];
#pragma unroll
        for (int c = 0; c < NZ; ++c)
          cz[c] = lin(dy == 0, lin_x<TP>(dx == 0, e[v][c][0][0], e[v][c][0][1]),
                      lin_x<TP>(dx == 0, e[v][c][1][0], e[v][c][1][1]));
        corr[v] = D == 3 ? lin(dz == 0, cz[0], cz[NZ - 1]) / TP(64) : cz[0] / TP(16);
      }
      const int64_t c = cidx(C, I, J, K);
      const TC a0 = q0[c] + TC(corr[0]);
      const TC a1 = q1[c] + TC(corr[1]);
      q0[c] = a0;
      q1[c] = a1;
      if (C.wt && near_boundary(C, I, J, K, D)) write_through<TC, D>(C, q0, q1, I, J, K, a0, a1);
    }
  }
}

// Tiles of BLOCK_THREADS consecutive blocks of a patch, x fastest.
inline void block_tiles(int patch, const int* cn, int nd, std::vector<Item>& out) {
  int64_t blocks = nd == 3 ? cn[2] + 1 : 1;
  blocks *= (int64_t)(cn[0] + 1) * (cn[1] + 1);
  for (int64_t b = 0; b < blocks; b += BLOCK_THREADS)
    out.push_back(Item{patch, (int)(b / BLOCK_THREADS), 0, 0});
}

// ---- reductions --------------------------------------------------------------

// Deterministic block sum of a double (fixed shuffle tree + fixed smem
// order).  Any block shape whose size is a multiple of 32 and at most 1024.
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double red[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nthreads = blockDim.x * blockDim.y * blockDim.z;
  const int lane = tid & 31, warp = tid >> 5;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (tid == 0) {
    for (int w = 0; w < nthreads / 32; ++w) s += red[w];
  }
  __syncthreads();
  return s;  // valid in thread 0
}

// Second stage of a two-stage reduction over `count` partial sums that the CTAs
// have stored (here: this CTA's by any of its threads): the last CTA to finish
// sums them in index order.  Returns true in thread 0 of that CTA with the total
// in `total`.
__device__ __forceinline__ bool last_block_sum(const double* partials, uint32_t* ticket,
                                               int nblocks, int count, double& total) {
  __shared__ bool is_last;
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nthreads = blockDim.x * blockDim.y * blockDim.z;
  __threadfence();
  __syncthreads();
  if (tid == 0) is_last = atomicAdd(ticket, 1u) == (uint32_t)nblocks - 1u;
  __syncthreads();
  if (!is_last) return false;
  __threadfence();
  double s = 0.0;
  for (int b = tid; b < count; b += nthreads) s += ((const volatile double*)partials)[b];
  const double tot = block_sum(s);
  if (tid == 0) {
    total = tot;
    *ticket = 0u;
    return true;
  }
  return false;
}

// The same with one partial sum per CTA, `mine` of thread 0.
__device__ __forceinline__ bool last_block_total(double mine, double* partials,
                                                 uint32_t* ticket, int nblocks,
                                                 double& total) {
  if (threadIdx.x + threadIdx.y + threadIdx.z == 0) partials[blockIdx.x] = mine;
  return last_block_sum(partials, ticket, nblocks, nblocks, total);
}

// ---- tile bodies ---------------------------------------------------------------
//
// One function per kernel that processes one Item (tile) of its work list.
// The grid kernels below run one tile per CTA; the batch kernels (batch.cuh)
// run the same bodies in a grid-stride loop over a device-resident list.
// Inactive patches (finished or idle batch slots) are skipped whole, which is
// uniform per CTA.

// RelaxGrid (one colour pass) + SetGhost(level, ipass) for physical faces.
// color 0 = ipass 1 = cells with even i+j(+k); color 1 = ipass 2.
template <class T, int D>
__device__ __forceinline__ void relax_item(const DevPatch* __restrict__ PT, const Item it,
                                           int color) {
  const DevPatch P = PT[it.patch];  // by value: fields stay in registers
  if (!P.active) return;
  const WorkPlace<D> w(it, P.n[0]);
  if (w.j > P.n[1]) return;
  const int i = w.i0 + ((w.i0 + w.j + w.k + color) & 1);
  if (i > P.n[0]) return;
  relax_cell<T, D>(P, i, w.j, w.k);
}

// The residual of the FP64 cells of one TILE_X x TILE_Y tile by one warp, a pair
// of cells a lane: out(i, j, k, two, r0, r1, q) for every pair inside (two: the
// second cell is inside too; q: phi of both).  Returns the tile's sum of rf^2
// (ErrorAFAS's SquareSum) in lane 0, in the order of block_sum with a thread per
// pair: each row by the shuffle tree, then the rows in order.
//
// A row of q comes as aligned pairs, once for the three rows that read it; the
// four rows' loads are independent of one another.  A CTA per tile, a thread per
// pair and each operand loaded where it is used, kept L1 at 76 % and memory at 28 %
// of their rates: the norm of 128^3 45 us, now 30.5; the defect (mixed.cuh) of
// 96 x 64 x 80 24 us, now 17, and of 24 masters of 32^3 and 64^3 154 us, now 110.
// (In 2D the norm of 96 masters takes 38 us either way.)
template <int D, class Out>
__device__ __forceinline__ double resid_rows(const DevPatch& P, const Item it, Out&& out) {
  const int lane = threadIdx.x & 31;
  const int i0 = it.tx * TILE_X + 2 * lane + 1, j0 = it.ty * TILE_Y + 1;
  const int k = D == 3 ? it.tz + 1 : 0;
  const bool on = i0 <= P.n[0], two = i0 < P.n[0];
  const int rows = min(TILE_Y, P.n[1] - j0 + 1);
  double acc[TILE_Y];
#pragma unroll
  for (int r = 0; r < TILE_Y; ++r) acc[r] = 0.0;
  if (on) {
    const int64_t c0 = cidx(P, i0, j0, k);
    const double* q0 = fld<double>(P.q[0]) + c0;
    const double* q1 = fld<double>(P.q[1]) + c0;
    const double* f0 = fld<double>(P.f[0]) + c0;
    const double* f1 = fld<double>(P.f[1]) + c0;
    double2 a[2][TILE_Y + 2];  // rows j0 - 1 ... j0 + TILE_Y of the pair
#pragma unroll
    for (int r = 0; r < TILE_Y + 2; ++r)
      if (r <= rows + 1) {
        a[0][r] = load_pair<double>(q0 + (r - 1) * P.sy);
        a[1][r] = load_pair<double>(q1 + (r - 1) * P.sy);
      }
#pragma unroll
    for (int r = 0; r < TILE_Y; ++r) {
      if (r >= rows) break;
      const int64_t o = r * P.sy;
      const double2 g0 = load_pair<double>(f0 + o), g1 = load_pair<double>(f1 + o);
      Problem::Stencil<double, D> lo, hi;
      lo.pc = a[0][r + 1].x;
      lo.mc = a[1][r + 1].x;
      hi.pc = a[0][r + 1].y;
      hi.mc = a[1][r + 1].y;
      lo.pm[0] = q0[o - 1];
      lo.mm[0] = q1[o - 1];
      lo.pp[0] = hi.pc;
      lo.mp[0] = hi.mc;
      hi.pm[0] = lo.pc;
      hi.mm[0] = lo.mc;
      hi.pp[0] = two ? q0[o + 2] : 0.0;
      hi.mp[0] = two ? q1[o + 2] : 0.0;
      lo.pm[1] = a[0][r].x;
      lo.mm[1] = a[1][r].x;
      lo.pp[1] = a[0][r + 2].x;
      lo.mp[1] = a[1][r + 2].x;
      hi.pm[1] = a[0][r].y;
      hi.mm[1] = a[1][r].y;
      hi.pp[1] = a[0][r + 2].y;
      hi.mp[1] = a[1][r + 2].y;
      if (D == 3) {
        const double2 zm0 = load_pair<double>(q0 + o - P.sz), zp0 = load_pair<double>(q0 + o + P.sz);
        const double2 zm1 = load_pair<double>(q1 + o - P.sz), zp1 = load_pair<double>(q1 + o + P.sz);
        lo.pm[D - 1] = zm0.x;
        lo.pp[D - 1] = zp0.x;
        lo.mm[D - 1] = zm1.x;
        lo.mp[D - 1] = zp1.x;
        hi.pm[D - 1] = zm0.y;
        hi.pp[D - 1] = zp0.y;
        hi.mm[D - 1] = zm1.y;
        hi.mp[D - 1] = zp1.y;
      }
      double o0, o1;
      double2 r0, r1;
      Problem::OperatorCell<double, D>(lo, P.tmp1, P.tmp2, P.alpha, o0, o1);
      r0.x = g0.x - o0;
      r1.x = g1.x - o1;
      Problem::OperatorCell<double, D>(hi, P.tmp1, P.tmp2, P.alpha, o0, o1);
      r0.y = g0.y - o0;
      r1.y = g1.y - o1;
      acc[r] = r0.x * r0.x + r1.x * r1.x;
      if (two) acc[r] += r0.y * r0.y + r1.y * r1.y;
      out(i0, j0 + r, k, two, r0, r1, a[0][r + 1]);
    }
  }
  double s = 0.0;
#pragma unroll
  for (int r = 0; r < TILE_Y; ++r) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[r] += __shfl_down_sync(0xffffffffu, acc[r], o);
    s += acc[r];
  }
  return s;
}

template <class TC, class TP, int D>
__device__ __forceinline__ void restrict_item(const DevPatch* __restrict__ PT, const Item it) {
  const DevPatch C = PT[it.patch];
  if (!C.active) return;
  const DevPatch P = PT[C.parent];
  const WorkPlace<D> w(it, C.cn[0]);
  if (w.j > C.cn[1]) return;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int ic = w.a0 + t * w.W;
    if (ic > C.cn[0]) break;
    restrict_cell<TC, TP, D>(C, P, ic, w.j, w.k);
  }
}

template <class TC, class TP, int D>
__device__ __forceinline__ void coarse_load_item(const DevPatch* __restrict__ PT, const Item it) {
  const DevPatch C = PT[it.patch];
  if (!C.active) return;
  const DevPatch P = PT[C.parent];
  const WorkPlace<D> w(it, C.cn[0]);
  if (w.j > C.cn[1]) return;
#pragma unroll 1
  for (int t = 0; t < 2; ++t) {
    const int ic = w.a0 + t * w.W;
    if (ic > C.cn[0]) break;
    coarse_load_cell<TC, TP, D>(C, P, ic, w.j, w.k);
  }
}

template <class TC, class TP, int D>
__device__ __forceinline__ void correct_item(const DevPatch* __restrict__ PT, const Item it) {
  const DevPatch C = PT[it.patch];
  if (!C.active) return;
  const DevPatch P = PT[C.parent];
  int u = it.tx * BLOCK_THREADS + threadIdx.x + 32 * threadIdx.y;
  const int m = u % (C.cn[0] + 1);
  u /= C.cn[0] + 1;
  const int n = D == 3 ? u % (C.cn[1] + 1) : u, p = D == 3 ? u / (C.cn[1] + 1) : 0;
  if (D == 3 ? p > C.cn[2] : n > C.cn[1]) return;
  correct_block<TC, TP, D>(C, P, m, n, p);
}

// GetSourceFunction + UpdateSourceFunction on one level (afas:312-367,
// 427-486): f = Source(qold) + 0.  newstep_only (batches): only masters
// whose new time step starts now; they keep no qold, so qold = q (the
// reference's CopyQToQold just before, lib/bsamroutines.f90:659-661).
template <class T, int D>
__device__ __forceinline__ void source_item(const DevPatch* __restrict__ PT, const Item it,
                                            int newstep_only) {
  const DevPatch P = PT[it.patch];
  if (!P.active || (newstep_only && !P.newstep)) return;
  const int j = it.ty * TILE_Y + threadIdx.y + 1;
  const int k = (D == 3) ? it.tz + 1 : 0;
  if (j > P.n[1]) return;
  const int i0 = (it.tx * 32 + threadIdx.x) * 2 + 1;
  const T* qo = fld<T>(P.qo[0] ? P.qo[0] : P.q[0]);
  T* f0 = fld<T>(P.f[0]);
  T* f1 = fld<T>(P.f[1]);
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int i = i0 + t;
    if (i > P.n[0]) break;
    const int64_t c = cidx(P, i, j, k);
    T a, b;
    Problem::SourceCell<T>(qo[c], T(P.alpha), a, b);
    f0[c] = a;
    f1[c] = b;
  }
}

// ---- grid kernels (one tile per CTA) --------------------------------------------

template <class T, int D>
__global__ void __launch_bounds__(BLOCK_THREADS)
    k_relax(const DevPatch* __restrict__ PT, const Item* __restrict__ items, int color) {
  after_previous();
  relax_item<T, D>(PT, items[blockIdx.x], color);
}

// ErrorAFAS / L2Error / SquareSum (afas:108-221), errortype 1:
// residual = sqrt(sum rf^2 / (nrvars * ncells)) over the finest level.
template <int D>
__global__ void __launch_bounds__(BLOCK_THREADS, D == 2 ? 5 : 4)
    k_resid_norm(const DevPatch* __restrict__ PT, const Item* __restrict__ items,
                 double* __restrict__ partials, DevStatus* __restrict__ st, int nitems,
                 double denom, double tol) {
  after_previous();
  const int b = blockIdx.x * TILE_Y + threadIdx.y;  // a tile per warp
  if (b < nitems) {
    const Item it = items[b];
    const double s = resid_rows<D>(PT[it.patch], it,
                                   [](int, int, int, bool, double2, double2, double2) {});
    if (threadIdx.x == 0) partials[b] = s;
  }
  double total;
  if (last_block_sum(partials, &st->ticket, gridDim.x, nitems, total)) {
    const double r = sqrt(total / denom);
    st->sumsq = total;
    st->residual = r;
    st->converged = (r < tol) ? 1 : 0;
  }
}

template <class TC, class TP, int D>
__global__ void __launch_bounds__(BLOCK_THREADS)
    k_restrict(const DevPatch* __restrict__ PT, const Item* __restrict__ items) {
  after_previous();
  restrict_item<TC, TP, D>(PT, items[blockIdx.x]);
}

template <class TC, class TP, int D>
__global__ void __launch_bounds__(BLOCK_THREADS)
    k_coarse_load(const DevPatch* __restrict__ PT, const Item* __restrict__ items) {
  after_previous();
  coarse_load_item<TC, TP, D>(PT, items[blockIdx.x]);
}

template <class TC, class TP, int D>
__global__ void __launch_bounds__(BLOCK_THREADS)
    k_correct(const DevPatch* __restrict__ PT, const Item* __restrict__ items) {
  after_previous();
  correct_item<TC, TP, D>(PT, items[blockIdx.x]);
}

template <class T, int D>
__global__ void __launch_bounds__(BLOCK_THREADS)
    k_source(const DevPatch* __restrict__ PT, const Item* __restrict__ items) {
  source_item<T, D>(PT, items[blockIdx.x], 0);
}

// The 2D ring cell g of a patch with m1 x m2 interior cells (bottom row, top
// row, left column, right column).
__device__ __forceinline__ void ring2(int g, int m1, int m2, int& gi, int& gj) {
  if (g < m1 + 2) {
    gi = g;
    gj = 0;
  } else if (g < 2 * (m1 + 2)) {
    gi = g - (m1 + 2);
    gj = m2 + 1;
  } else if (g < 2 * (m1 + 2) + m2) {
    gi = 0;
    gj = g - 2 * (m1 + 2) + 1;
  } else {
    gi = m1 + 1;
    gj = g - 2 * (m1 + 2) - m2 + 1;
  }
}

// The 3D ring cell g of a patch with m1 x m2 x m3 interior cells, in
// order: the two k planes, then the 2D ring of each interior plane.
__device__ __forceinline__ void ring3(int g, int m1, int m2, int m3, int& gi, int& gj, int& gk) {
  const int plane = (m1 + 2) * (m2 + 2), rg2 = 2 * (m1 + 2) + 2 * m2;
  if (g < 2 * plane) {
    gk = g < plane ? 0 : m3 + 1;
    const int r = g % plane;
    gi = r % (m1 + 2);
    gj = r / (m1 + 2);
  } else {
    const int r0 = g - 2 * plane;
    gk = 1 + r0 / rg2;
    ring2(r0 % rg2, m1, m2, gi, gj);
  }
}

// SetBC (boundary.f90:598-891), preceded by PeriodicBC on periodic faces
// (boundary.f90:76-83, 417-483), at one ring cell of a patch, any face codes: a
// ghost is written when at least one of the dimensions it lies outside of has a
// physical or periodic face; its value is the face maps of those dimensions
// (ascending; a periodic face maps a value to itself) applied to the cell
// reflected across them (across a periodic face, the cell at the other end).
template <class T, int D>
__device__ __forceinline__ void setbc_elem(const DevPatch& P, int g0, int g1, int g2) {
  const int co[3] = {g0, g1, g2};
  int src[3] = {g0, g1, g2};
  int codes[3] = {BC_NONE, BC_NONE, BC_NONE};
  bool write = false;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    if (co[d] == 0 && P.bc[2 * d] != BC_NONE) {
      src[d] = P.bc[2 * d] == BC_PERIODIC ? P.n[d] : 1;
      codes[d] = P.bc[2 * d];
      write = true;
    } else if (co[d] == P.n[d] + 1 && P.bc[2 * d + 1] != BC_NONE) {
      src[d] = P.bc[2 * d + 1] == BC_PERIODIC ? 1 : P.n[d];
      codes[d] = P.bc[2 * d + 1];
      write = true;
    }
  }
  if (!write) return;
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    T* q = fld<T>(P.q[v]);
    T val = q[cidx(P, src[0], src[1], src[2])];
#pragma unroll
    for (int d = 0; d < D; ++d)
      if (codes[d] != BC_NONE) val = bc_map<T>(codes[d], val);
    q[cidx(P, co[0], co[1], co[2])] = val;
  }
}

// SetBC of a list of patches, a thread per ring cell (blockIdx.y selects the
// patch; the grid strides over its ring).  Over every cell of the box instead it
// took 20 us at 128^3 and 558 us for 512 problems of a batch.
constexpr int SETBC_THREADS = 128;
template <class T, int D>
__global__ void __launch_bounds__(SETBC_THREADS)
    k_setbc_list(const DevPatch* __restrict__ PT, const int* __restrict__ patches) {
  const DevPatch& P = PT[patches[blockIdx.y]];
  const int m1 = P.n[0], m2 = P.n[1], m3 = P.n[2];
  const int ring2d = 2 * (m1 + 2) + 2 * m2;
  const int64_t ring = D == 2 ? ring2d : 2 * (int64_t)(m1 + 2) * (m2 + 2) + (int64_t)m3 * ring2d;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < ring;
       g += (int64_t)gridDim.x * blockDim.x) {
    int gi, gj, gk = 0;
    if (D == 2) ring2((int)g, m1, m2, gi, gj);
    else ring3((int)g, m1, m2, m3, gi, gj, gk);
    setbc_elem<T, D>(P, gi, gj, gk);
  }
}

// CTAs per patch of k_setbc_list for patches of at most `cells` cells.
inline unsigned setbc_blocks(int nd, int64_t cells) {
  // A square (cube) of that many cells; longer rings stride.
  double side = 1.0;
  while ((nd == 2 ? side * side : side * side * side) < (double)cells) side *= 1.25;
  const double ring = nd == 2 ? 4.0 * (side + 2.0) : 6.0 * (side + 2.0) * (side + 2.0);
  return (unsigned)std::max(1.0, std::min(1024.0, ring / SETBC_THREADS + 1.0));
}

// ---- device-side V-cycle loop (MultigridIterations, afas:69-104) -----------

// Start of a MultigridIterations call: no V-cycle done yet.
static __global__ void k_mg_begin(DevStatus* __restrict__ st) {
  st->iters = 0;
  st->converged = 0;
}

// End of one V-cycle: record the residual and decide whether the conditional
// WHILE node of the step graph runs another V-cycle.  Stops at convergence
// (residual < qerrortol), after maxvcycles, on a non-finite residual (the
// host reports it) or when a kernel recorded an error.
static __global__ void k_mg_loop(DevStatus* __restrict__ st, double* __restrict__ trace, int maxv,
                          double tol, cudaGraphConditionalHandle handle) {
  after_previous();
  const int it = st->iters + 1;
  st->iters = it;
  const double r = st->residual;
  if (it <= maxv) trace[it - 1] = r;
  const bool conv = r < tol;
  st->converged = conv ? 1 : 0;
  const bool again = !conv && it < maxv && isfinite(r) && st->kerr == 0;
  cudaGraphSetConditional(handle, again ? 1u : 0u);
}

// One of the two sums of Energy2D (problem.f90:330-361) over a 2D patch
// interior: which = 0, sum of Ff(c); which = 1, sum of f1(i) + f1(i-1) +
// f2(j) + f2(j-1) with f1 = (c(i+1) - c(i))^2, f2 = (c(j+1) - c(j))^2 (the
// ghost ring supplies the outer differences).
template <class T>
__global__ void __launch_bounds__(BLOCK_THREADS)
    k_energy2(const DevPatch* __restrict__ PT, const Item* __restrict__ items,
              double* __restrict__ partials, DevStatus* __restrict__ st, int nitems, int which) {
  const Item it = items[blockIdx.x];
  const DevPatch P = PT[it.patch];
  const int j = it.ty * TILE_Y + threadIdx.y + 1;
  const int i0 = (it.tx * 32 + threadIdx.x) * 2 + 1;
  const T* c = fld<T>(P.q[0]);
  auto C = [&](int i, int jj) { return (double)c[cidx(P, i, jj, 0)]; };
  double acc = 0.0;
  if (j <= P.n[1]) {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int i = i0 + t;
      if (i > P.n[0]) break;
      if (which == 0) {
        acc += Problem::Ff(C(i, j), P.alpha);
      } else {
        const double a = C(i + 1, j) - C(i, j), b = C(i, j) - C(i - 1, j);
        const double u = C(i, j + 1) - C(i, j), w = C(i, j) - C(i, j - 1);
        acc += a * a + b * b + u * u + w * w;
      }
    }
  }
  const double bs = block_sum(acc);
  double total;
  if (last_block_total(bs, partials, &st->ticket, nitems, total)) st->esum = total;
}

// h^d * sum(phi) over a patch interior (AfterStep2D/3D integral(1)).
template <class T, int D>
__global__ void __launch_bounds__(BLOCK_THREADS)
    k_mass(const DevPatch* __restrict__ PT, const Item* __restrict__ items,
           double* __restrict__ partials, DevStatus* __restrict__ st, int nitems, double hd) {
  const Item it = items[blockIdx.x];
  const DevPatch P = PT[it.patch];
  const int j = it.ty * TILE_Y + threadIdx.y + 1;
  const int k = (D == 3) ? it.tz + 1 : 0;
  const int i0 = (it.tx * 32 + threadIdx.x) * 2 + 1;
  const T* q0 = fld<T>(P.q[0]);
  double acc = 0.0;
  if (j <= P.n[1]) {
    if (i0 <= P.n[0]) acc += (double)q0[cidx(P, i0, j, k)];
    if (i0 + 1 <= P.n[0]) acc += (double)q0[cidx(P, i0 + 1, j, k)];
  }
  const double bs = block_sum(acc);
  double total;
  if (last_block_total(bs, partials, &st->ticket, nitems, total)) st->mass = hd * total;
}

}  // namespace bsam
