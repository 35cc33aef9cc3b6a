// chain.cuh -- the coarse end of the V-cycle in shared memory, by one
// thread-block cluster.
//
// AFASVcycle (afas:488-521) from a top level down to the coarsest and back is
// a chain of dependent passes (eight colour passes, a restriction, a coarse
// load and a correction per level) over levels that are far too small for the
// GPU.  As launches they cost 5-10 us each whatever their size, and one CTA
// working in global memory takes about 1.4 us a pass.  k_chain holds the whole
// chain in the shared memory of up to 16 CTAs (one cluster): every level is
// cut into slabs of rows (2D) or planes (3D), one per CTA, with one halo row on
// either side; the thread that changes a slab's first or last row stores the
// new value into the neighbour's halo too (distributed shared memory), so a
// cluster barrier is all that separates two passes.  The smallest levels
// (CHAIN_TAIL_CELLS) belong to the cluster's first CTA alone.
//
// What bounds a pass is the instructions that one warp issues (two to three
// clocks each with a warp or two per scheduler) and the barrier, so everything
// that can be is taken out of it: a thread keeps a pair of cells -- one of each
// colour -- with their state, right-hand side and neighbours' addresses in
// registers over a whole smoothing stage, and a neighbour across a face is read
// as the face's map of the cell itself (SetBC after every pass makes the ghost
// just that), so that no ghosts are written on the way.  Restriction and
// residual join the pairs of one coarse cell with shuffles; corrections read
// the coarse level directly.  (A thread per 2 x 2 block, nothing to exchange but
// twice the instructions per thread, took 88 us for a V-cycle of 128^2 where this
// takes 53; pairs with ghosts written through 68.)
//
// Measured, one V-cycle (FP64): a 32^2 problem 84 -> 27 us, 128^2 217 -> 53 us
// (24 launches and a single-CTA kernel before; the solve's V-cycle loop is in the
// kernel too, see ChainLoop), 16^3 and below 54 us (128 us for 8^3 and below and
// 75 us of launches for 16^3 before).
//
// The per-cell arithmetic is the problem module's, on the same operands in the
// same order as in the grid kernels, so every value is the same bit for bit.
#pragma once
#include <algorithm>
#include <array>
#include <vector>

#include "kernels.cuh"

namespace bsam {

// A 128^2 level gives each of 16 CTAs 512 pairs of cells: one per thread.  (A
// cluster barrier takes 396 clocks with 256 threads a CTA, 476 with 512.)
constexpr int CHAIN_THREADS = 512;
constexpr int CHAIN_MAX_CTAS = 16;
constexpr int CHAIN_MAX_LEVELS = 12;
// Levels of at most this many cells are held by one CTA, where a pass needs no
// cluster barrier (0.25 us with 512 threads, 0.45 when it has to wait for stores
// to other CTAs).  At 1024 (32^2 there too) a V-cycle of 128^2 took 55.5 us
// against 52.9: the slabs above then reach into one CTA's memory for all of it.
constexpr int CHAIN_TAIL_CELLS = 512;
// A chain whose top has at most this many cells runs on one CTA (32^2: 27 us a
// V-cycle there).
constexpr int CHAIN_SINGLE_CELLS = 1024;

struct ChainLevel {
  int32_t patch;       // record
  int32_t n[3];
  int32_t ns;          // rows (2D) / planes (3D)
  int32_t pitch;       // elements of a row with its ghosts
  int32_t sstr;        // elements of a row (2D) / plane (3D)
  int32_t prec, delta;
  int32_t bc[6];
  int32_t maps;        // some face changes the value it copies (BC_REFLECT, BC_NEGATE)
  uint32_t w, h;       // pairs of a row, pairs of rows (3D)
  uint32_t mw, mh;     // x / w = umulhi(x, mw) and x / h likewise, for any index of the level
  int32_t active;      // CTAs that hold rows of it
  int32_t units;       // what they are dealt: pairs of rows, or rows when ns is odd
  // Byte offsets of the (phi, mu) pairs, the right-hand sides, the snapshot and
  // the base; in the kernel, addresses in the CTA's shared window.
  uint32_t q, f, qs, bs;
  double tmp1, tmp2, tmp3, alpha;
};

struct ChainPlan {
  int32_t nlev;    // levels, top first
  int32_t nslab;   // the first nslab of them are held by several CTAs
  int32_t nu;      // smoothing sweeps
  int32_t ctas;    // CTAs of the cluster
  uint32_t rsum;   // byte offset of the residual's row sums (first CTA)
  uint32_t smem;   // bytes
  ChainLevel L[CHAIN_MAX_LEVELS];
};

// MultigridIterations' loop in the kernel (the chain's top is the finest
// level, FP64): V-cycles until the residual is below tol, at most maxv.
// maxv = 0: one V-cycle, no residual.
struct ChainLoop {
  int32_t maxv, pad_;
  double tol, denom;
  DevStatus* st;
  double* trace;
};

// This CTA's part of a level: rows lo .. lo + nr - 1 in row slots 1 .. nr, and
// the CTAs whose halo slots its first and last row feed (null at the level's
// own faces).
struct ChainSlab {
  int32_t lo, nr;
  int32_t lo_t, hi_t;    // the row slots there
  int32_t lo_r, hi_r;    // their ranks, -1 at the level's own faces
};

// Rows [first, first + count) of CTA r of a level.
__host__ __device__ __forceinline__ void chain_rows(const ChainLevel& L, int r, int& first, int& count) {
  const int per = L.ns % 2 ? 1 : 2;
  const int a = r * L.units / L.active, b = (r + 1) * L.units / L.active;
  first = a * per + 1;
  count = (b - a) * per;
}

// CTA `rank`'s part of a level; no rows (nr = 0) beyond the level's active CTAs.
template <int D>
__host__ __device__ __forceinline__ ChainSlab chain_slab(const ChainLevel& L, int rank) {
  ChainSlab S{};
  S.lo = 1;
  S.lo_r = S.hi_r = -1;
  if (rank >= L.active) return S;
  chain_rows(L, rank, S.lo, S.nr);
  const bool per = L.bc[2 * D - 2] == BC_PERIODIC;
  if (L.active > 1 && (rank > 0 || per)) {
    const int nb = rank > 0 ? rank - 1 : L.active - 1;
    int first, count;
    chain_rows(L, nb, first, count);
    S.lo_r = nb;
    S.lo_t = count + 1;
  }
  if (L.active > 1 && (rank + 1 < L.active || per)) {
    S.hi_r = rank + 1 < L.active ? rank + 1 : 0;
    S.hi_t = 0;
  }
  return S;
}

// The CTA that holds row k (1-based) of a level: the last one that starts at or
// before it.
__device__ __forceinline__ int chain_owner(const ChainLevel& L, int k) {
  const int u = L.ns % 2 ? k : (k + 1) / 2;
  return (u * L.active - 1) / L.units;
}

template <int D>
__host__ __device__ __forceinline__ int chain_idx(const ChainLevel& L, int i, int j, int t) {
  return D == 2 ? i + t * L.sstr : i + j * L.pitch + t * L.sstr;
}

// Both components of a value side by side: one shared-memory access each way.
template <class T> struct ChainV;
template <> struct ChainV<float> { using V = float2; };
template <> struct ChainV<double> { using V = double2; };

// Shared memory is addressed by 32-bit addresses, this CTA's in its own window,
// another CTA's in the cluster's (the compiler's pointers made it work the
// window's base out anew at every access, a third of a pass's instructions).
__device__ __forceinline__ uint32_t chain_base() {
  extern __shared__ __align__(128) unsigned char chain_raw[];
  return (uint32_t)__cvta_generic_to_shared(chain_raw);
}

// The address of this CTA's address `a` in CTA `rank`.
__device__ __forceinline__ uint32_t chain_map_rank(uint32_t a, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}

#define CHAIN_ACCESS(V, T, C, SUF)                                                              \
  __device__ __forceinline__ V chain_ld(uint32_t a, V) {                                        \
    V v;                                                                                        \
    asm volatile("ld.shared.v2." SUF " {%0, %1}, [%2];" : "=" C(v.x), "=" C(v.y) : "r"(a));     \
    return v;                                                                                   \
  }                                                                                             \
  __device__ __forceinline__ V chain_ld_cluster(uint32_t a, V) {                                \
    V v;                                                                                        \
    asm volatile("ld.shared::cluster.v2." SUF " {%0, %1}, [%2];"                                \
                 : "=" C(v.x), "=" C(v.y)                                                       \
                 : "r"(a));                                                                     \
    return v;                                                                                   \
  }                                                                                             \
  __device__ __forceinline__ void chain_st(uint32_t a, V v) {                                   \
    asm volatile("st.shared.v2." SUF " [%0], {%1, %2};" ::"r"(a), C(v.x), C(v.y) : "memory");   \
  }                                                                                             \
  __device__ __forceinline__ void chain_st_cluster(uint32_t a, V v) {                           \
    asm volatile("st.shared::cluster.v2." SUF " [%0], {%1, %2};" ::"r"(a), C(v.x), C(v.y)       \
                 : "memory");                                                                   \
  }                                                                                             \
  __device__ __forceinline__ T chain_ld(uint32_t a, T) {                                        \
    T v;                                                                                        \
    asm volatile("ld.shared." SUF " %0, [%1];" : "=" C(v) : "r"(a));                            \
    return v;                                                                                   \
  }                                                                                             \
  __device__ __forceinline__ void chain_st(uint32_t a, T v) {                                   \
    asm volatile("st.shared." SUF " [%0], %1;" ::"r"(a), C(v) : "memory");                      \
  }                                                                                             \
  __device__ __forceinline__ void chain_st_cluster(uint32_t a, T v) {                           \
    asm volatile("st.shared::cluster." SUF " [%0], %1;" ::"r"(a), C(v) : "memory");             \
  }
CHAIN_ACCESS(float2, float, "f", "f32")
CHAIN_ACCESS(double2, double, "d", "f64")
#undef CHAIN_ACCESS

// The cluster's barrier, by all its threads (release and acquire).
__device__ __forceinline__ void chain_cluster_sync() {
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// bc_map without branches on the value (2 + (-v) rounds as 2 - v).
template <class T> __device__ __forceinline__ T chain_map(int code, T v) {
  const T w = (code == BC_REFLECT || code == BC_NEGATE) ? -v : v;
  return code == BC_REFLECT ? T(2) + w : w;
}

__host__ __device__ __forceinline__ uint32_t chain_div(uint32_t x, uint32_t d, uint32_t m) {
#ifdef __CUDA_ARCH__
  return d == 1 ? x : __umulhi(x, m);
#else
  return d == 1 ? x : (uint32_t)(((uint64_t)x * m) >> 32);
#endif
}

// A cell: its index, and per dimension and side the address of the cell that
// is read as its neighbour there; the maps its values go through, four bits each.
template <class T, int D> struct ChainCell {
  int c;
  uint32_t at[2 * D];
  uint32_t code;
  T p, m, f0, f1, b;  // state, right-hand side, base (correction form)
};

template <class T>
__host__ __device__ __forceinline__ uint32_t chain_byte(uint32_t field, int idx) {
  return field + (uint32_t)idx * (uint32_t)sizeof(typename ChainV<T>::V);
}

// The neighbours of the cell at index X.c, coordinates (i, j), row slot t.
template <class T, int D>
__host__ __device__ __forceinline__ void chain_nb(const ChainLevel& L, const ChainSlab& S, int i,
                                                  int j, int t, ChainCell<T, D>& X) {
  X.code = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const bool slow = d == D - 1;
    const int st = d == 0 ? 1 : (slow ? L.sstr : L.pitch);
    const int n = slow ? L.ns : L.n[d], x = d == 0 ? i : (slow ? t : j);
    const int blo = L.bc[2 * d], bhi = L.bc[2 * d + 1];
    const bool lo = x == 1 && !(slow && S.lo_r >= 0);
    const bool hi = x == (slow ? S.nr : n) && !(slow && S.hi_r >= 0);
    const bool per = blo == BC_PERIODIC;
    X.at[2 * d] = chain_byte<T>(L.q, X.c + (lo ? (per ? (n - 1) * st : 0) : -st));
    X.at[2 * d + 1] = chain_byte<T>(L.q, X.c + (hi ? (per ? -(n - 1) * st : 0) : st));
    if (lo && !per) X.code |= (uint32_t)blo << (8 * d);
    if (hi && !per) X.code |= (uint32_t)bhi << (8 * d + 4);
  }
}

// The same with the ghosts as the caller's arrays hold them, which is how the
// first sweep of a solve finds them (the faces' maps of the cells by then,
// unless the caller left others).  A pass updates the periodic ghosts of the
// next one (fed from the other end, of the other colour): all but the first
// pass read those in place.
template <class T, int D>
__host__ __device__ __forceinline__ void chain_nb_raw(const ChainLevel& L, bool first,
                                                      ChainCell<T, D>& X) {
  X.code = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const int st = d == 0 ? 1 : (d == D - 1 ? L.sstr : L.pitch);
    if (!first && L.bc[2 * d] == BC_PERIODIC) continue;
    X.at[2 * d] = chain_byte<T>(L.q, X.c - st);
    X.at[2 * d + 1] = chain_byte<T>(L.q, X.c + st);
  }
}

template <class T, int D, bool DELTA>
__device__ __forceinline__ void chain_operator(const ChainLevel& L,
                                               const Problem::Stencil<T, D>& s, T base, T& o0,
                                               T& o1) {
  if (DELTA)
    Problem::OperatorCell<T, D, true>(s, T(L.tmp1), T(L.tmp2), T(L.alpha), o0, o1, base);
  else
    Problem::OperatorCell<T, D>(s, T(L.tmp1), T(L.tmp2), T(L.alpha), o0, o1);
}

// The copies of cell c, row slot t, in the halos of the neighbours: addresses in
// the cluster's shared window, 0 where there is none (static data lies there).
struct ChainPush {
  uint32_t lo, hi;
};
template <class T>
__device__ __forceinline__ ChainPush chain_push(const ChainLevel& L, const ChainSlab& S, int c,
                                                int t) {
  ChainPush p{0u, 0u};
  if (t == 1 && S.lo_r >= 0)
    p.lo = chain_map_rank(chain_byte<T>(L.q, c + (S.lo_t - t) * L.sstr), S.lo_r);
  if (t == S.nr && S.hi_r >= 0)
    p.hi = chain_map_rank(chain_byte<T>(L.q, c + (S.hi_t - t) * L.sstr), S.hi_r);
  return p;
}

// What the phases share; everything is uniform over the CTA.
struct ChainCtx {
  const ChainPlan* PL;
  const ChainSlab* S;      // per level
  int rank;
};

// ---- cells ----------------------------------------------------------------------

// State, right-hand side and base of a cell.
template <class T, int D, bool DELTA>
__device__ __forceinline__ void chain_fetch(const ChainLevel& L, ChainCell<T, D>& X) {
  using V = typename ChainV<T>::V;
  const V q = chain_ld(chain_byte<T>(L.q, X.c), V{});
  const V f = chain_ld(chain_byte<T>(L.f, X.c - L.sstr), V{});  // f has no halo row
  X.p = q.x;
  X.m = q.y;
  X.f0 = f.x;
  X.f1 = f.y;
  X.b = DELTA ? chain_ld(L.bs + (uint32_t)(X.c - L.sstr) * (uint32_t)sizeof(T), T(0)) : T(0);
}

// Its stencil; `move`: bytes from the state to the field that is read.
template <class T, int D>
__device__ __forceinline__ void chain_stencil(const ChainLevel& L, const ChainCell<T, D>& X,
                                              uint32_t move, Problem::Stencil<T, D>& s) {
  using V = typename ChainV<T>::V;
  s.pc = X.p;
  s.mc = X.m;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const V lo = chain_ld(X.at[2 * d] + move, V{}), hi = chain_ld(X.at[2 * d + 1] + move, V{});
    s.pm[d] = lo.x;
    s.pp[d] = hi.x;
    s.mm[d] = lo.y;
    s.mp[d] = hi.y;
  }
  if (L.maps) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const int lo = (X.code >> (8 * d)) & 15, hi = (X.code >> (8 * d + 4)) & 15;
      s.pm[d] = chain_map<T>(lo, s.pm[d]);
      s.pp[d] = chain_map<T>(hi, s.pp[d]);
      s.mm[d] = chain_map<T>(lo, s.mm[d]);
      s.mp[d] = chain_map<T>(hi, s.mp[d]);
    }
  }
}

// Stores a cell's state, here and in the halos that hold it (`shift` bytes from
// where p points).
template <class T, int D, bool SLAB>
__device__ __forceinline__ void chain_put(const ChainLevel& L, const ChainCell<T, D>& X,
                                          const ChainPush& p, uint32_t shift) {
  using V = typename ChainV<T>::V;
  V v;
  v.x = X.p;
  v.y = X.m;
  chain_st(chain_byte<T>(L.q, X.c), v);
  if (SLAB) {
    if (p.lo) chain_st_cluster(p.lo + shift, v);
    if (p.hi) chain_st_cluster(p.hi + shift, v);
  }
}

// RelaxGrid at a cell.
template <class T, int D, bool DELTA>
__device__ __forceinline__ void chain_relax(const ChainLevel& L, ChainCell<T, D>& X) {
  Problem::Stencil<T, D> s;
  chain_stencil<T, D>(L, X, 0u, s);
  if (DELTA)
    Problem::RelaxCell<T, D, true>(s, X.f0, X.f1, T(L.tmp1), T(L.tmp2), T(L.tmp3), T(L.alpha),
                                   X.p, X.m, X.b);
  else
    Problem::RelaxCell<T, D>(s, X.f0, X.f1, T(L.tmp1), T(L.tmp2), T(L.tmp3), T(L.alpha), X.p,
                             X.m);
}

// The second half of CoarseLoadingFunction: f += Operator(qs), q == qs still.
template <class T, int D, bool DELTA>
__device__ __forceinline__ void chain_add_load(const ChainLevel& L, ChainCell<T, D>& X) {
  using V = typename ChainV<T>::V;
  Problem::Stencil<T, D> s;
  chain_stencil<T, D>(L, X, L.qs - L.q, s);
  T o0, o1;
  chain_operator<T, D, DELTA>(L, s, X.b, o0, o1);
  X.f0 = X.f0 + o0;
  X.f1 = X.f1 + o1;
  V v;
  v.x = X.f0;
  v.y = X.f1;
  chain_st(chain_byte<T>(L.f, X.c - L.sstr), v);
}

// ---- pairs ----------------------------------------------------------------------
//
// Fine cells 2 ic - 1 and 2 ic of a row.  Pairs are numbered so that the 2 (2D)
// or 4 (3D) pairs of one coarse cell are neighbouring lanes: bit d - 1 of the
// pair's number is its row's place in dimension d (0: odd coordinate).

template <class T, int D> struct ChainPair {
  ChainCell<T, D> A, B;  // the cells of colours 0 and 1 (even and odd coordinate sums)
  int ic, jc, tc;        // coarse x, y (3D), and row of the slab in pairs (1-based)
  int t, j;              // row slot, y (3D)
  int c;                 // index of the left-hand cell
  bool on, right;        // right: A is the right-hand cell
  ChainPush push;        // of the left-hand cell
  __device__ __forceinline__ uint32_t shift(bool a) const {  // of cell A (a) or B
    return a == right ? (uint32_t)sizeof(typename ChainV<T>::V) : 0u;
  }
};

// The pairs of a CTA's slab.
template <int D>
__host__ __device__ __forceinline__ int chain_pairs(const ChainLevel& L, const ChainSlab& S) {
  return (int)(L.w * L.h) * (S.nr >> 1) << (D - 1);
}

// Does a CTA run a level's phases?  Every thread of one that does runs them (whole
// warps, for the shuffles; threads without a pair of their own work on pair 0 and
// store nothing).  A CTA without rows of the level (more CTAs than units) only
// keeps the barriers: it has no pair 0, and the cell across a periodic face that
// chain_nb would give it lies a whole level away, beyond its shared memory.
__host__ __device__ __forceinline__ bool chain_runs(const ChainSlab& S) { return S.nr > 0; }

template <class T, int D>
__host__ __device__ __forceinline__ void chain_pair(const ChainLevel& L, const ChainSlab& S,
                                                    int idx, ChainPair<T, D>& R) {
  constexpr int SUB = D - 1;  // bits of the pair in its coarse cell
  R.on = idx < chain_pairs<D>(L, S);
  const uint32_t sub = idx & ((1 << SUB) - 1), u = R.on ? (uint32_t)idx >> SUB : 0u;
  const uint32_t r = chain_div(u, L.w, L.mw);
  R.ic = (int)(u - r * L.w) + 1;
  const uint32_t z = D == 3 ? chain_div(r, L.h, L.mh) : r;
  R.tc = (int)z + 1;
  R.jc = D == 3 ? (int)(r - z * L.h) + 1 : 0;
  R.t = 2 * R.tc - 1 + (int)(sub >> (SUB - 1));
  R.j = D == 3 ? 2 * R.jc - 1 + (int)(sub & 1) : 0;
  const int i0 = 2 * R.ic - 1;
  // Slabs start at odd rows, so slot and row have the same parity.
  R.right = (i0 + R.j + R.t) & 1;
  const int c0 = chain_idx<D>(L, i0, R.j, R.t);
  R.c = c0;
  R.A.c = c0 + (R.right ? 1 : 0);
  R.B.c = c0 + (R.right ? 0 : 1);
  chain_nb<T, D>(L, S, i0 + (R.right ? 1 : 0), R.j, R.t, R.A);
  chain_nb<T, D>(L, S, i0 + (R.right ? 0 : 1), R.j, R.t, R.B);
}

// RestrictSolution and the restricted residual (the first half of
// CoarseLoadingFunction) of the pairs of a coarse cell into level P, in the
// memory of the CTA that holds the coarse row: q, its snapshot qs, the base,
// and the residual in f.  Sums in the reference's order of the children (x
// fastest, from the high end).  Every lane of the warp calls it.
template <class T, class TP, int D, bool DELTA>
__device__ __forceinline__ void chain_down(const ChainLevel& L, const ChainSlab& S,
                                           const ChainPair<T, D>& R, const ChainLevel& P) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int NP = 1 << (D - 1);  // pairs of a coarse cell
  T rA0 = T(0), rA1 = T(0), rB0 = T(0), rB1 = T(0);
  {
    Problem::Stencil<T, D> s;
    T o0, o1;
    chain_stencil<T, D>(L, R.A, 0u, s);
    chain_operator<T, D, DELTA>(L, s, R.A.b, o0, o1);
    rA0 = R.A.f0 - o0;
    rA1 = R.A.f1 - o1;
    chain_stencil<T, D>(L, R.B, 0u, s);
    chain_operator<T, D, DELTA>(L, s, R.B.b, o0, o1);
    rB0 = R.B.f0 - o0;
    rB1 = R.B.f1 - o1;
  }
  // Right-hand and left-hand values.
  auto hi = [&](T a, T b) { return R.right ? a : b; };
  auto lo = [&](T a, T b) { return R.right ? b : a; };
  const int lane = threadIdx.x & 31, sub = lane & (NP - 1);
  T v[4];  // phi, mu, residuals: sums over the children
  T vb = T(0);
  if (D == 2) {
    // The upper pair's lane sums phi and its residual, the lower one's mu and
    // its residual: each sends the other what it needs.
    const bool up = sub == 1;
    const T sr = up ? hi(R.A.m, R.B.m) : hi(R.A.p, R.B.p), sl = up ? lo(R.A.m, R.B.m) : lo(R.A.p, R.B.p);
    const T tr = up ? hi(rA1, rB1) : hi(rA0, rB0), tl = up ? lo(rA1, rB1) : lo(rA0, rB0);
    const T gr = __shfl_xor_sync(FULL, sr, 1), gl = __shfl_xor_sync(FULL, sl, 1);
    const T hr = __shfl_xor_sync(FULL, tr, 1), hl = __shfl_xor_sync(FULL, tl, 1);
    const T mr = up ? hi(R.A.p, R.B.p) : hi(R.A.m, R.B.m), ml = up ? lo(R.A.p, R.B.p) : lo(R.A.m, R.B.m);
    const T nr = up ? hi(rA0, rB0) : hi(rA1, rB1), nl = up ? lo(rA0, rB0) : lo(rA1, rB1);
    // Upper pair first.
    v[0] = ((up ? mr : gr) + (up ? ml : gl)) + (up ? gr : mr) + (up ? gl : ml);
    v[2] = ((up ? nr : hr) + (up ? nl : hl)) + (up ? hr : nr) + (up ? hl : nl);
    if (DELTA) {
      const T br = hi(R.A.b, R.B.b), bl = lo(R.A.b, R.B.b);
      const T or_ = __shfl_xor_sync(FULL, br, 1), ol = __shfl_xor_sync(FULL, bl, 1);
      vb = br + bl + or_ + ol;  // used by the upper lane alone
    }
  } else {
    const T w8[4][2] = {{hi(R.A.p, R.B.p), lo(R.A.p, R.B.p)},
                        {hi(R.A.m, R.B.m), lo(R.A.m, R.B.m)},
                        {hi(rA0, rB0), lo(rA0, rB0)},
                        {hi(rA1, rB1), lo(rA1, rB1)}};
    const T wb[2] = {hi(R.A.b, R.B.b), lo(R.A.b, R.B.b)};
#pragma unroll
    for (int k = NP - 1; k >= 0; --k) {
      const int src = (lane & ~(NP - 1)) + k;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const T r = __shfl_sync(FULL, w8[g][0], src), l = __shfl_sync(FULL, w8[g][1], src);
        v[g] = k == NP - 1 ? r + l : v[g] + r + l;
      }
      if (DELTA) {
        const T r = __shfl_sync(FULL, wb[0], src), l = __shfl_sync(FULL, wb[1], src);
        vb = k == NP - 1 ? r + l : vb + r + l;
      }
    }
  }
  const T wt = D == 2 ? T(0.25) : T(0.125);
  // 2D: the pair's two lanes exchange their sums, so that one stores the state
  // and the other the right-hand side; 3D: every lane has all four.
  using V = typename ChainV<TP>::V;
  V q, res;
  if (D == 2) {
    const T a = __shfl_xor_sync(FULL, sub ? v[2] : v[0], 1);
    q.x = TP(wt * v[0]);
    q.y = TP(wt * a);
    res.x = TP(wt * a);
    res.y = TP(wt * v[2]);
  } else {
    q.x = TP(wt * v[0]);
    q.y = TP(wt * v[1]);
    res.x = TP(wt * v[2]);
    res.y = TP(wt * v[3]);
  }
  if (!R.on || sub > 1) return;
  // Lane 1 stores the state (2D: it is the upper pair's, whose sums are phi's),
  // lane 0 the right-hand side.
  const int kc = (S.lo - 1) / 2 + R.tc;  // the coarse row
  const int own = P.active == 1 ? 0 : chain_owner(P, kc);
  int first = 1, count = P.ns;
  if (P.active > 1) chain_rows(P, own, first, count);
  const int t = kc - first + 1;
  if (sub == 0) {
    const int fc = chain_idx<D>(P, R.ic, R.jc, t - 1);
    chain_st_cluster(chain_map_rank(chain_byte<TP>(P.f, fc), own), res);
    return;
  }
  auto put = [&](int rank, int slot) {
    const int c = chain_idx<D>(P, R.ic, R.jc, slot);
    chain_st_cluster(chain_map_rank(chain_byte<TP>(P.q, c), rank), q);
    chain_st_cluster(chain_map_rank(chain_byte<TP>(P.qs, c), rank), q);
  };
  put(own, t);
  if (DELTA) {
    const int fc = chain_idx<D>(P, R.ic, R.jc, t - 1);
    chain_st_cluster(chain_map_rank(P.bs + (uint32_t)fc * (uint32_t)sizeof(TP), own),
                       TP(wt * vb));
  }
  // The halos of the coarse rows next to the owner's slab.
  if (P.active > 1) {
    const bool per = P.bc[2 * D - 2] == BC_PERIODIC;
    if (t == 1 && (own > 0 || per)) {
      const int nb = own > 0 ? own - 1 : P.active - 1;
      int a, n;
      chain_rows(P, nb, a, n);
      put(nb, n + 1);
    }
    if (t == count && (own + 1 < P.active || per)) put(own + 1 < P.active ? own + 1 : 0, 0);
  }
}

// CorrectFine of a pair from the change q - qs of the coarse level P, read in
// the CTA that holds the coarse row (whose halo rows are next to it).  A fine
// cell takes 3/4 of its own coarse cell (near) and 1/4 of the next one on its
// side (far) per dimension, x first: lin_x's sums, whose two terms commute.
template <class T, class TP, int D, bool SLAB>
__device__ __forceinline__ void chain_up(const ChainLevel& L, const ChainSlab& S,
                                         ChainPair<T, D>& R, const ChainLevel& P) {
  const int kc = (S.lo - 1) / 2 + R.tc;
  const int own = P.active == 1 ? 0 : chain_owner(P, kc);
  int first = 1, count = P.ns;
  if (P.active > 1) chain_rows(P, own, first, count);
  using V = typename ChainV<TP>::V;
  const int c = chain_idx<D>(P, R.ic, R.jc, kc - first + 1);
  const uint32_t q = chain_map_rank(chain_byte<TP>(P.q, c), own);
  const uint32_t s = q + (P.qs - P.q);
  // Far side of dimension d: the index offset and the face's map.
  auto far = [&](int d, bool high, int x, int n, int st, int& off, int& code) {
    const int bc = P.bc[2 * d + (high ? 1 : 0)];
    const bool face = x == (high ? n : 1);
    const bool halo = d == D - 1 && P.active > 1 && (!face || bc == BC_PERIODIC);
    code = BC_COPY;
    off = high ? st : -st;
    if (!face || halo) return;
    off = bc == BC_PERIODIC ? (high ? -(n - 1) * st : (n - 1) * st) : 0;
    if (bc != BC_PERIODIC) code = bc;
  };
  int xl, xh, cl, ch, yo = 0, yc = BC_COPY, zo, zc;
  far(0, false, R.ic, P.n[0], 1, xl, cl);
  far(0, true, R.ic, P.n[0], 1, xh, ch);
  if (D == 3) far(1, !(R.j & 1), R.jc, P.n[1], P.pitch, yo, yc);
  far(D - 1, !(R.t & 1), kc, P.ns, P.sstr, zo, zc);
  auto e = [&](int k, int cx, int cy, int cz) {
    V a = chain_ld_cluster(q + k * (int)sizeof(V), V{}), b = chain_ld_cluster(s + k * (int)sizeof(V), V{});
    if (P.maps) {
      auto m = [&](TP x) { return chain_map<TP>(cz, chain_map<TP>(cy, chain_map<TP>(cx, x))); };
      a.x = m(a.x);
      a.y = m(a.y);
      b.x = m(b.x);
      b.y = m(b.y);
    }
    a.x = a.x - b.x;
    a.y = a.y - b.y;
    return a;
  };
  // 3 near + far.
  auto mix = [](V n, V f) {
    V r;
    r.x = TP(3) * n.x + f.x;
    r.y = TP(3) * n.y + f.y;
    return r;
  };
  // Left and right values of one coarse row (offset k, maps cy, cz).
  auto row = [&](int k, int cy, int cz, V& l, V& r) {
    const V n = e(k, BC_COPY, cy, cz);
    l = mix(n, e(k + xl, cl, cy, cz));
    r = mix(n, e(k + xh, ch, cy, cz));
  };
  V l, r, l2, r2;
  row(0, BC_COPY, BC_COPY, l, r);
  if (D == 3) {
    row(yo, yc, BC_COPY, l2, r2);
    l = mix(l, l2);
    r = mix(r, r2);
  }
  row(zo, BC_COPY, zc, l2, r2);
  if (D == 3) {
    V l3, r3;
    row(yo + zo, yc, zc, l3, r3);
    l2 = mix(l2, l3);
    r2 = mix(r2, r3);
  }
  l = mix(l, l2);
  r = mix(r, r2);
  const TP w = D == 2 ? TP(16) : TP(64);
  R.A.p = R.A.p + T((R.right ? r.x : l.x) / w);
  R.A.m = R.A.m + T((R.right ? r.y : l.y) / w);
  R.B.p = R.B.p + T((R.right ? l.x : r.x) / w);
  R.B.m = R.B.m + T((R.right ? l.y : r.y) / w);
  chain_put<T, D, SLAB>(L, R.A, R.push, R.shift(true));
  chain_put<T, D, SLAB>(L, R.B, R.push, R.shift(false));
}

// ---- stages ---------------------------------------------------------------------

// The barrier between the phases of a level: the cluster's, or in the tail the
// one of the warps that take part.
template <bool SLAB> struct ChainSync {
  int warps;
  __device__ __forceinline__ void operator()() const {
    if (SLAB) chain_cluster_sync();
    else if (warps == 1) asm volatile("bar.warp.sync 0xffffffff;" ::: "memory");
    else asm volatile("bar.sync 1, %0;" ::"r"(32 * warps) : "memory");
  }
};

// A level's visit on the way down (coarse load, pre-smoothing, then restriction
// and residual into the next level) or up (correction from it, then
// post-smoothing).  SINGLE: at most a pair per thread, whose registers hold it
// throughout; else every phase loads and stores the pairs.
template <class T, class TP, int D, bool DELTA, bool SLAB, bool SINGLE>
__device__ __forceinline__ void chain_visit_pairs(const ChainCtx& X, int l, bool up, bool raw,
                                                  const ChainLevel& L, const ChainSlab& S,
                                                  const ChainLevel& P, ChainSync<SLAB> sync) {
  const int nt = SLAB ? (int)blockDim.x : 32 * sync.warps;
  ChainPair<T, D> R;
  R.on = false;
  auto load = [&](int idx) {
    chain_pair<T, D>(L, S, idx, R);
    R.push = chain_push<T>(L, S, R.c, R.t);
    // Lanes without a pair work on pair 0's values and store nothing.
    chain_fetch<T, D, DELTA>(L, R.A);
    chain_fetch<T, D, DELTA>(L, R.B);
  };
  const int total = chain_pairs<D>(L, S);
  // One phase over the pairs of this thread (whole warps, for the shuffles).
  auto each = [&](auto body) {
    if constexpr (SINGLE) {
      body();
    } else {
      for (int base = threadIdx.x & ~31; base < total; base += nt) {
        load(base + (threadIdx.x & 31));
        body();
      }
    }
  };
  if (SINGLE) load(threadIdx.x);
  if (up) {
    each([&] {
      if (R.on) chain_up<T, TP, D, SLAB>(L, S, R, P);
    });
    sync();
  } else if (l > 0) {
    each([&] {
      if (!R.on) return;
      chain_add_load<T, D, DELTA>(L, R.A);
      chain_add_load<T, D, DELTA>(L, R.B);
    });
  }
  const int passes = 2 * X.PL->nu;
  for (int p = 0; p < passes; p += 2) {
    const bool held = raw && p == 0;
    each([&] {
      if (held) chain_nb_raw<T, D>(L, true, R.A);
      chain_relax<T, D, DELTA>(L, R.A);
      if (R.on) chain_put<T, D, SLAB>(L, R.A, R.push, R.shift(true));
      if (held) chain_nb<T, D>(L, S, 2 * R.ic - (R.right ? 0 : 1), R.j, R.t, R.A);
    });
    sync();
    each([&] {
      if (held) chain_nb_raw<T, D>(L, false, R.B);
      chain_relax<T, D, DELTA>(L, R.B);
      if (R.on) chain_put<T, D, SLAB>(L, R.B, R.push, R.shift(false));
      if (held) chain_nb<T, D>(L, S, 2 * R.ic - (R.right ? 1 : 0), R.j, R.t, R.B);
    });
    sync();
  }
  if (!up) {
    each([&] { chain_down<T, TP, D, DELTA>(L, S, R, P); });
    sync();
  }
}

// The coarsest level, a cell per thread: load and smoothing.
template <class T, int D, bool DELTA, bool SLAB>
__device__ __forceinline__ void chain_visit_cells(const ChainCtx& X, int l, bool raw,
                                                  const ChainLevel& L, const ChainSlab& S,
                                                  ChainSync<SLAB> sync) {
  const int nt = SLAB ? (int)blockDim.x : 32 * sync.warps;
  const int w = L.n[0], h = D == 3 ? L.n[1] : 1, total = w * h * S.nr;
  const bool single = total <= nt;
  ChainCell<T, D> C;
  int i = 1, j = 0, t = 1, color = -1;
  ChainPush push{0u, 0u};
  auto load = [&](int k) {
    const int r = k / w;
    i = k - r * w + 1;
    t = D == 3 ? r / h + 1 : r + 1;
    j = D == 3 ? r - (t - 1) * h + 1 : 0;
    color = (i + j + S.lo + t - 1) & 1;
    C.c = chain_idx<D>(L, i, j, t);
    chain_nb<T, D>(L, S, i, j, t, C);
    chain_fetch<T, D, DELTA>(L, C);
    push = chain_push<T>(L, S, C.c, t);
  };
  auto each = [&](auto body) {
    if (single) {
      if ((int)threadIdx.x < total) body();
      return;
    }
    for (int k = threadIdx.x; k < total; k += nt) {
      load(k);
      body();
    }
  };
  if (single && (int)threadIdx.x < total) load(threadIdx.x);
  if (l > 0) each([&] { chain_add_load<T, D, DELTA>(L, C); });
  for (int p = 0; p < 2 * X.PL->nu; ++p) {
    each([&] {
      if (color != (p & 1)) return;
      if (raw && p < 2) chain_nb_raw<T, D>(L, p == 0, C);
      chain_relax<T, D, DELTA>(L, C);
      chain_put<T, D, SLAB>(L, C, push, 0u);
      if (raw && p < 2) chain_nb<T, D>(L, S, i, j, t, C);
    });
    sync();
  }
}

// A visit of level l: up, from the coarser level; raw, ghosts of the first sweep
// as the arrays hold them.
template <class T, class TP, int D, bool DELTA, bool SLAB>
__device__ __noinline__ void chain_visit_t(const ChainCtx& X, int l, bool up, bool raw) {
  const ChainLevel L = X.PL->L[l];  // by value: its fields stay in registers
  const ChainSlab S = X.S[l];
  const bool last = l + 1 == X.PL->nlev;
  if (SLAB && !chain_runs(S)) {
    // The barriers of a visit: two a sweep, and where there is a coarser level one
    // after the correction (up) or the restriction (down).
    for (int b = 2 * X.PL->nu + (last ? 0 : 1); b > 0; --b) chain_cluster_sync();
    return;
  }
  const int cells = L.n[0] * (D == 3 ? L.n[1] : 1) * S.nr, work = last ? cells : cells >> 1;
  const ChainSync<SLAB> sync{min(max((work + 31) / 32, 1), (int)blockDim.x / 32)};
  if (!SLAB && (int)threadIdx.x >= 32 * sync.warps) {
    __syncthreads();
    return;
  }
  if (last) {
    chain_visit_cells<T, D, DELTA, SLAB>(X, l, raw, L, S, sync);
  } else {
    const ChainLevel& P = X.PL->L[l + 1];
    if (work <= (int)blockDim.x)
      chain_visit_pairs<T, TP, D, DELTA, SLAB, true>(X, l, up, raw, L, S, P, sync);
    else
      chain_visit_pairs<T, TP, D, DELTA, SLAB, false>(X, l, up, raw, L, S, P, sync);
  }
  if (!SLAB) __syncthreads();
}

template <class T, class TP, int D, bool DELTA>
__device__ __forceinline__ void chain_visit_s(const ChainCtx& X, int l, bool up, bool raw) {
  if (l < X.PL->nslab) chain_visit_t<T, TP, D, DELTA, true>(X, l, up, raw);
  else chain_visit_t<T, TP, D, DELTA, false>(X, l, up, raw);
}

template <int D, bool MIXED>
__device__ __forceinline__ void chain_visit(const ChainCtx& X, int l, bool up, bool raw) {
  if (!MIXED) {
    chain_visit_s<double, double, D, false>(X, l, up, raw);
    return;
  }
  const bool cf = X.PL->L[l].prec == PREC_F32;
  const bool pf = cf && l + 1 < X.PL->nlev && X.PL->L[l + 1].prec == PREC_F32;
  if (!cf) chain_visit_s<double, double, D, true>(X, l, up, raw);
  else if (pf) chain_visit_s<float, float, D, true>(X, l, up, raw);
  else chain_visit_s<float, double, D, true>(X, l, up, raw);
}

// AFASVcycle of the whole chain, in shared memory.
template <int D, bool MIXED>
__device__ __forceinline__ void chain_vcycle(const ChainCtx& X, bool raw) {
  const int ns = X.PL->nslab, nl = X.PL->nlev;
  for (int l = 0; l < ns; ++l) chain_visit<D, MIXED>(X, l, false, raw && l == 0);
  if (nl > ns) {
    if (X.rank == 0) {
      for (int l = ns; l < nl; ++l) chain_visit<D, MIXED>(X, l, false, raw && l == 0);
      for (int l = nl - 2; l >= ns; --l) chain_visit<D, MIXED>(X, l, true, false);
    }
    if (ns > 0) chain_cluster_sync();
  }
  for (int l = min(ns, nl - 1) - 1; l >= 0; --l) chain_visit<D, MIXED>(X, l, true, false);
}

// ErrorAFAS of the top level (FP64), summed in the order of resid_rows
// and last_block_sum: per tile of 64 x TILE_Y cells a shuffle
// tree per row, the rows in order; the tiles by 128 strided sums and the same
// tree.  Valid in thread 0 of CTA 0.
template <int D>
__device__ __noinline__ double chain_resid(const ChainCtx& X) {
  const ChainLevel L = X.PL->L[0];
  const ChainSlab S = X.S[0];
  const uint32_t sums = X.PL->rsum;  // CTA 0's
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nseg = (L.n[0] + TILE_X - 1) / TILE_X;
  const int ny = D == 3 ? L.n[1] : L.ns;
  const int rows = S.nr * (D == 3 ? L.n[1] : 1);
  for (int w = warp; w < rows * nseg; w += CHAIN_THREADS / 32) {
    const int r = w / nseg, seg = w - r * nseg;
    const int t = D == 3 ? r / L.n[1] + 1 : r + 1, j = D == 3 ? r - (t - 1) * L.n[1] + 1 : 0;
    double acc = 0.0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = seg * TILE_X + 2 * lane + 1 + h;
      if (i <= L.n[0]) {
        ChainCell<double, D> C;
        C.c = chain_idx<D>(L, i, j, t);
        chain_nb<double, D>(L, S, i, j, t, C);
        chain_fetch<double, D, false>(L, C);
        Problem::Stencil<double, D> s;
        chain_stencil<double, D>(L, C, 0u, s);
        double o0, o1;
        chain_operator<double, D, false>(L, s, 0.0, o0, o1);
        const double r0 = C.f0 - o0, r1 = C.f1 - o1;
        acc += r0 * r0 + r1 * r1;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      const int row = (S.lo + t - 2) * (D == 3 ? L.n[1] : 1) + (D == 3 ? j - 1 : 0);
      chain_st_cluster(chain_map_rank(sums + 8u * (uint32_t)(row * nseg + seg), 0), acc);
    }
  }
  if (X.PL->nslab > 0) chain_cluster_sync();
  else __syncthreads();
  double total = 0.0;
  if (X.rank == 0) {
    const int nz = D == 3 ? L.ns : 1, ty = (ny + TILE_Y - 1) / TILE_Y;
    double s = 0.0;
    if (threadIdx.x < BLOCK_THREADS)
      for (int b = threadIdx.x; b < nseg * ty * nz; b += BLOCK_THREADS) {
        const int seg = b % nseg, y = (b / nseg) % ty, z = b / (nseg * ty);
        double tile = 0.0;
#pragma unroll
        for (int k = 0; k < TILE_Y; ++k) {
          const int j = y * TILE_Y + k;
          tile += j < ny ? chain_ld(sums + 8u * (uint32_t)((z * ny + j) * nseg + seg), 0.0) : 0.0;
        }
        s += tile;
      }
    __shared__ double red[BLOCK_THREADS / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0 && warp < BLOCK_THREADS / 32) red[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 0; w < BLOCK_THREADS / 32; ++w) total += red[w];
  }
  return total;
}

// The top level from global memory into this CTA's slab: q with ghosts and halo
// rows, f and the base inside.
template <class T, int D>
__device__ __forceinline__ void chain_load_top(const DevPatch& G, const ChainLevel& L,
                                               const ChainSlab& S) {
  using V = typename ChainV<T>::V;
  const int64_t gs = D == 2 ? G.sy : G.sz;
  const int ex = L.n[0] + 2, ey = D == 3 ? L.n[1] + 2 : 1;
  auto copy = [&](uint32_t dst, const T* s0, const T* s1, int rows, int first) {
    const int total = ex * ey * rows;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      const int r = e / ex, i = e - r * ex;
      const int t = D == 3 ? r / ey : r, j = D == 3 ? r - t * ey : 0;
      const int64_t g = i + (D == 3 ? j * G.sy : 0) + (first + t) * gs;
      const int c = i + j * L.pitch + t * L.sstr;
      if (s1) {
        V v;
        v.x = s0[g];
        v.y = s1[g];
        chain_st(chain_byte<T>(dst, c), v);
      } else {
        chain_st(dst + (uint32_t)c * (uint32_t)sizeof(T), s0[g]);
      }
    }
  };
  copy(L.q, fld<T>(G.q[0]), fld<T>(G.q[1]), S.nr + 2, S.lo - 1);
  copy(L.f, fld<T>(G.f[0]), fld<T>(G.f[1]), S.nr, S.lo);
  if (L.delta) copy(L.bs, fld<T>(G.bs), (const T*)nullptr, S.nr, S.lo);
}

// A level's slab to global memory: q with the ghosts that SetBC gives it (face
// maps in ascending dimension), and f inside.
template <class T, int D>
__device__ __forceinline__ void chain_store(const DevPatch& G, const ChainLevel& L,
                                            const ChainSlab& S, bool with_f) {
  const int64_t gs = D == 2 ? G.sy : G.sz;
  const int ex = L.n[0] + 2, ey = D == 3 ? L.n[1] + 2 : 1;
  // The level's own ghost rows belong to its first and last slab.
  const int t0 = S.lo == 1 ? 0 : 1, t1 = S.lo + S.nr - 1 == L.ns ? S.nr + 1 : S.nr;
  using V = typename ChainV<T>::V;
  // The cell that ghost coordinate x of an extent n takes, and its map.
  auto source = [](int x, int n, int lo, int hi, int& code) {
    code = x == 0 ? lo : (x == n + 1 ? hi : (int)BC_COPY);
    if (x >= 1 && x <= n) return x;
    return (x == 0) == (code == BC_PERIODIC) ? n : 1;
  };
  for (int e = threadIdx.x; e < ex * ey * (t1 - t0 + 1); e += blockDim.x) {
    const int i = e % ex, r = e / ex;
    const int j = D == 3 ? r % ey : 0, t = t0 + (D == 3 ? r / ey : r);
    int cx, cy = BC_COPY, ct = BC_COPY;
    const int si = source(i, L.n[0], L.bc[0], L.bc[1], cx);
    const int sj = D == 3 ? source(j, L.n[1], L.bc[2], L.bc[3], cy) : 0;
    int st = t;  // a halo slot fed by another CTA holds the row itself
    if ((t == 0 && S.lo_r < 0) || (t == S.nr + 1 && S.hi_r < 0))
      st = source(t, S.nr, L.bc[2 * D - 2], L.bc[2 * D - 1], ct);
    const int c = chain_idx<D>(L, si, sj, st);
    auto m = [&](T v) { return chain_map<T>(ct, chain_map<T>(cy, chain_map<T>(cx, v))); };
    const int64_t g = i + (D == 3 ? j * G.sy : 0) + (S.lo - 1 + t) * gs;
    const V q = chain_ld(chain_byte<T>(L.q, c), V{});
    fld<T>(G.q[0])[g] = m(q.x);
    fld<T>(G.q[1])[g] = m(q.y);
    if (with_f && i >= 1 && i <= L.n[0] && t >= 1 && t <= S.nr &&
        (D == 2 || (j >= 1 && j <= L.n[1]))) {
      const V f = chain_ld(chain_byte<T>(L.f, c - L.sstr), V{});
      fld<T>(G.f[0])[g] = f.x;
      fld<T>(G.f[1])[g] = f.y;
    }
  }
}

// A cluster of ctas CTAs per chain (one CTA when no level is cut).
// MIXED: the levels are correction-form levels (FP32 or FP64), else FP64.
template <int D, bool MIXED>
__global__ void __launch_bounds__(CHAIN_THREADS, 1)
    k_chain(const DevPatch* __restrict__ PT, const ChainPlan* __restrict__ plans, ChainLoop loop) {
  after_previous();
  __shared__ ChainPlan PL;
  __shared__ ChainSlab slabs[CHAIN_MAX_LEVELS];
  __shared__ int again;
  int rank, ctas;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ctas));
  const ChainPlan* plan = plans + blockIdx.x / ctas;
  for (int w = threadIdx.x; w < (int)(sizeof(ChainPlan) / 4); w += CHAIN_THREADS)
    reinterpret_cast<uint32_t*>(&PL)[w] = reinterpret_cast<const uint32_t*>(plan)[w];
  __syncthreads();
  if ((int)threadIdx.x < PL.nlev) {
    ChainLevel& L = PL.L[threadIdx.x];
    L.q += chain_base();
    L.f += chain_base();
    L.qs += chain_base();
    L.bs += chain_base();
    if (threadIdx.x == 0) PL.rsum += chain_base();
    slabs[threadIdx.x] = chain_slab<D>(L, rank);
  }
  __syncthreads();
  const ChainCtx X{&PL, slabs, rank};
  const DevPatch& G = PT[PL.L[0].patch];
  if (rank < PL.L[0].active) {
    if (MIXED && PL.L[0].prec == PREC_F32) chain_load_top<float, D>(G, PL.L[0], slabs[0]);
    else chain_load_top<double, D>(G, PL.L[0], slabs[0]);
  }
  chain_cluster_sync();  // every CTA of the cluster runs: its memory may be written
  int it = 0;
  for (;;) {
    chain_vcycle<D, MIXED>(X, it == 0);
    if (loop.maxv == 0) break;
    const double total = chain_resid<D>(X);
    ++it;
    if (rank == 0 && threadIdx.x == 0) {
      const double r = sqrt(total / loop.denom);
      loop.trace[it - 1] = r;
      const bool conv = r < loop.tol;
      const int go = !conv && it < loop.maxv && isfinite(r) ? 1 : 0;
      const uint32_t flag = (uint32_t)__cvta_generic_to_shared(&again);
      for (int c = 0; c < ctas; ++c)
        asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(chain_map_rank(flag, c)), "r"(go)
                     : "memory");
      if (!go) {
        loop.st->sumsq = total;
        loop.st->residual = r;
        loop.st->converged = conv ? 1 : 0;
        loop.st->iters = it;
      }
    }
    chain_cluster_sync();
    if (!*(volatile int*)&again) break;
  }
  // The fields go back to global memory: the top's state, and in the FP64
  // form every level's state and right-hand side, which a caller may read.
  for (int l = 0; l < (MIXED ? 1 : PL.nlev); ++l) {
    if (rank >= PL.L[l].active) continue;
    const DevPatch& W = PT[PL.L[l].patch];
    if (MIXED && PL.L[l].prec == PREC_F32) chain_store<float, D>(W, PL.L[l], slabs[l], false);
    else chain_store<double, D>(W, PL.L[l], slabs[l], l > 0);
  }
  chain_cluster_sync();  // no CTA leaves while another may still read its memory
}

// ---- chains of a batch, a CTA each ---------------------------------------------------

// Lays out the FP64 chain from record `top` down its parent links in this CTA's
// shared memory, as chain_layout does for one CTA, and fills in the records'
// faces and constants; a level per lane of the first warp.  (From the host it
// would be 2 KB for every problem admitted.)
template <int D, bool DELTA>
__device__ __forceinline__ void chain_plan(const DevPatch* __restrict__ PT, int top, int nu,
                                           ChainPlan& PL, ChainSlab* slabs) {
  if (threadIdx.x >= 32) return;
  const int l = threadIdx.x;
  int p = l < CHAIN_MAX_LEVELS ? top : -1;
  for (int s = 0; s < l && p >= 0; ++s) p = PT[p].parent;
  const unsigned levels = __ballot_sync(0xffffffffu, p >= 0);
  const DevPatch& P = PT[max(p, 0)];
  const int n0 = P.n[0], n1 = P.n[1], ns = P.n[D - 1];
  const int pitch = n0 + 2, sstr = D == 3 ? pitch * (n1 + 2) : pitch;
  const uint32_t q = 16u * (uint32_t)((ns + 2) * sstr), f = 16u * (uint32_t)(ns * sstr);
  const uint32_t b = DELTA ? (8u * (uint32_t)(ns * sstr) + 15u) / 16u * 16u : 0u;
  const uint32_t mine = p >= 0 ? q + f + (l > 0 ? q : 0u) + b : 0u;
  uint32_t end = mine;
#pragma unroll
  for (int o = 1; o < 32; o *= 2) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, end, o);
    if (l >= o) end += x;
  }
  if (l == 0) {
    PL.nlev = __popc(levels);
    PL.nslab = 0;
    PL.nu = nu;
    PL.ctas = 1;
  }
  if (p < 0) return;
  ChainLevel& L = PL.L[l];
  L.patch = p;
  L.n[0] = n0;
  L.n[1] = n1;
  L.n[2] = P.n[2];
  L.ns = ns;
  L.pitch = pitch;
  L.sstr = sstr;
  L.prec = PREC_F64;
  L.delta = DELTA ? 1 : 0;
  int maps = 0;
#pragma unroll
  for (int face = 0; face < 6; ++face) {
    const int code = P.bc[face];
    L.bc[face] = code;
    if (face < 2 * D && (code == BC_REFLECT || code == BC_NEGATE)) maps = 1;
  }
  L.maps = maps;
  auto magic = [](uint32_t d) { return d == 1u ? 0u : 0xffffffffu / d + 1u; };
  L.w = (uint32_t)max(1, n0 / 2);
  L.h = (uint32_t)(D == 3 ? max(1, n1 / 2) : 1);
  L.mw = magic(L.w);
  L.mh = magic(L.h);
  L.active = 1;
  L.units = ns % 2 ? ns : ns / 2;
  L.q = chain_base() + end - mine;
  L.f = L.q + q;
  L.qs = l > 0 ? L.f + f : 0u;
  L.bs = L.f + f + (l > 0 ? q : 0u);
  L.tmp1 = P.tmp1;
  L.tmp2 = P.tmp2;
  L.tmp3 = P.tmp3;
  L.alpha = P.alpha;
  ChainSlab S{};
  S.lo = 1;
  S.nr = ns;
  S.lo_r = S.hi_r = -1;
  slabs[l] = S;
}

// AFASVcycle of bottom chains that fit in a CTA's shared memory, a CTA per chain
// at a time.  DELTA: correction-form levels.  all: every level's fields go back
// to global memory, not only the top's state.
// In global memory (bottom.cuh) a chain is some 60 phases of about 1.4 us each
// whose loads wait on L2: 96 chains of 32^2 and below took 85 us, now 41; 24 of
// 8^3 and below 128, now 41; 512 of 32^2 in correction form, two CTAs of 256
// threads per SM in two waves, 127, now 96.
constexpr int BATCH_CHAIN_THREADS = 256;
template <int D, bool DELTA>
__global__ void __launch_bounds__(BATCH_CHAIN_THREADS, 2)
    kb_chain(const DevPatch* __restrict__ PT, const Item* __restrict__ tops,
             const int* __restrict__ count, int nu, int all) {
  __shared__ ChainPlan PL;
  __shared__ ChainSlab slabs[CHAIN_MAX_LEVELS];
  const int n = *count;
  for (int b = blockIdx.x; b < n; b += gridDim.x) {
    const int top = tops[b].patch;
    if (!PT[top].active) continue;  // uniform per CTA
    __syncthreads();  // the previous chain's memory is no longer read
    chain_plan<D, DELTA>(PT, top, nu, PL, slabs);
    __syncthreads();
    chain_load_top<double, D>(PT[top], PL.L[0], slabs[0]);
    __syncthreads();
    const ChainCtx X{&PL, slabs, 0};
    for (int l = 0; l < PL.nlev; ++l)
      chain_visit_t<double, double, D, DELTA, false>(X, l, false, l == 0);
    for (int l = PL.nlev - 2; l >= 0; --l)
      chain_visit_t<double, double, D, DELTA, false>(X, l, true, false);
    for (int l = 0; l < (all ? PL.nlev : 1); ++l)
      chain_store<double, D>(PT[PL.L[l].patch], PL.L[l], slabs[l], l > 0);
  }
}

// ---- host side -------------------------------------------------------------------

constexpr size_t CHAIN_SMEM_MAX = 227 * 1024 - 4096;  // dynamic; the rest holds the plan

// Lays out the chain of levels of extents n[l] (top first; n[l][2] = 1 in 2D,
// each half of the one before) with value types prec[l] in the shared memory of
// at most max_ctas CTAs.  loop: with room for the residual's row sums.  Returns
// false when it does not fit.  Patches, faces and constants are the caller's
// to fill in (chain_faces).
inline bool chain_layout(int nd, const std::vector<std::array<int, 3>>& n,
                         const std::vector<int>& prec, bool delta, int nu, int max_ctas,
                         bool loop, ChainPlan& C) {
  C = ChainPlan{};
  const int nl = (int)n.size();
  if (nl < 1 || nl > CHAIN_MAX_LEVELS) return false;
  auto cells = [&](int l) { return (int64_t)n[l][0] * n[l][1] * n[l][2]; };
  C.nlev = nl;
  C.nu = nu;
  const int slow = nd - 1;
  if (cells(0) > CHAIN_SINGLE_CELLS && max_ctas > 1)
    while (C.nslab < nl && cells(C.nslab) > CHAIN_TAIL_CELLS) ++C.nslab;
  C.ctas = 1;
  int64_t off = 0;
  auto place = [&](int64_t bytes) {
    const int64_t at = off;
    off += (bytes + 15) / 16 * 16;
    return (uint32_t)std::min<int64_t>(at, UINT32_MAX);
  };
  auto magic = [](uint32_t d) {
    return d == 1 ? 0u : (uint32_t)(((uint64_t(1) << 32) + d - 1) / d);
  };
  for (int l = 0; l < nl; ++l) {
    ChainLevel& L = C.L[l];
    for (int d = 0; d < 3; ++d) L.n[d] = n[l][d];
    for (int d = 0; d < nd; ++d) {
      if (l + 1 < nl && n[l][d] != 2 * n[l + 1][d]) return false;
    }
    L.ns = n[l][slow];
    L.prec = prec[l];
    L.delta = delta ? 1 : 0;
    L.w = (uint32_t)std::max(1, n[l][0] / 2);
    L.h = (uint32_t)(nd == 3 ? std::max(1, n[l][1] / 2) : 1);
    L.mw = magic(L.w);
    L.mh = magic(L.h);
    L.units = L.ns % 2 ? L.ns : L.ns / 2;
    L.active = l < C.nslab ? std::min(max_ctas, L.units) : 1;
    while (C.ctas < L.active) C.ctas *= 2;
    const int64_t pitch = n[l][0] + 2, sstr = nd == 3 ? pitch * (n[l][1] + 2) : pitch;
    if (sstr > (int64_t)CHAIN_SMEM_MAX) return false;
    L.pitch = (int)pitch;
    L.sstr = (int)sstr;
    const int64_t rows =
        (int64_t)((L.units + L.active - 1) / L.active) * (L.ns % 2 ? 1 : 2);
    const int64_t es = prec[l] == PREC_F32 ? 4 : 8;
    L.q = place(2 * (rows + 2) * sstr * es);
    L.f = place(2 * rows * sstr * es);
    L.qs = l > 0 ? place(2 * (rows + 2) * sstr * es) : 0;
    L.bs = delta ? place(rows * sstr * es) : 0;
    if (off > (int64_t)CHAIN_SMEM_MAX) return false;
  }
  if (loop) {
    const int64_t rows = (int64_t)n[0][1] * n[0][2];
    C.rsum = place(8 * rows * ((n[0][0] + TILE_X - 1) / TILE_X));
    if (off > (int64_t)CHAIN_SMEM_MAX) return false;
  }
  C.smem = (uint32_t)off;
  return true;
}

// Level l's record, faces and constants.
inline void chain_faces(ChainPlan& C, int l, int record, const DevPatch& P) {
  ChainLevel& L = C.L[l];
  L.patch = record;
  for (int f = 0; f < 6; ++f) {
    L.bc[f] = P.bc[f];
    if (f < 2 * P.ndims && (P.bc[f] == BC_REFLECT || P.bc[f] == BC_NEGATE)) L.maps = 1;
  }
  L.tmp1 = P.tmp1;
  L.tmp2 = P.tmp2;
  L.tmp3 = P.tmp3;
  L.alpha = P.alpha;
}

}  // namespace bsam
