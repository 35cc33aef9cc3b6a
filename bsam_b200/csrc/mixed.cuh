// mixed.cuh -- FP64 outer loop around an FP32 FAS V-cycle in correction form.
//
// The mixed form keeps an FP64 master of the finest level (q64, f64).  Each
// V-cycle solves for a correction e of q64 on the "twin" patch and the
// levels below it, which hold FP32 values (small levels FP64):
//
//   r64  = f64 - L64(q64)                    FP64 defect (+ its L2 norm)
//   e    = 0,  base = fl32(phi64),  g = fl32(r64)
//   e   <- FAS V-cycle on  L(base + e) - L(base) = g
//   q64 += e                                  FP64 update
//
// Written for the correction, the inner operator's nonlinear part is
// Dfc(base + e) - Dfc(base) = alpha e (3c^2 + 3ce + e^2) (problem_ch.cuh,
// DfcDelta) and every other term is linear in e, so FP32 rounding scales with
// the correction, not with q; the defect enters the FP32 cycle with its full
// relative precision.  The FAS recursion applies unchanged to e, with each
// level's base restricted from the finer one.  Convergence is judged on the
// FP64 defect of q64, exactly as MultigridIterations judges the FP64 form
// (afas:94-101).
#pragma once
#include "kernels.cuh"

namespace bsam {

// Defect of one master tile by one warp: ErrorAFAS of q64 (the same norm as
// k_resid_norm) plus the twin's start (e = 0), base and right-hand side.
// Returns the tile's sum of squares in lane 0.  zero: e = 0 is stored (a batch's
// fused stage starts from it without reading it).
template <class TW, int D>
__device__ __forceinline__ double defect_rows(const DevPatch& M, const DevPatch& W, const Item it,
                                              bool zero) {
  using V = typename PairOf<TW>::V;
  TW* e0 = fld<TW>(W.q[0]);
  TW* e1 = fld<TW>(W.q[1]);
  TW* f0 = fld<TW>(W.f[0]);
  TW* f1 = fld<TW>(W.f[1]);
  TW* bs = fld<TW>(W.bs);
  return resid_rows<D>(
      M, it, [&](int i, int j, int k, bool two, double2 r0, double2 r1, double2 q) {
        const int64_t c = cidx(W, i, j, k);
        if (two) {
          auto put = [&](TW* p, TW x, TW y) { *reinterpret_cast<V*>(p + c) = V{x, y}; };
          put(f0, TW(r0.x), TW(r0.y));
          put(f1, TW(r1.x), TW(r1.y));
          put(bs, TW(q.x), TW(q.y));
          if (zero) {
            put(e0, TW(0), TW(0));
            put(e1, TW(0), TW(0));
          }
        } else {
          f0[c] = TW(r0.x);
          f1[c] = TW(r1.x);
          bs[c] = TW(q.x);
          if (zero) e0[c] = e1[c] = TW(0);
        }
        if (!zero || !W.wt) return;
        // Ghosts across the faces; those across two or three are not read here (no
        // patch has its parent on the finest level).
        auto ghost = [&](int64_t g, int code, bool pair) {
          const TW z = bc_map<TW>(code, TW(0));
          e0[g] = e1[g] = z;
          if (pair) e0[g + 1] = e1[g + 1] = z;
        };
        if (i == 1) ghost(c - 1, W.bc[0], false);
        if (i + (int)two == W.n[0]) ghost(c + 1 + (int)two, W.bc[1], false);
        if (j == 1) ghost(c - W.sy, W.bc[2], two);
        if (j == W.n[1]) ghost(c + W.sy, W.bc[3], two);
        if (D == 3) {
          if (k == 1) ghost(c - W.sz, W.bc[4], two);
          if (k == W.n[2]) ghost(c + W.sz, W.bc[5], two);
        }
      });
}

// q64 += e on one work tile of a twin; ghosts by write-through.
template <class TW, int D>
__device__ __forceinline__ void update_item(const DevPatch* __restrict__ PT, const Item it) {
  const DevPatch W = PT[it.patch];
  const DevPatch M = PT[W.master];
  if (!M.active) return;
  const WorkPlace<D> w(it, M.n[0]);
  if (w.j > M.n[1]) return;
  double* q0 = fld<double>(M.q[0]);
  double* q1 = fld<double>(M.q[1]);
  const TW* e0 = fld<TW>(W.q[0]);
  const TW* e1 = fld<TW>(W.q[1]);
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int i = w.a0 + t * w.W;
    if (i > M.n[0]) break;
    const int64_t c = cidx(M, i, w.j, w.k), cw = cidx(W, i, w.j, w.k);
    const double na = q0[c] + (double)e0[cw];
    const double nb = q1[c] + (double)e1[cw];
    q0[c] = na;
    q1[c] = nb;
    if (M.wt && near_boundary(M, i, w.j, w.k, D))
      write_through<double, D>(M, q0, q1, i, w.j, w.k, na, nb);
  }
}

// Defect kernel over the masters' tiles, with the FP64 norm in d_status.
template <class TW, int D>
__global__ void __launch_bounds__(BLOCK_THREADS, 4)
    k_defect(const DevPatch* __restrict__ PT, const Item* __restrict__ items,
             double* __restrict__ partials, DevStatus* __restrict__ st, int nitems,
             double denom, double tol) {
  after_previous();
  const int b = blockIdx.x * TILE_Y + threadIdx.y;  // a tile per warp
  if (b < nitems) {
    const Item it = items[b];
    const DevPatch& M = PT[it.patch];
    const double s = defect_rows<TW, D>(M, PT[M.twin], it, true);
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

template <class TW, int D>
__global__ void __launch_bounds__(BLOCK_THREADS)
    k_update(const DevPatch* __restrict__ PT, const Item* __restrict__ items) {
  after_previous();
  update_item<TW, D>(PT, items[blockIdx.x]);
}

}  // namespace bsam
