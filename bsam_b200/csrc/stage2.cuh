// stage2.cuh -- a whole 2D smoothing stage of a single problem's level, with the
// transfer that belongs to it, in one launch.
//
// A level of a single 2D problem that is too large for one cluster's shared
// memory (chain.cuh) has some 10^4 to 10^6 cells: its passes as launches are
// bound by launch latency (5.3 us each from 100^2 to 512^2).  Here a CTA holds a
// tile of TX x TY cells with a halo of 4 in shared memory and runs all colour
// passes of the stage there -- pass p on the tile grown by 2 nu - 1 - p cells --
// then stores the tile.  Halo cells are recomputed from the same inputs as in
// their own tile, so every value is that of the per-pass kernels, bit for bit.
//   dir 0 (q -> qb): the stage before the coarse correction, then
//          RestrictSolution of the tile's coarse cells into the parent
//   dir 1 (qb -> q): CorrectFine of the tile as it is loaded, then the stage;
//          in the mixed form's finest level the result is added to the FP64
//          master instead of being stored (update_item)
// Neighbours across a physical face are read as the face's map of the cell
// itself; a periodic dimension's halo wraps around.
//
// Bound by latency: 250 CTAs of four dependent passes on a 320 x 200 FP64
// level take 9.0 us, where its 5 launches (four passes and the transfer) took
// 27; 512^2 FP32 12.5 us with the update of the master, where 6 launches took
// 33.  A V-cycle of 320 x 200 went from 98 to 73 us and of 512^2 mixed from 190
// to 140.  Tiles are small (the batch's fused stage uses 56 x 16 or 56 x 32)
// because a level gives each SM one or a few of them: the time of one CTA
// counts, not the halo's share.
#pragma once
#include "kernels.cuh"

namespace bsam {

template <class T> struct Stage2V;
template <> struct Stage2V<float> { using V = float2; };
template <> struct Stage2V<double> { using V = double2; };

template <class T, bool DELTA, int TY_> struct Stage2 {
  static constexpr int TX = 32, TY = TY_, H = 4;
  static constexpr int W = TX + 2 * H, R = TY + 2 * H;
  static constexpr int THREADS = 256;
  static constexpr size_t SMEM = sizeof(T) * (DELTA ? 5 : 4) * W * R;
};

// Change of the coarse solution prolongated to fine cell (I, J): correct_cell's
// expression.
template <class TP>
__device__ __forceinline__ void stage2_correction(const DevPatch& C, const DevPatch& P, int I,
                                                  int J, TP (&corr)[2]) {
  const int m = I >> 1, n = J >> 1;
  const bool ex = (I & 1) == 0, ey = (J & 1) == 0;
  const int64_t c = cidx(P, C.off[0] + m, C.off[1] + n, 0);
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    const TP* pq = fld<TP>(P.q[v]) + c;
    const TP* ps = fld<TP>(P.qs[v]) + c;
    auto e = [&](int64_t o) { return pq[o] - ps[o]; };
    const TP b0 = lin_x<TP>(ex, e(0), e(1));
    const TP b1 = lin_x<TP>(ex, e(P.sy), e(P.sy + 1));
    corr[v] = lin_x<TP>(ey, b0, b1) / TP(16);
  }
}

// blockIdx = tile.  The level is one patch, all faces physical or periodic
// (periodic extents even).  upd: the patch has an FP64 master to update.
template <class T, bool DELTA, int TY>
__global__ void __launch_bounds__(256)
    k_stage2(const DevPatch* __restrict__ PT, int patch, int dir, int nu, int upd) {
  after_previous();
  using S = Stage2<T, DELTA, TY>;
  using V = typename Stage2V<T>::V;
  extern __shared__ __align__(16) unsigned char stage2_raw[];
  V* sq = reinterpret_cast<V*>(stage2_raw);
  V* sf = sq + S::W * S::R;
  T* sb = reinterpret_cast<T*>(sf + S::W * S::R);
  const DevPatch P = PT[patch];
  const int n0 = P.n[0], n1 = P.n[1];
  const int gx0 = (int)blockIdx.x * S::TX + 1 - S::H, gy0 = (int)blockIdx.y * TY + 1 - S::H;
  const bool px = P.bc[0] == BC_PERIODIC, py = P.bc[2] == BC_PERIODIC;
  // The cell that tile column x (row y) holds: its own index, wrapped in a
  // periodic dimension; -1 outside the patch and its ghosts.
  auto wrap = [](int i, int n) {
    i = (i - 1) % n;
    return (i < 0 ? i + n : i) + 1;
  };
  auto col = [&](int i) { return px ? wrap(i, n0) : (i >= 0 && i <= n0 + 1 ? i : -1); };
  auto row = [&](int j) { return py ? wrap(j, n1) : (j >= 0 && j <= n1 + 1 ? j : -1); };
  const DevPatch* par = P.parent >= 0 ? PT + P.parent : nullptr;
  {
    const T* q0 = fld<T>(dir == 0 ? P.q[0] : P.qb[0]);
    const T* q1 = fld<T>(dir == 0 ? P.q[1] : P.qb[1]);
    const T* f0 = fld<T>(P.f[0]);
    const T* f1 = fld<T>(P.f[1]);
    for (int e = threadIdx.x; e < S::W * S::R; e += S::THREADS) {
      const int y = e / S::W, x = e - y * S::W;
      const int i = col(gx0 + x), j = row(gy0 + y);
      V q{}, f{};
      T b = T(0);
      if (i >= 0 && j >= 0) {
        const int64_t c = cidx(P, i, j, 0);
        q.x = q0[c];
        q.y = q1[c];
        if (i >= 1 && i <= n0 && j >= 1 && j <= n1) {
          f.x = f0[c];
          f.y = f1[c];
          if (DELTA) b = fld<T>(P.bs)[c];
          if (dir == 1 && par) {
            if (P.pprec == PREC_F32) {
              float corr[2];
              stage2_correction<float>(P, *par, i, j, corr);
              q.x = q.x + T(corr[0]);
              q.y = q.y + T(corr[1]);
            } else {
              double corr[2];
              stage2_correction<double>(P, *par, i, j, corr);
              q.x = q.x + T(corr[0]);
              q.y = q.y + T(corr[1]);
            }
          }
        }
      }
      sq[e] = q;
      sf[e] = f;
      if (DELTA) sb[e] = b;
    }
  }
  __syncthreads();
  const T tmp1 = T(P.tmp1), tmp2 = T(P.tmp2), tmp3 = T(P.tmp3), alpha = T(P.alpha);
  const int passes = 2 * nu;
  for (int p = 0; p < passes; ++p) {
    const int grow = passes - 1 - p;
    // The ghosts as the arrays hold them, where no pass of this stage has
    // rewritten them yet: before a correction the first pass of either colour
    // (a periodic ghost of the second is fed by the first).
    const bool held = dir == 0 && p < 2;
    for (int e = threadIdx.x; e < (S::W / 2) * S::R; e += S::THREADS) {
      const int y = e / (S::W / 2), x0 = 2 * (e - y * (S::W / 2));
      const int j = gy0 + y;
      const int x = x0 + ((gx0 + x0 + j + p) & 1), i = gx0 + x;
      if (x < S::H - grow || x >= S::H + S::TX + grow || y < S::H - grow ||
          y >= S::H + TY + grow)
        continue;
      if (!px && (i < 1 || i > n0)) continue;
      if (!py && (j < 1 || j > n1)) continue;
      const int c = y * S::W + x;
      const V own = sq[c];
      V w = sq[c - 1], ea = sq[c + 1], s = sq[c - S::W], n = sq[c + S::W];
      auto face = [&](int code, V& v) {
        if (held) return;  // the tile holds the ghost itself
        v.x = bc_map<T>(code, own.x);
        v.y = bc_map<T>(code, own.y);
      };
      if (!px) {
        if (i == 1) face(P.bc[0], w);
        if (i == n0) face(P.bc[1], ea);
      }
      if (!py) {
        if (j == 1) face(P.bc[2], s);
        if (j == n1) face(P.bc[3], n);
      }
      if (held && p == 0 && (px || py)) {
        // The periodic ghosts as stored (the tile's halo holds the cells).
        const int iw = px ? wrap(i, n0) : i, jw = py ? wrap(j, n1) : j;
        auto ghost = [&](int gi, int gj, V& v) {
          const int64_t g = cidx(P, gi, gj, 0);
          v.x = fld<T>(P.q[0])[g];
          v.y = fld<T>(P.q[1])[g];
        };
        if (px && iw == 1) ghost(0, jw, w);
        if (px && iw == n0) ghost(n0 + 1, jw, ea);
        if (py && jw == 1) ghost(iw, 0, s);
        if (py && jw == n1) ghost(iw, n1 + 1, n);
      }
      Problem::Stencil<T, 2> st;
      st.pc = own.x;
      st.mc = own.y;
      st.pm[0] = w.x;
      st.pp[0] = ea.x;
      st.pm[1] = s.x;
      st.pp[1] = n.x;
      st.mm[0] = w.y;
      st.mp[0] = ea.y;
      st.mm[1] = s.y;
      st.mp[1] = n.y;
      const V f = sf[c];
      V o;
      if (DELTA)
        Problem::RelaxCell<T, 2, true>(st, f.x, f.y, tmp1, tmp2, tmp3, alpha, o.x, o.y, sb[c]);
      else
        Problem::RelaxCell<T, 2>(st, f.x, f.y, tmp1, tmp2, tmp3, alpha, o.x, o.y);
      sq[c] = o;
    }
    __syncthreads();
  }
  // The tile's own cells.
  const DevPatch* M = upd && P.master >= 0 ? PT + P.master : nullptr;
  T* o0 = fld<T>(dir == 0 ? P.qb[0] : P.q[0]);
  T* o1 = fld<T>(dir == 0 ? P.qb[1] : P.q[1]);
  for (int e = threadIdx.x; e < S::TX * TY; e += S::THREADS) {
    const int y = e / S::TX, x = e - y * S::TX;
    const int i = gx0 + S::H + x, j = gy0 + S::H + y;
    if (i > n0 || j > n1) continue;
    const V v = sq[(y + S::H) * S::W + x + S::H];
    if (M) {
      double* m0 = fld<double>(M->q[0]);
      double* m1 = fld<double>(M->q[1]);
      const int64_t c = cidx(*M, i, j, 0);
      const double a = m0[c] + (double)v.x, b = m1[c] + (double)v.y;
      m0[c] = a;
      m1[c] = b;
      if (M->wt && near_boundary(*M, i, j, 0, 2))
        write_through<double, 2>(*M, m0, m1, i, j, 0, a, b);
      continue;
    }
    const int64_t c = cidx(P, i, j, 0);
    o0[c] = v.x;
    o1[c] = v.y;
    if (P.wt && near_boundary(P, i, j, 0, 2)) write_through<T, 2>(P, o0, o1, i, j, 0, v.x, v.y);
  }
  if (dir != 0 || !par) return;
  // RestrictSolution of the tile's coarse cells (restrict_cell's expressions).
  const DevPatch& Q = *par;
  auto restrict_tile = [&](auto zero) {
    using TP = decltype(zero);
    for (int e = threadIdx.x; e < (S::TX / 2) * (TY / 2); e += S::THREADS) {
      const int y = e / (S::TX / 2), x = e - y * (S::TX / 2);
      const int ic = (gx0 + S::H + 1) / 2 + x, jc = (gy0 + S::H + 1) / 2 + y;
      if (ic > P.cn[0] || jc > P.cn[1]) continue;
      const int c = (2 * y + 1 + S::H) * S::W + 2 * x + 1 + S::H;  // fine cell (2 ic, 2 jc)
      const V a = sq[c], b = sq[c - 1], d = sq[c - S::W], g = sq[c - S::W - 1];
      const TP v0 = TP(T(0.25) * (a.x + b.x + d.x + g.x));
      const TP v1 = TP(T(0.25) * (a.y + b.y + d.y + g.y));
      const int pi = P.off[0] + ic, pj = P.off[1] + jc;
      const int64_t pc = cidx(Q, pi, pj, 0);
      TP* pq0 = fld<TP>(Q.q[0]);
      TP* pq1 = fld<TP>(Q.q[1]);
      TP* ps0 = fld<TP>(Q.qs[0]);
      TP* ps1 = fld<TP>(Q.qs[1]);
      pq0[pc] = v0;
      pq1[pc] = v1;
      ps0[pc] = v0;
      ps1[pc] = v1;
      if (Q.wt && near_boundary(Q, pi, pj, 0, 2)) {
        write_through<TP, 2>(Q, pq0, pq1, pi, pj, 0, v0, v1);
        write_through<TP, 2>(Q, ps0, ps1, pi, pj, 0, v0, v1);
      }
      if (DELTA && Q.delta)
        fld<TP>(Q.bs)[pc] =
            TP(T(0.25) * (sb[c] + sb[c - 1] + sb[c - S::W] + sb[c - S::W - 1]));
    }
  };
  if (P.pprec == PREC_F32) restrict_tile(0.f);
  else restrict_tile(0.0);
}

}  // namespace bsam
