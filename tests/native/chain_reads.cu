// Replays on the host which shared-memory addresses the chain kernel's threads
// form for their pairs of cells (chain_slab, chain_pair, chain_nb of chain.cuh), for
// every CTA and level of a chain, and checks that each lies in the level's own
// field: no CUDA call is made.  Prints the number of chains seen, the number that
// have a CTA without rows on a paired level under a periodic last dimension, and
// the number of chains with an address out of range.
#include <cstdio>
#include <cstdlib>

#include "chain.cuh"

using namespace bsam;

template <class T, int D>
static bool in_field(const ChainLevel& L, int rows, uint32_t at) {
  const int64_t size = (int64_t)(rows + 2) * L.sstr * (int64_t)sizeof(typename ChainV<T>::V);
  return at >= L.q && at + sizeof(typename ChainV<T>::V) <= L.q + (uint64_t)size;
}

template <class T, int D>
static bool pair_ok(const ChainLevel& L, const ChainSlab& S, int rows, int idx) {
  ChainPair<T, D> R;
  chain_pair<T, D>(L, S, idx, R);
  bool ok = true;
  for (int cell = 0; cell < 2; ++cell)
    for (int raw = 0; raw < 3; ++raw) {  // as mapped, first pass, second pass
      ChainCell<T, D> X = cell ? R.B : R.A;
      if (raw) chain_nb_raw<T, D>(L, raw == 1, X);
      ok = ok && in_field<T, D>(L, rows, chain_byte<T>(L.q, X.c));
      for (int k = 0; k < 2 * D; ++k) ok = ok && in_field<T, D>(L, rows, X.at[k]);
      const int64_t f = X.c - L.sstr;  // right-hand side and base have no halo row
      ok = ok && f >= 0 && f < (int64_t)rows * L.sstr;
    }
  return ok;
}

struct Tally {
  long chains = 0, idle = 0, bad = 0;
};

// The chain from extents n down to the coarsest level, one form and face rule.
template <int D>
static void replay(const int (&n)[3], int prec_top, bool delta, const int (&bc)[6], bool loop,
                   int max_ctas, bool all_pairs, Tally& t) {
  std::vector<std::array<int, 3>> ext;
  std::vector<int> prec;
  std::array<int, 3> e{n[0], n[1], D == 3 ? n[2] : 1};
  for (;;) {
    ext.push_back(e);
    prec.push_back((int64_t)e[0] * e[1] * e[2] > 4096 ? prec_top : (int)PREC_F64);
    bool even = true;
    for (int d = 0; d < D; ++d) even = even && e[d] % 2 == 0;
    if (!even) break;
    for (int d = 0; d < D; ++d) e[d] /= 2;
  }
  for (int d = 0; d < D; ++d)  // a periodic dimension is even or 1 on every level
    if (bc[2 * d] == BC_PERIODIC && ext.back()[d] % 2 && ext.back()[d] > 1) return;
  ChainPlan C;
  if (!chain_layout(D, ext, prec, delta, 2, max_ctas, loop, C)) return;
  for (int l = 0; l < C.nlev; ++l)
    for (int f = 0; f < 6; ++f) C.L[l].bc[f] = bc[f];
  ++t.chains;
  bool idle = false, ok = true;
  for (int l = 0; l + 1 < C.nlev; ++l) {
    const ChainLevel& L = C.L[l];
    const int rows = (L.units + L.active - 1) / L.active * (L.ns % 2 ? 1 : 2);
    for (int r = 0; r < (l < C.nslab ? C.ctas : 1); ++r) {
      const ChainSlab S = chain_slab<D>(L, r);
      idle = idle || (S.nr == 0 && bc[2 * D - 1] == BC_PERIODIC);
      if (!chain_runs(S)) continue;
      const int pairs = chain_pairs<D>(L, S);
      const int step = all_pairs ? 1 : pairs > 64 ? pairs / 64 : 1;
      for (int i = 0; i < pairs; i += step)
        ok = ok && (L.prec == PREC_F32 ? pair_ok<float, D>(L, S, rows, i)
                                       : pair_ok<double, D>(L, S, rows, i));
      for (int i = pairs - 1; i < pairs + 1; ++i)  // the last pair and a thread without one
        ok = ok && (L.prec == PREC_F32 ? pair_ok<float, D>(L, S, rows, i)
                                       : pair_ok<double, D>(L, S, rows, i));
    }
  }
  t.idle += idle;
  if (!ok) {
    ++t.bad;
    if (t.bad <= 10) std::fprintf(stderr, "out of range: %d x %d x %d\n", n[0], n[1], n[2]);
  }
}

int main() {
  Tally t;
  auto faces = [](int x, int last, int nd, int (&bc)[6]) {
    for (int f = 0; f < 6; ++f) bc[f] = BC_NONE;
    for (int f = 0; f < 2 * nd; ++f) bc[f] = BC_REFLECT;
    if (x) bc[0] = bc[1] = BC_PERIODIC;
    if (last) bc[2 * nd - 2] = bc[2 * nd - 1] = BC_PERIODIC;
  };
  for (int px = 0; px < 2; ++px)
    for (int pl = 0; pl < 2; ++pl)
      for (int ctas : {16, 8}) {
        int bc[6];
        faces(px, pl, 2, bc);
        for (int a = 2; a <= 512; a += 2)
          for (int b = 2; b <= 256; b += 2) {
            const int n[3] = {a, b, 1};
            const bool all = a * b < 256 || (a % 34 == 0 && b % 26 == 0);
            replay<2>(n, PREC_F64, false, bc, true, ctas, all, t);
            if ((a + b) % 8 == 0) replay<2>(n, PREC_F32, true, bc, false, ctas, all, t);
          }
        faces(px, pl, 3, bc);
        for (int a = 2; a <= 40; a += 2)
          for (int b = 2; b <= 40; b += 2)
            for (int c = 2; c <= 64; c += 2) {
              const int n[3] = {a, b, c};
              replay<3>(n, PREC_F64, false, bc, true, ctas, false, t);
              if ((a + b + c) % 8 == 0) replay<3>(n, PREC_F32, true, bc, false, ctas, false, t);
            }
      }
  std::printf("%ld %ld %ld\n", t.chains, t.idle, t.bad);
  return t.bad != 0;
}
