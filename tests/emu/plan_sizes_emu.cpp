// The expert-plan kernels at sizes that plan_emu.cpp does not have, with its checks: more pairs than a CTA's threads keep between
// counting and placing, eight rows per CTA, and tiles of 256 rows, which share an expert's rows evenly.
//   g++ -std=c++20 -O1 -pthread -DB200_EMU -I tests/emu -x c++ tests/emu/plan_sizes_emu.cpp -o plan_sizes_emu
#define main plan_emu_main
#include "plan_emu.cpp"
#undef main

#include <tuple>

// Tiles of 256 rows: as few as hold the expert's rows, shared evenly in steps of 32. Looked over here, then written over with full
// tiles for the checks of everything else.
static int check_any(const char* what, const std::vector<int>& idx, int Et, int bt, int P, Plan p, int max_tiles, bool want_err) {
  int bad = 0, ti = 0;
  if (bt == 256)
    for (int e = 0; e < Et; ++e) {
      const int c = p.offsets[e + 1] - p.offsets[e], few = (c + bt - 1) / bt, step = few > 1 ? (c + 32 * few - 1) / (32 * few) * 32 : bt;
      for (int i = 0; i < few && ti < max_tiles; ++i, ++ti) {
        const int4 t = p.tiles[ti];
        if (t.x != e || t.y != p.offsets[e] + i * step || t.z <= 0 || t.z != std::min(step, c - i * step)) {
          std::printf("%s: tile %d of expert %d\n", what, ti, e);
          ++bad;
        }
        p.tiles[ti].y = p.offsets[e] + i * bt;
        p.tiles[ti].z = std::min(bt, c - i * bt);
      }
    }
  return bad + check(what, idx, Et, bt, P, p, max_tiles, want_err);
}

int main() {
  constexpr int E = 256, K = 8, P = K + 1, Et = E + 1, PER_LANE = 8, KEPT = 5 * 1024;
  std::mt19937 rng(6);
  std::normal_distribution<float> nd(0.f, 1.f);
  int bad = 0;

  // one CTA, half of the pairs at one expert, some served elsewhere, two bad indexes
  for (auto [n_pairs, bt] : {std::pair{KEPT, 16}, {KEPT + 1, 32}, {9300, 256}}) {
    const int max_tiles = 900;
    std::vector<int> idx(n_pairs);
    for (int i = 0; i < n_pairs; ++i) idx[i] = i % 2 ? std::max(-1, static_cast<int>(rng() % (Et + 40)) - 40) : E;
    for (int pass = 0; pass < 2; ++pass) {
      if (pass == 1) idx[1234] = idx[n_pairs - 1] = Et + 3;
      Plan p(Et, n_pairs, max_tiles);
      run_cta(1024, 0, 0, [&] {
        moe_plan_kernel(idx.data(), n_pairs, Et, bt, p.offsets.data(), p.tiles.data(), &p.n_tiles, max_tiles, p.perm.data(),
                        p.inv.data(), &p.err, P, p.src_rows.data());
      });
      bad += check_any(pass ? "plan (bad indexes)" : "plan", idx, Et, bt, P, p, max_tiles, pass == 1);
    }
  }

  // the grid forms with eight and 32 rows per CTA
  for (auto [T, bt, per_cta] : {std::tuple{97, 16, 8}, {280, 256, 32}}) {
    std::vector<float> logits(T * (E + 1));
    for (auto& v : logits) v = nd(rng) * 2.f;
    const int n_pairs = T * P, max_tiles = std::min(Et, n_pairs) + n_pairs / bt + 1;
    std::vector<float> wts(n_pairs);
    for (int with_work = 0; with_work < 2; ++with_work) {
      std::vector<int> idx(n_pairs, -5), work(2 * 1024, 0);
      unsigned ticket = 0;
      Plan p(Et, n_pairs, max_tiles);
      gridDim.x = (T + per_cta - 1) / per_cta;
      for (unsigned bx = 0; bx < gridDim.x; ++bx)
        run_cta(1024, bx, 0, [&] {
          moe_route_plan_grid_kernel<PER_LANE>(logits.data(), E + 1, T, E, K, 1, wts.data(), idx.data(), nullptr, Et, bt,
                                               p.offsets.data(), p.tiles.data(), &p.n_tiles, max_tiles, p.perm.data(), p.inv.data(),
                                               &p.err, p.src_rows.data(), &ticket, with_work ? work.data() : nullptr);
        });
      if (with_work) {
        gridDim.x = 3;
        for (unsigned bx = 0; bx < gridDim.x; ++bx)
          run_cta(256, bx, 0, [&] {
            moe_scatter_kernel(idx.data(), n_pairs, Et, p.offsets.data(), work.data() + 1024, p.perm.data(), p.inv.data(), &p.err, P,
                               p.src_rows.data());
          });
      }
      bad += check_any(with_work ? "grid route + scan, then scatter" : "grid route, last CTA plans", idx, Et, bt, P, p, max_tiles, false);
      if (ticket != 0) { std::printf("the ticket word was not put back to zero\n"); ++bad; }
    }
  }
  if (bad) return 1;
  std::printf("OK expert plan: more pairs than kept, eight rows per CTA, even tiles of 256 rows\n");
  return 0;
}
