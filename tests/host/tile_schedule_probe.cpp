// The checks of schedule_probe.cpp on schedules for factors in symmetric tiles, and
// the scratch of those: y_k and x_k in rows of their own on more than one CTA per half.
//
//   tile_schedule_probe N m p nrhs slots cl
//
// (slots: 1 to 16 per item, cl: 1, 2 or 4 CTAs per half, imposed on every launch where
// a front's groups allow it)
// 1. schedule_probe.cpp's checks: the same cell solves however they are launched, the
//    output planes, no unordered access to a trace line, output region or scratch range;
// 2. the scratch of the items of one launch is disjoint, that of launches of different
//    sweeps (or, one launch per step, of different shifts) too, every item starts at
//    an even element and ends within the pool.
// Prints "ok launches=<n> imposed=<launches of that shape>" after the first check's line.
#include "internal.h"

static int g_slots = 0, g_cl = 0;
struct TilePlan : lsw::FrontPlan {
  TilePlan() {
    sym = true;
    rmin = 1;
    forced_cl.assign(4096, g_cl);
  }
};
#define FrontPlan TilePlan
#define main schedule_main
#include "schedule_probe.cpp"
#undef main
#undef FrontPlan

int main(int argc, char** argv) {
  if (argc != 7) {
    std::fprintf(stderr, "usage: tile_schedule_probe N m p nrhs slots cl\n");
    return 2;
  }
  g_slots = std::atoi(argv[5]);
  g_cl = std::atoi(argv[6]);
  if (const int rc = schedule_main(6, argv)) return rc;
  const int N = std::atoi(argv[1]), m = std::atoi(argv[2]), p = std::atoi(argv[3]), nrhs = std::atoi(argv[4]);
  std::vector<DevCell> cells = make_cells(N, m, p);
  int max_n = 0;
  for (DevCell& c : cells) {
    c.blk = SymTiles::elems(c.ny);
    max_n = std::max(max_n, std::max(c.nx, c.ny));
  }
  const long long LP = ((max_n + 7) / 8) * 8, n_dof = (long long)N * m + N - 1 + 2 * p - 1;
  int bad = 0, launches = 0, imposed = 0;
  for (bool lanes : {false, true}) {
    const Built b = build(cells, N, nrhs, lanes, LP, n_dof * n_dof, g_slots);
    // ranges by the chain that they belong to: a sweep, a shift, or the whole pool
    std::map<int, std::pair<long long, long long>> chain;
    for (const Front& f : b.fronts) {
      launches += f.item_count > 0;
      imposed += f.item_count > 0 && f.slots_cap == g_slots && f.cluster == g_cl;
      std::vector<std::pair<long long, long long>> r;
      for (int i = f.item_begin; i < f.item_begin + f.item_count; ++i) {
        const DevItem& it = b.items[i];
        const DevCell& c = cells[it.cell];
        const long long len = (long long)(c.nx + 1) * front_rpad(it.slot_count) * c.ny * (f.cluster > 1 ? 2 : 1);
        if (it.scratch_off % 2 || it.scratch_off < 0 || it.scratch_off + len > f.scratch_elems) ++bad;
        r.emplace_back(it.scratch_off, it.scratch_off + len);
        int key = -1;                      // alone on the device
        if (f.lane >= 0) key = f.lane;
        else if (!f.mixed)
          for (int s = 0; s < 4; ++s)
            if (i - f.item_begin >= f.sh_begin[s] && i - f.item_begin < f.sh_begin[s + 1]) key = 100 + s;
        if (key < 0) continue;
        auto& q = chain.emplace(key, r.back()).first->second;
        q.first = std::min(q.first, r.back().first);
        q.second = std::max(q.second, r.back().second);
      }
      std::sort(r.begin(), r.end());
      for (size_t i = 1; i < r.size(); ++i) bad += r[i].first < r[i - 1].second;
    }
    for (auto x = chain.begin(); x != chain.end(); ++x)
      for (auto y = std::next(x); y != chain.end(); ++y)
        bad += x->second.first < y->second.second && y->second.first < x->second.second;
  }
  if (bad) {
    std::printf("%d scratch ranges overlap or leave the pool\n", bad);
    return 1;
  }
  std::printf("ok launches=%d imposed=%d\n", launches, imposed);
  return 0;
}
