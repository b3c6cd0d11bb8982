// Host rules that choose how a launch on one GPU is cut (csrc/host_layout.h): tokens per gating task and per
// COMBINE task over every token count, against the counters and tasks they have to fit.  No GPU.
#include <cstdio>

#include "host_layout.h"

using namespace fdmoe;

static int failures = 0;
#define CHECK(cond)                                                            \
  do {                                                                         \
    if (!(cond) && ++failures < 20) std::printf("  FAILED %s (line %d)\n", #cond, __LINE__); \
  } while (0)

int main() {
  for (int grid : {1, 2, 37, 148}) {
    for (int most : {1, 3, 8, 16}) {
      for (int max_tokens : {0, 1, 2, 7, 100, 147, 148, 149, 300, 1183, 1184, 1185, 4096, 40000}) {
        Geometry g;
        g.H = 2048; g.I = 768; g.E = g.El = 128; g.K = 8;
        g.max_tokens_local = g.max_tokens_max = max_tokens;
        g.max_tokens_sum = max_tokens;
        g.combine_group = most;
        g.small_groups = max_tokens < grid ? max_tokens : grid;
        CHECK(FinishGeometry(g, grid));
        for (int t = 1; t <= max_tokens; t += 1 + t / 97) {
          // every COMBINE group has a counter, and every task of the launch a slot
          const int cg = CombineGroup(t, grid, most);
          CHECK(cg >= 1 && cg <= most);
          const size_t groups = ((size_t)t + cg - 1) / cg;
          CHECK(groups <= CombineGroups(g));
          CHECK(groups <= (size_t)grid || cg == most);
          // gating tasks: one of the forms the kernel has; exact ones in one wave
          const int gr = GateRows(t, grid);
          CHECK(gr == 1 || gr == 2 || gr == 32 || gr == 64 || gr == 128);
          const size_t gates = ((size_t)t + gr - 1) / gr;
          CHECK(gr > 2 || gates <= (size_t)grid);
          const uint64_t tiles = ((uint64_t)t * g.K / FDMOE_TILE_M + g.El) * (g.H / FDMOE_TILE_N2);
          CHECK(tiles + groups + (gr > 2 ? (uint64_t)t / 2 + gates : 0) + 1 <= g.queue_cap);
        }
      }
    }
  }
  if (failures) std::printf("%d checks failed\n", failures);
  return failures != 0;
}
