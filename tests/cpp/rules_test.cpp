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
          // (GATEFIX tasks: one per tile of one or two tokens, else two tokens each, rounded up per tile)
          const uint64_t fix = gr <= 2 ? gates : (uint64_t)t / 2 + gates;
          CHECK(tiles + groups + fix + 1 <= WorstCaseQueueTasks(g));
          CHECK(WorstCaseQueueTasks(g) <= g.queue_cap);
          // tiles that a caller may ask for: the same bound
          for (int rows : {1, 2, 3, 32, 64, 128, 256}) {
            CHECK(GateRowsFit(rows, t, grid, 1) == (rows == 2 || rows == 32 || rows == 64 || rows == 128 || (rows == 1 && t <= grid)));
            CHECK(GateRowsFit(rows, t, grid, 2) == (rows == 32 || rows == 64 || rows == 128));
            const uint64_t tl = ((uint64_t)t + rows - 1) / rows;
            if (GateRowsFit(rows, t, grid, 1))
              CHECK(tiles + groups + (rows <= 2 ? tl : (uint64_t)t / 2 + tl) + 1 <= WorstCaseQueueTasks(g));
          }
        }
      }
    }
  }
  // wide FFN tasks: both sides of the line of three FFN1 tasks of 256 rows per worker
  {
    Geometry g;
    g.H = 2048; g.I = 768; g.E = g.El = 128; g.K = 8;
    CHECK(WideRows(g, 0, 148) == kNoWideRows);
    CHECK(WideRows(g, 2367, 148) == kNoWideRows && WideRows(g, 2368, 148) == FDMOE_TILE_M);  // 73 and 74 m-tile pairs x 6
    g.H = 4096; g.I = 1536;
    CHECK(WideRows(g, 1183, 148) == kNoWideRows && WideRows(g, 1184, 148) == FDMOE_TILE_M);  // 36 and 37 x 12
    CHECK(WideRows(g, 1 << 20, 1) == FDMOE_TILE_M);
  }
  if (failures) std::printf("%d checks failed\n", failures);
  return failures != 0;
}
