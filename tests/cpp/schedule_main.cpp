// Prints the rules of schedule.h.  Usage:
//   schedule_main cluster COUNT N CLUSTERS   whether the cluster tridiagonalisation pays
//   schedule_main bucket N                   size bucket
//   schedule_main scf TILED EARLY GAPLESS BLOCK MAX_ITER FEW ALL (CONVERGED FROM STEPS)...
//                                            the SCF loop over molecules that converge
//                                            in iteration CONVERGED and need STEPS
//                                            purification steps from iteration FROM on,
//                                            20 before; prints the number of iterations of
//                                            each effort, then each molecule's status
//                                            (1 converged, 2 max_iter) and waits
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>
#include "schedule.h"

struct Mol { int converged, from, steps, iter = 0, status = 0, waits = 0; bool flag = false; };

static void scf(bool tiled, int early, bool gapless, int block, int max_iter, int few, int all, std::vector<Mol> mols) {
  int used[3] = {0, 0, 0};
  nddo::BlockCounts slots[2] = {};
  nddo::run_blocks(
      block, max_iter, true, nddo::EffortPlan(tiled, early, gapless),
      [&](int effort) {
        ++used[effort];
        for (Mol& m : mols) {
          if (m.status) continue;
          const int need = m.iter >= m.from ? m.steps : 20, have = !tiled || effort > 0 ? all : few;
          m.flag = need > have && effort < 2;
          if (m.flag) { ++m.waits; continue; }
          if (++m.iter == m.converged) m.status = 1;
          else if (m.iter >= max_iter) m.status = 2;
        }
      },
      [&](int slot) {
        slots[slot] = {0, 0};
        for (const Mol& m : mols) { slots[slot].active += !m.status; slots[slot].waiting += !m.status && m.flag; }
      },
      [&](int slot) { return slots[slot]; });
  std::printf("%d %d %d", used[0], used[1], used[2]);
  for (const Mol& m : mols) std::printf(" %d %d", m.status, m.waits);
  std::printf("\n");
}

int main(int argc, char** argv) {
  const std::string mode = argc > 1 ? argv[1] : "";
  auto arg = [&](int k) { return std::atoi(argv[k]); };
  if (mode == "cluster" && argc == 5) std::printf("%d\n", (int)nddo::hh_cluster_pays(arg(2), arg(3), arg(4)));
  else if (mode == "bucket" && argc == 3) std::printf("%d\n", nddo::size_bucket(arg(2)));
  else if (mode == "scf" && argc >= 12 && (argc - 9) % 3 == 0) {
    std::vector<Mol> mols;
    for (int k = 9; k < argc; k += 3) mols.push_back({arg(k), arg(k + 1), arg(k + 2)});
    scf(arg(2), arg(3), arg(4), arg(5), arg(6), arg(7), arg(8), mols);
  } else return 2;
  return 0;
}
