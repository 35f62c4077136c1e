// Prints the rules of schedule.h.  Usage:
//   schedule_main cluster COUNT N CLUSTERS   whether the cluster tridiagonalisation pays
//   schedule_main bucket N                   size bucket
#include <cstdio>
#include <cstdlib>
#include <string>
#include "schedule.h"

int main(int argc, char** argv) {
  const std::string mode = argc > 1 ? argv[1] : "";
  auto arg = [&](int k) { return std::atoi(argv[k]); };
  if (mode == "cluster" && argc == 5) std::printf("%d\n", (int)nddo::hh_cluster_pays(arg(2), arg(3), arg(4)));
  else if (mode == "bucket" && argc == 3) std::printf("%d\n", nddo::size_bucket(arg(2)));
  else return 2;
  return 0;
}
