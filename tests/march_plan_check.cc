// Host driver for the marching passes' division of a grid (csrc/ssa_march_plan.h): reads lines
// "Mx My sms" and prints for each of the three passes (halo, extra rows, alignment as ssa_mg.cu
// gives them) strips, rows a chunk, chunks and blocks, then the doubles the partial sums need.
#include <iostream>

#include "ssa_march_plan.h"

using namespace pism_gpu;

int main() {
  int Mx, My, sms;
  while (std::cin >> Mx >> My >> sms) {
    for (const MarchPlan &p : {march_plan(Mx, My, 1, 2, 2, sms, 8, 1), march_plan(Mx, My, 1, 2, 1, sms, 10, 1),
                               march_plan_apply(Mx, My, sms)})
      std::cout << p.strips << ' ' << p.R << ' ' << p.chunks << ' ' << p.blocks << ' ';
    std::cout << march_partials(Mx, My, sms) << '\n';
  }
  return 0;
}
