// Host driver for the end of the mixed-precision refinement (ssa_state.h): reads lines
//   <rtol> <max_refine> <n> { <iter> <status> }*n { <r2> <b2> }*(n + 1)
// the outcome of each inner solve and the residual before it, and prints the refinement's state
// twice: with every pass taken (an inner solve that finds the tolerance met ends the loop), and
// with the passes refine_more() leaves out, then the passes each took.
#include <cstdio>
#include <cstdlib>
#include <iostream>
#include <sstream>
#include <string>
#include <vector>

#include "ssa_state.h"

using namespace pism_gpu;

struct Record {
  int iter, status;
};
struct Norms {
  double r2, b2;
};

static void run(double rtol, int max_refine, const std::vector<Record> &rec, const std::vector<Norms> &norms, bool skip) {
  PState P{};
  picard_start(P);
  P.rtol = rtol;
  int taken = 0;
  for (size_t k = 0; k < rec.size(); ++k) {
    // the inner solve's start (k32_init): done at once where the tolerance is met, NaN included
    const double rn = sqrt(norms[k].r2), bn = sqrt(norms[k].b2);
    const bool met = !(rn > rtol * bn) || bn == 0.0;
    KState st{};
    st.outer_r2 = norms[k].r2;
    st.outer_b2 = norms[k].b2;
    st.iter = met ? 0 : rec[k].iter;
    st.status = met ? KSP_OUTER_DONE : rec[k].status;
    refine_end(P, st, max_refine);
    ++taken;
    if (!P.go) break;
    if (skip && !refine_more(P, norms[k + 1].r2, norms[k + 1].b2, max_refine)) break;
  }
  printf("%d %d %d %d %d %d %lld %.17g %d %d\n", P.refine, P.refine_done, P.go, P.ksp_its, P.ksp_status, P.refine_steps,
         P.inner_passes, P.final_res, P.refine_passes, taken);
}

int main() {
  std::string line;
  while (std::getline(std::cin, line)) {
    std::istringstream in(line);
    auto num = [&] {
      std::string t;
      in >> t;
      return strtod(t.c_str(), nullptr);
    };
    const double rtol = num();
    const int max_refine = (int)num(), n = (int)num();
    std::vector<Record> rec(n);
    std::vector<Norms> norms(n + 1);
    for (auto &r : rec) {
      r.iter = (int)num();
      r.status = (int)num();
    }
    for (auto &q : norms) {
      q.r2 = num();
      q.b2 = num();
    }
    run(rtol, max_refine, rec, norms, false);
    run(rtol, max_refine, rec, norms, true);
  }
  return 0;
}
