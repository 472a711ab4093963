// Checks the layout of the resident small-level cycle (csrc/ssa_small_plan.h resident_plan) on
// the level chains given on stdin, one "first nlev Mx My ax ay Mx My ax ay ..." line each:
// every item of a register level belongs to one thread of one CTA, a CTA's items fit its
// threads, the window of a CTA beside the lead holds every row its items' stencils read at the
// index the kernel forms, the lead's arrays lie apart inside the shared memory, and the
// neighbour tables' indices fit 16 bits.  Prints "ok <wide> <bytes>", "none" where the levels
// do not fit, or "bad <reason>".
#include <cstdio>
#include <sstream>
#include <iostream>
#include <string>
#include <vector>

#include "ssa_small_plan.h"

using namespace pism_gpu;

static int wrap(int a, int n) { return a < 0 ? a + n : (a >= n ? a - n : a); }

int main() {
  std::string line;
  while (std::getline(std::cin, line)) {
    std::istringstream in(line);
    int first, nlev;
    in >> first >> nlev;
    std::vector<int> Mx(nlev), My(nlev), ax(nlev), ay(nlev);
    for (int l = 0; l < nlev; ++l) in >> Mx[l] >> My[l] >> ax[l] >> ay[l];
    ResidentPlan P;
    const int max_smem = 220 * 1024, last = nlev - 1;
    if (!resident_plan(first, last, Mx.data(), My.data(), ax.data(), ay.data(), max_smem, P)) {
      std::printf("none\n");
      continue;
    }
    const char *bad = nullptr;
    auto N = [&](int l) { return Mx[l] * My[l]; };
    // the lead's shared memory
    std::vector<char> used(P.smem, 0);
    auto claim = [&](int at, int bytes) {
      if (at % 16 != 0 || at < 0 || at + bytes > P.smem) { bad = "outside the shared memory or misaligned"; return; }
      for (int b = at; b < at + bytes; ++b) {
        if (used[b]) bad = "two arrays overlap";
        used[b] = 1;
      }
    };
    for (int l = P.reg; l <= last; ++l) claim(P.vec[l], 24 * N(l));
    for (int l = P.reg + 1; l < last; ++l) {
      const int items = small_span(N(l + 1));
      if (items > SR_THREADS) bad = "a level's items exceed the lead's threads";
      claim(P.op[l], 160 * items);
      claim(P.nb[l], 18 * items);
      if (N(l) >= 65535) bad = "neighbour index";
    }
    // the register levels
    for (int lv = P.first; lv <= P.reg && !bad; ++lv) {
      const bool lead = lv == P.reg;
      const int parts = lead ? 1 : SC_CTAS - 1, span = small_span(N(lv + 1));
      std::vector<int> seen(N(lv), 0);
      for (int c = 0; c < parts && !bad; ++c) {
        int b0 = 0, b1 = span, w0 = 0, nrows = Mx[lv];
        if (!lead) {
          small_chunk(span, parts, c, 32, b0, b1);
          if (b1 <= b0) continue;
          int r0, r1;
          small_down_rows(ax[lv], My[lv + 1], N(lv + 1), b0, b1, r0, r1);
          small_window(Mx[lv], r0, r1, w0, nrows);
          if (32 * nrows * My[lv] > P.smem) bad = "a window exceeds the shared memory";
        }
        if (b0 % 32 || b1 % 32) bad = "a chunk is not whole warps";
        if (b1 - b0 > SR_THREADS * SR_ITEMS) bad = "a CTA has more items than threads";
        for (int it = b0; it < b1 && !bad; ++it) {
          const int kc = it >> 2, pi = (it >> 1) & 1, pj = it & 1;
          if (kc >= N(lv + 1) || pi >= ax[lv] || pj >= ay[lv]) continue;
          const int i = (kc / My[lv + 1]) * ax[lv] + pi, j = (kc % My[lv + 1]) * ay[lv] + pj;
          if (i >= Mx[lv] || j >= My[lv]) continue;
          seen[i * My[lv] + j] += 1;
          for (int di = -1; di <= 1; ++di) {
            const int ii = wrap(i + di, Mx[lv]);
            int r = ii - w0;
            if (r < 0) r += Mx[lv];
            else if (r >= nrows) r -= Mx[lv];
            if (r < 0 || r >= nrows) { bad = "a stencil row is outside the window"; break; }
            int row = w0 + r;   // the row staged there, as the kernel wraps it
            if (row < 0) row += Mx[lv];
            else if (row >= Mx[lv]) row -= Mx[lv];
            if (row != ii) bad = "another row is staged there";
            int k = w0 * My[lv] + r * My[lv];   // and its first cell
            if (k < 0) k += N(lv);
            else if (k >= N(lv)) k -= N(lv);
            if (k != ii * My[lv]) bad = "another cell is staged there";
          }
        }
      }
      for (int k = 0; k < N(lv) && !bad; ++k)
        if (seen[k] != 1) bad = "a cell is not covered once";
    }
    if (bad) std::printf("bad %s\n", bad);
    else std::printf("ok %d %d\n", P.wide, P.smem);
  }
  return 0;
}
