"""The queue of the persistent kernels' tickets, on the host: the kernels' own
functions compiled into a small program.  Every place of the queue is one ticket
and every ticket one place, whichever CTAs ask and however late; a CTA's first
places are its share of each length of trajectory; a warp's count of its windows
never comes back to its first."""
import os
import subprocess

import pytest

from conftest import ROOT
from geliosphere_gb300 import build

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "kernels.cuh"
using namespace gelio;

template <class R> int check(unsigned long long total, unsigned ctas, unsigned warps, unsigned per_sm, bool alike) {
  const Placement p = place<R>(total, ctas, warps, per_sm, trajectories_per_lane(alike));
  if (p.warps < 1 || p.warps > warps || p.lanes > 32 || (total && p.lanes < 1)) return 1;
  const unsigned long long places = total > p.dealt ? total : p.dealt;
  std::vector<char> seen(total, 0);
  unsigned long long got = 0;
  for (unsigned long long at = 0; at < places; ++at) {
    const unsigned long long t = ticket_at(at, p, ctas);
    if (t >= places) return 2;
    if (t >= total) continue;
    if (seen[t]) return 3;
    seen[t] = 1;
    ++got;
  }
  if (got != total) return 4;
  if (ticket_at(places, p, ctas) < total || ticket_at(places + 12345, p, ctas) < total) return 5;
  // a CTA that asks b-th: warp w starts with chunk w * ctas + b
  for (unsigned b = 0; b < ctas && total; b += 7)
    for (unsigned w = 0; w < p.warps; ++w)
      if (ticket_at((unsigned long long)(b * p.warps + w) * p.lanes, p, ctas) !=
          (unsigned long long)(w * ctas + b) * p.lanes) return 6;
  return 0;
}

int main() {
  const unsigned shapes[][3] = {{304, 8, 2}, {152, 8, 1}, {456, 3, 3}, {608, 4, 4}, {1216, 1, 8}, {1, 1, 1}, {304, 8, 0}};
  const unsigned long long totals[] = {0, 1, 2, 151, 152, 303, 305, 500, 2431, 2432, 2433, 9727, 9729, 19456, 19457, 38911,
                                       38913, 77823, 77824, 77825, 116736, 116737, 233473, 350209, 1000003};
  for (auto &s : shapes)
    for (auto n : totals) for (int alike = 0; alike < 2; ++alike) {
      const int f = check<float>(n, s[0], s[1], s[2], alike), d = check<double>(n, s[0], s[1], s[2], alike);
      if (f || d) { printf("total %llu ctas %u warps %u per sm %u: %d %d\n", n, s[0], s[1], s[2], f, d); return 1; }
    }
  unsigned w = 0;
  if ((w = next_window(w)) != 1u || (w = next_window(w)) != 2u) return 2;
  for (w = 0xfffffff0u; w != 9u; w = next_window(w))
    if (w < 2u) { puts("a late window counts as the first"); return 3; }
  puts("ok");
}
"""


LENGTHS = r"""
#include <cstdio>
#include "kernels.cuh"
using namespace gelio;

static bool differ(int injection, float lo, float hi, int points) {
  gelio_sim_params p{};
  p.injection = injection; p.inj_min = lo; p.inj_max = p.injection_max = hi; p.inj_points = points;
  return lengths_differ(p);
}

int main() {
  const int lg = GELIO_INJ_LOG_GRID, lu = GELIO_INJ_LOG_UNIFORM, ru = GELIO_INJ_REFERENCE_UNIFORM, cu = GELIO_INJ_CPU_UNIFORM;
  const bool wide = differ(lg, 0.01f, 100, 100) && differ(lg, 0.1f, 3.1f, 33) && differ(lg, 1, 100, 10) && differ(lu, 0.01f, 100, 1) &&
                    differ(lu, 0.3f, 100, 1) && differ(ru, 0, 101, 1) && differ(cu, 0, 5, 1) && differ(GELIO_INJ_SOLARPROP_GRID, 0, 0, 0);
  const bool narrow = differ(lg, 0.1f, 0.1f, 1) || differ(lg, 0.01f, 100, 1) || differ(lg, 50, 100, 7) || differ(lg, 0.01f, 0.3f, 33) ||
                      differ(lg, 0.01f, 1, 33) || differ(lu, 0.01f, 3, 1) || differ(lu, 0.03f, 10, 1) || differ(ru, 0, 1, 1) || differ(cu, 0, 0.2f, 1);
  // more than six (two) trajectories a lane only on all warps; FP64 steps and sample runs always
  unsigned fewer[2] = {0, 0};
  for (unsigned long long n = 1; n < 500000; n += 777)
    for (int alike = 0; alike < 2; ++alike) {
      const unsigned most = trajectories_per_lane(alike);
      const Placement p = place<float>(n, 304, 8, 2, most);
      if (p.warps < 8 && n > 304ull * p.warps * 32 * most) return 1;
      fewer[alike] += p.warps < 8;
      if (place<float>(n, 304, 8, 0, most).warps != 8 || place<double>(n, 304, 8, 2, most).warps != 8) return 2;
    }
  puts(wide && !narrow && fewer[0] > 2 * fewer[1] && fewer[1] > 0 ? "ok" : "no");
}
"""


def run_program(tmp_path, text):
    src, exe = tmp_path / "tickets.cu", tmp_path / "tickets"
    src.write_text(text)
    cc = build.nvcc()
    if subprocess.run([cc, "--version"], capture_output=True).returncode != 0:
        pytest.skip("no nvcc")
    subprocess.run([cc, *build.ARCH, "-std=c++17", "-O1", "-I" + build.CSRC, "-I" + os.path.join(ROOT, "include"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


def test_every_place_is_a_ticket(tmp_path):
    run_program(tmp_path, PROGRAM)


def test_which_simulations_go_on_fewer_warps(tmp_path):
    """Those with a few trajectories much longer than most, by their injection; others
    up to two trajectories a lane."""
    run_program(tmp_path, LENGTHS)
