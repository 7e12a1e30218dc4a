"""The decode kernel's cuts of the keys, compiled for the host: every plan covers every key, with, without and with a too
small workspace (which is launched as without one)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SWEEP = r"""
#include <cstdio>
#include "scan_plan.h"
using namespace tyr;
int main() {
  long long plans = 0, bad = 0, ws = 0;
  for (int sm : {148, 132, 20, 1})
    for (int d : {64, 128})
      for (long long units = 1; units <= 4096; units += units < 330 ? 1 : 97)
        for (int len = 1; len <= 65536; len += len < 70 ? 1 : 1 + len / 9) {
          bool pays;
          for (int splits : {1, 2, 5, 64}) {
            const ScanPlan own = own_scan_plan(d, units, len, splits, sm, &pays);
            bad += !own.covers(len) || own.needs_workspace() || own.n_splits > splits || (own.warps != 4 && own.warps != 8);
          }
          for (bool have : {false, true}) {
            const ScanPlan s = few_rows_plan(d, units, len, have, sm);
            if (!s.covers(len) || (!have && s.needs_workspace()) || s.n_splits > kMaxWsChunks || (s.warps != 4 && s.warps != 8)) {
              if (bad++ < 5) std::printf("sm %d d %d units %lld len %d workspace %d: cluster %d splits %d chunk %d\n", sm, d, units, len,
                                         have, s.cluster, s.n_splits, s.chunk_len);
            }
            // the last CTA of a plan with partials has keys: the merge reads a slot per chunk
            bad += s.needs_workspace() && (long long)s.chunk_len * (s.n_splits - 1) >= len;
            ws += s.needs_workspace();
            ++plans;
          }
        }
  ScanPlan unset;
  bad += unset.covers(1);  // a plan nobody filled in is refused by the launch
  std::printf("%lld plans, %lld with a workspace, %lld bad\n", plans, ws, bad);
  return bad || ws == 0 || ws == plans;
}
"""


def test_every_plan_covers_every_key(tmp_path):
    src, exe = tmp_path / "sweep.cpp", tmp_path / "sweep"
    src.write_text(SWEEP)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "tyr_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
