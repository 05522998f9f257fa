"""The H_x walk that the tracker takes by default (no GPU): the rule, compiled from its header, on the
shipped problems' tables that lie beside its lines."""
import os
import shutil
import subprocess

import pytest

import ghc

CSRC = os.path.join(ghc.HERE, "csrc")
ENTRY, ROW, BALANCED = 0, 1, 2
SOURCE = """
#include <cstdint>
#include <cstdio>
#include <vector>
#include "ghc_internal.h"
int main() {
  int N, n;
  while (std::scanf("%d %d", &N, &n) == 2) {
    std::vector<uint16_t> off(n);
    for (auto& o : off) {
      int v;
      if (std::scanf("%d", &v) != 1) return 1;
      o = (uint16_t)v;
    }
    std::printf("%d\\n", ghc::flat_eval_pays(off.data(), N));
  }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_default_walk_of_shipped_problems(tmp_path):
    want = {"6pt_RS_abs_pos": ENTRY, "generalized_3views_6lines": BALANCED, "3pt_rel_pos_homog": BALANCED,
            "3view_triangulation": BALANCED, "optimal_PnP_quat": BALANCED, "dual_reciever_TDOA_5pt": BALANCED,
            "5pt_rel_pos_alg_form_quat": BALANCED, "4view_triangulation": BALANCED, "P3P_10x10": BALANCED,
            "generalized_3views_4pts": ROW, "uncalibrated_trifocal_rel_pos_CY": ROW, "trifocal_2op1p_30x30": ROW}
    (tmp_path / "walk.cpp").write_text(SOURCE)
    exe = str(tmp_path / "walk")
    subprocess.check_call(["g++", "-std=c++17", "-I", CSRC, str(tmp_path / "walk.cpp"), "-o", exe])
    lines = []
    for name in want:
        pb = ghc.Problem(name)
        off = [int(v) for v in pb.compiled_hx()[1]]
        lines.append(" ".join(map(str, [pb.N, len(off)] + off)))
    out = subprocess.run([exe], input="\n".join(lines), capture_output=True, text=True, check=True).stdout.split()
    assert dict(zip(want, map(int, out))) == want
