"""The CTA size of batches beyond one wave (no GPU): the choice, compiled from its header, at the register
limits that the kernels are compiled for -- the most paths on an SM, the usual size where none has more."""
import os
import shutil
import subprocess

import pytest

import ghc

CSRC = os.path.join(ghc.HERE, "csrc")
SOURCE = """
#include <cstdio>
#include "ghc_internal.h"
int main() {
  int tables, per_sub, W, max_block, max_threads, block, threads;
  while (std::scanf("%d %d %d %d %d %d %d", &tables, &per_sub, &W, &max_block, &max_threads, &block, &threads) == 7)
    std::printf("%d\\n", ghc::widest_block(tables, per_sub, W, max_block, max_threads, block, threads));
}
"""
SM, RESERVED = 228 * 1024, 1024


def _want(tables, per_sub, W, max_block, max_threads, block, threads):
    best, most = block, threads
    for b in range(64, max_block + 1, 32):
        cta = tables + b // W * per_sub + RESERVED
        if cta <= SM and min(SM // cta * b, max_threads) > most:
            best, most = b, min(SM // cta * b, max_threads)
    return best


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_widest_block(tmp_path):
    (tmp_path / "shape.cpp").write_text(SOURCE)
    exe = str(tmp_path / "shape")
    subprocess.check_call(["g++", "-std=c++17", "-I", CSRC, str(tmp_path / "shape.cpp"), "-o", exe])
    cases = [(t, s, W, 256, most, 128, usual) for t in (600, 5000, 40000) for s in (912, 2032, 3824, 18512)
             for W in (8, 16) for most in (512, 768, 1024) for usual in (128, 384, 512, 768) if usual <= most]
    cases.append((1500, 2032, 8, 256, 1024, 128, 768))  # room above 768 threads, which 512 as the limit would hide
    out = subprocess.run([exe], input="\n".join(" ".join(map(str, c)) for c in cases), capture_output=True, text=True,
                         check=True).stdout.split()
    assert [int(v) for v in out] == [_want(*c) for c in cases]
    assert int(out[-1]) > 128
