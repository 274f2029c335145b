"""The grid barrier's word (csrc/wig_wait.h), compiled for the CPU: however
many CTAs of however many give up, in whatever order with the arrivals still
coming, no wait that reads the word from then on passes."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include "wig_wait.h"
#include <cstdio>
using namespace wig;
int main() {
    // as many CTAs as a grid has, all giving up but `late`, which arrive after
    for (uint32_t n = 2; n <= 148; n++)
        for (uint32_t barriers = 1; barriers <= 64u * 30u; barriers += 613u)
            for (uint32_t gave = 1; gave <= n; gave++) {
                const uint32_t target = n * barriers;
                uint32_t word = target - (n - gave) - 1u;  // the arrivals before
                if (barrierOver(word, target)) return printf("passed early\n"), 1;
                for (uint32_t k = 0; k < gave; k++) {
                    word |= BARRIER_GAVE_UP;
                    if (!barrierGaveUp(word) || !barrierOver(word, target)) return printf("lost at %u of %u\n", k, n), 1;
                }
                for (uint32_t k = 0; k < n; k++) {
                    word += 1u;
                    if (!barrierGaveUp(word)) return printf("arrival %u of %u took it away\n", k, n), 1;
                }
            }
    // and none given up: passed at the last arrival, not before
    return barrierOver(147u, 148u) || !barrierOver(148u, 148u) || barrierGaveUp(148u) || barrierGaveUp(148u * 64u * 30u);
}
"""


def test_a_barrier_given_up_stays_so(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    src, exe = tmp_path / "wait.cpp", tmp_path / "wait"
    src.write_text(MAIN)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "worldinagrain_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_the_barrier_gives_up_by_that_word():
    with open(os.path.join(ROOT, "worldinagrain_b200", "csrc", "wig_fast.cu")) as f:
        s = f.read()
    sync = s[s.index("struct GridGroup"):]
    sync = sync[: sync.index("};")]
    assert "atomicOr(&st->bar_count, BARRIER_GAVE_UP)" in sync
    assert "atomicAdd(&st->bar_count" not in sync and "atomicExch(&st->bar_count" not in sync
