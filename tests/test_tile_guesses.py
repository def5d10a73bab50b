"""The guesses of how many 128-row tiles a float32 call's experts take (``dispatched_tiles`` in csrc/layer.cu), which the host makes for every
product: their values, and that what they cost does not grow with the number of rows.  No GPU: compiles the file and calls the function."""
import math
import subprocess

import pytest

from qutai_b200 import build

PROGRAM = """
#include <math.h>
#include <stdio.h>
static long evaluations = 0;
static double counted(double value) { ++evaluations; return erfc(value); }
#define erfc counted
#include "layer.cu"
int main() {
    const long long loads[][3] = {%s};
    for (auto& load : loads) {
        qmoe_route_t r = {};
        r.tokens = load[0]; r.experts = (int)load[1]; r.top_k = (int)load[2];
        long long tiles[3];
        evaluations = 0;
        qmoe::dispatched_tiles(&r, tiles);
        printf("%%lld %%lld %%lld %%ld\\n", tiles[0], tiles[1], tiles[2], evaluations);
    }
}
"""
# tokens, experts, top_k: a row or none per expert, the sizes of layers, rows past a million on one expert
LOADS = [(1, 8, 1), (64, 64, 6), (209, 32, 2), (2048, 8, 2), (4096, 4, 1), (100_000, 1, 1), (1_000_000, 2, 2), (16_000_000, 1, 1)]


def test_guesses_of_tiles_and_what_they_cost(tmp_path):
    try:
        nvcc = build.nvcc_path()
    except RuntimeError:
        pytest.skip("no nvcc on this machine")
    source, program = tmp_path / "guesses.cu", tmp_path / "guesses"
    source.write_text(PROGRAM % ", ".join("{%d, %d, %d}" % load for load in LOADS))
    done = subprocess.run([nvcc, *build.ARCH_FLAGS, "-std=c++17", "--expt-relaxed-constexpr", "-I", build.INCLUDE, "-I", build.CSRC, str(source), "-o",
                           str(program), "-Xlinker", "--unresolved-symbols=ignore-all"], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert done.returncode == 0, done.stdout
    lines = subprocess.run([str(program)], stdout=subprocess.PIPE, text=True, check=True).stdout.split("\n")
    for (tokens, experts, top_k), line in zip(LOADS, lines):
        *tiles, evaluations = map(int, line.split())
        rows = tokens * top_k
        mean = rows / experts
        firsts = (0.5 + 128 * i for i in range(int((mean + 6 * math.sqrt(mean) + 1) / 128) + 1))
        certain = sum(0.5 * math.erfc((first - mean) / math.sqrt(2 * mean)) for first in firsts if first < mean + 6 * math.sqrt(mean) + 1)
        half = rows / 128 + 0.5 * experts
        want = [max(1, int(guess)) for guess in (certain * experts + 0.5, half + 0.5, half + 0.5 * math.sqrt(experts))]
        assert all(abs(got - guess) <= 1e-6 * guess for got, guess in zip(tiles, want)), (tokens, tiles, want)
        # six standard deviations to either side of the mean
        assert evaluations <= 12 * math.sqrt(mean) / 128 + 3, (tokens, evaluations)
