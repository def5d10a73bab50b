"""Which form of the float32 tile kernel a product takes (``tile_form`` in csrc/gemm_simt.cu): the rule that the GPU test of the forms restates,
and products of which both sides were measured.  No GPU: compiles the file and calls the function."""
import random
import subprocess

import pytest

from qutai_b200 import build
from test_gpu_float32_tile_forms import ONE, ROWS, SMS, SPLIT_ROWS, TWO, WIDE, tile_form

PROGRAM = """
#include <stdio.h>
#include "gemm_simt.cu"
namespace qmoe { int sm_count() { return %d; } }
int main() {
    int mode, count, a_kfast, b_kfast, groups;
    long long m_extent, tiles[3], mean;
    while (scanf("%%d %%d %%d %%d %%d %%lld %%lld %%lld %%lld %%lld", &mode, &count, &a_kfast, &b_kfast, &groups, &m_extent, tiles, tiles + 1, tiles + 2, &mean) == 10) {
        qmoe::SimtGemmArgs g[qmoe::kSimtProducts] = {};
        for (int i = 0; i < count; ++i) {
            scanf("%%lld %%lld %%lld", &g[i].M, &g[i].K, &g[i].N);
            g[i].mode = mode == 0 ? qmoe::SG_PLAIN : mode == 1 ? qmoe::SG_ROWS : qmoe::SG_K;
            g[i].a_cs = a_kfast; g[i].a_rs = !a_kfast; g[i].b_rs = b_kfast; g[i].b_cs = !b_kfast;
            for (int t = 0; t < 3; ++t) g[i].row_tiles[t] = tiles[t];
            g[i].mean_rows = mean;
        }
        printf("%%d\\n", qmoe::tile_form(g, count, m_extent, groups));
    }
}
"""


@pytest.fixture(scope="module")
def forms(tmp_path_factory):
    try:
        nvcc = build.nvcc_path()
    except RuntimeError:
        pytest.skip("no nvcc on this machine")
    source, program = (tmp_path_factory.mktemp("rule") / name for name in ("rule.cu", "rule"))
    source.write_text(PROGRAM % SMS)
    done = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=compute_100a", "-std=c++17", "--expt-relaxed-constexpr", "-I", build.INCLUDE, "-I", build.CSRC, str(source), "-o",
                           str(program), "-Xlinker", "--unresolved-symbols=ignore-all"], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert done.returncode == 0, done.stdout

    def ask(questions):
        lines = []
        for shapes, kwargs in questions:
            mode, tiles = kwargs.get("mode", 0), kwargs.get("row_tiles", (0, 0, 0))
            extent = 0 if mode == SPLIT_ROWS else shapes[0][0]
            lines.append(" ".join(map(str, (mode, len(shapes), int(kwargs.get("a_kfast", True)), int(kwargs.get("b_kfast", False)), kwargs.get("groups", 1), extent,
                                            *tiles, kwargs.get("mean_rows", 0), *(value for shape in shapes for value in shape)))))
        out = subprocess.run([str(program)], input="\n".join(lines), stdout=subprocess.PIPE, text=True, check=True).stdout
        return [int(line) for line in out.split()]

    return ask


def test_products_that_were_measured_in_every_form(forms):
    questions = [
        # plain products, us as two to an SM, one, wide
        ([(4096, 1024, 1024)], {}, WIDE),                                   # 200, 208, 189
        ([(1024, 4096, 2048)], {}, ONE),                                    # 427, 405, 728
        ([(640, 640, 2560)], {}, ONE),                                      # 72, 68, 120
        ([(6684, 140, 4020)], dict(a_kfast=False), TWO),                    # 169, wide 172: 4 % by rounds, many of them
        # products of layers; guesses of tiles as dispatched_tiles makes them
        ([(8448, 760, 1408)], dict(mode=ROWS, row_tiles=(68, 68, 69)), TWO),             # dX of 4096 x 1408 x 760, 2 of 8: the call 3464, wide 3571
        ([(6128, 448, 1984)], dict(mode=ROWS, row_tiles=(40, 40, 42)), TWO),             # 4096 x 1984 x 448, 1 of 16: the call 1851, by rounds alone 2020:
        ([(6128, 1984, 448)], dict(mode=ROWS, row_tiles=(40, 40, 42)), TWO),             # d_h wide, and
        ([(1984, 0, 448), (448, 0, 1984), (448, 0, 1984)], dict(mode=SPLIT_ROWS, groups=16, a_kfast=False, mean_rows=256), TWO),     # the weight gradients
        ([(5120, 1024, 512)], dict(mode=ROWS, row_tiles=(36, 36, 37)), ONE),             # dX of 2048 x 512 x 1024, 2 of 8: 225, one 203
    ]
    assert forms([(shapes, kwargs) for shapes, kwargs, _ in questions]) == [want for _, _, want in questions]


def test_the_rule_restated_for_the_gpu_test_is_the_rule(forms):
    rng = random.Random(3)
    questions = []
    for _ in range(3000):
        mode, count = rng.choice((0, ROWS, SPLIT_ROWS)), rng.choice((1, 1, 2, 3))
        m = rng.randint(1, 9000)
        shapes = [(m if mode == ROWS else rng.randint(1, 9000), rng.randint(16, 1000), rng.randint(65, 5000)) for _ in range(count if mode else 1)]
        kwargs = dict(mode=mode, a_kfast=rng.random() < 0.5, b_kfast=rng.random() < 0.5)
        if mode == ROWS:
            kwargs["row_tiles"] = tuple(rng.randint(1, 80) for _ in range(3)) if rng.random() < 0.5 else (rng.randint(1, 80),) * 3
        if mode == SPLIT_ROWS:
            kwargs.update(groups=rng.randint(1, 64), mean_rows=rng.choice((16, 127, 128, 500)))
        questions.append((shapes, kwargs))
    got = forms(questions)
    assert {form: got.count(form) > 50 for form in (TWO, ONE, WIDE)} == {TWO: True, ONE: True, WIDE: True}
    assert got == [tile_form(shapes, **kwargs) for shapes, kwargs in questions]
