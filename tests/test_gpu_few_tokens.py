"""The streamed products' form for at most 32 tokens, against the kernel for many rows, around its steps of 16 rows and at its limits.
Needs a B200: ``-m gpu``."""
import pytest

import test_gpu_few_rows as few_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,width,hidden", [
    ((0, 1, 15, 16), 64, 128),               # 32 tokens; fewer k-blocks than stages
    ((32,), 584, 136),                       # one expert with every row, widths that fill no tile
    ((33,), 584, 136),                       # one token more: the form with 128 rows per stage
    ((0, 17, 2, 0, 0, 13), 1032, 264),       # two steps of 16 rows; more k-blocks than stages
    ((1,) * 30, 2048, 1408),                 # more than two tiles per SM: the form with 128 rows per stage
])
def test_products_of_few_tokens(counts, width, hidden, kernel_variant):
    few_rows.test_streamed_products_match_the_kernel_for_many_rows(counts, width, hidden, kernel_variant)
