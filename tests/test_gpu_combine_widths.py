"""The backward of the combine with two, four and eight 16-byte pieces of a row per lane, at widths that end inside the first, the second and the
third round of pieces.  Needs a B200: ``-m gpu``."""
import pytest

import test_gpu_parity as parity

pytestmark = pytest.mark.gpu

# 16-byte pieces of a row: up to 127 go in rounds of 64, up to 255 in rounds of 128, above that in rounds of 256
PIECES = [2, 65, 127, 128, 129, 161, 255, 256, 257, 300, 513]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("T,E,k,pieces", [(37, 5, (1, 2, 3, 4, 5)[i % 5], pieces) for i, pieces in enumerate(PIECES)] + [(130, 9, 8, 129), (130, 9, 6, 257)])
def test_rows_that_end_inside_a_round_of_pieces(T, E, k, pieces, dtype):
    parity.test_permute_combine_and_backwards(T, E, k, pieces * (4 if dtype == "float32" else 8), dtype)
