"""float32 products in each form of the tile kernel (two tiles to an SM, one, tiles of 256 columns): the bits of the general kernel, which adds in
the same order.  Needs a B200: ``-m gpu``."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS, (TWO, ONE, WIDE), (ROWS, SPLIT_ROWS) = 148, range(3), (1, 2)


def tile_form(shapes, *, mode=0, a_kfast=True, b_kfast=False, groups=1, row_tiles=(0, 0, 0), mean_rows=0):
    """The rule of ``tile_form`` in csrc/gemm_simt.cu, restated (test_tile_form_rule.py compares the two): (M, K, N) of the products of a launch."""
    if a_kfast and b_kfast or (mean_rows if mode == SPLIT_ROWS else shapes[0][1]) < 128:
        return TWO
    narrow = wide = 0
    for guess in row_tiles:
        # products whose rows are the group's share their row tiles
        tiles = [guess or -(-(m if mode == SPLIT_ROWS else shapes[0][0]) // 128) for m, _, _ in shapes]
        counts = [groups * sum(count * -(-n // columns) for count, (_, _, n) in zip(tiles, shapes)) for columns in (128, 256)]
        narrow, wide = max((narrow, wide), tuple(counts))
    if narrow <= SMS:
        return ONE
    return WIDE if mode not in (ROWS, SPLIT_ROWS) and len(shapes) == 1 and narrow <= 2 * SMS and wide <= SMS else TWO


# (m, k, n) and the form: wide tiles with 4, 132, 252 and 256 columns in the last and 68, 128 and 4 rows; one tile to an SM, few and as many as
# there are; two, many and, with inner sizes below the rule's 128, few; inner sizes of whole slices, one value more and one less
SHAPES = [(2500, 128, 1028, WIDE), (2560, 143, 1156, WIDE), (2564, 129, 1276, WIDE), (4096, 260, 1024, WIDE), (644, 301, 2500, ONE), (508, 144, 4732, ONE),
          (640, 640, 2560, ONE), (4100, 129, 1280, TWO), (2500, 124, 1028, TWO), (1024, 16, 1024, TWO), (2048, 33, 1028, TWO), (2044, 47, 1156, TWO),
          (4096, 64, 1276, TWO), (4100, 48, 1000, TWO)]


@pytest.mark.parametrize("form", ["nn", "tn", "tt"])
@pytest.mark.parametrize("m,k,n,tiles_of", SHAPES)
def test_tile_forms_give_the_bits_of_the_general_kernel(form, m, k, n, tiles_of, kernel_variant):
    from gpu_util import to_device
    from qutai_b200 import lib
    from qutai_b200.storage import DeviceStorage

    k = k if form == "tn" else -(-k // 4) * 4       # whole 16-byte pieces along what is contiguous
    assert tile_form([(m, k, n)], a_kfast=form[0] == "n", b_kfast=form[1] == "t") == tiles_of and lib.device_info()["sm_count"] == SMS
    rng = np.random.default_rng(m + k + n)
    a, b = (to_device(rng.standard_normal(size).astype(np.float32), "float32") for size in (m * k, k * n))

    def product():
        out = DeviceStorage(m * n, "float32")
        lib.call("qmoe_memset", out.ptr, 0xFF, out.nbytes, 0)
        lib.call("qmoe_gemm", a.ptr, lib.QMOE_F32, b.ptr, lib.QMOE_F32, out.ptr, lib.QMOE_F32, m, k, n, int(form[0] == "t"), int(form[1] == "t"), 0, 0)
        return out.tobytes()

    tiles = product()
    kernel_variant(lib.VARIANT_NO_FLOAT32_TILES)
    assert tiles == product()
