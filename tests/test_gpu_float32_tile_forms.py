"""float32 products in each form of the tile kernel (two tiles to an SM, one, tiles of 256 columns): the bits of the general kernel, which adds in
the same order.  Needs a B200: ``-m gpu``."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (m, k, n): by the rule of 148 SMs one round of single tiles; one of wide tiles, the last column tile with 4, 132 and 252 columns; rounds of two;
# inner sizes of whole slices, one value more and one less
SHAPES = [(1024, 16, 1024), (2048, 33, 1028), (2044, 47, 1156), (4096, 64, 1276), (4100, 48, 1000), (640, 640, 2560)]


@pytest.mark.parametrize("form", ["nn", "tn", "tt"])
@pytest.mark.parametrize("m,k,n", SHAPES)
def test_tile_forms_give_the_bits_of_the_general_kernel(form, m, k, n, kernel_variant):
    from gpu_util import to_device
    from qutai_b200 import lib
    from qutai_b200.storage import DeviceStorage

    k = k if form == "nn" and k % 4 == 0 or form == "tn" else -(-k // 4) * 4       # whole 16-byte pieces along what is contiguous
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
