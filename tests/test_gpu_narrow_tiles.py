"""Plain products of a few tiles (128 x 64 tiles, one CTA each): the same bits as 128 x 256 tiles, and the exact product within
bfloat16.  Needs a B200: ``-m gpu``."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows, inner, columns: one row more than a tile, one column group more or less than a tile, inner sizes around a k-block, as many
# tiles as SMs (148) and two more, which run as 256 x 256 tiles
SHAPES = [(129, 64, 8), (130, 72, 64), (257, 520, 72), (602, 512, 512), (300, 4096, 136), (4736, 64, 256), (4737, 64, 256)]


def _operands(form, rows, inner, columns):
    rng = np.random.default_rng(rows + inner + columns)
    shapes = {"nt": ((rows, inner), (columns, inner)), "nn": ((rows, inner), (inner, columns)), "tn": ((rows, inner), (rows, columns))}
    return [rng.standard_normal(shape) for shape in shapes[form]]


@pytest.mark.parametrize("form", ["nt", "nn", "tn"])
@pytest.mark.parametrize("rows,inner,columns", SHAPES)
def test_narrow_tiles_give_the_bits_of_wide_tiles(form, rows, inner, columns, kernel_variant):
    from gpu_util import to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.storage import DeviceStorage

    a, b = (to_device(value, "bfloat16") for value in _operands(form, rows, inner, columns))
    m, k, n = (inner, rows, columns) if form == "tn" else (rows, inner, columns)      # tn: a weight gradient over `rows`, any number of them
    kind = "float32" if form == "tn" else "bfloat16"

    def product():
        out = DeviceStorage(m * n, kind)
        lib.call("qmoe_memset", out.ptr, 0xFF, out.nbytes, 0)       # NaN: everything has to be written
        lib.call("qmoe_gemm", a.ptr, lib.QMOE_BF16, b.ptr, lib.QMOE_BF16, out.ptr, lib.DTYPE_CODES[kind], m, k, n, int(form == "tn"), int(form == "nt"), 0, 0)
        assert lib.device_status() == 0
        return out

    narrow = product()
    kernel_variant(lib.VARIANT_SINGLE_CTA_GEMM)
    assert narrow.tobytes() == product().tobytes()
    x, y = (to_host(value, like.shape) for value, like in zip((a, b), _operands(form, rows, inner, columns)))
    exact = {"nt": lambda: x @ y.T, "nn": lambda: x @ y, "tn": lambda: x.T @ y}[form]()
    # bfloat16 has 8 significant bits: rounding moves a value by up to 2^-8 of itself (half of the last place, 2^-9, just below a power of
    # two); what is added in tensor memory loses its low bits, 2^-22 of the running sum per 16 products
    bound = (2.0 ** -8 if kind == "bfloat16" else 0.0) * np.abs(exact) + 2.0 ** -22 * (k / 16 + 4) * (np.abs(x).max() * np.abs(y).max() * np.sqrt(k) * 4)
    assert (np.abs(to_host(narrow, (m, n)) - exact) <= bound).all()
