"""The per-op backend function table (``qutai_b200.cuda_lm``) against the oracle, written after the
upstream GPU tests of the same functions (tests/test_lm_moe.py:140-162,
tests/test_lm_bfloat16.py:129-167, tests/test_gemm_precision.py)."""
import os

import numpy as np
import pytest

from conftest import golden_files
from oracle import moe_oracle as oracle

pytestmark = pytest.mark.gpu


def close(actual, expected, tolerance):
    actual, expected = np.asarray(actual, dtype=np.float64), np.asarray(expected, dtype=np.float64)
    assert actual.shape == expected.shape
    assert np.all(np.abs(actual - expected) <= tolerance * np.maximum(1.0, np.abs(expected)))


def test_route_pack_has_stable_token_slot_order_across_blocks():
    from gpu_util import to_device, to_host
    from qutai_b200 import cuda_lm

    rows, experts, top_k = 517, 5, 3
    scores = np.array([[((row * 37 + expert * 11) % 101) / 13 for expert in range(experts)] for row in range(rows)],
                      dtype=np.float32)
    reference = oracle.routing(scores.astype(np.float64), top_k)
    values = to_device(scores, "float32")
    for _ in range(3):
        route = cuda_lm.routing(values, rows, experts, top_k)
        assert route["counts"] == reference["counts"]
        for expert, count in enumerate(route["counts"]):
            ids = to_host(cuda_lm.take(route["ids"], expert * route["capacity"], count))
            slots = to_host(cuda_lm.take(route["slots"], expert * route["capacity"], count))
            assert np.array_equal(ids, reference["ids"][expert])
            assert np.array_equal(slots, reference["slots"][expert])
        assert np.array_equal(to_host(route["indices"]).reshape(rows, top_k), reference["indices"])
        assert np.array_equal(to_host(route["locations"]).reshape(rows, top_k), reference["locations"])


def test_router_fp32_and_bfloat16_expert_gather_combine():
    from gpu_util import to_device, to_host
    from qutai_b200 import cuda_lm

    scores = np.array([[3, 1, -2], [0, 2, 1], [1, -2, 4], [-1, 3, 2], [4, 0, 1]], dtype=np.float32)
    raw_values = np.array([0.03 * i - 0.2 for i in range(20)]).reshape(5, 4)
    raw_gradient = np.array([0.05 * i - 0.4 for i in range(20)]).reshape(5, 4)
    values, gradient = to_device(raw_values, "bfloat16"), to_device(raw_gradient, "bfloat16")
    reference, reference_g = oracle.round_bf16(raw_values), oracle.round_bf16(raw_gradient)
    route = cuda_lm.routing(to_device(scores, "float32"), 5, 3, 2)
    outputs = tuple((e, cuda_lm.route_gather(values, route, e, 4)) for e in range(3) if route["counts"][e])
    combined = cuda_lm.combine(outputs, route["weights"], route, 4)
    gradients = cuda_lm.combine_backward(gradient, outputs, route["weights"], route, 4)
    cpu_route = oracle.routing(scores.astype(np.float64), 2)
    assert route["counts"] == cpu_route["counts"] == (3, 3, 4)
    cpu_outputs = [(e, oracle.route_gather(reference, cpu_route, e)) for e in range(3) if cpu_route["counts"][e]]
    expected = oracle.combine(cpu_outputs, cpu_route["weights"], cpu_route)
    expected_dy, expected_dw = oracle.combine_backward(reference_g, cpu_outputs, cpu_route["weights"], cpu_route)
    assert (route["weights"].dtype, route["aux"].dtype, combined.dtype) == ("float32", "float32", "bfloat16")
    assert combined.nbytes == 40
    close(to_host(combined, (5, 4)), expected, 0.012)
    for (e, storage), want_rows in zip(outputs, cpu_outputs):
        assert np.array_equal(to_host(storage).reshape(-1, 4), want_rows[1])
    for actual, want in zip(gradients[:-1], expected_dy):
        close(to_host(actual).reshape(-1, 4), want, 0.012)
    assert gradients[-1].dtype == "float32"
    close(to_host(gradients[-1], (5, 2)), expected_dw, 0.012)
    # bfloat16 scores are widened exactly before routing
    again = cuda_lm.routing(to_device(scores, "bfloat16"), 5, 3, 2)
    assert again["counts"] == route["counts"] and np.array_equal(to_host(again["indices"]), to_host(route["indices"]))
    # routing backward: both paths
    g = np.random.default_rng(0).standard_normal((5, 2)).astype(np.float32)
    close(to_host(cuda_lm.routing_backward(to_device(g, "float32"), route), (5, 3)), oracle.routing_backward(g, cpu_route), 1e-5)
    close(to_host(cuda_lm.routing_backward(to_device(np.array([0.5]), "float32"), route, True), (5, 3)),
          oracle.routing_backward([0.5], cpu_route, True), 1e-5)


@pytest.mark.parametrize("transpose_left", [False, True])
@pytest.mark.parametrize("transpose_right", [False, True])
def test_gemm_transposes_mixed_precision_and_accumulate(transpose_left, transpose_right):
    from gpu_util import to_device, to_host
    from qutai_b200 import cuda_lm

    rows, inner, cols = 65, 129, 33     # partial tiles in every dimension
    rng = np.random.default_rng(3)
    a, b = rng.standard_normal((rows, inner)), rng.standard_normal((inner, cols))
    a16, b32 = oracle.round_bf16(a), b.astype(np.float32).astype(np.float64)
    left = to_device(a16.T if transpose_left else a16, "bfloat16")
    right = to_device(b32.T if transpose_right else b32, "float32")
    kw = dict(transpose_left=transpose_left, transpose_right=transpose_right)
    product = a16 @ b32
    out = cuda_lm.gemm(left, right, rows, inner, cols, **kw)
    assert out.dtype == "float32"
    close(to_host(out, (rows, cols)), product, 5e-5)   # fp32 accumulation of 129 products
    rounded = cuda_lm.gemm(left, right, rows, inner, cols, out_dtype="bfloat16", **kw)
    assert rounded.dtype == "bfloat16" and rounded.nbytes == rows * cols * 2
    assert np.array_equal(to_host(rounded, (rows, cols)), oracle.round_bf16(to_host(out, (rows, cols))))  # RNE of the fp32 result
    cuda_lm.gemm(left, right, rows, inner, cols, out=out, accumulate=True, **kw)
    close(to_host(out, (rows, cols)), 2 * product, 5e-5)
    with pytest.raises(ValueError):
        cuda_lm.gemm(left, right, rows, inner, cols, accumulate=True, **kw)          # accumulate needs out
    square = to_device(np.eye(16), "float32")
    with pytest.raises(ValueError):
        cuda_lm.gemm(square, square, 16, 16, 16, out=square)                           # out must not overlap an input
    with pytest.raises(ValueError):
        cuda_lm.gemm(square, square, 16, 16, 16, out_dtype="float64")


def test_gemm_long_inner_dimension_keeps_fp32_sums():
    from gpu_util import to_device, to_host
    from qutai_b200 import cuda_lm

    rows, inner, cols = 129, 8193, 65
    a, b = np.ones((rows, inner)), np.full((inner, cols), 0.5)
    out = cuda_lm.gemm(to_device(a, "bfloat16"), to_device(b, "bfloat16"), rows, inner, cols)
    assert np.array_equal(to_host(out, (rows, cols)), np.full((rows, cols), inner * 0.5))  # exact in fp32


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_silu_forward_and_backward(dtype):
    from gpu_util import to_device, to_host
    from qutai_b200 import cuda_lm

    rng = np.random.default_rng(4)
    rnd = oracle.round_bf16 if dtype == "bfloat16" else (lambda v: v.astype(np.float32).astype(np.float64))
    x, g = rnd(rng.standard_normal(1000) * 4), rnd(rng.standard_normal(1000))
    x[:4] = [0.0, -80.0, 80.0, -1e-3]
    x = rnd(x)
    tol = 0.012 if dtype == "bfloat16" else 2e-6
    close(to_host(cuda_lm.silu(to_device(x, dtype))), oracle.silu(x), tol)
    close(to_host(cuda_lm.silu_backward(to_device(g, dtype), to_device(x, dtype))), oracle.silu_backward(g, x), tol)


def test_upstream_style_expert_loop_matches_golden_layer():
    """The upstream ``SparseMoE.__call__`` written against this function table
    (src/qutai/lm/layers.py:376-402) reproduces the golden fixture of the upstream CPU layer."""
    from gpu_util import to_device, to_host
    from qutai_b200 import cuda_lm as b

    g = np.load(os.path.join(os.path.dirname(golden_files("layer")[0]), "layer_mid.npz"))
    T, d = g["x"].shape
    E, h = g["gate"].shape[0], g["gate"].shape[1]
    k = int(g["top_k"])
    x = to_device(g["x"], "float32")
    scores = b.gemm(x, to_device(g["router"], "float32"), T, d, E, transpose_right=True)
    route = b.routing(scores, T, E, k)
    assert route["counts"] == tuple(g["counts"].tolist())
    outputs = []
    for e in range(E):
        if route["counts"][e]:
            xe, c = b.route_gather(x, route, e, d), route["counts"][e]
            gate = b.gemm(xe, to_device(g["gate"][e], "float32"), c, d, h, transpose_right=True)
            up = b.gemm(xe, to_device(g["up"][e], "float32"), c, d, h, transpose_right=True)
            act = b.silu(gate)
            outputs.append((e, (act, up, c)))
    # element-wise product silu(gate) * up through the table's gemm is not available; use numpy for that one op
    ys = []
    for e, (act, up, c) in outputs:
        hidden = to_device(to_host(act) * to_host(up), "float32")
        ys.append((e, b.gemm(hidden, to_device(g["down"][e], "float32"), c, h, d, transpose_right=True)))
    y = b.combine(tuple(ys), route["weights"], route, d)
    assert oracle.max_rel_err(to_host(y, (T, d)), g["y"]) <= 1e-4
    assert abs(to_host(route["aux"])[0] - float(g["aux"])) <= 1e-5
    # gather backward of one expert: rows scattered into zeros
    e0 = ys[0][0]
    grad_rows = np.random.default_rng(1).standard_normal((route["counts"][e0], d)).astype(np.float32)
    scattered = to_host(b.route_gather_backward(to_device(grad_rows, "float32"), route, e0, d), (T, d))
    cpu_route = oracle.routing(to_host(scores, (T, E)), k)
    assert np.array_equal(scattered, oracle.route_gather_backward(grad_rows, cpu_route, e0))


@pytest.mark.parametrize("rows,inner,cols", [(128, 64, 72), (384, 1024, 264), (1024, 264, 1024)])
def test_gemm_takes_the_tensor_cores_for_the_three_products_of_a_linear_layer(rows, inner, cols, kernel_variant):
    """bf16 x bf16 in the forms of a linear layer's forward (x W^T), input gradient (g W) and weight gradient
    (g^T x, float32) run on the tcgen05 kernels when the sizes allow, and give what the CUDA-core kernel gives."""
    from gpu_util import to_device, to_host
    from qutai_b200 import cuda_lm, lib

    rng = np.random.default_rng(rows + cols)
    x, w = oracle.round_bf16(rng.standard_normal((rows, inner))), oracle.round_bf16(rng.standard_normal((cols, inner)) * 0.1)
    g = oracle.round_bf16(rng.standard_normal((rows, cols)))
    xs, ws, gs = to_device(x, "bfloat16"), to_device(w, "bfloat16"), to_device(g, "bfloat16")
    count = lib.load().qmoe_tensor_core_launch_count

    def products():
        y = cuda_lm.gemm(xs, ws, rows, inner, cols, transpose_right=True, out_dtype="bfloat16")
        dx = cuda_lm.gemm(gs, ws, rows, cols, inner, out_dtype="bfloat16")
        dw = cuda_lm.gemm(gs, xs, cols, rows, inner, transpose_left=True, out_dtype="float32")
        return to_host(y, (rows, cols)), to_host(dx, (rows, inner)), to_host(dw, (cols, inner))

    before = count()
    fast = products()
    assert count() - before == 3
    kernel_variant(lib.VARIANT_PLAIN_GEMM_ON_CUDA_CORES)
    before = count()
    slow = products()
    assert count() == before
    for got, reference, exact in zip(fast, slow, (x @ w.T, g @ w, g.T @ x)):
        assert oracle.max_rel_err(got, exact) <= 1e-2
        assert oracle.max_rel_err(got, reference) <= 8e-3          # both round fp32 sums of the same products to bf16 (or keep fp32)
    # a row count that is not a multiple of 128 stays on the CUDA cores (a tile of the tensor-core kernel writes 128 rows)
    kernel_variant(lib.VARIANT_PLAIN_GEMM_ON_CUDA_CORES, 0)
    before = count()
    cuda_lm.gemm(to_device(x[:100], "bfloat16"), ws, 100, inner, cols, transpose_right=True, out_dtype="bfloat16")
    assert count() == before


@pytest.mark.parametrize("rows,cols_out,cols_in", [(8192, 1024, 1024), (4104, 256, 1024), (1096, 512, 264)])
def test_split_weight_gradient_of_a_linear_layer(rows, cols_out, cols_in):
    """``qmoe_gemm_wgrad_split``: g^T x with the rows cut into ranges that run side by side, the ranges' products
    added in a fixed order — the value of the one-launch product, the same bits on every run; row counts that leave a
    ragged last range included."""
    from gpu_util import to_device, to_host
    from qutai_b200 import cuda_lm, lib
    from qutai_b200.storage import DeviceStorage

    rng = np.random.default_rng(rows)
    x, g = oracle.round_bf16(rng.standard_normal((rows, cols_in))), oracle.round_bf16(rng.standard_normal((rows, cols_out)))
    xs, gs = to_device(x, "bfloat16"), to_device(g, "bfloat16")
    partials = lib.load().qmoe_gemm_wgrad_partials(cols_out, rows, cols_in)
    assert partials > 64 + cols_out * cols_in                 # these shapes are split
    scratch, out = DeviceStorage(partials, "float32"), DeviceStorage(cols_out * cols_in, "float32")
    results = []
    for _ in range(2):
        lib.call("qmoe_gemm_wgrad_split", gs.ptr, xs.ptr, out.ptr, scratch.ptr, cols_out, rows, cols_in, 0)
        results.append(to_host(out, (cols_out, cols_in)))
    assert np.array_equal(results[0], results[1])
    assert lib.device_status() == 0
    assert oracle.max_rel_err(results[0], g.T @ x) <= 1e-5
    whole = to_host(cuda_lm.gemm(gs, xs, cols_out, rows, cols_in, transpose_left=True, out_dtype="float32"), (cols_out, cols_in))
    assert oracle.max_rel_err(results[0], whole) <= 1e-5
    # a shape with enough tiles of its own is not split, and the call says so
    assert lib.load().qmoe_gemm_wgrad_partials(32000, 8192, 1024) == 0
    with pytest.raises(ValueError):
        lib.call("qmoe_gemm_wgrad_split", gs.ptr, xs.ptr, out.ptr, scratch.ptr, 32000, 8192, 1024, 0)


@pytest.mark.parametrize("rows,inner,cols", [(129, 64, 72), (200, 264, 512), (602, 512, 128), (1001, 1024, 264)])
def test_gemm_takes_ragged_row_counts_to_the_tensor_cores(rows, inner, cols, kernel_variant):
    """Row counts that fill no whole tile: the three products of a linear layer give what the CUDA-core kernel gives, and
    what lies behind the last row of a result keeps its bits."""
    from gpu_util import to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.storage import DeviceStorage

    rng = np.random.default_rng(rows)
    x, w = oracle.round_bf16(rng.standard_normal((rows, inner))), oracle.round_bf16(rng.standard_normal((cols, inner)) * 0.1)
    g = oracle.round_bf16(rng.standard_normal((rows, cols)))
    xs, ws, gs = to_device(x, "bfloat16"), to_device(w, "bfloat16"), to_device(g, "bfloat16")
    bf16, f32 = lib.QMOE_BF16, lib.QMOE_F32
    count = lib.load().qmoe_tensor_core_launch_count

    def product(a, b, m, k, n, ta, tb, dtype, code):
        out = DeviceStorage((m + 3) * n, dtype)
        lib.call("qmoe_memset", out.ptr, 0x3C, out.nbytes, 0)
        lib.call("qmoe_gemm", a.ptr, bf16, b.ptr, bf16, out.ptr, code, m, k, n, ta, tb, 0, 0)
        raw = np.frombuffer(out.tobytes(), dtype=np.uint8)
        assert np.all(raw[m * n * (2 if code == bf16 else 4):] == 0x3C)
        return to_host(out, (m + 3, n))[:m]

    def products():
        return (product(xs, ws, rows, inner, cols, 0, 1, "bfloat16", bf16), product(gs, ws, rows, cols, inner, 0, 0, "bfloat16", bf16),
                product(gs, xs, cols, rows, inner, 1, 0, "float32", f32))

    before = count()
    fast = products()
    assert count() - before == 3
    kernel_variant(lib.VARIANT_PLAIN_GEMM_ON_CUDA_CORES)
    for got, slow, exact in zip(fast, products(), (x @ w.T, g @ w, g.T @ x)):
        assert oracle.max_rel_err(got, exact) <= 1e-2
        assert oracle.max_rel_err(got, slow) <= 8e-3
    assert lib.device_status() == 0


# Whether a float32 product runs on the 128 x 128 tiles: the last column.  Ragged edges, an inner size that is no multiple of the
# 16-deep slice (100, 20, 36) or, where no pitch is made of it, of a 16-byte piece (37), narrow and few tiles.
@pytest.mark.parametrize("m,k,n,ta,tb,tiles", [
    *((m, k, n, ta, tb, True) for m, k, n in ((1028, 100, 1156), (1284, 20, 1284), (9476, 16, 132), (1160, 520, 1032)) for ta in (0, 1) for tb in (0, 1)),
    (1284, 37, 1156, 1, 0, True), (1284, 17, 1156, 1, 0, True), (1281, 36, 1155, 0, 1, True),
    (9476, 4, 132, 0, 1, False), (1284, 15, 1156, 1, 0, False), (1284, 37, 1156, 0, 1, False), (1284, 37, 1156, 1, 1, False), (1282, 36, 1156, 1, 0, False),
    *((m, k, n, ta, tb, False) for m, k, n in ((128, 16, 128), (1000, 37, 900), (4097, 100, 132), (700, 260, 1028)) for ta in (0, 1) for tb in (0, 1)),
    (9600, 36, 64, 0, 1, False), (64, 36, 9600, 0, 1, False)])
def test_float32_gemm_in_every_orientation(m, k, n, ta, tb, tiles, kernel_variant):
    """float32 products on the 128 x 128 tiles and on the general kernel: one fp32 FMA chain per output in the same order, so the
    same bits, and an error of at most k roundings of sums of |a||b|.  The
    dispatch rule is restated here, so that no case misses the kernel it is for."""
    from gpu_util import to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.storage import DeviceStorage

    pitches = (m if ta else k, k if tb else n)
    assert tiles == (min(m, n) > 64 and k >= 16 and all(pitch % 4 == 0 for pitch in pitches) and -(-m // 128) * -(-n // 128) * 2 >= lib.device_info()["sm_count"])
    rng = np.random.default_rng(m + k + n)
    a, b = (rng.standard_normal(shape).astype(np.float32) for shape in ((k, m) if ta else (m, k), (n, k) if tb else (k, n)))
    sa, sb = to_device(a, "float32"), to_device(b, "float32")

    def product():
        out = DeviceStorage((m + 1) * n, "float32")
        lib.call("qmoe_memset", out.ptr, 0x3C, out.nbytes, 0)
        lib.call("qmoe_gemm", sa.ptr, lib.QMOE_F32, sb.ptr, lib.QMOE_F32, out.ptr, lib.QMOE_F32, m, k, n, ta, tb, 0, 0)
        return out

    first = product()
    kernel_variant(lib.VARIANT_NO_FLOAT32_TILES)
    assert first.tobytes() == product().tobytes()                     # the row behind the result included
    got = to_host(first, (m + 1, n))[:m]
    a64, b64 = (a.T if ta else a).astype(np.float64), (b.T if tb else b).astype(np.float64)
    bound = k * 2.0 ** -24 * (np.abs(a64) @ np.abs(b64)) * 1.01
    assert np.all(np.abs(got - a64 @ b64) <= bound)


def test_float32_gemm_with_more_row_tiles_than_a_grid_axis():
    """x W^T goes one product per launch with a row of tiles per step of the grid's y axis, which ends at 65535; beyond, the tiles
    follow one another in x.  The rows around that line and the last ones, to k roundings of sums of |a||b|."""
    from gpu_util import to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.storage import DeviceStorage

    m, k, n = 65535 * 128 + 5, 16, 68
    a, out = DeviceStorage(m * k, "float32"), DeviceStorage(m * n, "float32")
    a.fill_normal(0.0, 1.0, 7)
    b = np.random.default_rng(7).standard_normal((n, k)).astype(np.float32)
    sb = to_device(b, "float32")
    lib.call("qmoe_gemm", a.ptr, lib.QMOE_F32, sb.ptr, lib.QMOE_F32, out.ptr, lib.QMOE_F32, m, k, n, 0, 1, 0, 0)
    for first, rows in ((0, 130), (m - 140, 140)):
        x = to_host(a.view(first * k, rows * k), (rows, k)).astype(np.float64)
        got = to_host(out.view(first * n, rows * n), (rows, n))
        assert np.all(np.abs(got - x @ b.T.astype(np.float64)) <= k * 2.0 ** -24 * (np.abs(x) @ np.abs(b.T.astype(np.float64))) * 1.01)


@pytest.mark.parametrize("rows,cols_out,cols_in", [(129, 64, 72), (301, 264, 512), (602, 512, 136), (1001, 1024, 264), (4503, 128, 256)])
def test_ragged_weight_gradients_are_as_exact_as_an_fma_chain(rows, cols_out, cols_in, kernel_variant):
    """bf16 operands, fp32 result, a row count that is no multiple of 8: the tensor cores take the rows in pieces that are added
    in fp32, and the result is no further from the exact product than the CUDA cores' chain of fp32 FMAs.  Two pieces, pieces of
    every length from 64 to 512 rows, and ragged last ones; with terms of both signs and of one sign."""
    from gpu_util import to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.storage import DeviceStorage

    rng = np.random.default_rng(rows)
    count = lib.load().qmoe_tensor_core_launch_count

    def error(g, x, launches):
        gs, xs, out, before = to_device(g, "bfloat16"), to_device(x, "bfloat16"), DeviceStorage(cols_out * cols_in, "float32"), count()
        lib.call("qmoe_gemm", gs.ptr, lib.QMOE_BF16, xs.ptr, lib.QMOE_BF16, out.ptr, lib.QMOE_F32, cols_out, rows, cols_in, 1, 0, 0, 0)
        exact = g.astype(np.float64).T @ x.astype(np.float64)
        difference = np.linalg.norm(to_host(out, exact.shape) - exact) / np.linalg.norm(exact)
        assert count() - before == launches and lib.device_status() == 0
        return difference

    operands = [oracle.round_bf16(rng.standard_normal((rows, n))) for n in (cols_out, cols_in)]
    both_signs, one_sign = operands, [np.abs(a) for a in operands]
    pieces = [error(*o, 1) for o in (both_signs, one_sign)]
    kernel_variant(lib.VARIANT_PLAIN_GEMM_ON_CUDA_CORES)
    for got, chain in zip(pieces, (error(*o, 0) for o in (both_signs, one_sign))):
        assert got <= chain


@pytest.mark.parametrize("rows", [1, 7, 127])
def test_short_ragged_weight_gradients_stay_on_the_cuda_cores(rows):
    from gpu_util import to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.storage import DeviceStorage

    rng = np.random.default_rng(rows)
    g, x = (oracle.round_bf16(rng.standard_normal((rows, n))) for n in (64, 72))
    gs, xs, out, before = to_device(g, "bfloat16"), to_device(x, "bfloat16"), DeviceStorage(64 * 72, "float32"), lib.load().qmoe_tensor_core_launch_count()
    lib.call("qmoe_gemm", gs.ptr, lib.QMOE_BF16, xs.ptr, lib.QMOE_BF16, out.ptr, lib.QMOE_F32, 64, rows, 72, 1, 0, 0, 0)
    assert lib.load().qmoe_tensor_core_launch_count() == before
    g64, x64 = g.astype(np.float64), x.astype(np.float64)
    assert np.all(np.abs(to_host(out, (64, 72)) - g64.T @ x64) <= rows * 2.0 ** -24 * (np.abs(g64).T @ np.abs(x64)) * 1.01)


@pytest.mark.parametrize("rows,inner,tensor_cores", [(129, 32, 0), (4503, 56, 0), (129, 64, 1), (256, 8, 1), (128, 32, 1), (127, 64, 0)])
def test_thin_ragged_products_stay_on_the_cuda_cores(rows, inner, tensor_cores):
    from gpu_util import to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.storage import DeviceStorage

    rng = np.random.default_rng(rows + inner)
    x, w = (oracle.round_bf16(rng.standard_normal((n, inner))) for n in (rows, 72))
    xs, ws, out = to_device(x, "bfloat16"), to_device(w, "bfloat16"), DeviceStorage(rows * 72, "bfloat16")
    before = lib.load().qmoe_tensor_core_launch_count()
    lib.call("qmoe_gemm", xs.ptr, lib.QMOE_BF16, ws.ptr, lib.QMOE_BF16, out.ptr, lib.QMOE_BF16, rows, inner, 72, 0, 1, 0, 0)
    assert lib.load().qmoe_tensor_core_launch_count() - before == tensor_cores
    exact = x.astype(np.float64) @ w.astype(np.float64).T
    # one rounding to bf16 of an fp32 sum
    assert np.all(np.abs(to_host(out, exact.shape) - exact) <= 2.0 ** -8 * np.abs(exact) + inner * 2.0 ** -23 * (np.abs(x) @ np.abs(w).T))
