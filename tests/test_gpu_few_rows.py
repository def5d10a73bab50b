"""Few rows per expert: the weight-streaming forward products (``stream_gemm_kernel``) against the kernel for many rows, and
the one-block routing against the oracle, at the sizes where either can go wrong.  Needs a B200: ``-m gpu``."""
import numpy as np
import pytest

from oracle import moe_oracle as oracle

pytestmark = pytest.mark.gpu


# 64 experts, 50 rows on average: enough tiles of 256 columns for the down product that holds two weight tiles per stage
MANY = (0, 127, 128, 129, 300, 1, 15, 17) + (33, 0, 64, 31, 49, 96, 2, 48) * 7


@pytest.mark.parametrize("counts,width,hidden", [
    ((0, 1, 15, 16, 17), 64, 128),           # around one 16-row step, an expert without rows
    ((127, 128, 129, 0, 3), 72, 136),        # around one 128-row chunk, widths that fill no tile
    ((300, 2, 0, 40, 33), 264, 1032),        # an expert with three chunks, several k blocks and tiles
    ((1,), 2048, 8),                         # one row, the narrowest hidden width
    (MANY, 648, 136),                        # the last 256-column tile of the down product holds 136, one full weight tile and 8 columns
    (MANY, 584, 136),                        # it holds 72: the second weight tile lies outside, at the last expert behind the last weight
    (MANY, 768, 200),                        # whole tiles
])
def test_streamed_products_match_the_kernel_for_many_rows(counts, width, hidden, kernel_variant):
    import ctypes

    from gpu_util import RouteTables, to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.storage import DeviceStorage

    experts, tokens = len(counts), sum(counts)
    if counts is MANY:      # the rule for two weight tiles per stage
        assert 32 * experts < tokens <= 96 * experts and -(-width // 256) * experts >= lib.device_info()["sm_count"]
    rng = np.random.default_rng(tokens + width)
    choice = np.repeat(np.arange(experts), counts)
    scores = np.zeros((tokens, experts), dtype=np.float32)
    scores[np.arange(tokens), rng.permutation(choice)] = 5.0
    tables = RouteTables(tokens, experts, 1)
    tables.run(to_device(scores, "float32"))
    assert tuple(tables.host("counts").tolist()) == counts
    rows = tables.rows_bound
    x = to_device(rng.standard_normal((tokens, width)), "bfloat16")
    weights = [to_device(rng.standard_normal(shape) / np.sqrt(shape[-1]), "bfloat16")
               for shape in ((experts, hidden, width), (experts, hidden, width), (experts, width, hidden))]
    dispatched = DeviceStorage(rows * width, "bfloat16")
    lib.call("qmoe_permute", tables.ref, x.ptr, dispatched.ptr, lib.QMOE_BF16, width, 0)
    ex = lib.Experts()
    ex.experts, ex.dtype, ex.engine, ex.width, ex.hidden = experts, lib.QMOE_BF16, lib.ENGINE_TCGEN05, width, hidden
    ex.w_gate, ex.w_up, ex.w_down = (w.ptr for w in weights)
    used = int(tables.host("offsets")[experts])

    def forward():
        g, u, h, y = (DeviceStorage(rows * n, "bfloat16") for n in (hidden, hidden, hidden, width))
        for buffer in (g, u, h, y):
            lib.call("qmoe_memset", buffer.ptr, 0xFF, buffer.nbytes, 0)       # NaN: every row of a tile has to be written
        lib.call("qmoe_expert_forward", tables.ref, ctypes.byref(ex), dispatched.ptr, g.ptr, u.ptr, h.ptr, y.ptr, 0)
        assert lib.device_status() == 0
        return [to_host(b, (rows, -1))[:used] for b in (g, u, h, y)]

    streamed = forward()
    kernel_variant(lib.VARIANT_NO_STREAM_GEMM)
    for got, want in zip(streamed, forward()):
        assert np.all(np.isfinite(got))
        # the same fp32 sums in another order, rounded to bf16: at most one step (2^-8) of the largest value apart
        assert oracle.max_rel_err(got, want) <= 2.0 ** -7
    source = tables.host("row_source")[:used]
    for got in streamed:
        assert not np.any(got[source < 0])                                    # pad rows hold zeros


@pytest.mark.parametrize("tokens,experts,top_k", [(1, 1, 1), (1, 256, 8), (31, 33, 4), (33, 32, 3), (128, 256, 8), (128, 64, 6), (129, 64, 6), (97, 5, 5)])
def test_one_block_routing_matches_the_oracle(tokens, experts, top_k):
    """Both sides of the token limit, every width of a lane's expert list, ties, and scores of the lowest values."""
    from gpu_util import RouteTables, check_route_against_oracle, to_device

    rng = np.random.default_rng(tokens * 3 + experts)
    scores = rng.standard_normal((tokens, experts)).astype(np.float32)
    scores[:, ::3] = np.round(scores[:, ::3])                                 # ties, zeros of both signs among them
    scores[tokens // 2] = -0.0
    scores[-1, : experts // 2] = np.finfo(np.float32).min
    tables = RouteTables(tokens, experts, top_k)
    tables.run(to_device(scores, "float32"))
    check_route_against_oracle(tables, oracle.routing(scores, top_k))
    # readers of the per-block probability sums add them over the blocks
    sums = tables.host("block_colsum", (-1, experts)).sum(axis=0)
    assert np.abs(sums - tables.host("probs", (tokens, experts)).sum(axis=0)).max() <= 1e-5 * tokens


def test_a_layer_of_few_rows_reads_no_pad_row_it_did_not_write():
    """Inside a layer call the pad rows of few-row experts are zeroed only to a multiple of 16 rows: with every workspace
    buffer full of NaN beforehand, forward and backward give the same bits as with a fresh workspace."""
    from gpu_util import make_layer, run_layer
    from qutai_b200 import lib

    T, d, E, k, h = 70, 136, 6, 2, 264
    rng = np.random.default_rng(5)
    x, grad_y = (oracle.round_bf16(rng.standard_normal((T, d))) for _ in range(2))
    router = rng.standard_normal((E, d)).astype(np.float32) * 0.05
    gate, up = (rng.standard_normal((E, h, d)).astype(np.float32) / np.sqrt(d) for _ in range(2))
    down = rng.standard_normal((E, d, h)).astype(np.float32) / np.sqrt(h)
    layer = make_layer(x.shape, router, gate, up, down, k, engine="tcgen05")
    first = run_layer(layer, x, grad_y, 0.5, "bfloat16")
    buf = layer._saved[0]["buf"]
    for name in ("x_dispatched", "g", "u", "h", "y_dispatched", "dy_dispatched", "d_h", "d_g", "d_u"):
        lib.call("qmoe_memset", buf[name].ptr, 0xFF, buf[name].nbytes, 0)
    again = run_layer(layer, x, grad_y, 0.5, "bfloat16")
    assert first["counts"] == again["counts"]
    for name in ("y", "dx", "d_router"):
        assert np.array_equal(first[name], again[name]), name
    for name in ("d_gate", "d_up", "d_down"):
        for a, b in zip(first[name], again[name]):
            assert (a is None and b is None) or np.array_equal(a, b), name


@pytest.mark.parametrize("with_norm", [False, True])
def test_layer_calls_fill_every_pad_row_unless_asked_not_to(with_norm):
    """The dispatched buffers of a whole-layer (whole-block) call, full of NaN beforehand: every pad row is zero afterwards, as the
    layout promises, for a caller that has not set ``EXPERTS_SHORT_PADS``; one that has gets the same output."""
    import ctypes

    from gpu_util import make_layer, to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.layers import MoEFeedForward, RMSNorm, Tensor

    T, d, E, k, h = 70, 136, 6, 2, 264
    rng = np.random.default_rng(6)
    x = Tensor(to_device(rng.standard_normal((T, d)), "bfloat16"), (T, d))
    router = rng.standard_normal((E, d)).astype(np.float32) * 0.05
    gate, up = (rng.standard_normal((E, h, d)).astype(np.float32) / np.sqrt(d) for _ in range(2))
    down = rng.standard_normal((E, d, h)).astype(np.float32) / np.sqrt(h)
    layer = make_layer((T, d), router, gate, up, down, k, engine="tcgen05")
    call = MoEFeedForward(RMSNorm(d, 1e-6), layer) if with_norm else layer
    out, _ = call.forward(x)
    work = layer._saved[0]
    buf, struct = work["buf"], call._blocks[id(work)]["struct"] if with_norm else work["layer"]
    experts = struct.layer.experts if with_norm else struct.experts
    assert experts.reserved == lib.EXPERTS_SHORT_PADS
    first, experts.reserved = out.storage.tobytes(), 0
    names = ("x_dispatched", "g", "u", "h", "y_dispatched")
    for name in names:
        lib.call("qmoe_memset", buf[name].ptr, 0xFF, buf[name].nbytes, 0)
    lib.call("qmoe_block_forward" if with_norm else "qmoe_layer_forward", ctypes.byref(struct), 0)
    assert out.storage.tobytes() == first and lib.device_status() == 0
    used = int(to_host(buf["offsets"])[E])
    pads = to_host(buf["row_source"])[:used] < 0
    for name in names:
        rows = to_host(buf[name], (work["rows_bound"], -1))[:used]
        assert np.all(np.isfinite(rows)) and not np.any(rows[pads]), name
