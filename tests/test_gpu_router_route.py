"""Router logits and routing of a handful of tokens in one launch (up to 32 logits): the bits of the two launches it replaces, and with the
norm in front the exact logits within float32.  Needs a B200: ``-m gpu``."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one logit, as many as the block has warps, one token more; every expert chosen; widths that take several rounds, part of one, and no
# 16-byte pieces
SHAPES = [(1, 1, 1, 64), (4, 8, 2, 1024), (1, 32, 6, 72), (32, 1, 1, 520), (3, 9, 8, 100), (2, 8, 8, 37), (5, 8, 2, 2048)]


@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("tokens,experts,top_k,width", SHAPES)
def test_router_and_routing_in_one_launch(tokens, experts, top_k, width, dtype, norm):
    from gpu_util import RouteTables, make_layer, to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.layers import MoEFeedForward, RMSNorm, Tensor
    from qutai_b200.storage import DeviceStorage

    rng = np.random.default_rng(tokens * experts + width)
    draw = lambda *shape: rng.standard_normal(shape).astype(np.float32)
    hidden = 8
    layer = make_layer((tokens, width), draw(experts, width) * 0.3, draw(experts, hidden, width), draw(experts, hidden, width),
                       draw(experts, width, hidden), top_k)
    x = to_device(draw(tokens, width), dtype)
    call = MoEFeedForward(RMSNorm(width, 1e-6), layer) if norm else layer
    call.forward(Tensor(x, (tokens, width)))
    assert lib.device_status() == 0
    buffers = layer._saved[0]["buf"]
    scores = buffers["scores"]
    if norm:
        values, weights = to_host(x, (tokens, width)), to_host(layer.router.weight.storage, (experts, width))
        normed = values / np.sqrt((values ** 2).mean(1, keepdims=True) + 1e-6)
        # width products per logit in float32, summed by 32 lanes in four chains each: at most 2^-23 of the sum of sizes per step of a chain
        bound = 2.0 ** -23 * (width / 128 + 12) * (np.abs(normed) @ np.abs(weights).T)
        assert (np.abs(to_host(scores, (tokens, experts)) - normed @ weights.T) <= bound).all()
    else:
        apart = DeviceStorage(tokens * experts, "float32")
        lib.call("qmoe_router_forward", x.ptr, lib.DTYPE_CODES[dtype], layer.router.weight.storage.ptr, apart.ptr, 0, tokens, width, experts, 0)
        assert apart.tobytes() == scores.tobytes()
    tables = RouteTables(tokens, experts, top_k)
    tables.run(scores)
    for name in ("probs", "gate_weights", "expert_index", "dest_row", "row_source", "counts", "offsets", "meta", "utilization", "aux"):
        assert tables.buf[name].tobytes() == buffers[name].tobytes(), name
