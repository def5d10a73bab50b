"""``qmoe_publish_counts``: per-expert counts to pinned host memory.  Needs a B200: ``-m gpu``."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("experts", [1, 31, 64, 256])
def test_counts_reach_the_host(experts):
    from gpu_util import to_device
    from qutai_b200 import lib

    host, event = ctypes.c_void_p(), ctypes.c_uint64()
    lib.call("qmoe_host_alloc", ctypes.byref(host), 4 * experts)
    lib.call("qmoe_event_create", ctypes.byref(event))
    values = np.random.default_rng(experts).integers(0, 2 ** 31 - 1, experts, dtype=np.int32)
    counts = to_device(values, "int32")
    lib.call("qmoe_publish_counts", counts.ptr, host, experts, event.value, 0)
    lib.call("qmoe_event_sync", event.value)
    assert list(ctypes.cast(host, ctypes.POINTER(ctypes.c_int32))[:experts]) == values.tolist()
    for bad in ((0, host, experts), (counts.ptr, None, experts), (counts.ptr, host, 0)):
        with pytest.raises(ValueError):
            lib.call("qmoe_publish_counts", *bad, 0, 0)
    lib.call("qmoe_event_destroy", event.value)
    lib.load().qmoe_host_free(host)


@pytest.mark.parametrize("tokens,experts,top_k", [(40, 8, 2), (3000, 64, 6)])
def test_counts_of_a_routing_enqueued_just_before(tokens, experts, top_k):
    """No wait between the routing and the kernel that hands its counts to the host, several routings in a row on the same tables."""
    from gpu_util import RouteTables, to_device
    from oracle import moe_oracle as oracle
    from qutai_b200 import lib

    rng = np.random.default_rng(tokens)
    host, event = ctypes.c_void_p(), ctypes.c_uint64()
    lib.call("qmoe_host_alloc", ctypes.byref(host), 4 * experts)
    lib.call("qmoe_event_create", ctypes.byref(event))
    tables = RouteTables(tokens, experts, top_k)
    scores = [(rng.standard_normal((tokens, experts)) + rng.standard_normal(experts)).astype(np.float32) for _ in range(6)]
    for values, storage in [(s, to_device(s, "float32")) for s in scores]:
        tables.run(storage)
        lib.call("qmoe_publish_counts", tables.buf["counts"].ptr, host, experts, event.value, 0)
        lib.call("qmoe_event_sync", event.value)
        assert tuple(ctypes.cast(host, ctypes.POINTER(ctypes.c_int32))[:experts]) == oracle.routing(values, top_k)["counts"]
    lib.call("qmoe_event_destroy", event.value)
    lib.load().qmoe_host_free(host)


def test_last_counts_are_those_of_the_last_of_two_forwards():
    from gpu_util import make_layer, to_device
    from oracle import moe_oracle as oracle
    from qutai_b200.layers import Tensor

    tokens, d, experts, top_k, hidden = 900, 128, 8, 2, 64
    rng = np.random.default_rng(3)
    router = (rng.standard_normal((experts, d)) * 0.2).astype(np.float32)
    weights = [(rng.standard_normal(shape) / 8).astype(np.float32) for shape in ((experts, hidden, d), (experts, hidden, d), (experts, d, hidden))]
    layer = make_layer((tokens, d), router, *weights, top_k)
    inputs = [rng.standard_normal((tokens, d)).astype(np.float32) * 4 for _ in range(2)]
    storages = [Tensor(to_device(x, "float32"), (tokens, d)) for x in inputs]
    wanted = [oracle.routing((x @ router.T), top_k)["counts"] for x in inputs]
    assert wanted[0] != wanted[1]
    for order in ((0, 1), (1, 0)):
        for which in order:
            layer(storages[which])
        assert layer.last_counts == wanted[order[-1]]
