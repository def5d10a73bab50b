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
