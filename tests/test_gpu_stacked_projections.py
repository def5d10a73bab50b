"""``qmoe_rope_qkv`` against ``qmoe_rope`` and plain copies, bit for bit.  Needs a B200: ``-m gpu``."""
import numpy as np
import pytest

from oracle import moe_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,time,heads,kv_heads,dim", [
    (1, 1, 1, 1, 8),           # the smallest of everything: three heads in one group of eight
    (2, 5, 6, 1, 64),          # exactly one group
    (1, 7, 7, 1, 64),          # nine: the last value head alone in its group
    (3, 33, 16, 4, 64),        # keys and values in one group, positions that fill no block
    (2, 301, 9, 3, 24),        # a group that holds queries and keys, one with keys and values; three pieces per head
])
def test_projections_side_by_side_and_apart(batch, time, heads, kv_heads, dim):
    from gpu_util import to_device
    from qutai_b200 import lib
    from qutai_b200.storage import DeviceStorage

    rng = np.random.default_rng(time)
    rows, all_heads = batch * time, heads + 2 * kv_heads
    packed = oracle.round_bf16(rng.standard_normal((rows, all_heads, dim)))
    parts = np.split(packed, [heads, heads + kv_heads], axis=1)
    counts = (heads, kv_heads, kv_heads)

    def rotated(values, count, inverse):
        out = DeviceStorage(values.size, "bfloat16")
        lib.call("qmoe_rope", values.ptr, out.ptr, lib.QMOE_BF16, batch, time, count, dim, 10000.0, 3, inverse, 0)
        return out

    def bits(storage, count):
        return np.frombuffer(storage.tobytes(), dtype=np.uint16).reshape(rows, count, dim)

    devices = [to_device(part, "bfloat16") for part in parts]
    out = [DeviceStorage(rows * count * dim, "bfloat16") for count in counts]
    lib.call("qmoe_rope_qkv", to_device(packed, "bfloat16").ptr, *(o.ptr for o in out), batch, time, heads, kv_heads, dim, 10000.0, 3, 0, 0)
    want = [rotated(devices[0], heads, 0), rotated(devices[1], kv_heads, 0), devices[2]]
    for got, expected, count in zip(out, want, counts):
        assert np.array_equal(bits(got, count), bits(expected, count))
    together = DeviceStorage(packed.size, "bfloat16")
    lib.call("qmoe_rope_qkv", together.ptr, *(d.ptr for d in devices), batch, time, heads, kv_heads, dim, 10000.0, 3, 1, 0)
    want = [rotated(devices[0], heads, 1), rotated(devices[1], kv_heads, 1), devices[2]]
    assert np.array_equal(bits(together, all_heads), np.concatenate([bits(w, count) for w, count in zip(want, counts)], axis=1))
    with pytest.raises(ValueError):
        lib.call("qmoe_rope_qkv", together.ptr + 2, *(d.ptr for d in devices), batch, time, heads, kv_heads, dim, 10000.0, 0, 0, 0)
    with pytest.raises(ValueError):
        lib.call("qmoe_rope_qkv", together.ptr, *(d.ptr for d in devices), batch, time, heads, kv_heads, dim - 2, 10000.0, 0, 0, 0)
