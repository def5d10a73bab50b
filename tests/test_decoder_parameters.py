"""``Decoder.parameters`` (what an optimizer trains) against ``Decoder.named_parameters`` (what a checkpoint holds), on a fake
allocator (no GPU)."""
import ctypes
from itertools import count

import pytest

from qutai_b200 import lib, storage
from qutai_b200.decoder import Config, Decoder
from qutai_b200.layers import Tensor
from qutai_b200.storage import DeviceStorage

CONFIG = Config(vocab_size=16, d_model=64, n_heads=1, n_kv_heads=1, n_layers=2, n_experts=3, top_k=1, d_expert=8)


class Extended(Decoder):
    def named_parameters(self):
        return [*super().named_parameters(), ("scale", self.scale)]


@pytest.mark.parametrize("kind", [Decoder, Extended])
def test_parameters_are_the_named_ones_in_their_order(monkeypatch, kind):
    class FakeDevice:
        def qmoe_free(self, address):
            return 0

    addresses = count(1 << 20, 1 << 20)

    def call(name, *args):
        if name == "qmoe_malloc":
            ctypes.cast(args[0], ctypes.POINTER(ctypes.c_uint64))[0] = next(addresses)

    monkeypatch.setattr(lib, "load", FakeDevice)
    monkeypatch.setattr(lib, "call", call)
    monkeypatch.setattr(storage, "_cache", {})
    monkeypatch.setattr(storage, "_cached_bytes", 0)
    model = kind(CONFIG, seed=0)
    model.scale = Tensor(DeviceStorage(1, "float32"), (), requires_grad=True)
    named = [parameter for _, parameter in model.named_parameters()]
    assert len(named) == (3 if kind is Extended else 2) + CONFIG.n_layers * (7 + 3 * CONFIG.n_experts)
    assert [id(p) for p in model.parameters()] == [id(p) for p in named]
