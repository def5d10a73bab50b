"""Which weights the projections of ``qutai_b200.decoder.GQA`` multiply with, on a fake device (no GPU): it keeps, per address, of
which weight and of which of its states a bf16 copy was last made there, and notes what every product reads."""
import ctypes

import pytest

from qutai_b200 import lib, storage
from qutai_b200.decoder import GQA, Config, Linear
from qutai_b200.layers import Tensor
from qutai_b200.storage import DeviceStorage

CONFIG = Config(vocab_size=16, d_model=128, n_heads=2, n_kv_heads=1, n_layers=1, n_experts=2, top_k=1, d_expert=8)
BATCH, TIME = 1, 5


class FakeDevice:
    def __init__(self):
        self.next, self.state, self.copies, self.read = 0x1000, {}, {}, []

    def qmoe_free(self, address):
        return 0

    def qmoe_gemm_wgrad_partials(self, m, k, n):
        return 0

    def call(self, name, *args):
        if name == "qmoe_malloc":
            ctypes.cast(args[0], ctypes.POINTER(ctypes.c_uint64))[0] = self.next
            self.next += 1 << 24
        elif name == "qmoe_cast_bf16":
            source, destination, count, _ = args
            self.copies[destination] = (2 * count, source, self.state.get(source, 0))
        elif name == "qmoe_gemm" and args[9] == 0:        # not a weight gradient: the second operand is a weight
            address, end = args[2], args[2] + 2 * args[7] * args[8]
            while address < end:
                nbytes, source, state = self.copies.get(address, (end - address, None, None))
                self.read.append((source, state))
                address += nbytes


@pytest.fixture
def device(monkeypatch):
    fake = FakeDevice()
    monkeypatch.setattr(lib, "load", lambda: fake)
    monkeypatch.setattr(lib, "call", fake.call)
    monkeypatch.setattr(storage, "_cache", {})
    monkeypatch.setattr(storage, "_cached_bytes", 0)
    return fake


def read_by(device, attention, backward=False):
    rows, width = BATCH * TIME, CONFIG.d_model
    device.read.clear()
    _, saved = attention.forward(DeviceStorage(rows * width, "bfloat16"), BATCH, TIME)
    if backward:
        device.read.clear()
        attention.backward(DeviceStorage(rows * width, "bfloat16"), saved, BATCH, TIME)
    return list(device.read)


def current(device, *layers):
    return [(layer.weight.storage.ptr, device.state.get(layer.weight.storage.ptr, 0)) for layer in layers]


def write(device, *layers):
    for layer in layers:
        device.state[layer.weight.storage.ptr] = device.state.get(layer.weight.storage.ptr, 0) + 1
        layer.weight.storage.touch()


def separate(attention):
    pass


def tied(attention):
    attention.v.weight = attention.k.weight


def one_buffer(attention):
    layers = (attention.q, attention.k, attention.v)
    flat = DeviceStorage(sum(layer.weight.storage.size for layer in layers), "float32")
    start = 0
    for layer in layers:
        size = layer.weight.storage.size
        layer.weight = Tensor(flat.view(start, size), layer.weight.shape, requires_grad=True)
        start += size


@pytest.mark.parametrize("arrange", [separate, tied, one_buffer])
def test_every_projection_reads_its_own_weight_as_it_is_now(device, arrange):
    attention = GQA(CONFIG, seed=0)
    arrange(attention)
    layers = (attention.q, attention.k, attention.v, attention.out)
    assert read_by(device, attention) == current(device, *layers)
    for written in (layers[:3], layers[1:2], layers[2:]):
        write(device, *written)
        assert read_by(device, attention) == current(device, *layers)
        assert read_by(device, attention, backward=True) == current(device, attention.out, *layers[:3])


def test_a_replaced_projection_is_the_one_that_runs(device):
    class Adapted(Linear):
        runs = 0

        def forward(self, x, rows):
            self.runs += 1
            return super().forward(x, rows)

    attention = GQA(CONFIG, seed=0)
    read_by(device, attention)
    attention.q = Linear(CONFIG.d_model, CONFIG.d_model, std=0.02, seed=1)
    attention.v = Adapted(CONFIG.d_model, attention.kv_width, std=0.02, seed=2)
    layers = (attention.q, attention.k, attention.v, attention.out)
    assert read_by(device, attention) == current(device, *layers)
    assert attention.v.runs == 1
    assert read_by(device, attention, backward=True) == current(device, attention.out, *layers[:3])
