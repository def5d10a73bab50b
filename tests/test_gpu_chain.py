"""Kernels launched in a chain, each set up while the one before it ends, against the same steps with the device waited for after
every launch (``QUTAI_MOE_SYNC=1``): the same bits.  A kernel that read before its predecessor had written would read what the step
before, on other inputs, left in the same buffers.  Needs a B200: ``-m gpu``."""
import hashlib
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 5


def block_steps(dtype, tokens):
    """Norm, layer and residual, forward and backward, on a new input every step, enqueued without a wait between the kernels."""
    from gpu_util import make_layer, to_device
    from qutai_b200.layers import MoEFeedForward, RMSNorm, Tensor

    d, E, k, h = 256, 8, 2, 264
    rng = np.random.default_rng(tokens)
    draw = lambda *shape: rng.standard_normal(shape).astype(np.float32)
    layer = make_layer((tokens, d), draw(E, d) * 0.2, draw(E, h, d) / 16, draw(E, h, d) / 16, draw(E, d, h) / 16, k)
    block = MoEFeedForward(RMSNorm(d, 1e-6), layer)
    inputs = [[Tensor(to_device(draw(tokens, d) * (step + 1), dtype), (tokens, d)) for _ in range(2)] for step in range(STEPS)]
    aux_gradient = Tensor(to_device(np.array([0.1]), "float32"), ())
    kept = []
    for x, g in inputs:
        for parameter in block.parameters():
            parameter.zero_grad()
        y, aux = block.forward(x)
        dx = block.backward(g, aux_gradient)
        kept += [y.storage, dx.storage, aux.storage.copy(), layer.router.weight.grad.storage.copy(), block.ffn_norm.weight.grad.storage.copy()]
        kept += [expert.up.weight.grad.storage.copy() for expert in layer.experts if expert.up.weight.grad is not None]
    return kept


def decoder_steps():
    from qutai_b200.decoder import Config, Decoder
    from qutai_b200.optim import AdamW

    config = Config(vocab_size=400, d_model=128, n_heads=2, n_kv_heads=1, n_layers=2, n_experts=4, top_k=2, d_expert=136)
    model = Decoder(config, seed=1)
    rng = np.random.default_rng(2)
    optimizer, kept = AdamW(model.parameters(), learning_rate=1e-3), []
    for _ in range(STEPS):
        model.zero_grad()
        kept.append(model.loss(rng.integers(0, config.vocab_size, (2, 150)).tolist()).storage)
        model.backward()
        model.clip_grad_norm(1.0)
        optimizer.step()
    return kept + [parameter.storage for parameter in model.parameters()]


def main():
    from qutai_b200 import lib

    for name, steps in (("bfloat16 1500", lambda: block_steps("bfloat16", 1500)), ("bfloat16 40", lambda: block_steps("bfloat16", 40)),
                        ("float32 700", lambda: block_steps("float32", 700)), ("decoder", decoder_steps)):
        print(name, *(hashlib.sha256(storage.tobytes()).hexdigest()[:16] for storage in steps()))
    assert lib.device_status() == 0


def test_chained_steps_give_the_bits_of_steps_one_launch_at_a_time():
    outputs = []
    for sync in ("0", "1"):
        done = subprocess.run([sys.executable, os.path.abspath(__file__)], env=dict(os.environ, QUTAI_MOE_SYNC=sync), stdout=subprocess.PIPE,
                              stderr=subprocess.STDOUT, text=True, timeout=300)
        assert done.returncode == 0, done.stdout
        outputs.append([line for line in done.stdout.splitlines() if line.startswith(("bfloat16", "float32", "decoder"))])
    assert len(outputs[0]) == 4 and outputs[0] == outputs[1]


if __name__ == "__main__":
    here = os.path.dirname(os.path.abspath(__file__))
    sys.path[:0] = [here, os.path.dirname(here)]
    main()
