"""Products for few rows that fetch tables and weights before they wait for the kernel ahead of them: forwards with new weights and
another routing each time, against the same with the device waited for after every launch (``QUTAI_MOE_SYNC=1``): the same bits.
Needs a B200: ``-m gpu``."""
import hashlib
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def forwards(tokens, norm):
    """Every forward converts new weights, routes new rows and starts right behind the last one, in the same buffers."""
    from gpu_util import make_layer, to_device
    from qutai_b200.layers import MoEFeedForward, RMSNorm, Tensor

    d, E, k, h = 512, 8, 2, 328
    rng = np.random.default_rng(tokens)
    draw = lambda *shape: rng.standard_normal(shape).astype(np.float32)
    layer = make_layer((tokens, d), draw(E, d) * 0.2, draw(E, h, d) / 16, draw(E, h, d) / 16, draw(E, d, h) / 16, k)
    call = MoEFeedForward(RMSNorm(d, 1e-6), layer) if norm else layer
    inputs = [Tensor(to_device(draw(tokens, d), "bfloat16"), (tokens, d)) for _ in range(12)]
    kept = []
    for step, x in enumerate(inputs):
        if step % 3 == 0:
            for seed, weights in enumerate((layer._gate, layer._up, layer._down)):
                weights.fill_normal(0.0, 0.05, 100 * step + seed)
        kept.append(call.forward(x)[0].storage)
    return kept


def main():
    from qutai_b200 import lib

    for tokens in (1, 5, 32, 33, 300):      # up to 32 tokens both products start early, above the first of them
        for norm in (False, True):
            print("tokens", tokens, norm, *(hashlib.sha256(storage.tobytes()).hexdigest()[:16] for storage in forwards(tokens, norm)))
    assert lib.device_status() == 0


def test_early_products_give_the_bits_of_one_launch_at_a_time():
    outputs = []
    for sync in ("0", "1"):
        done = subprocess.run([sys.executable, os.path.abspath(__file__)], env=dict(os.environ, QUTAI_MOE_SYNC=sync), stdout=subprocess.PIPE,
                              stderr=subprocess.STDOUT, text=True, timeout=300)
        assert done.returncode == 0, done.stdout
        outputs.append([line for line in done.stdout.splitlines() if line.startswith("tokens")])
    assert len(outputs[0]) == 10 and outputs[0] == outputs[1]


if __name__ == "__main__":
    here = os.path.dirname(os.path.abspath(__file__))
    sys.path[:0] = [here, os.path.dirname(here)]
    main()
