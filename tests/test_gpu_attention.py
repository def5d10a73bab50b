"""Causal self-attention with grouped key/value heads (``qutai_b200.attention`` over ``qmoe_attention_forward`` /
``_backward``, tcgen05, head width 64, bf16) against the fixtures the upstream CPU backend produced, against the oracle
on other shapes (sequence lengths that are not multiples of the 128-position block, one and many blocks, key/value
groups of 1, 2 and 4 heads), and at the size of the full decoder step through sampled heads.  Needs a B200: ``-m gpu``."""
import os
import sys

import numpy as np
import pytest

from conftest import golden_files
from oracle import moe_oracle as oracle

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "golden"))
from attention_inputs import attention_inputs  # noqa: E402

pytestmark = pytest.mark.gpu

BF16_TOL = 2e-2              # max |a - b| / max |b| per tensor (the bar of the layer's bf16 outputs and gradients)
BF16_ELEMENT_TOL = 0.08      # |x - y| <= 0.08 max(rms(y), |y|)


def run_attention(q, k, v, grad, heads, kv_heads):
    from gpu_util import to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.attention import attention
    from qutai_b200.layers import Tensor

    tensors = [Tensor(to_device(a, "bfloat16"), a.shape) for a in (q, k, v)]
    out = attention(*tensors, heads, kv_heads)
    assert out.parents == tuple(tensors)
    dq, dk, dv = out.backward_rule(to_device(grad, "bfloat16"))
    assert lib.device_status() == 0
    return dict(out=to_host(out.storage, q.shape), dq=to_host(dq, q.shape), dk=to_host(dk, k.shape), dv=to_host(dv, v.shape))


def check(got, want, element_tol=BF16_ELEMENT_TOL):
    for name in ("out", "dq", "dk", "dv"):
        if not np.any(want[name]):        # a single position: the gradients of q and k are exactly zero upstream
            assert np.abs(got[name]).max() <= 1e-6, name
            continue
        assert oracle.max_rel_err(got[name], want[name]) <= BF16_TOL, name
        assert oracle.elementwise_err(got[name], want[name], bf16=True, unit=oracle.rms(want[name])) <= element_tol, name


@pytest.mark.parametrize("path", golden_files("attention"), ids=os.path.basename)
def test_attention_matches_the_upstream_fixture(path):
    g = np.load(path)
    heads, kv_heads = int(g["heads"]), int(g["kv_heads"])
    q, k, v, grad = attention_inputs(int(g["batch"]), int(g["time"]), heads, kv_heads, int(g["seed"]), float(g["scale"]))
    got = run_attention(q, k, v, grad, heads, kv_heads)
    check(got, g)
    again = run_attention(q, k, v, grad, heads, kv_heads)
    for name in ("out", "dq", "dk", "dv"):                 # no atomics anywhere: the same bits on every run
        assert np.array_equal(again[name], got[name]), name


@pytest.mark.parametrize("batch,time,heads,kv_heads", [(1, 128, 1, 1), (2, 129, 2, 1), (1, 256, 4, 1), (3, 300, 4, 2),
                                                       (1, 1000, 2, 2), (2, 64, 8, 2)])
def test_attention_matches_the_oracle(batch, time, heads, kv_heads):
    q, k, v, grad = attention_inputs(batch, time, heads, kv_heads, seed=time * 7 + heads, scale=0.8)
    out, lse = oracle.attention_forward(q, k, v, heads, kv_heads)
    dq, dk, dv = oracle.attention_backward(grad, q, k, v, out, lse, heads, kv_heads)
    check(run_attention(q, k, v, grad, heads, kv_heads), dict(out=out, dq=dq, dk=dk, dv=dv))


def test_attention_at_the_size_of_the_decoder_step():
    """4 sequences of 2048 positions, 16 heads in 4 key/value groups (one rank's share of the full decoder step):
    two sampled sequences x key/value groups against the oracle (a group's heads depend on nothing else).  The
    tensor-wide bar is the usual 2e-2; the element-wise one is 0.2 of the tensor's root mean square here: over 2048
    keys dS = P (dP - delta) loses digits where dP and delta (formed from the bf16 output) nearly cancel, and the
    worst of two million elements was 0.11."""
    batch, time, heads, kv_heads, dim = 4, 2048, 16, 4, 64
    q, k, v, grad = attention_inputs(batch, time, heads, kv_heads, seed=99, scale=0.6)
    got = run_attention(q, k, v, grad, heads, kv_heads)
    group = heads // kv_heads
    for b, g in ((0, 0), (3, 2)):
        wide = slice(g * group * dim, (g + 1) * group * dim)
        narrow = slice(g * dim, (g + 1) * dim)
        qs, ks, vs, gs = q[b:b + 1, :, wide], k[b:b + 1, :, narrow], v[b:b + 1, :, narrow], grad[b:b + 1, :, wide]
        out, lse = oracle.attention_forward(qs, ks, vs, group, 1)
        dq, dk, dv = oracle.attention_backward(gs, qs, ks, vs, out, lse, group, 1)
        check(dict(out=got["out"][b:b + 1, :, wide], dq=got["dq"][b:b + 1, :, wide], dk=got["dk"][b:b + 1, :, narrow],
                   dv=got["dv"][b:b + 1, :, narrow]), dict(out=out, dq=dq, dk=dk, dv=dv), element_tol=0.2)


def test_attention_rejects_what_it_does_not_cover():
    from gpu_util import to_device
    from qutai_b200.attention import attention
    from qutai_b200.layers import Tensor

    q = Tensor(to_device(np.zeros((1, 4, 64)), "bfloat16"), (1, 4, 64))
    kv = Tensor(to_device(np.zeros((1, 4, 64)), "bfloat16"), (1, 4, 64))
    with pytest.raises(ValueError):
        attention(q, kv, kv, 2, 1)                      # head width 32
    q32 = Tensor(to_device(np.zeros((1, 4, 64)), "float32"), (1, 4, 64))
    with pytest.raises(ValueError):
        attention(q32, kv, kv, 1, 1)                    # float32
    q3 = Tensor(to_device(np.zeros((1, 4, 192)), "bfloat16"), (1, 4, 192))
    kv2 = Tensor(to_device(np.zeros((1, 4, 128)), "bfloat16"), (1, 4, 128))
    with pytest.raises(ValueError):
        attention(q3, kv2, kv2, 3, 2)                   # heads not a multiple of kv_heads


@pytest.mark.parametrize("batch,time,heads,kv_heads,scale", [(1, 2, 2, 1, 1.0), (2, 63, 2, 2, 1.0), (1, 65, 3, 1, 1.0), (1, 127, 2, 1, 1.0),
                                                             (1, 255, 4, 2, 1.0), (2, 257, 2, 1, 1.0), (1, 640, 4, 4, 3.0)])
def test_attention_at_the_edges_of_blocks_and_with_growing_scores(batch, time, heads, kv_heads, scale):
    """Lengths one off the 64- and 128-position blocks, and scores that grow along the sequence, so that the maximum of a
    row rises by more than 2^8 between its key blocks and the accumulated output has to be rescaled."""
    q, k, v, grad = attention_inputs(batch, time, heads, kv_heads, seed=time * 5 + heads, scale=scale)
    k = oracle.round_bf16(k * (1.0 + 3.0 * np.arange(time)[None, :, None] / time))
    out, lse = oracle.attention_forward(q, k, v, heads, kv_heads)
    dq, dk, dv = oracle.attention_backward(grad, q, k, v, out, lse, heads, kv_heads)
    # with scores of scale^2 the softmax is nearly one-hot and dS = P (dP - delta) cancels: the element bar is that of the
    # 2048-position test there
    check(run_attention(q, k, v, grad, heads, kv_heads), dict(out=out, dq=dq, dk=dk, dv=dv), element_tol=0.2 if scale > 1 else BF16_ELEMENT_TOL)


def test_attention_of_one_hot_rows_returns_the_value_row():
    """Scores of about 8e5 that grow by 2048 (256 after the scale) from one position to the next: in every row the
    probability of the last position is 1 and all others are below exp(-256), so the output is that position's value row,
    exactly, and the gradient of q vanishes up to rounding.  A base of the exponentials that is rounded (half an ulp of 1.5e5 is
    2^-7) shows as a probability other than 1."""
    batch, time, heads, kv_heads = 1, 300, 2, 1
    at = np.arange(time)
    q = np.full((batch, time, heads * 64), 64.0)
    k = np.empty((batch, time, 64))
    k[0, :, :32], k[0, :, 32:] = (128 + at % 128)[:, None], (128 + 128 * (at // 128))[:, None]      # exact in bf16
    rng = np.random.default_rng(0)
    v, grad = oracle.round_bf16(rng.standard_normal(k.shape)), oracle.round_bf16(rng.standard_normal(q.shape))
    got = run_attention(q, k, v, grad, heads, kv_heads)
    assert np.array_equal(got["out"], np.concatenate([v, v], axis=2))
    # dS = P (dP - delta): two fp32 sums of the same 64 products in different orders, at most 64 roundings of their size apart,
    # times keys of up to 384 over 8
    bound = 384 / 8 * 64 * 2.0 ** -24 * np.abs(grad).max() * np.abs(v).max() * 64
    assert np.abs(got["dq"]).max() <= bound


@pytest.mark.parametrize("batch,time,heads,kv_heads", [(2, 2048, 8, 8), (4, 1024, 16, 4), (1, 4096, 4, 1)])
def test_attention_backward_repeats_its_bits(batch, time, heads, kv_heads):
    """Many key blocks with a diagonal block in each, whose row warps take longer than the others': the warps that share a
    block's probabilities drift apart, and every repetition has to give the same bits all the same."""
    from gpu_util import to_device
    from qutai_b200 import lib
    from qutai_b200.attention import attention_backward, attention_forward
    from qutai_b200.layers import Tensor

    inputs = attention_inputs(batch, time, heads, kv_heads, seed=time, scale=1.0)
    q, k, v, grad = (Tensor(to_device(a, "bfloat16"), a.shape) for a in inputs)
    out, lse = attention_forward(q, k, v, heads, kv_heads)
    first = None
    for _ in range(25):
        bits = [part.tobytes() for part in attention_backward(grad, q, k, v, out, lse, heads, kv_heads)]
        first = first or bits
        assert bits == first
    assert lib.device_status() == 0


@pytest.mark.parametrize("time", [200, 256, 300])
def test_attention_gradients_of_a_key_that_no_query_sees(time):
    """A key with an infinite component, so that every query's score of it is -inf: its probability is zero everywhere, and its
    gradients too, whether or not the sequence fills its last block of queries."""
    heads, kv_heads, hidden = 2, 1, 70
    q, k, v, grad = attention_inputs(1, time, heads, kv_heads, seed=time, scale=1.0)
    q[:, :, 0::64] = -1.0
    k[:, :, 0] = 0.0
    without = k.copy()
    k[0, hidden, 0], without[0, hidden, 0] = np.inf, 2.0 ** 100
    got = run_attention(q, k, v, grad, heads, kv_heads)
    out, lse = oracle.attention_forward(q, without, v, heads, kv_heads)
    dq, dk, dv = oracle.attention_backward(grad, q, without, v, out, lse, heads, kv_heads)
    for name in ("dk", "dv"):
        assert np.all(np.isfinite(got[name])) and not np.any(got[name][0, hidden]), name
    check(dict(got, dq=dq), dict(out=out, dq=dq, dk=dk, dv=dv))       # dq holds 0 * inf, as a product with that key does


@pytest.mark.parametrize("time", [130, 300])
def test_attention_rows_with_infinities_and_nan_stay_by_themselves(time):
    """Query rows that hold NaN and infinities give NaN rows; every other row of the output keeps its bits, in the same block and in
    others."""
    from gpu_util import to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.attention import attention_forward
    from qutai_b200.layers import Tensor

    heads, kv_heads = 2, 1
    q, k, v, _ = attention_inputs(1, time, heads, kv_heads, seed=time, scale=1.0)

    def rows(values):
        tensors = [Tensor(to_device(a, "bfloat16"), a.shape) for a in (values, k, v)]
        out, lse = attention_forward(*tensors, heads, kv_heads)
        assert lib.device_status() == 0
        return to_host(out, q.shape)[0], to_host(lse, (time, heads))

    wild = q.copy()
    wild[0, 5, 3], wild[0, 64, 64:], wild[0, 127, 7], wild[0, time - 1, 0] = np.nan, np.inf, -np.inf, np.nan
    (plain, plain_lse), (got, got_lse) = rows(q), rows(wild)
    bad = np.zeros((time, heads), dtype=bool)
    bad[5, 0] = bad[64, 1] = bad[127, 0] = bad[time - 1, 0] = True
    wide = np.repeat(bad, 64, axis=1)
    assert np.isnan(got[wide]).all() and np.isnan(got_lse[bad]).all()
    assert np.array_equal(got[~wide], plain[~wide]) and np.array_equal(got_lse[~bad], plain_lse[~bad])


@pytest.mark.parametrize("batch,time,heads,kv_heads", [(1, 1, 1, 1), (2, 129, 4, 2), (1, 300, 2, 1)])
def test_attention_delta_is_summed_in_the_order_of_the_row(batch, time, heads, kv_heads):
    """delta = sum of grad_out * out: products of two bf16 numbers are exact in fp32, the pairs of a row are rounded once and
    added from the first to the last, so numpy gives the same bits."""
    import ctypes

    from gpu_util import to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.attention import attention_forward
    from qutai_b200.layers import Tensor
    from qutai_b200.storage import DeviceStorage

    rng = np.random.default_rng(time)
    q, k, v, grad = (oracle.round_bf16(rng.standard_normal((batch, time, 64 * h))).astype(np.float32) for h in (heads, kv_heads, kv_heads, heads))
    tensors = [Tensor(to_device(x, "bfloat16"), x.shape) for x in (q, k, v)]
    out, lse = attention_forward(*tensors, heads, kv_heads)
    a = lib.Attention()
    a.batch, a.time, a.heads, a.kv_heads, a.dim, a.dtype = batch, time, heads, kv_heads, 64, lib.QMOE_BF16
    gradients = [DeviceStorage(x.size, "bfloat16") for x in (q, k, v)]
    delta, gradient = DeviceStorage(lse.size, "float32"), to_device(grad, "bfloat16")
    a.q, a.k, a.v = (tensor.storage.ptr for tensor in tensors)
    a.dq, a.dk, a.dv = (storage.ptr for storage in gradients)
    a.out, a.lse, a.grad_out, a.delta = out.ptr, lse.ptr, gradient.ptr, delta.ptr
    lib.call("qmoe_attention_backward", ctypes.byref(a), 0)
    products = to_host(out, (-1, 64)).astype(np.float32) * grad.reshape(-1, 64)
    want = np.zeros(len(products), dtype=np.float32)
    for column in range(0, 64, 2):
        want += products[:, column] + products[:, column + 1]
    assert np.array_equal(to_host(delta, (-1,)).astype(np.float32), want)
