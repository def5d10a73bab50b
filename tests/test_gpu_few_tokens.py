"""The streamed products' form for at most 32 tokens, against the kernel for many rows, around its steps of 16 rows and at its limits.
Needs a B200: ``-m gpu``."""
import ctypes

import numpy as np
import pytest

import test_gpu_few_rows as few_rows
from oracle import moe_oracle as oracle

pytestmark = pytest.mark.gpu


def few_tokens(tokens, top_k, experts, tiles_per_expert, sms=148):
    """The rule of ``few_tokens`` in csrc/gemm_stream.cu, restated: at most 32 tokens, and two tiles per SM for the experts that uniform load reaches."""
    return tokens <= 32 and (1 - (1 - min(1, top_k / experts)) ** tokens) * experts * tiles_per_expert <= 2 * sms


@pytest.mark.parametrize("counts,width,hidden,forms", [      # forms: whether gate and up, and down, are in the form for few tokens
    ((0, 1, 15, 16), 64, 128, (True, True)),                 # 32 tokens; fewer k-blocks than stages
    ((32,), 584, 136, (True, True)),                         # one expert with every row, widths that fill no tile
    ((33,), 584, 136, (False, False)),                       # one token more
    ((0, 17, 2, 0, 0, 13), 1032, 264, (True, True)),         # two steps of 16 rows; more k-blocks than stages
    ((1,) * 30, 2048, 1408, (True, False)),                  # 211 tiles of the hidden width and 306 of the other, against two for every SM
    ((1,) * 30, 1408, 2048, (False, True)),                  # the other way round: down by itself in the form for few tokens, which then does not start early
    ((1,) * 30, 2048, 2048, (False, False)),
])
def test_products_of_few_tokens(counts, width, hidden, forms, kernel_variant):
    from qutai_b200 import lib

    assert lib.device_info()["sm_count"] == 148
    assert forms == tuple(few_tokens(sum(counts), 1, len(counts), -(-columns // 128)) for columns in (hidden, width))
    few_rows.test_streamed_products_match_the_kernel_for_many_rows(counts, width, hidden, kernel_variant)


@pytest.mark.parametrize("tokens,top_k,counts", [
    (20, 4, (33, 40, 7, 0)),                             # one row and eight rows past a stage's 32
    (32, 4, (128, 0, 0, 0)),                             # four tiles of rows, no pad row
    (32, 8, (129, 65, 31, 0, 1, 30, 0, 0)),              # past 128 rows: the pads of a last chunk that starts a 128-row tile
    (2, 2, (480, 0, 0, 0)),                              # more tiles than the CTAs that two tokens get
])
def test_tables_with_more_rows_for_an_expert_than_tokens(tokens, top_k, counts, kernel_variant):
    """Tables that the caller filled: an expert's count is bounded by the dispatched rows alone."""
    from gpu_util import RouteTables, to_device, to_host
    from qutai_b200 import lib
    from qutai_b200.storage import DeviceStorage

    experts, width, hidden = len(counts), 584, 264
    tables = RouteTables(tokens, experts, top_k)
    padded = [-(-count // lib.ROW_PAD) * lib.ROW_PAD for count in counts]
    offsets = np.concatenate([[0], np.cumsum(padded)])
    used, rows = int(offsets[-1]), tables.rows_bound
    assert used <= rows and max(counts) > 32 >= tokens
    owners = np.repeat(np.arange(experts), np.array(padded) // lib.ROW_PAD)
    for name, values in (("counts", counts), ("offsets", offsets), ("meta", (used, used // lib.ROW_PAD, sum(counts), 0)),
                         ("tile_expert", np.resize(owners, rows // lib.ROW_PAD))):
        tables.buf[name].upload_bytes(np.asarray(values, dtype=np.int32).tobytes())
    held = np.zeros(rows, dtype=bool)
    for first, count in zip(offsets, counts):
        held[first:first + count] = True
    rng = np.random.default_rng(tokens + experts)
    x = to_device(rng.standard_normal((rows, width)) * held[:, None], "bfloat16")
    ex = lib.Experts()
    weights = [to_device(rng.standard_normal(shape) / np.sqrt(shape[-1]), "bfloat16")
               for shape in ((experts, hidden, width), (experts, hidden, width), (experts, width, hidden))]
    ex.experts, ex.dtype, ex.engine, ex.width, ex.hidden = experts, lib.QMOE_BF16, lib.ENGINE_TCGEN05, width, hidden
    ex.w_gate, ex.w_up, ex.w_down = (w.ptr for w in weights)

    def forward():
        buffers = [DeviceStorage(rows * n, "bfloat16") for n in (hidden, hidden, hidden, width)]
        for buffer in buffers:
            lib.call("qmoe_memset", buffer.ptr, 0xFF, buffer.nbytes, 0)       # NaN: every row of a tile has to be written
        lib.call("qmoe_expert_forward", tables.ref, ctypes.byref(ex), x.ptr, *(buffer.ptr for buffer in buffers), 0)
        assert lib.device_status() == 0
        return [to_host(buffer, (rows, -1))[:used] for buffer in buffers]

    streamed = forward()
    kernel_variant(lib.VARIANT_NO_STREAM_GEMM)
    for got, want in zip(streamed, forward()):
        assert np.all(np.isfinite(got))
        assert oracle.max_rel_err(got, want) <= 2.0 ** -7       # as in test_gpu_few_rows
        assert not np.any(got[~held[:used]])                    # pad rows hold zeros
