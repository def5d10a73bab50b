"""The work that users of this package have it do, as a list of measurable cases.

A case is a dict of plain values.  ``prepare`` makes what a program holds before the call (inputs, weights, the layer
or model object), ``run`` is one pass through the package's public entry points, ``work`` the bytes and operations
that pass cannot do without, ``tolerance`` what two correct implementations of the same precision differ by.

Kinds of case:
  layer      ``SparseMoE`` (or, with ``norm``, ``MoEFeedForward``: norm before and residual after), forward or
             forward + backward, bfloat16 or float32 activations
  replay     ``SparseMoE.capture_forward`` once, then ``ForwardGraph.replay`` per call: the serving loop of decoding
  attention  ``attention_forward`` (prefill) or forward + backward, grouped key/value heads of width 64
  head       ``LMHead`` forward + backward: tied head and its cross-entropy loss
  decoder    one training step of ``Decoder``: loss, backward, optionally gradient clipping, ``AdamW``
"""
import math

import numpy as np
import torch

from qutai_b200.attention import attention_backward, attention_forward
from qutai_b200.decoder import Config, Decoder
from qutai_b200.head import LMHead
from qutai_b200.layers import MoEFeedForward, RMSNorm, SparseMoE, Tensor
from qutai_b200.optim import AdamW
from qutai_b200.storage import DeviceStorage

TORCH = {"float32": torch.float32, "bfloat16": torch.bfloat16}
BYTES = {"float32": 4, "bfloat16": 2}


# -- the cases ----------------------------------------------------------------------------------------------------
def _layer(name, tokens, d, experts, top_k, hidden, *, dtype="bfloat16", train=True, norm=False, skew=False):
    case = dict(kind="layer", tokens=tokens, d=d, experts=experts, top_k=top_k, hidden=hidden, dtype=dtype, train=train, norm=norm,
                skew=skew)
    return case if name is None else dict(case, name=name)


def _replay(name, tokens, d, experts, top_k, hidden):
    case = dict(kind="replay", tokens=tokens, d=d, experts=experts, top_k=top_k, hidden=hidden, dtype="bfloat16", skew=True)
    return case if name is None else dict(case, name=name)


def _attention(name, batch, time, heads, kv_heads, *, train):
    case = dict(kind="attention", batch=batch, time=time, heads=heads, kv_heads=kv_heads, train=train)
    return case if name is None else dict(case, name=name)


def _head(name, batch, time, width, vocab):
    case = dict(kind="head", batch=batch, time=time, width=width, vocab=vocab)
    return case if name is None else dict(case, name=name)


def _decoder(name, batch, time, d, heads, kv_heads, blocks, experts, top_k, hidden, vocab, *, clip):
    case = dict(kind="decoder", batch=batch, time=time, d=d, heads=heads, kv_heads=kv_heads, blocks=blocks, experts=experts, top_k=top_k,
                hidden=hidden, vocab=vocab, clip=clip)
    return case if name is None else dict(case, name=name)


def listed():
    return [
        # Decoding: 64 sequences, one position each, through the 64-expert layer; the call that a serving loop replays.
        _replay("decode_64_replay", 64, 2048, 64, 6, 1408),
        # The smallest call: a block's feed-forward half on a handful of rows, launched step by step (no recording).
        _layer("decode_4_rows", 4, 1024, 8, 2, 2816, train=False, norm=True),
        # Prefill of one prompt of odd length through the 64-expert layer, skewed load.
        _layer("prefill_1003_rows", 1003, 2048, 64, 6, 1408, train=False, skew=True),
        # float32 activations (the package's default dtype upstream): a small model's layer, forward and backward.
        _layer("train_float32", 2048, 512, 8, 2, 1024, dtype="float32"),
        # Fine-tuning with an odd number of rows: norm, layer and residual in one, forward and backward.
        _layer("train_3001_rows", 3001, 1024, 16, 2, 2048, norm=True),
        # The two training shapes of the layer: few wide experts with near-uniform load, many narrow ones with skewed load.
        _layer("train_8_experts", 16384, 1024, 8, 2, 2816),
        _layer("train_64_experts", 32768, 2048, 64, 6, 1408, skew=True),
        # Attention of a training step (4 x 2048 positions) and of a prefill with odd lengths, forward only.
        _attention("attention_train", 4, 2048, 16, 4, train=True),
        _attention("attention_prefill", 3, 1501, 16, 4, train=False),
        # The tied head and its loss over a 32000-token vocabulary.
        _head("head_train", 4, 2048, 1024, 32000),
        # A training step of a small model on short sequences with gradient clipping: many small launches.
        _decoder("decoder_small", 2, 301, 512, 8, 2, 2, 8, 2, 1024, 8000, clip=True),
        # A training step at the width, vocabulary and sequence length of the 12-block model, four of its blocks.
        _decoder("decoder_train", 4, 2048, 1024, 16, 4, 4, 16, 2, 2048, 32000, clip=False),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case from the ranges above: sizes log-uniform, most of them no multiple of a tile."""
    while True:
        kind = rng.choice(["layer", "layer", "layer", "layer", "layer", "replay", "attention", "attention", "head", "decoder"])
        if kind in ("layer", "replay"):
            experts = rng.choice([4, 8, 16, 32, 64])
            top_k = rng.choice([1, 2, 2, 4, 6])
            d, hidden = 64 * rng.randint(4, 32), 8 * _log(rng, 32, 352)
            if top_k > experts:
                continue
        if kind == "replay":
            case = _replay(None, _log(rng, 1, 256), d, experts, top_k, hidden)
        elif kind == "layer":
            train, dtype = rng.random() < 0.6, "float32" if rng.random() < 0.2 else "bfloat16"
            low = max(64, -(-8 * experts // top_k)) if train else 1       # training steps have rows for every expert, or nearly
            tokens = _log(rng, low, 4096 if dtype == "float32" else 32768)
            case = _layer(None, tokens, d, experts, top_k, hidden, dtype=dtype, train=train, norm=rng.random() < 0.5,
                          skew=rng.random() < 0.5)
            if dtype == "float32" and work(case)["flops"] > 2e11:
                continue
        elif kind == "attention":
            kv_heads = rng.choice([1, 2, 4, 8])
            case = _attention(None, _log(rng, 1, 16), _log(rng, 64, 8192), kv_heads * rng.choice([1, 2, 4]), kv_heads, train=rng.random() < 0.5)
            if case["batch"] * case["time"] > 32768 or work(case)["flops"] > 1e12:
                continue
        elif kind == "head":
            case = _head(None, _log(rng, 1, 8), _log(rng, 32, 2048), 64 * rng.randint(4, 32), 8 * _log(rng, 500, 6000))
            if case["batch"] * case["time"] > 8192:
                continue
        else:
            kv_heads = rng.choice([1, 2, 4])
            heads = kv_heads * rng.choice([2, 4])
            case = _decoder(None, _log(rng, 1, 8), _log(rng, 64, 2048), 64 * heads, heads, kv_heads, rng.randint(1, 4), rng.choice([4, 8, 16]), 2,
                            64 * rng.randint(8, 32), 8 * _log(rng, 250, 4000), clip=rng.random() < 0.5)
            if case["batch"] * case["time"] > 8192:
                continue
        largest = work(_layer(None, 32768, 2048, 64, 6, 1408))
        mine = work(case)
        if mine["flops"] <= largest["flops"] and mine["bytes"] <= largest["bytes"]:
            return case


# -- inputs -------------------------------------------------------------------------------------------------------
class _Memory:
    """What ``torch.as_tensor`` reads of a device buffer; keeps the buffer alive while the tensor lives."""
    __slots__ = ("__cuda_array_interface__", "storage")


def _tensor(storage, shape):
    """A storage of this package as a torch tensor over the same memory."""
    memory = _Memory()
    memory.storage = storage
    kind = "<f4" if storage.dtype == "float32" else "<i2"
    memory.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": kind, "data": (storage.ptr, False), "version": 2}
    tensor = torch.as_tensor(memory, device="cuda")
    return tensor if kind == "<f4" else tensor.view(torch.bfloat16)


def _given(tensor):
    """A torch tensor as the package's ``Tensor`` over the same memory."""
    names = {torch.float32: "float32", torch.bfloat16: "bfloat16", torch.int64: "int64"}
    return Tensor(DeviceStorage.wrap(tensor.data_ptr(), tensor.numel(), names[tensor.dtype], owner=tensor), tuple(tensor.shape))


class _LayerConfig:
    def __init__(self, case):
        self.d_model, self.n_experts, self.top_k, self.d_expert, self.n_layers = (case["d"], case["experts"], case["top_k"], case["hidden"], 12)


def _normal(generator, shape, dtype):
    return torch.randn(shape, generator=generator, device="cuda", dtype=torch.float32).to(TORCH[dtype])


def _make_layer(case, generator, seed, stream=0):
    """The layer as its constructor initialises it.  ``skew``: some experts are liked more than others — a column of the
    input that is one for every row carries a bias per expert, N(0, 0.5)."""
    layer = SparseMoE(_LayerConfig(case), seed=seed, stream=stream)
    x = _normal(generator, (case["tokens"], case["d"]), case["dtype"])
    if case["skew"]:
        x[:, -1] = 1
        router = layer.router.weight
        _tensor(router.storage, router.shape)[:, -1] = torch.randn(case["experts"], generator=generator, device="cuda") * 0.5
        router.storage.touch()
    return layer, x


def _token_ids(case, seed):
    """Token ids as a text has them: Zipf(1.1) over the vocabulary."""
    weights = np.arange(1, case["vocab"] + 1, dtype=np.float64) ** -1.1
    return np.random.default_rng(seed).choice(case["vocab"], size=(case["batch"], case["time"]), p=weights / weights.sum())


def prepare(case, seed):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    kind, state = case["kind"], dict(case=case)
    if kind == "layer":
        layer, x = _make_layer(case, generator, seed)
        state["layer"], state["x"] = layer, _given(x)
        state["call"] = MoEFeedForward(RMSNorm(case["d"], 1e-6), layer) if case["norm"] else layer
        if case["train"]:
            state["g"] = _given(_normal(generator, (case["tokens"], case["d"]), case["dtype"]))
            state["g_aux"] = _given(torch.full((1,), 0.01, device="cuda"))
        state["call"].forward(state["x"])                 # the operand copies of the weights, which a program makes once
    elif kind == "replay":
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        layer, x = _make_layer(case, generator, seed, stream.cuda_stream)
        torch.cuda.synchronize()
        graph = layer.capture_forward(_given(x))
        y, aux = graph.replay()
        state.update(stream=stream, x=x, graph=graph, y=_tensor(y.storage, y.shape), aux=_tensor(aux.storage, (1,)))
    elif kind == "attention":
        shape = (case["batch"], case["time"])
        state["q"] = _given(_normal(generator, (*shape, case["heads"] * 64), "bfloat16"))
        for name in ("k", "v"):
            state[name] = _given(_normal(generator, (*shape, case["kv_heads"] * 64), "bfloat16"))
        state["g"] = _given(_normal(generator, (*shape, case["heads"] * 64), "bfloat16"))
    elif kind == "head":
        state["hidden"] = _given(_normal(generator, (case["batch"], case["time"], case["width"]), "bfloat16"))
        state["weight"] = _given(_normal(generator, (case["vocab"], case["width"]), "float32") * 0.02)
        state["labels"] = _given(torch.from_numpy(_token_ids(case, seed)).to("cuda").reshape(-1)).storage
        state["head"] = LMHead()
        state["head"].forward(state["hidden"], state["weight"], state["labels"])
    else:
        config = Config(vocab_size=case["vocab"], d_model=case["d"], n_heads=case["heads"], n_kv_heads=case["kv_heads"], n_layers=case["blocks"],
                        n_experts=case["experts"], top_k=case["top_k"], d_expert=case["hidden"])
        model = Decoder(config, seed=seed)
        tokens = _token_ids(case, seed).tolist()
        model.loss(tokens)                                # makes the operand copies that the optimizer then keeps current
        state.update(model=model, tokens=tokens, optimizer=AdamW(model.parameters(), learning_rate=1e-4, shadows=model.operand_shadows()))
        state["weights"] = [_tensor(p.storage, p.shape) for p in (model.embedding.weight, model.norm.weight)]
        for block in model.blocks:
            dense = (block.attn_norm, block.ffn_norm, block.attn.q, block.attn.k, block.attn.v, block.attn.out, block.ffn.router)
            state["weights"] += [_tensor(part.weight.storage, part.weight.shape) for part in dense]
            state["weights"] += [_all_experts([getattr(expert, name).weight for expert in block.ffn.experts])[0] for name in ("gate", "up", "down")]
    return state


# -- one pass -----------------------------------------------------------------------------------------------------
def _all_experts(values):
    """Tensors of consecutive experts that lie side by side in memory (the layer keeps one buffer per kind), as one torch
    tensor each; ``None`` (no row reached that expert) ends a tensor."""
    result, i = [], 0
    while i < len(values):
        if values[i] is None:
            i += 1
            continue
        first, end = values[i], i + 1
        nbytes = first.size * 4
        while end < len(values) and values[end] is not None and values[end].storage.ptr == first.storage.ptr + (end - i) * nbytes:
            end += 1
        whole = DeviceStorage.wrap(first.storage.ptr, first.size * (end - i), "float32", owner=first.storage)
        result.append(_tensor(whole, (end - i, *first.shape)))
        i = end
    return result


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "layer":
        layer, call = state["layer"], state["call"]
        if not case["train"]:
            y, aux = call.forward(state["x"])
            return [_tensor(y.storage, y.shape), _tensor(aux.storage, (1,))]
        for parameter in call.parameters():
            parameter.zero_grad()
        y, aux = call.forward(state["x"])
        dx = call.backward(state["g"], state["g_aux"])
        router = layer.router.weight.grad
        outputs = [_tensor(y.storage, y.shape), _tensor(aux.storage, (1,)), _tensor(dx.storage, dx.shape), _tensor(router.storage, router.shape)]
        if case["norm"]:
            outputs.append(_tensor(call.ffn_norm.weight.grad.storage, (case["d"],)))
        for name in ("gate", "up", "down"):
            outputs += _all_experts([getattr(expert, name).weight.grad for expert in layer.experts])
        return outputs
    if kind == "replay":
        state["graph"].replay()
        return [state["y"], state["aux"]]
    if kind == "attention":
        q, k, v, heads, kv_heads = state["q"], state["k"], state["v"], case["heads"], case["kv_heads"]
        out, lse = attention_forward(q, k, v, heads, kv_heads)
        outputs = [_tensor(out, q.shape), _tensor(lse, (*q.shape[:2], heads))]
        if case["train"]:
            gradients = attention_backward(state["g"], q, k, v, out, lse, heads, kv_heads)
            outputs += [_tensor(gradient, like.shape) for gradient, like in zip(gradients, (q, k, v))]
        return outputs
    if kind == "head":
        head = state["head"]
        loss = head.forward(state["hidden"], state["weight"], state["labels"])
        d_hidden, d_weight = head.backward()
        return [_tensor(loss.storage, (1,)), _tensor(d_hidden.storage, d_hidden.shape), _tensor(d_weight.storage, d_weight.shape)]
    model, optimizer = state["model"], state["optimizer"]
    model.zero_grad()
    loss = model.loss(state["tokens"])
    model.backward()
    outputs = [_tensor(loss.storage, (1,))]
    if case["clip"]:
        outputs.append(model.clip_grad_norm(1.0))
    optimizer.step()
    return outputs + state["weights"]


# -- what a pass cannot do without ----------------------------------------------------------------------------------
def _layer_work(tokens, d, experts, top_k, hidden, size, train):
    reached = experts * (1.0 - (1.0 - top_k / experts) ** tokens)          # experts that some row reaches
    weights = 3.0 * reached * d * hidden
    products = 6.0 * tokens * top_k * d * hidden + 2.0 * tokens * d * experts
    if not train:
        return {"bytes": 2.0 * tokens * d * size + weights * size + 4.0 * experts * d, "flops": products}
    return {"bytes": 4.0 * tokens * d * size + weights * (size + 4) + 8.0 * experts * d, "flops": 3 * products}


def _attention_work(batch, time, heads, kv_heads, train):
    pairs = batch * heads * (time * (time + 1) / 2)
    wide, narrow = batch * time * heads * 128.0, batch * time * kv_heads * 128.0        # bytes of q (out, dq ..) and of k (v, dk, dv)
    if not train:
        return {"bytes": 2 * wide + 2 * narrow + batch * time * heads * 4.0, "flops": 256.0 * pairs}
    return {"bytes": 4 * wide + 4 * narrow + batch * time * heads * 4.0, "flops": (256.0 + 640.0) * pairs}


def _head_work(rows, width, vocab, weight_bytes):
    return {"bytes": 4.0 * rows * width + vocab * width * (weight_bytes + 4.0), "flops": 6.0 * rows * width * vocab}


def work(case):
    kind = case["kind"]
    if kind in ("layer", "replay"):
        return _layer_work(case["tokens"], case["d"], case["experts"], case["top_k"], case["hidden"], BYTES[case["dtype"]],
                           case.get("train", False))
    if kind == "attention":
        return _attention_work(case["batch"], case["time"], case["heads"], case["kv_heads"], case["train"])
    if kind == "head":
        return _head_work(case["batch"] * (case["time"] - 1), case["width"], case["vocab"], 2)
    rows, d, blocks = case["batch"] * case["time"], case["d"], case["blocks"]
    narrow = 64 * case["kv_heads"]
    dense = 2 * d * d + 2 * d * narrow                                                   # projections of one block
    parameters = case["vocab"] * d + d + blocks * (dense + 2 * d + case["experts"] * d * (1 + 3 * case["hidden"]))
    layer = _layer_work(rows, d, case["experts"], case["top_k"], case["hidden"], 2, True)
    attention = _attention_work(case["batch"], case["time"], case["heads"], case["kv_heads"], True)
    head = _head_work(case["batch"] * (case["time"] - 1), d, case["vocab"], 2)
    # every parameter, both of its moments: read and written; its bf16 copy read and written, its gradient made
    return {"bytes": 32.0 * parameters + 12.0 * rows * d, "flops": head["flops"] + blocks * (layer["flops"] + attention["flops"] + 6.0 * rows * dense)}


def tolerance(case):
    """About four times what was measured against the same path in float64 on the device's own routing (layer,
    attention, head), over sizes from a few rows to thousands."""
    kind = case["kind"]
    if kind in ("layer", "replay"):
        # float32: 1.0e-6, largest 7.6e-6; bfloat16: 4.4e-3, largest 0.055 (gradients of experts with few rows; 0.11
        # once, for an entry of dx in which large terms cancel)
        return {"rel": 4e-6, "max": 4e-5} if case["dtype"] == "float32" else {"rel": 1.6e-2, "max": 0.25}
    if kind == "attention":
        return {"rel": 1e-2, "max": 0.25}                  # 2.5e-3 (dq), largest 0.057
    if kind == "head":
        return {"rel": 1e-2, "max": 0.03}                  # 2.8e-3 (d_hidden), largest 7.3e-3
    # The step's outputs are the loss, the gradient norm and every updated weight.  A hidden state that is rounded the
    # other way can send a row to another expert, and AdamW's first step turns a gradient's sign into a full step:
    # with the embedding table disturbed by 2^-10 the weights moved by 5.3e-3, the largest by 0.028 of the weights' size.
    return {"rel": 2e-2, "max": 0.1}
