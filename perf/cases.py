"""Timed cases of the GRU scan: what a user of the package has it do, through its public entry points.

Every case is one ``GRULayer`` call: inference (``out, h_T = layer(x, h0)`` without gradients), or a
training step (the same call, the backward pass from the gradient that the rest of the model hands
to ``out``, and the gradients of every parameter).  Training at one fixed shape is captured once
with ``graphed.GraphedStep``, the package's own way to run such a loop; training on batches of
varying length, and inference, call the layer directly.

Keys of a case: ``kind`` of the hidden weights, sequence length ``T``, batch ``B``, input width
``I``, hidden width ``H``; ``train``; ``graph`` (captured step); ``x_grad`` (the layer sits on top
of others, so the gradient with respect to its input is wanted too); bit widths of the weight, input
and hidden-state quantisers (32: none); ``nblocks`` (diagonal blocks of a monarch layer, factors of
a butterfly).
"""

from __future__ import annotations

import math

import torch

import gru_triton_b200 as gru
from gru_triton_b200.graphed import GraphedStep


def _case(name, kind, T, B, I, H, **options):
    case = dict(name=name, kind=kind, T=T, B=B, I=I, H=H, train=False, graph=False, x_grad=False,
                weight_bits=32, input_bits=32, hidden_bits=32, nblocks=1)
    case.update(options)
    return case


def listed():
    return [
        # one time step of one sequence, as a streaming recogniser makes for every frame: pure latency
        _case("dense_stream_step", "dense", 1, 1, 256, 256),
        # a deployed model with the stock int8 recipe (weights, input and state on int8 grids) on one batch of utterances
        _case("dense_int8_infer", "dense", 100, 64, 128, 512, weight_bits=8, input_bits=8, hidden_bits=8),
        # the headline training step of the benchmark
        _case("dense_train", "dense", 64, 32, 512, 512, train=True, graph=True),
        # the same layer at an ordinary training batch
        _case("dense_train_b256", "dense", 64, 256, 512, 512, train=True, graph=True),
        # a stacked layer on batches of varying length: sizes that no tile divides
        _case("dense_train_ragged", "dense", 41, 257, 120, 608, train=True, x_grad=True),
        # quantisation-aware training of a large layer: the shard that one of eight GPUs has of a batch of 4096
        _case("dense_qat_shard", "dense", 512, 512, 1024, 1024, train=True, graph=True, weight_bits=8, hidden_bits=8),
        # the same with half of that batch on one GPU: the largest case
        _case("dense_qat_large", "dense", 512, 2048, 1024, 1024, train=True, weight_bits=8, hidden_bits=8),
        # block-diagonal hidden weights with a frozen int8 state, the benchmark's training step
        _case("monarch_train", "monarch", 64, 32, 512, 512, train=True, graph=True, hidden_bits=8, nblocks=8),
        # butterfly hidden weights, the benchmark's training step
        _case("butterfly_train", "butterfly", 128, 64, 1024, 1024, train=True, graph=True),
        # a stacked butterfly layer whose width is no power of two, on batches of varying length
        _case("butterfly_train_ragged", "butterfly", 50, 19, 384, 384, train=True, x_grad=True),
        # diagonal hidden weights over long sequences, int8 state: the benchmark's inference pass
        _case("diagonal_infer", "diagonal", 1024, 256, 1024, 1024, hidden_bits=8),
        # training a stacked diagonal layer on long sequences of varying length
        _case("diagonal_train", "diagonal", 500, 96, 512, 1024, train=True, x_grad=True),
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["dense", "dense", "monarch", "butterfly", "diagonal"])
    T, B = _log_int(rng, 1, 512), _log_int(rng, 1, 1024)
    while T * B > 65536:
        T, B = max(1, T // 2), max(1, B // 2 + 1)
    H, I, nblocks = _log_int(rng, 32, 1024), _log_int(rng, 32, 1024), 1
    # widths are multiples of eight in most models; one in five is not
    if rng.random() < 0.8:
        H, I = max(32, H // 8 * 8), max(32, I // 8 * 8)
    if kind == "dense" and rng.random() < 0.3:
        H = rng.choice([256, 512, 768, 1024])
    if kind == "monarch":
        nblocks = rng.choice([2, 4, 8, 16])
        H = max(32, H // nblocks * nblocks)
    if kind == "butterfly":
        nblocks = rng.choice([1, 1, 2])
    train = rng.random() < 0.65
    int8 = rng.random() < 0.4
    return dict(kind=kind, T=T, B=B, I=I, H=H, train=train, graph=train and rng.random() < 0.5,
                x_grad=train and rng.random() < 0.5, weight_bits=8 if int8 and kind == "dense" else 32,
                input_bits=8 if int8 and rng.random() < 0.3 else 32, hidden_bits=8 if int8 else 32, nblocks=nblocks)


def _layer(case, seed):
    """The layer with the package's own initialisation; quantised states calibrated on a few batches
    of eight sequences and frozen, as ``GRULayer.calibrate`` / ``freeze`` have it."""
    recipe = gru.QuantRecipe(weight=gru.QuantizerConfig(bits=case["weight_bits"], axis=0, name="W"),
                             input_act=gru.QuantizerConfig(bits=case["input_bits"], name="x"),
                             hidden=gru.QuantizerConfig(bits=case["hidden_bits"], name="h"))
    structure = None
    if case["kind"] != "dense":
        structure = gru.StructureConfig(kind=case["kind"], nblocks=case["nblocks"], butterfly_nblocks=case["nblocks"])
    with torch.random.fork_rng(devices=[]):
        torch.manual_seed(seed)
        layer = gru.GRULayer(case["I"], case["H"], recipe, gate_layout="fused", structure_hidden=structure)
    layer = layer.cuda().train(case["train"])
    cell = layer.cell
    if case["hidden_bits"] < 32 or case["input_bits"] < 32:
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        batches = [torch.randn(128, 8, case["I"], device="cuda", generator=gen) for _ in range(4)]
        layer.calibrate(batches, n_batches=len(batches))
        for q in (cell.quant_x, cell.quant_h_in, cell.quant_h_out):
            q.freeze()                      # weight scales stay dynamic: they follow the weights
    return layer


def prepare(case, seed):
    layer = _layer(case, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed + 2)
    T, B, I, H = case["T"], case["B"], case["I"], case["H"]
    x = torch.randn(T, B, I, device="cuda", generator=gen)
    h0 = torch.randn(B, H, device="cuda", generator=gen).mul_(0.1)
    state = dict(case=case, layer=layer, inputs=[x, h0])
    if case["train"]:
        # what a mean loss over the batch hands back
        state["inputs"].append(torch.randn(T, B, H, device="cuda", generator=gen).div_(T * B))

        def step(x, h0, dout):
            layer.zero_grad(set_to_none=True)
            if case["x_grad"]:
                x = x.detach().requires_grad_(True)
            out, h_T = layer(x, h0)
            out.backward(dout)
            grads = [p.grad for p in layer.parameters()]
            return (out.detach(), h_T.detach(), *([x.grad] if case["x_grad"] else []), *grads)

        state["step"] = GraphedStep(step, state["inputs"]) if case["graph"] else step
    return state


def run(state):
    if state["case"]["train"]:
        return state["step"](*state["inputs"])
    with torch.no_grad():
        return state["layer"](*state["inputs"])


def work(case):
    T, B, I, H = case["T"], case["B"], case["I"], case["H"]
    n, hpad = case["nblocks"], 1 << max(1, math.ceil(math.log2(H)))
    # hidden weights, and multiply-adds of one hidden product of one row
    weights, macs = {"dense": (3 * H * H, 3 * H * H), "monarch": (3 * H * H // n, 3 * H * H // n), "diagonal": (3 * H, 3 * H),
                     "butterfly": (6 * n * hpad * int(math.log2(hpad)), 6 * n * hpad * int(math.log2(hpad)))}[case["kind"]]
    params = weights + 3 * H * I + 6 * H
    rows = T * B
    floats = rows * (I + H) + B * H + params                      # x, h0, parameters in; out out
    flops = 2.0 * rows * (3 * H * I + macs)
    if case["train"]:
        floats += rows * H + params                               # the gradient of out in; the gradients out
        flops += 2.0 * rows * (3 * H * I + 2 * macs)
        if case["x_grad"]:
            floats += rows * I
            flops += 2.0 * rows * 3 * H * I
    return {"bytes": 4.0 * floats, "flops": flops}


def tolerance(case):
    """About four times what was measured against the same layer in 64 bits, and on inputs changed in their last bit.

    On an int8 grid a state that falls next to a half-way point may land on either code, and in a dense layer one such
    code moves all others of its sequence a little, so whole sequences part within the quantisation noise (rel 7e-3
    seen; 6e-4 where only a block of the state, or a unit of its own, follows).  In fp32 the sums over all rows that
    make the weight gradients are the least exact (5e-6; the outputs alone 7e-7)."""
    if case["hidden_bits"] < 32:
        return {"rel": 0.027 if case["kind"] == "dense" else 0.01, "max": 0.2}
    return {"rel": 2e-5, "max": 3e-4} if case["train"] else {"rel": 3e-6, "max": 2e-5}


def _fake_quant64(v, scale, top):
    """Round to the grid and clamp, in 64 bits; the gradient goes straight through inside the range."""
    q = v / scale
    code = q.detach().round()
    inside = (code >= -top) & (code <= top)
    return (code.clamp(-top, top) + (q - q.detach()) * inside) * scale


def _weight64(w, bits):
    if bits >= 32:
        return w
    top = 2 ** (bits - 1) - 1
    amax = torch.maximum(w.amax(1, keepdim=True).abs(), w.amin(1, keepdim=True).abs())
    return _fake_quant64(w, amax.clamp(min=1e-8) / top, top)


def _hidden64(case, weights):
    """h [B,H] -> the hidden products [3,B,H] of the gates r, z, n (``weights``: one tensor per gate)."""
    kind, H = case["kind"], case["H"]
    if kind == "dense":
        W = torch.stack([_weight64(w, case["weight_bits"]) for w in weights])
        return lambda h: torch.matmul(h, W.transpose(1, 2))
    W = torch.stack(weights)
    if kind == "diagonal":
        return lambda h: h * W[:, None, :]
    if kind == "monarch":
        def blocks(h):
            return torch.einsum("bni,gnoi->gbno", h.reshape(h.shape[0], W.shape[1], -1), W).reshape(3, h.shape[0], H)
        return blocks
    W = W[:, 0]                                          # [3, factors, log2 n, n/2, 2 (new), 2 (old)]
    log_n, n = W.shape[2], 2 * W.shape[3]

    def butterfly(h):
        v = torch.nn.functional.pad(h, (0, n - H)).expand(3, -1, -1)
        for f in range(W.shape[1]):
            for s in range(log_n) if f % 2 == 0 else reversed(range(log_n)):
                stage = s if f % 2 == 0 else log_n - 1 - s
                tw = W[:, f, stage].reshape(3, 1, n >> (s + 1), 1 << s, 2, 2)
                old = v.reshape(3, -1, n >> (s + 1), 2, 1 << s)
                a, b = old[:, :, :, 0], old[:, :, :, 1]
                v = torch.stack((tw[..., 0, 0] * a + tw[..., 0, 1] * b, tw[..., 1, 0] * a + tw[..., 1, 1] * b), 3)
                v = v.reshape(3, -1, n)
        return v[:, :, :H]
    return butterfly


def exact(case, seed):
    """The same outputs from plain torch operations in 64 bits; none where the states of all steps would not fit."""
    if case["train"] and case["T"] * case["B"] * case["H"] > 3e8:
        return None
    state = prepare(dict(case, graph=False), seed)
    cell, inputs = state["layer"].cell, [t.double() for t in state["inputs"]]
    params = [(name, p.detach().double().requires_grad_(case["train"])) for name, p in state["layer"].named_parameters()]
    by = {name.split(".", 1)[1]: p for name, p in params}
    scale = {name: float(getattr(cell, name).scale) for name in ("quant_x", "quant_h_in", "quant_h_out")}

    def on_grid(v, name, bits):
        return v if bits >= 32 else _fake_quant64(v, scale[name], 2 ** (bits - 1) - 1)

    with torch.set_grad_enabled(case["train"]):
        x = inputs[0].requires_grad_(case["train"] and case["x_grad"])
        hidden = {"dense": "W_h{}", "diagonal": "struct_Wh_{}.weight", "monarch": "struct_Wh_{}.weight",
                  "butterfly": "struct_Wh_{}.b.twiddle"}[case["kind"]]
        product = _hidden64(case, [by[hidden.format(g)] for g in "rzn"])
        xq = on_grid(x, "quant_x", case["input_bits"])
        gi = [xq @ _weight64(by[f"W_i{g}"], case["weight_bits"]).t() + by[f"b_i{g}"] for g in "rzn"]
        h, outs = inputs[1], []
        for t in range(case["T"]):
            gh_r, gh_z, gh_n = product(on_grid(h, "quant_h_in", case["hidden_bits"]))
            r = torch.sigmoid(gi[0][t] + gh_r + by["b_hr"])
            z = torch.sigmoid(gi[1][t] + gh_z + by["b_hz"])
            n = torch.tanh(gi[2][t] + r * (gh_n + by["b_hn"]))
            h = on_grid((1 - z) * n + z * h, "quant_h_out", case["hidden_bits"])
            outs.append(h)
        out = torch.stack(outs)
        if not case["train"]:
            return out, h
        wanted = ([x] if case["x_grad"] else []) + [p for _, p in params]
        return (out.detach(), h.detach(), *torch.autograd.grad(out, wanted, inputs[2]))
