"""Performance cases: the work users of this framework have it do, through its public entry points.

Kinds of case
  train        one optimizer step of GptTrainer: `accum` micro-batches (forward, loss, backward), then the update.
               feed "device": token tensors already in HBM; feed "pipeline": host arrays through AsyncInputPipeline,
               the way a training program with a data loader runs.
  evaluate     GptTrainer.evaluate over `accum` batches (forward and loss only).
  step         one token of incremental decoding (GptTrainer.forward_step) behind `context` cached tokens.
  generate     GptTrainer.generate: a prompt of `context` tokens, then `new` tokens, greedy; and the logits it ended on.
  engine_linear, engine_attention
               one Linear layer / one attention layer, forward and backward, as the C++ engine drop-in issues them:
               fp32 primitives of the C ABI in the (features, tokens) layout of the reference's layers.

Model sizes are those of the repository's benchmark configurations and tests, or generic ones between them.
"""
import ctypes as C
import math

import numpy as np
import torch

import __graft_entry__ as entry

nnb = entry.load_package()

GELU, SWIGLU = nnb.ACT_GELU, nnb.ACT_SWIGLU
LAYER, RMS = nnb.NORM_LAYER, nnb.NORM_RMS
LEARNED, SINUSOIDAL, ALIBI, ROPE = nnb.POS_LEARNED, nnb.POS_SINUSOIDAL, nnb.POS_ALIBI, nnb.POS_ROPE
FP32, BF16 = nnb.FP32, nnb.BF16

TINY = dict(vocab=512, d=128, heads=4, layers=2, ff=512, act=GELU, norm=LAYER, pos=LEARNED)
SMALL = dict(vocab=4096, d=384, heads=6, layers=6, ff=1024, act=SWIGLU, norm=RMS, pos=SINUSOIDAL)
BASE = dict(vocab=8192, d=768, heads=12, layers=12, ff=2048, act=SWIGLU, norm=RMS, pos=ALIBI)
PACKED = dict(vocab=16384, d=1024, heads=16, layers=16, ff=2816, act=SWIGLU, norm=RMS, pos=LEARNED)


def _train(name, model, seq, batch, accum=1, precision=BF16, feed="device", docs=False, mask=False, clip=0.0, muon=False):
    c = dict(model, kind="train", seq=seq, batch=batch, accum=accum, precision=precision, feed=feed, docs=docs, mask=mask, clip=clip, muon=muon)
    return dict(c, name=name) if name else c


def _infer(name, kind, model, seq, batch=1, accum=1, context=0, new=0, precision=BF16):
    c = dict(model, kind=kind, seq=seq, batch=batch, accum=accum, precision=precision, context=context, new=new)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a first experiment in the reference's own precision: the smallest model, all launch latency
        _train("train_tiny_fp32", TINY, 128, 8, precision=FP32),
        # someone else's model: nothing is a multiple of a tile, padded sequences with a loss mask, clipping
        _train("train_ragged", dict(vocab=1000, d=320, heads=5, layers=4, ff=856, act=GELU, norm=LAYER, pos=LEARNED), 200, 12, mask=True, clip=1.0),
        # a small language model trained from a data loader on the host
        _train("train_small", SMALL, 256, 32, feed="pipeline", clip=1.0),
        # the benchmark model: gradient accumulation over two micro-batches, from the host
        _train("train_base", BASE, 1024, 16, accum=2, feed="pipeline"),
        # the largest model: packed documents in long windows, Muon on the matrices and AdamW on the rest
        _train("train_packed_muon", PACKED, 2048, 8, docs=True, muon=True),
        # long context: heads of 128, rotary positions, a large vocabulary
        _train("train_long", dict(vocab=32768, d=1024, heads=8, layers=4, ff=2816, act=SWIGLU, norm=RMS, pos=ROPE), 8192, 2, clip=1.0),
        # validation loss of the benchmark model between epochs
        _infer("evaluate_base", "evaluate", BASE, 1024, batch=16, accum=2),
        # one token of a small model, little context: pure latency
        _infer("step_small", "step", SMALL, 256, context=40),
        # one token of the benchmark model late in its window
        _infer("step_base", "step", BASE, 1024, context=900),
        # a prompt and a short answer
        _infer("generate_base", "generate", BASE, 1024, context=501, new=16),
        # the C++ engine drop-in: the layers of a small model, one primitive at a time
        dict(name="engine_linear", kind="engine_linear", out=1024, inp=384, tokens=8192),
        dict(name="engine_attention", kind="engine_attention", heads=48, seq=256, dk=64),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _model(rng, most_d, most_layers):
    dk = rng.choice([32, 64, 64, 64, 128])
    heads = max(1, round(_log(rng, 128, most_d) / dk))
    d = dk * heads
    act = rng.choice([GELU, SWIGLU, SWIGLU])
    ff = max(64, 8 * round((4.0 if act == GELU else 8.0 / 3.0) * d * rng.uniform(0.9, 1.1) / 8))
    return dict(vocab=8 * round(_log(rng, 512, 32768) / 8), d=d, heads=heads, layers=round(_log(rng, 1, most_layers)), ff=ff, act=act,
                norm=rng.choice([LAYER, RMS, RMS]), pos=rng.choice([LEARNED, SINUSOIDAL, ALIBI, ROPE]))


def draw(rng):
    """One more case of the same kinds and ranges: sizes over their logarithms, odd sequence lengths among them."""
    kind = rng.choices(["train", "evaluate", "step", "generate", "engine_linear", "engine_attention"], [50, 10, 12, 10, 9, 9])[0]
    if kind == "engine_linear":
        return dict(kind=kind, out=round(_log(rng, 128, 2048)), inp=round(_log(rng, 128, 1024)), tokens=round(_log(rng, 256, 8192)))
    if kind == "engine_attention":
        seq = round(_log(rng, 32, 512))
        dk = rng.choice([32, 64, 128])
        return dict(kind=kind, heads=max(1, round(_log(rng, 4, 48) * min(1.0, (256 / seq) ** 2 * 64 / dk))), seq=seq, dk=dk)
    if kind in ("step", "generate"):
        model = _model(rng, 1024, 12)
        seq = round(_log(rng, 128, 2048))
        precision = rng.choice([BF16, BF16, BF16, FP32])
        if kind == "step":
            return _infer(None, kind, model, seq, context=min(seq - 1, round(_log(rng, 8, seq))), precision=precision)
        new = rng.randint(4, 24)
        return _infer(None, kind, model, seq, context=max(1, min(seq - new, 512, round(_log(rng, 8, seq)))), new=new, precision=precision)
    while True:
        precision = rng.choice([BF16, BF16, BF16, BF16, FP32])
        full = precision == BF16
        model = _model(rng, 1024 if full else 384, 16 if full else 6)
        seq = round(_log(rng, 64, 8192 if full else 512))
        if rng.random() < 0.5:
            seq = max(128, 128 * round(seq / 128))
        batch = max(1, round(_log(rng, 512, 16384 if full else 4096) / seq))
        accum = rng.choice([1, 1, 2])
        if kind == "evaluate":
            c = _infer(None, kind, model, seq, batch=batch, accum=accum, precision=precision)
        else:
            c = _train(None, model, seq, batch, accum, precision, rng.choice(["device", "pipeline"]), rng.random() < 0.25, rng.random() < 0.25,
                       rng.choice([0.0, 1.0]), full and rng.random() < 0.25)
        # fp32, and heads of 128 at a sequence length that is no whole number of tiles, are a fraction of the tensor-core paths' rate
        ragged_128 = full and model["d"] // model["heads"] == 128 and seq % 128 != 0
        if batch * seq <= 16384 and work(c)["flops"] <= (2.0e11 if ragged_128 or not full else 1.2e13):
            return c


# ---------------------------------------------------------------------------------------------- inputs
def _config(c):
    return nnb.GptConfig(c["vocab"], c["d"], c["heads"], c["layers"], c["ff"], c["seq"], c["batch"], c["act"], c["norm"], c["pos"], c["precision"])


def _trainer(c, gen):
    """A trainer in mid-run: weights N(0, 0.02), norm scales near 1, moments of the size gradients have, step 1000."""
    tr = nnb.GptTrainer(_config(c), lr=3e-4, muon=bool(c.get("muon")), muon_lr=0.01)
    tr.params.normal_(0.0, 0.02, generator=gen)
    for name, (off, r, k) in zip(tr.param_names(), tr.table):
        if name.endswith(".gamma"):
            tr.params[off:off + r * k].add_(1.0)
    tr.refresh_shadow()
    if c["kind"] == "train":
        tr.m.normal_(0.0, 1e-5, generator=gen)
        tr.v.uniform_(5e-10, 1.5e-9, generator=gen)
        tr.t = 1000
    return tr


def _batch(c, gen, zipf):
    """Token ids Zipf(1.1), labels the next token; documents of geometric length (mean 300); a mask without the padding."""
    B, S = c["batch"], c["seq"]
    u = torch.rand(B, S + 1, device="cuda", generator=gen)
    ids = torch.searchsorted(zipf, u).clamp_(max=c["vocab"] - 1).to(torch.int32)
    tokens, labels = ids[:, :-1].contiguous().view(-1), ids[:, 1:].contiguous().view(-1)
    docs = mask = None
    if c.get("docs"):
        docs = (torch.rand(B, S, device="cuda", generator=gen) < 1.0 / 300.0).to(torch.int32).cumsum(1, dtype=torch.int32).contiguous().view(-1)
    if c.get("mask"):
        length = torch.randint(S // 2, S + 1, (B, 1), device="cuda", generator=gen)
        mask = (torch.arange(S, device="cuda")[None, :] < length).to(torch.float32).contiguous().view(-1)
    return tokens, labels, mask, docs


def _normal(gen, *shape, std=1.0):
    return torch.randn(*shape, device="cuda", generator=gen) * std


def prepare(case, seed):
    c = dict(case)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if c["kind"] == "engine_linear":
        m, k, n = c["out"], c["inp"], c["tokens"]
        s = dict(c=c, W=_normal(gen, m, k, std=0.02), b=_normal(gen, m, std=0.02), X=_normal(gen, k, n), G=_normal(gen, m, n, std=1e-3), acc=_normal(gen, m, k, std=1e-3))
        s.update({k_: torch.empty(shape, device="cuda") for k_, shape in
                  (("mm", (m, n)), ("Y", (m, n)), ("dW", (m, k)), ("gradW", (m, k)), ("db", (m,)), ("dX", (k, n)))})
        return s
    if c["kind"] == "engine_attention":
        h, S, dk = c["heads"], c["seq"], c["dk"]
        causal = torch.full((S, S), -math.inf, device="cuda").triu_(1)
        s = dict(c=c, Q=_normal(gen, h * dk, S), K=_normal(gen, h * dk, S), V=_normal(gen, h * S, dk), G=_normal(gen, h * S, dk, std=1e-3), mask=causal)
        s.update({k_: torch.empty(shape, device="cuda") for k_, shape in
                  (("row_max", (h * S,)), ("denom", (h * S,)), ("O", (h * S, dk)), ("P", (h * S, S)), ("R", (h * S,)),
                   ("dQ", (h * dk, S)), ("dK", (h * dk, S)), ("dV", (h * dk, S)))})
        return s
    tr = _trainer(c, gen)
    zipf = torch.arange(1, c["vocab"] + 1, device="cuda", dtype=torch.float64).pow_(-1.1).cumsum_(0)
    zipf = (zipf / zipf[-1]).to(torch.float32)
    if c["kind"] in ("train", "evaluate"):
        batches = [_batch(c, gen, zipf) for _ in range(c["accum"])]
        if c.get("feed") == "pipeline":
            batches = [tuple(None if t is None else t.cpu() for t in b) for b in batches]
            return dict(c=c, tr=tr, batches=batches, pipe=nnb.AsyncInputPipeline(tr))
        return dict(c=c, tr=tr, batches=batches)
    prompt = torch.searchsorted(zipf, torch.rand(c["context"] + 1, device="cuda", generator=gen)).clamp_(max=c["vocab"] - 1).tolist()
    if c["kind"] == "step":
        tr.generate(prompt[:-1], 0)                     # fills the cache
        return dict(c=c, tr=tr, token=prompt[-1])
    return dict(c=c, tr=tr, prompt=prompt[:-1])


# ---------------------------------------------------------------------------------------------- one pass
def _p(t):
    return C.c_void_p(t.data_ptr())


def _engine_linear(s):
    """Linear::forward (matmul, bias broadcast) and ::backward (weight gradient added up, bias gradient, input gradient)."""
    m, k, n = s["c"]["out"], s["c"]["inp"], s["c"]["tokens"]
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    nnb.call("cuda_matmul", _p(s["W"]), _p(s["X"]), _p(s["mm"]), m, k, k, n, 0, 0, st)
    nnb.call("cuda_broadcast_row", _p(s["mm"]), _p(s["b"]), _p(s["Y"]), m, n, 0, st)
    nnb.call("cuda_matmul", _p(s["G"]), _p(s["X"]), _p(s["dW"]), m, n, k, n, 0, 1, st)
    nnb.call("cuda_elementwise_binary", _p(s["acc"]), _p(s["dW"]), _p(s["gradW"]), m * k, 0, st)
    nnb.call("cuda_reduce_row", _p(s["G"]), _p(s["db"]), m, n, 0, st)
    nnb.call("cuda_matmul", _p(s["W"]), _p(s["G"]), _p(s["dX"]), m, k, m, n, 1, 0, st)
    return {k_: s[k_] for k_ in ("Y", "gradW", "db", "dX")}


def _engine_attention(s):
    """The two-pass attention of the reference's layers: row maxima, denominators, values; then the gradients."""
    h, S, dk = s["c"]["heads"], s["c"]["seq"], s["c"]["dk"]
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    alpha = C.c_float(1.0 / math.sqrt(dk))
    Q, K, V, G, mask, mx, den, P = (_p(s[k]) for k in ("Q", "K", "V", "G", "mask", "row_max", "denom", "P"))
    nnb.call("nnb200_bmm_reduce", Q, K, mask, mx, h, S, S, dk, 1, 1, 0, alpha, 1, st)
    nnb.call("nnb200_bmm_softmax_denom", Q, K, mx, mask, den, h, S, S, dk, 1, 0, alpha, st)
    nnb.call("nnb200_bmm_softmax_apply", Q, K, V, mx, den, mask, _p(s["O"]), h, S, S, dk, dk, 1, 0, alpha, st)
    nnb.call("nnb200_batched_matmul", G, V, P, h * S, dk, h * S, dk, h, 0, 1, C.c_float(1.0), st)
    nnb.call("nnb200_bmm_softmax_backward_q", Q, K, P, mx, den, mask, _p(s["dQ"]), _p(s["R"]), h, S, S, dk, 1, 0, alpha, st)
    nnb.call("nnb200_bmm_softmax_backward_kv", Q, K, P, G, _p(s["R"]), mx, den, mask, _p(s["dK"]), _p(s["dV"]), h, S, S, dk, dk, 1, 0, alpha, st)
    return {k: s[k] for k in ("row_max", "denom", "O", "P", "R", "dQ", "dK", "dV")}


def run(state):
    c = state["c"]
    if c["kind"] == "engine_linear":
        return _engine_linear(state)
    if c["kind"] == "engine_attention":
        return _engine_attention(state)
    tr = state["tr"]
    if c["kind"] == "evaluate":
        loss = tr.evaluate(state["batches"])
        return {"loss": loss, "logit_gradient": tr.logits()}
    if c["kind"] == "step":
        return tr.forward_step(state["token"], c["context"], c["context"])
    if c["kind"] == "generate":
        tokens = tr.generate(state["prompt"], c["new"], temperature=0.0)
        last = c["context"] + c["new"] - 1
        return {"tokens": np.array(tokens, np.int64), "logits": tr.forward_step(tokens[-1], last, last)}
    n = c["accum"]
    if c["feed"] == "pipeline":
        pipe = state["pipe"]
        for i, b in enumerate(state["batches"]):
            pipe.submit(*b)
            pipe.run(grad_scale=1.0 / n, last=i == n - 1)
    else:
        for i, b in enumerate(state["batches"]):
            tr.micro_step(*b, grad_scale=1.0 / n, last=i == n - 1)
    tr.optimizer_step(clip=c["clip"] or None)
    return {"loss": tr.loss_tensor(), "params": tr.params, "m": tr.m, "v": tr.v}


# ---------------------------------------------------------------------------------------------- floors and tolerances
def _sizes(c):
    d, ff, V, L = c["d"], c["ff"], c["vocab"], c["layers"]
    matrices = L * (4 * d * d + (3 if c["act"] == SWIGLU else 2) * d * ff)
    embeddings = V * d + (c["seq"] * d if c["pos"] == LEARNED else 0)
    return matrices, V * d, embeddings


def work(case):
    c = case
    if c["kind"] == "engine_linear":
        m, k, n = c["out"], c["inp"], c["tokens"]
        # W, X, G, the accumulator and the bias read; Y, the weight, bias and input gradients written
        return {"bytes": 4.0 * (m * k + k * n + m * n + m * k + m + m * n + m * k + m + k * n), "flops": 6.0 * m * k * n}
    if c["kind"] == "engine_attention":
        h, S, dk = c["heads"], c["seq"], c["dk"]
        # Q, K, V, G, mask read; O, dQ, dK, dV, P, row statistics written.  Seven products: S, O, P, S again in each of the
        # two gradient calls (their inputs do not hold it), dQ, dK, dV - the causal half, except P, which is whole
        return {"bytes": 4.0 * (8 * h * S * dk + S * S + h * S * S + 3 * h * S), "flops": 2.0 * h * S * S * dk * (7 * 0.5 + 1.0)}
    matrices, head, embeddings = _sizes(c)
    wbytes = 2.0 if c["precision"] == BF16 else 4.0
    if c["kind"] in ("step", "generate"):
        read = wbytes * (matrices + head)
        n, cached = (1, c["context"]) if c["kind"] == "step" else (c["new"], c["context"] + c["new"] / 2)
        # every generated token reads the weights and the cached keys and values (fp32); the prompt reads the weights once
        kv = 8.0 * c["layers"] * c["d"] * cached
        flops = 2.0 * (matrices + head) * n + 4.0 * c["layers"] * c["d"] * cached * n
        total = n * (read + kv)
        if c["kind"] == "generate":
            total += read + 8.0 * c["layers"] * c["d"] * c["context"]
            flops += 2.0 * matrices * c["context"] + 2.0 * c["layers"] * c["d"] * c["context"] ** 2
        return {"bytes": total, "flops": flops}
    N = c["batch"] * c["seq"]
    keys = min(300.0, c["seq"]) if c.get("docs") else (c["seq"] + 1) / 2.0     # keys a query may attend to, on average
    per_token = 2.0 * (matrices + head) + 4.0 * c["layers"] * c["d"] * keys
    if c["kind"] == "evaluate":
        logits = 2.0 if c["precision"] == BF16 else 4.0
        return {"bytes": wbytes * (matrices + head) + 4.0 * embeddings + N * c["vocab"] * logits, "flops": per_token * N * c["accum"]}
    params = matrices + head + embeddings
    flops = 3.0 * per_token * N * c["accum"]
    if c.get("muon"):
        d, ff = c["d"], c["ff"]
        ns = lambda a, b: 5.0 * (4.0 * min(a, b) ** 2 * max(a, b) + 2.0 * min(a, b) ** 3)      # five Newton-Schulz iterations of one matrix
        flops += c["layers"] * (4 * ns(d, d) + ns(ff * (2 if c["act"] == SWIGLU else 1), d) + ns(d, ff))
    # weights read once, gradients written and read, parameters and both moments read and written, the bf16 copy written
    return {"bytes": params * (wbytes + 8.0 + 24.0 + (2.0 if c["precision"] == BF16 else 0.0)) + 8.0 * N * c["accum"], "flops": flops}


def tolerance(case):
    if case["kind"] in ("engine_linear", "engine_attention"):
        return {"rel": 1e-5, "max": 1e-3}                  # fp32 sums of up to 8192 terms, one exponential
    if case["kind"] in ("step", "generate"):
        return {"rel": 5e-5, "max": 1e-3, "differ": 0.0}   # fp32 activations through up to 16 layers; greedy tokens the same
    if case["precision"] == FP32:
        return {"rel": 3e-5, "max": 3e-3}                  # fp32 through up to 6 layers forward and backward; squares in the second moment
    return {"rel": 2e-2, "max": 0.8}                       # bf16 activations and gradients; single gradients cancel to less than their rounding
