"""The work whose speed counts: training iterations and pipeline-stage token slices.

Three kinds of case, each through the package's public entry points:

* ``step``:  one training iteration, ``Trainer.train_step``: the input travels from pinned host
  memory, forward, backward and the mixed-precision Adam run on the device, the loss comes back.
* ``grads``: forward and backward without the optimizer, ``Trainer.compute_grads``, on an input
  that is on the device already.
* ``slice``: what one layer of a pipeline stage does for one token slice, forward and data
  gradients, through ``terapipe_b200.ops.functional``.  With several stages a ``Trainer`` runs
  exactly these calls between its transfers; one GPU has no neighbour, so they are called here
  directly.  The earlier slices' keys and values (the first ``ctx`` positions) and the later
  slices' output gradients are in the buffers, as they are in a stage.

Lists of lengths are texts ("3,2" or "128*16") because a case holds plain values only.
"""
import math

import torch

from terapipe_b200.models.config import MODEL_CONFIGS
from terapipe_b200.ops import functional as F
from terapipe_b200.runtime.trainer import Trainer

_DTYPE = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _step(name, model, layers, batch, batch_slices, seq_slices, dtype, activation, kind="step"):
    return {"name": name, "kind": kind, "model": model, "layers": layers, "batch": batch,
            "batch_slices": batch_slices, "seq_slices": seq_slices, "dtype": dtype,
            "activation": activation}


def _slice(name, hidden, head_dim, tp, seq, batch, tokens, ctx, dtype, activation):
    return {"name": name, "kind": "slice", "hidden": hidden, "head_dim": head_dim, "tp": tp,
            "seq": seq, "batch": batch, "tokens": tokens, "ctx": ctx, "dtype": dtype,
            "activation": activation}


def listed():
    return [
        # the smallest model of the registry with the slices of the correctness runs: a wall of
        # tiny kernels, where launches and latencies are all that counts
        _step("step test 8 slices", "test", 24, 2, "2", "16*8", "fp16", "gelu"),
        # a small model, unsliced, with the reference's own activation
        _step("step gpt2-1hm whole", "gpt2-1hm-single-device", 10, 4, "4", "2048", "fp16", "relu"),
        # the headline workload (GPT3-1B shape, batch 8, 16 uniform slices) in its one-device depth
        _step("step gpt3-1b 16 slices", "gpt3-1b-single-device", 5, 8, "8", "128*16", "fp16", "gelu"),
        # 13B width with the planner's 8 slices
        _step("step gpt3-13b 8 slices", "gpt3-13b-single-device", 1, 8, "8", "256*8", "fp16", "gelu"),
        # heads of 80 columns, an odd batch, decreasing slices as the planner gives them
        _step("step gpt3-2b uneven", "gpt3-2b-single-device", 3, 3, "3", "424,376,344,320,304,280",
              "bf16", "gelu"),
        # batch and token slices together, nothing a multiple of a tile: 25 heads, batch 3 + 2
        _step("step gpt2-1b batch slices", "gpt2-1b-single-device", 4, 5, "3,2",
              "297,281,265,257,251,241,233,223", "fp16", "gelu"),
        # the widest layer (GPT3-175B), 8 slices, few tokens for its weights: the largest case
        _step("step gpt3-175b wide", "gpt3-175b-single-node", 1, 2, "2", "256*8", "fp16", "gelu"),
        # gradients without the optimizer (evaluation of another optimizer, verification runs)
        _step("grads gpt3-3hm", "gpt3-3hm", 4, 2, "2", "512*4", "bf16", "gelu", kind="grads"),
        # one stage's slice of the headline pipeline, at the end of the sequence
        _slice("slice 1b last", 2048, 128, 1, 2048, 8, 128, 1920, "fp16", "gelu"),
        # ... of the 13B pipeline (tensor parallel 2), early in the sequence
        _slice("slice 13b early", 5120, 128, 2, 2048, 8, 256, 256, "fp16", "gelu"),
        # ... of the 44B pipeline (tensor parallel 4): a long slice of a small batch
        _slice("slice 44b long", 6144, 128, 4, 2048, 4, 512, 768, "bf16", "gelu"),
        # a short ragged slice of a small model: batch 1, 64-column heads, odd lengths
        _slice("slice small ragged", 768, 64, 1, 1024, 1, 77, 299, "fp16", "relu"),
    ]


_SINGLE = ("test", "gpt2-1hm-single-device", "gpt2-3hm-single-device", "gpt2-1b-single-device",
           "gpt3-1hm", "gpt3-3hm", "gpt3-7hm", "gpt3-1b-single-device",
           "gpt3-2b-single-device", "gpt3-6b-single-device", "gpt3-13b-single-device", "megatron-1b")
_MOST_FLOPS = 3.5e13


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _partition(rng, total, parts):
    """`parts` lengths that add up to `total`: uniform, or decreasing with an odd remainder."""
    if parts == 1 or (total % parts == 0 and rng.random() < 0.4):
        return "%d*%d" % (total // parts, parts)
    weights = sorted((1.0 + rng.random() for _ in range(parts)), reverse=True)
    lengths = [max(1, int(total * w / sum(weights))) for w in weights]
    lengths[0] += total - sum(lengths)
    return ",".join(str(v) for v in lengths)


def draw(rng):
    # ReLU is what the reference's layer computes, and it knows fp16 only
    dtype, activation = rng.choice((("fp16", "gelu"), ("fp16", "relu"), ("bf16", "gelu")))
    if rng.random() < 0.4:
        hidden, head_dim = rng.choice(((768, 64), (1024, 64), (1600, 64), (2048, 128), (4096, 128),
                                       (5120, 128), (6144, 128)))
        heads = hidden // head_dim
        tp = rng.choice([n for n in (1, 2, 4) if heads % n == 0])
        seq = rng.choice((1024, 2048, 2048, 4096))
        batch = rng.randint(1, 8)
        tokens = _log_int(rng, 16, min(1024, 4096 // batch))
        ctx = rng.randint(0, seq - tokens)
        if rng.random() < 0.5:      # uniform schedules: everything a multiple of 8
            tokens, ctx = max(8, tokens // 8 * 8), ctx // 8 * 8
        case = _slice("", hidden, head_dim, tp, seq, batch, tokens, ctx, dtype, activation)
    else:
        kind = "grads" if activation == "gelu" and rng.random() < 0.35 else "step"
        model = rng.choice(_SINGLE)
        layers = MODEL_CONFIGS[model][0]
        layers = rng.randint(1, min(layers, 5 if kind == "grads" else 12))
        seq = MODEL_CONFIGS[model][2]
        batch = rng.randint(1, 8)
        batch_slices = "%d" % batch
        if batch > 1 and rng.random() < 0.3:
            first = rng.randint(1, batch - 1)
            batch_slices = "%d,%d" % (max(first, batch - first), min(first, batch - first))
        seq_slices = _partition(rng, seq, rng.choice((1, 2, 4, 6, 8, 13, 16)))
        case = _step("", model, layers, batch, batch_slices, seq_slices, dtype, activation, kind)
        while work(case)["flops"] > _MOST_FLOPS:
            if case["layers"] > 1:
                case["layers"] -= 1
            else:
                case["batch"] -= 1
                case["batch_slices"] = "%d" % case["batch"]
    del case["name"]
    return case


# ------------------------------------------------------------------------------- preparation
def _lengths(text):
    out = []
    for part in text.split(","):
        n, _, times = part.partition("*")
        out += [int(n)] * int(times or 1)
    return out


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _prepare_trainer(case, seed):
    # a loss scale that keeps the gradients of mean(output) in fp16's normal range
    trainer = Trainer(case["model"], batch_size=case["batch"], n_layers=case["layers"],
                      batch_slices=_lengths(case["batch_slices"]),
                      seq_slices=_lengths(case["seq_slices"]), dtype=case["dtype"],
                      activation=case["activation"], lr=1e-6, seed=seed, loss_scale=32768.0)
    c = trainer.config
    # hidden states as an embedding that is not quite centred gives them
    x = torch.randn(c.seq_len, c.batch_size, c.embedding_dim, device="cuda", generator=_generator(seed))
    x = (x + 0.25).to(_DTYPE[case["dtype"]])
    return {"trainer": trainer, "x": x.cpu().pin_memory() if case["kind"] == "step" else x}


def _prepare_slice(case, seed):
    g, dt = _generator(seed), _DTYPE[case["dtype"]]
    H, D, tp = case["hidden"], case["head_dim"], case["tp"]
    h = H // D // tp                       # heads, attention width and FFN width of this rank
    Hl, Fl = h * D, 4 * H // tp
    L, b, t, c = case["seq"], case["batch"], case["tokens"], case["ctx"]
    T = t * b

    def normal(*shape, std=1.0, dtype=dt):
        return (torch.randn(*shape, device="cuda", generator=g) * std).to(dtype)

    def weight(n, k):
        return normal(n, k, std=math.sqrt(2.0 / (n + k)))

    def empty(*shape, dtype=dt):
        return torch.empty(*shape, device="cuda", dtype=dtype)

    f32 = torch.float32
    s = {"D": D, "h": h, "b": b, "t": t, "c": c, "L": L, "act": case["activation"],
         "x": normal(T, H), "dy": normal(T, H, std=1e-2),
         "w_qkv": weight(3 * Hl, H), "b_qkv": normal(3 * Hl, std=0.02), "w_o": weight(H, Hl),
         "b_o": normal(H, std=0.02), "w_1": weight(Fl, H), "b_1": normal(Fl, std=0.02),
         "w_2": weight(H, Fl), "b_2": normal(H, std=0.02),
         "g1": 1 + normal(H, std=0.05), "e1": normal(H, std=0.05),
         "g2": 1 + normal(H, std=0.05), "e2": normal(H, std=0.05),
         "qkv": normal(L, b, 3 * Hl), "do": normal(L * b, Hl, std=1e-2),
         "lse": empty(b * h, L, dtype=f32), "delta": empty(b * h, L, dtype=f32)}
    # what the other slices of the sequence have left behind: their outputs' statistics
    o = empty(L * b, Hl)
    F.attn_fwd(s["qkv"], b, h, D, L, 0, o, s["lse"])
    s["delta"].copy_((o.float() * s["do"].float()).view(L, b, h, D).sum(-1).permute(1, 2, 0).reshape(b * h, L))
    for name, width in (("ln1", H), ("xmid", H), ("ln2", H), ("y", H), ("ao", Hl), ("fa", Fl), ("fz", Fl),
                        ("dfc", Fl), ("dln", H), ("dmid", H), ("dqkv", 3 * Hl), ("dx", H)):
        s[name] = empty(T, width)
    for name in ("m1", "r1", "m2", "r2"):
        s[name] = empty(T, dtype=f32)
    for name in ("dg1", "de1", "dg2", "de2"):
        s[name] = torch.zeros(H, device="cuda")
    s["scratch"] = empty(F.layernorm_bwd_scratch_floats(T, H), dtype=f32)
    return s


def prepare(case, seed):
    return _prepare_slice(case, seed) if case["kind"] == "slice" else _prepare_trainer(case, seed)


# ------------------------------------------------------------------------------- one pass
def _run_slice(s):
    b, h, D, t, c, L = s["b"], s["h"], s["D"], s["t"], s["c"], s["L"]
    act, T = s["act"], t * b
    fz = s["fz"] if act == "gelu" else None
    rows = slice(c * b, c * b + T)
    qkv, dao = s["qkv"].view(L * b, -1)[rows], s["do"][rows]
    # forward of the layer
    F.layernorm_fwd(s["x"], s["g1"], s["e1"], s["ln1"], s["m1"], s["r1"])
    F.gemm(s["ln1"], s["w_qkv"], qkv, bias=s["b_qkv"])
    F.attn_fwd(s["qkv"], b, h, D, t, c, s["ao"], s["lse"])
    F.gemm(s["ao"], s["w_o"], s["xmid"], bias=s["b_o"], residual=s["x"])
    F.layernorm_fwd(s["xmid"], s["g2"], s["e2"], s["ln2"], s["m2"], s["r2"])
    F.gemm(s["ln2"], s["w_1"], s["fa"], bias=s["b_1"], act=act, aux_out=fz)
    F.gemm(s["fa"], s["w_2"], s["y"], bias=s["b_2"], residual=s["xmid"])
    # data gradients of the layer
    F.gemm(s["dy"], s["w_2"], s["dfc"], b_mn=True, dact=act, aux_in=s["fa"] if fz is None else fz)
    F.gemm(s["dfc"], s["w_1"], s["dln"], b_mn=True)
    F.layernorm_bwd(s["dln"], s["xmid"], s["m2"], s["r2"], s["g2"], s["dmid"], s["dg2"], s["de2"],
                    s["scratch"], dres=s["dy"])
    F.gemm(s["dmid"], s["w_o"], dao, b_mn=True)
    F.attn_bwd(s["qkv"], b, h, D, t, c, L, s["ao"], s["do"], s["lse"], s["delta"], s["dqkv"])
    F.gemm(s["dqkv"], s["w_qkv"], s["dln"], b_mn=True)
    F.layernorm_bwd(s["dln"], s["x"], s["m1"], s["r1"], s["g1"], s["dx"], s["dg1"], s["de1"],
                    s["scratch"], dres=s["dmid"])
    out = {"qkv": qkv, "ao": s["ao"], "lse": s["lse"][:, c:c + t], "xmid": s["xmid"], "fa": s["fa"],
           "y": s["y"], "dmid": s["dmid"], "dqkv": s["dqkv"], "dx": s["dx"],
           "delta": s["delta"][:, c:c + t], "dg1": s["dg1"], "de1": s["de1"], "dg2": s["dg2"],
           "de2": s["de2"], "m1": s["m1"], "r1": s["r1"], "m2": s["m2"], "r2": s["r2"]}
    if act == "gelu":
        # (single elements of it are all or nothing under ReLU, where the sign of a value that is
        # zero to rounding decides; dmid, dx and the LayerNorm gradients are made from all of it)
        out["dfc"] = s["dfc"]
    return out


def run(state):
    if "trainer" not in state:
        return _run_slice(state)
    trainer = state["trainer"]
    if state["x"].is_cuda:
        return trainer.compute_grads(state["x"])
    loss = trainer.train_step(state["x"])
    e = trainer.engine
    return {"loss": loss, "output": e.output(), "master": e.master, "exp_avg": e.exp_avg,
            "exp_avg_sq": e.exp_avg_sq}


# ------------------------------------------------------------------------------- what it takes
def work(case):
    if case["kind"] == "slice":
        H, D, tp = case["hidden"], case["head_dim"], case["tp"]
        h = H // D // tp
        Hl, Fl = h * D, 4 * H // tp
        L, b, t, c = case["seq"], case["batch"], case["tokens"], case["ctx"]
        T = t * b
        weights = 4 * H * Hl + 2 * H * Fl
        own, past, later = t * (t + 1) / 2, t * c, t * (L - c - t)
        # pairs of a query and a key: forward and dQ see the past and the slice itself, dK / dV
        # the slice itself and the later queries (scores of the shared pairs computed once)
        pairs = 4 * (past + own) + 6 * past + 10 * own + 8 * later
        flops = 4.0 * T * weights + b * h * D * pairs
        values = (2 * weights + T * (2 * H + 3 * Hl)           # both passes' weights, x, dy, qkv
                  + 2 * c * b * Hl + 2 * (L - c - t) * b * Hl   # cached K, V; later Q, dO
                  + T * (3 * H + 2 * Hl + 2 * Fl + 3 * Hl + H))
        return {"bytes": 2.0 * values, "flops": flops}
    n_layers, (_, H, L, heads) = case["layers"], MODEL_CONFIGS[case["model"]]
    rows = L * case["batch"]
    weights, params = 12 * H * H, 12 * H * H + 13 * H
    # per layer: three products per weight; attention over the causal half, two products forward
    # and five backward
    flops = n_layers * (6.0 * rows * weights + 14.0 * case["batch"] * H * (L * (L + 1) / 2))
    # the input and the output once; per parameter the 16-bit value and either the fp32 gradient
    # or the optimizer's three fp32 values both ways and the new 16-bit value
    per_param = 6 if case["kind"] == "grads" else 2 + 24 + 2
    return {"bytes": 4.0 * rows * H + n_layers * params * per_param, "flops": flops}


def tolerance(case):
    # About four times what the outputs differ by from the same computation in 64 bits, rounded to
    # 16 bits at the same places (slice: fp16 5.7e-4, bf16 4.2e-3, fp16 with ReLU 4.9e-3, where
    # the sign of a value that is zero to rounding decides about a whole term), or from the fp32
    # pipeline with the same weights (24 layers in fp16 1.3e-3, 12 layers in bf16 8e-3).
    if case["kind"] == "slice":
        rel = 0.017 if case["dtype"] == "bf16" else 0.0025 if case["activation"] == "gelu" else 0.02
    else:
        rel = 0.005 if case["dtype"] == "fp16" else 0.03
    return {"rel": rel}
