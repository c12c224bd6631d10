"""Cases that stand for what a training program has this framework do, through its public entry points: whole training
steps (captured once and replayed, or run on the tape), forward passes without gradients, and the flat optimizer pass,
from a step of some ten microseconds to one of some ten milliseconds, in f32, bf16 and f16.

A case is a dict; `kind` says which program it is:
  mlp, cnn, encoder, decoder   the models built into the library, `mode` "static" (StaticStep, fed from pinned host memory every
                               step, its losses read one step behind) or "tape" (zero_grad, loss, backward, optimizer)
  block                        a pre-norm transformer block that the program composes from F.* itself, `mode` "train" or "eval"
  classifier                   a GELU classifier composed from F.*, trained on the tape with AdamW
  optimizer                    inf/nan check, unscale and Adam over one flat buffer (gradients f32 or bf16)
"""
import math

import numpy as np
import torch

import modernchainer_b200 as mc
from modernchainer_b200.api import BF16, F, F16, AdamW, MomentumSGD, Variable, clip_grad_norm

LOWP = {"bf16": BF16, "f16": F16}
_context = []


def context():
    """One context for the whole program, as a user's process has."""
    if not _context:
        _context.append(mc.Context(0))
    return _context[0]


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest training step: launches and latency are all there is (784-100-10, batch 128)
        dict(name="mlp_static", kind="mlp", mode="static", dtype="f32", batch=128, dims_in=784, hidden=100, classes=10),
        # a program's own classifier, widths and batch that nothing divides, trained on the tape
        dict(name="classifier_tape", kind="classifier", dtype="f32", batch=250, dims_in=1000, hidden=515, classes=37),
        # small CNN on 32x32x3 images, batch 256
        dict(name="cnn_static", kind="cnn", mode="static", dtype="f32", batch=256, cin=3, c1=32, c2=64, hw=32, classes=10),
        # 28x28 grey images, channel counts off the tensor-core grid, on the tape
        dict(name="cnn_tape_odd", kind="cnn", mode="tape", dtype="f32", batch=100, cin=1, c1=20, c2=50, hw=28, classes=10),
        # one encoder block at its benchmark size: d 512, 8 heads, FFN 2048, seq 256, batch 32, bf16
        dict(name="encoder_static_bf16", kind="encoder", mode="static", dtype="bf16", batch=32, seq=256, d=512, heads=8, ff=2048),
        # an image-patch sequence (odd length) in f16; the program waits for the scaler's verdict every step
        dict(name="encoder_tape_f16", kind="encoder", mode="tape", dtype="f16", batch=16, seq=197, d=768, heads=12, ff=3072),
        # full-precision training without autocast, the framework's default, with gradient clipping
        dict(name="block_train_f32", kind="block", mode="train", dtype="f32", batch=16, seq=100, d=256, heads=8, ff=1024),
        # a small language model, byte-sized vocabulary, on the tape: many small launches
        dict(name="decoder_tape_small", kind="decoder", mode="tape", dtype="bf16", batch=8, seq=256, d=256, heads=4, ff=1024, layers=4, vocab=256),
        # a middle-sized language model whose vocabulary is no multiple of anything, wide heads
        dict(name="decoder_static_odd", kind="decoder", mode="static", dtype="bf16", batch=6, seq=500, d=512, heads=4, ff=2048, layers=4, vocab=10007),
        # the headline configuration: 12 layers, d 768, vocabulary 32000, 8 x 1024 tokens, bf16
        dict(name="decoder_static_large", kind="decoder", mode="static", dtype="bf16", batch=8, seq=1024, d=768, heads=12, ff=3072, layers=12, vocab=32000),
        # scoring one short sequence: forward only
        dict(name="block_eval_bf16", kind="block", mode="eval", dtype="bf16", batch=1, seq=128, d=768, heads=12, ff=3072),
        # the optimizer pass alone: 125M parameters, bf16 gradients
        dict(name="optimizer_flat", kind="optimizer", dtype="bf16", n=125_000_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _transformer_sizes(rng, most_tokens, most_d):
    hd = rng.choice([32, 48, 64, 64, 64, 80, 96, 128])
    heads = max(1, min(_log(rng, 2, 16), most_d // hd))
    seq = min(_log(rng, 16, 2048), most_tokens)
    batch = max(1, min(_log(rng, 1, 64), most_tokens // seq))
    d = heads * hd
    return dict(batch=batch, seq=seq, d=d, heads=heads, ff=rng.choice([2 * d, 4 * d, 4 * d])), batch * seq


def draw(rng):
    kind = rng.choice(["mlp", "classifier", "cnn", "encoder", "encoder", "decoder", "decoder", "block", "block", "optimizer"])
    mode = rng.choice(["static", "tape"])
    if kind in ("mlp", "classifier"):
        case = dict(kind=kind, dtype="f32", batch=_log(rng, 1, 2048), dims_in=_log(rng, 8, 2048), hidden=_log(rng, 16, 2048), classes=_log(rng, 2, 1000))
        return dict(case, mode=mode) if kind == "mlp" else case
    if kind == "cnn":
        case = dict(kind=kind, mode=mode, dtype="f32", cin=rng.choice([1, 3]), c1=_log(rng, 8, 64), c2=_log(rng, 8, 128), hw=4 * rng.randint(4, 16), classes=_log(rng, 2, 200))
        per_image = case["hw"] ** 2 * case["c1"] * (case["cin"] + case["c2"] / 4)
        return dict(case, batch=max(1, min(_log(rng, 1, 512), int(4e8 / per_image))))
    if kind == "optimizer":
        return dict(kind=kind, dtype=rng.choice(["bf16", "f32"]), n=_log(rng, 20_000, 125_000_000))
    dtype = rng.choice(["bf16", "bf16", "bf16", "f16", "f32"])
    full = dtype == "f32"
    sizes, tokens = _transformer_sizes(rng, 2048 if full else 8192, 512 if full else 1024)
    if kind == "encoder":
        return dict(sizes, kind=kind, mode=mode, dtype=dtype)
    if kind == "block":
        return dict(sizes, kind=kind, mode=rng.choice(["train", "eval"]), dtype=dtype)
    layers = rng.randint(1, 3 if full else 6)
    vocab = _log(rng, 200, 32000)
    if rng.random() < 0.5:
        vocab = (vocab + 63) // 64 * 64
    most = 4e9 if full else (2e10 if vocab % 8 else 2.6e11)
    vocab = max(200, min(vocab, int(most / (tokens * sizes["d"])) // 8 * 8 + vocab % 8))
    return dict(sizes, kind=kind, mode=mode, dtype=dtype, layers=layers, vocab=vocab)


# ------------------------------------------------------------------ what a program has in hand
class Outcome(dict):
    """What one pass left behind.  Loss, parameters, gradients and activations stay on the device, as in a training loop;
    looking at an entry reads it back."""

    def __init__(self, **readers):
        super().__init__(readers)

    def __getitem__(self, key):
        return super().__getitem__(key)()


def _flat(values):
    return np.concatenate([np.ravel(v) for v in values])


def _trained(loss, params, gradients=True):
    out = Outcome(loss=loss, parameters=lambda: _flat(p.data for p in params))
    if gradients:  # a replayed step keeps its gradients to itself
        dict.__setitem__(out, "gradients", lambda: _flat(p.grad for p in params))
    return out


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _io(case, rng):
    """Inputs and targets of one batch."""
    kind, b = case["kind"], case["batch"]
    if kind in ("mlp", "classifier"):
        return rng.standard_normal((b, case["dims_in"]), dtype=np.float32), rng.integers(0, case["classes"], b)
    if kind == "cnn":
        return rng.random((b, case["cin"], case["hw"], case["hw"]), dtype=np.float32), rng.integers(0, case["classes"], b)
    if kind == "decoder":  # next-token prediction
        ids = rng.integers(0, case["vocab"], (b, case["seq"] + 1))
        return np.ascontiguousarray(ids[:, :-1]), np.ascontiguousarray(ids[:, 1:])
    shape = (b, case["seq"], case["d"])
    return rng.standard_normal(shape, dtype=np.float32), rng.standard_normal(shape, dtype=np.float32)


def _model_cfg(case, seed):
    if case["kind"] == "mlp":
        return [case["dims_in"], case["hidden"], case["classes"]]
    if case["kind"] == "cnn":
        return [case["cin"], case["c1"], case["c2"], case["hw"], case["classes"]]
    if case["kind"] == "encoder":
        return [case["d"], case["heads"], case["ff"], 0]
    return [case["vocab"], case["d"], case["heads"], case["ff"], case["layers"], seed]


def _weights(ctx, rng, shapes):
    """Parameters of a composed model: He-normal matrices, unit gains (g), zero biases (b)."""
    p = {}
    for name, shape in shapes.items():
        if len(shape) == 2:
            w = rng.standard_normal(shape, dtype=np.float32) * np.float32(math.sqrt(2.0 / shape[1]))
        else:
            w = (np.ones if name.startswith("g") else np.zeros)(shape, np.float32)
        p[name] = Variable(ctx, w)
    return p


def _block_shapes(case):
    d, ff = case["d"], case["ff"]
    return dict(g1=(d,), b1=(d,), wq=(d, d), bq=(d,), wk=(d, d), bk=(d,), wv=(d, d), bv=(d,), wo=(d, d), bo=(d,),
                g2=(d,), b2=(d,), w1=(ff, d), bf1=(ff,), w2=(d, ff), bf2=(d,))


def prepare(case, seed):
    ctx, rng, kind = context(), np.random.default_rng(seed), case["kind"]
    s = dict(case=case, ctx=ctx)
    if kind == "optimizer":
        n, gen = case["n"], torch.Generator("cuda").manual_seed(seed)
        s["p"] = torch.randn(n, device="cuda", generator=gen) * 0.02
        s["m"] = torch.randn(n, device="cuda", generator=gen) * 1e-3
        s["v"] = torch.rand(n, device="cuda", generator=gen) * 1e-6
        g = torch.randn(n, device="cuda", generator=gen) * (1e-3 * 65536.0)
        s["g"] = g.bfloat16() if case["dtype"] == "bf16" else g
        s["shadow"] = torch.empty(n, device="cuda", dtype=torch.bfloat16)
        s["flag"] = torch.zeros(1, device="cuda", dtype=torch.int32)
        s["step"] = 100
        return s
    x, y = _io(case, rng)
    lowp = LOWP.get(case["dtype"])
    if kind in ("block", "classifier"):
        if kind == "block":
            shapes = _block_shapes(case)
        else:
            i, h, c = case["dims_in"], case["hidden"], case["classes"]
            shapes = dict(w1=(h, i), b1=(h,), w2=(h, h), b2=(h,), w3=(c, h), b3=(c,))
        s["weights"] = _weights(ctx, rng, shapes)
        s["params"] = list(s["weights"].values())
        s["opt"] = AdamW(ctx, 1e-3, 0.01) if kind == "classifier" else MomentumSGD(ctx, 1e-2, 0.9)
    else:
        s["model"] = mc.Model(ctx, kind, _model_cfg(case, seed))
        s["params"] = s["model"].parameters()
        # with Adam, an entry whose gradient is rounding noise (the key-projection bias) moves by the full rate in a random
        # direction: in f32 the transformers are trained with momentum, so that results can be compared to rounding
        if kind in ("mlp", "cnn"):
            s["opt"] = mc.Adam(ctx, 1e-3)
        else:
            s["opt"] = MomentumSGD(ctx, 1e-2, 0.9) if lowp is None else mc.Adam(ctx, 1e-4)
    s["arena"] = mc.Arena(ctx, s["params"])
    s["scaler"] = mc.GradScaler(ctx, 65536.0) if lowp is not None else None
    s["lowp"] = lowp
    if case.get("mode") == "static":
        s["x"], s["y"] = _pinned(x), _pinned(y)
        s["step"] = mc.StaticStep(s["model"], s["opt"], x, y, scaler=s["scaler"], autocast_dtype=lowp)
    else:
        s["x"], s["y"] = Variable.constant(ctx, x), Variable.constant(ctx, y)
    return s


# ------------------------------------------------------------------ one pass
def _block(s):
    case, p, x = s["case"], s["weights"], s["x"]
    b, n, d = case["batch"], case["seq"], case["d"]
    h = F.reshape(F.layer_norm(x, p["g1"], p["b1"], 1e-5), (b * n, d))
    q, k, v = (F.reshape(F.linear(h, p["w" + c], p["b" + c]), (b, n, d)) for c in "qkv")
    a = F.reshape(F.multi_head_attention(q, k, v, case["heads"], False), (b * n, d))
    x = F.add(x, F.reshape(F.linear(a, p["wo"], p["bo"]), (b, n, d)))
    h = F.reshape(F.layer_norm(x, p["g2"], p["b2"], 1e-5), (b * n, d))
    h = F.linear(F.linear_activation(h, p["w1"], p["bf1"], "gelu"), p["w2"], p["bf2"])
    return F.add(x, F.reshape(h, (b, n, d)))


def _loss(s):
    p, x, y = s.get("weights"), s["x"], s["y"]
    if s["case"]["kind"] == "classifier":
        h = F.gelu(F.linear(x, p["w1"], p["b1"]))
        h = F.gelu(F.linear(h, p["w2"], p["b2"]))
        return F.softmax_cross_entropy(F.linear(h, p["w3"], p["b3"]), y)
    if s["case"]["kind"] == "block":
        diff = F.sub(_block(s), y)
        return F.mean(F.mul(diff, diff))
    return s["model"].loss(x, y)


def _optimizer_pass(s):
    ctx, lib = s["ctx"], s["ctx"].lib
    g_dt, n = (mc.BF16 if s["case"]["dtype"] == "bf16" else mc.F32), s["case"]["n"]
    s["step"] += 1
    ctx.check(lib.mcb_memset(ctx.h, s["flag"].data_ptr(), 0, 4))
    ctx.check(lib.mcb_check_finite(ctx.h, s["g"].data_ptr(), g_dt, n, s["flag"].data_ptr()))
    ctx.check(lib.mcb_adam_flat(ctx.h, s["p"].data_ptr(), s["g"].data_ptr(), g_dt, s["m"].data_ptr(), s["v"].data_ptr(), s["shadow"].data_ptr(), n,
                                1e-3, 0.9, 0.999, 1e-8, s["step"], 1.0 / 65536.0, s["flag"].data_ptr()))
    return {k: s[k] for k in ("p", "m", "v", "shadow", "flag")}


def run(s):
    case, params = s["case"], s.get("params")
    if case["kind"] == "optimizer":
        return _optimizer_pass(s)
    if case.get("mode") == "static":
        s["step"].run_pipelined(s["x"], s["y"])
        return _trained(s["step"].loss, params, gradients=False)
    if case.get("mode") == "eval":
        with mc.no_grad():
            if s["lowp"] is None:
                y = _block(s)
            else:
                with mc.autocast(s["lowp"]):
                    y = _block(s)
        return Outcome(y=lambda: y.data)
    mc.zero_grad(params)
    if s["lowp"] is None:
        loss = _loss(s)
        loss.backward()
        if case["kind"] == "block":
            clip_grad_norm(params, 1.0)
        s["opt"].update(params)
    else:
        with mc.autocast(s["lowp"]):
            loss = _loss(s)
        s["scaler"].scale_loss(loss).backward()
        if case["kind"] == "encoder":
            s["scaler"].step(s["opt"], params)  # waits for the verdict, as the reference's loop does
        else:
            s["scaler"].step_async(s["opt"], params)
    return _trained(lambda: loss.data, params)


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "optimizer":  # p, m, v read and written, g read, the 16-bit copy written
        return {"bytes": case["n"] * (26.0 + (2.0 if case["dtype"] == "bf16" else 4.0)), "flops": 12.0 * case["n"]}
    b = case["batch"]
    if kind in ("mlp", "classifier"):
        i, h, c = case["dims_in"], case["hidden"], case["classes"]
        weights = i * h + h * c + (h * h if kind == "classifier" else 0)
        first = i * h  # the input needs no gradient
        macs, count, io = b * (3 * weights - first), weights + (2 * h if kind == "classifier" else h) + c, b * (4 * i + 8)
    elif kind == "cnn":
        hw, c0, c1, c2, c = case["hw"], case["cin"], case["c1"], case["c2"], case["classes"]
        conv1, conv2, fc = hw * hw * c1 * c0 * 9, (hw // 2) ** 2 * c2 * c1 * 9, c2 * (hw // 4) ** 2 * c
        macs, count, io = b * (2 * conv1 + 3 * conv2 + 3 * fc), c1 * c0 * 9 + c2 * c1 * 9 + fc + c1 + c2 + c, b * (4 * c0 * hw * hw + 8)
    else:
        t, d, ff = b * case["seq"], case["d"], case["ff"]
        layers = case.get("layers", 1)
        attn = layers * b * case["seq"] ** 2 * d * (0.5 if kind == "decoder" else 1.0)  # one of the two products of the forward pass
        weights, count = layers * (4 * d * d + 2 * d * ff), layers * (4 * d * d + 2 * d * ff + 9 * d + ff)
        if kind == "decoder":
            weights, count, io = weights + case["vocab"] * d, count + 2 * case["vocab"] * d + 2 * d, 16 * t
        else:
            io = 8 * t * d
        if case.get("mode") == "eval":
            return {"bytes": 4.0 * count + io, "flops": 2.0 * (t * weights + 2 * attn)}
        macs = 3 * t * weights + 7 * attn
    state = 2 if kind != "block" and not (case["dtype"] == "f32" and kind in ("encoder", "decoder")) else 1  # Adam's moments, or momentum
    return {"bytes": count * 4.0 * (3 + 2 * state) + io, "flops": 2.0 * macs}


def tolerance(case):
    kind, dtype, static = case["kind"], case["dtype"], case.get("mode") == "static"
    if kind == "optimizer":  # elementwise f32 arithmetic; the 16-bit copy may round the other way
        return {"rel": 1e-5, "max": 8e-3}
    if dtype in LOWP:
        if static:  # the updated parameters: where a gradient is no larger than its own rounding, Adam's step may have either sign
            return {"rel": 1e-3, "max": 0.1}
        if case.get("mode") == "eval":
            return {"rel": 1e-2 if dtype == "bf16" else 2e-3, "max": 0.1}
        # gradients and activations carry 8 (or 11) bits, and single entries of small tensors cancel: two ways to round the same
        # bf16 step differ by 1.8e-2 in the gradients of the second step
        return {"rel": 2.5e-2, "max": 0.9} if dtype == "bf16" else {"rel": 5e-3, "max": 0.5}
    if kind in ("mlp", "cnn"):  # a ReLU or max-pool decision that flips on the last bit moves a whole gradient path
        return {"rel": 1e-4 if static else 1e-3, "max": 0.1 if static else 0.5}
    if kind == "classifier":  # Adam's first steps divide each gradient by its own size
        return {"rel": 1e-4, "max": 0.1}
    return {"rel": 2e-5, "max": 5e-3}
