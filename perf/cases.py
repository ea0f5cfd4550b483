"""The work whose speed this framework is judged by: single layers and whole training steps
through the public entry points, from the smallest layer of LeNet to a CosmoFlow step.

A case is a dict of plain values; ``prepare`` makes its state on the GPU from a seed, ``run`` does
one pass, ``exact`` is the same pass in 64-bit PyTorch.  Layers run forward and backward on 16-bit
activations with fp32 master weights and fp32 gradient buffers, as the executor calls them; models
are built from the front end and stepped with ``train_step`` / ``evaluate_step``.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

import lbann_b200 as lbann
from lbann_b200.data.readers import ArrayReader
from lbann_b200.exec.trainer import ExecTrainer
from lbann_b200.models.cosmoflow import construct_cosmoflow_model
from lbann_b200.models.transformer import construct_gpt_model
from lbann_b200.ops import native, nn
from lbann_b200.ops.attention import attention_packed
from lbann_b200.utils import options

_DT = {"bf16": torch.bfloat16, "fp16": torch.float16}
_SLOPE = 0.3            # leaky-ReLU slope of CosmoFlow
_LR = 1e-5              # small enough that hundreds of steps on one mini-batch stay in fp16 range
_EPS = 1e-5


# ------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # LeNet's first fully-connected layer at its mini-batch of 64: launches and host time count
        dict(name="fc_lenet", kind="linear", rows=64, cin=400, cout=120, act="relu", dtype="bf16"),
        # a dense layer whose sizes are no multiples of anything (tabular and auto-encoder models)
        dict(name="fc_ragged", kind="linear", rows=1000, cin=1155, cout=777, act="none", dtype="bf16"),
        # feed-forward projection of the GPT benchmark over four sequences of tokens
        dict(name="fc_tokens", kind="linear", rows=8192, cin=2048, cout=8192, act="none", dtype="bf16"),
        # causal self-attention of the GPT benchmark (16 heads of 128), two sequences
        dict(name="attention_gpt", kind="attention", batch=2, seq=2048, heads=16, causal=True, dtype="bf16"),
        # an encoder's short bidirectional attention
        dict(name="attention_encoder", kind="attention", batch=3, seq=384, heads=4, causal=False, dtype="fp16"),
        # ResNet-50: a 3x3 convolution + batch norm + ReLU of the first stage
        dict(name="conv2d_stage1", kind="conv", batch=32, cin=64, cout=64, d=0, h=56, w=56, k=3, stride=1, dtype="bf16"),
        # ResNet-50: the strided 3x3 convolution at the head of the second stage
        dict(name="conv2d_stride2", kind="conv", batch=32, cin=128, cout=128, d=0, h=56, w=56, k=3, stride=2,
             dtype="bf16"),
        # 3-D U-Net: first convolution of the second level, on a volume that is no power of two
        dict(name="conv3d_unet", kind="conv", batch=1, cin=32, cout=64, d=45, h=52, w=60, k=3, stride=1, dtype="bf16"),
        # the headline workload: one CosmoFlow training step, 128^3 volumes, mini-batch 8, fp16 + AMP
        dict(name="cosmoflow_128", kind="cosmoflow", width=128, batch=8, dtype="fp16"),
        # the per-GPU share of a larger job: one 64^3 volume
        dict(name="cosmoflow_64", kind="cosmoflow", width=64, batch=1, dtype="fp16"),
        # a training step of a GPT decoder (embedding, two blocks, 50304-word head, Adam)
        dict(name="gpt_train", kind="gpt", layers=2, d_model=1024, heads=8, seq=1024, vocab=50304, batch=4, train=True,
             dtype="bf16"),
        # scoring one sequence with the same network: forward only
        dict(name="gpt_evaluate", kind="gpt", layers=2, d_model=1024, heads=8, seq=512, vocab=50304, batch=1, train=False,
             dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "attention", "attention", "conv", "conv", "cosmoflow", "gpt"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "linear":
        rows, cin, cout = _log(rng, 1, 16384), _log(rng, 16, 8192), _log(rng, 8, 8192)
        if rng.random() < 0.6:                       # most layers are sized in multiples of 8
            cin, cout = (cin + 7) // 8 * 8, (cout + 7) // 8 * 8
        return dict(kind=kind, rows=rows, cin=cin, cout=cout, act=rng.choice(["none", "relu", "leaky"]), dtype=dtype)
    if kind == "attention":
        batch, heads = _log(rng, 1, 8), _log(rng, 1, 16)
        if rng.random() < 0.2:                       # any length; the framework computes those layer by layer
            seq = _log(rng, 16, 600)
        else:
            seq = 128 * _log(rng, 1, 32)
        while batch * heads * seq * seq > 16 * 2 * 4096 * 4096:
            batch = max(1, batch // 2)
            heads = heads if batch > 1 else max(1, heads // 2)
        return dict(kind=kind, batch=batch, seq=seq, heads=heads, causal=rng.random() < 0.6, dtype=dtype)
    if kind == "conv":
        chans = [8, 16, 24, 32, 48, 64, 96, 128, 256, 512]
        cin, cout, k = rng.choice(chans[1:]), rng.choice(chans[1:]), rng.choice([1, 3, 3, 3, 5])
        stride = rng.choice([1, 1, 1, 2])
        if rng.random() < 0.4:
            k, cin, cout = min(k, 3), min(cin, 256), min(cout, 256)
            d, h, w = _log(rng, 6, 64), _log(rng, 6, 64), _log(rng, 6, 64)
        else:
            d, h, w = 0, _log(rng, 7, 112), _log(rng, 7, 112)
        batch = _log(rng, 1, 64)
        taps = k ** (3 if d else 2)
        while batch > 1 and batch * max(1, d) * h * w * (cin + cout) * (1 + taps * min(cin, cout) / 512) > 3e9:
            batch //= 2
        return dict(kind=kind, batch=batch, cin=cin, cout=cout, d=d, h=h, w=w, k=k, stride=stride, dtype=dtype)
    if kind == "cosmoflow":
        width = rng.choice([32, 64, 64, 128])
        return dict(kind=kind, width=width, batch=rng.randint(1, 7 if width == 128 else 16), dtype=dtype)
    d_model = 128 * rng.choice([2, 4, 6, 8])
    return dict(kind=kind, layers=rng.randint(1, 3), d_model=d_model, heads=d_model // 128, seq=128 * rng.randint(1, 8),
                vocab=rng.choice([1000, 5003, 30522, 50304]), batch=rng.randint(1, 4), train=rng.random() < 0.7, dtype="bf16")


# ------------------------------------------------------------------------------------ the inputs
def _rng(seed, tag=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + tag)


def _randn(g, *shape, scale=1.0):
    return torch.randn(*shape, generator=g, device="cuda") * scale


_ACT = {"none": native.ACT_NONE, "relu": native.ACT_RELU, "leaky": native.ACT_LEAKY}


def _linear_tensors(c, seed):
    g, dt = _rng(seed), _DT[c["dtype"]]
    return dict(x=_randn(g, c["rows"], c["cin"]).to(dt), w=_randn(g, c["cout"], c["cin"], scale=(2.0 / c["cin"]) ** 0.5),
                b=_randn(g, c["cout"], scale=0.1), dy=_randn(g, c["rows"], c["cout"]).to(dt))


def _conv_sizes(c):
    nd = 3 if c["d"] else 2
    size = [c["d"], c["h"], c["w"]][3 - nd:]
    out = [(s + 2 * (c["k"] // 2) - c["k"]) // c["stride"] + 1 for s in size]
    return nd, size, out


def _conv_tensors(c, seed):
    g, dt = _rng(seed), _DT[c["dtype"]]
    nd, size, out = _conv_sizes(c)
    fmt = torch.channels_last_3d if nd == 3 else torch.channels_last
    x = torch.relu(_randn(g, c["batch"], c["cin"], *size)).to(dt).contiguous(memory_format=fmt)
    w = _randn(g, c["cout"], c["cin"], *[c["k"]] * nd, scale=(2.0 / (c["cin"] * c["k"] ** nd)) ** 0.5)
    dy = _randn(g, c["batch"], c["cout"], *out).to(dt).contiguous(memory_format=fmt)
    return dict(x=x, w=w, scale=1 + _randn(g, c["cout"], scale=0.1), bias=_randn(g, c["cout"], scale=0.1), dy=dy)


def _attention_tensors(c, seed):
    g, dt = _rng(seed), _DT[c["dtype"]]
    e = c["heads"] * 128
    return dict(qkv=_randn(g, c["batch"], c["seq"], 3 * e).to(dt), dy=_randn(g, c["batch"], c["seq"], e).to(dt))


def _handles(dtype, *values):
    """Weight handles whose gradients share one buffer, as they do in a parameter arena."""
    flat = torch.zeros(sum((v.numel() + 63) // 64 * 64 for v in values), device="cuda")
    made, at = [], 0
    for v in values:
        grad = flat[at:at + v.numel()].view(v.shape)
        at += (v.numel() + 63) // 64 * 64
        made.append(nn.WeightHandle(v.requires_grad_(True), grad, v.detach().to(dtype)))
    return flat, made


def _cosmoflow_channels(width):
    return (32, 64, 128, 256, 256)[:int(math.log2(width)) - 2]


def _model_inputs(c, seed):
    g = _rng(seed)
    if c["kind"] == "cosmoflow":
        w = c["width"]
        vol = torch.exp(_randn(g, c["batch"], 4, w, w, w, scale=0.5))        # log-normal densities
        target = torch.rand(c["batch"], 4, generator=g, device="cuda") * 2 - 1
        return {"samples": vol.to(_DT[c["dtype"]]), "responses": target}
    tok = torch.randint(0, c["vocab"], (c["batch"], c["seq"] + 1), generator=g, device="cuda")
    return {"samples": tok.int()}                    # whole numbers: 16-bit floats cannot hold a vocabulary


def _weight(name, shape, seed):
    """Initial values of a weight: a function of its name, its shape and the seed."""
    if name.endswith("causal_values"):
        return None
    g = _rng(seed, 1 + sum((i + 1) * ord(ch) for i, ch in enumerate(name)) % 997)
    v = _randn(g, *shape)
    if name.endswith("_kernel"):
        return v * (2.0 / math.prod(shape[1:])) ** 0.5
    if name.endswith("norm_weight") or name.endswith("norm1_weight") or name.endswith("norm2_weight"):
        return 1 + 0.1 * v
    if name.endswith("_bias"):
        return 0.05 * v
    if name.endswith("_matrix"):
        return v / shape[-1] ** 0.5
    return 0.02 * v                                                       # embeddings, LM head


def _build(c, seed):
    options.current().set("use_cuda_graph", True)       # as the training benchmark runs its steps
    if c["kind"] == "cosmoflow":
        w = c["width"]
        model = construct_cosmoflow_model(w, 4, 4, channels=_cosmoflow_channels(w), pool_mode="max", conv_bias=False,
                                          name="cosmoflow")
        if c["dtype"] == "fp16":
            model.amp = lbann.AmpOptions(enabled=True, init_scale=128.0)
        arrays = {"samples": np.zeros((1, 4, w, w, w), np.float32), "responses": np.zeros((1, 4), np.float32)}
    else:
        model = construct_gpt_model(vocab_size=c["vocab"], seq_len=c["seq"], d_model=c["d_model"], num_heads=c["heads"],
                                    num_layers=c["layers"], ffn_dim=4 * c["d_model"])
        arrays = {"samples": np.zeros((1, c["seq"] + 1), np.float32)}
    exp = lbann.proto.serialize.build_experiment(
        trainer=lbann.Trainer(mini_batch_size=c["batch"], random_seed=1), model=model,
        data_reader=lbann.reader_pb2.DataReader(), optimizer=lbann.Adam(learn_rate=_LR, beta1=0.9, beta2=0.99, eps=1e-8))
    trainer = ExecTrainer(exp, default_dtype=c["dtype"], readers={"train": ArrayReader(arrays)}, background_io=False)
    m = trainer.build_model(exp.model)
    for w in m.weights:
        v = _weight(w.name, tuple(w.values.shape), seed)
        if v is not None:
            w.set_values(v)
    return trainer, m


def prepare(case, seed):
    c = case
    if c["kind"] == "linear":
        t = _linear_tensors(c, seed)
        flat, (wh, bh) = _handles(_DT[c["dtype"]], t["w"], t["b"])
        return dict(case=c, x=t["x"].requires_grad_(True), dy=t["dy"], flat=flat, wh=wh, bh=bh)
    if c["kind"] == "conv":
        t = _conv_tensors(c, seed)
        flat, (wh, sh, bh) = _handles(_DT[c["dtype"]], t["w"], t["scale"], t["bias"])
        return dict(case=c, x=t["x"].requires_grad_(True), dy=t["dy"], flat=flat, wh=wh, sh=sh, bh=bh,
                    mean=torch.zeros(c["cout"], device="cuda"), var=torch.ones(c["cout"], device="cuda"))
    if c["kind"] == "attention":
        t = _attention_tensors(c, seed)
        return dict(case=c, x=t["qkv"].requires_grad_(True), dy=t["dy"])
    trainer, m = _build(c, seed)
    return dict(case=c, trainer=trainer, model=m, inputs=_model_inputs(c, seed))


# -------------------------------------------------------------------------------------- one pass
def run(state):
    s, c = state, state["case"]
    if c["kind"] == "linear":
        s["flat"].zero_()
        y = nn.linear(s["x"], s["wh"], s["bh"], _ACT[c["act"]], _SLOPE if c["act"] == "leaky" else 0.0)
        dx, = torch.autograd.grad(y, s["x"], s["dy"])
        return dict(y=y, dx=dx, dw=s["wh"].grad, db=s["bh"].grad)
    if c["kind"] == "attention":
        y = attention_packed(s["x"], c["heads"], 1.0 / math.sqrt(128), c["causal"])
        dx, = torch.autograd.grad(y, s["x"], s["dy"])
        return dict(y=y, dx=dx)
    if c["kind"] == "conv":
        nd = 3 if c["d"] else 2
        s["flat"].zero_()
        s["wh"].bump()                              # the optimizer has changed the weights since the last step
        pad, stride = (c["k"] // 2,) * nd, (c["stride"],) * nd
        y = nn.convolution(s["x"], s["wh"], None, (c["k"],) * nd, pad, stride, (1,) * nd)
        y = nn.batch_norm(y, s["sh"], s["bh"], s["mean"], s["var"], True, _EPS, 0.9, act=native.ACT_RELU)
        dx, = torch.autograd.grad(y, s["x"], s["dy"])
        return dict(y=y, dx=dx, dw=s["wh"].grad, dscale=s["sh"].grad, dbias=s["bh"].grad, mean=s["mean"], var=s["var"])
    m = s["model"]
    if not c.get("train", True):
        loss = m.evaluate_step(s["inputs"], "validation", c["batch"])
        return dict(loss=loss, logits=m.activation("gpt_head_instance1"))
    loss = m.train_step(s["inputs"], c["batch"])
    out = dict(loss=loss)
    for w in m.weights:
        if w.gradient is not None:
            out["grad " + w.name], out["new " + w.name] = w.gradient, w.values
    return out


# ------------------------------------------------------------------------ what a pass cannot avoid
def work(case):
    c = case
    if c["kind"] == "linear":
        r, i, o = c["rows"], c["cin"], c["cout"]
        # x and dy read, y and dx written in 16 bits; the 16-bit weight read, its fp32 gradient written
        return dict(bytes=2 * (2 * r * i + 2 * r * o) + 6 * i * o + 8 * o, flops=6 * r * i * o)
    if c["kind"] == "attention":
        b, s, e = c["batch"], c["seq"], c["heads"] * 128
        pairs = b * c["heads"] * (s * (s + 1) / 2 if c["causal"] else s * s)
        return dict(bytes=2 * b * s * e * (3 + 1 + 1 + 3), flops=14 * 128 * pairs)
    if c["kind"] == "conv":
        nd, size, out = _conv_sizes(c)
        n_in, n_out = c["batch"] * math.prod(size), c["batch"] * math.prod(out)
        weight = c["cin"] * c["cout"] * c["k"] ** nd
        return dict(bytes=2 * (2 * n_in * c["cin"] + 2 * n_out * c["cout"]) + 8 * weight, flops=6 * n_out * weight)
    if c["kind"] == "cosmoflow":
        flops, size, cin, weights = 0, c["width"] ** 3, 4, 0
        first = True
        for ch in _cosmoflow_channels(c["width"]):
            flops += (4 if first else 6) * size * 27 * cin * ch * c["batch"]
            weights += 27 * cin * ch
            first, size, cin = False, size // 8, ch
        for a, b in ((size * cin, 2048), (2048, 256), (256, 4)):
            flops += 6 * a * b * c["batch"]
            weights += a * b
        # the volumes; per weight the gradient written and value, moments, 16-bit copy read or written
        return dict(bytes=2 * 4 * c["width"] ** 3 * c["batch"] + 32 * weights, flops=flops)
    tokens, e, layers = c["batch"] * c["seq"], c["d_model"], c["layers"]
    weights = layers * 12 * e * e + c["vocab"] * e
    pairs = layers * c["batch"] * c["heads"] * c["seq"] * (c["seq"] + 1) / 2
    if c["train"]:
        return dict(bytes=32 * (weights + c["vocab"] * e), flops=6 * weights * tokens + 14 * 128 * pairs)
    return dict(bytes=2 * weights + 2 * tokens * c["vocab"], flops=2 * weights * tokens + 4 * 128 * pairs)


def tolerance(case):
    """bf16 keeps 8 bits and fp16 11: a value rounded once is 2^-9 (2^-12) off, about 0.4 of that
    in the norm (0.0017 and 0.0003 against 64 bits for a matrix product or an attention).  Behind a
    ReLU, a leaky ReLU or a max pooling a rounding that moves a value across the threshold moves a
    whole gradient value: 0.035 against 64 bits for convolution + batch norm + ReLU in bf16."""
    if case["kind"] in ("cosmoflow", "gpt", "conv"):
        return {"rel": 0.03, "max": 0.99}
    return {"rel": 0.008, "max": 0.3}


# ------------------------------------------------------------------------------- in 64 bits
def _exact_linear(c, seed):
    t = {k: v.double() for k, v in _linear_tensors(c, seed).items()}
    w, b, x = t["w"].to(_DT[c["dtype"]]).double().requires_grad_(True), t["b"].requires_grad_(True), t["x"].requires_grad_(True)
    y = F.linear(x, w, b)
    y = torch.relu(y) if c["act"] == "relu" else F.leaky_relu(y, _SLOPE) if c["act"] == "leaky" else y
    dx, dw, db = torch.autograd.grad(y, (x, w, b), t["dy"])
    return dict(y=y, dx=dx, dw=dw, db=db)


def _exact_attention(c, seed):
    t = {k: v.double() for k, v in _attention_tensors(c, seed).items()}
    s, heads = c["seq"], c["heads"]
    keep = torch.ones(s, s, dtype=torch.bool, device="cuda").tril() if c["causal"] else None
    ys, dxs = [], []
    for i in range(c["batch"]):                     # one sequence and head at a time: the scores are large in 64 bits
        y, dx = torch.empty(s, heads * 128, device="cuda", dtype=torch.double), torch.empty_like(t["qkv"][i])
        for h in range(heads):
            cols = [slice(j * heads * 128 + h * 128, j * heads * 128 + (h + 1) * 128) for j in range(3)]
            q, k, v = (t["qkv"][i][:, col].clone().requires_grad_(True) for col in cols)
            p = q @ k.t() / math.sqrt(128)
            o = torch.softmax(p if keep is None else p.masked_fill(~keep, -math.inf), -1) @ v
            at = slice(h * 128, (h + 1) * 128)
            for col, g in zip(cols, torch.autograd.grad(o, (q, k, v), t["dy"][i][:, at])):
                dx[:, col] = g
            y[:, at] = o.detach()
        ys.append(y)
        dxs.append(dx)
    return dict(y=torch.stack(ys), dx=torch.stack(dxs))


def _conv_by_taps(x, w, stride, pad):
    """A convolution as one matrix product for each filter tap (64-bit tensors, channels last inside)."""
    nd, k = x.dim() - 2, w.shape[2]
    out = [(s + 2 * pad - k) // stride + 1 for s in x.shape[2:]]
    xp = F.pad(x, (pad,) * (2 * nd)).permute(0, *range(2, nd + 2), 1)
    y = 0
    for tap in range(k ** nd):
        at = [tap // k ** (nd - 1 - i) % k for i in range(nd)]
        view = xp[(slice(None),) + tuple(slice(a, a + (o - 1) * stride + 1, stride) for a, o in zip(at, out))]
        y = y + view @ w[(slice(None), slice(None)) + tuple(at)].t()
    return y.permute(0, nd + 1, *range(1, nd + 1))


def _exact_conv(c, seed):
    nd, size, out = _conv_sizes(c)
    if c["batch"] * math.prod(size) * (c["cin"] + c["cout"]) * c["k"] ** nd > 6e9:
        return None                                 # the tap products would not fit or take too long in 64 bits
    t = {k: v.double() for k, v in _conv_tensors(c, seed).items()}
    x = t["x"].requires_grad_(True)
    w, scale, bias = (t[n].requires_grad_(True) for n in ("w", "scale", "bias"))
    u = _conv_by_taps(x, w, c["stride"], c["k"] // 2)
    dims, shape = [0] + list(range(2, nd + 2)), [1, -1] + [1] * nd
    n = u.numel() / u.shape[1]
    mean, var = u.mean(dims), (u.var(dims, unbiased=False) * n / (n - 1)).clamp(min=_EPS)
    y = torch.relu((u - mean.view(shape)) / torch.sqrt(var.view(shape) + _EPS) * scale.view(shape) + bias.view(shape))
    dx, dw, dscale, dbias = torch.autograd.grad(y, (x, w, scale, bias), t["dy"])
    return dict(y=y, dx=dx, dw=dw, dscale=dscale, dbias=dbias, mean=0.1 * mean, var=0.9 + 0.1 * var)


def _train_outputs(loss, p):
    loss.backward()
    out = dict(loss=loss.detach().float())
    for name, v in p.items():
        out["grad " + name] = v.grad
        # Adam's first step from zero moments: the bias-corrected moments are g and g^2
        out["new " + name] = (v - _LR * v.grad / (v.grad.abs() + 1e-8)).detach()
    return out


def _exact_cosmoflow(c, seed):
    if c["width"] == 128:
        return None                                 # 64-bit activations of full-size volumes: over the time limit
    t = {k: v.double() for k, v in _model_inputs(c, seed).items()}
    p, cin, size = {}, 4, c["width"]
    for i, ch in enumerate(_cosmoflow_channels(c["width"])):
        p[f"cosmoflow_conv{i + 1}_kernel"] = (ch, cin, 3, 3, 3)
        cin, size = ch, size // 2
    for i, (a, b) in enumerate(((cin * size ** 3, 2048), (2048, 256), (256, 4))):
        p[f"cosmoflow_fc{i + 1}_matrix"], p[f"cosmoflow_fc{i + 1}_bias"] = (b, a), (b,)
    p = {n: _weight(n, s, seed).double().requires_grad_(True) for n, s in p.items()}
    h = t["samples"]
    for i in range(len(_cosmoflow_channels(c["width"]))):
        h = F.max_pool3d(F.leaky_relu(_conv_by_taps(h, p[f"cosmoflow_conv{i + 1}_kernel"], 1, 1), _SLOPE), 2)
    h = h.flatten(1)
    for i in range(3):
        h = F.linear(h, p[f"cosmoflow_fc{i + 1}_matrix"], p[f"cosmoflow_fc{i + 1}_bias"])
        h = F.leaky_relu(h, _SLOPE) if i < 2 else h
    out = _train_outputs(F.mse_loss(h, t["responses"]), p)
    scale = 128.0 if c["dtype"] == "fp16" else 1.0  # the gradients a step leaves behind carry the loss scale
    return {k: v * scale if k.startswith("grad ") else v for k, v in out.items()}


def _exact_gpt(c, seed):
    s, e, heads = c["seq"], c["d_model"], c["heads"]
    shapes = {"gpt_token_embeddings": (c["vocab"], e), "gpt_positions_positions": (s, e), "gpt_lm_head": (c["vocab"], e),
              "gpt_final_norm_weight": (e,), "gpt_final_norm_bias": (e,)}
    for i in range(c["layers"]):
        n = f"gpt_block{i}_"
        for which in ("norm1", "norm2"):
            shapes[n + which + "_weight"], shapes[n + which + "_bias"] = (e,), (e,)
        for which, (o, a) in dict(attention_qkv=(3 * e, e), attention_output=(e, e), fc1=(4 * e, e), fc2=(e, 4 * e)).items():
            shapes[n + which + "_matrix"], shapes[n + which + "_bias"] = (o, a), (o,)
    p = {n: _weight(n, sh, seed).double().requires_grad_(True) for n, sh in shapes.items()}
    tok = _model_inputs(c, seed)["samples"].long()
    hidden = torch.ones(s, s, dtype=torch.bool, device="cuda").triu(1)
    x = p["gpt_token_embeddings"][tok[:, :s]] + p["gpt_positions_positions"]
    for i in range(c["layers"]):
        n = f"gpt_block{i}_"
        h = F.layer_norm(x, (e,), p[n + "norm1_weight"], p[n + "norm1_bias"], _EPS)
        qkv = F.linear(h, p[n + "attention_qkv_matrix"], p[n + "attention_qkv_bias"])
        q, k, v = (t.reshape(-1, s, heads, 128).transpose(1, 2) for t in qkv.split(e, dim=-1))
        att = torch.softmax((q @ k.transpose(-1, -2) / math.sqrt(128)).masked_fill(hidden, -math.inf), -1) @ v
        x = x + F.linear(att.transpose(1, 2).reshape(-1, s, e), p[n + "attention_output_matrix"],
                         p[n + "attention_output_bias"])
        h = F.layer_norm(x, (e,), p[n + "norm2_weight"], p[n + "norm2_bias"], _EPS)
        x = x + F.linear(F.gelu(F.linear(h, p[n + "fc1_matrix"], p[n + "fc1_bias"])), p[n + "fc2_matrix"], p[n + "fc2_bias"])
    logits = F.linear(F.layer_norm(x, (e,), p["gpt_final_norm_weight"], p["gpt_final_norm_bias"], _EPS), p["gpt_lm_head"])
    loss = F.cross_entropy(logits.reshape(-1, c["vocab"]), tok[:, 1:].reshape(-1))
    if not c["train"]:
        return dict(loss=loss.detach(), logits=logits.detach())
    return _train_outputs(loss, p)


def exact(case, seed):
    return {"linear": _exact_linear, "attention": _exact_attention, "conv": _exact_conv, "cosmoflow": _exact_cosmoflow,
            "gpt": _exact_gpt}[case["kind"]](case, seed)
