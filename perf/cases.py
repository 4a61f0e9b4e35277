"""Performance cases of the framework: training steps and forward passes through its public modules.

Families (the ``kind`` of a case) and the work they stand for:

``mlp``      networks of Linear - GELU - LayerNorm blocks with a classification head (``models.wide_mlp``): the
             headline training step, its serving form at small batches, and the same network at ordinary, odd and
             ragged sizes in each GEMM precision (fp32 is the default, bf16 autocast and tf32 are options)
``mnist``    ``models.mnist_classifier`` as the repository configures it: launch-bound training and single-sample
             inference
``embed``    ``models.EmbeddingClassifier`` over Zipf-distributed token ids, SGD with momentum and weight decay
``encoder``  ``nn.TransformerEncoderLayer``: a training step (bf16 or fp32) and inference
``attn``     ``nn.MultiHeadAttention`` without gradients over a whole prompt (prefill), causal or not
``conv``     ``models.vision.BasicBlock``: two 3 x 3 convolutions, the first one possibly strided, and a shortcut
``rnn``      ``nn.LSTM`` / ``nn.GRU`` over a ``[T, B, F]`` sequence

A training pass is a whole step: zero_grad, forward, loss, backward, optimizer update.  The optimizers start from
restored state (non-zero moments), as in a run that has been going for a while.
"""
from __future__ import annotations

import contextlib
import math

import torch

import ferrum_b200 as fb
from ferrum_b200 import data, nn, optim
from ferrum_b200.models import BasicBlock, EmbeddingClassifier, mnist_classifier, wide_mlp

MAX_OUTPUTS = 64


# ------------------------------------------------------------------------------------------------- the listed cases
def listed():
    return [
        # one digit classified as it arrives: latency and launch count are all there is
        dict(name="mnist_infer_b1", kind="mnist", mode="infer", prec="fp32", batch=1),
        # the repository's MNIST-shaped training configuration (batch 128, Adam, fp32): launch-bound training
        dict(name="mnist_train_b128", kind="mnist", mode="train", prec="fp32", batch=128),
        # a medium network trained in the default precision
        dict(name="mlp_train_fp32_1024x4", kind="mlp", mode="train", prec="fp32", din=1024, width=1024, depth=4,
             classes=1000, batch=1024),
        # tabular data: no width, batch or class count is a multiple of anything
        dict(name="mlp_train_bf16_ragged", kind="mlp", mode="train", prec="bf16", din=333, width=1001, depth=2,
             classes=37, batch=777),
        # the headline network answering a small batch of requests: every weight is read once
        dict(name="mlp_serve_bf16_b16", kind="mlp", mode="infer", prec="bf16", din=1024, width=4096, depth=8,
             classes=1000, batch=16),
        # the headline training step (bench.py)
        dict(name="mlp_train_bf16_4096x8", kind="mlp", mode="train", prec="bf16", din=1024, width=4096, depth=8,
             classes=1000, batch=8192),
        # the repository's embedding-classifier training configuration
        dict(name="embed_train_b512", kind="embed", mode="train", prec="bf16", vocab=50000, dim=1024, tokens=256,
             hidden=4096, classes=512, batch=512),
        # a transformer layer in bf16 training at the sequence length of the attention benchmarks
        dict(name="encoder_train_bf16_s1024", kind="encoder", mode="train", prec="bf16", heads=16, hd=64, ff=4096,
             batch=8, seq=1024),
        # a small transformer layer in the default precision over an odd number of tokens
        dict(name="encoder_infer_fp32_s197", kind="encoder", mode="infer", prec="fp32", heads=6, hd=64, ff=1536,
             batch=3, seq=197),
        # prefill of one long prompt, causal, head dimension 128
        dict(name="attn_prefill_bf16_s8192", kind="attn", mode="infer", prec="bf16", heads=16, hd=128, batch=1,
             seq=8192, causal=True),
        # a down-sampling residual block of an image network in bf16 training
        dict(name="conv_train_bf16_56px", kind="conv", mode="train", prec="bf16", cin=64, cout=128, stride=2,
             batch=64, size=56),
        # a recurrent layer trained over a sequence: a serial chain of small products
        dict(name="lstm_train_fp32_t64", kind="rnn", mode="train", prec="fp32", cell="lstm", feat=128, hidden=256,
             layers=1, batch=32, seq=64),
    ]


# ---------------------------------------------------------------------------------------------------- drawn cases
def _log(rng, lo, hi, step=1):
    """A whole number spread over the logarithm of [lo, hi], a multiple of ``step``."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(step, int(round(v / step)) * step)


def _size(rng, lo, hi):
    """Two of three sizes are multiples of 8 as most networks have them, the others any number."""
    return _log(rng, lo, hi, 8) if rng.random() < 0.67 else _log(rng, lo, hi) | 1


def draw(rng):
    kind = rng.choice(["mnist", "mlp", "mlp", "mlp", "embed", "encoder", "encoder", "attn", "conv", "rnn"])
    mode = rng.choice(["train", "infer"])
    while True:
        if kind == "mnist":
            c = dict(kind=kind, mode=mode, prec=rng.choice(["fp32", "bf16"]), batch=_log(rng, 1, 4096))
        elif kind == "mlp":
            c = dict(kind=kind, mode=mode, prec=rng.choice(["fp32", "bf16", "bf16", "tf32"]), din=_size(rng, 16, 2048),
                     width=_size(rng, 64, 4096), depth=rng.randint(1, 6), classes=_size(rng, 8, 1000),
                     batch=_log(rng, 1, 8192))
        elif kind == "embed":
            c = dict(kind=kind, mode=mode, prec="bf16", vocab=_log(rng, 1000, 50000), dim=_log(rng, 64, 1024, 8),
                     tokens=_log(rng, 8, 256), hidden=_log(rng, 256, 4096, 8), classes=_size(rng, 8, 512),
                     batch=_log(rng, 16, 512))
        elif kind == "encoder":
            heads, hd = rng.choice([2, 4, 6, 8, 12, 16]), rng.choice([32, 64, 64, 128])
            c = dict(kind=kind, mode=mode, prec=rng.choice(["fp32", "bf16", "bf16"]), heads=heads, hd=hd,
                     ff=4 * heads * hd, batch=_log(rng, 1, 16), seq=_log(rng, 16, 2048))
        elif kind == "attn":
            c = dict(kind=kind, mode="infer", prec="bf16", heads=rng.choice([4, 8, 16]), hd=rng.choice([64, 128]),
                     batch=_log(rng, 1, 4), seq=_log(rng, 128, 8192), causal=rng.random() < 0.67)
        elif kind == "conv":
            c = dict(kind=kind, mode=mode, prec=rng.choice(["bf16", "bf16", "fp32"]), cin=_log(rng, 16, 256, 8),
                     cout=_log(rng, 16, 256, 8), stride=rng.choice([1, 2]), batch=_log(rng, 1, 64),
                     size=_log(rng, 14, 56))
        else:
            c = dict(kind=kind, mode=mode, prec="fp32", cell=rng.choice(["lstm", "gru"]), feat=_size(rng, 16, 512),
                     hidden=_log(rng, 32, 512, 8), layers=rng.randint(1, 2), batch=_log(rng, 1, 128),
                     seq=_log(rng, 8, 128))
        w = work(c)
        if w["flops"] <= (1.5e12 if c["prec"] == "bf16" else 1.2e11):  # within the cost of the listed cases
            return c


# ------------------------------------------------------------------------------------------------ inputs and models
def _restore(opt, seed):
    """Moments of a run under way, through the checkpoint interface."""
    g = torch.Generator(device="cuda").manual_seed(seed + 7)
    st = {"optim.step": torch.tensor(100)}
    for i, p in enumerate(opt.params):
        m = torch.randn(p.shape, device="cuda", generator=g)
        if isinstance(opt, optim.Adam):
            st[f"optim.m.{i}"] = m.mul_(1e-4)
            st[f"optim.v.{i}"] = torch.rand(p.shape, device="cuda", generator=g).add_(0.5).mul_(1e-6)
        else:
            st[f"optim.velocity.{i}"] = m.mul_(1e-4)
    opt.load_state_tensors(st)
    return opt


def prepare(case, seed):
    c, kind = case, case["kind"]
    fb.manual_seed(seed)
    dev = fb.Device.Cuda(torch.cuda.current_device())
    g = torch.Generator(device="cuda").manual_seed(seed + 1)

    def randn(*shape):
        return torch.randn(*shape, device="cuda", generator=g)

    s = dict(case=dict(case), target=None)
    if kind == "mnist":
        model = mnist_classifier(device=dev)
        s["x"] = torch.rand(c["batch"], 784, device="cuda", generator=g)
        s["target"], s["loss"] = torch.randint(0, 10, (c["batch"],), device="cuda", generator=g), nn.nll_loss
        adam = 1e-3
    elif kind == "mlp":
        model = wide_mlp(c["din"], c["width"], c["depth"], c["classes"], device=dev)
        s["x"] = randn(c["batch"], c["din"])
        s["target"] = torch.randint(0, c["classes"], (c["batch"],), device="cuda", generator=g)
        s["loss"], adam = nn.cross_entropy, 3e-4
    elif kind == "embed":
        # dropout draws a new mask at each call: left out, so that two runs can be compared
        model = EmbeddingClassifier(c["vocab"], c["dim"], c["hidden"], c["classes"], p_drop=0.0, device=dev)
        ids = data.zipf_indices(c["vocab"], 1.1, c["batch"] * c["tokens"], seed=seed)
        s["x"] = torch.from_numpy(ids).reshape(c["batch"], c["tokens"]).cuda()
        s["target"] = torch.randint(0, c["classes"], (c["batch"],), device="cuda", generator=g)
        s["loss"], adam = nn.cross_entropy, None
        sgd = optim.SGDConfig(lr=0.1, momentum=0.9, weight_decay=1e-4)
    elif kind in ("encoder", "attn"):
        d = c["heads"] * c["hd"]
        model = (nn.TransformerEncoderLayer(d, c["heads"], c["ff"], device=dev) if kind == "encoder"
                 else nn.MultiHeadAttention(d, c["heads"], device=dev))
        s["x"] = randn(c["batch"], c["seq"], d)
        s["target"], s["loss"], adam = randn(c["batch"], c["seq"], d), nn.mse_loss, None
        sgd = optim.SGDConfig(lr=0.01, momentum=0.9)
    elif kind == "conv":
        model = BasicBlock(c["cin"], c["cout"], c["stride"], device=dev)
        s["x"] = randn(c["batch"], c["cin"], c["size"], c["size"])
        so = (c["size"] - 1) // c["stride"] + 1
        s["target"], s["loss"], adam = randn(c["batch"], c["cout"], so, so), nn.mse_loss, None
        sgd = optim.SGDConfig(lr=0.01, momentum=0.9)
    else:
        cls = nn.LSTM if c["cell"] == "lstm" else nn.GRU
        model = cls(c["feat"], c["hidden"], c["layers"], device=dev)
        s["x"] = randn(c["seq"], c["batch"], c["feat"])
        s["target"], s["loss"], adam = randn(c["seq"], c["batch"], c["hidden"]), nn.mse_loss, None
        sgd = optim.SGDConfig(lr=0.01, momentum=0.9)
    s["model"] = model
    if c["mode"] == "train":
        model.train()
        opt = (optim.Adam(model.parameters(), optim.AdamConfig(lr=adam)) if adam
               else optim.SGD(model.parameters(), sgd))
        s["opt"] = _restore(opt, seed)
    else:
        model.eval()
    return s


# ----------------------------------------------------------------------------------------------------------- a pass
@contextlib.contextmanager
def _precision(prec):
    if prec == "bf16":
        with fb.autocast():
            yield
    elif prec == "tf32":
        before = fb.matmul_precision()
        fb.matmul_precision("tf32")
        try:
            yield
        finally:
            fb.matmul_precision(before)
    else:
        yield


def _forward(s):
    model, c = s["model"], s["case"]
    if c["kind"] == "attn":
        return model.forward_attn(s["x"], s["x"], s["x"], causal=c["causal"])
    if c["kind"] == "rnn":
        return model.forward_seq(s["x"])
    return model(s["x"])


def run(state):
    s = state
    prec = s["case"]["prec"]
    if s["case"]["mode"] == "infer":
        with torch.no_grad(), _precision(prec):
            return _forward(s)
    opt = s["opt"]
    opt.zero_grad()
    with _precision(prec):
        y = _forward(s)
        y = y[0] if s["case"]["kind"] == "rnn" else y
        loss = s["loss"](y, s["target"])
        if prec == "tf32":  # a setting of the process, read in the backward pass too
            loss.backward()
    if prec != "tf32":
        loss.backward()
    opt.step()
    return _outputs(s, y, loss)


def _outputs(s, y, loss):
    """The loss, the forward result, every parameter, its gradient and the optimizer's moments; where that would be
    too many tensors, gradients and moments of the matrices alone."""
    opt = s["opt"]
    ps = opt.params
    state = [opt.m, opt.v] if isinstance(opt, optim.Adam) else [opt.velocity]
    keep = [i for i, p in enumerate(ps) if p.dim() > 1] if 2 + (2 + len(state)) * len(ps) > MAX_OUTPUTS else range(len(ps))
    out = dict(loss=loss, y=y, params=list(ps), grads=[ps[i].grad for i in keep])
    for k, st in enumerate(state):
        out[f"moment{k}"] = [st[i] for i in keep]
    return out


# ------------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    """Multiply-adds of the products, counted as two operations each (three products per layer in training, the one
    for the input's gradient left out where nobody asks for it), and the bytes of inputs, outputs and weights: in
    training every parameter and moment is read and written once and every gradient written once."""
    c, kind = case, case["kind"]
    B, train = c["batch"], c["mode"] == "train"
    act = 2 if c["prec"] == "bf16" else 4
    first = other = 0.0     # forward operations of the layers on the input (no input gradient) and of the rest
    nmom = 1
    if kind == "mnist":
        first, other = 2.0 * B * 784 * 256, 2.0 * B * 256 * 10
        params, io, nmom = 784 * 256 + 256 * 13 + 10 + 2560, B * (784 + 10) * 4, 2
    elif kind == "mlp":
        W, D = c["width"], c["depth"]
        first = 2.0 * B * c["din"] * W
        other = 2.0 * B * ((D - 1) * W * W + W * c["classes"])
        params = c["din"] * W + (D - 1) * W * W + 3 * D * W + (W + 1) * c["classes"]
        io, nmom = B * (c["din"] * 4 + c["classes"] * act), 2
    elif kind == "embed":
        other = 2.0 * B * (c["dim"] * c["hidden"] + c["hidden"] * c["classes"])
        head = c["dim"] * c["hidden"] + c["hidden"] + (c["hidden"] + 1) * c["classes"]
        rows = min(c["vocab"], B * c["tokens"])
        params = head + (c["vocab"] if train else rows) * c["dim"]
        io = B * c["tokens"] * 8 + B * c["classes"] * act
    elif kind in ("encoder", "attn"):
        d, S = c["heads"] * c["hd"], c["seq"]
        core = 4.0 * B * S * S * d * (0.5 if c.get("causal") else 1.0)
        other = 8.0 * B * S * d * d + core + (4.0 * B * S * d * c["ff"] if kind == "encoder" else 0.0)
        params = 4 * d * (d + 1) + (2 * d * c["ff"] + c["ff"] + 5 * d if kind == "encoder" else 0)
        io = B * S * d * (4 + (4 if kind == "encoder" else act))
    elif kind == "conv":
        so = (c["size"] - 1) // c["stride"] + 1
        short = c["cin"] if c["stride"] != 1 or c["cin"] != c["cout"] else 0
        first = 2.0 * B * so * so * c["cout"] * (c["cin"] * 9 + short)
        other = 2.0 * B * so * so * c["cout"] * c["cout"] * 9
        params = c["cout"] * (9 * c["cin"] + 9 * c["cout"] + short)
        io = B * (c["cin"] * c["size"] ** 2 + c["cout"] * so * so) * 4
    else:
        G, H, T = 4 if c["cell"] == "lstm" else 3, c["hidden"], c["seq"]
        first = 2.0 * T * B * G * H * c["feat"]
        other = 2.0 * T * B * G * H * H * (2 * c["layers"] - 1)
        params = G * H * (c["feat"] + H + 2) + (c["layers"] - 1) * G * H * (2 * H + 2)
        io = T * B * (c["feat"] + H) * 4
    if train:
        return {"bytes": io + params * 4.0 * (2 + 2 * nmom + 1), "flops": 2 * first + 3 * other}
    return {"bytes": io + params * float(act if kind != "embed" else 4), "flops": first + other}


def tolerance(case):
    """What the order of the sums and the rounding points of the types give.  With ReLU in a training step a
    pre-activation next to zero may fall on either side: its whole gradient goes or stays, so the share p of such
    units shows as sqrt(p) in the gradients, and single values can be off by much."""
    relu = case["mode"] == "train" and case["kind"] in ("mnist", "encoder", "conv")
    if case["prec"] == "bf16":
        return {"rel": 0.02 if relu else 0.01, "max": 0.9 if relu else 0.4}
    if case["prec"] == "tf32":
        return {"rel": 0.002, "max": 0.08}
    return {"rel": 1e-3, "max": 0.9} if relu else {"rel": 2e-5, "max": 1e-3}
