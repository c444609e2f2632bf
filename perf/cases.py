"""Performance cases: the layers, blocks and steps that training programs run through this framework's entry points.

Sizes are those of the benchmark models (ResNet-50 at batch 8 to 256, a BERT-large-shaped encoder, a CTR model in
parameter-server mode), of the tests, and generic ragged ones around them.  ``listed`` names the fixed cases, ``draw``
gives another one from the same ranges, and the kinds share their code:

    conv_bn      convolution + batch norm + ReLU, training, forward and backward
    block        ResNet bottleneck block, training, forward and backward (with a projection when it changes shape)
    block_eval   the same block at inference, captured as a CUDA graph: a handful of small launches
    stem         fp32 images -> 7x7 convolution + batch norm + ReLU + max pool, forward and weight gradient
    linear       dense layer with bias and activation, forward and backward
    encoder      one transformer encoder layer, forward and backward
    layer_norm   LayerNorm(x + residual), forward and backward
    mlm_head     vocabulary projection and softmax cross-entropy, forward and backward
    ctr_step     one training step of the click model in parameter-server mode, captured as a CUDA graph
    adamw        optimizer step over a list of bf16 parameters with fp32 master weights
    ps           parameter-server step: pull the rows of a batch, push their gradients (server-side Adagrad)
"""
import math

import torch
import torch.nn.functional as F

from tips_b200.models.bert import BertLayer
from tips_b200.models.ctr import CtrTrainer
from tips_b200.models.resnet50 import Bottleneck
from tips_b200.ops.conv import Conv2d, conv2d
from tips_b200.ops.linear import Linear, linear
from tips_b200.ops.norm import BatchNorm2d, LayerNorm
from tips_b200.ops.optim import FusedAdamW
from tips_b200.ops.pointwise import softmax_cross_entropy
from tips_b200.ops.pool import MaxPool3x3S2
from tips_b200.ps.gpu import ShardedEmbedding
from tips_b200.utils.misc import make_subgraph

DEV = "cuda"
BF16 = torch.bfloat16
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # ResNet-50 stage 1, its most frequent shape at the benchmark's batch: few channels, many pixels
        {"name": "conv3x3_56_c64", "kind": "conv_bn", "batch": 256, "size": 56, "cin": 64, "cout": 64, "k": 3, "stride": 1},
        # stage 2 entry: the block that halves the resolution (3x3 stride 2, 1x1 stride 2 projection)
        {"name": "block_56_s2", "kind": "block", "batch": 64, "size": 56, "cin": 256, "width": 128, "stride": 2},
        # stage 3, the stage with the most blocks
        {"name": "block_14", "kind": "block", "batch": 128, "size": 14, "cin": 1024, "width": 256, "stride": 1},
        # a classifier's request of one image: latency of a short chain of launches
        {"name": "block_eval_7_b1", "kind": "block_eval", "batch": 1, "size": 7, "cin": 2048, "width": 512, "stride": 1},
        # input of a training step as a loader delivers it
        {"name": "stem_224", "kind": "stem", "batch": 64, "size": 224, "cout": 64},
        # feed-forward layer of the encoder at 32 sequences of 512 tokens
        {"name": "ffn_16384", "kind": "linear", "rows": 16384, "k": 1024, "n": 4096, "act": "gelu", "bias": True},
        # a ResNet classifier head: ragged output count, few rows
        {"name": "classifier_256", "kind": "linear", "rows": 256, "k": 2048, "n": 1000, "act": "none", "bias": True},
        # one encoder layer at 8 sequences of 512 tokens
        {"name": "encoder_8x512", "kind": "encoder", "batch": 8, "seq": 512, "hidden": 1024, "heads": 16, "ffn": 4096},
        # masked-language-model head: 77 masked positions of each of 16 sequences
        {"name": "mlm_head_1232", "kind": "mlm_head", "rows": 1232, "hidden": 1024, "vocab": 30528},
        # the click model's whole step at the benchmark's batch: 26 fields of 64 plus 13 dense features
        {"name": "ctr_step_8192", "kind": "ctr_step", "batch": 8192, "fields": 26, "rows": 50000, "dim": 64, "h1": 512, "h2": 256},
        # optimizer step over two encoder layers (25 M parameters)
        {"name": "adamw_25M", "kind": "adamw", "hidden": 1024, "ffn": 4096, "layers": 2, "vocab": 0},
        # parameter-server step of the click model at the benchmark's batch, ids Zipf(1.05)
        {"name": "ps_8192x26", "kind": "ps", "batch": 8192, "fields": 26, "rows": 50000, "dim": 64},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["conv_bn", "conv_bn", "block", "block_eval", "stem", "linear", "linear", "encoder",
                       "layer_norm", "layer_norm", "mlm_head", "ctr_step", "adamw", "ps"])
    if kind == "conv_bn":
        size, chans = rng.choice([(56, (64, 128, 256)), (28, (64, 128, 256, 512)), (14, (256, 512, 1024)),
                                  (7, (512, 1024, 2048)), (rng.randrange(9, 45), (64, 128, 192, 320))])
        cin, cout = rng.choice(chans), rng.choice(chans)
        k = rng.choice([1, 3])
        if k == 3:
            cin, cout = min(cin, 512), min(cout, 512)
        stride = rng.choice([1, 1, 2])
        work = size * size * max(cin * k * k * cout / 150, cin, cout)
        most = max(4, min(256, int(256 * 56 * 56 * 245 / work)))
        return {"kind": kind, "batch": round(_log(rng, 4, most)), "size": size, "cin": cin, "cout": cout, "k": k, "stride": stride}
    if kind in ("block", "block_eval"):
        size, width, cin, stride = rng.choice([(56, 64, 64, 1), (56, 64, 256, 1), (56, 128, 256, 2), (28, 128, 512, 1),
                                               (28, 256, 512, 2), (14, 256, 1024, 1), (14, 512, 1024, 2),
                                               (7, 512, 2048, 1)])
        if kind == "block":
            batch = round(_log(rng, 8, 64 if size > 28 else 128))
        else:
            batch = round(_log(rng, 1, 16))
        return {"kind": kind, "batch": batch, "size": size, "cin": cin, "width": width, "stride": stride}
    if kind == "stem":
        return {"kind": kind, "batch": round(_log(rng, 4, 64)), "size": rng.choice([128, 160, 192, 224, rng.randrange(64, 224)]), "cout": 64}
    if kind == "linear":
        k, n = rng.choice([(1024, 4096), (4096, 1024), (1024, 3072), (1024, 1024), (2048, 1000), (512, 256), (1728, 512),
                           (8 * rng.randrange(8, 200), 8 * rng.randrange(8, 200))])
        return {"kind": kind, "rows": round(_log(rng, 64, 16384)), "k": k, "n": n,
                "act": rng.choice(["none", "relu", "gelu"]), "bias": rng.random() < 0.8}
    if kind == "encoder":
        hidden, heads = rng.choice([(1024, 16), (768, 12), (512, 8)])
        return {"kind": kind, "batch": rng.randrange(1, 9), "seq": rng.choice([64, 128, 256, 384, 512]), "hidden": hidden,
                "heads": heads, "ffn": 4 * hidden}
    if kind == "layer_norm":
        dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
        cols = rng.choice([256, 768, 1024, 1024 if dtype == "fp32" else 2048, 8 * rng.randrange(8, 128 if dtype == "fp32" else 192)])
        return {"kind": kind, "rows": round(_log(rng, 64, 65536)), "cols": cols, "dtype": dtype}
    if kind == "mlm_head":
        hidden = rng.choice([512, 768, 1024])
        return {"kind": kind, "rows": round(_log(rng, 32, 1232)), "hidden": hidden, "vocab": rng.choice([30528, 64 * rng.randrange(16, 470)])}
    if kind == "ctr_step":
        fields, dim = rng.choice([(26, 64), (8, 32), (16, 16), (26, 32)])
        h1 = rng.choice([128, 256, 512])
        return {"kind": kind, "batch": round(_log(rng, 256, 8192)), "fields": fields, "rows": round(_log(rng, 1000, 50000)),
                "dim": dim, "h1": h1, "h2": h1 // 2}
    if kind == "adamw":
        hidden = rng.choice([128, 512, 768, 1024])
        return {"kind": kind, "hidden": hidden, "ffn": 4 * hidden, "layers": rng.choice([1, 2]), "vocab": rng.choice([0, rng.randrange(1000, 4000)])}
    return {"kind": "ps", "batch": round(_log(rng, 256, 8192)), "fields": rng.choice([4, 13, 26]), "rows": round(_log(rng, 1000, 50000)),
            "dim": rng.choice([16, 32, 64])}


# ---------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed * 7919 + 11)


def _normal(g, *shape, dtype=BF16, scale=1.0, nhwc=False):
    t = (torch.randn(*shape, generator=g, device=DEV) * scale).to(dtype)
    return t.contiguous(memory_format=torch.channels_last) if nhwc else t


def _grad(g, *shape):
    """Upstream gradient behind a ReLU: uniform, so that one value that crosses the ReLU's threshold stays bounded."""
    t = ((torch.rand(*shape, generator=g, device=DEV) - 0.5) * 0.02).to(BF16)
    return t.contiguous(memory_format=torch.channels_last)


def _out_size(size, k, stride):
    return (size + 2 * (k // 2) - k) // stride + 1


def _init_bn(bn, g):
    with torch.no_grad():
        bn.weight.copy_(1.0 + 0.1 * torch.randn(bn.num_features, generator=g, device=DEV))
        bn.bias.copy_(0.1 * torch.randn(bn.num_features, generator=g, device=DEV))
        bn.running_mean.copy_(0.1 * torch.randn(bn.num_features, generator=g, device=DEV))
        bn.running_var.copy_(0.5 + torch.rand(bn.num_features, generator=g, device=DEV))


def _init_conv(conv, g, gain=2.0):
    with torch.no_grad():
        fan_in = conv.weight[0].numel()
        conv.weight.copy_(torch.randn(conv.weight.shape, generator=g, device=DEV) * math.sqrt(gain / fan_in))


def _block(case, g):
    cin, width, stride = case["cin"], case["width"], case["stride"]
    m = Bottleneck(cin, width, stride, downsample=(stride != 1 or cin != 4 * width)).to(device=DEV, dtype=BF16)
    for mod in m.modules():
        if isinstance(mod, Conv2d):
            _init_conv(mod, g)
        elif isinstance(mod, BatchNorm2d):
            _init_bn(mod, g)
    return m


def _linear_init(lin, g, std=None):
    with torch.no_grad():
        std = 1.0 / math.sqrt(lin.in_features) if std is None else std
        lin.weight.copy_(torch.randn(lin.weight.shape, generator=g, device=DEV) * std)
        if lin.bias is not None:
            lin.bias.copy_(torch.randn(lin.bias.shape, generator=g, device=DEV) * 0.1)


def _zipf_ids(g, batch, fields, rows, alpha=1.05):
    u = torch.rand(batch, fields, generator=g, device=DEV, dtype=torch.float64)
    e = 1.0 - alpha
    x = ((float(rows) ** e - 1.0) * u + 1.0) ** (1.0 / e)
    return (x.floor().to(torch.int64) - 1).clamp_(0, rows - 1)


def _adamw_shapes(case):
    h, f = case["hidden"], case["ffn"]
    layer = [(3 * h, h), (3 * h,), (h, h), (h,), (h,), (h,), (f, h), (f,), (h, f), (h,), (h,), (h,)]
    return layer * case["layers"] + ([(case["vocab"], h), (case["vocab"],)] if case["vocab"] else [])


def _inputs(case, seed):
    """Everything random of a case, as tensors and modules that both the framework's pass and the exact one use."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "conv_bn":
        conv = Conv2d(case["cin"], case["cout"], case["k"], case["stride"], case["k"] // 2).to(device=DEV, dtype=BF16)
        bn = BatchNorm2d(case["cout"], relu=True).to(DEV)
        _init_conv(conv, g)
        _init_bn(bn, g)
        x = _normal(g, case["batch"], case["cin"], case["size"], case["size"], nhwc=True).relu_()
        o = _out_size(case["size"], case["k"], case["stride"])
        dy = _grad(g, case["batch"], case["cout"], o, o)
        return {"conv": conv, "bn": bn, "x": x.requires_grad_(), "dy": dy}
    if kind in ("block", "block_eval"):
        m = _block(case, g)
        x = _normal(g, case["batch"], case["cin"], case["size"], case["size"], nhwc=True).relu_()
        if kind == "block_eval":
            return {"m": m.eval(), "x": x}
        o = _out_size(case["size"], 3, case["stride"])
        dy = _grad(g, case["batch"], 4 * case["width"], o, o)
        return {"m": m.train(), "x": x.requires_grad_(), "dy": dy}
    if kind == "stem":
        conv = Conv2d(3, case["cout"], 7, 2, 3).to(device=DEV, dtype=BF16)
        bn = BatchNorm2d(case["cout"], relu=True).to(DEV)
        _init_conv(conv, g)
        _init_bn(bn, g)
        images = _normal(g, case["batch"], 3, case["size"], case["size"], dtype=torch.float32)
        o = (_out_size(case["size"], 7, 2) - 1) // 2 + 1
        dy = _grad(g, case["batch"], case["cout"], o, o)
        return {"conv": conv, "bn": bn, "pool": MaxPool3x3S2(), "x": images, "dy": dy}
    if kind == "linear":
        lin = Linear(case["k"], case["n"], bias=case["bias"], act=case["act"]).to(device=DEV, dtype=BF16)
        _linear_init(lin, g)
        x = _normal(g, case["rows"], case["k"])
        return {"lin": lin, "x": x.requires_grad_(), "dy": _normal(g, case["rows"], case["n"], scale=0.01)}
    if kind == "encoder":
        m = BertLayer(case["hidden"], case["heads"], case["ffn"]).to(device=DEV, dtype=BF16)
        for mod in m.modules():
            if isinstance(mod, Linear):
                _linear_init(mod, g)
        x = _normal(g, case["batch"], case["seq"], case["hidden"])
        return {"m": m, "x": x.requires_grad_(), "dy": _normal(g, *x.shape, scale=0.01)}
    if kind == "layer_norm":
        dt = DTYPES[case["dtype"]]
        ln = LayerNorm(case["cols"], eps=1e-12).to(device=DEV, dtype=dt)
        with torch.no_grad():
            ln.weight.copy_(1.0 + 0.1 * torch.randn(case["cols"], generator=g, device=DEV))
            ln.bias.copy_(0.1 * torch.randn(case["cols"], generator=g, device=DEV))
        shape = (case["rows"], case["cols"])
        x, r = _normal(g, *shape, dtype=dt), _normal(g, *shape, dtype=dt)
        return {"ln": ln, "x": x.requires_grad_(), "r": r.requires_grad_(), "dy": _normal(g, *shape, dtype=dt, scale=0.01)}
    if kind == "mlm_head":
        h = _normal(g, case["rows"], case["hidden"])
        w = _normal(g, case["vocab"], case["hidden"], scale=0.02)
        b = _normal(g, case["vocab"], scale=0.02)
        labels = torch.randint(0, case["vocab"], (case["rows"],), generator=g, device=DEV)
        labels[::16] = -100  # unused slots
        return {"h": h.requires_grad_(), "w": w.requires_grad_(), "b": b.requires_grad_(), "labels": labels}
    if kind == "ctr_step":
        ids = _zipf_ids(g, case["batch"], case["fields"], case["rows"])
        dense = _normal(g, case["batch"], CTR_DENSE)
        labels = (torch.rand(case["batch"], generator=g, device=DEV) < 0.25).to(torch.float32)
        dims = [(case["fields"] * case["dim"] + CTR_DENSE + 63) // 64 * 64, case["h1"], case["h2"], 1]
        params = []
        for i in range(3):
            params.append(_normal(g, dims[i + 1], dims[i], scale=1.0 / math.sqrt(dims[i])))
            params.append(_normal(g, dims[i + 1], scale=0.1))
        return {"ids": ids, "dense": dense, "labels": labels, "params": params}
    if kind == "adamw":
        shapes = _adamw_shapes(case)
        params = [torch.nn.Parameter(_normal(g, *s, scale=0.02)) for s in shapes]
        grads = [_normal(g, *s, scale=1e-3) for s in shapes]
        return {"params": params, "grads": grads}
    ids = _zipf_ids(g, case["batch"], case["fields"], case["rows"])
    grads = _normal(g, case["batch"], case["fields"] * case["dim"], scale=1e-2)
    return {"ids": ids, "grads": grads}


ADAMW = {"lr": 1e-3, "betas": (0.9, 0.999), "eps": 1e-8, "weight_decay": 0.01}
PS_LR, PS_EPS = 0.05, 1e-8
CTR_DENSE, CTR_LR, CTR_WARM = 13, 1e-3, 4  # dense features, Adam's rate, steps until the trainer replays its graph


def _ps_tables(case, seed):
    """Rows and Adagrad accumulators of a table in mid-training."""
    g = _gen(seed + 1)
    shape = (case["rows"], case["dim"])
    for _ in range(case["fields"]):
        yield 0.05 * torch.randn(shape, generator=g, device=DEV), 0.01 + 0.1 * torch.rand(shape, generator=g, device=DEV)


def _fill_tables(t, case, seed):
    for f, (rows, acc) in enumerate(_ps_tables(case, seed)):  # with one server, row id is local row id
        t.local_shard(f).copy_(rows)
        t.local_shard(f, state=True).copy_(acc)


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = s["kind"] = case["kind"]
    if kind == "block_eval":
        with torch.no_grad():
            s["graph"] = make_subgraph(s["m"], s["x"])
    elif kind == "adamw":
        s["opt"] = FusedAdamW(s["params"], **ADAMW)
        s["opt"].build()
    elif kind == "ps":
        s["table"] = ShardedEmbedding(case["fields"], case["rows"], case["dim"], optimizer="adagrad", lr=PS_LR, eps=PS_EPS,
                                      expected_batch=case["batch"], device=torch.device(DEV, torch.cuda.current_device()))
        _fill_tables(s["table"], case, seed)
        s["x"] = torch.empty(case["batch"], case["fields"] * case["dim"], dtype=BF16, device=DEV)
    elif kind == "ctr_step":
        tr = CtrTrainer(case["fields"], case["rows"], case["dim"], CTR_DENSE, (case["h1"], case["h2"]), table_lr=PS_LR,
                        mlp_lr=CTR_LR, expected_batch=case["batch"], graph=True,
                        device=torch.device(DEV, torch.cuda.current_device()))
        _fill_tables(tr.tables, case, seed)
        with torch.no_grad():
            for p, v in zip(tr.mlp.parameters(), s["params"]):
                p.copy_(v.view(p.shape))
        tr.opt.refresh_master_from_params()
        for _ in range(CTR_WARM):
            tr.train_step(s["ids"], s["dense"], s["labels"])
        s["trainer"] = tr
    return s


# ---------------------------------------------------------------- one pass

def _clear(params):
    for p in params:
        p.grad = None


def run(state):
    kind = state["kind"]
    if kind == "conv_bn":
        conv, bn, x = state["conv"], state["bn"], state["x"]
        _clear([x, conv.weight, bn.weight, bn.bias])
        stats = torch.zeros(2, conv.out_channels, dtype=torch.float32, device=x.device)
        y = bn(conv2d(x, conv.weight, conv.stride, conv.padding, stats), stats=stats)
        y.backward(state["dy"])
        return [y.detach(), x.grad, conv.weight.grad, bn.weight.grad, bn.bias.grad, bn.running_mean, bn.running_var]
    if kind == "block":
        m, x = state["m"], state["x"]
        _clear([x, *m.parameters()])
        y = m(x)
        y.backward(state["dy"])
        return [y.detach(), x.grad, *[p.grad for p in m.parameters()], *m.buffers()]
    if kind == "block_eval":
        return state["graph"](state["x"])
    if kind == "stem":
        conv, bn = state["conv"], state["bn"]
        _clear([conv.weight, bn.weight, bn.bias])
        stats = torch.zeros(2, conv.out_channels, dtype=torch.float32, device=state["x"].device)
        y = state["pool"](bn(conv(state["x"], stats=stats), stats=stats))
        y.backward(state["dy"])
        return [y.detach(), conv.weight.grad, bn.weight.grad, bn.bias.grad, bn.running_mean, bn.running_var]
    if kind == "linear":
        lin, x = state["lin"], state["x"]
        _clear([x, *lin.parameters()])
        y = lin(x)
        y.backward(state["dy"])
        return [y.detach(), x.grad, *[p.grad for p in lin.parameters()]]
    if kind == "encoder":
        m, x = state["m"], state["x"]
        _clear([x, *m.parameters()])
        y = m(x)
        y.backward(state["dy"])
        return [y.detach(), x.grad, *[p.grad for p in m.parameters()]]
    if kind == "layer_norm":
        ln, x, r = state["ln"], state["x"], state["r"]
        _clear([x, r, *ln.parameters()])
        y = ln(x, residual=r)
        y.backward(state["dy"])
        return [y.detach(), x.grad, r.grad, ln.weight.grad, ln.bias.grad]
    if kind == "mlm_head":
        h, w, b = state["h"], state["w"], state["b"]
        _clear([h, w, b])
        logits = linear(h, w, b)
        loss = softmax_cross_entropy(logits, state["labels"])
        loss.backward()
        return [loss.detach(), logits.detach(), h.grad, w.grad, b.grad]
    if kind == "ctr_step":
        tr = state["trainer"]
        loss = tr.train_step(state["ids"], state["dense"], state["labels"])
        return [loss, *[p.detach() for p in tr.mlp.parameters()], *[tr.tables.local_shard(f) for f in range(tr.fields)]]
    if kind == "adamw":
        opt = state["opt"]
        for p, g in zip(state["params"], state["grads"]):
            p.grad = g
        opt.step()
        return [*[p.detach() for p in state["params"]], *[t for fs in opt.build() for t in (fs.master, fs.state["exp_avg"], fs.state["exp_avg_sq"])]]
    t = state["table"]
    t.pull(state["ids"], out=state["x"])
    t.push(state["ids"], state["grads"])
    rows = [t.local_shard(f) for f in range(t.num_fields)]
    acc = [t.local_shard(f, state=True) for f in range(t.num_fields)]
    return [state["x"], *rows, *acc]


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind == "conv_bn":
        o = _out_size(case["size"], case["k"], case["stride"])
        x = case["batch"] * case["size"] ** 2 * case["cin"]
        y = case["batch"] * o * o * case["cout"]
        w = case["cin"] * case["cout"] * case["k"] ** 2
        return {"bytes": 2 * (2 * x + 2 * y + 2 * w), "flops": 3 * 2 * case["batch"] * o * o * w}
    if kind in ("block", "block_eval"):
        n, s, cin, width, stride = (case[k] for k in ("batch", "size", "cin", "width", "stride"))
        o = _out_size(s, 3, stride)
        w1, w2, w3 = cin * width, 9 * width * width, 4 * width * width
        macs = n * (s * s * w1 + o * o * (w2 + w3))
        weights = w1 + w2 + w3
        if stride != 1 or cin != 4 * width:
            macs += n * o * o * cin * 4 * width
            weights += cin * 4 * width
        x, y = n * s * s * cin, n * o * o * 4 * width
        if kind == "block_eval":
            return {"bytes": 2 * (x + y + weights), "flops": 2 * macs}
        return {"bytes": 2 * (2 * x + 2 * y + 2 * weights), "flops": 6 * macs}
    if kind == "stem":
        c = _out_size(case["size"], 7, 2)
        p = (c - 1) // 2 + 1
        return {"bytes": case["batch"] * (case["size"] ** 2 * 3 * 4 + 2 * p * p * case["cout"] * 2),
                "flops": 2 * 2 * case["batch"] * c * c * case["cout"] * 147}
    if kind == "linear":
        m, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": 2 * (2 * m * k + 2 * m * n + 2 * k * n), "flops": 3 * 2 * m * k * n}
    if kind == "encoder":
        t, h, f = case["batch"] * case["seq"], case["hidden"], case["ffn"]
        w = 4 * h * h + 2 * h * f
        att = 2 * case["batch"] * case["seq"] ** 2 * h  # multiply-adds of the two products
        return {"bytes": 2 * (4 * t * h + 2 * w), "flops": 3 * 2 * t * w + 2 * att * 3.5}
    if kind == "layer_norm":
        e = 4 if case["dtype"] == "fp32" else 2
        # x, residual and dy read, y and the two equal input gradients (one tensor) written
        return {"bytes": e * 5 * case["rows"] * case["cols"], "flops": 16 * case["rows"] * case["cols"]}
    if kind == "mlm_head":
        r, h, v = case["rows"], case["hidden"], case["vocab"]
        return {"bytes": 2 * (2 * r * h + 2 * v * h + r * v), "flops": 3 * 2 * r * h * v}
    if kind == "adamw":
        n = sum(math.prod(s) for s in _adamw_shapes(case))
        return {"bytes": n * (2 + 2 + 3 * 8), "flops": 16 * n}
    items = case["batch"] * case["fields"]
    distinct = min(items, case["rows"] * case["fields"]) // 2
    # ids, pulled rows and gradients once, every distinct row and its accumulator read and written
    if kind == "ctr_step":  # the gradients of the rows stay inside; master weights, state and parameters of the MLP
        n = case["fields"] * case["dim"] * case["h1"] + case["h1"] * case["h2"]
        return {"bytes": items * 8 + distinct * case["dim"] * 4 * 4 + 26 * n, "flops": 3 * 2 * case["batch"] * n}
    return {"bytes": items * 8 + 2 * items * case["dim"] * 2 + distinct * case["dim"] * 4 * 4, "flops": 8 * items * case["dim"]}


def tolerance(case):
    """Between implementations of the same precision.  Measured against ``exact``: 0.0017 for one bf16 rounding (dense
    layers, pulled rows), 0.004 to 0.006 through an encoder layer; 0.03 (a batch norm) to 0.09 (a block) where a rounding
    moves values across the threshold of a ReLU or changes the winner of a pooling window, so that those are bounded by
    the most that can be asked for."""
    kind = case["kind"]
    if kind in ("conv_bn", "block", "stem"):
        return {"rel": 0.03, "max": 0.99}
    if kind == "block_eval":
        return {"rel": 0.012, "max": 0.2}
    if kind == "encoder":
        return {"rel": 0.024, "max": 0.4}
    if kind in ("linear", "mlm_head"):
        # a ReLU's mask is that of the value before its rounding, or of the bf16 output
        return {"rel": 0.01, "max": 0.5 if case.get("act") == "relu" else 0.05}
    if kind == "layer_norm":
        return {"rel": 1e-5, "max": 1e-3} if case["dtype"] == "fp32" else {"rel": 0.01, "max": 0.05}
    if kind == "ctr_step":
        return {"rel": 0.01, "max": 0.5}
    return {"rel": 0.007, "max": 0.05}


# ---------------------------------------------------------------- the same in 64 bits

def _d(t):
    return t.detach().double()


def _leaf(t):
    return _d(t).clone().requires_grad_()


class _Params:
    """64-bit copies of a module's parameters, in the order of parameters()."""

    def __init__(self, module):
        self.map = {n: _leaf(p) for n, p in module.named_parameters()}
        self.running = {n: _d(b).clone() for n, b in module.named_buffers()}

    def grads(self):
        return [p.grad for p in self.map.values()]


def _conv64(x, w, stride, pad):
    return F.conv2d(x, w.permute(0, 3, 1, 2), stride=stride, padding=pad)


def _bn64(x, p, name, training, relu, residual=None, eps=1e-5):
    dot = name + "." if name else ""
    y = F.batch_norm(x, p.running[dot + "running_mean"], p.running[dot + "running_var"], p.map[dot + "weight"],
                     p.map[dot + "bias"], training, 0.1, eps)
    if residual is not None:
        y = y + residual
    return F.relu(y) if relu else y


def _block64(m, p, x, training):
    out = _bn64(_conv64(x, p.map["conv1.weight"], 1, 0), p, "bn1", training, True)
    stride = m.conv2.stride
    identity = x if m.down is None else _bn64(_conv64(x, p.map["down.conv.weight"], stride, 0), p, "down.bn", training, False)
    out = _bn64(_conv64(out, p.map["conv2.weight"], stride, 1), p, "bn2", training, True)
    return _bn64(_conv64(out, p.map["conv3.weight"], 1, 0), p, "bn3", training, True, residual=identity)


def _encoder64(p, x, heads):
    lin = lambda t, n: F.linear(t, p.map[n + ".weight"], p.map[n + ".bias"])
    norm = lambda t, n: F.layer_norm(t, (t.shape[-1],), p.map[n + ".weight"], p.map[n + ".bias"], 1e-12)
    b, s, h = x.shape
    q, k, v = lin(x, "qkv").view(b, s, 3, heads, h // heads).permute(2, 0, 3, 1, 4)
    att = torch.softmax(q @ k.transpose(-1, -2) / math.sqrt(h // heads), dim=-1) @ v
    x = norm(lin(att.transpose(1, 2).reshape(b, s, h), "proj") + x, "ln1")
    return norm(lin(F.gelu(lin(x, "fc1")), "fc2") + x, "ln2")


def _ctr64(case, seed, s):
    """The warm-up steps and one more: pull, MLP, mean cross-entropy, Adam, Adagrad on the rows."""
    tables = [[_d(w), _d(a)] for w, a in _ps_tables(case, seed)]
    params = [_d(p) for p in s["params"]]
    m, v = [torch.zeros_like(p) for p in params], [torch.zeros_like(p) for p in params]
    ids, dim = s["ids"], case["dim"]
    pad = params[0].shape[1] - case["fields"] * dim - CTR_DENSE
    for step in range(1, CTR_WARM + 2):
        emb = torch.cat([t[0][ids[:, f]] for f, t in enumerate(tables)], dim=1).requires_grad_()
        leaves = [p.clone().requires_grad_() for p in params]
        y = F.pad(torch.cat([emb, _d(s["dense"])], dim=1), (0, pad))
        y = F.relu(F.linear(y, leaves[0], leaves[1]))
        y = F.relu(F.linear(y, leaves[2], leaves[3]))
        loss = F.binary_cross_entropy_with_logits(F.linear(y, leaves[4], leaves[5]).view(-1), _d(s["labels"]))
        loss.backward()
        for i, p in enumerate(leaves):
            m[i] = 0.9 * m[i] + 0.1 * p.grad
            v[i] = 0.999 * v[i] + 0.001 * p.grad * p.grad
            params[i] = params[i] - CTR_LR * (m[i] / (1 - 0.9 ** step)) / ((v[i] / (1 - 0.999 ** step)).sqrt() + 1e-8)
        for f, t in enumerate(tables):
            g = torch.zeros_like(t[0]).index_add_(0, ids[:, f], emb.grad[:, f * dim:(f + 1) * dim])
            t[1] = t[1] + g * g
            t[0] = t[0] - PS_LR * g / (t[1].sqrt() + PS_EPS)
    return [loss.detach(), *params[:4], params[4].view(1, -1), params[5], *[t[0] for t in tables]]


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if work(case)["flops"] > 3e12:
        return None
    if kind in ("conv_bn", "stem"):
        conv, bn = s["conv"], s["bn"]
        pc, pb = _Params(conv), _Params(bn)
        # the images of the stem are rounded to bf16 when they enter the framework
        x = _leaf(s["x"].to(BF16))
        y = _bn64(_conv64(x, pc.map["weight"], conv.stride, conv.padding), pb, "", True, True)
        if kind == "stem":
            y = F.max_pool2d(y, 3, stride=2, padding=1)
        y.backward(_d(s["dy"]))
        tail = [pc.map["weight"].grad, *pb.grads(), pb.running["running_mean"], pb.running["running_var"]]
        return [y.detach(), *([x.grad] if kind == "conv_bn" else []), *tail]
    if kind == "block":
        p, x = _Params(s["m"]), _leaf(s["x"])
        y = _block64(s["m"], p, x, True)
        y.backward(_d(s["dy"]))
        return [y.detach(), x.grad, *p.grads(), *p.running.values()]
    if kind == "block_eval":
        return _block64(s["m"], _Params(s["m"]), _d(s["x"]), False).detach()
    if kind == "linear":
        p, x = _Params(s["lin"]), _leaf(s["x"])
        y = F.linear(x, p.map["weight"], p.map.get("bias"))
        y = {"relu": F.relu, "gelu": F.gelu}.get(case["act"], lambda t: t)(y)
        y.backward(_d(s["dy"]))
        return [y.detach(), x.grad, *p.grads()]
    if kind == "encoder":
        p, x = _Params(s["m"]), _leaf(s["x"])
        y = _encoder64(p, x, case["heads"])
        y.backward(_d(s["dy"]))
        return [y.detach(), x.grad, *p.grads()]
    if kind == "layer_norm":
        p, x, r = _Params(s["ln"]), _leaf(s["x"]), _leaf(s["r"])
        y = F.layer_norm(x + r, (case["cols"],), p.map["weight"], p.map["bias"], 1e-12)
        y.backward(_d(s["dy"]))
        return [y.detach(), x.grad, r.grad, *p.grads()]
    if kind == "mlm_head":
        h, w, b = _leaf(s["h"]), _leaf(s["w"]), _leaf(s["b"])
        logits = F.linear(h, w, b)
        loss = F.cross_entropy(logits, s["labels"], ignore_index=-100)
        loss.backward()
        return [loss.detach(), logits.detach(), h.grad, w.grad, b.grad]
    if kind == "ctr_step":
        return _ctr64(case, seed, s)
    if kind == "adamw":
        b1, b2 = ADAMW["betas"]
        new, means, squares = [], [], []
        for p, g in zip(s["params"], s["grads"]):
            w, g = _d(p), _d(g)
            m, v = (1 - b1) * g, (1 - b2) * g * g
            w = w * (1 - ADAMW["lr"] * ADAMW["weight_decay"]) - ADAMW["lr"] * (m / (1 - b1)) / ((v / (1 - b2)).sqrt() + ADAMW["eps"])
            new.append(w)
            means.append(m)
            squares.append(v)
        # the flat buffers' layout (order and alignment of the parameters) is the framework's own
        buckets = len(FusedAdamW([torch.nn.Parameter(p.detach().clone()) for p in s["params"]], **ADAMW).build())
        return [*new, *([None] * (3 * buckets))]
    ids, grads = s["ids"], _d(s["grads"])
    pulled, rows, acc = [], [], []
    for f, (w, a) in enumerate(_ps_tables(case, seed)):
        w, a, i = _d(w), _d(a), ids[:, f]
        pulled.append(w[i])
        g = torch.zeros_like(w).index_add_(0, i, grads[:, f * case["dim"]:(f + 1) * case["dim"]])
        a = a + g * g
        rows.append(w - PS_LR * g / (a.sqrt() + PS_EPS))
        acc.append(a)
    return [torch.cat(pulled, dim=1), *rows, *acc]
