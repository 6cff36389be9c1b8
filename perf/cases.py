"""The workloads by which this framework's speed is judged, through its public entry points.

A case is a dict of plain values.  ``listed`` gives the named ones, ``draw`` one more of the same
ranges, ``prepare`` what a program holds before the call (model, engine, batch on the GPU), ``run``
one pass, ``work`` the bytes and operations that the pass cannot do without, ``tolerance`` how far
two correct implementations at the same precision may be apart, ``exact`` the outputs in 64 bits.

Kinds: whole training steps of the decoder and convolution models through ``TrainEngine``, the
forward / backward of a pipeline stage's slice of a model, evaluation passes that return logits,
the attention operator by itself, and the 2-bit gradient codec.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from necklace_b200.comm.symm import SymmetricHeap
from necklace_b200.models.gpt2 import GPT2, GPT2Config
from necklace_b200.models.llama import Llama, LlamaConfig
from necklace_b200.models.resnet import ResNet
from necklace_b200.ops import (attention_qkv, dequantize_flat, matrix_dequantize, matrix_quantize,
                               quantize_flat)
from necklace_b200.ops.conv import BatchNorm2d, Conv2d
from necklace_b200.parallel.engine import GradCompConfig, OptimConfig, TrainEngine
from necklace_b200.parallel.flat import FlatParams

DEV = "cuda"


def listed() -> list[dict]:
    return [
        # the model of the smoke run and of a first experiment: everything is launch latency
        _gpt2_step("gpt2_tiny_step", n_layer=2, n_head=4, vocab=1000, B=2, S=256),
        # the benchmark's headline: GPT-2 medium, 8 x 1024 tokens, the step captured in a graph
        _gpt2_step("gpt2_medium_step", n_layer=24, n_head=16, vocab=50257, B=8, S=1024, graph=True),
        # accumulation over two micro-batches with clipping, sequences cut to an odd length and a
        # tenth of the targets ignored (padding), issued eagerly
        _gpt2_step("gpt2_accum_clip_step", n_layer=12, n_head=12, vocab=50257, B=6, S=771, micro=2,
                   clip=1.0),
        # scoring one prompt: forward only, logits of every position
        {"name": "gpt2_medium_logits", "kind": "gpt2_logits", "n_layer": 24, "n_head": 16,
         "vocab": 50257, "B": 1, "S": 333},
        # the data-parallel benchmark: ResNet-50, 256 images, 2-bit gradients with error feedback
        {"name": "resnet50_step", "kind": "resnet_step", "layers": "3,4,6,3", "N": 256, "H": 224,
         "W": 224, "codec": True, "graph": True},
        # convolution, batch norm and ReLU of a network of one's own: an odd batch of images that
        # are not square, there and back
        {"name": "conv_unit_ragged", "kind": "conv_unit", "cin": 64, "cout": 128, "k": 3,
         "stride": 1, "N": 33, "H": 40, "W": 53},
        # evaluation of a small batch with the running statistics
        {"name": "resnet50_infer", "kind": "resnet_infer", "layers": "3,4,6,3", "N": 37, "H": 224,
         "W": 224},
        # a pipeline stage's slice of the dp+pp+mp benchmark model: one micro-batch there and back
        {"name": "llama7b_stage", "kind": "llama_stage", "n_layer": 2, "n_head": 32, "d_ff": 11008,
         "B": 2, "S": 2048, "backward": True},
        # one layer of the dp+zr+mp model on a long odd sequence, forward only (recomputation,
        # evaluation)
        {"name": "llama13b_layer_fwd", "kind": "llama_stage", "n_layer": 1, "n_head": 40,
         "d_ff": 13824, "B": 1, "S": 4001, "backward": False},
        # a small Llama trained whole on one GPU, single odd sequence
        {"name": "llama_small_step", "kind": "llama_step", "n_layer": 4, "n_head": 8, "d_ff": 2752,
         "vocab": 32000, "B": 1, "S": 1501, "graph": False},
        # bidirectional attention on lengths that are not a multiple of a tile
        {"name": "attention_full", "kind": "attention", "B": 3, "H": 12, "S": 1111, "D": 64,
         "causal": False, "backward": True},
        # the codec on the flat gradient of ResNet-50 (25,557,032 parameters)
        {"name": "codec_resnet50", "kind": "codec", "n": 25557032, "ncol": 0, "fp32": False},
    ]


def _gpt2_step(name=None, *, n_layer, n_head, vocab, B, S, micro=1, clip=0.0, graph=False):
    c = {"kind": "gpt2_step", "n_layer": n_layer, "n_head": n_head, "vocab": vocab, "B": B, "S": S,
         "micro": micro, "clip": clip, "graph": graph}
    return {"name": name, **c} if name else c


def draw(rng) -> dict:
    def log(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["gpt2_step", "gpt2_step", "gpt2_logits", "resnet_step", "conv_unit",
                       "resnet_infer", "llama_stage", "llama_stage", "llama_step", "attention",
                       "codec"])
    if kind == "gpt2_step":
        micro = rng.choice([1, 1, 2])
        return _gpt2_step(n_layer=log(2, 24), n_head=rng.randint(2, 16), vocab=log(1000, 50257),
                          B=micro * log(1, 8 // micro), S=log(33, 1024), micro=micro,
                          clip=rng.choice([0.0, 1.0]), graph=rng.choice([False, True]))
    if kind == "gpt2_logits":
        return {"kind": kind, "n_layer": log(2, 24), "n_head": rng.randint(2, 16),
                "vocab": log(1000, 50257), "B": log(1, 8), "S": log(17, 1024)}
    if kind in ("resnet_step", "resnet_infer"):
        # 3 x 224 x 224 x 256 at most; small batches of odd sizes are as likely as large ones
        c = {"kind": kind, "layers": rng.choice(["3,4,6,3", "1,1,1,1", "2,2,2,2"]),
             "N": log(8, 256), "H": log(64, 224), "W": log(64, 224)}
        if kind == "resnet_step":
            c.update(codec=rng.choice([False, True]), graph=rng.choice([False, True]))
        return c
    if kind == "conv_unit":
        # the layers of a residual network and what lies between: wide images have few channels
        cin, cout = 8 * log(4, 128), 8 * log(4, 128)
        hw = max(7, 56 * 64 // max(cin, cout))
        return {"kind": kind, "cin": cin, "cout": cout, "k": rng.choice([1, 3, 3]),
                "stride": rng.choice([1, 1, 2]), "N": log(8, 256), "H": rng.randint(hw // 2, hw),
                "W": rng.randint(hw // 2, hw)}
    if kind == "llama_stage":
        B = rng.choice([1, 2])
        return {"kind": kind, "n_layer": rng.choice([1, 2]), "n_head": log(2, 40),
                "d_ff": 8 * log(64, 1728), "B": B, "S": log(65, 4096 // B),
                "backward": rng.choice([False, True])}
    if kind == "llama_step":
        return {"kind": kind, "n_layer": log(1, 8), "n_head": rng.randint(2, 8),
                "d_ff": 8 * log(32, 512), "vocab": log(1000, 32000), "B": log(1, 4),
                "S": log(33, 2048), "graph": rng.choice([False, True])}
    if kind == "attention":
        return {"kind": kind, "B": log(1, 8), "H": log(1, 32), "S": log(33, 2048),
                "D": rng.choice([64, 128]), "causal": rng.choice([False, True]),
                "backward": rng.choice([False, True])}
    if rng.choice([False, True]):
        return {"kind": "codec", "n": log(1001, 400000000 // 12), "ncol": 0,
                "fp32": rng.choice([False, True])}
    ncol = log(33, 4096)
    return {"kind": "codec", "n": log(33, 8192), "ncol": ncol, "fp32": True}


# ------------------------------------------------------------------------------------ prepare
def prepare(case: dict, seed: int) -> dict:
    return _PREPARE[case["kind"]](case, seed)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _tokens(c, seed):
    g = _gen(seed + 1)
    t = torch.randint(0, c["vocab"], (c["B"], c["S"] + 1), generator=g, device=DEV)
    x, y = t[:, :-1].contiguous(), t[:, 1:].contiguous()
    if c.get("micro", 1) > 1:                      # padded batches ignore a part of the targets
        y[torch.rand(y.shape, generator=g, device=DEV) < 0.1] = -100
    return x, y


def _adam():
    return OptimConfig("adam", lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1)


def _warm(engine, steps, *inputs):
    for _ in range(steps):                         # the step that captures the graph
        engine.step(*inputs)


def _prepare_gpt2(c, seed):
    torch.manual_seed(seed)
    d = 64 * c["n_head"]
    cfg = GPT2Config(n_layer=c["n_layer"], d_model=d, n_head=c["n_head"], d_ff=4 * d,
                     vocab=c["vocab"], max_seq=1024)
    model = GPT2(cfg, device=DEV)
    x, y = _tokens(c, seed)
    if c["kind"] == "gpt2_logits":
        return {"kind": c["kind"], "model": model, "x": x}
    eng = TrainEngine(model, optim=_adam(), micro_batches=c["micro"],
                      clip_grad_norm=c["clip"] or None, use_cuda_graph=c["graph"])
    if c["graph"]:
        _warm(eng, 1, x, y)
    return {"kind": c["kind"], "engine": eng, "x": x, "y": y}


def _resnet_like_trained(module, g):
    """Values as in the middle of a training run: the last norm of a block starts at zero and
    has grown, running statistics have left their start."""
    bns = [m for m in module.modules() if isinstance(m, BatchNorm2d)]
    stats = torch.empty(2, sum(m.C for m in bns), device=DEV)
    stats[0].normal_(0.0, 0.1, generator=g)
    stats[1].uniform_(0.5, 1.5, generator=g)
    o = 0
    for name, m in module.named_modules():
        if isinstance(m, BatchNorm2d):
            m.running_mean, m.running_var = stats[0, o:o + m.C], stats[1, o:o + m.C]
            o += m.C
            if name.endswith("bn3"):
                m.weight.data.fill_(0.2)
    return stats


def _prepare_resnet(c, seed):
    torch.manual_seed(seed)
    g = _gen(seed + 1)
    net = ResNet(1000, tuple(int(v) for v in c["layers"].split(",")), 64, device=DEV)
    stats = _resnet_like_trained(net, g)
    x = torch.randn(c["N"], c["H"], c["W"], 3, generator=g, device=DEV).bfloat16()
    y = torch.randint(0, 1000, (c["N"],), generator=g, device=DEV)
    if c["kind"] == "resnet_infer":
        return {"kind": c["kind"], "model": net.eval(), "x": x}
    kw = {}
    if c["codec"]:
        n = sum(p.numel() for p in net.parameters())
        heap = SymmetricHeap(int(n * (2 + 2 + 0.25 + 1) * 1.05) + (64 << 20))
        kw = dict(mode="dp", group=heap.peer_group(), heap=heap,
                  grad_comp=GradCompConfig(grad_comp_threshold=1e-3))
    eng = TrainEngine(net, optim=OptimConfig("sgd", lr=0.1, beta1=0.9), use_cuda_graph=c["graph"],
                      **kw)
    _warm(eng, 2 if c["graph"] else 0, x, y)       # SGD's first step is never the captured one
    return {"kind": c["kind"], "engine": eng, "x": x, "y": y, "stats": stats}


def _prepare_conv_unit(c, seed):
    torch.manual_seed(seed)
    g = _gen(seed + 1)
    k, st = c["k"], c["stride"]
    net = torch.nn.Sequential(Conv2d(c["cin"], c["cout"], k, st, k // 2, device=DEV),
                              BatchNorm2d(c["cout"], relu=True, device=DEV))
    x = torch.randn(c["N"], c["H"], c["W"], c["cin"], generator=g, device=DEV).relu().bfloat16()
    dy = torch.randn(c["N"], (c["H"] - 1) // st + 1, (c["W"] - 1) // st + 1, c["cout"],
                     generator=g, device=DEV).bfloat16()
    return {"kind": c["kind"], "model": net, "flat": FlatParams(net), "x": x.requires_grad_(True),
            "dy": dy}


def _prepare_llama_stage(c, seed):
    d = 128 * c["n_head"]
    cfg = LlamaConfig(n_layer=32, d_model=d, n_head=c["n_head"], d_ff=c["d_ff"], max_seq=c["S"])
    net = Llama(cfg, device=DEV, layers=range(c["n_layer"]), with_embed=False, with_head=False,
                seed=seed)
    g = _gen(seed + 1)
    x = torch.randn(c["B"], c["S"], d, generator=g, device=DEV).bfloat16()
    if not c["backward"]:
        return {"kind": c["kind"], "model": net, "x": x}
    dy = torch.randn(c["B"], c["S"], d, generator=g, device=DEV).bfloat16()
    return {"kind": c["kind"], "model": net, "flat": FlatParams(net), "x": x.requires_grad_(True),
            "dy": dy}


def _prepare_llama_step(c, seed):
    d = 128 * c["n_head"]
    cfg = LlamaConfig(n_layer=c["n_layer"], d_model=d, n_head=c["n_head"], d_ff=c["d_ff"],
                      vocab=c["vocab"], max_seq=c["S"])
    net = Llama(cfg, device=DEV, seed=seed)
    eng = TrainEngine(net, optim=_adam(), use_cuda_graph=c["graph"])
    x, y = _tokens(c, seed)
    if c["graph"]:
        _warm(eng, 1, x, y)
    return {"kind": c["kind"], "engine": eng, "x": x, "y": y}


def _prepare_attention(c, seed):
    g = _gen(seed)
    width = c["H"] * c["D"]
    qkv = torch.randn(c["B"], c["S"], 3 * width, generator=g, device=DEV).bfloat16()
    st = {"kind": c["kind"], "qkv": qkv, "H": c["H"], "causal": c["causal"], "dout": None}
    if c["backward"]:
        st["dout"] = torch.randn(c["B"], c["S"], width, generator=g, device=DEV).bfloat16()
        qkv.requires_grad_(True)
    return st


def _prepare_codec(c, seed):
    g = _gen(seed)
    shape = (c["n"], c["ncol"]) if c["ncol"] else (c["n"],)
    grad = torch.randn(shape, generator=g, device=DEV) * 1e-3
    st = {"kind": c["kind"], "ncol": c["ncol"], "thr": 1e-3,
          "grad": grad if c["fp32"] else grad.bfloat16()}
    if not c["ncol"]:
        st["residual"] = torch.randn(c["n"], generator=g, device=DEV) * 3e-4
        st["out"] = torch.empty(c["n"], dtype=st["grad"].dtype, device=DEV)
    return st


_PREPARE = {"gpt2_step": _prepare_gpt2, "gpt2_logits": _prepare_gpt2, "resnet_step": _prepare_resnet,
            "resnet_infer": _prepare_resnet, "conv_unit": _prepare_conv_unit,
            "llama_stage": _prepare_llama_stage, "llama_step": _prepare_llama_step,
            "attention": _prepare_attention, "codec": _prepare_codec}


# ---------------------------------------------------------------------------------------- run
def run(st: dict):
    kind = st["kind"]
    if kind in ("gpt2_step", "llama_step"):
        loss = st["engine"].step(st["x"], st["y"])
        return {"loss": loss, "grads": st["engine"].flat.grad, "weights": st["engine"].master}
    if kind == "resnet_step":
        # the weights and not the gradients: see tolerance()
        loss = st["engine"].step(st["x"], st["y"])
        return {"loss": loss, "weights": st["engine"].master, "stats": st["stats"]}
    if kind in ("gpt2_logits", "resnet_infer"):
        with torch.no_grad():
            return st["model"](st["x"])
    if kind == "llama_stage" and "flat" not in st:
        with torch.no_grad():
            return st["model"](st["x"])
    if kind in ("llama_stage", "conv_unit"):
        st["flat"].begin_step()
        y = st["model"](st["x"])
        st["x"].grad = None
        y.backward(st["dy"])
        st["flat"].finish_backward()
        return {"y": y.detach(), "dx": st["x"].grad, "grads": st["flat"].grad}
    if kind == "attention":
        if st["dout"] is None:
            with torch.no_grad():
                return attention_qkv(st["qkv"], st["H"], st["causal"])
        out = attention_qkv(st["qkv"], st["H"], st["causal"])
        st["qkv"].grad = None
        out.backward(st["dout"])
        return {"out": out.detach(), "dqkv": st["qkv"].grad}
    if st["ncol"]:
        codes, resid = matrix_quantize(st["grad"], st["thr"])
        return {"codes": codes, "residual": resid,
                "decoded": matrix_dequantize(codes, st["grad"].shape[0], st["thr"])}
    codes = quantize_flat(st["grad"], st["residual"], st["thr"])
    return {"codes": codes, "residual": st["residual"],
            "decoded": dequantize_flat(codes, st["out"], st["thr"])}


# --------------------------------------------------------------------------------------- work
def work(case: dict) -> dict:
    c, kind = case, case["kind"]
    if kind in ("gpt2_step", "gpt2_logits", "llama_step", "llama_stage"):
        T = c["B"] * c["S"]
        if kind.startswith("gpt2"):
            d = 64 * c["n_head"]
            per, table = 12 * d * d, c["vocab"] * d
            n = c["n_layer"] * per + table + 1024 * d
        else:
            d = 128 * c["n_head"]
            per, table = 4 * d * d + 3 * d * c["d_ff"], c.get("vocab", 0) * d
            n = c["n_layer"] * per + 2 * table
        # matrix products per token, and causal attention (half of the score matrix)
        fwd = T * (2 * (c["n_layer"] * per + table) + c["n_layer"] * 2 * c["S"] * d)
        if kind.endswith("step"):
            # gradient written and read (bf16), three fp32 states read and written, bf16 copy read
            # in forward and backward and written
            return {"bytes": n * (2 * 2 + 3 * 8 + 3 * 2) + T * 16, "flops": 3 * fwd}
        if kind == "gpt2_logits":
            return {"bytes": 2 * n + 8 * T + 2 * T * c["vocab"], "flops": fwd}
        if c["backward"]:
            return {"bytes": 2 * n * 3 + 2 * T * d * 4, "flops": 3 * fwd}
        return {"bytes": 2 * n + 2 * T * d * 2, "flops": fwd}
    if kind in ("resnet_step", "resnet_infer"):
        macs, n, H, W = _resnet_macs(c)
        img = c["N"] * c["H"] * c["W"] * 3
        if kind == "resnet_infer":
            return {"bytes": 2 * n + 2 * img + 2 * 1000 * c["N"], "flops": 2 * macs * c["N"]}
        # no gradient of the images; weights and momentum in fp32, bf16 copy and gradient
        return {"bytes": n * (2 * 2 + 2 * 8 + 3 * 2) + 2 * img,
                "flops": 6 * macs * c["N"] - 2 * c["N"] * H * W * 147 * 64}
    if kind == "conv_unit":
        h, w = (c["H"] - 1) // c["stride"] + 1, (c["W"] - 1) // c["stride"] + 1
        n = c["cin"] * c["cout"] * c["k"] ** 2
        x, y = c["N"] * c["H"] * c["W"] * c["cin"], c["N"] * h * w * c["cout"]
        return {"bytes": 2 * (2 * x + 2 * y) + 2 * 3 * n, "flops": 6 * n * c["N"] * h * w}
    if kind == "attention":
        n, pairs = c["B"] * c["S"] * c["H"] * c["D"], c["B"] * c["H"] * c["S"] * c["S"] * c["D"]
        fl = 4 * pairs * (0.5 if c["causal"] else 1)
        if c["backward"]:
            return {"bytes": 2 * n * (3 + 1 + 1 + 3), "flops": 3.5 * fl}
        return {"bytes": 2 * n * 4, "flops": fl}
    n = c["n"] * (c["ncol"] or 1)
    e = 4 if c["fp32"] else 2
    # gradient in, residual in (flat form) and out, codes out and in, decoded values out
    return {"bytes": n * (e + (4 if c["ncol"] else 8) + 0.5 + e), "flops": 0}


def _bottleneck_macs(cin, width, stride, blocks, H, W):
    """(multiply-adds per image, parameters, output height, width)"""
    h, w = (H - 1) // stride + 1, (W - 1) // stride + 1
    macs = H * W * cin * width + h * w * (9 * width * width + 4 * width * width)
    n = cin * width + 13 * width * width
    if stride != 1 or cin != 4 * width:
        macs, n = macs + h * w * cin * 4 * width, n + cin * 4 * width
    macs += (blocks - 1) * h * w * 17 * width * width
    return macs, n + (blocks - 1) * 17 * width * width, h, w


def _resnet_macs(c):
    """(multiply-adds per image, parameters, stem output height, width)"""
    H, W = (c["H"] - 1) // 2 + 1, (c["W"] - 1) // 2 + 1
    macs, n = H * W * 147 * 64, 147 * 64
    h, w, cin = (H - 1) // 2 + 1, (W - 1) // 2 + 1, 64
    for i, blocks in enumerate(int(v) for v in c["layers"].split(",")):
        m, k, h, w = _bottleneck_macs(cin, 64 << i, 1 if i == 0 else 2, blocks, h, w)
        macs, n, cin = macs + m, n + k, 256 << i
    return macs + 2048 * 1000, n + 2048 * 1000, H, W


# ---------------------------------------------------------------------------------- tolerance
def tolerance(case: dict):
    """Measured: the same model with the same weights and batch at reduced sizes on the CPU path
    (bf16 at the same places, fp32 sums in another order) against the GPU, times about four.

    gpt2_step      gradients 0.5 - 1.0 %, single values 0.7 of the root mean square
    gpt2_logits    1.3 %, 0.06 (24 layers)
    resnet_step    weights 0.1 %, 0.22.  The gradients themselves differ by 23 %: a bf16 rounding
                   that falls the other way moves a value across a ReLU's zero, and the masks of
                   fifty layers multiply; their sum in the weights is what two runs can share
    conv_unit      0.04 %, 0.013; one flipped ReLU mask moves single gradients of a narrow
                   1x1 convolution by up to half of the root mean square
    resnet_infer   0.4 %, 0.016
    llama_stage    0.3 %, 0.04
    llama_step     0.8 %, 0.27
    attention      0.26 %, 0.07
    codec          the codes, the residual and the decoded values are the same bits
    """
    return {"gpt2_step": {"rel": 3e-2, "max": 0.99}, "gpt2_logits": {"rel": 3e-2, "max": 0.25},
            "resnet_step": {"rel": 4e-3, "max": 0.88}, "conv_unit": {"rel": 2e-3, "max": 0.5},
            "resnet_infer": {"rel": 1.6e-2, "max": 0.07}, "llama_stage": {"rel": 1.2e-2, "max": 0.16},
            "llama_step": {"rel": 3e-2, "max": 0.99}, "attention": {"rel": 1e-2, "max": 0.28},
            "codec": "exact"}[case["kind"]]


# -------------------------------------------------------------------------------------- exact
def exact(case: dict, seed: int):
    """The outputs of ``run`` in plain torch and 64 bits.  Inputs, weights and the layout of the
    flat gradient come from the state of ``prepare``.  The updated weights of an optimizer step are
    left out: Adam's first update is the sign of the gradient.  So is the whole convolution step,
    whose gradients have no digits to compare (see ``tolerance``)."""
    kind = case["kind"]
    if kind == "resnet_step":
        return None
    st = prepare(case, seed)
    with torch.enable_grad():
        return _EXACT[kind](case, st)


def _leaves64(flat):
    return {n: p.detach().double().requires_grad_(True) for n, p in zip(flat.names, flat.params)}


def _flat_grad64(flat, w):
    """The gradients at their places in the flat buffer."""
    out = torch.zeros(flat.numel, dtype=torch.float64, device=DEV)
    for n, o in zip(flat.names, flat.offsets):
        if w[n].grad is not None:
            out[o:o + w[n].numel()] = w[n].grad.reshape(-1)
    return out


def _softmax_attention64(q, k, v, causal):
    s = (q @ k.transpose(-1, -2)) / math.sqrt(q.shape[-1])
    if causal:
        s = s.masked_fill(~torch.ones(s.shape[-2:], dtype=torch.bool, device=DEV).tril(),
                          float("-inf"))
    return torch.softmax(s, -1) @ v


def _attention64(qkv, H, causal, rotate=False):
    B, S, C3 = qkv.shape
    q, k, v = qkv.view(B, S, 3, H, C3 // 3 // H).permute(2, 0, 3, 1, 4)
    if rotate:
        half = q.shape[-1] // 2
        a = torch.arange(S, dtype=torch.float64, device=DEV)[:, None] * 10000.0 ** (
            -torch.arange(half, dtype=torch.float64, device=DEV) / half)
        cos, sin = a.cos(), a.sin()
        q, k = (torch.cat([t[..., :half] * cos - t[..., half:] * sin,
                           t[..., half:] * cos + t[..., :half] * sin], -1) for t in (q, k))
    # a head of every sample at a time: the score matrices of all heads take too much memory
    out = [checkpoint(_softmax_attention64, q[:, h], k[:, h], v[:, h], causal, use_reentrant=False)
           for h in range(H)]
    return torch.stack(out, 2).reshape(B, S, C3 // 3)


def _gpt2_block64(x, w, pre, H):
    C = x.shape[-1]

    def ln(t, n):
        return F.layer_norm(t, (C,), w[pre + n + ".weight"], w[pre + n + ".bias"], 1e-5)

    def lin(t, n):
        return t @ w[pre + "w_" + n].t() + w[pre + "b_" + n]

    x = x + lin(_attention64(lin(ln(x, "ln1"), "qkv"), H, True), "proj")
    return x + lin(F.gelu(lin(ln(x, "ln2"), "fc1"), approximate="tanh"), "fc2")


def _gpt2_logits64(c, w, idx):
    table = w["embed.emb.wte"]
    x = table[idx] + w["embed.emb.wpe"][:idx.shape[1]]
    for i in range(c["n_layer"]):
        x = checkpoint(_gpt2_block64, x, w, f"blocks.{i}.", c["n_head"], use_reentrant=False)
    x = F.layer_norm(x, x.shape[-1:], w["head.ln_f.weight"], w["head.ln_f.bias"], 1e-5)
    return x @ table[:c["vocab"]].t()


def _llama_block64(x, w, pre, H):
    def rms(t, n):
        return t * torch.rsqrt(t.square().mean(-1, keepdim=True) + 1e-6) * w[pre + n + ".weight"]

    x = x + _attention64(rms(x, "ln1") @ w[pre + "w_qkv"].t(), H, True, True) @ w[pre + "w_o"].t()
    g, u = (rms(x, "ln2") @ w[pre + "w_gu"].t()).chunk(2, -1)
    return x + (F.silu(g) * u) @ w[pre + "w_down"].t()


def _llama_blocks64(c, w, x):
    for i in range(c["n_layer"]):
        x = checkpoint(_llama_block64, x, w, f"blocks.{i}.", c["n_head"], use_reentrant=False)
    return x


def _llama_logits64(c, w, idx):
    x = _llama_blocks64(c, w, w["embed.wte"][idx])
    x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w["head.norm.weight"]
    return x @ w["head.w_out"][:c["vocab"]].t()


def _exact_step(c, st):
    flat = st["engine"].flat
    w, total = _leaves64(flat), 0.0
    logits = _gpt2_logits64 if c["kind"] == "gpt2_step" else _llama_logits64
    k = c.get("micro", 1)
    for x, y in zip(st["x"].chunk(k), st["y"].chunk(k)):
        loss = F.cross_entropy(logits(c, w, x).flatten(0, 1), y.reshape(-1), ignore_index=-100)
        loss.backward()
        total = total + loss.detach() / k
    return {"loss": total, "grads": _flat_grad64(flat, w), "weights": None}


def _exact_gpt2_logits(c, st):
    with torch.no_grad():
        w = {n: p.double() for n, p in st["model"].named_parameters()}
        return _gpt2_logits64(c, w, st["x"])


def _there_and_back64(st, w, fn):
    x = st["x"].detach().double().requires_grad_(True)
    y = fn(x)
    y.backward(st["dy"].double())
    return {"y": y.detach(), "dx": x.grad, "grads": _flat_grad64(st["flat"], w)}


def _exact_llama_stage(c, st):
    if not c["backward"]:
        with torch.no_grad():
            w = {n: p.double() for n, p in st["model"].named_parameters()}
            return _llama_blocks64(c, w, st["x"].double())
    w = _leaves64(st["flat"])
    return _there_and_back64(st, w, lambda x: _llama_blocks64(c, w, x))


def _conv64(x, w, k, stride, pad):
    """``x`` [N, H, W, C], ``w`` [out, (kh, kw, c) and padding]."""
    N, H, W, C = x.shape
    t = F.pad(x, (0, 0, pad, pad, pad, pad))
    h, v = (H + 2 * pad - k) // stride + 1, (W + 2 * pad - k) // stride + 1
    taps = [t[:, i:i + (h - 1) * stride + 1:stride, j:j + (v - 1) * stride + 1:stride]
            for i in range(k) for j in range(k)]
    return torch.cat(taps, -1) @ w[:, :k * k * C].t()


def _exact_conv_unit(c, st):
    w = _leaves64(st["flat"])

    def fn(x):
        y = _conv64(x, w["0.weight"], c["k"], c["stride"], c["k"] // 2)
        var, mean = torch.var_mean(y, (0, 1, 2), unbiased=False)
        return torch.relu((y - mean) * torch.rsqrt(var + 1e-5) * w["1.weight"] + w["1.bias"])

    return _there_and_back64(st, w, fn)


def _exact_resnet_infer(c, st):
    net = st["model"]

    def unit(x, conv, bn):
        y = _conv64(x, conv.weight.double(), conv.k, conv.stride, conv.pad)
        a = bn.weight.double() * torch.rsqrt(bn.running_var.double() + 1e-5)
        return (y - bn.running_mean.double()) * a + bn.bias.double()

    def features(x):
        x = torch.relu(unit(x, net.conv1, net.bn1)).permute(0, 3, 1, 2)
        x = F.max_pool2d(x, 3, 2, 1).permute(0, 2, 3, 1)
        for layer in (net.layer1, net.layer2, net.layer3, net.layer4):
            for b in layer:
                idt = x if b.down_conv is None else unit(x, b.down_conv, b.down_bn)
                y = torch.relu(unit(torch.relu(unit(x, b.conv1, b.bn1)), b.conv2, b.bn2))
                x = torch.relu(unit(y, b.conv3, b.bn3) + idt)
        return x.mean((1, 2))

    with torch.no_grad():
        f = torch.cat([features(x.double()) for x in st["x"].split(32)])
        return f @ net.fc_weight.double()[:1000].t() + net.fc_bias.double()[:1000]


def _exact_attention(c, st):
    qkv = st["qkv"].detach().double().requires_grad_(c["backward"])
    out = _attention64(qkv, c["H"], c["causal"])
    if not c["backward"]:
        return out
    out.backward(st["dout"].double())
    return {"out": out.detach(), "dqkv": qkv.grad}


def _exact_codec(c, st):
    # which value is over the threshold is decided on the 32-bit sum
    a = st["grad"].float() + (st["residual"] if not c["ncol"] else 0.0)
    thr = float(torch.tensor(st["thr"], dtype=torch.float32))
    dec = (a >= thr).double().mul_(thr) - (a <= -thr).double().mul_(thr)
    return {"codes": None, "residual": a.double() - dec, "decoded": dec}


_EXACT = {"gpt2_step": _exact_step, "llama_step": _exact_step, "gpt2_logits": _exact_gpt2_logits,
          "llama_stage": _exact_llama_stage, "conv_unit": _exact_conv_unit,
          "resnet_infer": _exact_resnet_infer, "attention": _exact_attention,
          "codec": _exact_codec}
