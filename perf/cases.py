"""The work that a user of this framework has it do, as cases that can be timed.

Four kinds of case, each through the public entry point that a program uses for it:

  gemm   `self_ops.approx_gemm_op` on float tensors of codes, forward and backward (both gradients): the operator API
  conv   an `AppConv2d` layer in training: observers, quantisation, LUT convolution, de-quantisation and their backward
  linear an `AppLinear` layer in training, the same for a token matrix
  model  a whole network: a training pass (forward, loss, backward) or an evaluation pass (forward under no_grad)

The tables are those of the synthetic multiplier (`lutgemm_luts`), max(0, x*y + e) with window-difference gradients.
"""
from __future__ import annotations

import math
import os
import sys

import torch
import torch.nn.functional as F

# the package of the repository that is the working folder
_PKG = os.path.join(os.getcwd(), "appmult-aware-retraining_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import self_ops  # noqa: E402
from lutgemm_dp import OverlappedGradReducer  # noqa: E402
from lutgemm_layers import AppConv2d, AppLinear, prepare as prepare_model  # noqa: E402
from lutgemm_luts import synthetic_multiplier, window_difference_gradients  # noqa: E402
from lutgemm_models import MODELS, lut_macs_per_image  # noqa: E402
from self_ops.ops_py import approx_ops as op_state  # noqa: E402


def listed():
    return [
        # one small linear layer through the operator API (the single-layer benchmark configuration): launch-bound
        dict(name="gemm7_256x512x256", kind="gemm", bits=7, m=256, k=512, n=256),
        # odd sizes, nothing a multiple of a vector or a tile
        dict(name="gemm7_1000x777x333", kind="gemm", bits=7, m=1000, k=777, n=333),
        # the square sweep: the headline size at 8 bits, and the two narrow tables at their ordinary sizes
        dict(name="gemm8_4096", kind="gemm", bits=8, m=4096, k=4096, n=4096),
        dict(name="gemm6_2048", kind="gemm", bits=6, m=2048, k=2048, n=2048),
        dict(name="gemm4_1024", kind="gemm", bits=4, m=1024, k=1024, n=1024),
        # ResNet-18 (CIFAR shape) stage 1: many output positions, few channels, 7 bits
        dict(name="conv7_64x64_3x3_at32", kind="conv", bits=7, b=256, cin=64, cout=64, h=32, kernel=3, stride=1, pad=1),
        # ResNet-18 stage 3 to stage 4: stride 2, many channels, 8 bits
        dict(name="conv8_256x512_3x3s2_at8", kind="conv", bits=8, b=256, cin=256, cout=512, h=8, kernel=3, stride=2, pad=1),
        # ResNet-50 (ImageNet shape) bottleneck reduction: 1x1, 8 bits
        dict(name="conv8_256x64_1x1_at56", kind="conv", bits=8, b=64, cin=256, cout=64, h=56, kernel=1, stride=1, pad=0),
        # ViT-S MLP: 64 images of 197 tokens, 384 -> 1536, 7 bits
        dict(name="linear7_12608x384x1536", kind="linear", bits=7, m=12608, k=384, n=1536),
        # evaluation of a small batch: latency of the forward path of a whole network
        dict(name="resnet18_eval_b16", kind="model", model="resnet18", train=False, bits=7, b=16),
        # the two training workloads with their own batch sizes
        dict(name="resnet18_train_b256", kind="model", model="resnet18", train=True, bits=7, b=256),
        dict(name="vit_s_train_b64", kind="model", model="vit_s", train=True, bits=7, b=64),
    ]


# most LUT-MACs of one drawn pass (forward and both gradients): below a third of the largest listed case
_DRAW_MACS = 2.0e11


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channels(rng, lo, hi):
    c = _log_uniform(rng, lo, hi)
    return c if rng.random() < 0.3 else max(8, (c + 4) // 8 * 8)  # mostly multiples of 8, as networks have them


def draw(rng):
    """One more case of the same ranges: 7 and 8 bits in two of three, 4 and 6 bits in the others."""
    bits = rng.choice([7, 7, 8, 8, 6, 4])
    kind = rng.choice(["gemm", "gemm", "conv", "conv", "conv", "linear", "model"])
    while True:
        if kind == "gemm":
            case = dict(kind=kind, bits=bits, m=_log_uniform(rng, 64, 16384), k=_log_uniform(rng, 32, 8192),
                        n=_log_uniform(rng, 16, 8192))
            if rng.random() < 0.5:  # whole multiples of 64 as often as odd sizes
                for d in "mkn":
                    case[d] = max(64, case[d] // 64 * 64)
            macs = case["m"] * case["k"] * case["n"]
        elif kind == "conv":
            kernel = rng.choice([1, 3, 3, 3, 5, 7])
            stride = rng.choice([1, 1, 2])
            case = dict(kind=kind, bits=bits, b=_log_uniform(rng, 8, 256), cin=_channels(rng, 3, 512),
                        cout=_channels(rng, 16, 512), h=_log_uniform(rng, max(kernel, 4), 64), kernel=kernel, stride=stride,
                        pad=kernel // 2)
            macs = _conv_macs(case)
        elif kind == "linear":
            case = dict(kind=kind, bits=bits, m=_log_uniform(rng, 32, 16384), k=_channels(rng, 64, 2048),
                        n=_channels(rng, 10, 2048))
            macs = case["m"] * case["k"] * case["n"]
        else:
            # a forward pass of any small batch, or a training pass
            name = rng.choice(["resnet18", "resnet18", "resnet50", "vit_s"])
            train = rng.random() < 0.5
            most = {"resnet18": 256, "resnet50": 12, "vit_s": 14}[name]
            case = dict(kind=kind, model=name, train=train, bits=rng.choice([7, 8]), b=_log_uniform(rng, 1 if not train else 4, most))
            return case
        if 1e6 < macs <= _DRAW_MACS / 3:
            return case


def _conv_out(case):
    return (case["h"] + 2 * case["pad"] - case["kernel"]) // case["stride"] + 1


def _conv_macs(case):
    return case["b"] * _conv_out(case) ** 2 * case["cin"] * case["kernel"] ** 2 * case["cout"]


# ---- tables -----------------------------------------------------------------------------------------------------------
_TABLES = {}  # bit-width -> the three device tables; a program loads its table file once, before anything else


def _tables(bits):
    if bits not in _TABLES:
        fp = synthetic_multiplier(bits, seed=0)
        ga, gb = window_difference_gradients(fp, max(1, (1 << bits) // 16))
        self_ops.set_lookup_tables(torch.device("cuda"), fp, ga, gb, bits)
        _TABLES[bits] = (op_state.lut_appmult, op_state.lut_grad_a, op_state.lut_grad_b)
    return _TABLES[bits]


def _use_tables(tables):
    # a program has one multiplier and installs its tables once; here several bit-widths share a process
    op_state.lut_appmult, op_state.lut_grad_a, op_state.lut_grad_b = tables


# ---- states -------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    state = dict(kind=case["kind"], tables=_tables(case["bits"]))

    def randn(*shape):
        return torch.randn(*shape, generator=gen, device=dev)

    if case["kind"] == "gemm":
        # uniform codes and a N(0,1) gradient, as the operator benchmarks have them
        def codes(*shape):
            return torch.randint(0, 1 << case["bits"], shape, generator=gen, device=dev).float().requires_grad_(True)

        state.update(a=codes(case["m"], case["k"]), w=codes(case["k"], case["n"]), g=randn(case["m"], case["n"]))
        return state
    torch.manual_seed(seed)  # module initialisers draw from the global generators
    if case["kind"] == "conv":
        layer = AppConv2d(case["cin"], case["cout"], case["kernel"], case["stride"], case["pad"], bias=False,
                          a_bits=case["bits"], w_bits=case["bits"], conv_impl="layer")
        torch.nn.init.kaiming_normal_(layer.weight, mode="fan_out", nonlinearity="relu")
        ho = _conv_out(case)
        # activations after a ReLU, and the memory format in which networks are trained
        x = F.relu(randn(case["b"], case["cin"], case["h"], case["h"])).contiguous(memory_format=torch.channels_last)
        g = randn(case["b"], case["cout"], ho, ho).contiguous(memory_format=torch.channels_last)
        layer = layer.to(dev).to(memory_format=torch.channels_last)
    elif case["kind"] == "linear":
        layer = AppLinear(case["k"], case["n"], a_bits=case["bits"], w_bits=case["bits"], impl="layer").to(dev)
        x, g = randn(case["m"], case["k"]), randn(case["m"], case["n"])  # as after a layer norm
    else:
        ctor, shape, classes = MODELS[case["model"]]
        model = ctor(classes).to(dev)
        prepare_model(model, a_bits=case["bits"], w_bits=case["bits"], conv_impl="layer")
        model = model.to(memory_format=torch.channels_last).train()
        state.update(model=model, images=randn(case["b"], *shape), train=case["train"],
                     labels=torch.randint(0, classes, (case["b"],), generator=gen, device=dev))
        if case["train"]:
            state["reducer"] = OverlappedGradReducer(model.parameters())
        else:
            _use_tables(state["tables"])
            with torch.no_grad():
                model(state["images"])  # the observers have seen data
            model.eval()
        return state
    layer.train()
    state.update(layer=layer, x=x.requires_grad_(True), g=g)
    return state


def run(state):
    _use_tables(state["tables"])
    if state["kind"] == "gemm":
        a, w = state["a"], state["w"]
        a.grad = w.grad = None
        out = self_ops.approx_gemm_op(a, w)
        out.backward(state["g"])
        return {"out": out.detach(), "grad_a": a.grad, "grad_w": w.grad}
    if state["kind"] in ("conv", "linear"):
        layer, x = state["layer"], state["x"]
        x.grad = None
        for p in layer.parameters():
            p.grad = None
        out = layer(x)
        out.backward(state["g"])
        return {"out": out.detach(), "grad_x": x.grad, "grads": [p.grad for p in layer.parameters()]}
    model = state["model"]
    if not state["train"]:
        with torch.no_grad():
            return {"logits": model(state["images"])}
    reducer = state["reducer"]
    reducer.zero_grad()
    logits = model(state["images"])
    loss = F.cross_entropy(logits, state["labels"])
    loss.backward()
    reducer.finish()
    return {"logits": logits.detach(), "loss": loss.detach(), "grads": reducer.flat}


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
_PER_IMAGE = {}


def _model_counts(name):
    """(LUT-MACs per image, parameters) of a network."""
    if name not in _PER_IMAGE:
        ctor, shape, classes = MODELS[name]
        model = ctor(classes)
        _PER_IMAGE[name] = (lut_macs_per_image(model, shape), sum(p.numel() for p in model.parameters()),
                            math.prod(shape), classes)
    return _PER_IMAGE[name]


def work(case):
    """A LUT-MAC counts as two operations (the look-up's product and its addition); a training pass has three per
    (m, k, n).  Bytes: fp32 inputs, weights and incoming gradients once in, results and gradients once out."""
    if case["kind"] in ("gemm", "linear"):
        m, k, n = case["m"], case["k"], case["n"]
        macs, values = m * k * n, 2 * (m * k + k * n + m * n)
    elif case["kind"] == "conv":
        macs = _conv_macs(case)
        ho = _conv_out(case)
        values = 2 * (case["b"] * case["cin"] * case["h"] ** 2 + case["cin"] * case["cout"] * case["kernel"] ** 2
                      + case["b"] * case["cout"] * ho * ho)
    else:
        per_image, params, pixels, classes = _model_counts(case["model"])
        passes = 3 if case["train"] else 1
        return {"bytes": 4.0 * (case["b"] * (pixels + classes) + params * (2 if case["train"] else 1)),
                "flops": 2.0 * passes * per_image * case["b"]}
    return {"bytes": 4.0 * values, "flops": 6.0 * macs}


def tolerance(case):
    """The integer sums are exact, so forward results of one operator or layer differ by roundings of the
    de-quantisation only; gradients are fp32 sums of up to a few hundred thousand terms.  The same gradients with their
    sums in another order (the broadcast against the slab kernels) and, for operators, against 64-bit sums differ by at
    most: operators 1.2e-6, layers 4.7e-6, all gradients of a network 1.1e-5."""
    if case["kind"] == "model":
        return {"rel": 5e-5 if case["train"] else 1e-5}
    return {"rel": 5e-6 if case["kind"] == "gemm" else 2e-5}
