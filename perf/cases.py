"""What users of this library have it do, as measurable cases over the public entry points.

    listed()              the named cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   inputs (and carried state) on the GPU, from the seed alone
    run(state)            one pass through the entry points, outputs whole
    work(case)            bytes and flops of one pass that the path cannot do without
    tolerance(case)       how far another correct implementation at the same precision may be off

A case has a ``kind``, which says who calls what:

    forward   ``mlstm_matmul``: the parallel form without gradients
    train     ``Triton_mLSTM.apply`` and its backward (``gated``: with the output gate as eighth argument)
    scan      ``mlstm_scan``: forward with output gate
    long      ``mlstm_chunkwise``: a long sequence, forward
    scantrain ``mlstm_scan`` on inputs that require gradients
    segment   ``mlstm_scan`` with ``initial`` and ``return_state``: a prompt read in segments, or, with one
              or a few tokens, the decoding step after it
"""
import importlib
import math

import torch

PKG = importlib.import_module("xlstm-triton-cuda-implementation_b200")

_DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
_CHUNK = 256          # the block length of the chunkwise form (the entry points' default)


def _case(kind, dtype, B, NH, S, D, gated=False, f_mean=3.0, name=None):
    c = dict(kind=kind, dtype=dtype, B=B, NH=NH, S=S, D=D, gated=gated, f_mean=f_mean)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # the C++ driver's single head (S = 640, D = 128, fp16): a call that is nearly all latency
        _case("forward", "fp16", 1, 1, 640, 128, f_mean=0.0, name="forward_one_head_fp16"),
        # a few short sequences at inference, 16-bit, with a length that is a multiple of nothing
        _case("scan", "bf16", 4, 8, 333, 64, gated=True, name="scan_short_ragged_bf16"),
        # the matmul demo: fp32, forward + backward through the autograd function
        _case("train", "fp32", 1, 4, 2048, 64, f_mean=0.0, name="train_demo_fp32_d64"),
        # fp32 training at a model's head dimension: reproducing or debugging a run in full precision
        _case("train", "fp32", 1, 4, 1024, 256, name="train_fp32_d256"),
        # a small model's training step with output gate and a ragged length
        _case("train", "bf16", 2, 8, 1000, 128, gated=True, name="train_gated_ragged_bf16_d128"),
        # the model-scale training step, the benchmark's workload
        _case("train", "bf16", 16, 8, 4096, 256, name="train_model_bf16_d256"),
        # wide heads, trained in 16 bits
        _case("train", "bf16", 4, 8, 2048, 512, name="train_wide_bf16_d512"),
        # the scan demo: fp32, D = 1024, output gate
        _case("scan", "fp32", 1, 4, 2048, 1024, gated=True, f_mean=0.0, name="scan_demo_fp32_d1024"),
        # a long context read in one call
        _case("long", "bf16", 1, 8, 65536, 128, name="long_forward_bf16_d128"),
        # training on long sequences, linear in the length
        _case("scantrain", "bf16", 1, 8, 16384, 128, gated=True, name="long_train_bf16_d128"),
        # one segment of a batch of prompts, with the state carried in and out
        _case("segment", "bf16", 4, 8, 2048, 256, gated=True, name="segment_prefill_bf16_d256"),
        # the decoding step behind it: one token per sequence
        _case("segment", "bf16", 16, 8, 1, 128, gated=True, name="decode_one_token_bf16_d128"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One case of the ranges behind the listed ones.  Lengths over their logarithm, half of them as they fall and half
    on a multiple of 64; batches and heads as far as the largest listed cases pay for them: ``pairs`` bounds what the
    forms with every earlier position taken directly cost, ``values`` what the ones that are linear in the length do."""
    kind, pairs, values = rng.choice([
        ("forward", 5e11, 2e8), ("train", 5e11, 2e8), ("train", 1e11, 1e8), ("train32", 2.2e9, 1e8), ("wide", 2e11, 1e8),
        ("scan", 4e10, 1e8), ("long", 1e16, 1.4e8), ("scantrain", 1e16, 7e7), ("segment", 1e16, 7e7), ("decode", 1e16, 1e8)])
    while True:
        half = rng.choice(["bf16", "bf16", "fp16"])
        B, NH = _log_int(rng, 1, 16), rng.choice([1, 2, 4, 6, 8])
        gated, f_mean = rng.random() < 0.5, rng.choice([3.0, 3.0, 1.0, 0.0])
        if kind == "forward":
            c = _case("forward", half, B, NH, _log_int(rng, 100, 4096), rng.choice([64, 128, 256]), f_mean=f_mean)
        elif kind == "train":
            c = _case("train", half, B, NH, _log_int(rng, 128, 4096), rng.choice([64, 128, 256]), gated, f_mean)
        elif kind == "train32":
            c = _case("train", "fp32", rng.choice([1, 1, 2]), NH, _log_int(rng, 128, 2048), rng.choice([32, 64, 128, 256]), gated, f_mean)
        elif kind == "wide":
            c = _case("train", half, B, NH, _log_int(rng, 256, 4096), rng.choice([512, 512, 768, 1024]), gated, f_mean)
        elif kind == "scan":
            c = _case("scan", rng.choice(["fp32", half]), rng.choice([1, 2, 4]), NH, _log_int(rng, 128, 4096),
                      rng.choice([64, 128, 256, 512, 1024]), True, f_mean)
        elif kind == "long":
            c = _case("long", half, rng.choice([1, 1, 2]), NH, _log_int(rng, 4096, 65536), rng.choice([128, 128, 256]), f_mean=f_mean)
        elif kind == "scantrain":
            c = _case("scantrain", half, rng.choice([1, 1, 2]), NH, _log_int(rng, 2048, 16384), rng.choice([128, 256]), True, f_mean)
        elif kind == "segment":
            c = _case("segment", half, B, NH, _log_int(rng, 64, 4096), rng.choice([128, 256]), gated, f_mean)
        else:
            c = _case("segment", half, _log_int(rng, 1, 64), NH, rng.choice([1, 1, 1, 2, 4, 8]), rng.choice([128, 256]), gated, f_mean)
        if rng.random() < 0.5 and c["S"] >= 128:
            c["S"] = c["S"] // 64 * 64
        n = c["B"] * c["NH"] * c["S"] * c["D"]
        if n * c["S"] <= pairs and n <= values:
            return c


def _carried_state(c, g, dev):
    """The state behind an earlier part of the sequence: what ``return_state`` of the call before gave."""
    BH, D, T = c["B"] * c["NH"], c["D"], 192
    k, v = (torch.randn(BH, T, D, device=dev, generator=g) * D ** -0.5 for _ in range(2))
    f = c["f_mean"] + torch.randn(BH, T, device=dev, generator=g)
    i = torch.randn(BH, T, device=dev, generator=g)
    F = torch.nn.functional.logsigmoid(f).double().cumsum(1)
    a = i.double() - F
    A = a.max(1).values
    kw = k * torch.exp(a - A[:, None]).float()[:, :, None]
    return kw.transpose(1, 2) @ v, kw.sum(1), F[:, -1].clone(), A


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(int(seed))
    dt, shape = _DTYPES[case["dtype"]], (case["B"], case["NH"], case["S"], case["D"])
    # the demos draw q, k, v ~ N(0, 1) in fp32; at model scale they are normalised, N(0, 1 / D)
    scale = 1.0 if case["dtype"] == "fp32" and case["f_mean"] == 0.0 else case["D"] ** -0.5
    s = dict(kind=case["kind"])
    x = {n: (torch.randn(shape, device=dev, generator=g) * scale).to(dt) for n in ("q", "k", "v")}
    x["f"] = (case["f_mean"] + torch.randn(shape[:3], device=dev, generator=g)).to(dt)
    x["i"] = torch.randn(shape[:3], device=dev, generator=g).to(dt)
    if case["gated"]:
        x["o"] = torch.randn(shape, device=dev, generator=g).to(dt)
    if case["kind"] in ("train", "scantrain"):
        for t in x.values():
            t.requires_grad_(True)
        s["dh"] = torch.randn(shape, device=dev, generator=g)      # h is float32 whatever the inputs are
    if case["kind"] == "segment":
        s["initial"] = _carried_state(case, g, dev)
    s["x"] = x
    return s


def run(state):
    x, kind = state["x"], state["kind"]
    q, k, v, f, i, o = (x.get(n) for n in ("q", "k", "v", "f", "i", "o"))
    if kind == "forward":
        return PKG.mlstm_matmul(q, k, v, f, i)
    if kind == "scan":
        return PKG.mlstm_scan(q, k, v, f, i, o)
    if kind == "long":
        return PKG.mlstm_chunkwise(q, k, v, f, i, _CHUNK)
    if kind == "segment":
        if o is None:
            return PKG.mlstm_chunkwise(q, k, v, f, i, _CHUNK, initial=state["initial"], return_state=True)
        return PKG.mlstm_scan(q, k, v, f, i, o, initial=state["initial"], return_state=True)
    if kind == "train":
        h = PKG.Triton_mLSTM.apply(q, k, v, f, i, 32, 4) if o is None else PKG.Triton_mLSTM.apply(q, k, v, f, i, 32, 4, o)
    else:
        h = PKG.mlstm_scan(q, k, v, f, i, o)
    return (h.detach(),) + torch.autograd.grad(h, list(x.values()), state["dh"])


def work(case):
    B, NH, S, D = case["B"], case["NH"], case["S"], case["D"]
    es, rows = (4 if case["dtype"] == "fp32" else 2), B * NH * S
    grads = case["kind"] in ("train", "scantrain")
    inputs = rows * es * ((4 if case["gated"] else 3) * D + 2)
    nbytes = inputs + rows * 4 * D                                  # h in float32
    if grads:
        nbytes += rows * 4 * D + inputs                             # dh in, gradients of every input out
    if case["kind"] == "segment":
        nbytes += 2 * B * NH * (4 * D * D + 4 * D + 16)             # the state in and out
    # per position: either every earlier position taken directly, or the part inside a block of 256 and the carried
    # state's update and use (two contractions each; the backward adds five to two), whichever is less
    whole = 4 * D * (S + 1) / 2
    carried = 4 * D * (min(S, _CHUNK) + 1) / 2 + 4 * D * D
    per_row = carried if case["kind"] == "segment" else min(whole, carried)
    return {"bytes": float(nbytes), "flops": float(rows * per_row * (3.5 if grads else 1.0))}


def tolerance(case):
    if case["dtype"] == "fp32":
        if case["kind"] == "scan" and case["D"] not in (64, 128):
            return {"rel": 2e-3}      # single tf32 products, the scan entry's default (10 bits of mantissa)
        return {"rel": 1e-4}          # fp32-level products; the gradient of f is a difference of sums over the sequence
    return {"rel": 1e-2}              # 16-bit operands
