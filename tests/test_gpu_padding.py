"""GPU tests of left padding: input gates of -inf in front of a sequence.

A position with an input gate of -inf contributes nothing, and one with no finite gate at or before it sees nothing: its h, its
gradients and its row sum are exactly 0 and its m is -inf.  The positions behind the padding give what the sequence without
it gives (the oracle on the cut sequence), in every form of the forward and the backward, wherever the padding ends:
inside a reference block of the gate vectors (64), a tile (128), a block of the chunkwise form (256) or on their edges.
"""
import importlib

import pytest
import torch

from oracle import mlstm_oracle as orc

pytestmark = pytest.mark.gpu

TOL_F32 = 3e-4
TOL_16 = 1e-2
PKG = "xlstm-triton-cuda-implementation_b200"
NAMES = ("q", "k", "v", "f", "i")


@pytest.fixture(scope="module")
def gc():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from tests import gpu_cases
    return gpu_cases


def _padded(gc, pads, S, D, dtype, seed, slices=None):
    """One slice per entry of ``pads`` (``slices``: as many, the entries in turn), that many gates of -inf in front."""
    n = slices or len(pads)
    x = gc.make_inputs(1, n, S, D, dtype, f_mean=2.0, qkv_scale=D ** -0.5, seed=seed, with_o=True)
    for s in range(n):
        x["i"][0, s, :pads[s % len(pads)]] = -float("inf")
    return x


def _finite(x, pads):
    """The same inputs with gates of -200 in place of -inf and no upstream gradient there: beside a gate of order 1 a weight of
    exp(-200) is 0 in fp32, so what is behind the padding has the same value and, in the same form, the same rounding."""
    y = {n: t.clone() for n, t in x.items()}
    for s in range(x["q"].shape[1]):
        y["i"][0, s, :pads[s % len(pads)]] = -200.0
        y["dh"][0, s, :pads[s % len(pads)]] = 0.0
    return y


def _check(x, pads, run, tol, check_slices=None):
    """``run(x)``: name -> tensor [1, slices, S, ...].  Names: h, m, b and the gradients; gated where there is a ``do``.
    The bound is ``tol`` or, where the form's own rounding at these inputs is larger (df of the chunkwise backward, a running
    sum; tf32 products that cancel in a sequence of one position), the error without infinite gates: padding adds none."""
    got, finite = run(x), run(_finite(x, pads))
    S = x["q"].shape[2]
    gated = "do" in got
    for s in check_slices or range(x["q"].shape[1]):
        pad = pads[s % len(pads)]
        for n, t in got.items():
            front = t[0, s, :pad]
            assert bool(((front == -float("inf")) if n == "m" else (front == 0)).all()), (n, s)
        if pad == S:
            continue
        y = {n: t[:, s:s + 1, pad:] for n, t in x.items()}
        h, m, b, _ = orc.matmul_forward(*(y[n] for n in NAMES), return_state=True)
        ref = dict(h=h, b=b)
        if any(n.startswith("d") for n in got):
            sg = torch.sigmoid(y["o"].double())
            dh = y["dh"].double() * (y["o"].double() * sg if gated else 1.0)
            ref.update(zip(("dq", "dk", "dv", "df", "di"), orc.matmul_backward(dh, *(y[n] for n in NAMES))))
            ref["df"][..., 0] = 0.0
            ref["do"] = y["dh"].double() * h * sg * (1.0 + y["o"].double() * (1.0 - sg))
        for n, t in got.items():
            if n != "m":      # (m counts the forget gates of the padding in: an absolute scale of its own)
                err, own = (orc.max_abs_rel(r[:, s:s + 1, pad:].float(), ref[n]) for r in (t, finite[n]))
                assert err < max(tol, 1.1 * own), (n, s, pad, err, own)


def _parallel(gc, flags, gated):
    def run(x):
        d = [x[n].cuda() for n in NAMES]
        h, m, b = gc.PKG.mlstm_matmul_forward(*d, flags=flags)
        grads = gc.PKG.mlstm_matmul.__globals__["_backward"](x["dh"].cuda(), *d, h, m, b, flags, x["o"].cuda() if gated else None)
        got = dict(zip(("h", "m", "b", "dq", "dk", "dv", "df", "di", "do"), (h, m, b) + grads))
        return got if gated else {n: t for n, t in got.items() if n != "do"}
    return run


@pytest.mark.parametrize("dtype,S,D,flags,gated", [
    (torch.bfloat16, 700, 128, 0, True), (torch.bfloat16, 700, 256, 0, False), (torch.float16, 330, 64, 0, True),
    (torch.bfloat16, 300, 512, 0, True),       # two passes
    (torch.float32, 330, 128, 0, False),       # split bf16 products
    (torch.float32, 330, 256, 4, False),       # tf32
    (torch.float32, 330, 96, 0, True),         # CUDA cores in two stages
    (torch.float32, 330, 96, 1, False),        # and in one
])
def test_parallel_forms(gc, dtype, S, D, flags, gated):
    pads = (0, 1, 63, 64, 100, 129, S - 1, S)
    x = _padded(gc, pads, S, D, dtype, seed=S + D)
    _check(x, pads, _parallel(gc, flags, gated), TOL_16 if dtype != torch.float32 or flags & 4 else TOL_F32)


@pytest.mark.parametrize("D", [128, 256])
def test_chunkwise_form_behind_the_parallel_entry_points(gc, D):
    S, pads = 2050, (0, 1, 100, 256, 300, 640, 2049, 2050)
    x = _padded(gc, pads, S, D, torch.bfloat16, seed=D, slices=64)
    _check(x, pads, _parallel(gc, 0, True), TOL_16, check_slices=range(56, 64))


@pytest.mark.parametrize("chunk", [256, 128])      # 128: an odd number of tiles per block, single CTAs
@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 128), (torch.float16, 256)])
def test_chunkwise_entry_points(gc, dtype, D, chunk):
    """Forward, backward and the state carried out, which goes on through a second call (also when the first was all padding)."""
    S, cut, pads = 900, 520, (0, 1, 100, 256, 300, 520, 899)
    x = _padded(gc, pads, S, D, dtype, seed=D + chunk)

    def whole(x):
        t = {n: x[n].cuda().requires_grad_(True) for n in NAMES}
        h = gc.PKG.mlstm_chunkwise(*(t[n] for n in NAMES), chunk)
        grads = torch.autograd.grad(h, [t[n] for n in NAMES], x["dh"].cuda())
        return dict(zip(("h", "dq", "dk", "dv", "df", "di"), (h.detach(),) + grads))

    def in_two(x):
        part = lambda a, b: [x[n][:, :, a:b].contiguous().cuda() for n in NAMES]
        h1, st1 = gc.PKG.mlstm_chunkwise(*part(0, cut), chunk, return_state=True)
        h2, st2 = gc.PKG.mlstm_chunkwise(*part(cut, S), chunk, initial=st1, return_state=True)
        states.append((st1, st2))
        return dict(h=torch.cat([h1, h2], 2))
    _check(x, pads, whole, TOL_16)
    states = []
    _check(x, pads, in_two, TOL_16)
    st1, st2 = states[0]
    empty = [s for s, pad in enumerate(pads) if pad >= cut]
    assert bool((st1[0][empty] == 0).all()) and bool((st1[1][empty] == 0).all()) and bool((st1[3][empty] == -float("inf")).all())
    assert all(bool(torch.isfinite(s).all()) for s in st2)


@pytest.mark.parametrize("T", [1, 4, 16])
@pytest.mark.parametrize("D", [128, 256])
def test_decoding_step(gc, D, T):
    """T positions at a time from an empty state, through padding of 0 .. 33 positions, all in csrc/step.cu."""
    S, pads = 48, (0, 1, 5, 16, 33, 48)
    x = _padded(gc, pads, S, D, torch.bfloat16, seed=T)
    states = []

    def steps(x):
        st, out = None, []
        for a in range(0, S, T):
            part = [x[n][:, :, a:a + T].contiguous().cuda() for n in NAMES]
            h, st = gc.PKG.mlstm_chunkwise(*part, initial=st, return_state=True)
            out.append(h)
        states.append(st)
        return dict(h=torch.cat(out, 2))
    _check(x, pads, steps, 1e-4)       # exact inputs, fp32 sums of at most 256 terms
    st = states[0]
    assert bool((st[0][-1] == 0).all()) and float(st[3][-1]) == -float("inf")
    assert all(bool(torch.isfinite(s[:-1]).all()) for s in st)
