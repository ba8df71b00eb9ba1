"""GPU parity tests of the parallel (matmul) path, through the C ABI, against the CPU oracle.

Tolerances (max |a-b| / max |b|): 1e-4 forward / 3e-4 gradients for fp32 inputs (the reference computes
IEEE fp32 dots; here the CUDA-core path and, at D = 64 and 128, the split tensor-core form), 1e-2 for
16-bit and tf32 tensor-core math (the reference's own check tolerance, utils.py:4).
"""
import numpy as np
import pytest
import torch

from oracle import mlstm_oracle as orc

pytestmark = pytest.mark.gpu

TOL_F32 = 1e-4
TOL_16 = 1e-2


@pytest.fixture(scope="module")
def gc():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from tests import gpu_cases
    return gpu_cases


@pytest.mark.parametrize("name", ["matmul_s128_d32_f0.npz", "matmul_s192_d64_f3.npz", "matmul_s768_d32_f1.npz"])
def test_fp32_against_reference_golden(gc, golden_dir, name):
    z = np.load(f"{golden_dir}/{name}")
    x = {k: torch.from_numpy(z[k]) for k in ("q", "k", "v", "f", "i", "dh")}
    h, m, b = gc.run_forward(x)
    assert orc.max_abs_rel(h, torch.from_numpy(z["h"])) < TOL_F32
    ok, frac = orc.check(h, torch.from_numpy(z["h"]))
    assert ok, frac
    grads = gc.run_backward(x, h, m, b)
    for key, g in zip(("dq", "dk", "dv", "df", "di"), grads):
        ref = torch.from_numpy(z[key]).clone()
        if key == "df":
            ref[..., 0] = 0.0
            assert float(g[..., 0].abs().max()) == 0.0
        assert orc.max_abs_rel(g, ref) < 2e-4, key


def test_bf16_against_reference_golden_long(gc, golden_dir):
    """S = 1024, D = 128, bf16: the tensor-core forward and backward against the reference's own PyTorch
    forward / backward on the same bf16 values (fixture made by tests/golden/make_golden.py)."""
    from tests.test_oracle import load_long_bf16
    x, ref = load_long_bf16(golden_dir)
    h, m, b = gc.run_forward(x, h_dtype=torch.bfloat16, flags=gc._lib.F_FORCE_TC)
    assert orc.max_abs_rel(h.float(), ref["h"]) < TOL_16
    grads = gc.run_backward(x, h, m, b, flags=gc._lib.F_FORCE_TC)
    for key, g in zip(("dq", "dk", "dv", "df", "di"), grads):
        r = ref[key].clone()
        if key == "df":
            r[..., 0] = 0.0
        assert orc.max_abs_rel(g.float(), r) < TOL_16, key


@pytest.mark.parametrize("B,NH,S,D,f_mean", [
    (1, 4, 2048, 64, 0.0),     # the reference demo / configuration 2
    (2, 3, 200, 40, 3.0),      # ragged S, D not a tile multiple
    (1, 2, 64, 8, -3.0),
    (1, 1, 3, 16, 0.0),        # three steps
])
def test_fp32_simt_forward_backward(gc, B, NH, S, D, f_mean):
    x = gc.make_inputs(B, NH, S, D, torch.float32, f_mean=f_mean, seed=S + D)
    flags = gc._lib.F_FORCE_SIMT
    h, m, b = gc.run_forward(x, flags=flags)
    ef = gc.errors_forward(x, h, m, b)
    assert ef["h"] < TOL_F32 and ef["m"] < 1e-5 and ef["b"] < TOL_F32, ef
    eb = gc.errors_backward(x, gc.run_backward(x, h, m, b, flags=flags), torch.float32)
    assert all(v < 3e-4 for v in eb.values()), eb


@pytest.mark.parametrize("B,NH,S,D,f_mean,scale", [
    (1, 4, 2048, 64, 0.0, 1.0),      # the reference demo / configuration 2, through the default path
    (1, 2, 328, 128, 1.0, 128 ** -0.5),
    (2, 2, 200, 64, 3.0, 1.0),       # ragged S
    (1, 2, 192, 128, -0.5, 1.0),     # strong decay, last 64-position block pure padding
    (1, 1, 1, 64, 0.0, 1.0),         # a single step (forward only, see test_single_step_sequence)
])
def test_fp32_split_tensor_core_forward_backward(gc, B, NH, S, D, f_mean, scale):
    """fp32 inputs at D = 64 / 128 take the tensor cores by default with operands split into two bf16 halves
    (three products per fp32 product): the fp32 tolerances apply, and the elementwise comparator must pass."""
    x = gc.make_inputs(B, NH, S, D, torch.float32, f_mean=f_mean, qkv_scale=scale, seed=S + D)
    assert gc._lib.lib().mlstm_mm_fwd_workspace(B, NH, S, D, 0, 0) > gc._lib.lib().mlstm_mm_fwd_workspace(B, NH, S, D, 0, 8)
    h, m, b = gc.run_forward(x, flags=gc._lib.F_FORCE_TC)
    ef = gc.errors_forward(x, h, m, b)
    assert ef["h"] < TOL_F32 and ef["m"] < 1e-5 and ef["b"] < TOL_F32, ef
    assert ef["h_check_frac"] == 0.0, ef
    if S > 1:
        eb = gc.errors_backward(x, gc.run_backward(x, h, m, b, flags=gc._lib.F_FORCE_TC), torch.float32)
        assert all(v < 3e-4 for k, v in eb.items() if k != "check_frac"), eb
        assert eb["check_frac"] == 0.0, eb


def test_single_step_sequence(gc):
    """S = 1.  Forward must match; the backward of a lone step is a difference of two terms that agree
    to about 1e-6 relative (dC/n + db = dC/n * (1 - |b|/n)), so only its structure is checked."""
    x = gc.make_inputs(1, 1, 1, 16, torch.float32, seed=17)
    h, m, b = gc.run_forward(x)
    ef = gc.errors_forward(x, h, m, b)
    assert ef["h"] < TOL_F32 and ef["b"] < TOL_F32, ef
    dq, dk, dv, df, di = gc.run_backward(x, h, m, b)
    assert all(bool(torch.isfinite(t).all()) for t in (dq, dk, dv, df, di))
    assert float(df.abs().max()) == 0.0
    assert orc.max_abs_rel(dv, gc.oracle_backward(x, torch.float32)[2]) < TOL_F32


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("S,f_mean", [(128, 0.0), (512, 3.0), (328, 0.0)])
def test_tensor_core_forward_backward(gc, dtype, D, S, f_mean):
    x = gc.make_inputs(1, 3, S, D, dtype, f_mean=f_mean, qkv_scale=D ** -0.5, seed=D + S)
    flags = gc._lib.F_FORCE_TC
    for h_dtype in (torch.float32, dtype):
        h, m, b = gc.run_forward(x, h_dtype=h_dtype, flags=flags)
        ef = gc.errors_forward(x, h, m, b)
        assert ef["h"] < TOL_16 and ef["m"] < 1e-5 and ef["b"] < TOL_16, (h_dtype, ef)
        assert ef["h_check_frac"] < gc.CHECK_FRAC_16 and ef["h_first_tile_row_rel"] < gc.ROW_REL_16, (h_dtype, ef)
        eb = gc.errors_backward(x, gc.run_backward(x, h, m, b, flags=flags), h_dtype)
        assert all(v < TOL_16 for v in eb.values()), (h_dtype, eb)


@pytest.mark.parametrize("dtype,D,S", [(torch.float16, 64, 192), (torch.bfloat16, 128, 192), (torch.float16, 256, 320),
                                       (torch.bfloat16, 256, 448)])
def test_strong_decay_with_a_fully_padded_column_block(gc, dtype, D, S):
    """Ragged S whose last 128-row tile ends in a 64-position block of pure padding, with forget gates around
    sigmoid(-0.5): the row term of the exponent alone reaches 2^140 for late keys, and the padded block has no
    reference to balance it.  Its columns weigh 0; the product must be 0, not NaN (regression)."""
    x = gc.make_inputs(1, 2, S, D, dtype, f_mean=-0.5, qkv_scale=D ** -0.5, seed=S + D)
    flags = gc._lib.F_FORCE_TC
    h, m, b = gc.run_forward(x, h_dtype=dtype, flags=flags)
    ef = gc.errors_forward(x, h, m, b)
    assert ef["h"] < TOL_16 and ef["b"] < TOL_16, ef
    assert ef["h_check_frac"] < gc.CHECK_FRAC_16 and ef["h_first_tile_row_rel"] < gc.ROW_REL_16, ef
    grads = gc.run_backward(x, h, m, b, flags=flags)
    assert all(bool(torch.isfinite(t.float()).all()) for t in grads)
    eb = gc.errors_backward(x, grads, dtype)
    assert all(v < TOL_16 for v in eb.values()), eb


@pytest.mark.parametrize("D", [64, 128, 256])
def test_tf32_tensor_core_forward_backward(gc, D):
    """fp32 inputs on the tensor cores (tf32 operands, fp32 accumulate), opt-in by flag."""
    x = gc.make_inputs(1, 2, 328, D, torch.float32, f_mean=1.0, qkv_scale=D ** -0.5, seed=D)
    flags = gc._lib.F_FORCE_TC | gc._lib.F_ALLOW_TF32
    h, m, b = gc.run_forward(x, flags=flags)
    ef = gc.errors_forward(x, h, m, b)
    # tf32 keeps 10 mantissa bits of every operand: about 1e-3 on h, 1e-3 .. 5e-3 on gradients (measured)
    assert ef["h"] < 3e-3 and ef["m"] < 1e-5 and ef["b"] < 3e-3, ef
    eb = gc.errors_backward(x, gc.run_backward(x, h, m, b, flags=flags), torch.float32)
    assert all(v < TOL_16 for v in eb.values()), eb


@pytest.mark.parametrize("dtype,D,S,f_mean", [
    (torch.bfloat16, 512, 400, 2.0),      # ragged: three full row tiles and a bit
    (torch.float16, 768, 128, 0.0),
    (torch.float32, 512, 300, 1.0),       # tf32 operands (by flag); an odd number of row tiles
    (torch.bfloat16, 512, 1300, 3.0),     # eleven row tiles
])
def test_head_dimensions_above_256_take_the_two_pass_form(gc, dtype, D, S, f_mean):
    """The parallel forward (float32 h) and backward at D = 512, 768: gated S x S matrices to scratch, then plain
    contractions, on the tensor cores; h, m, b and the five gradients against the oracle.  The workspace query
    says which form a call gets: the two-pass one needs room for the gated matrices."""
    x = gc.make_inputs(1, 2, S, D, dtype, f_mean=f_mean, qkv_scale=D ** -0.5, seed=D + S)
    flags = gc._lib.F_ALLOW_TF32 if dtype == torch.float32 else 0
    L = gc._lib.lib()
    dt = gc._lib.dtype_code(x["q"])
    Spad = (S + 127) // 128 * 128
    es = 4 if dtype == torch.float32 else 2
    assert L.mlstm_mm_fwd_workspace(1, 2, S, D, dt, flags) >= 2 * Spad * Spad * es
    assert L.mlstm_mm_fwd_workspace(1, 2, S, D, dt, flags | gc._lib.F_FORCE_SIMT) < Spad * Spad * es
    h, m, b = gc.run_forward(x, flags=flags)
    ef = gc.errors_forward(x, h, m, b)
    tol = 3e-3 if dtype == torch.float32 else TOL_16
    assert ef["h"] < tol and ef["m"] < 1e-5 and ef["b"] < tol, ef
    assert ef["h_check_frac"] < gc.CHECK_FRAC_16 and ef["h_first_tile_row_rel"] < gc.ROW_REL_16, ef
    # the same call on the CUDA cores agrees
    h2, m2, b2 = gc.run_forward(x, flags=gc._lib.F_FORCE_SIMT)
    assert orc.max_abs_rel(h, h2) < tol and orc.max_abs_rel(b, b2) < tol and torch.equal(m, m2)
    assert L.mlstm_mm_bwd_workspace(1, 2, S, D, dt, gc._lib.dtype_code(h), flags) >= 4 * Spad * Spad * es
    grads = gc.run_backward(x, h, m, b, flags=flags)
    eb = gc.errors_backward(x, grads, torch.float32)
    assert all(v < TOL_16 for v in eb.values()), eb
    # the CUDA-core backward of the same call agrees
    grads2 = gc.run_backward(x, h, m, b, flags=gc._lib.F_FORCE_SIMT)
    for name, g1, g2 in zip(("dq", "dk", "dv", "df", "di"), grads, grads2):
        assert orc.max_abs_rel(g1, g2) < TOL_16, name


def test_two_pass_form_in_slice_groups(gc):
    """Nine slices at S = 4096, D = 512: the backward keeps two gated matrices per slice (64 MB here), so it runs in
    two groups of slices (eight, then one) through the same scratch, the forward in one.  Slices of both groups agree
    with the same slice computed alone."""
    B, NH, S, D = 1, 9, 4096, 512
    x = gc.make_inputs(B, NH, S, D, torch.bfloat16, f_mean=3.0, qkv_scale=D ** -0.5, seed=99)
    L = gc._lib.lib()
    dt = gc._lib.dtype_code(x["q"])
    assert L.mlstm_mm_bwd_workspace(B, NH, S, D, dt, 0, 0) < 700 << 20     # two matrices of eight slices, not of nine
    h, m, b = gc.run_forward(x)
    grads = gc.run_backward(x, h, m, b)
    for hd in (0, 7, 8):
        one = {n: t[:, hd:hd + 1].contiguous() for n, t in x.items()}
        h1, m1, b1 = gc.run_forward(one)
        assert orc.max_abs_rel(h[:, hd:hd + 1], h1) < 1e-6 and orc.max_abs_rel(b[:, hd:hd + 1], b1) < 1e-6
        for name, g_all, g_one in zip(("dq", "dk", "dv", "df", "di"), grads, gc.run_backward(one, h1, m1, b1)):
            assert orc.max_abs_rel(g_all[:, hd:hd + 1], g_one) < 1e-6, (hd, name)
    # and one slice of the second group against the oracle
    one = {n: t[:, 8:9].contiguous() for n, t in x.items()}
    eb = gc.errors_backward(one, [g[:, 8:9] for g in grads], torch.float32)
    assert all(v < TOL_16 for v in eb.values()), eb


def test_calls_back_to_back_on_one_workspace(gc):
    """Forty forward + backward calls enqueued without a synchronize, alternating two input sets, all through the same
    cached workspace: a call's first kernel clears the status block and the passes are launched programmatically (they
    may start under the tail of the kernel before them), so this is where a missing dependency would show.  The
    results of the last two calls must equal those of the same calls made alone."""
    dev = torch.device("cuda", 0)
    sets = []
    for seed in (1, 2):
        x = gc.make_inputs(2, 3, 384, 128, torch.bfloat16, f_mean=2.0, qkv_scale=128 ** -0.5, seed=seed)
        sets.append({n: t.to(dev) for n, t in x.items()})
    def call(d):
        h, m, b = gc.PKG.mlstm_matmul_forward(d["q"], d["k"], d["v"], d["f"], d["i"])
        return (h, m, b) + tuple(gc.PKG.mlstm_matmul_backward(d["dh"], d["q"], d["k"], d["v"], d["f"], d["i"], h, m, b))
    alone = []
    for d in sets:
        out = call(d)
        torch.cuda.synchronize()
        alone.append([t.clone() for t in out])
    last = [None, None]
    for it in range(40):
        last[it & 1] = call(sets[it & 1])
    torch.cuda.synchronize()
    for k in range(2):
        for a, b in zip(last[k], alone[k]):
            assert torch.equal(a, b)


def test_tensor_core_matches_simt_on_device(gc):
    """Same 16-bit inputs through both kernel families."""
    x = gc.make_inputs(2, 2, 640, 128, torch.bfloat16, f_mean=3.0, qkv_scale=128 ** -0.5, seed=3)
    h1, m1, b1 = gc.run_forward(x, flags=gc._lib.F_FORCE_TC)
    h2, m2, b2 = gc.run_forward(x, flags=gc._lib.F_FORCE_SIMT)
    assert orc.max_abs_rel(h1, h2) < TOL_16
    assert torch.equal(m1, m2)
    g1 = gc.run_backward(x, h2, m2, b2, flags=gc._lib.F_FORCE_TC)
    g2 = gc.run_backward(x, h2, m2, b2, flags=gc._lib.F_FORCE_SIMT)
    for a, b_ in zip(g1, g2):
        assert orc.max_abs_rel(a.float(), b_.float()) < TOL_16


def test_autograd_function_matches_reference_api(gc):
    """Triton_mLSTM.apply(q,k,v,f,i,SB,NUM_WARPS) + h.backward(dh), as the reference demo does."""
    x = gc.make_inputs(1, 2, 256, 64, torch.float32, seed=11)
    dev = torch.device("cuda", 0)
    t = {n: x[n].to(dev).requires_grad_(True) for n in ("q", "k", "v", "f", "i")}
    h = gc.PKG.Triton_mLSTM.apply(t["q"], t["k"], t["v"], t["f"], t["i"], 32, 4)
    assert h.dtype == torch.float32
    h.backward(x["dh"].to(dev))
    ref = gc.oracle_backward(x, torch.float32)
    for n, r in zip(("q", "k", "v", "f", "i"), ref):
        assert t[n].grad.dtype == t[n].dtype
        assert orc.max_abs_rel(t[n].grad, r) < 3e-4, n
    h2 = gc.PKG.mlstm_matmul(*(t[n].detach() for n in ("q", "k", "v", "f", "i")), SB=32, num_warps=4)
    assert torch.equal(h2, h.detach())


@pytest.mark.parametrize("dtype,D", [(torch.float32, 64), (torch.bfloat16, 256)])
def test_autograd_function_with_output_gate(gc, dtype, D):
    """The optional eighth argument o of Triton_mLSTM.apply: h * silu(o), and gradients for all six inputs."""
    x = gc.make_inputs(1, 2, 256, D, dtype, f_mean=1.0, qkv_scale=D ** -0.5, seed=D + 5, with_o=True)
    dev = torch.device("cuda", 0)
    names = ("q", "k", "v", "f", "i", "o")
    t = {n: x[n].to(dev).requires_grad_(True) for n in names}
    h = gc.PKG.Triton_mLSTM.apply(t["q"], t["k"], t["v"], t["f"], t["i"], 32, 4, t["o"])
    assert h.dtype == torch.float32
    h.backward(x["dh"].to(dev))
    # reference: the oracle's forward and closed-form backward around the gate's own derivative
    od = x["o"].double()
    sig = torch.sigmoid(od)
    h_inner = orc.matmul_forward(x["q"], x["k"], x["v"], x["f"], x["i"], dtype=torch.float64)
    dhd = x["dh"].double()
    ref = dict(zip(("q", "k", "v", "f", "i"), orc.matmul_backward(dhd * od * sig, x["q"], x["k"], x["v"], x["f"], x["i"])))
    ref["o"] = dhd * h_inner * sig * (1 + od * (1 - sig))
    tol = 3e-4 if dtype == torch.float32 else TOL_16
    assert orc.max_abs_rel(h.detach(), h_inner * od * sig) < tol
    for n in names:
        assert t[n].grad.dtype == t[n].dtype
        assert orc.max_abs_rel(t[n].grad, ref[n]) < tol, n
    with pytest.raises(ValueError):
        gc.PKG.Triton_mLSTM.apply(t["q"], t["k"], t["v"], t["f"], t["i"], 32, 4, t["o"][..., :8])


@pytest.mark.parametrize("which", ["dh", "o"])
@pytest.mark.parametrize("entry,S,D,dtype", [
    ("matmul", 130, 64, torch.float32), ("matmul", 256, 128, torch.bfloat16),
    ("scan", 256, 128, torch.float16),       # the parallel kernels behind mlstm_scan
    ("scan", 1280, 128, torch.bfloat16),     # the chunkwise backward
])
def test_gated_backward_takes_unaligned_gradients(gc, entry, S, D, dtype, which):
    """A contiguous upstream gradient (or o) that starts one element behind a 16-byte boundary, as a view into a flat buffer
    does: the same gradients as from an aligned one.  The gate's derivative then has a kernel of its own, with the same fp32
    arithmetic up to the order of its products: a rounding of the gradients' type apart (bf16: 2^-8)."""
    x = gc.make_inputs(1, 2, S, D, dtype, f_mean=2.0, qkv_scale=D ** -0.5, seed=S, with_o=True)
    names = ("q", "k", "v", "f", "i", "o")

    def run(off):
        def place(t, shift):
            buf = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
            view = buf[shift:shift + t.numel()].view(t.shape)
            view.copy_(t)
            assert view.is_contiguous() and (view.data_ptr() % 16 != 0) == (shift != 0)
            return view
        t = {n: place(x[n], off if n == which else 0).requires_grad_(True) for n in names}
        if entry == "matmul":
            h = gc.PKG.Triton_mLSTM.apply(*(t[n] for n in names[:5]), 32, 4, t["o"])
        else:
            h = gc.PKG.mlstm_scan(*(t[n] for n in names))
        return torch.autograd.grad(h, [t[n] for n in names], place(x["dh"], off if which == "dh" else 0))

    tol = 1e-5 if dtype == torch.float32 else 2.0 ** -8
    for n, a, r in zip(names, run(1), run(0)):
        assert orc.max_abs_rel(a.float(), r.float().cpu()) < tol, n


@pytest.mark.parametrize("f_mean", [3.0, 0.0])
def test_model_scale_slice_properties(gc, f_mean):
    """Configuration-4 shape per slice (S=4096, D=256, bf16) on a few slices, with retention-biased gates
    (the configuration's own) and with N(0,1) gates: oracle parity on one slice, and slice independence
    (each slice equals the same slice run alone)."""
    x = gc.make_inputs(1, 3, 4096, 256, torch.bfloat16, f_mean=f_mean, qkv_scale=256 ** -0.5, seed=0)
    h, m, b = gc.run_forward(x, h_dtype=torch.bfloat16)
    grads = gc.run_backward(x, h, m, b)
    one = {k: v[:, 1:2].contiguous() for k, v in x.items()}
    h1, m1, b1 = gc.run_forward(one, h_dtype=torch.bfloat16)
    assert torch.equal(h1, h[:, 1:2])
    g1 = gc.run_backward(one, h1, m1, b1)
    for a, b_ in zip(g1, grads):
        assert torch.equal(a, b_[:, 1:2])
    ef = gc.errors_forward(one, h1, m1, b1)
    assert ef["h"] < TOL_16, ef
    assert ef["h_check_frac"] < gc.CHECK_FRAC_16, ef
    eb = gc.errors_backward(one, g1, torch.bfloat16)
    assert all(v < TOL_16 for v in eb.values()), eb


def test_bounded_wait_runs_out_and_the_device_stays_usable(gc):
    """The waits of every kernel are bounded; this makes one run out on purpose, the allowed way: a warp waits
    (limit: two million cycles, about a millisecond) on a barrier that nothing completes, then stores a code in the
    status word.  mlstm_read_status must report MLSTM_E_TIMEOUT with that code, and ordinary work must still pass."""
    import ctypes
    L = gc._lib.lib()
    dev = torch.device("cuda", 0)
    ws = torch.zeros(4096, dtype=torch.uint8, device=dev)
    stream = gc._lib.stream_ptr(dev)
    assert L.mlstm_selftest_wait_timeout(ws.data_ptr(), ws.numel(), 2_000_000, stream) == 0
    code = ctypes.c_int(0)
    assert L.mlstm_read_status(ws.data_ptr(), ctypes.byref(code), stream) == -7   # MLSTM_E_TIMEOUT
    assert code.value == 4000
    assert b"gave up" in L.mlstm_status_string(-7)
    assert L.mlstm_selftest_wait_timeout(ws.data_ptr(), 16, 2_000_000, stream) == -5
    assert L.mlstm_selftest_wait_timeout(ws.data_ptr(), ws.numel(), 0, stream) == -1
    # the context is intact: an ordinary call on the same device passes and reports a clean status
    x = gc.make_inputs(1, 2, 256, 64, torch.bfloat16, f_mean=1.0, qkv_scale=0.125, seed=2)
    h, m, b = gc.run_forward(x, flags=gc._lib.F_FORCE_TC)
    ef = gc.errors_forward(x, h, m, b)
    assert ef["h"] < TOL_16, ef


def test_argument_errors(gc):
    L = gc._lib.lib()
    assert L.mlstm_mm_fwd(None, None, None, None, None, None, None, None, None, 0, 1, 1, 8, 8, 0, 0, 0, None) == -1
    x = gc.make_inputs(1, 1, 64, 12, torch.float32)
    with pytest.raises(gc._lib.MlstmError):
        gc.run_forward(x)  # D not a multiple of 8
    x = gc.make_inputs(1, 1, 64, 32, torch.float32)
    with pytest.raises(gc._lib.MlstmError):
        gc.run_forward(x, flags=gc._lib.F_FORCE_TC)  # fp32 at D = 32 has no tensor-core path


@pytest.mark.parametrize("BH,S,D,gated,pad", [
    (64, 2048, 128, False, 0),      # the smallest that takes the chunkwise form
    (33, 4001, 256, True, 0),       # ragged last block, an odd number of tiles
    (66, 2049, 128, False, 640),    # one position in the last block; input gates of -inf in front (left padding)
])
def test_long_sequences_take_the_chunkwise_form(gc, BH, S, D, gated, pad):
    """The parallel entry points' chunkwise route against the oracle (first and last slice) and against the quadratic kernel,
    whose error it may not exceed by more than the noise of the measure (a quarter)."""
    dt = torch.bfloat16
    x = gc.make_inputs(1, BH, S, D, dt, f_mean=3.0, qkv_scale=D ** -0.5, seed=S, with_o=gated)
    if pad:
        x["i"][:, :, :pad] = -float("inf")
    dev = {n: t.cuda() for n, t in x.items()}
    args = [dev[n] for n in ("q", "k", "v", "f", "i")]
    res = []
    for flags in (0, gc._lib.F_FORCE_TC):
        h, m, b = gc.PKG.mlstm_matmul_forward(*args, flags=flags)
        if pad:
            h[:, :, :pad] = 0.0          # rows without a finite gate have no value
            dev["dh"][:, :, :pad] = 0.0
        gr = None if pad else gc.PKG.mlstm_matmul.__globals__["_backward"](dev["dh"], *args, h, m, b, flags, dev.get("o"))
        res.append((h, m, b, gr))
    (h, m, b, gr), (h2, m2, b2, gr2) = res
    for sl in (0, BH - 1):
        y = {n: t[:, sl:sl + 1, pad:] for n, t in x.items()}
        ref, _, b_ref, _ = orc.matmul_forward(y["q"], y["k"], y["v"], y["f"], y["i"], return_state=True)
        err = lambda t, r: float((t.double().cpu() - r).norm() / r.norm())
        cut = lambda t: t[:, sl:sl + 1, pad:]
        assert err(cut(h), ref) < 1.25 * err(cut(h2), ref)
        if gr is None:
            continue
        sg = torch.sigmoid(y["o"].double()) if gated else None
        dh = y["dh"].double() * (y["o"].double() * sg if gated else 1.0)
        refs = list(orc.matmul_backward(dh, y["q"], y["k"], y["v"], y["f"], y["i"]))
        refs[3][..., 0] = 0.0
        if gated:
            refs.append(y["dh"].double() * ref * sg * (1.0 + y["o"].double() * (1.0 - sg)))
        for name, a, a2, r in zip(("dq", "dk", "dv", "df", "di", "do"), gr, gr2, refs):
            assert err(cut(a), r) < 1.25 * err(cut(a2), r), name


def test_chunkwise_route_without_room_for_its_states(gc):
    """With less memory than the block states need (the process' share is cut for the call) the parallel entry points run the
    quadratic kernels: what MLSTM_F_FORCE_TC gives, bit for bit."""
    B, NH, S, D = 1, 64, 2048, 256                       # states: 128 MB forward, 256 MB backward; scratch without: 1.5 and 69 MB
    x = gc.make_inputs(B, NH, S, D, torch.bfloat16, f_mean=3.0, qkv_scale=D ** -0.5, seed=9)
    d, dh = [x[n].cuda() for n in ("q", "k", "v", "f", "i")], x["dh"].cuda()

    forward = lambda flags: gc.PKG.mlstm_matmul_forward(*d, flags=flags)
    want = forward(gc._lib.F_FORCE_TC)
    backward = lambda flags: gc.PKG.mlstm_matmul_backward(dh, *d, *want, flags=flags)
    want_grads = backward(gc._lib.F_FORCE_TC)
    assert not torch.equal(want[0], forward(0)[0])       # (another order of summation)
    assert gc._lib.lib().mlstm_tc_supported(S, D, 2) == 1

    def limited(fn, scratch):
        """fn with room for its results and ``scratch`` bytes beside them"""
        gc._lib._WS_CACHE.clear()
        torch.cuda.empty_cache()
        results = sum(t.numel() * t.element_size() for t in (want if fn is forward else want_grads))
        room = torch.cuda.memory_reserved() + results + scratch
        torch.cuda.set_per_process_memory_fraction(room / torch.cuda.get_device_properties(0).total_memory)
        try:
            return fn(0)
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
    for fn, scratch, ref in ((forward, 64 << 20, want), (backward, 160 << 20, want_grads)):
        for a, r in zip(limited(fn, scratch), ref):
            assert torch.equal(a, r)


def test_chunkwise_route_in_slice_groups(gc):
    """More states than a set may hold (1 GB or 74 slices at D = 256): the slices go in two groups of 80.  A slice's results
    do not depend on the slices beside it: both groups equal the same slices called on their own, in one group each."""
    BH, S, D, cut = 160, 7100, 256, 80
    g = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *shape: torch.randn(shape, device="cuda", generator=g)
    q, k, v, o = ((rnd(1, BH, S, D) * s).bfloat16() for s in (D ** -0.5, D ** -0.5, D ** -0.5, 1.0))
    f, i, dh = (3.0 + rnd(1, BH, S)).bfloat16(), rnd(1, BH, S).bfloat16(), rnd(1, BH, S, D)
    backward = gc.PKG.mlstm_matmul.__globals__["_backward"]

    def run(sl):
        x = [t[:, sl].contiguous() for t in (q, k, v, f, i)]
        h, m, b = gc.PKG.mlstm_matmul_forward(*x)
        return (h, m, b) + backward(dh[:, sl].contiguous(), *x, h, m, b, 0, o[:, sl].contiguous())
    whole = run(slice(0, BH))
    for sl in (slice(0, cut), slice(cut, BH)):
        for a, part in zip(whole, run(sl)):
            assert torch.equal(a[:, sl], part)


@pytest.mark.parametrize("B,NH,S,D,dtype", [
    (1, 2, 64, 8, torch.float32),          # one tile
    (2, 1, 65, 32, torch.float32),         # a tile and one row
    (1, 3, 200, 72, torch.float32),        # a partial column tile
    (1, 2, 321, 256, torch.float32),
    (1, 2, 130, 96, torch.float16),
    (1, 2, 8190, 8, torch.float32),        # the longest: slices in groups of one
])
def test_cuda_core_arithmetic_in_two_stages(gc, B, NH, S, D, dtype):
    """Head dimensions outside the tensor-core set: against the one-stage kernel (the same fp32 products, added up in another
    order: sums of S terms, S * 2^-24 of the largest at worst) and, where it is quick, the oracle."""
    x = gc.make_inputs(B, NH, S, D, dtype, f_mean=1.0, qkv_scale=D ** -0.5, seed=S + D, with_o=True)
    h, m, b = gc.run_forward(x)
    h1, m1, b1 = gc.run_forward(x, flags=gc._lib.F_FORCE_SIMT)
    tol = TOL_F32 if dtype == torch.float32 else 1e-3     # 16 bits: the gradients are rounded to 2^-11
    assert orc.max_abs_rel(h, h1.cpu()) < TOL_F32
    assert orc.max_abs_rel(b, b1.cpu()) < TOL_F32
    assert torch.equal(m, m1)
    g, g1 = gc.run_backward(x, h, m, b), gc.run_backward(x, h1, m1, b1, flags=gc._lib.F_FORCE_SIMT)
    for name, a, r in zip(("dq", "dk", "dv", "df", "di"), g, g1):
        assert orc.max_abs_rel(a, r.cpu()) < 3 * tol, name
    o = x["o"].cuda()
    scan = gc.PKG.mlstm_scan(*(x[n].cuda() for n in ("q", "k", "v", "f", "i")), o, 1, 1, allow_tf32=False)
    assert orc.max_abs_rel(scan, (h * torch.nn.functional.silu(o.float())).cpu()) < tol
    if S <= 400:
        assert orc.max_abs_rel(h, gc.oracle_forward(x)[0]) < TOL_F32
        for name, a, r in zip(("dq", "dk", "dv", "df", "di"), g, gc.oracle_backward(x, torch.float32)):
            assert orc.max_abs_rel(a, r) < 3 * tol, name


@pytest.mark.parametrize("D,S,f_mean", [(32, 384, 1.0), (96, 320, 1.0), (256, 384, 1.0), (32, 640, 0.0)])
def test_two_stages_are_no_farther_from_64_bits_than_one(gc, D, S, f_mean):
    """Strong decay makes row and column parts of an exponent tens where their sum is of order 1.  The two-stage form adds them
    with the rests of their rounding: its errors (2-norm, against the fp64 oracle, 16 slices) are below the one-stage
    kernel's, up to a tenth for what is left to chance in sums of the same length."""
    x = gc.make_inputs(2, 8, S, D, torch.float32, f_mean=f_mean, qkv_scale=D ** -0.5, seed=D + S)
    ref = (gc.oracle_forward(x)[0],) + tuple(gc.oracle_backward(x, torch.float32))
    errs = []
    for flags in (0, gc._lib.F_FORCE_SIMT):
        h, m, b = gc.run_forward(x, flags=flags)
        got = (h,) + tuple(gc.run_backward(x, h, m, b, flags=flags))
        errs.append([float((g.double().cpu() - r).norm() / r.norm()) for g, r in zip(got, ref)])
    for name, two, one in zip(("h", "dq", "dk", "dv", "df", "di"), *errs):
        if name != "df":      # (a running sum: its error is a random walk, and of either size)
            assert two < 1.1 * one, (name, two, one)
