"""The tcgen05 grouped GEMM kernels (bf16/fp16, feature sizes that are multiples of 64 and >= 256)
against fp32 matmuls and against the FFMA kernels on the same inputs."""
import ctypes
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fc():
    from fastermoe_b200 import fmoe_cuda
    return fmoe_cuda


@pytest.fixture(autouse=True)
def _default_form(fc):
    """Every test starts and ends with the library's own choice of GEMM kernels."""
    fc.set_gemm_form("auto")
    yield
    fc.set_gemm_form("auto")


def device_status():
    from fastermoe_b200 import _lib
    v = ctypes.c_int32(-1)
    assert _lib.lib.fmoe_device_status(ctypes.byref(v)) == 0
    return v.value


def reference(x, counts, w, b, gy, act=None):
    x, w, gy = x.float(), w.float(), gy.float()
    y = torch.zeros(x.shape[0], w.shape[1], device=x.device)
    gx, gw = torch.zeros_like(x), torch.zeros_like(w)
    gb = torch.zeros(w.shape[0], w.shape[1], device=x.device)
    p = 0
    for e, c in enumerate(counts):
        s = slice(p, p + c)
        y[s] = x[s] @ w[e].t() + (b[e].float() if b is not None else 0)
        gx[s] = gy[s] @ w[e]
        gw[e] = gy[s].t() @ x[s]
        gb[e] = gy[s].sum(0)
        p += c
    return y, gx, gw, gb


def close(got, want):
    """16-bit result against the fp32 product of the same 16-bit inputs.  Accumulation is fp32 on both
    sides, so what separates them is one rounding of the output: relative 2^-9 for bf16.  rtol 2e-2 is
    the bound the layer is specified to; the absolute floor (four such roundings of a typical element)
    only covers entries that cancel to almost nothing."""
    want = want.float()
    rms = float(want.pow(2).mean().sqrt()) if want.numel() else 0.0
    torch.testing.assert_close(got.float(), want, rtol=2e-2, atol=4 * 2.0 ** -9 * rms)


CASES = [
    ([128], 256, 256),
    ([1], 256, 256),
    ([100, 0, 0, 29], 256, 320),
    ([300, 0, 77], 512, 256),
    ([257, 511, 64, 128], 1024, 512),
    ([700, 900], 256, 1024),
    ([63, 65, 127, 129, 191, 193, 1, 0], 320, 576),
    ([0, 0, 0, 0], 256, 256),
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("counts,fin,fout", CASES)
@pytest.mark.parametrize("bias", [True, False])
def test_tc_against_fp32(fc, dtype, counts, fin, fout, bias):
    torch.manual_seed(sum(counts) + fin + fout)
    E, B = len(counts), sum(counts)
    pad = 5  # rows past the last segment hold NaNs: they must never reach an output
    x = torch.full((B + pad, fin), float("nan"), device="cuda", dtype=dtype)
    gy = torch.full((B + pad, fout), float("nan"), device="cuda", dtype=dtype)
    x[:B] = torch.randn(B, fin, device="cuda").to(dtype)
    gy[:B] = torch.randn(B, fout, device="cuda").to(dtype)
    w = ((torch.rand(E, fout, fin, device="cuda") * 2 - 1) / np.sqrt(fin)).to(dtype)
    b = ((torch.rand(E, fout, device="cuda") * 2 - 1) / np.sqrt(fin)).to(dtype) if bias else None
    cnt = torch.tensor(counts, dtype=torch.int64)
    y = fc.linear_forward(x, cnt, w, b)
    gx, gw, gb = fc.linear_backward(gy, x, cnt, w, b)
    wy, wgx, wgw, wgb = reference(x[:B], counts, w, b, gy[:B])
    assert device_status() == 0
    if B:
        close(y[:B], wy)
        close(gx[:B], wgx)
    close(gw, wgw)
    close(gb, wgb)
    assert torch.isfinite(gw.float()).all() and torch.isfinite(gb.float()).all()


@pytest.mark.parametrize("act", ["relu", "gelu"])
def test_tc_fused_epilogues_match_ffma(fc, act):
    """Bias + activation (forward) and activation backward (input gradient) in the tensor-core
    epilogues against the FFMA kernels, which apply the same formulas in fp32."""
    from fastermoe_b200 import _lib
    torch.manual_seed(1)
    counts, d, h = [300, 0, 157, 431], 256, 512
    E, B = len(counts), sum(counts)
    off = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int64, device="cuda")
    x = torch.randn(B, d, device="cuda").bfloat16()
    w1 = ((torch.rand(E, h, d, device="cuda") * 2 - 1) / np.sqrt(d)).bfloat16()
    b1 = ((torch.rand(E, h, device="cuda") * 2 - 1) / np.sqrt(d)).bfloat16()
    gh = torch.randn(B, h, device="cuda").bfloat16()
    code = {"relu": _lib.ACT_RELU, "gelu": _lib.ACT_GELU}[act]

    def both():
        # the derivative buffer is only written for GELU (ReLU's backward reads the output)
        y, pre = fc.linear_forward_act(x, off, w1, b1, code, want_pre=(act == "gelu"))
        if pre is None:
            pre = torch.zeros(1, device="cuda")
        # backward of a layer whose input came from an activation: a saved buffer of x's shape
        # (ReLU: the activation output, only its sign matters; GELU: the saved derivative)
        pre_in = torch.randn(B, d, device="cuda").bfloat16()
        torch.manual_seed(5)
        gx, gw, gb = fc.linear_backward_act(gh, x, off, w1, pre_in, code)
        return y, pre, gx, gw, gb

    torch.manual_seed(7)
    tc = both()
    fc.set_gemm_form("simt")
    torch.manual_seed(7)
    ff = both()
    fc.set_gemm_form("auto")
    for name, a, b_ in zip(["y", "pre", "gx", "gw", "gb"], tc, ff):
        # both sides round to bf16: they may differ by one unit in the last place of either
        rms = float(b_.float().pow(2).mean().sqrt())
        torch.testing.assert_close(a.float(), b_.float(), rtol=2e-2, atol=8 * 2.0 ** -9 * rms, msg=lambda m, n=name: f"{n}: {m}")
    assert device_status() == 0


def test_tc_accumulate_weight_gradient(fc):
    from fastermoe_b200 import _lib
    torch.manual_seed(2)
    counts, d, h = [200, 312], 256, 256
    off = torch.tensor([0, 200, 512], dtype=torch.int64, device="cuda")
    x = torch.randn(512, d, device="cuda").bfloat16()
    gy = torch.randn(512, h, device="cuda").bfloat16()
    w = torch.randn(2, h, d, device="cuda").bfloat16()
    gw0 = torch.randn(2, h, d, device="cuda").bfloat16()
    gb0 = torch.randn(2, h, device="cuda").bfloat16()
    _, gw, gb = fc.linear_backward_act(gy, x, off, w, None, _lib.ACT_NONE, grad_w=gw0.clone(), grad_b=gb0.clone(),
                                       accumulate=True)
    _, _, wgw, wgb = reference(x, counts, w, None, gy)
    close(gw, wgw + gw0.float())
    close(gb, wgb + gb0.float())


def test_benchmark_shapes_against_fp32(fc):
    """All six products of the benchmark layer (16384 tokens x top-2 = 32768 rows over 16 experts,
    d_model 1024, d_hidden 4096, bf16; the sizes at which the library picks the CTA-pair kernels)
    against fp32 matmuls of the same bf16 inputs, including the fused bias + GELU epilogue, the
    saved-derivative input gradient and the column sums that give the first layer's bias gradient."""
    from fastermoe_b200 import _lib
    torch.manual_seed(3)
    E, d, h, B = 16, 1024, 4096, 32768
    counts = np.random.default_rng(0).multinomial(B, np.ones(E) / E)
    off = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int64, device="cuda")
    bf = torch.bfloat16
    x = torch.randn(B, d, device="cuda").to(bf)
    w1 = ((torch.rand(E, h, d, device="cuda") * 2 - 1) / np.sqrt(d)).to(bf)
    b1 = ((torch.rand(E, h, device="cuda") * 2 - 1) / np.sqrt(d)).to(bf)
    w2 = ((torch.rand(E, d, h, device="cuda") * 2 - 1) / np.sqrt(h)).to(bf)
    b2 = ((torch.rand(E, d, device="cuda") * 2 - 1) / np.sqrt(h)).to(bf)
    gy = torch.randn(B, d, device="cuda").to(bf)
    hid, deriv = fc.linear_forward_act(x, off, w1, b1, _lib.ACT_GELU, want_pre=True)         # product 1
    y, _ = fc.linear_forward_act(hid, off, w2, b2, _lib.ACT_NONE)                            # product 2
    gh, gw2, gb2, gb1 = fc.linear_backward_act(gy, hid, off, w2, deriv, _lib.ACT_GELU,       # products 3, 4
                                               want_gx_colsum=True)
    gx, gw1, _ = fc.linear_backward_act(gh, x, off, w1, None, _lib.ACT_NONE, need_bias=False)  # products 5, 6
    assert device_status() == 0
    p = 0
    for e, c in enumerate(counts):
        sl = slice(p, p + int(c))
        p += int(c)
        xe, ge = x[sl].float(), gy[sl].float()
        pre = xe @ w1[e].float().t() + b1[e].float()
        close(hid[sl], torch.nn.functional.gelu(pre))
        cdf = 0.5 * (1 + torch.erf(pre * 0.7071067811865476))
        want_deriv = cdf + pre * torch.exp(-0.5 * pre * pre) * 0.3989422804014327
        close(deriv[sl], want_deriv)
        # from here on every product is checked against fp32 math on the kernel's own 16-bit inputs
        he = hid[sl].float()
        close(y[sl], he @ w2[e].float().t() + b2[e].float())
        close(gh[sl], (ge @ w2[e].float()) * deriv[sl].float())
        close(gw2[e], ge.t() @ he)
        close(gb2[e], ge.sum(0))
        ghe = gh[sl].float()
        close(gb1[e], ghe.sum(0))
        close(gx[sl], ghe @ w1[e].float())
        close(gw1[e], ghe.t() @ xe)


def test_offsets_beyond_the_buffer_are_clamped(fc):
    """Segment offsets that live on the device are not seen by the host.  When they overshoot the
    buffers (or run backwards) the kernels clamp them: nothing is read or written past the rows
    given, rows past the clamped end keep their old contents, and status code 8 is raised."""
    from fastermoe_b200 import _lib
    torch.manual_seed(9)
    fin, fout, rows = 256, 512, 700
    for dtype in (torch.bfloat16, torch.float32):
        # counts claim 300 + 900 rows, the buffers hold 700 followed by poisoned padding
        off = torch.tensor([0, 300, 1200], dtype=torch.int64, device="cuda")
        x = torch.full((rows + 600, fin), float("nan"), device="cuda", dtype=dtype)
        gy = torch.full((rows + 600, fout), float("nan"), device="cuda", dtype=dtype)
        x[:rows] = torch.randn(rows, fin, device="cuda").to(dtype)
        gy[:rows] = torch.randn(rows, fout, device="cuda").to(dtype)
        w = ((torch.rand(2, fout, fin, device="cuda") * 2 - 1) / np.sqrt(fin)).to(dtype)
        y = torch.full((rows + 600, fout), 7.0, device="cuda", dtype=dtype)
        gx = torch.full((rows + 600, fin), 7.0, device="cuda", dtype=dtype)
        gw = torch.empty_like(w)
        gb = torch.empty(2, fout, device="cuda", dtype=dtype)
        code = _lib.BF16 if dtype == torch.bfloat16 else _lib.F32
        st = fc._stream()
        P = lambda t: ctypes.c_void_p(t.data_ptr())
        # the library is told the truth about the buffers (700 rows); only the offsets lie
        assert _lib.lib.fmoe_linear_forward(P(x), P(w), None, P(off), P(y), None, rows, fin, fout, 2, code, 0, st) == 0
        scratch = torch.empty(_lib.lib.fmoe_linear_scratch_bytes(rows, fin, fout, 2, code) + 16, dtype=torch.uint8, device="cuda")
        assert _lib.lib.fmoe_linear_backward(P(gy), P(x), P(w), P(off), None, P(gx), P(gw), P(gb), rows, fin, fout, 2,
                                             code, 0, 0, P(scratch), st) == 0
        torch.cuda.synchronize()
        assert (y[rows:] == 7).all() and (gx[rows:] == 7).all(), "rows past the buffer were written"
        wy, wgx, wgw, wgb = reference(x[:rows], [300, 400], w, None, gy[:rows])
        tol = close if dtype == torch.bfloat16 else (lambda a, b: torch.testing.assert_close(a.float(), b, rtol=1e-4, atol=1e-4))
        tol(y[:rows], wy); tol(gx[:rows], wgx); tol(gw, wgw); tol(gb, wgb)
        if dtype == torch.bfloat16:
            assert device_status() == 8
            assert _lib.lib.fmoe_device_status_clear() == 0
    # the reference-named operators take counts on the host and refuse a mismatch before launching
    with pytest.raises(RuntimeError, match="rows"):
        fc.linear_forward(x[:rows].contiguous(), torch.tensor([300, 900]), w)
    assert device_status() == 0


@pytest.mark.parametrize("form", ["pair", "auto"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_cta_pair_kernels(fc, form, dtype):
    """The cta_group::2 kernels (256-row tiles, one CTA pair per tile) against fp32 matmuls and,
    bit for bit, against the one-CTA kernels: both accumulate the same products in the same order.
    'pair' forces them for all three products; 'auto' is the default choice at a size where it
    picks pairs for the forward and input-gradient products."""
    from fastermoe_b200 import _lib
    torch.manual_seed(11)
    if form == "pair":
        counts, fin, fout = [2048 + 77, 300, 2600, 0, 1500, 255, 257], 512, 768
        fc.set_gemm_form("pair")
    else:
        counts, fin, fout = [9000, 12001, 8191, 10808], 256, 1024      # >= 512 rows per expert, >= 148 pair tiles
    E, B = len(counts), sum(counts)
    off = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int64, device="cuda")
    x = torch.randn(B, fin, device="cuda").to(dtype)
    gy = torch.randn(B, fout, device="cuda").to(dtype)
    w = ((torch.rand(E, fout, fin, device="cuda") * 2 - 1) / np.sqrt(fin)).to(dtype)
    b = ((torch.rand(E, fout, device="cuda") * 2 - 1) / np.sqrt(fin)).to(dtype)

    def run():
        y, pre = fc.linear_forward_act(x, off, w, b, _lib.ACT_GELU, want_pre=True)
        y0, _ = fc.linear_forward_act(x, off, w, b, _lib.ACT_NONE)
        gx, gw, gb = fc.linear_backward_act(gy, x, off, w, None, _lib.ACT_NONE)
        return y, pre, y0, gx, gw, gb

    got = run()
    fc.set_gemm_form("tc1")
    single = run()
    fc.set_gemm_form("auto")
    assert device_status() == 0
    for name, a_, b_ in zip(["y", "pre", "y0", "gx", "gw", "gb"], got, single):
        assert torch.equal(a_, b_), f"{name}: CTA-pair and one-CTA kernels differ"
    wy, wgx, wgw, wgb = reference(x, counts, w, b, gy)
    close(got[2], wy)
    close(got[3], wgx)
    close(got[4], wgw)
    close(got[5], wgb)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("form", ["auto", "pair"])
def test_input_gradient_column_sums(fc, dtype, form):
    """linear_backward_act(want_gx_colsum=True): per-expert column sums of the returned dX (the bias
    gradient of the layer below), from the tensor-core epilogue (16-bit) or the plain kernel (fp32)."""
    from fastermoe_b200 import _lib
    if form == "pair":
        if dtype == torch.float32:
            pytest.skip("fp32 takes the FFMA kernels")
        fc.set_gemm_form("pair")
        counts, fin, fout = [2048 + 77, 300, 2600, 0, 1500, 31, 33], 512, 256
    else:
        counts, fin, fout = [100, 0, 0, 29, 257, 32, 1, 511], 320, 256
    torch.manual_seed(5)
    E, B = len(counts), sum(counts)
    off = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int64, device="cuda")
    x = torch.randn(B, fin, device="cuda").to(dtype)
    gy = torch.randn(B, fout, device="cuda").to(dtype)
    w = ((torch.rand(E, fout, fin, device="cuda") * 2 - 1) / np.sqrt(fin)).to(dtype)
    saved = torch.rand(B, fin, device="cuda").to(dtype)          # stands for a saved GELU derivative
    for act_pre, act in ((None, _lib.ACT_NONE), (saved, _lib.ACT_GELU)):
        gx, gw, gb, cs = fc.linear_backward_act(gy, x, off, w, act_pre, act, want_gx_colsum=True)
        gx0, gw0, gb0 = fc.linear_backward_act(gy, x, off, w, act_pre, act)
        assert torch.equal(gx, gx0) and torch.equal(gw, gw0) and torch.equal(gb, gb0)
        want = torch.zeros(E, fin, device="cuda")
        p = 0
        for e, c in enumerate(counts):
            want[e] = gx[p:p + c].float().sum(0)
            p += c
        # fp32 sums of the kernel's own (rounded) dX, rounded once to the output type
        rms = float(want.pow(2).mean().sqrt())
        if dtype == torch.float32:
            torch.testing.assert_close(cs.float(), want, rtol=1e-5, atol=1e-5 * rms)
        else:
            torch.testing.assert_close(cs.float(), want, rtol=2e-2, atol=4 * 2.0 ** -9 * rms)
    assert device_status() == 0


TOKEN_MINOR = [
    # on the 64-element grid: the token-major kernels at the same row counts
    ([1, 31, 32, 33, 0, 63, 64, 65], 256, 384),
    ([3, 0, 0, 1], 2048, 1024),
    ([255, 256, 257, 0, 1, 129], 512, 256),
    ([700, 37], 256, 832),
    # widths off the 64-element grid, the smallest ones, columns that end inside a 32-column block
    ([100, 0, 29, 300], 200, 712),
    ([5, 70], 32, 40),
    ([33, 95, 64], 264, 72),
    ([1300, 1, 1500], 136, 328),
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("counts,fin,fout", TOKEN_MINOR)
def test_token_minor_products(fc, dtype, counts, fin, fout):
    """Forward (bias, GELU with its saved derivative), input gradient (with column sums) and weight gradient, against
    fp32.  Rows past the segments hold NaNs and the expert after each used one holds infinities: neither may show."""
    from fastermoe_b200 import _lib
    torch.manual_seed(sum(counts) + fin + fout)
    counts = [c for n in counts for c in (n, 0)]            # every other expert has no rows, and infinite weights
    E, B, pad = len(counts), sum(counts), 3
    x = torch.full((B + pad, fin), float("nan"), device="cuda", dtype=dtype)
    gy = torch.full((B + pad, fout), float("nan"), device="cuda", dtype=dtype)
    x[:B], gy[:B] = torch.randn(B, fin, device="cuda").to(dtype), torch.randn(B, fout, device="cuda").to(dtype)
    w = ((torch.rand(E, fout, fin, device="cuda") * 2 - 1) / np.sqrt(fin)).to(dtype)
    b = ((torch.rand(E, fout, device="cuda") * 2 - 1) / np.sqrt(fin)).to(dtype)
    saved = torch.rand(B + pad, fin, device="cuda").to(dtype)
    w[1::2] = float("inf")
    off = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int64, device="cuda")
    y, pre = fc.linear_forward_act(x, off, w, b, _lib.ACT_GELU, want_pre=True)
    plain, _ = fc.linear_forward_act(x, off, w, None, _lib.ACT_NONE)
    gx, gw, gb, cs = fc.linear_backward_act(gy, x, off, w, saved, _lib.ACT_GELU, want_gx_colsum=True)
    assert device_status() == 0
    p = 0
    for e, c in enumerate(counts):
        xe, ge = x[p:p + c].float(), gy[p:p + c].float()
        if c:
            z = xe @ w[e].float().t()
            close(plain[p:p + c], z)
            zb = (z + b[e].float()).requires_grad_(True)
            act = torch.nn.functional.gelu(zb)
            close(y[p:p + c], act.detach())
            close(pre[p:p + c], torch.autograd.grad(act.sum(), zb)[0])
            close(gx[p:p + c], (ge @ w[e].float()) * saved[p:p + c].float())
            # sums of the rounded rows
            want = gx[p:p + c].float().sum(0)
            torch.testing.assert_close(cs[e].float(), want, rtol=2e-2, atol=2.0 ** -8 * float(want.abs().max()))
        close(gw[e], ge.t() @ xe)
        close(gb[e], ge.sum(0))
        p += c


@pytest.mark.parametrize("act", ["relu", "none"])
def test_token_minor_epilogues(fc, act):
    """ReLU forward and backward and the plain products at a ragged size, against fp32."""
    from fastermoe_b200 import _lib
    torch.manual_seed(5)
    counts, fin, fout = [40, 0, 97], 328, 200
    code = {"relu": _lib.ACT_RELU, "none": _lib.ACT_NONE}[act]
    E, B = len(counts), sum(counts)
    x, gy = torch.randn(B, fin, device="cuda").bfloat16(), torch.randn(B, fout, device="cuda").bfloat16()
    w = ((torch.rand(E, fout, fin, device="cuda") * 2 - 1) / np.sqrt(fin)).bfloat16()
    b = torch.randn(E, fout, device="cuda").bfloat16()
    saved = torch.randn(B, fin, device="cuda").relu().bfloat16()
    off = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int64, device="cuda")
    y, _ = fc.linear_forward_act(x, off, w, b, code)
    gx, _, _ = fc.linear_backward_act(gy, x, off, w, saved if act == "relu" else None, code)
    p = 0
    for e, c in enumerate(counts):
        z = x[p:p + c].float() @ w[e].float().t() + b[e].float()
        close(y[p:p + c], z.relu() if act == "relu" else z)
        g = gy[p:p + c].float() @ w[e].float()
        close(gx[p:p + c], g * (saved[p:p + c].float() > 0) if act == "relu" else g)
        p += c


@pytest.mark.parametrize("what", ["no_scratch", "odd_address"])
@pytest.mark.parametrize("fin,fout", [(200, 136), (64, 64), (30, 50)])
def test_column_sums_without_scratch(what, fin, fout):
    """Off the 64-element grid the column sums need neither the scratch buffer nor an even number of elements before them."""
    from fastermoe_b200 import _lib
    counts = [17, 0, 23]
    B, E = sum(counts), len(counts)
    x, gy = torch.randn(B, fin, device="cuda").bfloat16(), torch.randn(B, fout, device="cuda").bfloat16()
    w = (torch.randn(E, fout, fin, device="cuda") / np.sqrt(fout)).bfloat16()
    off = torch.tensor([0, 17, 17, 40], device="cuda")
    gx, gw = torch.empty_like(x), torch.empty_like(w)
    cs = torch.empty(E * fin + 1, device="cuda", dtype=torch.bfloat16)[int(what == "odd_address"):]
    nbytes = _lib.lib.fmoe_linear_scratch_bytes(B, fin, fout, E, _lib.BF16)
    scratch = None if what == "no_scratch" else torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    ptr = [None if t is None else t.data_ptr() for t in (gy, x, w, off, None, gx, gw, None, cs)]
    rc = _lib.lib.fmoe_linear_backward_colsum(*ptr, B, fin, fout, E, _lib.BF16, _lib.ACT_NONE, 0,
                                              None if scratch is None else scratch.data_ptr(), None)
    assert rc == 0, _lib.lib.fmoe_last_error_string()
    torch.cuda.synchronize()
    p = 0
    for e, c in enumerate(counts):
        close(gx[p:p + c], gy[p:p + c].float() @ w[e].float())
        close(cs[e * fin:(e + 1) * fin], gx[p:p + c].float().sum(0))
        p += c


def gemm_kernels(call):
    """Template arguments (mode, bf16, pair, token-minor) of the tensor-core products that ``call`` launches."""
    import re
    call()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    found = []
    for e in prof.events():
        m = re.search(r"grouped_gemm_kernel<([^>]*)>", e.name)
        if m:
            words = re.sub(r"\((int|bool)\)", "", m.group(1)).replace("true", "1").replace("false", "0")
            found.append(tuple(int(w) for w in words.split(",")))
    return found


def test_forced_form_off_the_grid(fc):
    """"pair" and "tc1" force the form of widths off the 64-element grid too; "auto" goes by the rows per expert."""
    from fastermoe_b200 import _lib
    fin, fout = 200, 136
    w = torch.randn(2, fout, fin, device="cuda").bfloat16()
    for rows, auto in ((20, 0), (400, 1)):
        x = torch.randn(rows, fin, device="cuda").bfloat16()
        off = torch.tensor([0, rows // 2, rows], device="cuda")
        for form, pair in (("auto", auto), ("pair", 1), ("tc1", 0)):
            fc.set_gemm_form(form)
            ran = gemm_kernels(lambda: (fc.linear_forward_act(x, off, w, None, _lib.ACT_NONE),
                                        fc.linear_backward_act(x.new_ones(rows, fout), x, off, w, None, _lib.ACT_NONE)))
            assert sorted(ran)[:2] == [(0, 1, pair, 1), (1, 1, pair, 1)], (form, rows, ran)


TOKEN_MINOR_EDGES = [
    # the 32-token steps of one CTA and its 64-token tiles; widths with a column block of 8 and of 24
    ([1, 31, 32, 33, 0, 63, 64, 65], 264, 200),
    # the 64-token steps of a pair; its second CTA has 8 columns of 392 and none of 520
    ([127, 128, 129, 191, 192, 193], 392, 520),
    # segments that end on a 256-token tile, one before and one after it
    ([255, 256, 257, 0, 1, 512], 136, 328),
    ([700, 37], 72, 264),
    ([3, 0, 0, 1], 2056, 1032),
    ([5, 70], 32, 40),
]


@pytest.mark.parametrize("form", ["pair", "tc1"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("counts,fin,fout", TOKEN_MINOR_EDGES)
def test_token_minor_edges(fc, form, dtype, counts, fin, fout):
    """Both forms of the products off the 64-element grid at the edges of their steps and tiles."""
    fc.set_gemm_form(form)
    test_token_minor_products(fc, dtype, counts, fin, fout)


@pytest.mark.parametrize("form", ["pair", "tc1"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("act", ["relu", "none", "gelu", "silu"])
def test_token_minor_activations(fc, form, dtype, act):
    """Every activation in both forms: value and saved derivative forward, the saved factor backward, against fp32."""
    from fastermoe_b200 import _lib
    fc.set_gemm_form(form)
    code = {"relu": _lib.ACT_RELU, "none": _lib.ACT_NONE, "gelu": _lib.ACT_GELU, "silu": _lib.ACT_SILU}[act]
    fn = {"relu": torch.relu, "none": lambda z: z * 1, "gelu": torch.nn.functional.gelu, "silu": torch.nn.functional.silu}[act]
    counts, fin, fout = [40, 0, 97, 256, 5], 328, 200
    E, B = len(counts), sum(counts)
    x, gy = torch.randn(B, fin, device="cuda").to(dtype), torch.randn(B, fout, device="cuda").to(dtype)
    w = ((torch.rand(E, fout, fin, device="cuda") * 2 - 1) / np.sqrt(fin)).to(dtype)
    b = (torch.randn(E, fout, device="cuda") * 4).to(dtype)
    saved = (torch.randn(B, fin, device="cuda").relu() if act == "relu" else torch.randn(B, fin, device="cuda")).to(dtype)
    off = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int64, device="cuda")
    saves = act in ("gelu", "silu")
    y, pre = fc.linear_forward_act(x, off, w, b, code, want_pre=saves)
    alone, _ = fc.linear_forward_act(x, off, w, b, code)
    assert torch.equal(y, alone)                       # the value does not depend on whether the derivative is kept
    gx, _, _ = fc.linear_backward_act(gy, x, off, w, None if act == "none" else saved, code)
    factor = {"relu": (saved > 0).float(), "none": torch.ones_like(saved).float()}.get(act, saved.float())
    assert device_status() == 0
    p = 0
    for e, c in enumerate(counts):
        z = (x[p:p + c].float() @ w[e].float().t() + b[e].float()).requires_grad_(True)
        close(y[p:p + c], fn(z).detach())
        if saves and c:
            close(pre[p:p + c], torch.autograd.grad(fn(z).sum(), z)[0])
        close(gx[p:p + c], gy[p:p + c].float() @ w[e].float() * factor[p:p + c])
        p += c


BIAS_GRADIENTS = [
    # rows of the experts (long and empty ones among them), out_feat: every number of blocks that share a segment
    ([20] * 100, 4096),                         # one block
    ([140] * 15 + [0], 4096),                   # two, beside the products
    ([1] + [320] * 14 + [0], 4096),             # four, beside the products
    ([3, 0, 40, 1], 320),                       # eight, most of them without rows
    ([9000, 5, 0], 128),                        # eight, rows that eight does not divide; out_feat off the grid
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("counts,fout", BIAS_GRADIENTS)
def test_bias_gradient(fc, dtype, counts, fout):
    """Column sums per segment against fp64: fp32 sums of 16-bit rows, rounded once; the same from call to call, beside the
    products and (in a captured graph) in stream order before them."""
    from fastermoe_b200 import _lib
    E, B, fin = len(counts), sum(counts), 256
    off = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int64, device="cuda")
    x, gy = torch.randn(B, fin, device="cuda").to(dtype), torch.randn(B, fout, device="cuda").to(dtype)
    w = (torch.randn(E, fout, fin, device="cuda") / np.sqrt(fout)).to(dtype)
    runs = [fc.linear_backward_act(gy, x, off, w, None, _lib.ACT_NONE)[2] for _ in range(3)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = fc.linear_backward_act(gy, x, off, w, None, _lib.ACT_NONE)[2]
    graph.replay()
    assert all(torch.equal(r, captured) for r in runs)
    eps = torch.finfo(dtype).eps
    p = 0
    for e, c in enumerate(counts):
        rows = gy[p:p + c].double()
        # one rounding to the output type, and c fp32 additions of terms whose magnitudes add up to `size`
        want, size = rows.sum(0), rows.abs().sum(0)
        bound = 0.5 * eps * want.abs() + (c + 1) * 2.0 ** -24 * size * (1 + eps)
        assert bool(((captured[e].double() - want).abs() <= bound).all())
        p += c


def test_bias_gradient_from_threads(fc):
    """Two threads on streams of their own, their backward calls interleaved: the side stream that they share takes each
    gradient after its rows and before it is read."""
    import threading
    from fastermoe_b200 import _lib
    E, B, fin, fout = 4, 4096, 256, 512
    off = torch.arange(0, B + 1, B // E, device="cuda")
    w = torch.randn(E, fout, fin, device="cuda").bfloat16()
    torch.cuda.synchronize()
    wrong = []

    def work(seed):
        stream = torch.cuda.Stream()
        g = torch.Generator(device="cuda").manual_seed(seed)
        with torch.cuda.stream(stream):
            x = torch.randn(B, fin, device="cuda", generator=g).bfloat16()
            for _ in range(30):
                gy = torch.randint(-4, 5, (B, fout), device="cuda", generator=g).bfloat16()      # sums are exact in fp32
                gb = fc.linear_backward_act(gy, x, off, w, None, _lib.ACT_NONE)[2]
                want = gy.float().view(E, B // E, fout).sum(1).bfloat16()
                wrong.append((gb != want).sum())
            stream.synchronize()

    threads = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(wrong) == 60 and int(torch.stack(wrong).sum()) == 0
