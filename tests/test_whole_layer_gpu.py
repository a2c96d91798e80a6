"""The layer as one library call against the same layer operator by operator, and the calls that must not take it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ACTS = {"gelu": torch.nn.GELU, "relu": torch.nn.ReLU, "silu": torch.nn.SiLU}


def make(T, d, h, E, k, act="gelu", dtype=torch.bfloat16, bias=True, softmax=True, seed=0):
    from fastermoe_b200 import FMoETransformerMLP
    torch.manual_seed(seed)
    m = FMoETransformerMLP(num_expert=E, d_model=d, d_hidden=h, top_k=k, activation=ACTS[act](), bias=bias)
    for p in m.parameters():
        torch.nn.init.uniform_(p, -d ** -0.5, d ** -0.5)
    m.gate.softmax_scores = softmax
    x = torch.randn(T, d, device="cuda").to(dtype).requires_grad_(True)
    return m.cuda().to(dtype), x


def step(m, x, g):
    x.grad = None
    m.zero_grad()
    out = m(x)
    out.backward(g)
    return [out.detach(), x.grad] + [p.grad for p in m.parameters()]


@pytest.mark.parametrize("act", list(ACTS))
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,d,h,E,k,bias", [(1, 256, 512, 4, 2, True), (67, 256, 512, 8, 2, False), (130, 72, 200, 5, 3, True),
                                            (33, 30, 50, 3, 1, True), (700, 264, 136, 40, 8, False)])
def test_one_call_equals_the_operators(act, dtype, T, d, h, E, k, bias):
    """Same kernels in the same order: equal to the last bit, and every output is written."""
    m, x = make(T, d, h, E, k, act, dtype, bias)
    g = torch.randn(T, d, device="cuda").to(dtype)
    from fastermoe_b200 import fmoe_cuda as fc
    one = step(m, x, g)
    fc.set_profile(fc.Profile())            # operator by operator
    try:
        parts = step(m, x, g)
    finally:
        fc.set_profile(None)
    for a, b in zip(one, parts):
        assert torch.equal(a, b)
    with torch.no_grad():
        assert torch.equal(m(x), one[0])
    assert m(x.detach()).shape == x.shape and all(torch.isfinite(t.float()).all() for t in one)


def test_partial_gradients():
    """Only what requires a gradient gets one."""
    m, x = make(50, 256, 512, 4, 2)
    g = torch.randn(50, 256, device="cuda").bfloat16()
    want = step(m, x, g)
    m.experts.requires_grad_(False)
    got = step(m, x, g)
    assert torch.equal(got[1], want[1]) and m.experts.htoh4.weight.grad is None
    assert torch.equal(m.gate.gate.weight.grad, want[2 + [n for n, _ in m.named_parameters()].index("gate.gate.weight")])
    m.experts.requires_grad_(True)
    m.zero_grad()
    m(x.detach()).backward(g)
    assert all(torch.equal(p.grad, w) for p, w in zip(m.parameters(), want[2:]))
    m.zero_grad()
    m.requires_grad_(False)
    x.grad = None
    m(x).backward(g)
    assert torch.equal(x.grad, want[1])


def test_parameters_that_do_not_fit_are_refused():
    """The fused call leaves them to the single operators, whose checks raise."""
    for name, shape in (("htoh4", (4, 512, 264)), ("h4toh", (4, 256, 504)), ("htoh4", (3, 512, 256))):
        m, x = make(20, 256, 512, 4, 2)
        getattr(m.experts, name).weight = torch.nn.Parameter(torch.zeros(shape, device="cuda", dtype=torch.bfloat16))
        with pytest.raises((AssertionError, RuntimeError)):
            m(x)


@pytest.mark.parametrize("act", ["gelu", "silu"])
def test_hooks_are_called(act):
    m, x = make(20, 256, 512, 4, 2, act)
    base = m(x)
    seen = []
    hooks = [m.experts.register_forward_hook(lambda *a: seen.append("experts"))]
    if act == "silu":       # the two linears and the activation are calls of their own then
        hooks += [getattr(m.experts, n).register_forward_hook(lambda *a, n=n: seen.append(n)) for n in ("htoh4", "activation")]
    out = m(x)
    assert seen == (["htoh4", "activation", "experts"] if act == "silu" else ["experts"])
    torch.testing.assert_close(out, base, rtol=2e-2, atol=2e-2)
    for h in hooks:
        h.remove()
    rows, plain = [], m.expert_fn
    m.expert_fn = lambda inp, *a: (rows.append(tuple(inp.shape)), plain(inp, *a))[1]
    m(x)
    assert rows == [(40, 256)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d,h", [(256, 320), (72, 200)])
def test_silu_against_fp32(dtype, d, h):
    """Layer with SiLU against plain autograd on the same (rounded) tensors in fp64; bounds as for the other
    activations: fp32 1e-5 of a typical element, bf16 a few of its roundings."""
    T, E, k = 90, 4, 2
    m, x = make(T, d, h, E, k, "silu", dtype)
    g = torch.randn(T, d, device="cuda").to(dtype)
    out, gx, *grads = step(m, x, g)
    with torch.no_grad():
        idx, _ = m.gate(x)
    leaves = {n: p.detach().double().requires_grad_(True) for n, p in m.named_parameters()}
    xr = x.detach().double().requires_grad_(True)
    logits = xr @ leaves["gate.gate.weight"].t() + leaves["gate.gate.bias"]
    score = torch.softmax(torch.gather(logits, 1, idx), 1)
    rows = []
    for t in range(T):
        acc = 0
        for j in range(k):
            e = int(idx[t, j])
            mid = torch.nn.functional.silu(leaves["experts.htoh4.weight"][e] @ xr[t] + leaves["experts.htoh4.bias"][e])
            acc = acc + score[t, j] * (leaves["experts.h4toh.weight"][e] @ mid + leaves["experts.h4toh.bias"][e])
        rows.append(acc)
    want = torch.stack(rows)
    want.backward(g.double())
    rel = 1e-5 if dtype == torch.float32 else 2e-2
    for got, ref in [(out, want.detach()), (gx, xr.grad)] + [(a, leaves[n].grad) for a, (n, _) in zip(grads, m.named_parameters())]:
        assert float((got.double() - ref).norm()) <= rel * float(ref.norm())


@pytest.mark.parametrize("E,k", [(2, 2), (16, 1), (32, 8), (33, 4), (200, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_gate_softmax_in_the_selection(E, k, dtype):
    """Scores and logit gradients of the fused softmax against torch on the library's own selection."""
    from fastermoe_b200.functions import gate_topk
    torch.manual_seed(E + k)
    logits = (torch.randn(301, E, device="cuda") * 3).to(dtype)
    logits[0], logits[1, 0], logits[2] = float("-inf"), float("nan"), 0
    logits[3, 0], logits[4, 1] = float("inf"), float("-inf")
    a, b = logits.clone().requires_grad_(True), logits.clone().requires_grad_(True)
    val, idx = gate_topk(a, k, softmax=True)
    raw, idx2 = gate_topk(b, k)
    assert torch.equal(idx, idx2)
    want = torch.softmax(raw, -1)
    eps = torch.finfo(dtype).eps
    torch.testing.assert_close(val, want, rtol=2 * eps, atol=1e-6, equal_nan=True)
    g = torch.randn(301, k, device="cuda").to(dtype)
    val.backward(g)
    want.backward(g)
    # products and a difference of the same rounded scores: a few roundings of the largest term
    torch.testing.assert_close(a.grad, b.grad, rtol=4 * eps, atol=4 * eps, equal_nan=True)


@pytest.mark.parametrize("n,E,cap", [(1, 1, 0), (5000, 16, 100), (5000, 16, 10 ** 6), (300000, 7, 20000)])
def test_limit_and_prune(n, E, cap):
    from fastermoe_b200 import fmoe_cuda as fc
    g = np.random.default_rng(n).integers(-1, E, n)
    left = torch.full((E,), cap, dtype=torch.int32, device="cuda")
    granted, pruned = fc.limit_and_prune(torch.from_numpy(g).cuda(), left, E)
    want, seen = g.copy(), np.zeros(E, dtype=np.int64)
    for i, e in enumerate(g):
        if e >= 0:
            want[i] = e if seen[e] < cap else -1
            seen[e] += 1
    assert (pruned.cpu().numpy() == want).all()
    assert (granted.cpu().numpy() == np.minimum(seen, cap)).all()
    assert (left.cpu().numpy() == cap - seen).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,E", [(1, 2), (9, 16), (1500, 33), (40, 256), (300, 300)])
def test_balance_loss(T, E, dtype):
    """Value and logit gradient against the definition in fp64; 16-bit gradients are rounded once.  (300 experts: the
    form in torch operators, which rounds the probabilities and their mean to the logits' type.)"""
    from fastermoe_b200.gates.gshard_gate import balance_loss_top1
    torch.manual_seed(T + E)
    logits = torch.randn(T, E, device="cuda").to(dtype).requires_grad_(True)
    idx = torch.randint(0, E, (T, 2), device="cuda")
    loss = balance_loss_top1(idx[:, 0], logits, E, E)
    grad, = torch.autograd.grad(3 * loss, logits, retain_graph=True)
    ref = logits.detach().double().requires_grad_(True)
    share = torch.bincount(idx[:, 0], minlength=E).double() / T
    want = (share * torch.softmax(ref, 1).mean(0)).mean() * E ** 2
    want_grad, = torch.autograd.grad(3 * want, ref, create_graph=True)
    eps = torch.finfo(dtype).eps
    rel = 1e-5 if E <= 256 else 4 * eps + 1e-5
    assert loss.dtype == torch.float32 and abs(float(loss.detach()) - float(want.detach())) <= rel * float(want.detach())
    floor = float(want_grad.abs().max())
    if dtype == torch.float16:
        floor += 6e-8 / eps             # fp16 subnormals
    torch.testing.assert_close(grad.double(), want_grad.detach(), rtol=4 * eps + 1e-5, atol=(8 * eps + 1e-6) * floor)
    if dtype == torch.float32:          # the gradient has a gradient
        g, = torch.autograd.grad(loss, logits, create_graph=True)
        w, = torch.autograd.grad(want, ref, create_graph=True)
        torch.testing.assert_close(torch.autograd.grad((g * g).sum(), logits)[0].double(), torch.autograd.grad((w * w).sum(), ref)[0],
                                   rtol=1e-3, atol=1e-5 * float(w.abs().max()) ** 2)


def expert_gradients(m, x, idx, score, g, act):
    """Gradients of the experts' parameters and of x, given the choice of experts and its weights, by autograd in fp64."""
    fn = {"gelu": torch.nn.functional.gelu, "silu": torch.nn.functional.silu}[act]
    p = {n: t.detach().double().requires_grad_(True) for n, t in m.experts.named_parameters()}
    xr = x.detach().double().requires_grad_(True)
    hid = fn(torch.einsum("ehd,td->teh", p["htoh4.weight"], xr) + p["htoh4.bias"])
    y = torch.einsum("edh,teh->ted", p["h4toh.weight"], hid) + p["h4toh.bias"]
    rows = torch.gather(y, 1, idx.unsqueeze(-1).expand(-1, -1, y.shape[2]))
    (score.detach().double().unsqueeze(-1) * rows).sum(1).backward(g.double())
    return {n: t.grad for n, t in p.items()}, xr.grad


@pytest.mark.parametrize("form", ["one_call", "operators"])
@pytest.mark.parametrize("act", ["gelu", "silu"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d,h", [(256, 320), (72, 200)])
@pytest.mark.parametrize("trained", ["htoh4.bias", "htoh4.bias h4toh.weight h4toh.bias", "htoh4.weight", "h4toh.weight"])
def test_some_parameters_trained(form, act, dtype, d, h, trained):
    """Any subset of the experts' parameters may be trained while input and gate need no gradient: the first layer's bias
    needs the activation's derivative as much as its weight does.  Bounds as in test_silu_against_fp32."""
    m, x = make(90, d, h, 4, 2, act, dtype)
    x.requires_grad_(False)
    if form == "operators":
        m.experts.register_forward_hook(lambda *a: None)
    m.requires_grad_(False)
    for n in trained.split():
        m.experts.get_parameter(n).requires_grad_(True)
    g = torch.randn(90, d, device="cuda").to(dtype)
    idx, score = m.gate(x)
    want, _ = expert_gradients(m, x, idx, score, g, act)
    m(x).backward(g)
    rel = 1e-5 if dtype == torch.float32 else 2e-2
    for n, p in m.experts.named_parameters():
        if n in trained.split():
            assert float((p.grad.double() - want[n]).norm()) <= rel * float(want[n].norm()), n
        else:
            assert p.grad is None


@pytest.mark.parametrize("act", ["gelu", "silu"])
def test_input_gradient_of_strided_rows(act):
    """A call of the experts on a transposed input, first layer frozen: its gradient passes the activation."""
    m, x = make(40, 256, 320, 1, 1, act, torch.float32)
    m.experts.htoh4.requires_grad_(False)
    xt = x.detach().t().contiguous().t().requires_grad_(True)
    out = m.experts(xt, torch.tensor([40]))
    g = torch.randn_like(out)
    out.backward(g)
    one = torch.ones(40, 1, device="cuda")
    _, want = expert_gradients(m, x, torch.zeros(40, 1, dtype=torch.int64, device="cuda"), one, g, act)
    assert float((xt.grad.double() - want).norm()) <= 1e-5 * float(want.norm())


@pytest.mark.parametrize("param_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("low", [torch.bfloat16, torch.float16])
def test_gate_scores_under_autocast(low, param_dtype):
    """Autocast forms softmaxes in fp32: the scores, their dtype and the gate's gradients are those of the softmax
    operator on the selected logits, to the last bit."""
    m, x = make(64, 256, 512, 8, 2, "gelu", param_dtype)
    g = torch.randn(64, 2, device="cuda")
    grads = []
    for fused in (True, False):
        m.zero_grad()
        x.grad = None
        with torch.autocast("cuda", low):
            m.gate.softmax_scores = fused
            idx, score = m.gate(x)
            if not fused:
                score = torch.nn.functional.softmax(score, dim=-1)
        assert score.dtype == torch.float32
        score.backward(g)
        grads.append([idx, score.detach(), x.grad] + [p.grad for p in m.gate.parameters()])
    assert all(torch.equal(a, b) for a, b in zip(*grads))


def test_balance_loss_keeps_its_graph():
    """The second derivative reaches logits in any layout, and the choices may be overwritten after the call."""
    from fastermoe_b200.gates.gshard_gate import balance_loss_top1
    idx = torch.randint(0, 12, (30,), device="cuda")
    plain = torch.randn(30, 12, device="cuda")
    want = None
    for strided in (False, True):
        leaf = (plain.t().contiguous() if strided else plain.clone()).requires_grad_(True)
        choice = idx.clone()
        loss = balance_loss_top1(choice, leaf.t() if strided else leaf, 12, 12)
        choice.zero_()
        first, = torch.autograd.grad(loss, leaf, create_graph=True)
        second, = torch.autograd.grad((first * first).sum(), leaf)
        got = [t.detach().t() if strided else t.detach() for t in (first, second)]
        if want is None:
            ref = plain.double().requires_grad_(True)
            share = torch.bincount(idx, minlength=12).double() / 30
            g, = torch.autograd.grad((share * torch.softmax(ref, 1).mean(0)).sum() * 12, ref, create_graph=True)
            want = [g.detach(), torch.autograd.grad((g * g).sum(), ref)[0]]
        for a, w in zip(got, want):
            torch.testing.assert_close(a.double(), w, rtol=1e-4, atol=1e-5 * float(w.abs().max()))


def test_balance_loss_of_calls_left_to_torch():
    """Function transforms, forward mode, tracing and compilation see the loss as operators, and a call may count fewer
    choices than there are logits: the same values as the operators give in fp64."""
    from fastermoe_b200.gates.gshard_gate import balance_loss_top1
    import torch.autograd.forward_ad as fa
    idx = torch.randint(0, 12, (30,), device="cuda")
    logits = torch.randn(30, 12, device="cuda")
    tangent = torch.randn_like(logits)

    def loss(v, choice=idx):
        return balance_loss_top1(choice, v, 12, 12)

    def want(v, choice=idx):
        return (torch.bincount(choice, minlength=12).double() / 30 * torch.softmax(v, 1).mean(0)).sum() * 12

    def close(a, b):
        torch.testing.assert_close(a.double(), b.double(), rtol=1e-5, atol=1e-6)

    ref = logits.double().requires_grad_(True)
    grad, = torch.autograd.grad(want(ref), ref)
    slope = (grad * tangent.double()).sum()
    value, along = torch.func.jvp(loss, (logits,), (tangent,))
    close(value, want(logits.double()))
    close(along, slope)
    close(torch.func.grad(loss)(logits), grad)
    close(torch.func.vmap(loss)(torch.stack([logits, 2 * logits])), torch.stack([want(s * logits.double()) for s in (1, 2)]))
    with fa.dual_level():
        close(fa.unpack_dual(loss(fa.make_dual(logits, tangent))).tangent, slope)
    close(torch.jit.trace(loss, (logits,))(2 * logits), want(2 * logits.double()))
    close(torch.compile(loss, backend="eager", fullgraph=True)(logits), want(logits.double()))
    close(loss(logits, idx[:20]), want(logits.double(), idx[:20]))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_silu_with_a_strided_weight(dtype):
    """A SiLU layer takes a transposed weight (its linears copy it): same output and gradients as with the copy, up to
    the activation's rounding where it is an operator of its own."""
    m, x = make(20, 256, 512, 4, 2, "silu", dtype)
    g = torch.randn(20, 256, device="cuda").to(dtype)
    want = step(m, x, g)
    for lin in (m.experts.htoh4, m.experts.h4toh):
        lin.weight = torch.nn.Parameter(lin.weight.detach().transpose(1, 2).contiguous().transpose(1, 2))
    tol = 1e-5 if dtype == torch.float32 else 2e-2
    for a, b in zip(step(m, x, g), want):
        assert float((a.double() - b.double()).norm()) <= tol * float(b.double().norm())


@pytest.mark.parametrize("T,E", [(5000, 2), (70000, 16), (9001, 64), (3000, 65), (4097, 256)])
def test_balance_loss_of_many_tokens(T, E):
    """Every number of blocks, and of finishing threads per expert, that the sizes select, against the definition in fp64.
    An element of the gradient is p (w - sum p w): its error is a few roundings of the largest w, whatever cancels."""
    from fastermoe_b200.gates.gshard_gate import balance_loss_top1
    logits = torch.randn(T, E, device="cuda", requires_grad=True)
    idx = torch.randint(0, E, (T,), device="cuda")
    loss = balance_loss_top1(idx, logits, E, E)
    loss.backward()
    ref = logits.detach().double().requires_grad_(True)
    share = torch.bincount(idx, minlength=E).double() / T
    want = (share * torch.softmax(ref, 1).mean(0)).mean() * E ** 2
    want.backward()
    assert abs(float(loss.detach()) - float(want.detach())) <= 1e-5 * float(want.detach())
    w = E * share / T
    torch.testing.assert_close(logits.grad.double(), ref.grad, rtol=1e-5, atol=8 * 2.0 ** -23 * float(w.max()))
