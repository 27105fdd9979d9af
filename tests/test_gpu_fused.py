"""One-launch model set-up and one-call evaluation against the compositions of
tensor operations that define them: values, gradients, second gradients, and
the inputs they leave to the compositions.

Tolerance 1e-12 of the largest entry: sums of at most 61 products (61 x 1.1e-16 =
7e-15) over factors of order 1 to 100; the evaluation adds the eigen system's
1e-14 over at most 64 states."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(got, want, tol=1e-12):
    got, want = got.detach().cpu().numpy(), want.detach().cpu().numpy()
    assert got.shape == want.shape
    np.testing.assert_allclose(got, want, rtol=tol, atol=tol * max(np.abs(want).max(), 1e-300))


def _leaf(a):
    return torch.tensor(a, dtype=torch.float64, device="cuda").requires_grad_()


def _same(fn, compose, inputs, second=True):
    a, c = fn(*inputs), compose(*inputs)
    _close(a, c)
    g = torch.linspace(-1.0, 2.0, a.numel(), dtype=torch.float64, device="cuda").reshape(a.shape).sin()
    ga = torch.autograd.grad(a, inputs, g)
    for x, y in zip(ga, torch.autograd.grad(c, inputs, g)):
        _close(x, y)
    if second:
        outs = []
        for f in (fn, compose):
            first = torch.autograd.grad(f(*inputs), inputs, g, create_graph=True)
            outs.append(torch.autograd.grad(sum((t * t).sum() for t in first), inputs))
        for x, y in zip(*outs):
            _close(x, y)


@pytest.mark.parametrize("k", [1, 3, 4, 8, 32])
@pytest.mark.parametrize("kind", ["weibull", "gamma"])
@pytest.mark.parametrize("lead", [(3,), (), (2, 2)])
def test_category_rates(k, kind, lead):
    from torchtree_gb300 import site_models

    rng = np.random.default_rng(k)
    shape = _leaf(rng.uniform(0.2, 3.0, lead + (1,)))
    fn = getattr(site_models, kind + "_rates")
    compose = {"weibull": site_models._weibull, "gamma": site_models._gamma}[kind]
    rates, probs = fn(shape, k)
    want_r, want_p = compose(shape, k)
    assert probs.shape == want_p.shape and torch.equal(probs, want_p) and not probs.requires_grad
    assert type(rates.grad_fn).__name__.startswith("CategoryRates")
    if k > 1:  # one category's rate is constant
        _same(lambda s: fn(s, k)[0], lambda s: compose(s, k)[0], (shape,))


@pytest.mark.parametrize("b", [1, 3])
@pytest.mark.parametrize("model", ["gtr", "hky", "general2", "general20", "general61", "mg94"])
def test_rate_matrices(model, b):
    from torchtree_gb300 import substitution as sub

    rng = np.random.default_rng(b)
    S = {"gtr": 4, "hky": 4, "general2": 2, "general20": 20, "general61": 61, "mg94": 61}[model]
    pi = _leaf(rng.dirichlet(5.0 * np.ones(S), b))
    if model == "hky":
        params, fn, compose = (_leaf(rng.uniform(1, 5, (b, 1))),), sub.hky_q, sub._hky
    elif model == "mg94":
        params = tuple(_leaf(rng.uniform(0.2, 4, (b, 1))) for _ in range(3))
        fn, compose = sub.mg94_q, lambda a, w, k, p: sub._mg94(a, w, k, p, sub.UNIVERSAL_CODE)
    else:
        params = (_leaf(rng.gamma(1.0, 1.0, (b, S * (S - 1) // 2))),)
        fn = sub.gtr_q if model == "gtr" else (lambda r, p: sub.general_symmetric_q(r, p, S))
        compose = lambda r, p: sub._general(r, p, S)  # noqa: E731
    assert type(fn(*params, pi).grad_fn).__name__.startswith("ExchangeabilityQ")
    _same(fn, compose, (*params, pi))
    # strided inputs, and gradients for some of the inputs only
    wide = _leaf(np.repeat(params[0].detach().cpu().numpy(), 2, -1))
    q = fn(wide[:, ::2], *[p.detach() for p in params[1:]], pi.detach())
    _close(q, compose(*params, pi))
    assert torch.autograd.grad(q.sum() + (q * q).sum(), wide)[0].shape == wide.shape


def test_compositions_keep_what_the_kernels_do_not_take():
    from torchtree_gb300 import site_models, substitution as sub

    rng = np.random.default_rng(0)
    r, p = _leaf(rng.gamma(1.0, 1.0, (3, 6))), _leaf(rng.dirichlet(np.ones(4), 3))
    fused = sub.gtr_q(r, p)
    for q in (sub.gtr_q(r[0], p[0]), sub.gtr_q(r.cpu(), p.cpu())[0], sub.gtr_q(r.float(), p.float())[0],
              sub.gtr_q(r[:1], p)[0]):
        assert not type(q.grad_fn).__name__.startswith("ExchangeabilityQ")
        np.testing.assert_allclose(q.detach().cpu().numpy(), fused[0].detach().cpu().numpy(), rtol=2e-6, atol=1e-6)
    _, tangent = torch.func.jvp(lambda x: sub.gtr_q(x, p.detach()), (r.detach(),), (torch.ones_like(r),))
    _close(tangent, sub._general(torch.ones_like(r), p, 4))
    s = _leaf(rng.uniform(0.5, 1.0, (3, 1)))
    _, tangent = torch.func.jvp(lambda x: site_models.weibull_rates(x, 4)[0], (s.detach(),), (torch.ones_like(s),))
    assert tangent.shape == (3, 4)
    out = torch.func.vmap(lambda x: site_models.weibull_rates(x, 4)[0])(s.detach())
    _close(out, site_models.weibull_rates(s, 4)[0])
    with pytest.raises(RuntimeError):
        sub.gtr_q(_leaf(np.ones((3, 5))), p)
    inv = _leaf(np.full((3, 1), 0.2))
    assert site_models.weibull_rates(s, 4, invariant=inv)[0].shape == (3, 5)


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("S,K,b", [(4, 4, 3), (4, 1, 1), (7, 3, 2), (61, 2, 1)])
def test_one_call_evaluation_matches_the_separate_steps(precision, S, K, b):
    from torchtree_gb300 import substitution as sub, synthetic
    from torchtree_gb300.likelihood import PhyloLikelihood
    from torchtree_gb300.patterns import CompressedAlignment

    rng = np.random.default_rng(S + K)
    T, N = 9, 70
    topo = synthetic.yule_topology(T, rng)
    codes = rng.integers(0, S + 1, (T, N)).astype(np.uint8)
    aln = CompressedAlignment(codes, np.vstack([np.eye(S), np.ones((1, S))]), rng.integers(1, 4, N),
                              np.zeros((T, 0), np.uint8))
    bl, pi = _leaf(rng.exponential(0.1, (b, 2 * T - 3))), _leaf(rng.dirichlet(5.0 * np.ones(S), b))
    exch = rng.gamma(1.0, 1.0, (b, S * (S - 1) // 2))
    q = sub._general(torch.tensor(exch, device="cuda"), pi.detach(), S).requires_grad_()
    rates = _leaf(rng.uniform(0.2, 2.0, (b, K)))
    props = _leaf(rng.dirichlet(np.ones(K)))
    lik = PhyloLikelihood(topo, aln, S, K, batch=b, precision=precision)
    ins = (bl, q, pi, rates, props)

    def separate():
        return lik.evaluate_rate_matrix(sub.normalise(q, pi), pi, lik.node_branch_lengths(bl), rates,
                                        props.expand(b, K), pi)

    def once():
        return lik(bl, q, pi, rates, props.expand(b, K))

    assert type(once().grad_fn).__name__.startswith("EvaluateLikelihood")
    g = torch.linspace(0.5, 2.0, b, dtype=torch.float64, device="cuda")
    tol = 1e-12 if precision == "f64" else 1e-9  # FP32 matrices may round the other way where Q differs by an ulp
    a, c = once(), separate()
    _close(a, c, tol)
    for x, y in zip(torch.autograd.grad(once(), ins, g), torch.autograd.grad(separate(), ins, g)):
        _close(x, y, tol * 1e3 if precision == "f32" else tol * 10)
    # the stored partials of the first were overwritten by the second: its backward evaluates again
    first = once()
    once()
    for x, y in zip(torch.autograd.grad(first, ins, g), torch.autograd.grad(once(), ins, g)):
        _close(x, y, 1e-13)
    # a graph of the gradient, as the separate steps leave it
    w = g.clone().requires_grad_()
    seconds = []
    for f in (once, separate):
        first = torch.autograd.grad(f(), ins, w, create_graph=True)
        seconds.append(torch.autograd.grad(sum((t * t).sum() for t in first), (w, q), allow_unused=True))
    for x, y in zip(*seconds):
        _close(x, y, 1e-5 if precision == "f32" else 1e-10)
    # lnL only, one tensor without a gradient, and inputs that take the separate steps
    with torch.no_grad():
        _close(once(), a, 0.0)
    (gb,) = torch.autograd.grad(lik(bl, q.detach(), pi.detach(), rates.detach(), props.detach().expand(b, K)).sum(), bl)
    assert gb.shape == bl.shape
    clock = lik(torch.cat((bl, bl[:, :1]), 1), q, pi, rates, props.expand(b, K), clock_rates=torch.ones_like(bl[:, :1]))
    assert not type(clock.grad_fn).__name__.startswith("EvaluateLikelihood")
    assert lik.engine.device_status() == 0


def test_codon_gradient_from_a_thread_without_a_context():
    """The tensor-core adjoint encodes tensor maps through the driver; the call must
    not depend on an earlier runtime call of its thread."""
    import threading

    from torchtree_gb300 import synthetic
    from torchtree_gb300.engine import LikelihoodEngine

    S, T, N = 61, 5, 40
    rng = np.random.default_rng(1)
    topo = synthetic.yule_topology(T, rng)
    eng = LikelihoodEngine(topo.postorder, T, S, 1, rng.integers(0, S, (T, N)), np.eye(S), np.ones(N), precision="f32")
    t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    pi = t(np.full((1, S), 1.0 / S))
    q = t(np.ones((1, S, S)) / S)
    q = q - torch.diag_embed(q.sum(-1))
    one, bl = t(np.ones((1, 1))), t(rng.exponential(0.1, (1, 2 * T - 3)))
    grad = t(np.ones(1))
    want = None
    for _ in range(2):  # the second time every buffer of the call comes from the caching allocator
        _, work = eng.evaluate(q, pi, bl, one, one, True, True)
        want = [x.clone() for x in eng.evaluate_gradient(work, grad, 2 * T - 3, [True] * 5)]
    _, work = eng.evaluate(q, pi, bl, one, one, True, True)
    torch.cuda.synchronize()
    out = []

    def call():
        try:
            out.append(eng.evaluate_gradient(work, grad, 2 * T - 3, [True] * 5))
        except Exception as e:  # noqa: BLE001
            out.append(e)

    th = threading.Thread(target=call)
    th.start()
    th.join()
    assert not isinstance(out[0], Exception), out[0]
    for a, b in zip(out[0], want):
        assert torch.equal(a, b)
