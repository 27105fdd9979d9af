"""Gradients with a graph of their own (create_graph) and batches of incoming gradients
through the one-launch set-up and the one-call evaluation, where inputs depend on one
another as they do in a model: the rate matrix on the frequencies, the root frequencies
the rate matrix's.  Against the compositions of tensor operations and the separate steps.

Tolerance 1e-10 of the largest entry: FP64 sums of 40 patterns x 4 states and of the
4-state matrix products around them (1e-14), amplified by the second derivative's factors
of up to 1e3."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

T, N, B, K = 12, 40, 3, 4


def _close(got, want, tol=1e-10):
    got, want = got.detach().cpu().numpy(), want.detach().cpu().numpy()
    assert got.shape == want.shape
    np.testing.assert_allclose(got, want, rtol=tol, atol=tol * max(np.abs(want).max(), 1e-300))


def _leaf(a):
    return torch.tensor(a, dtype=torch.float64, device="cuda").requires_grad_()


def _model(site):
    """``(lnL of the leaves by the fused calls, the same by separate steps, the leaves)``."""
    from torchtree_gb300 import site_models, substitution as sub, synthetic
    from torchtree_gb300.likelihood import PhyloLikelihood
    from torchtree_gb300.patterns import CompressedAlignment

    rng = np.random.default_rng(7)
    topo = synthetic.yule_topology(T, rng)
    aln = CompressedAlignment(rng.integers(0, 5, (T, N)).astype(np.uint8), np.vstack([np.eye(4), np.ones((1, 4))]),
                              rng.integers(1, 4, N), np.zeros((T, 0), np.uint8))
    lik = PhyloLikelihood(topo, aln, 4, K, batch=B, precision="f64")
    leaves = (_leaf(rng.exponential(0.1, (B, 2 * T - 3))), _leaf(rng.gamma(2.0, 1.0, (B, 6))),
              _leaf(rng.dirichlet(5.0 * np.ones(4), B)), _leaf(rng.uniform(0.3, 1.5, (B, 1))))
    compose = {"weibull": site_models._weibull, "gamma": site_models._gamma}[site]

    def fused(bl, exch, pi, shape):
        rates, props = getattr(site_models, site + "_rates")(shape, K)
        lnl = lik(bl, sub.gtr_q(exch, pi), pi, rates, props)
        assert type(lnl.grad_fn).__name__.startswith("EvaluateLikelihood")
        return lnl

    def separate(bl, exch, pi, shape):
        rates, props = compose(shape, K)
        return lik.evaluate_rate_matrix(sub.normalise(sub._general(exch, pi, 4), pi), pi, lik.node_branch_lengths(bl),
                                        rates, props, pi)

    return fused, separate, leaves


@pytest.mark.parametrize("site", ["weibull", "gamma"])
def test_gradients_with_a_graph(site):
    fused, separate, leaves = _model(site)
    plain = torch.autograd.grad(fused(*leaves).sum(), leaves)
    firsts, seconds = [], []
    for f in (fused, separate):
        first = torch.autograd.grad(f(*leaves).sum(), leaves, create_graph=True)
        firsts.append(first)
        seconds.append(torch.autograd.grad(sum((t * t).sum() for t in first), leaves[1:]))
    for a, b, c in zip(plain, *firsts):
        _close(b, a)
        _close(b, c)
    for a, b in zip(*seconds):
        _close(a, b)


def test_rate_matrix_gradient_where_frequencies_depend_on_rates():
    from torchtree_gb300 import substitution as sub

    rng = np.random.default_rng(3)
    r = _leaf(rng.gamma(2.0, 1.0, (B, 6)))
    g = torch.tensor(rng.normal(size=(B, 4, 4)), device="cuda")
    outs = []
    for fn in (lambda x, p: sub.general_symmetric_q(x, p, 4), lambda x, p: sub._general(x, p, 4)):
        first = torch.autograd.grad(fn(r, torch.softmax(r[:, :4], -1)), r, g, create_graph=True)[0]
        outs.append((first, torch.autograd.grad((first * first).sum(), r)[0]))
    for a, b in zip(*outs):
        _close(a, b)


@pytest.mark.parametrize("site", ["weibull", "gamma"])
def test_batches_of_incoming_gradients(site):
    """``is_grads_batched`` and the vectorised Jacobian, with and without a graph."""
    fused, separate, leaves = _model(site)
    eye = torch.eye(B, dtype=torch.float64, device="cuda")
    outs = [torch.autograd.grad(f(*leaves), leaves, eye, is_grads_batched=True) for f in (fused, separate)]
    for a, b in zip(*outs):
        assert not a.requires_grad
        _close(a, b)
    for graph in (False, True):
        outs = [torch.autograd.functional.jacobian(f, leaves, vectorize=True, create_graph=graph)
                for f in (fused, separate)]
        for a, b in zip(*outs):
            _close(a, b)
