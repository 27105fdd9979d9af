"""Inputs that the one-launch set-up and the one-call evaluation leave to the compositions
of tensor operations: equal to the composition's own values, bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("categories", [4.0, np.int64(4), 3.5])
def test_category_counts_that_are_no_ints(categories):
    from torchtree_gb300 import site_models

    shape = torch.tensor([[0.3], [0.7]], dtype=torch.float64, device="cuda")
    rates, props = site_models.weibull_rates(shape, categories)
    want, want_p = site_models._weibull(shape, categories)
    for a, b in ((rates, want), (props, want_p)):  # (3.5 has no mean rate of one: NaN either way)
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
    assert rates.shape == (2, 4)


def test_negated_views():
    """Tensors whose negation is still to be done (``imag`` of a conjugate is one): what
    their storage holds is not their value."""
    from torchtree_gb300 import site_models, substitution as sub, synthetic
    from torchtree_gb300.likelihood import PhyloLikelihood
    from torchtree_gb300.patterns import CompressedAlignment

    rng = np.random.default_rng(2)
    b, T, K = 2, 6, 3
    t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    lazy = lambda x: torch._neg_view(-x)  # noqa: E731
    shape, exch, pi = t(rng.uniform(0.3, 1.0, (b, 1))), t(rng.gamma(2.0, 1.0, (b, 6))), t(rng.dirichlet(np.ones(4), b))
    assert lazy(shape).is_neg()
    for make in (site_models.weibull_rates, site_models.gamma_rates):
        assert torch.equal(make(lazy(shape), K)[0], make(shape, K)[0])
    q = sub.gtr_q(exch, pi)
    assert torch.equal(sub.gtr_q(lazy(exch), pi), q) and torch.equal(sub.gtr_q(exch, lazy(pi)), q)
    rates, props = site_models.weibull_rates(shape, K)
    bl = t(rng.exponential(0.1, (b, 2 * T - 3)))
    topo = synthetic.yule_topology(T, rng)
    aln = CompressedAlignment(rng.integers(0, 4, (T, 30)).astype(np.uint8), np.eye(4), np.ones(30),
                              np.zeros((T, 0), np.uint8))
    lik = PhyloLikelihood(topo, aln, 4, K, batch=b, precision="f64")
    want = lik(bl, q, pi, rates, props)
    np.testing.assert_allclose(lik(lazy(bl), q, pi, rates, props).cpu().numpy(), want.cpu().numpy(), rtol=1e-12)
    np.testing.assert_allclose(lik(bl, lazy(q), pi, rates, props).cpu().numpy(), want.cpu().numpy(), rtol=1e-12)
    x = bl.clone().requires_grad_()
    one = torch.ones(b, dtype=torch.float64, device="cuda")
    grads = [torch.autograd.grad(lik(x, q, pi, rates, props), x, g)[0] for g in (one, lazy(one))]
    np.testing.assert_allclose(grads[1].cpu().numpy(), grads[0].cpu().numpy(), rtol=1e-12)
