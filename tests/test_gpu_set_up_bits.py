"""The one-launch category rates and rate matrices, and the normalisation inside the
one-call evaluation, equal the compositions of tensor operations to the last bit: FP32
transition matrices are rounded from them.  Category and state counts that are powers of
two and not, batches on both sides of a warp and a CTA."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _t(a):
    return torch.tensor(a, dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("kind", ["weibull", "gamma"])
def test_rates(kind):
    from torchtree_gb300 import site_models

    rng = np.random.default_rng(1)
    fn, compose = getattr(site_models, kind + "_rates"), getattr(site_models, "_" + kind)
    for k in range(1, 33):
        for b in (1, 3, 33, 300):
            shape = _t(rng.uniform(0.2, 3.0, (b, 1)))
            (rates, props), (want, want_p) = fn(shape, k), compose(shape, k)
            assert torch.equal(rates, want) and torch.equal(props, want_p), (k, b)


@pytest.mark.parametrize("b", [1, 3, 40, 300])
def test_rate_matrices(b):
    from torchtree_gb300 import substitution as sub

    rng = np.random.default_rng(b)
    for S in (2, 3, 4, 5, 7, 16, 20, 31, 32, 33, 61, 64):
        r, pi = _t(rng.gamma(1.0, 1.0, (b, S * (S - 1) // 2))), _t(rng.dirichlet(5.0 * np.ones(S), b))
        assert torch.equal(sub.general_symmetric_q(r, pi, S), sub._general(r, pi, S)), S
    kappa, pi = _t(rng.uniform(0.5, 8.0, (b, 1))), _t(rng.dirichlet(5.0 * np.ones(4), b))
    assert torch.equal(sub.hky_q(kappa, pi), sub._hky(kappa, pi))
    alpha, beta, pi = *(_t(rng.uniform(0.1, 3.0, (b, 1))) for _ in range(2)), _t(rng.dirichlet(5.0 * np.ones(61), b))
    assert torch.equal(sub.mg94_q(alpha, beta, kappa, pi), sub._mg94(alpha, beta, kappa, pi, sub.UNIVERSAL_CODE))


@pytest.mark.parametrize("b", [1, 3, 40])
@pytest.mark.parametrize("S", [2, 3, 4, 5, 20, 33, 61, 64])
def test_normalised_matrix_and_eigen_system_of_an_evaluation(S, b):
    from torchtree_gb300 import substitution as sub, synthetic
    from torchtree_gb300.engine import LikelihoodEngine

    rng = np.random.default_rng(S + b)
    topo = synthetic.yule_topology(4, rng)
    eng = LikelihoodEngine(topo.postorder, 4, S, 1, rng.integers(0, S, (4, 8)).astype(np.uint8), np.eye(S), np.ones(8),
                           batch=b, precision="f64")
    pi = _t(rng.dirichlet(5.0 * np.ones(S), b))
    q = sub._general(_t(rng.gamma(1.0, 1.0, (b, S * (S - 1) // 2))), pi, S)
    one = torch.ones(b, 1, dtype=torch.float64, device="cuda")
    _, work = eng.evaluate(q, pi, _t(rng.exponential(0.1, (b, 5))), one, one, True, False)
    qn = sub.normalise(q, pi)
    assert torch.equal(work[:q.numel()].view_as(q), qn)
    for got, want in zip(eng.evaluation_parts(work), sub.device_eigen(qn, pi)):
        assert torch.equal(got, want)


def test_numbers_that_are_not_finite():
    """NaN and infinities go where the compositions put them, zeros keep their sign."""
    from torchtree_gb300 import site_models, substitution as sub

    rng = np.random.default_rng(5)
    odd = [np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-310]
    r, pi = rng.gamma(1.0, 1.0, (12, 6)), rng.dirichlet(5.0 * np.ones(4), 12)
    for i, v in enumerate(odd):
        r[i, i % 6] = v
        pi[6 + i, i % 4] = v
    for got, want in ((sub.gtr_q(_t(r), _t(pi)), sub._general(_t(r), _t(pi), 4)),
                      (sub.hky_q(_t(r[:, :1]), _t(pi)), sub._hky(_t(r[:, :1]), _t(pi)))):
        np.testing.assert_array_equal(got.cpu().numpy(), want.cpu().numpy())
        np.testing.assert_array_equal(np.signbit(got.cpu().numpy()), np.signbit(want.cpu().numpy()))
    shape = _t(np.array(odd + [-1.0, 1e300, 1e-3])[:, None])
    for kind in ("weibull", "gamma"):
        for k in (1, 4, 6):
            rates, _ = getattr(site_models, kind + "_rates")(shape, k)
            np.testing.assert_array_equal(rates.cpu().numpy(), getattr(site_models, "_" + kind)(shape, k)[0].cpu().numpy())
