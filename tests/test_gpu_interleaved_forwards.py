"""A value-only evaluation (or a change of the matrices) between an evaluation and its
backward, on the same engine: the backward evaluates again, whichever route both took.
Equal to the gradient without the evaluation in between, bit for bit: the same kernels on
the same inputs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("S", [4, 20])
def test_value_between_forward_and_backward(precision, S):
    from torchtree_gb300 import substitution as sub, synthetic
    from torchtree_gb300.likelihood import PhyloLikelihood
    from torchtree_gb300.patterns import CompressedAlignment

    T, N, K, b = 7, 50, 2, 2
    rng = np.random.default_rng(S)
    topo = synthetic.yule_topology(T, rng)
    aln = CompressedAlignment(rng.integers(0, S, (T, N)).astype(np.uint8), np.eye(S), rng.integers(1, 4, N),
                              np.zeros((T, 0), np.uint8))
    lik = PhyloLikelihood(topo, aln, S, K, batch=b, precision=precision)
    lik.rescale = True
    t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731

    def inputs():
        pi = t(rng.dirichlet(5.0 * np.ones(S), b))
        q = sub._general(t(rng.gamma(1.0, 1.0, (b, S * (S - 1) // 2))), pi, S)
        return [t(rng.exponential(0.1, (b, 2 * T - 3))), q, pi, t(rng.uniform(0.2, 2.0, (b, K))),
                t(rng.dirichlet(np.ones(K), b))]

    def eigen(x):
        lam, u, w = sub.eigen_system(x[1], x[2])
        bls = lik.node_branch_lengths(x[0])
        return lam, u, w, bls

    routes = {
        "one call": lambda x: lik(*x[:5]),
        "rate matrix": lambda x: lik.evaluate_rate_matrix(sub.normalise(x[1], x[2]), x[2], lik.node_branch_lengths(x[0]),
                                                          x[3], x[4], x[2]),
        "eigen": lambda x: lik.evaluate_eigen(*eigen(x), x[3], x[4], x[2]),
        "general": lambda x: lik.evaluate_general(sub.normalise(x[1], x[2]), lik.node_branch_lengths(x[0]), x[3], x[4],
                                                  x[2]),
        "matrices": lambda x: lik.evaluate_matrices(x[5], x[4], x[2]),
    }
    first, second = inputs(), inputs()
    for x in (first, second):
        x.append(t(0.9 * np.eye(S) + 0.1 * rng.dirichlet(np.ones(S), size=(b, 2 * T - 2, K, S))))
    for name, run in routes.items():
        leaves = [x.clone().requires_grad_() for x in first]
        grad = lambda v: [g for g in torch.autograd.grad(v.sum(), leaves, allow_unused=True)]  # noqa: E731
        want = grad(run(leaves))
        for other, between in routes.items():
            lnl = run(leaves)
            between(second)
            for a, c in zip(grad(lnl), want):
                assert (a is None and c is None) or torch.equal(a, c), (name, other)
        lnl = run(leaves)
        lik.engine.set_matrices(second[5])
        for a, c in zip(grad(lnl), want):
            assert (a is None and c is None) or torch.equal(a, c), name
