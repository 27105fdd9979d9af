"""The chain from dlnL/dP to dlnL/dQ, dlnL/dt and dlnL/dr of FP64 plans over
every form of the divided difference: branch lengths from 1e-8 (differences of
rounding size) to 40 (beyond the series), repeated eigenvalues, state counts at
the edges of the 4 x 4 tiles and of the column slabs, category counts that do
not divide the runs.  The plan's own dlnL/dP is the cotangent of torch's matrix
exponential on the CPU, so that only this chain is compared (the short branches'
P entries, about 1e-8, carry a relative error of 1e-8 themselves).

Tolerance: products with U and W (condition sqrt(max pi / min pi), at most 8
here) over S <= 64 terms each way give 2 x 64 x 8^2 x 1.1e-16 = 9e-13 of the size
of the terms, sum of tau |G| (of |Q| |G| for the lengths and rates): 2e-12 of it.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,K,b,flat", [(4, 1, 2, False), (4, 3, 1, True), (4, 5, 3, False), (5, 2, 1, False),
                                        (20, 5, 2, False), (20, 4, 1, True), (21, 1, 1, False), (33, 3, 2, False),
                                        (61, 4, 1, False), (64, 2, 2, True)])
def test_rate_matrix_gradient_ranges(S, K, b, flat):
    from torchtree_gb300.engine import LikelihoodEngine
    from torchtree_gb300.substitution import device_eigen

    T, N = 5, 23
    rng = np.random.default_rng(100 * S + K)
    post = [(5, 0, 1), (6, 2, 3), (7, 5, 6), (8, 7, 4)]
    codes = rng.integers(0, S, (T, N)).astype(np.uint8)
    w = rng.integers(1, 4, N).astype(np.float64)
    exch = np.ones((S, S)) if flat else rng.gamma(1.0, 1.0, (S, S))
    exch = np.triu(exch, 1) + np.triu(exch, 1).T
    pi = np.full(S, 1.0 / S) if flat else rng.uniform(0.2, 1.0, S)
    pi /= pi.sum()
    q = exch * pi
    np.fill_diagonal(q, -q.sum(1))
    q /= -(np.diag(q) * pi).sum()
    bl = np.array([1e-8, 1e-3, 0.3, 2.0, 0.05, 40.0, 7.0, 1e-5]) * rng.uniform(0.5, 1.0, (b, 8))
    rates = rng.uniform(0.1, 2.0, (b, K))
    props = rng.dirichlet(np.ones(K), size=b)

    qs = np.repeat(q[None], b, 0)
    eng = LikelihoodEngine(post, T, S, K, codes, np.eye(S), w, batch=b, precision="f64")
    t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    qd, pid = t(qs), t(np.repeat(pi[None], b, 0))
    eig = (*device_eigen(qd, pid), t(bl), t(rates))
    eng.set_eigen(*eig)
    eng.log_likelihood(t(props), pid, keep_partials=True)
    G, _, _ = eng.gradient(t(props), pid, want_matrices=True)
    got = [x.cpu().numpy() for x in eng.rate_matrix_gradient(*eig)]

    # torch's backward squares a block matrix scaled to the cotangent's size too: take it of norm 1
    size = np.linalg.norm(G.cpu().numpy(), axis=(-2, -1))  # [b,B,K]
    tau = bl[:, :, None] * rates[:, None]
    a = torch.tensor(qs[:, None, None] * tau[..., None, None]).requires_grad_()
    unit = G.cpu() / torch.tensor(np.maximum(size, 1e-300))[..., None, None]
    y = torch.autograd.grad(torch.linalg.matrix_exp(a), a, unit)[0].numpy() * size[..., None, None]
    dtau = (y * q).sum((-2, -1))
    want = [(y * tau[..., None, None]).sum((1, 2)), (dtau * rates[:, None]).sum(-1), (dtau * bl[:, :, None]).sum(1)]
    qn = np.linalg.norm(q)
    bound = [(size * tau).sum((1, 2))[:, None, None], qn * (size * rates[:, None]).sum(-1),
             qn * (size * bl[:, :, None]).sum(1)]
    for g, ref, scale in zip(got, want, bound):
        assert (np.abs(g - ref) <= 2e-12 * scale).all(), (np.abs(g - ref) / scale).max()
