"""Eigen systems in batches on both sides of the rule for the first sweeps' CTAs (76 matrices
of more than 32 states), at the state counts where the kernels change (5 with a dummy player,
32, 33, 64) and odd ones: one matrix's system does not depend on the batch it is in, bit for
bit (each matrix is a cluster's own; a row of the eigenvectors is one warp's own), and
U diag(lambda) W is Q, U W the identity (bounds as for the solver's LAPACK comparison)."""
import numpy as np
import pytest
import torch

from test_model_setup import _random_reversible

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,b", [(5, 77), (20, 160), (31, 3), (32, 2), (33, 76), (33, 77), (61, 2), (61, 90), (64, 78)])
def test_eigen_system_does_not_depend_on_the_batch(S, b):
    from torchtree_gb300 import substitution

    q, pi = (torch.tensor(x, device="cuda") for x in _random_reversible(np.random.default_rng(S + b), b, S))
    lam, u, w = substitution.device_eigen(q, pi)
    eye = torch.eye(S, dtype=torch.float64, device="cuda")
    assert float((u @ w - eye).abs().max()) <= 1e-12
    recon = u @ torch.diag_embed(lam) @ w
    assert float(((recon - q).abs().amax((-1, -2)) / q.abs().amax((-1, -2))).max()) <= 1e-11
    for i in (0, b // 2, b - 1):
        one = substitution.device_eigen(q[i:i + 1], pi[i:i + 1])
        assert all(torch.equal(x[i], y[0]) for x, y in zip((lam, u, w), one)), i
