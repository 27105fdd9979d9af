"""The one-call evaluation reports an eigen system that did not converge in the plan's status
word.  The matrix: after normalisation by frequencies of 1e35 its diagonal is of order 1e-36
and the rest 1e-46, which FP32 rotation angles round to 0 while the FP64 stopping rule
(1e-14 of the norm) does not: finite, and no sweep makes progress."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [4, 5, 40])  # the one-launch solver and both cluster shapes of the other
def test_unconverged_eigen_system_is_reported(S):
    from torchtree_gb300 import synthetic
    from torchtree_gb300.engine import LikelihoodEngine

    T, N = 5, 20
    rng = np.random.default_rng(S)
    topo = synthetic.yule_topology(T, rng)
    eng = LikelihoodEngine(topo.postorder, T, S, 1, rng.integers(0, S, (T, N)).astype(np.uint8), np.eye(S), np.ones(N),
                           precision="f64")
    t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    one, bl = t(np.ones((1, 1))), t(rng.exponential(0.1, (1, 2 * T - 3)))
    good = np.full((1, S, S), 1.0 / S) - np.eye(S)
    bad = np.full((1, S, S), 1e-10)
    bad[0, range(S), range(S)] = -1.0 - np.arange(S) / S
    assert eng.device_status() == 0
    eng.evaluate(t(bad), t(np.full((1, S), 1e35)), bl, one, one, True, False)
    assert eng.device_status(reset=True) == 2  # TT_ERR_UNSUPPORTED
    lnl, _ = eng.evaluate(t(good), t(np.full((1, S), 1.0 / S)), bl, one, one, True, False)
    assert eng.device_status() == 0 and bool(torch.isfinite(lnl).all())
