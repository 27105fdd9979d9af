"""FP32 codon plans hold a table of tip products only where their passes use one: not for
alignments of fewer than six 128-pattern tiles, few products or more than 128 codes, not
beyond the gradient budget; and a plan whose pattern slabs grow gets it then.  Values do
not depend on it (the post-order's products either way, bit for bit)."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

S = 61


def _engine(T, N, K, b, codes=62):
    from torchtree_gb300 import synthetic
    from torchtree_gb300.engine import LikelihoodEngine

    rng = np.random.default_rng(N)
    topo = synthetic.yule_topology(T, rng)
    table = np.concatenate([np.eye(S), np.ones((codes - S, S))])
    return LikelihoodEngine(topo.postorder, T, S, K, rng.integers(0, codes, (T, N)).astype(np.uint8), table, np.ones(N),
                            batch=b, precision="f32")


def _plan_bytes(T, N, K, b):
    """Workspace of a plan before its tips are set."""
    from torchtree_gb300 import _native, synthetic

    lib = _native.load()
    post = np.ascontiguousarray(np.asarray(synthetic.yule_topology(T, np.random.default_rng(N)).postorder, np.int32))
    handle, n = ctypes.c_void_p(), ctypes.c_size_t()
    _native.check(lib.tt_plan_create(ctypes.byref(handle), T, post.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), S, K,
                                     N, b, _native.TT_PRECISION_F32))
    _native.check(lib.tt_plan_workspace_bytes(handle, ctypes.byref(n)))
    lib.tt_plan_destroy(handle)
    return n.value


@pytest.mark.parametrize("T,N,K,b,codes,capacity", [
    (11, 640, 4, 9, 62, 0),   # five tiles of patterns
    (11, 641, 4, 9, 62, 64),  # six
    (11, 641, 4, 7, 62, 0),   # 11 x 4 x 7 x 6 products
    (11, 704, 4, 9, 70, 0), (20, 1409, 4, 9, 70, 128),  # more than 64 codes: 8,192 products in 12 tiles of patterns
    (20, 1409, 4, 8, 70, 0), (20, 1409, 4, 9, 129, 0)])
def test_table_is_held_where_it_is_used(T, N, K, b, codes, capacity):
    assert _engine(T, N, K, b, codes).workspace_bytes - _plan_bytes(T, N, K, b) == b * T * K * capacity * 64 * 4


def test_table_stays_within_the_budget_and_follows_the_slabs(monkeypatch):
    from torchtree_gb300 import _native

    T, N, K, b = 11, 704, 4, 9
    table = b * T * K * 64 * 64 * 4
    dev = torch.device("cuda")
    rng = np.random.default_rng(0)
    mats = torch.tensor(0.9 * np.eye(S) + 0.1 * rng.dirichlet(np.ones(S), size=(b, 2 * T - 2, K, S)), device=dev)
    pd = torch.full((b, K), 1.0 / K, dtype=torch.float64, device=dev)
    fd = torch.full((b, S), 1.0 / S, dtype=torch.float64, device=dev)

    def value(eng):
        eng.set_matrices(mats)
        return eng.log_likelihood(pd, fd, rescale=True)

    free = _engine(T, N, K, b)
    want = value(free)
    monkeypatch.setenv("TT_SLAB_PATTERNS", "256")
    eng = _engine(T, N, K, b)
    before = eng.workspace_bytes
    np.testing.assert_allclose(value(eng).cpu().numpy(), want.cpu().numpy(), rtol=1e-12)  # sums by slab
    eng.set_option(_native.TT_OPT_SLAB_PATTERNS, 0)
    assert eng.workspace_bytes == free.workspace_bytes > before
    assert torch.equal(value(eng), want)
    monkeypatch.delenv("TT_SLAB_PATTERNS")
    low, high = 1, free.workspace_bytes  # the smallest budget without slabs: the pattern buffers alone
    while high - low > 1:
        mid = (low + high) // 2
        monkeypatch.setenv("TT_GRADIENT_BUDGET_BYTES", str(mid))
        if _engine(T, N, K, b).get_option(_native.TT_OPT_SLAB_PATTERNS):
            low = mid
        else:
            high = mid
    for budget, held in ((high, 0), (high + table - 1, 0), (high + table, table)):
        monkeypatch.setenv("TT_GRADIENT_BUDGET_BYTES", str(budget))
        eng = _engine(T, N, K, b)
        assert eng.workspace_bytes == free.workspace_bytes - table + held
        assert torch.equal(value(eng), want)
