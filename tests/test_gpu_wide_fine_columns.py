"""FP64 codon levels in tiles of 16 patterns beside levels in tiles of 32: the columns past
the last pattern that a wider tile reads belong to this evaluation, not to whatever the
buffers held.  An evaluation with NaN matrices first leaves NaN in every column that is
written; the next evaluation on the same plan has to match the CPU oracle at the
repository's FP64 bound of 1e-10 of the largest entry.  Pattern counts whose last tile
of 32 is at most half full (301, 45, 100), with the internal children's products kept and
formed again (TT_WIDE_STORE_PRODUCTS=0)."""
import numpy as np
import pytest
import torch

from oracle import likelihood as OL

pytestmark = pytest.mark.gpu


def _fine(nodes, bk, n):
    """The rule of ``wide_fine_level`` (csrc/tt_wide.cuh)."""
    waves = lambda tile: -(-nodes * bk * -(-n // tile) // 152)  # noqa: E731
    return 130 * waves(16) < 200 * waves(32)


def _mixed_nodes(topo, T, bk, n):
    """Internal children that the post-order writes in tiles of 16 and the adjoint reads in tiles of 32."""
    height, depth, kids = {}, {2 * T - 2: 0}, {}
    for v, l, r in np.asarray(topo.postorder).reshape(-1, 3):
        kids[int(v)] = (int(l), int(r))
        height[int(v)] = 1 + max(height.get(int(l), 0), height.get(int(r), 0))
    for v in sorted(kids, key=lambda x: -height[x]):
        for c in kids[v]:
            depth[c] = depth[v] + 1
    level = lambda of: {v: sum(of[x] == of[v] for x in kids) for v in kids}  # noqa: E731
    up, down = level(height), level(depth)
    return sum(c in kids and _fine(up[c], bk, n) and not _fine(down[v], bk, n) for v in kids for c in kids[v])


@pytest.mark.parametrize("products", [True, False])
@pytest.mark.parametrize("N,T,seed", [(301, 60, 1), (45, 90, 2), (100, 90, 3)])
def test_padding_columns_are_this_evaluations_own(products, N, T, seed, monkeypatch):
    from torchtree_gb300 import synthetic
    from torchtree_gb300.engine import LikelihoodEngine

    S, K = 61, 4
    rng = np.random.default_rng(seed)
    topo = synthetic.yule_topology(T, rng)
    assert _mixed_nodes(topo, T, K, N) > 0
    table = np.concatenate([np.eye(S), np.ones((1, S))])
    codes = rng.integers(0, S + 1, (T, N)).astype(np.uint8)
    w = rng.integers(1, 4, N).astype(np.float64)
    mats = 0.9 * np.eye(S) + 0.1 * rng.dirichlet(0.5 * np.ones(S), size=(1, 2 * T - 2, K, S)) + 1e-3
    props, freqs = rng.dirichlet(np.ones(K), size=1), rng.dirichlet(np.ones(S), size=1)
    t = lambda a: torch.tensor(a, dtype=torch.float64, requires_grad=True)  # noqa: E731
    m, p, f = t(mats), t(props), t(freqs)
    tips = [torch.tensor(table[codes[i]].T) for i in range(T)]
    want = OL.treelikelihood_discrete_rescaled(tips + [None] * (T - 1), torch.tensor(w), topo.postorder_list(), m,
                                               f.unsqueeze(-2), p[..., None, None]).reshape(-1)
    ref = [want.detach().numpy()] + [x.numpy() for x in torch.autograd.grad(want.sum(), (m, f, p))]

    if not products:
        monkeypatch.setenv("TT_WIDE_STORE_PRODUCTS", "0")
    eng = LikelihoodEngine(topo.postorder, T, S, K, codes, table, w, precision="f64")
    dev = torch.device("cuda")
    pd, fd = torch.tensor(props, device=dev), torch.tensor(freqs, device=dev)
    for values in (np.full_like(mats, np.nan), mats):
        eng.set_matrices(torch.tensor(values, device=dev))
        lnl = eng.log_likelihood(pd, fd, rescale=True, keep_partials=True)
        got = [lnl, *eng.gradient(pd, fd, want_matrices=True)]
    np.testing.assert_allclose(got[0].cpu().numpy(), ref[0], rtol=1e-10)
    for x, r in zip(got[1:], ref[1:]):
        np.testing.assert_allclose(x.cpu().numpy(), r, rtol=1e-10, atol=1e-10 * np.abs(r).max())
