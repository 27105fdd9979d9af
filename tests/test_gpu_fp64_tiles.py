"""FP64 4-state kernels at the edges of their tiles: one warp holds 32 / KP
patterns (KP = categories padded to 1, 2, 4 or 8), so category counts on both
sides of the padding, pattern counts around a tile and around the adjoint's
tiles per warp, tips with and without ambiguous codes, the smallest trees.
lnL, dlnL/dP, dlnL/dpi and dlnL/dw against the CPU oracle's autograd.

Tolerance: the repository's FP64 parity bound, 1e-10 of the largest entry (each
entry is a sum of at most N = 20,000 terms of one sign after at most 24 levels
of 4-term products: below 20,100 roundings of 1.1e-16, 2.3e-12).
"""
import numpy as np
import pytest
import torch

from oracle import likelihood as OL

pytestmark = pytest.mark.gpu

AMBIGUOUS = np.vstack([np.eye(4), np.ones((1, 4)), [[1, 0, 1, 0], [0, 1, 1, 1]], [[0.5, 0.1, 0.0, 0.25]]])


def _problem(T, N, K, b, codes_used, seed):
    from torchtree_gb300 import synthetic

    rng = np.random.default_rng(seed)
    topo = synthetic.yule_topology(T, rng) if T > 2 else None
    post = np.asarray(topo.postorder if topo is not None else [(2, 0, 1)], dtype=np.int32)
    codes = rng.integers(0, codes_used, size=(T, N)).astype(np.uint8)
    if codes_used > 4:  # some tips without ambiguity, so every mix of children occurs
        codes[::2] %= 4
    w = rng.integers(0, 4, N).astype(np.float64)
    mats = rng.dirichlet(0.5 * np.ones(4), size=(b, 2 * T - 2, K, 4)) + 0.02
    props = rng.dirichlet(np.ones(K), size=b)
    freqs = rng.dirichlet(np.ones(4), size=b)
    return post, codes, AMBIGUOUS[:codes_used], w, mats, props, freqs


def _oracle(post, codes, table, w, mats, props, freqs):
    t = lambda a: torch.tensor(a, dtype=torch.float64, requires_grad=True)  # noqa: E731
    m, p, f = t(mats), t(props), t(freqs)
    T = codes.shape[0]
    tips = [torch.tensor(table[codes[i]].T) for i in range(T)]
    lnl = OL.treelikelihood_discrete_rescaled(tips + [None] * (T - 1), torch.tensor(w),
                                              [tuple(int(x) for x in r) for r in post], m, f.unsqueeze(-2),
                                              p[..., None, None]).reshape(-1)
    g = torch.autograd.grad(lnl.sum(), (m, f, p))
    return [lnl.detach().numpy()] + [x.numpy() for x in g]


CASES = [(2, 1, 1, 1, 4), (3, 33, 1, 2, 8), (9, 64, 2, 1, 8), (9, 17, 3, 2, 8), (24, 7, 4, 1, 4), (24, 257, 4, 2, 8),
         (9, 129, 5, 1, 8), (9, 31, 8, 2, 8), (5, 20000, 4, 1, 5), (5, 5003, 8, 3, 4)]


@pytest.mark.parametrize("T,N,K,b,codes_used", CASES)
@pytest.mark.parametrize("rescale", [True, False])
def test_fp64_tiles_match_oracle(T, N, K, b, codes_used, rescale):
    from torchtree_gb300.engine import LikelihoodEngine

    post, codes, table, w, mats, props, freqs = _problem(T, N, K, b, codes_used, 31 * T + N + K)
    want = _oracle(post, codes, table, w, mats, props, freqs)
    eng = LikelihoodEngine(post, T, 4, K, codes, table, w, batch=b, precision="f64")
    dev = torch.device("cuda")
    p, f = torch.tensor(props, device=dev), torch.tensor(freqs, device=dev)
    eng.set_matrices(torch.tensor(mats, device=dev))
    lnl, site = eng.log_likelihood(p, f, rescale=rescale, keep_partials=True, site=True)
    for _ in range(2):  # the adjoint leaves the stored partials usable
        dP, dpi, dc = eng.gradient(p, f, want_matrices=True)
    for got, ref in zip((lnl, dP, dpi, dc), want):
        np.testing.assert_allclose(got.cpu().numpy(), ref, rtol=1e-10, atol=1e-10 * np.abs(ref).max())
    np.testing.assert_allclose((site.cpu().numpy() * w).sum(-1), want[0], rtol=1e-10)


def test_fp64_impossible_pattern():
    """A pattern of likelihood zero: lnL is -inf, its gradient terms are zero, as for the other patterns' sum."""
    from torchtree_gb300.engine import LikelihoodEngine

    post, codes, table, w, mats, props, freqs = _problem(9, 40, 4, 1, 4, 5)
    w[:] = 1.0
    codes = np.concatenate([codes, codes[:, :1]], 1)  # pattern 40: the last tip takes a state no path reaches
    leaf = int(codes.shape[0] - 1)
    mats[:, leaf, :, :, 3] = 0.0
    codes[leaf, :40] %= 3
    codes[leaf, 40] = 3
    dev = torch.device("cuda")
    out = []
    for n in (40, 41):
        eng = LikelihoodEngine(post, 9, 4, 4, codes[:, :n], table, np.ones(n), batch=1, precision="f64")
        eng.set_matrices(torch.tensor(mats, device=dev))
        p, f = torch.tensor(props, device=dev), torch.tensor(freqs, device=dev)
        lnl = eng.log_likelihood(p, f, rescale=True, keep_partials=True)
        out.append((float(lnl[0]), *[x.cpu().numpy() for x in eng.gradient(p, f, want_matrices=True)]))
    assert np.isfinite(out[0][0]) and out[1][0] == -np.inf
    for a, c in zip(out[0][1:], out[1][1:]):
        np.testing.assert_allclose(c, a, rtol=1e-12, atol=1e-12 * np.abs(a).max())
