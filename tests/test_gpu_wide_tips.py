"""Tips of wide-state plans: table or column look-ups in place of products, at
the code counts where the look-up gives way to the product (64 codes for the
20-state post-order's tables, 4 ambiguous codes for the others), pattern counts
around the tiles (128, 256 per CTA step, 32 in FP64 codon plans), 20 and fewer
states, 61 states; every mix of tip and internal children.  lnL, dlnL/dP,
dlnL/dpi and dlnL/dw against the CPU oracle's autograd.

Tolerances are the repository's parity bounds: FP64 1e-10 of the largest entry
(sums of at most 400 patterns x 61 states, 61 x 400 x 1.1e-16 = 3e-12), FP32 lnL
1e-6 and gradients 1e-4."""
import numpy as np
import pytest
import torch

from oracle import likelihood as OL

pytestmark = pytest.mark.gpu


def _codes(S, extra, rng):
    """The unit vectors and `extra` other rows: all states, sets of states, a weighted one."""
    rows = [np.eye(S)]
    for e in range(extra):
        row = np.ones(S) if e == 0 else (rng.random(S) < 0.4).astype(float)
        row[rng.integers(S)] = 1.0
        row[rng.integers(S)] = 1.0
        if e == 1:
            row = rng.random(S)
        rows.append(row[None])
    return np.concatenate(rows)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("S,N,K,b,extra", [(20, 1, 1, 1, 0), (20, 129, 4, 2, 1), (20, 257, 3, 1, 4), (20, 300, 2, 1, 5),
                                           (20, 384, 1, 1, 44), (20, 200, 2, 1, 60), (7, 130, 4, 1, 2),
                                           (5, 255, 2, 2, 70), (61, 1, 1, 1, 0), (61, 33, 2, 1, 1), (61, 129, 2, 1, 4),
                                           (33, 97, 1, 2, 5), (64, 64, 1, 1, 3)])
def test_tip_lookups_match_oracle(precision, S, N, K, b, extra):
    from torchtree_gb300 import synthetic
    from torchtree_gb300.engine import LikelihoodEngine

    T = 11
    rng = np.random.default_rng(1000 * S + N + extra)
    topo = synthetic.yule_topology(T, rng)
    table = _codes(S, extra, rng)
    codes = rng.integers(0, table.shape[0], (T, N)).astype(np.uint8)
    codes[::3] %= S  # tips without ambiguity too
    w = rng.integers(0, 4, N).astype(np.float64)
    mats = 0.9 * np.eye(S) + 0.1 * rng.dirichlet(0.5 * np.ones(S), size=(b, 2 * T - 2, K, S)) + 1e-3
    props, freqs = rng.dirichlet(np.ones(K), size=b), rng.dirichlet(np.ones(S), size=b)

    t = lambda a: torch.tensor(a, dtype=torch.float64, requires_grad=True)  # noqa: E731
    m, p, f = t(mats), t(props), t(freqs)
    tips = [torch.tensor(table[codes[i]].T) for i in range(T)]
    want = OL.treelikelihood_discrete_rescaled(tips + [None] * (T - 1), torch.tensor(w), topo.postorder_list(), m,
                                               f.unsqueeze(-2), p[..., None, None]).reshape(-1)
    ref = [want.detach().numpy()] + [x.numpy() for x in torch.autograd.grad(want.sum(), (m, f, p))]

    eng = LikelihoodEngine(topo.postorder, T, S, K, codes, table, w, batch=b, precision=precision)
    dev = torch.device("cuda")
    pd, fd = torch.tensor(props, device=dev), torch.tensor(freqs, device=dev)
    eng.set_matrices(torch.tensor(mats, device=dev))
    lnl = eng.log_likelihood(pd, fd, rescale=True, keep_partials=True)
    dP, dpi, dc = eng.gradient(pd, fd, want_matrices=True)
    tol = (1e-10, 1e-10) if precision == "f64" else (1e-6, 1e-4)
    np.testing.assert_allclose(lnl.cpu().numpy(), ref[0], rtol=tol[0])
    for got, r in zip((dP, dpi, dc), ref[1:]):
        np.testing.assert_allclose(got.cpu().numpy(), r, rtol=tol[1], atol=tol[1] * np.abs(r).max())
    if precision == "f64":  # without rescaling: the same value
        lnl2 = eng.log_likelihood(pd, fd, rescale=False)
        np.testing.assert_allclose(lnl2.cpu().numpy(), ref[0], rtol=1e-10)
    assert eng.device_status() == 0


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("S", [20, 61])
def test_captured_pass_follows_tips_set_anew(precision, S):
    """A pass captured before the plan's tips (none ambiguous) are replaced by others of as
    many codes, with 3 and then 6 ambiguous ones, and its matrices by others: the replay
    gives what a new plan of those tips and matrices gives (the same kernels: FP64 1e-12;
    FP32 1e-6 and 1e-5 of the largest entry, for shared sums in another order)."""
    from torchtree_gb300 import _native, synthetic
    from torchtree_gb300.engine import LikelihoodEngine

    T, N, K = 9, 400, 2
    rng = np.random.default_rng(S)
    topo = synthetic.yule_topology(T, rng)
    tables = [np.concatenate([np.eye(S), np.eye(S)[:6 - e], _codes(S, e, rng)[S:]]) for e in (0, 3, 6)]
    codes = rng.integers(0, S + 6, (T, N)).astype(np.uint8)
    w = rng.integers(1, 4, N).astype(np.float64)
    dev = torch.device("cuda")
    pd = torch.tensor(rng.dirichlet(np.ones(K), size=1), device=dev)
    fd = torch.tensor(rng.dirichlet(np.ones(S), size=1), device=dev)
    mats = [torch.tensor(0.9 * np.eye(S) + 0.1 * rng.dirichlet(0.5 * np.ones(S), size=(1, 2 * T - 2, K, S)) + 1e-3,
                         device=dev) for _ in tables]

    def plan(table):
        return LikelihoodEngine(topo.postorder, T, S, K, codes, table, w, batch=1, precision=precision)

    def work(eng):
        lnl = eng.log_likelihood(pd, fd, rescale=True, keep_partials=True)
        return [lnl, *eng.gradient(pd, fd, want_matrices=True)]

    eng = plan(tables[0])
    eng.set_matrices(mats[0])
    work(eng)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = work(eng)
    for table, m in zip(tables, mats):
        host = np.ascontiguousarray(table)
        _native.check(eng.lib.tt_plan_set_tips(eng._plan, _native.ptr(codes), _native.ptr(host), host.shape[0],
                                               _native.ptr(w)))
        eng.set_matrices(m)
        graph.replay()
        fresh = plan(table)
        fresh.set_matrices(m)
        want = work(fresh)
        torch.cuda.synchronize()
        for i, (got, ref) in enumerate(zip(outs, want)):
            tol = 1e-12 if precision == "f64" else (1e-5 if i else 1e-6)
            np.testing.assert_allclose(got.cpu().numpy(), ref.cpu().numpy(), rtol=tol,
                                       atol=tol * float(ref.abs().max()))


@pytest.mark.parametrize("N,extra", [(704, 3), (769, 4), (768, 67), (700, 70)])
def test_codon_tip_product_tables_match_oracle(N, extra):
    """FP32 plans of 61 states large enough for the tips' tables of products: 64 codes and
    65 (the larger table), 128 codes and 131 (no table), whole and ragged tiles of 128
    patterns, two tips, one and none below a node.  Tolerances as above."""
    test_tip_lookups_match_oracle("f32", 61, N, 4, 9, extra)


def test_captured_codon_pass_rebuilds_tip_product_tables():
    """Matrices replaced between a captured large pass and its replay: the tables of tip
    products follow (the replay runs the same kernels as an eager pass: equal to 1e-12)."""
    from torchtree_gb300 import synthetic
    from torchtree_gb300.engine import LikelihoodEngine

    S, T, N, K, b = 61, 11, 800, 4, 9
    rng = np.random.default_rng(5)
    codes = rng.integers(0, S + 1, (T, N)).astype(np.uint8)
    eng = LikelihoodEngine(synthetic.yule_topology(T, rng).postorder, T, S, K, codes, _codes(S, 1, rng), np.ones(N),
                           batch=b, precision="f32")
    dev = torch.device("cuda")
    pd = torch.full((b, K), 1.0 / K, dtype=torch.float64, device=dev)
    fd = torch.full((b, S), 1.0 / S, dtype=torch.float64, device=dev)
    mats = [torch.tensor(rng.dirichlet(np.ones(S), size=(b, 2 * T - 2, K, S)), device=dev) for _ in range(2)]
    eng.set_matrices(mats[0])
    eng.log_likelihood(pd, fd)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = eng.log_likelihood(pd, fd)
    eng.set_matrices(mats[1])
    graph.replay()
    want = eng.log_likelihood(pd, fd)
    torch.cuda.synchronize()
    np.testing.assert_allclose(got.cpu().numpy(), want.cpu().numpy(), rtol=1e-12)
