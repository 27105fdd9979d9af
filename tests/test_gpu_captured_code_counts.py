"""A captured pass of a wide-state plan follows tips set anew with another number of codes:
across the limit of the 20-state tables (64), and for FP32 codon plans from the small table
of tip products (64) past it and past the large one's (128), with and without a table in
the captured pass.  The replay against the CPU oracle at the repository's parity bounds
(FP64 1e-10, FP32 lnL 1e-6 and gradients 1e-4)."""
import numpy as np
import pytest
import torch

from oracle import likelihood as OL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,precision,T,N,K,b,counts", [
    (20, "f32", 9, 300, 2, 1, (21, 60, 90, 20)), (20, "f64", 9, 300, 2, 1, (21, 60, 90, 20)),
    (20, "f32", 9, 300, 2, 1, (80, 23)), (61, "f64", 7, 100, 2, 1, (61, 66, 140)),
    (61, "f32", 7, 100, 2, 1, (61, 66, 140)), (61, "f32", 11, 704, 4, 9, (62, 70, 140, 61)),
    (61, "f32", 11, 704, 4, 9, (100, 64, 140))])
def test_captured_pass_follows_other_code_counts(S, precision, T, N, K, b, counts):
    from torchtree_gb300 import _native, synthetic
    from torchtree_gb300.engine import LikelihoodEngine

    rng = np.random.default_rng(S + N + counts[0])
    topo = synthetic.yule_topology(T, rng)
    w = rng.integers(1, 4, N).astype(np.float64)
    mats = 0.9 * np.eye(S) + 0.1 * rng.dirichlet(0.5 * np.ones(S), size=(b, 2 * T - 2, K, S)) + 1e-3
    props, freqs = rng.dirichlet(np.ones(K), size=b), rng.dirichlet(np.ones(S), size=b)
    sets = []
    for count in counts:
        table = np.concatenate([np.eye(S), (rng.random((count - S, S)) < 0.4) + 0.0])
        table[S:, 0] = 1.0
        sets.append((table, rng.integers(0, count, (T, N)).astype(np.uint8)))
    dev = torch.device("cuda")
    pd, fd = torch.tensor(props, device=dev), torch.tensor(freqs, device=dev)
    eng = LikelihoodEngine(topo.postorder, T, S, K, sets[0][1], sets[0][0], w, batch=b, precision=precision)
    eng.set_matrices(torch.tensor(mats, device=dev))

    def work():
        lnl = eng.log_likelihood(pd, fd, rescale=True, keep_partials=True)
        return [lnl, *eng.gradient(pd, fd, want_matrices=True)]

    work()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = work()
    t = lambda a: torch.tensor(a, dtype=torch.float64, requires_grad=True)  # noqa: E731
    tol = (1e-10, 1e-10) if precision == "f64" else (1e-6, 1e-4)
    for table, codes in sets:
        _native.check(eng.lib.tt_plan_set_tips(eng._plan, _native.ptr(codes), _native.ptr(np.ascontiguousarray(table)),
                                               table.shape[0], _native.ptr(w)))
        graph.replay()
        torch.cuda.synchronize()
        m, p, f = t(mats), t(props), t(freqs)
        tips = [torch.tensor(table[codes[i]].T) for i in range(T)]
        want = OL.treelikelihood_discrete_rescaled(tips + [None] * (T - 1), torch.tensor(w), topo.postorder_list(), m,
                                                   f.unsqueeze(-2), p[..., None, None]).reshape(-1)
        np.testing.assert_allclose(outs[0].cpu().numpy(), want.detach().numpy(), rtol=tol[0])
        for got, r in zip(outs[1:], torch.autograd.grad(want.sum(), (m, f, p))):
            r = r.numpy()
            np.testing.assert_allclose(got.cpu().numpy(), r, rtol=tol[1], atol=tol[1] * np.abs(r).max())
    assert eng.device_status() == 0
