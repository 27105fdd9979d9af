"""Time-tree kernels where their sort, merge and product can go wrong: tip
counts around the sort's padding (8 heights per thread, 256 at least), heights
closer than the sort key resolves, heights tied with each other and with tips,
negative and signed-zero times, spans that a log|J| product must not swallow.

Tolerance 1e-12 relative to the largest entry, the repository's bound for these
kernels (sums of at most 8,191 terms: 8,191 x 1.1e-16 = 9e-13)."""
import numpy as np
import pytest
import torch

from oracle import timetree as OT

pytestmark = pytest.mark.gpu


def _tree(T, times, seed):
    from torchtree_gb300 import synthetic
    from torchtree_gb300.timetree import TimeTree

    topo = synthetic.yule_topology(T, np.random.default_rng(seed))
    return topo, TimeTree(topo.postorder, times)


def _close(got, want):
    got, want = got.detach().cpu().numpy(), want.detach().numpy()
    np.testing.assert_allclose(got, want, rtol=1e-12, atol=1e-12 * np.abs(want).max())


def _coalescent(times, tree, h, theta):
    """Value and d/dtheta against the oracle; d/dheight against its definition,
    (C(l after, 2) - C(l before, 2)) / theta with tied events in node order (the
    oracle's argsort leaves the order of ties open, which the value does not see)."""
    hd, td = h.cuda().requires_grad_(), theta.cuda().requires_grad_()
    lp = tree.constant_coalescent(hd, td)
    tc = theta.clone().requires_grad_()
    want = OT.constant_coalescent(list(times), h, tc)
    _close(lp, want)
    gh, gth = torch.autograd.grad(lp.sum(), (hd, td))
    _close(gth, torch.autograd.grad(want.sum(), tc)[0])
    T = len(times)
    ref = np.empty((h.shape[0], T - 1))
    for i in range(h.shape[0]):
        every = np.concatenate([np.asarray(times), h[i].numpy()])
        order = np.lexsort((np.arange(2 * T - 1), every + 0.0))
        after = np.cumsum(np.where(order < T, 1.0, -1.0))
        pairs = 0.5 * after * (after - 1.0)
        pairs[-1] = 0.0
        diff = np.diff(np.concatenate([[0.0], pairs])) / float(theta[i])
        inner = order >= T
        ref[i, order[inner] - T] = diff[inner]
    _close(gh, torch.tensor(ref))


@pytest.mark.parametrize("T", [2, 3, 33, 256, 257, 258, 513, 1025, 4096])
def test_coalescent_at_the_sort_padding(T):
    rng = np.random.default_rng(T)
    times = np.round(rng.uniform(0.0, 2.0, T), 1)  # many tips share a time
    _, tree = _tree(T, times, T)
    h = torch.tensor(2.0 + rng.exponential(3.0, (3, T - 1)))
    h[1] = torch.round(h[1] * 4) / 4  # ties
    _coalescent(times, tree, h, torch.tensor(rng.lognormal(1.0, 0.3, 3)))


@pytest.mark.parametrize("step", [2.0 ** -52, 2.0 ** -44, 2.0 ** -41, 2.0 ** -38])
def test_coalescent_of_heights_closer_than_the_sort_key(step):
    T = 300
    rng = np.random.default_rng(3)
    times = rng.uniform(-1.0, 0.9, T)
    _, tree = _tree(T, times, 1)
    order = torch.tensor(rng.permutation(T - 1).astype(np.float64))
    h = torch.stack([1.0 + order * step, 1.0 - order * step, 1.0 + (order % 7) * step])
    theta = torch.tensor([0.5, 1.0, 2.0], dtype=torch.float64)
    hd = h.cuda().requires_grad_()
    lp = tree.constant_coalescent(hd, theta.cuda())
    (g,) = torch.autograd.grad(lp.sum(), hd)
    _close(lp, OT.constant_coalescent(list(times), h, theta))
    # by hand: the node of rank r (ties by index) has T - r lineages below it
    for i in range(3):
        rank = np.lexsort((np.arange(T - 1), h[i].numpy()))
        want = np.empty(T - 1)
        want[rank] = -(T - np.arange(T - 1) - 1.0) / float(theta[i])
        np.testing.assert_allclose(g[i].cpu().numpy(), want, rtol=1e-14)


def test_coalescent_signed_zero_and_negative_heights():
    times = np.array([0.0, -0.0, -2.0, 0.0, -1.0])
    _, tree = _tree(5, times, 2)
    h = torch.tensor([[-0.0, 0.0, 0.5, 1.0], [0.0, 0.25, 0.25, 3.0], [-1.0, -0.5, 0.0, 2.0]], dtype=torch.float64)
    _coalescent(times, tree, h, torch.tensor([1.0, 2.0, 0.1], dtype=torch.float64))


@pytest.mark.parametrize("T,scale", [(2, 1.0), (9, 1e-30), (70, 1e200), (700, 1e-3), (2000, 1e3)])
def test_log_det_product(T, scale):
    rng = np.random.default_rng(T)
    times = np.zeros(T)
    topo, tree = _tree(T, times, T)
    x = torch.tensor(rng.uniform(0.3, 0.9, (4, T - 1)))
    x[:, T - 2] = torch.tensor(scale * rng.uniform(0.5, 2.0, 4))
    h, bl, ld = tree.ratio_transform(x.cuda())
    hc, blc, ldc = OT.ratio_transform(topo.postorder_list(), list(times), x)
    for got, want in ((h, hc), (bl, blc), (ld, ldc)):
        _close(got, want)


def test_log_det_of_degenerate_spans():
    times = np.zeros(6)
    topo, tree = _tree(6, times, 4)
    x = torch.full((3, 5), 0.5, dtype=torch.float64)
    x[0, 4], x[1, 4], x[2, 4] = 0.0, -1.0, float("inf")  # log 0, log of a negative span, log inf
    _, _, ld = tree.ratio_transform(x.cuda())
    _, _, want = OT.ratio_transform(topo.postorder_list(), list(times), x)
    np.testing.assert_array_equal(ld.cpu().numpy(), want.numpy())
