"""Workloads for timing the likelihood engine through its public entry points.

Each case is one call that a sampler or an optimiser makes over and over: the
log-likelihood of a batch of parameter samples with its gradient
(HMC, ADVI, MAP), the log-likelihood alone (Metropolis moves, model
evidence), or the time-tree prior with its gradient.  The topology and the
alignment stay on the device, as they do in a run; the parameters are new on
every call.  ``exact`` restates the same mathematics in 64-bit torch.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from torchtree_gb300 import site_models, substitution, synthetic
from torchtree_gb300.likelihood import PhyloLikelihood
from torchtree_gb300.patterns import CompressedAlignment
from torchtree_gb300.timetree import TimeTree

CATEGORIES = 4
STATES = {"gtr": 4, "hky": 4, "nonrev": 4, "protein": 20, "codon": 61}


def _likelihood(name, model, tips, patterns, batch, precision, site, gaps=0.01, grad=True):
    return {"name": name, "kind": "likelihood", "model": model, "tips": tips, "patterns": patterns, "batch": batch,
            "precision": precision, "site": site, "gaps": gaps, "grad": grad}


def _timetree(name, tips, batch):
    return {"name": name, "kind": "timetree", "tips": tips, "batch": batch}


def listed():
    return [
        # one HMC chain on an influenza-sized set (69 taxa, 238 patterns): launches and latency
        _likelihood("dna_t69_b1_f32", "gtr", 69, 238, 1, "f32", "weibull"),
        # the same at the plug-in's default precision
        _likelihood("dna_t69_b1_f64", "gtr", 69, 238, 1, "f64", "weibull"),
        # a Metropolis move: likelihood only, odd sizes
        _likelihood("dna_t137_b1_f32_value", "gtr", 137, 1373, 1, "f32", "gamma", grad=False),
        # an ADVI step with 64 samples, 500 taxa x 10,000 sites
        _likelihood("dna_t500_b64_f32", "hky", 500, 6584, 64, "f32", "gamma", gaps=0.0),
        # the benchmark's default: 1,000 taxa x 100,000 sites, 8 samples
        _likelihood("dna_t1000_b8_f32", "gtr", 1000, 81808, 8, "f32", "gamma", gaps=0.0),
        # the 64-bit drop-in on a mid-sized set
        _likelihood("dna_t500_b4_f64", "hky", 500, 6584, 4, "f64", "gamma"),
        # a non-reversible DNA model (matrix exponential instead of an eigen system), default precision
        _likelihood("nonrev_t87_b3_f64", "nonrev", 87, 611, 3, "f64", "weibull"),
        # amino acids, 200 taxa x 5,000 sites
        _likelihood("protein_t200_b4_f32", "protein", 200, 4246, 4, "f32", "gamma"),
        # codons, 200 taxa x 3,000 codons, 16 samples
        _likelihood("codon_t200_b16_f32", "codon", 200, 2608, 16, "f32", "gamma", gaps=0.0),
        # codons on a small set, default precision
        _likelihood("codon_t60_b1_f64", "codon", 60, 301, 1, "f64", "weibull"),
        # the time-tree prior of one chain, and of a large batch of samples
        _timetree("timetree_t69_b1", 69, 1),
        _timetree("timetree_t1000_b16384", 1000, 16384),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case over the ranges of the listed ones (never dearer than the largest)."""
    if rng.random() < 0.2:
        case = _timetree(None, _log_uniform(rng, 20, 1500), _log_uniform(rng, 1, 16384))
        while case["tips"] * case["batch"] > 16384 * 1000:
            case["batch"] //= 2
        del case["name"]
        return case
    model = rng.choice(("gtr", "gtr", "hky", "protein", "codon", "nonrev"))
    precision = "f64" if model == "nonrev" else rng.choice(("f32", "f32", "f64"))
    wide = STATES[model] > 4
    tips = _log_uniform(rng, 20, 200 if wide else 1000)
    patterns = _log_uniform(rng, 100, 5000 if wide else 80000)
    batch = _log_uniform(rng, 1, 16 if wide else 64)
    # per-type limits keep a drawn case below the largest listed one of its kind
    limit = {("gtr", "f32"): 4e8, ("hky", "f32"): 4e8, ("gtr", "f64"): 1.3e7, ("hky", "f64"): 1.3e7,
             ("nonrev", "f64"): 3e6, ("protein", "f32"): 6e6, ("protein", "f64"): 3e5, ("codon", "f32"): 8e6,
             ("codon", "f64"): 8e4}[model, precision]
    while tips * patterns * batch > limit:
        if batch > 1:
            batch -= max(1, batch // 3)
        elif patterns > 300:
            patterns -= patterns // 3
        else:
            tips -= tips // 3
    case = _likelihood(None, model, tips, patterns, batch, precision, rng.choice(("weibull", "gamma")),
                       gaps=rng.choice((0.0, 0.01, 0.05)), grad=rng.random() < 0.75)
    del case["name"]
    return case


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _topology(tips, seed):
    return synthetic.yule_topology(tips, np.random.default_rng(seed))


def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _parameters(case, seed):
    """Model parameters as a sampler holds them (64 bits, on the device): free
    branch lengths [b, 2T-3], rate parameters, frequencies, site-model shape."""
    rng = np.random.default_rng([seed, 1])
    b, T, S = case["batch"], case["tips"], STATES[case["model"]]
    mean = 0.01 if S == 4 else 0.05
    bl = rng.exponential(mean, 2 * T - 3)[None] * rng.lognormal(0.0, 0.1, (b, 2 * T - 3))
    if case["model"] == "gtr":
        exch = np.repeat(rng.dirichlet(np.ones(6))[None], b, 0)
    elif case["model"] == "hky":
        exch = rng.lognormal(1.0, 0.5, (1, 1)).repeat(b, 0)
    elif case["model"] == "nonrev":
        exch = np.repeat(rng.gamma(2.0, 0.5, 12)[None], b, 0)
    elif case["model"] == "protein":
        exch = np.repeat(rng.gamma(1.0, 1.0, 190)[None], b, 0)
    else:  # kappa, omega
        exch = np.repeat(np.array([[rng.lognormal(1.0, 0.5), rng.gamma(2.0, 0.25) + 0.02]]), b, 0)
    exch = exch * rng.lognormal(0.0, 0.05, exch.shape)
    if case["model"] == "codon":
        pi = synthetic.f3x4_np(rng.dirichlet(2.0 * np.ones(4), 3))
    else:
        pi = rng.dirichlet(4.0 * np.ones(S))
    shape = 0.5 * rng.lognormal(0.0, 0.1, (b, 1))
    dev = _device()
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    return {"bl": t(bl), "exch": t(exch), "pi": t(np.repeat(pi[None], b, 0)), "shape": t(shape)}


def _rate_matrix(case, p):
    """Unnormalised rate matrix [b,S,S] in plain torch."""
    S, exch, pi = STATES[case["model"]], p["exch"], p["pi"]
    b, dev = exch.shape[0], exch.device
    if case["model"] == "nonrev":
        q = exch.new_zeros(b, S, S)
        off = ~torch.eye(S, dtype=torch.bool, device=dev)
        q = q.masked_scatter(off.expand(b, S, S), exch)
        return q - torch.diag_embed(q.sum(-1))
    if case["model"] == "hky":
        one = torch.ones_like(exch)
        upper = torch.cat((one, exch, one, one, exch, one), -1)
    elif case["model"] == "codon":
        ts, syn, non = (m.to(dev) for m in _codon_masks())
        one = exch.new_ones(())
        upper = torch.where(ts, exch[:, :1], one) * torch.where(non, exch[:, 1:], one)
        del syn  # alpha = 1
    else:
        upper = exch
    iu = torch.triu_indices(S, S, 1, device=dev)
    r = exch.new_zeros(b, S, S).index_put((torch.arange(b, device=dev)[:, None], iu[0], iu[1]), upper)
    q = (r + r.transpose(-1, -2)) * pi.unsqueeze(-2)
    return q - torch.diag_embed(q.sum(-1))


@functools.lru_cache(maxsize=None)
def _codon_masks():
    """(transition, synonymous, non-synonymous) of every pair of sense codons,
    row-major upper triangle; only pairs one nucleotide apart are classed."""
    code = "KNKNTTTTRSRSIIMIQHQHPPPPRRRRLLLLEDEDAAAAGGGGVVVV*Y*YSSSS*CWCLFLF"
    sense = [i for i in range(64) if code[i] != "*"]
    ts, syn, non = [], [], []
    for x, i in enumerate(sense):
        for j in sense[x + 1:]:
            d = [(i >> s & 3, j >> s & 3) for s in (4, 2, 0) if (i >> s & 3) != (j >> s & 3)]
            one = len(d) == 1
            ts.append(one and set(d[0]) in ({0, 2}, {1, 3}))
            syn.append(one and code[i] == code[j])
            non.append(one and code[i] != code[j])
    return tuple(torch.tensor(m) for m in (ts, syn, non))


def _normalised(q, pi):
    return q / -(torch.diagonal(q, dim1=-2, dim2=-1) * pi).sum(-1)[:, None, None]


def _alignment(case, seed, topo, p):
    """Site patterns evolved down the tree under sample 0's parameters, with
    gap codes scattered over the tips; weights 1 or more, as compression gives."""
    T, N, S = case["tips"], case["patterns"], STATES[case["model"]]
    dev = _device()
    gen = torch.Generator(dev).manual_seed(seed * 1000003 + 17)
    q = _normalised(_rate_matrix(case, p), p["pi"])[0].float()
    rates = torch.as_tensor(synthetic.discrete_weibull_np(0.6, CATEGORIES), dtype=torch.float32, device=dev)
    bl = torch.cat((p["bl"][0], p["bl"].new_zeros(1))).float()
    cum = torch.linalg.matrix_exp(q * (bl[:, None, None, None] * rates[None, :, None, None])).cumsum(-1)
    cat = torch.randint(CATEGORIES, (N,), generator=gen, device=dev)
    kids = {int(v): (int(l), int(r)) for v, l, r in topo.postorder}
    state = torch.zeros(2 * T - 1, N, dtype=torch.int64, device=dev)
    state[2 * T - 2] = torch.multinomial(p["pi"][0].float(), N, replacement=True, generator=gen)
    level = [2 * T - 2]
    per = max(1, 120_000_000 // (N * S))
    while level:
        pairs = [(c, v) for v in level for c in kids[v]]
        for i in range(0, len(pairs), per):
            c = torch.tensor([x[0] for x in pairs[i:i + per]], device=dev)
            v = torch.tensor([x[1] for x in pairs[i:i + per]], device=dev)
            rows = cum[c[:, None], cat, state[v]]
            u = torch.rand(len(c), N, 1, generator=gen, device=dev)
            state[c] = (u > rows).sum(-1).clamp_(max=S - 1)
        level = [c for c, _ in pairs if c >= T]
    codes = state[:T].to(torch.uint8)
    if case["gaps"]:
        codes[torch.rand(T, N, generator=gen, device=dev) < case["gaps"]] = S
    table = np.vstack([np.eye(S), np.ones((1, S))]) if case["gaps"] else np.eye(S)
    w = 1 + np.random.default_rng([seed, 2]).geometric(0.6, N) // 2
    return CompressedAlignment(codes=codes.cpu().numpy(), table=table, weights=w.astype(np.int64),
                               columns=np.zeros((T, 0), dtype=np.uint8))


def _time_inputs(case, seed):
    T, b = case["tips"], case["batch"]
    rng = np.random.default_rng([seed, 3])
    topo = _topology(T, seed)
    times = rng.uniform(0.0, 5.0, T)
    lb = np.zeros(T - 1)
    for v, l, r in topo.postorder:
        lb[v - T] = max(times[l] if l < T else lb[l - T], times[r] if r < T else lb[r - T])
    dev = _device()
    gen = torch.Generator(dev).manual_seed(seed * 1000003 + 29)
    kw = dict(generator=gen, dtype=torch.float64, device=dev)
    x = 0.05 + 0.9 * torch.rand(b, T - 1, **kw)
    x[:, T - 2] = lb[T - 2] + 0.5 + 5.0 * torch.rand(b, **kw)
    theta = torch.exp(1.0 + 0.3 * torch.randn(b, **kw))
    gbl = 100.0 * torch.randn(b, 2 * T - 2, **kw)  # what a likelihood's gradient brings for the branch lengths
    return topo, times, lb, x, theta, gbl


def prepare(case, seed):
    if case["kind"] == "timetree":
        topo, times, _, x, theta, gbl = _time_inputs(case, seed)
        tree = TimeTree(topo.postorder, times)
        one = torch.ones(case["batch"], dtype=torch.float64, device=x.device)
        return {"case": case, "tree": tree, "x": x.requires_grad_(), "theta": theta.requires_grad_(), "gbl": gbl,
                "one": one}
    topo = _topology(case["tips"], seed)
    p = _parameters(case, seed)
    aln = _alignment(case, seed, topo, p)
    lik = PhyloLikelihood(topo, aln, STATES[case["model"]], CATEGORIES, batch=case["batch"],
                          precision=case["precision"])
    lik.rescale = True  # a chain that has met an underflow, or always in 32 bits
    if case["grad"]:
        for t in p.values():
            t.requires_grad_()
    return {"case": case, "lik": lik, "p": p}


# ------------------------------------------------------------------- calls
def run(state):
    case = state["case"]
    if case["kind"] == "timetree":
        h, bl, ld = state["tree"].ratio_transform(state["x"])
        lp = state["tree"].constant_coalescent(h, state["theta"])
        gx, gth = torch.autograd.grad((lp + ld, bl), (state["x"], state["theta"]), (state["one"], state["gbl"]))
        return {"heights": h.detach(), "branches": bl.detach(), "log_det": ld.detach(), "log_prior": lp.detach(),
                "d_ratios": gx, "d_theta": gth}
    lik, p = state["lik"], state["p"]
    bl, exch, pi, shape = p["bl"], p["exch"], p["pi"], p["shape"]
    with torch.set_grad_enabled(case["grad"]):
        make = site_models.gamma_rates if case["site"] == "gamma" else site_models.weibull_rates
        rates, probs = make(shape, CATEGORIES)
        if case["model"] == "nonrev":
            q = substitution.normalise(_rate_matrix(case, p), pi)
            lnl = lik.evaluate_general(q, lik.node_branch_lengths(bl), rates, probs, pi)
        else:
            if case["model"] == "gtr":
                q = substitution.gtr_q(exch, pi)
            elif case["model"] == "hky":
                q = substitution.hky_q(exch, pi)
            elif case["model"] == "protein":
                q = substitution.general_symmetric_q(exch, pi, 20)
            else:
                q = substitution.mg94_q(torch.ones_like(exch[:, :1]), exch[:, 1:], exch[:, :1], pi)
            lnl = lik(bl, q, pi, rates, probs)
        if not case["grad"]:
            return {"lnl": lnl}
        g = torch.autograd.grad(lnl.sum(), (bl, exch, pi, shape))
    return {"lnl": lnl.detach(), "d_branches": g[0], "d_rates": g[1], "d_frequencies": g[2], "d_shape": g[3]}


def work(case):
    """Bytes: inputs read and outputs written once.  Operations: an internal
    child takes one S x S product per pattern and category in the post-order and
    two more in the adjoint (outside partial, gradient); a tip child is a column
    of its matrix (and a column sum of the gradient); plus the S products that
    join two children."""
    T, b = case["tips"], case["batch"]
    if case["kind"] == "timetree":
        return {"bytes": 8 * b * (7 * (T - 1) + 5), "flops": b * (T - 1) * 30}
    S, K, N, B = STATES[case["model"]], CATEGORIES, case["patterns"], 2 * T - 2
    n_exch = {"gtr": 6, "hky": 1, "nonrev": 12, "protein": 190, "codon": 2}[case["model"]]
    params = b * (B + n_exch + S + 1)
    passes = 3 if case["grad"] else 1
    per_site = (T - 2) * 2 * S * S * passes + (T - 1) * S * (1 + 3 * (passes > 1))
    matrices = b * B * K * 2 * S * S * S * passes
    return {"bytes": T * N + 8 * N + 8 * params * (2 if case["grad"] else 1) + 8 * b,
            "flops": b * K * N * per_site + matrices}


# ------------------------------------------------------------ 64-bit values
def _gamma_quantiles(shape):
    """Gamma(shape, 1) quantiles / shape at (2i+1)/(2K) [b,K], differentiable in shape:
    bisection and Newton on the series x^a e^-x sum_n x^n / Gamma(a+n+1)."""
    q = (2.0 * torch.arange(CATEGORIES, dtype=torch.float64, device=shape.device) + 1.0) / (2.0 * CATEGORIES)

    def cdf(a, x):
        n = torch.arange(200, dtype=torch.float64, device=x.device)
        terms = n * x.log().unsqueeze(-1) - torch.lgamma(a.unsqueeze(-1) + n + 1.0)
        return torch.exp(a * x.log() - x) * torch.exp(terms).sum(-1)

    def pdf(a, x):
        return torch.exp((a - 1.0) * x.log() - x - torch.lgamma(a))

    with torch.no_grad():
        lo = torch.full((shape.shape[0], CATEGORIES), -300.0, dtype=torch.float64, device=shape.device)
        hi = torch.full_like(lo, math.log(60.0))
        for _ in range(80):
            mid = 0.5 * (lo + hi)
            below = cdf(shape, mid.exp()) < q
            lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
        x = (0.5 * (lo + hi)).exp()
        for _ in range(3):
            x = x - (cdf(shape, x) - q) / pdf(shape, x)
        slope = pdf(shape, x)
    x = x - (cdf(shape, x) - q) / slope  # value x, derivative -(dF/da)/pdf
    return x / shape


def _exact_likelihood(case, seed):
    topo = _topology(case["tips"], seed)
    p = _parameters(case, seed)
    aln = _alignment(case, seed, topo, p)
    T, N, S, K, b = case["tips"], case["patterns"], STATES[case["model"]], CATEGORIES, case["batch"]
    dev = p["bl"].device
    codes = torch.as_tensor(aln.codes, device=dev).long()
    table = torch.as_tensor(aln.table, dtype=torch.float64, device=dev)
    weights = torch.as_tensor(aln.weights, dtype=torch.float64, device=dev)
    out = {k: [] for k in ("lnl", "bl", "exch", "pi", "shape")}
    group = max(1, min(b, (1 << 22) // (S * S * S)))  # samples at once
    chunk = max(64, min(N, 30_000_000_000 // (8 * 8 * T * K * S * group)))
    for s0 in range(0, b, group):
        leaf = {k: t[s0:s0 + group].detach().clone().requires_grad_(case["grad"]) for k, t in p.items()}
        g = leaf["bl"].shape[0]
        if case["site"] == "gamma":
            rates = _gamma_quantiles(leaf["shape"])
        else:
            u = (2.0 * torch.arange(K, dtype=torch.float64, device=dev) + 1.0) / (2.0 * K)
            rates = torch.pow(-torch.log(1.0 - u), 1.0 / leaf["shape"])
        rates = rates / rates.mean(-1, keepdim=True)
        q = _normalised(_rate_matrix(case, leaf), leaf["pi"])
        bl = torch.cat((leaf["bl"], leaf["bl"].new_zeros(g, 1)), -1)
        mats = torch.linalg.matrix_exp(q[:, None, None] * (bl[:, :, None] * rates[:, None])[..., None, None])
        cut = mats.detach().requires_grad_(case["grad"])  # gradients of all chunks gather here
        lnl = leaf["bl"].new_zeros(g)
        for n0 in range(0, N, chunk):
            part = _prune(topo, cut, leaf["pi"], codes[:, n0:n0 + chunk], table, weights[n0:n0 + chunk])
            lnl += part.detach()
            if case["grad"]:
                part.sum().backward()
            del part
        out["lnl"].append(lnl)
        if case["grad"]:
            mats.backward(cut.grad)
            for k, t in leaf.items():
                out[k].append(t.grad)
        del mats, cut
    if not case["grad"]:
        return {"lnl": torch.cat(out["lnl"])}
    r = {k: torch.cat(v) for k, v in out.items()}
    return {"lnl": r["lnl"], "d_branches": r["bl"], "d_rates": r["exch"], "d_frequencies": r["pi"],
            "d_shape": r["shape"]}


def _prune(topo, mats, pi, codes, table, weights):
    """Felsenstein pruning of one chunk of patterns, [g] log-likelihoods."""
    T = topo.tip_count
    part, scale = {}, 0.0

    def up(c):  # P_c x_c: [g,K,S,n]
        x = part.pop(c) if c >= T else table[codes[c]].T
        return mats[:, c] @ x

    for v, l, r in ((int(a), int(b), int(c)) for a, b, c in topo.postorder):
        x = up(l) * up(r)
        m = x.detach().amax((1, 2), keepdim=True)
        part[v] = x / m
        scale = scale + m.log()[:, 0, 0]
    site = (part[2 * T - 2] * pi[:, None, :, None]).sum(2).mean(1)  # equal category weights
    return ((site.log() + scale) * weights).sum(-1)


def _exact_timetree(case, seed):
    topo, times, lb, x, theta, gbl = _time_inputs(case, seed)
    T, b = case["tips"], case["batch"]
    dev = x.device
    x.requires_grad_()
    theta.requires_grad_()
    t = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    kids = {int(v): (int(l), int(r)) for v, l, r in topo.postorder}
    level, heights, order, ld = [2 * T - 2], [x[:, T - 2:]], [2 * T - 2], 0.0
    while True:
        pairs = [(c, i) for i, v in enumerate(level) for c in kids[v] if c >= T]
        if not pairs:
            break
        own = [c - T for c, _ in pairs]
        low = t(lb[own])
        span = heights[-1][:, [i for _, i in pairs]] - low
        heights.append(low + x[:, own] * span)
        ld = ld + span.log().sum(-1)
        level = [c for c, _ in pairs]
        order += level
    h = torch.cat(heights, -1)[:, np.argsort(order)]
    if not torch.is_tensor(ld):
        ld = x.new_zeros(b)
    every = torch.cat((t(times).expand(b, T), h), -1)
    parent = np.zeros(2 * T - 2, dtype=np.int64)
    for v, (l, r) in kids.items():
        parent[l] = parent[r] = v
    bl = every[:, parent] - every[:, :-1]
    times_sorted, idx = torch.sort(every, dim=-1, stable=True)
    lineages = torch.where(idx < T, 1.0, -1.0).to(torch.float64).cumsum(-1)[:, :-1]
    area = (0.5 * lineages * (lineages - 1.0) * (times_sorted[:, 1:] - times_sorted[:, :-1])).sum(-1)
    lp = -area / theta - (T - 1) * theta.log()
    one = torch.ones_like(lp)
    gx, gth = torch.autograd.grad((lp + ld, bl), (x, theta), (one, gbl))
    return {"heights": h.detach(), "branches": bl.detach(), "log_det": ld.detach(), "log_prior": lp.detach(),
            "d_ratios": gx, "d_theta": gth}


def exact(case, seed):
    return _exact_timetree(case, seed) if case["kind"] == "timetree" else _exact_likelihood(case, seed)
