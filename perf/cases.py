"""What the library's speed is measured on.

One case is a stretch of work that a phylogenetics program asks of the library
through its Python entry points: proposals of an MCMC chain along one dirty
path or over the whole tree, for DNA and protein alignments, in both forms
(FP64 and FP32), alone or many chains at once, and a training step of the
delayed-acceptance surrogate.  Alignments are simulated from the seed down a
Yule tree, compressed to distinct patterns, as a program has them in hand.

Kinds of cases:

``path``
    eight proposals of a chain through ``GpuCalculator``: a random internal
    node gets a new height, the path from it to the root is evaluated and the
    log-likelihood read; the first six are rejected, the seventh is accepted
    and the eighth moves the node back (accepted), so that a pass ends in the
    state it began with.
``tree``
    one evaluation of the whole tree (a tree-scale or model move), accepted;
    with ``sites`` the per-pattern log-likelihoods are read too, as topology
    tests and model comparisons do.
``trait``
    the reference engine's own call order: transition matrices in,
    per-pattern log-likelihoods of every category out, accepted.
``batch``
    chains of several alignments evaluated by one ``Batch``: two steps, in
    each of which one chain in sixteen re-evaluates its whole tree and the
    others a path; all rejected.
``surrogate``
    loss and gradient of a minibatch of proposal pairs.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from aspartik_gb300.calculator import Batch, Calculator
from aspartik_gb300.schedule import Topology
from aspartik_gb300.surrogate import Surrogate

ROOT = 0xFFFFFFFF
PROPOSALS = 8


def listed():
    return [
        # the smallest configuration (16 taxa, 1,000 sites, HKY, one
        # category): every proposal of a small chain; latency only
        dict(name="dna_path_f32_16x910", kind="path", states=4, form="f32", taxa=16,
             patterns=910, categories=1),
        # the largest configuration (256 taxa, 20,000 sites, GTR + Gamma4):
        # nine of ten proposals of a chain are such paths
        dict(name="dna_path_f32_256x17764", kind="path", states=4, form="f32", taxa=256,
             patterns=17764, categories=4),
        # the drop-in FP64 form on the middle configuration (64 taxa, 10,000
        # sites, GTR + Gamma4)
        dict(name="dna_path_f64_64x7855", kind="path", states=4, form="f64", taxa=64,
             patterns=7855, categories=4),
        # whole-tree moves of the middle configuration
        dict(name="dna_tree_f32_64x7855", kind="tree", states=4, form="f32", taxa=64,
             patterns=7855, categories=4, sites=False),
        # whole-tree moves of the largest configuration (the benchmark's step)
        dict(name="dna_tree_f32_256x17764", kind="tree", states=4, form="f32", taxa=256,
             patterns=17764, categories=4, sites=False),
        # the same tree in the drop-in FP64 form, with its site values
        dict(name="dna_tree_f64_256x17764", kind="tree", states=4, form="f64", taxa=256,
             patterns=17764, categories=4, sites=True),
        # a calculator as the reference's engine drives one (one category per
        # calculator), on an alignment of odd sizes
        dict(name="dna_trait_f64_37x1147", kind="trait", states=4, form="f64", taxa=37,
             patterns=1147, categories=1),
        # protein, 128 taxa, 5,000 sites, Gamma4: whole-tree moves
        dict(name="aa_tree_f32_128x4989", kind="tree", states=20, form="f32", taxa=128,
             patterns=4989, categories=4, sites=False),
        # and the dirty paths of the same chain
        dict(name="aa_path_f32_128x4989", kind="path", states=20, form="f32", taxa=128,
             patterns=4989, categories=4),
        # protein in the FP64 form on a smaller alignment of odd sizes, with
        # its site values
        dict(name="aa_tree_f64_61x2003", kind="tree", states=20, form="f64", taxa=61,
             patterns=2003, categories=4, sites=True),
        # 32 chains: four alignments with a temperature ladder of eight each
        dict(name="dna_batch_32", kind="batch", alignments=4, chains=8, taxa=184,
             patterns=4832, categories=4),
        # a training step of the surrogate at the driver's sizes (minibatches
        # of 512 pairs, 14 inputs, three hidden layers of 256)
        dict(name="surrogate_512x256", kind="surrogate", pairs=512, inputs=14, hidden=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["path", "path", "tree", "tree", "tree", "trait", "batch", "surrogate"])
    if kind == "surrogate":
        return dict(kind=kind, pairs=_log(rng, 32, 1024), inputs=rng.randint(6, 31),
                    hidden=32 * rng.randint(2, 12))
    if kind == "batch":
        return dict(kind=kind, alignments=rng.randint(1, 4), chains=rng.randint(2, 8),
                    taxa=rng.randint(24, 184), patterns=_log(rng, 500, 4832),
                    categories=rng.choice([1, 4, 4]))
    if kind == "trait":
        return dict(kind=kind, states=4, form=rng.choice(["f64", "f64", "f32"]),
                    taxa=_log(rng, 8, 128), patterns=_log(rng, 300, 10000),
                    categories=rng.choice([1, 1, 4]))
    protein = rng.random() < 0.4
    form = rng.choice(["f32", "f32", "f64"])
    case = dict(kind=kind, states=20 if protein else 4, form=form)
    if protein:
        case.update(taxa=_log(rng, 12, 128 if form == "f32" else 64),
                    patterns=_log(rng, 200, 4989 if form == "f32" else 2500),
                    categories=rng.choice([1, 4, 4, 5]))
    else:
        case.update(taxa=_log(rng, 8, 256), patterns=_log(rng, 300, 17764),
                    categories=rng.choice([1, 2, 3, 4, 4, 4]))
    if kind == "tree":
        case["sites"] = form == "f64"
    return case


# ---------------------------------------------------------------------------
# inputs


def _yule(taxa, rng, root_height):
    """parents and heights of a Yule tree (leaves first, parents after their
    children, the root last)."""
    n = 2 * taxa - 1
    parents = np.full(n, ROOT, dtype=np.uint32)
    heights = np.zeros(n)
    live, t = list(range(taxa)), 0.0
    for new in range(taxa, n):
        t += rng.exponential(1.0 / len(live))
        for _ in range(2):
            k = int(rng.integers(len(live)))
            live[k], live[-1] = live[-1], live[k]
            parents[live.pop()] = new
        heights[new] = t
        live.append(new)
    return parents, heights * (root_height / t)


def _eigen(rates, pi):
    """V, V^-1 and the eigenvalues of the reversible rate matrix with mean
    rate 1, and the matrix itself."""
    n = pi.size
    R = np.zeros((n, n))
    R[np.triu_indices(n, 1)] = rates
    Q = (R + R.T) * pi[None, :]
    Q -= np.diag(Q.sum(axis=1))
    Q /= -(np.diag(Q) @ pi)
    h = np.sqrt(pi)
    B = h[:, None] * Q / h[None, :]
    lam, U = np.linalg.eigh(0.5 * (B + B.T))
    return U / h[:, None], U.T * h[None, :], lam, Q


def _matrices(rates, pi, times):
    V, Vi, lam, _ = _eigen(rates, pi)
    return np.einsum("ik,...k,kj->...ij", V, np.exp(np.asarray(times)[..., None] * lam), Vi)


def _gamma(alpha, k):
    """The k median categories of Gamma(alpha, alpha), mean 1 (bisection on
    the regularised incomplete gamma function)."""
    if k == 1:
        return np.ones(1)
    a = torch.full((k,), float(alpha), dtype=torch.float64)
    want = (2 * torch.arange(k, dtype=torch.float64) + 1) / (2 * k)
    lo, hi = torch.full_like(a, -60.0), torch.full_like(a, 6.0)  # logarithms
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        low = torch.special.gammainc(a, mid.exp()) < want
        lo, hi = torch.where(low, mid, lo), torch.where(low, hi, mid)
    q = (0.5 * (lo + hi)).exp().numpy()
    return q / q.mean()


def _simulate(parents, heights, rates, pi, cats, sites, rng):
    """States [taxa][sites] evolved down the tree."""
    n, S = parents.size, pi.size
    P = np.clip(_matrices(rates, pi, np.where(parents == ROOT, 0.0, heights[np.minimum(
        parents, n - 1)] - heights)[:, None] * cats), 0.0, None)
    cdf = np.cumsum(P, axis=3)[..., :-1].astype(np.float32)
    at = rng.integers(0, cats.size, size=sites) * S
    states = np.empty((n, sites), dtype=np.uint8)
    states[n - 1] = rng.choice(S, size=sites, p=pi)
    for v in range(n - 2, -1, -1):
        rows = np.take(cdf[v].reshape(cats.size * S, S - 1), at + states[parents[v]], axis=0)
        states[v] = (rng.random(sites, dtype=np.float32)[:, None] > rows).sum(axis=1)
    return states[: (n + 1) // 2]


def _distinct(parents, heights, rates, pi, cats, patterns, rng):
    """Exactly `patterns` distinct columns and how often each was drawn."""
    sites, cols = int(1.15 * patterns) + 16, None
    for _ in range(8):
        more = np.ascontiguousarray(
            _simulate(parents, heights, rates, pi, cats, sites, rng).T)
        cols = more if cols is None else np.concatenate([cols, more])
        view = cols.view(np.dtype((np.void, cols.shape[1]))).reshape(-1)
        _, first, counts = np.unique(view, return_index=True, return_counts=True)
        if first.size >= patterns:
            break
        sites = 2 * cols.shape[0]
    keep = np.sort(first)[:patterns]
    leaves = np.ascontiguousarray(cols[keep].T)
    weights = counts[np.argsort(first)[:patterns]].astype(np.uint32)
    # sequences start late and end early: up to 3 % of either end is unknown
    S = pi.size
    for row in leaves:
        a, b = rng.integers(0, max(2, 3 * patterns // 100), size=2)
        row[:a] = S
        row[patterns - b:] = S
    return leaves, weights


def _model(S, rng):
    if S == 4:
        return rng.gamma(2.0, 1.0, size=6), rng.dirichlet([5.0] * 4)
    pi = np.maximum(rng.dirichlet([1.0] * 20), 1e-4)
    return rng.lognormal(0.0, 1.0, size=190), pi / pi.sum()


def _problem(case, rng):
    S, C = case.get("states", 4), case["categories"]
    parents, heights = _yule(case["taxa"], rng, 1.0 if case["taxa"] > 16 else 0.5)
    rates, pi = _model(S, rng)
    if S == 4 and C == 1:  # HKY, as the one-category configuration has it
        rates = np.array([1.0, 2.0, 1.0, 1.0, 2.0, 1.0])
    alpha = 0.5 if S == 4 else 1.0
    cats = _gamma(alpha, C)
    leaves, weights = _distinct(parents, heights, rates, pi, cats, case["patterns"], rng)
    return dict(parents=parents, heights=heights, rates=rates, pi=pi, alpha=alpha, cats=cats,
                leaves=leaves, weights=weights)


def _moves(problem, rng, count):
    """`count` (node, height) moves of internal nodes within their bounds."""
    parents, heights = problem["parents"], problem["heights"]
    n, L = parents.size, (parents.size + 1) // 2
    out = []
    for v in rng.integers(L, n, size=count):
        low = heights[np.nonzero(parents == v)[0]].max()
        high = heights[v] * 1.1 if v == n - 1 else heights[parents[v]]
        out.append((int(v), float(low + (high - low) * rng.uniform(0.2, 0.8))))
    return out


def _paths(problem, moves):
    """The dirty lists of each move from the problem's own heights."""
    lists = []
    for v, h in moves:
        heights = problem["heights"].copy()
        heights[v] = h
        lists.append(Topology(problem["parents"], heights).path(v))
    return lists


def _case_inputs(case, seed):
    """What prepare() and exact() both start from."""
    rng = np.random.default_rng([seed & 0x7FFFFFFF, 20])
    if case["kind"] == "surrogate":
        d, H, n = case["inputs"], case["hidden"], case["pairs"]
        dims = [d, H, H, H, 1]
        params = np.concatenate([np.concatenate([
            rng.uniform(-1, 1, size=o * i) / math.sqrt(i), rng.uniform(-0.05, 0.05, size=o)])
            for i, o in zip(dims[:-1], dims[1:])]).astype(np.float32)
        old = rng.normal(0.0, 1.0, size=(n, d)).astype(np.float32)
        new = (old + 0.1 * rng.normal(0.0, 1.0, size=(n, d))).astype(np.float32)
        delta = rng.normal(0.0, 1.0, size=n).astype(np.float32)
        return dict(params=params, x_new=new, x_old=old, delta=delta)
    if case["kind"] == "batch":
        problems, members = [], []
        for a in range(case["alignments"]):
            scale = (1.0, 0.19, 0.55, 0.32)[a]
            one = dict(taxa=max(8, int(case["taxa"] * scale)), categories=case["categories"],
                       patterns=max(200, int(case["patterns"] * scale)))
            problems.append(_problem(one, rng))
        for k in range(case["alignments"] * case["chains"]):
            p = dict(problems[k // case["chains"]])
            p["heights"] = p["heights"] * rng.uniform(0.9, 1.1)
            p["rates"], p["pi"] = _model(4, rng)
            members.append(dict(problem=p, moves=_moves(p, rng, 2)))
        return dict(members=members)
    problem = _problem(case, rng)
    got = dict(problem=problem)
    if case["kind"] == "path":
        moves = _moves(problem, rng, PROPOSALS - 1)
        v = moves[-1][0]
        got["moves"] = moves + [(v, float(problem["heights"][v]))]
    return got


def _calculator(case, problem):
    make = Calculator.GB300(0, case.get("form", "f32"))
    S, C = case.get("states", 4), case["categories"]
    leaves = problem["leaves"]
    if S == 4:  # bases as IUPAC bit codes, N where unknown
        leaves = np.array([1, 2, 4, 8, 15], np.uint8)[leaves]
    calc = (make.make20 if S == 20 else make.make4)(leaves, leaves.shape[1], num_categories=C)
    calc.set_weights(problem["weights"])
    calc.set_reversible(problem["rates"], problem["pi"])
    if C > 1:
        calc.set_gamma(problem["alpha"])
    return calc


def prepare(case, seed):
    got = _case_inputs(case, seed)
    kind = case["kind"]
    if kind == "surrogate":
        net = Surrogate(case["inputs"], case["hidden"])
        net.set_params(got["params"])
        return dict(kind=kind, net=net, data=(got["x_new"], got["x_old"], got["delta"]))
    if kind == "batch":
        calcs, steps = [], [[], []]
        for k, m in enumerate(got["members"]):
            p = m["problem"]
            calc = _calculator(case, p)
            full = Topology(p["parents"], p["heights"]).full()
            calc.propose_lengths(*full)
            calc.log_likelihood()
            calc.accept()
            paths = _paths(p, m["moves"])
            for j in range(2):
                steps[j].append(full if k % 16 == 3 * j else paths[j])
            calcs.append(calc)
        return dict(kind=kind, calcs=calcs, batch=Batch(calcs), steps=steps)
    p = got["problem"]
    calc = _calculator(case, p)
    full = Topology(p["parents"], p["heights"]).full()
    if kind == "trait":
        times = np.asarray(full[2])[:, :, None] * p["cats"]
        mats = np.ascontiguousarray(_matrices(p["rates"], p["pi"], times))
        return dict(kind=kind, calc=calc, args=(full[0], full[1], mats, p["pi"]))
    # a chain starts from its evaluated tree, the launch tuned as the
    # library's own driver tunes it
    calc.propose_lengths(*full)
    calc.log_likelihood()
    calc.accept()
    calc.autotune(*full)
    if kind == "tree":
        return dict(kind=kind, calc=calc, full=full, sites=case["sites"],
                    f64=case["form"] == "f64")
    return dict(kind=kind, calc=calc, lists=_paths(p, got["moves"]), f64=case["form"] == "f64")


def run(state):
    kind = state["kind"]
    if kind == "surrogate":
        loss, grad = state["net"].loss_grad(*state["data"])
        return dict(loss=loss, grad=grad)
    if kind == "batch":
        out = []
        for lists in state["steps"]:
            for calc, one in zip(state["calcs"], lists):
                calc.stage_lengths(*one)
            state["batch"].run()
            out += state["batch"].log_likelihoods().tolist()
            for calc in state["calcs"]:
                calc.reject()
        return out
    calc = state["calc"]
    if kind == "trait":
        calc.propose(*state["args"])
        out = calc.likelihoods()
        calc.accept()
        return out
    if kind == "tree":
        calc.propose_lengths(*state["full"])
        lnl = calc.log_likelihood()
        out = dict(lnl=np.float64(lnl) if state["f64"] else lnl)
        if state["sites"]:
            out["sites"] = calc.site_log_likelihoods()
        calc.accept()
        return out
    out = []
    for k, one in enumerate(state["lists"]):
        calc.propose_lengths(*one)
        out.append(calc.log_likelihood())
        if k < PROPOSALS - 2:
            calc.reject()
        else:
            calc.accept()
    return np.array(out) if state["f64"] else out


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _path_length(taxa):
    """Expected internal nodes from a random one of a Yule tree to its root."""
    return min(taxa - 1.0, max(1.0, 2.0 * (sum(1.0 / k for k in range(1, taxa + 1)) - 1.0) - 1.0))


def _evaluation(S, C, P, w, nodes, clean, internal, tips):
    """`nodes` evaluated: partials and scale counts written, `clean` partials
    read, `tips` tip rows read, weights read; `internal` matrix-vector
    products."""
    cols = C * P
    return dict(bytes=cols * ((nodes + clean) * (S * w + 4)) + P * (tips + 4),
                flops=cols * (internal * 2 * S * S + nodes * S))


def work(case):
    kind = case["kind"]
    if kind == "surrogate":
        d, H, n = case["inputs"], case["hidden"], case["pairs"]
        params = d * H + 2 * H * H + 4 * H + 1
        return dict(bytes=4.0 * (2 * params + n * (2 * d + 1)),
                    flops=2.0 * 2 * n * (2 * d * H + 6 * H * H + 3 * H))
    if kind == "batch":
        total = dict(bytes=0.0, flops=0.0)
        for a in range(case["alignments"]):
            scale = (1.0, 0.19, 0.55, 0.32)[a]
            L, P = max(8, int(case["taxa"] * scale)), max(200, int(case["patterns"] * scale))
            n = _path_length(L)
            path = _evaluation(4, case["categories"], P, 4, n, 0.6 * n, 1.6 * n - 1, 0.4 * n)
            full = _evaluation(4, case["categories"], P, 4, L - 1, 0, L - 2, L)
            for key in total:
                total[key] += case["chains"] * 2 * (path[key] + (full[key] - path[key]) / 16)
        return total
    S, C, P, L = case["states"], case["categories"], case["patterns"], case["taxa"]
    w = 8 if case["form"] == "f64" else 4
    if kind == "path":
        # a path's other children: about three in five are internal
        n = _path_length(L)
        one = _evaluation(S, C, P, w, n, 0.6 * n, 1.6 * n - 1, 0.4 * n + 1)
        return {k: PROPOSALS * v for k, v in one.items()}
    one = _evaluation(S, C, P, w, L - 1, 0, L - 2, L)
    if kind == "trait":
        one["bytes"] += 8 * C * P + 8 * (L - 1) * 2 * C * S * S
    elif case["sites"]:
        one["bytes"] += 8 * P
    return one


# ---------------------------------------------------------------------------
# the same in 64 bits


def _exact_columns(problem, heights, dev):
    """Log-likelihood [categories][patterns] by plain pruning in 64 bits."""
    parents, pi, cats = problem["parents"], problem["pi"], problem["cats"]
    n, S = parents.size, pi.size
    L = (n + 1) // 2
    t = np.where(parents == ROOT, 0.0, heights[np.minimum(parents, n - 1)] - heights)
    mats = torch.from_numpy(_matrices(problem["rates"], pi, t[:, None] * cats)).to(dev)
    leaves = torch.from_numpy(problem["leaves"].astype(np.int64)).to(dev)
    children = [[] for _ in range(n)]
    for v in range(n - 1):
        children[parents[v]].append(v)
    part, logs = {}, torch.zeros(len(cats), leaves.shape[1], dtype=torch.float64, device=dev)
    for v in range(L, n):  # parents follow their children
        x = None
        for ch in children[v]:
            m = mats[ch].transpose(1, 2)
            if ch < L:  # an unknown state sums to one over the last row
                y = torch.cat([m, torch.ones_like(m[:, :1])], dim=1)[:, leaves[ch], :]
            else:
                y = part.pop(ch) @ m
            x = y if x is None else x * y
        top = x.amax(dim=2)
        part[v] = x / top[..., None]
        logs += top.log()
    return (part[n - 1] @ torch.from_numpy(pi).to(dev)).log() + logs


def _exact_sites(problem, heights, dev):
    cols = _exact_columns(problem, heights, dev)
    return torch.logsumexp(cols, dim=0) - math.log(cols.shape[0])


def _exact_lnl(problem, heights, dev):
    w = torch.from_numpy(problem["weights"].astype(np.float64)).to(dev)
    return float(_exact_sites(problem, heights, dev) @ w)


def _exact_surrogate(case, got):
    d, H = case["inputs"], case["hidden"]
    dims = [d, H, H, H, 1]
    p = torch.from_numpy(got["params"].astype(np.float64)).requires_grad_(True)
    new, old, delta = (torch.from_numpy(got[k].astype(np.float64))
                       for k in ("x_new", "x_old", "delta"))

    def f(x):
        at = 0
        for k, (i, o) in enumerate(zip(dims[:-1], dims[1:])):
            x = x @ p[at: at + o * i].reshape(o, i).T + p[at + o * i: at + o * i + o]
            at += o * i + o
            if k < 3:
                x = torch.nn.functional.gelu(x, approximate="tanh")
        return x[:, 0]

    r = f(new) - f(old) - delta
    loss = (r * r).mean()
    loss.backward()
    return dict(loss=loss.item(), grad=p.grad.numpy())


def exact(case, seed):
    got = _case_inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "surrogate":
        return _exact_surrogate(case, got)
    if kind == "batch":
        out = []
        for j in range(2):
            for k, m in enumerate(got["members"]):
                heights = m["problem"]["heights"].copy()
                if k % 16 != 3 * j:
                    v, h = m["moves"][j]
                    heights[v] = h
                out.append(_exact_lnl(m["problem"], heights, dev))
        return out
    p = got["problem"]
    if kind == "trait":
        cols = _exact_columns(p, p["heights"], dev)
        return (cols[0] if cols.shape[0] == 1 else cols).cpu().numpy()
    if kind == "tree":
        sites = _exact_sites(p, p["heights"], dev)
        lnl = float(sites @ torch.from_numpy(p["weights"].astype(np.float64)).to(dev))
        out = dict(lnl=np.float64(lnl) if case["form"] == "f64" else lnl)
        if case["sites"]:
            out["sites"] = sites.cpu().numpy()
        return out
    out = []
    for v, h in got["moves"]:
        heights = p["heights"].copy()
        heights[v] = h
        out.append(_exact_lnl(p, heights, dev))
    return np.array(out) if case["form"] == "f64" else out
