"""The workloads that the likelihood path is timed on, through the calls that a program makes.

A case names a kind of use (`KINDS`), the alignment's size, the model family (4, 20 or 61 states,
1 to 8 rate categories) and the form (FP64 or mixed, NORM or SAFE scaling).  Inputs are simulated
down a random tree under a random model of that family, all drawn from the seed alone.

listed()            the cases that are timed
draw(rng)           one more case of the same ranges
prepare(case, seed) session, tree and data as a program holds them before the call
run(state)          one pass through the public entry points
work(case)          bytes and operations one pass cannot do without
exact(case, seed)   what run() returns, in 64-bit torch without the library's kernels
"""
import math

import numpy as np
import torch

from gems_b200 import PhyloTree, Session, synth
from gems_b200 import api


def listed():
    return [
        # the plain FP64 configuration: a small tree's lnL, then the derivatives of every branch
        # (16 taxa, 10,000 sites of 3,801 patterns: a few microseconds of device work per call)
        dict(name="dna_branches", kind="branches", states=4, ncat=4, precision="fp64",
             scaling="norm", taxa=16, patterns=3_801, gaps=0.0, branches=29),
        # a step of tree search: both NNIs of a few internal branches, five Newton loops each,
        # on a gene-sized alignment with its pattern count left ragged
        dict(name="dna_nni", kind="nni", states=4, ncat=4, precision="mixed", scaling="norm",
             taxa=100, patterns=4_703, gaps=0.05, branches=4),
        # one round of branch lengths on a new tree (after a model change): traversals of a few
        # nodes, theta and a Newton loop for each of the branches
        dict(name="dna_optimise", kind="optimise", states=4, ncat=4, precision="fp64",
             scaling="safe", taxa=50, patterns=18_501, gaps=0.05),
        # the large DNA configuration in both forms: a from-scratch lnL of 512 taxa
        dict(name="dna_lnl_fp64", kind="lnl", states=4, ncat=4, precision="fp64",
             scaling="norm", taxa=512, patterns=600_000, gaps=0.05),
        dict(name="dna_lnl_mixed", kind="lnl", states=4, ncat=4, precision="mixed",
             scaling="norm", taxa=512, patterns=1_000_000, gaps=0.05),
        # the protein configuration (100,000 sites) in both forms
        dict(name="protein_lnl_fp64", kind="lnl", states=20, ncat=4, precision="fp64",
             scaling="norm", taxa=128, patterns=98_762, gaps=0.0),
        dict(name="protein_lnl_mixed", kind="lnl", states=20, ncat=4, precision="mixed",
             scaling="norm", taxa=128, patterns=98_762, gaps=0.0),
        # branch lengths of a protein tree
        dict(name="protein_optimise", kind="optimise", states=20, ncat=4, precision="fp64",
             scaling="norm", taxa=40, patterns=9_707, gaps=0.02),
        # ModelFinder: candidate codon models on one alignment, each at a new Gamma shape
        dict(name="codon_models", kind="models", states=61, ncat=4, precision="mixed",
             scaling="safe", taxa=200, patterns=3_780, gaps=0.0, models=32),
        # one codon model in the FP64 form: lnL and the derivatives of some branches
        dict(name="codon_branches", kind="branches", states=61, ncat=4, precision="fp64",
             scaling="safe", taxa=200, patterns=3_780, gaps=0.0, branches=8),
        # ultrafast bootstrap: the current tree's lnL from its resident partials, then every
        # replicate's from the same pattern likelihoods
        dict(name="dna_rell", kind="rell", states=4, ncat=4, precision="mixed", scaling="norm",
             taxa=64, patterns=450_000, gaps=0.05, replicates=256),
        # an alignment as read from a file, encoded and compressed to patterns on the device
        dict(name="dna_ingest", kind="ingest", states=4, taxa=256, patterns=170_000,
             sites=200_000, gaps=0.05),
    ]


#: (kind, states, precisions, taxa range, pattern range, categories)
KINDS = [
    ("branches", 4, ("fp64", "mixed"), (8, 64), (500, 50_000), (1, 4, 8)),
    ("nni", 4, ("fp64", "mixed"), (12, 200), (500, 50_000), (1, 4)),
    ("optimise", 4, ("fp64", "mixed"), (8, 60), (500, 50_000), (1, 4, 8)),
    ("lnl", 4, ("fp64", "mixed"), (32, 512), (20_000, 600_000), (1, 4, 8)),
    ("lnl", 20, ("fp64", "mixed"), (8, 128), (1_000, 100_000), (1, 2, 4, 8)),
    ("branches", 20, ("fp64", "mixed"), (8, 128), (500, 40_000), (1, 4, 8)),
    ("optimise", 20, ("fp64",), (8, 40), (500, 12_000), (1, 4)),
    ("models", 61, ("mixed",), (16, 200), (300, 4_000), (1, 4, 8)),
    ("branches", 61, ("fp64",), (8, 200), (300, 4_000), (1, 4, 8)),
    ("rell", 4, ("fp64", "mixed"), (16, 64), (10_000, 500_000), (4,)),
    ("ingest", 4, (None,), (16, 256), (5_000, 200_000), (1,)),
]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind, states, precs, taxa, patterns, cats = rng.choice(KINDS)
    case = dict(kind=kind, states=states, taxa=_log_uniform(rng, *taxa),
                gaps=rng.choice([0.0, 0.02, 0.05]))
    # a small tree has few distinct columns
    case["patterns"] = min(_log_uniform(rng, *patterns), 20 * case["taxa"] ** 2)
    if kind == "ingest":
        case["sites"] = int(case["patterns"] * rng.uniform(1.0, 1.5))
        return case
    case.update(ncat=rng.choice(cats), precision=rng.choice(precs),
                scaling="safe" if states == 61 else rng.choice(["norm", "safe"]))
    if kind == "lnl" and states == 4:  # the device memory of three states
        per = case["taxa"] * case["ncat"] * (32 if case["precision"] == "fp64" else 16)
        case["patterns"] = min(case["patterns"], int(35e9 / per))
    if kind == "branches":
        case["branches"] = rng.randint(1, min(12, 2 * case["taxa"] - 3))
    if kind == "nni":
        case["branches"] = rng.randint(1, 4)
    if kind == "models":
        case["models"] = rng.randint(2, 16 if case["ncat"] == 8 else 32)
    if kind == "rell":
        case["replicates"] = _log_uniform(rng, 32, 256)
    return case


# ---- inputs ------------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _model(states, ncat, rng):
    if states == 4:
        return synth.dna_gtr(rng, ncat, 0.5)
    if states == 20:
        return synth.protein(rng, ncat, 0.8)
    return synth.codon_gy(rng, ncat, 0.5, freerate=ncat == 8)


def _rate_matrix(model):
    """The reversible rate matrix of the model, one substitution per site."""
    n = model.nstates
    freq = np.asarray(model.freq, np.float64)
    freq = freq / freq.sum()
    q = np.zeros((n, n))
    q[np.triu_indices(n, 1)] = model.exch_upper
    q = (q + q.T) * freq
    np.fill_diagonal(q, 0.0)
    q /= float(freq @ q.sum(1))
    np.fill_diagonal(q, -q.sum(1))
    return q, freq


def _transition(model, lengths, device):
    """P_c(t) of every length and category: [len][C][n][n], 64 bits."""
    q, _ = _rate_matrix(model)
    a = torch.as_tensor(np.multiply.outer(np.asarray(lengths, np.float64), model.rates))
    return torch.matrix_exp(a.to(device)[..., None, None] * torch.as_tensor(q).to(device))


def _neighbours(tree):
    adj = [[] for _ in range(tree.nnodes)]
    for e, (u, v) in enumerate(zip(tree.eu.tolist(), tree.ev.tolist())):
        adj[u].append((v, e))
        adj[v].append((u, e))
    return adj


def _simulate(tree, model, sites, seed, gaps):
    """Tip states [taxa][sites] (uint8) drawn down the tree, `gaps` of the cells unknown."""
    dev, n = _device(), model.nstates
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    cum = _transition(model, tree.length, dev).clamp_min(0).cumsum(-1).float()
    def pick(p, shape):
        w = torch.as_tensor(np.asarray(p, np.float64) / np.sum(p)).cumsum(0).float().to(dev)
        r = torch.rand(shape, generator=g, device=dev)
        return torch.searchsorted(w, r).clamp_max(len(p) - 1)
    cat = pick(model.props, sites)
    adj, root = _neighbours(tree), tree.ntaxa
    out = torch.empty((tree.ntaxa, sites), dtype=torch.uint8, device=dev)
    todo = [(root, -1, pick(model.freq, sites).to(torch.uint8))]
    while todo:
        x, dad, state = todo.pop()
        if x < tree.ntaxa:
            out[x] = state
            continue
        row = cat * n + state.long()
        for y, e in adj[x]:
            if y == dad:
                continue
            r = torch.rand(sites, generator=g, device=dev)
            child = (r[:, None] > cum[e].reshape(-1, n)[row]).sum(1).clamp_max(n - 1)
            todo.append((y, x, child.to(torch.uint8)))
    if gaps > 0:
        for k in range(tree.ntaxa):
            gone = torch.rand(sites, generator=g, device=dev) < gaps
            out[k][gone] = synth.state_unknown(n)
    return out.cpu().numpy()


def _alignment(tree, model, case, seed):
    """(patterns [taxa][K], weights): the first K distinct columns of an alignment simulated down
    the tree, with how often each comes up in it."""
    want, taxa = case["patterns"], case["taxa"]
    if want * taxa > 30_000_000:  # hundreds of taxa: every column is its own pattern
        return _simulate(tree, model, want, seed, case["gaps"]), np.ones(want)
    sites = want + want // 16 + 64
    while True:
        aln = synth.compress(_simulate(tree, model, sites, seed, case["gaps"]), model.nstates)
        if aln.npat >= want:
            return np.ascontiguousarray(aln.patterns[:, :want]), aln.weights[:want].copy()
        if sites > 512 * want:
            raise ValueError("the tree has too few distinct columns")
        sites *= 2


def _inputs(case, seed):
    """(tree, models, patterns, weights) of a case: candidate models share the tree and data."""
    rng = np.random.default_rng([int(seed), 17])
    n = case["states"]
    mean = {4: 0.05 if case["taxa"] > 64 else 0.1, 20: 0.15, 61: 0.1}[n]
    tree = synth.random_tree(case["taxa"], mean, int(seed) + 11)
    models = [_model(n, case.get("ncat", 4), rng) for _ in range(case.get("models", 1))]
    return (tree, models, *_alignment(tree, models[0], case, seed))


def _columns(case, patterns, weights, seed):
    """An alignment of case["sites"] columns that holds every pattern, in a random order."""
    rng = np.random.default_rng([int(seed), 37])
    more = rng.choice(len(weights), case["sites"] - len(weights), p=weights / weights.sum())
    order = rng.permutation(np.concatenate([np.arange(len(weights)), more]))
    return np.ascontiguousarray(patterns[:, order])


def _branches(tree, count, internal=False):
    """`count` branches spread over the tree as (node, dad)."""
    edges = [(u, v) for u, v in zip(tree.eu.tolist(), tree.ev.tolist())
             if not internal or min(u, v) >= tree.ntaxa]
    count = min(count, len(edges))
    return [edges[(i * len(edges)) // count] for i in range(count)]


def _session(case, model, patterns, weights, spare=0):
    taxa, npat = patterns.shape
    s = Session(taxa, npat, case["states"], case["ncat"], taxa - 2 + spare,
                precision=case["precision"], scaling=case["scaling"])
    s.upload_tips(patterns)
    s.upload_patterns(weights)
    s.set_model(model.eval, model.evec, model.inv_evec, model.rates, model.props)
    return s


def _shapes(case, models, seed):
    """A new Gamma shape for each candidate model: its category rates."""
    rng = np.random.default_rng([int(seed), 29])
    if case["ncat"] == 1:
        return [np.ones(1) for _ in models]
    return [synth.gamma_rates(float(rng.uniform(0.2, 1.5)), case["ncat"]) for _ in models]


def _replicates(case, weights, seed):
    rng = np.random.default_rng([int(seed), 31])
    total = int(weights.sum())
    return np.stack([rng.multinomial(total, weights / weights.sum())
                     for _ in range(case["replicates"])]).astype(np.float32)


def prepare(case, seed):
    tree, models, patterns, weights = _inputs(case, seed)
    kind = case["kind"]
    if kind == "ingest":
        letters = np.full(256, ord("-"), np.uint8)
        letters[:4] = np.frombuffer(b"ACGT", np.uint8)
        columns = _columns(case, patterns, weights, seed)
        return dict(kind=kind, states=case["states"], seqs=letters[columns])
    state = dict(kind=kind, pattern_lh=case["precision"] == "fp64")
    if kind == "models":
        sessions = [_session(case, m, patterns, weights) for m in models]
        state["trees"] = [PhyloTree(s, tree.eu, tree.ev, tree.length) for s in sessions]
        state["rates"] = _shapes(case, models, seed)
        return state
    s = _session(case, models[0], patterns, weights, spare=2 if kind == "nni" else 0)
    state["session"], state["tree"] = s, PhyloTree(s, tree.eu, tree.ev, tree.length)
    state["edges"] = (tree.eu, tree.ev, tree.length)
    if kind in ("branches", "nni"):
        state["branches"] = _branches(tree, case["branches"], internal=kind == "nni")
        state["lengths"] = [state["tree"].getBranchLength(u, v) for u, v in state["branches"]]
    if kind == "nni":
        state["tree"].computeLikelihood()
    if kind == "rell":
        state["tree"].computeLikelihood()
        s.upload_reweightings(_replicates(case, weights, seed))
    return state


# ---- one pass ----------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "ingest":
        ing = api.Ingest(state["seqs"], state["states"])
        patterns, weights, site_pattern, const_char = ing.read()
        ing.close()
        return dict(patterns=patterns, weights=weights, site_pattern=site_pattern,
                    const_char=const_char)
    if kind == "models":
        return api.evaluate_rates_batch(state["trees"], state["rates"])
    t = state["tree"]
    if kind == "lnl":
        t.clearAllPartialLH()
        if state["pattern_lh"]:
            lnl, plh = t.computeLikelihood(pattern_lh=True)
            return dict(lnl=lnl, pattern_lh=plh)
        return dict(lnl=t.computeLikelihood())
    if kind == "branches":
        t.clearAllPartialLH()
        lnl = t.computeLikelihood()
        return dict(lnl=lnl, derv=[t.computeFuncDerv(u, v, x, new_branch=True) for (u, v), x in
                                   zip(state["branches"], state["lengths"])])
    if kind == "nni":
        return [[(lnl, lens) for _, _, lnl, lens in t.evaluateNNI(u, v)]
                for u, v in state["branches"]]
    if kind == "optimise":
        t = PhyloTree(state["session"], *state["edges"])
        lnl = t.optimizeAllBranches(1, 0.001, 100)
        return dict(lnl=lnl, lengths=t.getBranchLengths())
    if kind == "rell":
        return dict(lnl=t.computeLikelihood(), replicates=state["session"].reweighted_lnl())
    raise ValueError(kind)


# ---- what a pass cannot do without -------------------------------------------------------

def _traversal(case):
    """(bytes, flops) of one from-scratch traversal: every tip byte and weight read once, every
    partial and its counters written once (they stay resident for the calls after), and one n x n
    product per internal child (half of a binary tree's children are tips), n products of the two
    messages."""
    c, n, p = case["ncat"], case["states"], case["patterns"]
    elem = 8 if case["precision"] == "fp64" else 4
    nodes = case["taxa"] - 2
    counters = 2 * (c if case["scaling"] == "safe" else 1)
    return (p * (case["taxa"] + 8) + nodes * p * (c * n * elem + counters),
            p * c * ((nodes - 1) * 2.0 * n * n + nodes * n))


def work(case):
    kind, p, taxa = case["kind"], case["patterns"], case["taxa"]
    if kind == "ingest":
        return dict(bytes=taxa * case["sites"] + 4 * case["sites"] + (taxa + 9) * p, flops=0)
    c, n = case["ncat"], case["states"]
    elem = 8 if case["precision"] == "fp64" else 4
    tb, tf = _traversal(case)
    row = c * n * elem
    if kind == "lnl":
        return dict(bytes=tb + 8 * p, flops=tf)
    if kind == "models":
        return dict(bytes=case["models"] * tb, flops=case["models"] * tf)
    if kind == "rell":
        return dict(bytes=p * (2 * row + 16 + 4 * case["replicates"]),
                    flops=p * (2.0 * c * n * n + 2.0 * case["replicates"]))
    # per branch: the partial on its far side (about one node's update as the calls walk on), then
    # both ends' rows read once per Newton loop or derivative
    one_b, one_f = tb / (taxa - 2), tf / (taxa - 2)
    per_b, per_f = one_b + 2 * p * row, one_f + 8.0 * p * c * n
    if kind == "branches":
        k = case["branches"]
        return dict(bytes=tb + k * per_b, flops=tf + k * per_f)
    if kind == "optimise":
        k = 2 * taxa - 3
        return dict(bytes=tb + k * per_b, flops=tf + k * per_f)
    # nni: two swaps, five branches each
    k = 10 * case["branches"]
    return dict(bytes=k * per_b, flops=k * per_f)


# ---- in 64 bits --------------------------------------------------------------------------

def _exact_lnl(tree, model, patterns, branch, derivatives, chunk=65536):
    """Pattern log-likelihoods [npat] rooted in the branch, with the first and second derivatives
    of the pattern likelihood over the likelihood when asked, by pruning with rescaled rows."""
    dev, n = _device(), model.nstates
    adj, (u, v) = _neighbours(tree), branch
    trans = _transition(model, tree.length, dev)
    q, freq = _rate_matrix(model)
    q, freq = torch.as_tensor(q).to(dev), torch.as_tensor(freq).to(dev)
    rates = torch.as_tensor(np.asarray(model.rates, np.float64)).to(dev)
    props = torch.as_tensor(np.asarray(model.props, np.float64)).to(dev)
    table = torch.ones((256, n), dtype=torch.float64, device=dev)
    table[:n] = torch.eye(n, dtype=torch.float64, device=dev)
    out = []
    for p0 in range(0, patterns.shape[1], chunk):
        tips = torch.as_tensor(patterns[:, p0:p0 + chunk].astype(np.int64)).to(dev)

        def below(top, dad):
            """([P][C][n], log scale [P]) of the subtree at `top` away from `dad`."""
            order, todo = [], [(top, dad)]
            while todo:
                x, d = todo.pop()
                order.append((x, d))
                todo += [(y, x) for y, _ in adj[x] if y != d and x >= tree.ntaxa]
            done = {}
            for x, d in reversed(order):
                if x < tree.ntaxa:
                    continue
                part, scale = None, torch.zeros(tips.shape[1], dtype=torch.float64, device=dev)
                for y, e in adj[x]:
                    if y == d:
                        continue
                    if y < tree.ntaxa:
                        m = (trans[e] @ table.T).permute(2, 0, 1)[tips[y]]
                    else:
                        child, s = done.pop(y)
                        m = torch.einsum("cxy,pcy->pcx", trans[e], child)
                        scale = scale + s
                    part = m if part is None else part * m
                big = part.amax((1, 2)).clamp_min(1e-300)
                done[x] = (part / big[:, None, None], scale + big.log())
            if top < tree.ntaxa:
                row = table[tips[top]][:, None, :].expand(-1, len(rates), -1)
                return row, torch.zeros(tips.shape[1], dtype=torch.float64, device=dev)
            return done[top]

        (a, sa), (b, sb) = below(u, v), below(v, u)
        e = next(e for y, e in adj[u] if y == v)
        a = a * freq * props[:, None]
        like = torch.einsum("pcx,cxy,pcy->p", a, trans[e], b)
        got = [like.log() + sa + sb]
        if derivatives:
            d1 = rates[:, None, None] * (q @ trans[e])
            d2 = rates[:, None, None] * (q @ d1)
            got += [torch.einsum("pcx,cxy,pcy->p", a, d, b) / like for d in (d1, d2)]
        out.append(torch.stack(got))
    return torch.cat(out, 1).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("nni", "optimise"):
        return None  # an optimiser's result: no closed value
    tree, models, patterns, weights = _inputs(case, seed)
    if kind == "ingest":
        patterns = _columns(case, patterns, weights, seed)
        cols = np.ascontiguousarray(patterns.T).view(np.dtype((np.void, patterns.shape[0])))
        _, first, count = np.unique(cols.ravel(), return_index=True, return_counts=True)
        return dict(patterns=None, weights=count[np.argsort(first)].astype(np.float64),
                    site_pattern=None, const_char=None)
    at = (0, next(y for y, _ in _neighbours(tree)[0]))
    if kind == "models":
        got = []
        for m, r in zip(models, _shapes(case, models, seed)):
            m.rates, m.props = r, np.full(len(r), 1.0 / len(r))
            got.append(float(weights @ _exact_lnl(tree, m, patterns, at, False)[0]))
        return np.array(got)
    plh = _exact_lnl(tree, models[0], patterns, at, False)[0]
    lnl = float(weights @ plh)
    if kind == "lnl":
        return dict(lnl=lnl, pattern_lh=plh) if case["precision"] == "fp64" else dict(lnl=lnl)
    if kind == "rell":
        return dict(lnl=lnl, replicates=_replicates(case, weights, seed).astype(np.float64) @ plh)
    derv = []
    for br in _branches(tree, case["branches"]):
        _, d1, d2 = _exact_lnl(tree, models[0], patterns, br, True)
        # an optimiser minimises: the negated derivatives
        derv.append((-float(weights @ d1), float(weights @ (d1 * d1 - d2))))
    return dict(lnl=lnl, derv=derv)
