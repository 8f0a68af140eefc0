"""FP64 20-state traversal (eight patterns per warp on the FP64 mma): pattern counts at the edges
of a warp's and a block's patterns, category counts in one pass (1 to 4) and in several (5, 8),
NORM and SAFE, a deep tree that rescales, packets against the whole traversal.  Against the FP64
oracle: lnL to 1e-9, scale counters exact, and partials to 1e-10 of their pattern's largest value
(two chained sums of 20 terms round to about 40 x 1.1e-16 of their largest term, and the
eigen-space sums of these trees cancel by far less than 1e4)."""
import numpy as np
import pytest

from conftest import ptn_invar
from gems_b200 import GemsError, PhyloTree, synth
from gems_b200.api import full_traversal
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def case(ncat, npat, seed, ntaxa=12, blen=0.15, p_invar=0.0):
    rng = np.random.default_rng(seed)
    model = synth.protein(rng, ncat, 0.8)
    model.p_invar = p_invar
    tree = synth.random_tree(ntaxa, blen, seed + 1)
    aln = synth.simulate(tree, model, 2 * npat + 64, seed + 2, gap_frac=0.05)
    assert aln.npat >= npat
    aln.patterns = np.ascontiguousarray(aln.patterns[:, :npat])
    aln.weights = aln.weights[:npat].copy()
    return tree, model, aln


def check(tree, model, aln, safe):
    ot = orc.OracleTree(tree, model, aln, safe=safe, const_char=aln.const_char())
    gt = PhyloTree.from_case(tree, model, aln, precision="fp64",
                             scaling="safe" if safe else "norm", invar=ptn_invar(model, aln))
    lo, plo = ot.computeLikelihood(pattern_lh=True)
    lg, plg = gt.computeLikelihood(pattern_lh=True)
    assert abs(lg - lo) <= 1e-9 * abs(lo), (lg, lo)
    assert np.allclose(plg, plo, rtol=1e-9, atol=1e-12)
    most = 0
    checked = 0
    for u, v in zip(tree.eu.tolist(), tree.ev.tolist()):
        for node, dad in ((u, v), (v, u)):
            if node < tree.ntaxa:
                continue
            try:
                po, so = ot.getPartial(node, dad)
                pg, sg = gt.getPartial(node, dad)
            except (AssertionError, GemsError):
                continue
            np.testing.assert_array_equal(sg, so)
            most = max(most, int(sg.max()))
            scale = np.abs(po).max(axis=(1, 2), keepdims=True) + 1e-300
            assert np.max(np.abs(pg - po) / scale) < 1e-10
            checked += 1
    assert checked >= tree.ntaxa - 2
    gt.close()
    gt.session.close()
    return most


@pytest.mark.parametrize("npat", [1, 7, 8, 9, 31, 33, 64, 65, 129])
@pytest.mark.parametrize("ncat,safe", [(1, True), (4, False), (4, True), (5, False)])
def test_pattern_edges(gpu, npat, ncat, safe):
    check(*case(ncat, npat, 400 + npat), safe)


@pytest.mark.parametrize("ncat", [1, 2, 3, 4, 5, 8, 11])
@pytest.mark.parametrize("safe", [False, True], ids=["norm", "safe"])
def test_categories(gpu, ncat, safe):
    check(*case(ncat, 301, 440 + ncat, p_invar=0.1 if ncat == 2 else 0.0), safe)


@pytest.mark.parametrize("ncat", [4, 6])
@pytest.mark.parametrize("safe", [False, True], ids=["norm", "safe"])
def test_deep_tree_rescales(gpu, ncat, safe):
    assert check(*case(ncat, 90, 470, ntaxa=220, blen=1.0), safe) >= 2


@pytest.mark.parametrize("ncat", [3, 4, 8])
@pytest.mark.parametrize("safe", [False, True], ids=["norm", "safe"])
def test_packets_equal_whole(gpu, ncat, safe):
    """One op over a pattern range at a time (no child forwarded, ranges that start inside a
    warp's patterns) leaves the slots of the whole traversal, bit for bit."""
    tree, model, aln = case(ncat, 77, 480, ntaxa=20)
    scaling = "safe" if safe else "norm"
    whole = PhyloTree.from_case(tree, model, aln, scaling=scaling)
    parts = PhyloTree.from_case(tree, model, aln, scaling=scaling)
    ops, _ = full_traversal(tree)
    whole.session.traverse(ops)
    for op in ops:
        for lo, hi in ((0, 5), (5, 37), (37, 77)):
            parts.session.compute_partial(op, lo, hi)
    for slot in range(tree.ntaxa - 2):
        for a, b in zip(whole.session.get_partial(slot), parts.session.get_partial(slot)):
            np.testing.assert_array_equal(a, b)
    for t in (whole, parts):
        t.close()
        t.session.close()
