"""Mixed 20-state traversal (two patterns per lane, op tables in a ring): category counts on every
lane split (1 to 16, with idle lanes), pattern counts at the edges of a warp's and a block's
patterns, op lists shorter and longer than the ring, NORM and SAFE, +I, a deep tree that rescales,
packets against the whole traversal.  Against the FP64 oracle: lnL to 1e-6; a pattern's lnL to the
first-order rounding bound of its FP32 chain, 24 roundings (a 20-term sum, a product, P and the
tip row) of 2^-24 per node."""
import numpy as np
import pytest

from conftest import ptn_invar
from gems_b200 import PhyloTree, synth
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
    gt = PhyloTree.from_case(tree, model, aln, precision="mixed",
                             scaling="safe" if safe else "norm", invar=ptn_invar(model, aln))
    lo, plo = ot.computeLikelihood(pattern_lh=True)
    lg, plg = gt.computeLikelihood(pattern_lh=True)
    assert abs(lg - lo) <= 1e-6 * abs(lo), (lg, lo)
    assert np.max(np.abs(plg - plo)) <= (tree.ntaxa - 1) * 24 * 2.0 ** -24
    most = 0
    ops, _ = full_traversal(tree)
    gt.session.traverse(ops)
    for slot in range(tree.ntaxa - 2):
        most = max(most, int(gt.session.get_partial(slot)[1].max()))
    gt.close()
    gt.session.close()
    return most


@pytest.mark.parametrize("npat", [1, 15, 16, 17, 33, 63, 64, 65, 97, 193, 385])
@pytest.mark.parametrize("ncat,safe", [(1, False), (2, True), (4, False), (4, True), (7, False)])
def test_pattern_edges(gpu, npat, ncat, safe):
    check(*case(ncat, npat, 500 + npat), safe)


@pytest.mark.parametrize("ncat", [1, 2, 3, 4, 5, 6, 8, 9, 14, 16])
@pytest.mark.parametrize("safe", [False, True], ids=["norm", "safe"])
def test_categories(gpu, ncat, safe):
    check(*case(ncat, 211, 540 + ncat, p_invar=0.1 if ncat == 2 else 0.0), safe)


@pytest.mark.parametrize("ntaxa", [3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("ncat", [4, 8])
def test_short_op_lists(gpu, ntaxa, ncat):
    check(*case(ncat, 40, 560 + ntaxa, ntaxa=ntaxa, blen=0.4), False)


@pytest.mark.parametrize("ncat", [4, 6])
@pytest.mark.parametrize("safe", [False, True], ids=["norm", "safe"])
def test_deep_tree_rescales(gpu, ncat, safe):
    assert check(*case(ncat, 90, 570, ntaxa=220, blen=1.0), safe) >= 2


@pytest.mark.parametrize("ncat", [3, 4, 8])
@pytest.mark.parametrize("safe", [False, True], ids=["norm", "safe"])
def test_packets_equal_whole(gpu, ncat, safe):
    """One op over a range of patterns at a time (no child forwarded) leaves the slots of the
    whole traversal, bit for bit."""
    tree, model, aln = case(ncat, 300, 580, ntaxa=20)
    scaling = "safe" if safe else "norm"
    whole = PhyloTree.from_case(tree, model, aln, precision="mixed", scaling=scaling)
    parts = PhyloTree.from_case(tree, model, aln, precision="mixed", scaling=scaling)
    ops, _ = full_traversal(tree)
    whole.session.traverse(ops)
    assert parts.session.pattern_granule() == (128 if ncat <= 4 else 1)
    for op in ops:
        for lo, hi in ((0, 128), (128, 256), (256, 300)):
            parts.session.compute_partial(op, lo, hi)
    for slot in range(tree.ntaxa - 2):
        for a, b in zip(whole.session.get_partial(slot), parts.session.get_partial(slot)):
            np.testing.assert_array_equal(a, b)
    for t in (whole, parts):
        t.close()
        t.session.close()
