"""FP64 20-state traversal with more than four categories: several warps share a group of patterns
where there are few, one warp holds all categories where there are many.  A traversal of many
patterns and ranges of few (categories that split evenly over the warps and ones that do not) leave
the same partials and counters, bit for bit, on a tree that rescales; and a small alignment gives
the oracle's lnL to 1e-9 (rounding of 1e3 sums of 20 terms: far below)."""
import numpy as np
import pytest

from gems_b200 import PhyloTree, synth
from gems_b200.api import full_traversal
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def case(ncat, npat, ntaxa, blen):
    rng = np.random.default_rng(900 + ncat)
    model = synth.protein(rng, ncat, 0.8)
    tree = synth.random_tree(ntaxa, blen, 901)
    pats = rng.integers(0, 20, (ntaxa, npat)).astype(np.uint8)
    pats[rng.random((ntaxa, npat)) < 0.05] = synth.state_unknown(20)
    return tree, model, synth.Alignment(ntaxa, 20, npat, pats, np.ones(npat))


@pytest.mark.parametrize("ncat", [5, 6, 8, 9, 11, 13, 16])
@pytest.mark.parametrize("scaling", ["norm", "safe"])
def test_ranges_equal_whole(gpu, ncat, scaling):
    npat = 9_601
    tree, model, aln = case(ncat, npat, 100, 1.0)
    whole = PhyloTree.from_case(tree, model, aln, scaling=scaling)
    parts = PhyloTree.from_case(tree, model, aln, scaling=scaling)
    ops, _ = full_traversal(tree)
    whole.session.traverse(ops)
    step = 2_003
    for op in ops:
        for lo in range(0, npat, step):
            parts.session.compute_partial(op, lo, min(lo + step, npat))
    most = 0
    for slot in range(0, tree.ntaxa - 2, 7):
        a, b = whole.session.get_partial(slot), parts.session.get_partial(slot)
        np.testing.assert_array_equal(a[0], b[0])
        np.testing.assert_array_equal(a[1], b[1])
        most = max(most, int(a[1].max()))
    assert most >= 1
    for t in (whole, parts):
        t.close()
        t.session.close()


@pytest.mark.parametrize("ncat", range(5, 17))
@pytest.mark.parametrize("safe", [False, True], ids=["norm", "safe"])
def test_few_patterns(gpu, ncat, safe):
    tree, model, aln = case(ncat, 37, 9, 0.3)
    lo, plo = orc.OracleTree(tree, model, aln, safe=safe).computeLikelihood(pattern_lh=True)
    t = PhyloTree.from_case(tree, model, aln, scaling="safe" if safe else "norm")
    lg, plg = t.computeLikelihood(pattern_lh=True)
    assert abs(lg - lo) <= 1e-9 * abs(lo)
    assert np.allclose(plg, plo, rtol=1e-9, atol=1e-12)
    t.close()
    t.session.close()
