"""Short op lists that a 4-state branch call runs in its own launch give the bits of the separate
traversal (a session held to a launch shape of its kernels): partials, counters, lnL, derivatives
and Newton lengths, for the category counts and pattern counts at the edges of a lane group's and
a block's patterns, lists of one op to the longest, tips with gaps, +I, and a tree that rescales."""
import numpy as np
import pytest

from conftest import ptn_invar
from gems_b200 import GemsError, PhyloTree, synth

pytestmark = pytest.mark.gpu


def pair(ncat, npat, seed, safe, precision, ntaxa=12, blen=0.1, p_invar=0.0):
    rng = np.random.default_rng(seed)
    model = synth.dna_gtr(rng, ncat, 0.5)
    model.p_invar = p_invar
    tree = synth.random_tree(ntaxa, blen, seed + 1)
    aln = synth.simulate(tree, model, 40 * npat + 64, seed + 2, gap_frac=0.05)
    npat = min(npat, aln.npat)
    aln.patterns = np.ascontiguousarray(aln.patterns[:, :npat])
    aln.weights = aln.weights[:npat].copy()
    out = []
    for separate in (False, True):
        t = PhyloTree.from_case(tree, model, aln, precision=precision,
                                scaling="safe" if safe else "norm", invar=ptn_invar(model, aln))
        if separate:
            t.session.set_autotune(False, force_shape=0)
        out.append(t)
    return tree, out


def same(tree, trees):
    got = []
    for t in trees:
        r = []
        for u, v in zip(tree.eu.tolist(), tree.ev.tolist()):
            for node, dad in ((u, v), (v, u)):
                if node < tree.ntaxa:
                    continue
                try:
                    r.append(t.getPartial(node, dad))
                except GemsError:
                    r.append(None)
        got.append(r)
    seen = 0
    for a, b in zip(*got):
        assert (a is None) == (b is None)
        if a is not None:
            np.testing.assert_array_equal(a[0], b[0])
            np.testing.assert_array_equal(a[1], b[1])
            seen += 1
    return seen


def walk(tree, trees):
    (a, b) = trees
    assert a.computeLikelihood(pattern_lh=True)[0] == b.computeLikelihood(pattern_lh=True)[0]
    assert same(tree, trees) >= tree.ntaxa - 2
    for u, v, x in list(zip(tree.eu.tolist(), tree.ev.tolist(), tree.length.tolist()))[::3]:
        assert a.computeFuncDerv(u, v, x, True) == b.computeFuncDerv(u, v, x, True)
        a.optimizeOneBranch(u, v)
        b.optimizeOneBranch(u, v)
        assert a.getBranchLength(u, v) == b.getBranchLength(u, v)
    same(tree, trees)
    n = a.session.launch_count(), b.session.launch_count()
    for t in trees:
        t.close()
        t.session.close()
    return n


@pytest.mark.parametrize("ncat", [2, 3, 4, 5, 8, 16])
@pytest.mark.parametrize("safe", [False, True], ids=["norm", "safe"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_categories(gpu, ncat, safe, precision):
    fused, separate = walk(*pair(ncat, 333, 800 + ncat, safe, precision,
                                 p_invar=0.2 if ncat == 4 else 0.0))
    assert fused < separate


@pytest.mark.parametrize("npat", [1, 31, 64, 65, 127, 129, 257, 1025])
@pytest.mark.parametrize("precision,safe", [("fp64", True), ("mixed", False)])
def test_pattern_edges(gpu, npat, precision, safe):
    walk(*pair(4, npat, 820 + npat, safe, precision, ntaxa=18))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("safe", [False, True], ids=["norm", "safe"])
def test_rescaling(gpu, precision, safe):
    """A deep tree (its first traversal is a separate launch either way): the updates of the walk
    over its branches rescale."""
    tree, trees = pair(4, 150, 860, safe, precision, ntaxa=200, blen=1.2)
    for t in trees:
        t.session.set_newton_share(8)
    walk(tree, trees)
