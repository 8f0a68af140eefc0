"""The branch lnL of many mixed sessions in one launch gives the bits of each session's own call:
more sessions than one launch takes, and as many pattern groups per session as its blocks can
hold and more, 20 and 61 states, NORM and SAFE, one op list and a list per session."""
import numpy as np
import pytest

from gems_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nstates,scaling,npat,nsess", [
    (20, "norm", 70, 2), (20, "norm", 24_000, 2), (20, "safe", 3_000, 33),
    (61, "safe", 100, 3), (61, "safe", 2_600, 33),
])
def test_batch_equals_alone(nstates, scaling, npat, nsess):
    from gems_b200 import PhyloTree, compute_likelihood_batch
    rng = np.random.default_rng(31 + npat)
    model = (synth.codon_gy(rng, 1, 0.7) if nstates == 61 else synth.protein(rng, 2, 0.7))
    tree = synth.random_tree(6, 0.4, 32)
    aln = synth.simulate(tree, model, 3 * npat, 33, gap_frac=0.05)
    npat = min(npat, aln.npat)
    aln.patterns = np.ascontiguousarray(aln.patterns[:, :npat])
    aln.weights = np.ascontiguousarray(aln.weights[:npat])
    trees = [PhyloTree.from_case(tree, model, aln, precision="mixed", scaling=scaling)
             for _ in range(nsess)]
    for k, t in enumerate(trees):
        t.session.set_rates(model.rates * (1.0 + 0.01 * k), model.props)
    for lengths in (False, True):
        if lengths:
            for k, t in enumerate(trees):
                e = k % tree.nedges
                t.setLength(int(tree.eu[e]), int(tree.ev[e]), 0.05 + 0.01 * k)
        alone = []
        for t in trees:
            t.clearAllPartialLH()
            alone.append(t.computeLikelihood())
            t.clearAllPartialLH()
        together = compute_likelihood_batch(trees)
        assert list(together) == alone
    for t in trees:
        t.close()
        t.session.close()
