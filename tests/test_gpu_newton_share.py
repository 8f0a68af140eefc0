"""Newton loops of sessions that share the GPU, with more patterns than their blocks hold: small
blocks on many SMs, one cluster of them and several, theta formed in the launch, read as stored and
read again in every evaluation.  The lengths are those of the whole GPU's loop to 1e-8 (the same
sums, grouped by other blocks: rounding, far below the loop's own tolerance)."""
import numpy as np
import pytest

from gems_b200 import PhyloTree, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ncat,npat,share,precision,scaling", [
    (4, 16, 5_000, 4, "fp64", "safe"), (4, 16, 20_000, 2, "mixed", "norm"),
    (4, 1, 33_001, 16, "fp64", "norm"), (4, 4, 2_600, 64, "mixed", "safe"),
    (20, 4, 5_000, 4, "fp64", "norm"), (20, 7, 3_001, 16, "fp64", "safe"),
    (20, 4, 3_001, 16, "mixed", "safe"), (61, 1, 1_500, 16, "fp64", "safe"),
    (61, 9, 700, 16, "fp64", "norm"), (61, 4, 700, 16, "mixed", "safe"),
])
def test_lengths(gpu, n, ncat, npat, share, precision, scaling):
    rng = np.random.default_rng(51)
    make = {4: synth.dna_gtr, 20: synth.protein, 61: synth.codon_gy}[n]
    model = make(rng, ncat, 0.5)
    tree = synth.random_tree(12, 0.2, 52)
    pats = rng.integers(0, n, (12, npat)).astype(np.uint8)
    pats[:, :] = np.where(rng.random((12, npat)) < 0.7, pats[:1], pats)
    aln = synth.Alignment(12, n, npat, pats, np.ones(npat))
    edges = list(zip(tree.eu.tolist(), tree.ev.tolist()))[::4]
    got = []
    for k in (1, share):
        t = PhyloTree.from_case(tree, model, aln, precision=precision, scaling=scaling)
        t.session.set_newton_share(k)
        for u, v in edges:
            t.optimizeOneBranch(u, v)
        got.append(t.getBranchLengths())
        t.close()
        t.session.close()
    np.testing.assert_allclose(got[1], got[0], rtol=1e-8, atol=1e-10)
