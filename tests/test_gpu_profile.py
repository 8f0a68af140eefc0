"""Kernel timing runs node updates and theta in launches of their own (so that their ids have
times): derivatives, Newton lengths, lnL and theta have the bits of a session without it."""
import numpy as np
import pytest

from gems_b200 import PhyloTree, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ncat,precision,scaling", [
    (4, 4, "fp64", "norm"), (4, 4, "fp64", "safe"), (4, 4, "mixed", "safe"), (4, 1, "mixed", "norm"),
    (20, 4, "fp64", "safe"), (20, 4, "mixed", "norm"), (61, 3, "fp64", "safe"),
])
def test_same_bits_and_every_id_counts(gpu, n, ncat, precision, scaling):
    rng = np.random.default_rng(41)
    make = {4: synth.dna_gtr, 20: synth.protein, 61: synth.codon_gy}[n]
    model = make(rng, ncat, 0.5)
    tree = synth.random_tree(12, 0.2, 42)
    aln = synth.simulate(tree, model, 900, 43, gap_frac=0.05)
    runs = []
    for on in (False, True):
        t = PhyloTree.from_case(tree, model, aln, precision=precision, scaling=scaling)
        t.session.profile(on)
        out = [t.computeLikelihood()]
        for u, v, x in zip(tree.eu.tolist(), tree.ev.tolist(), tree.length.tolist()):
            out.append(t.computeFuncDerv(u, v, x, True))
            out.append(t.computeLikelihoodFromBuffer())
            t.optimizeOneBranch(u, v)
        out += t.getBranchLengths().tolist()
        counts = [t.session.profile_read(k)[1] for k in range(6)]
        assert all(counts) if on else not any(counts)
        runs.append(out)
        t.close()
        t.session.close()
    assert runs[0] == runs[1]
