"""Op tables of the 61-state tensor-core traversal (images of internal children, tip tables with
the unknown state's row) at category counts that fill the two category groups of a block unevenly
and at the largest: few taxa, so that most children are tips, every state and gaps among them,
against the FP64 oracle and the FP32 CUDA-core form at the bars of the mixed form."""
import numpy as np
import pytest

from gems_b200 import PhyloTree, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncat,ntaxa", [(1, 3), (2, 5), (3, 9), (5, 5), (16, 9)])
def test_tables(gpu, ncat, ntaxa):
    rng = np.random.default_rng(200 + ncat)
    model = synth.codon_gy(rng, ncat, 0.5)
    tree = synth.random_tree(ntaxa, 0.2, 201 + ncat)
    aln = synth.simulate(tree, model, 500, 202 + ncat, gap_frac=0.1)
    lo = orc.OracleTree(tree, model, aln, safe=True).computeLikelihood()
    res = []
    for tc in (True, False):
        gt = PhyloTree.from_case(tree, model, aln, precision="mixed", scaling="safe")
        gt.session.set_tensor_cores(tc)
        lg, plg = gt.computeLikelihood(pattern_lh=True)
        assert abs(lg - lo) <= 1e-6 * abs(lo), (tc, lg, lo)
        res.append(plg)
        gt.close()
        gt.session.close()
    assert np.max(np.abs(res[0] - res[1]) / (np.abs(res[1]) + 1)) < 1e-5
