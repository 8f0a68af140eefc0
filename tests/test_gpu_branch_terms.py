"""Branch terms (lanes of a warp share a pattern's theta): lnL, derivatives, lnL from the stored
theta and the Newton loop, for blocks that split evenly over the lanes and ones that leave lanes
partly empty (odd blocks: 61 states with an odd category count), pattern counts around a block's,
tip and internal branches, NORM and SAFE, and a Newton grid so small that most patterns are read
again at every evaluation.  Against the FP64 oracle: FP64 1e-9 (sums of up to 1e3 x 976 terms of
one sign or nearly: rounding far below), mixed 1e-6 for lnL and 1e-5 of |ddf| for derivatives."""
import numpy as np
import pytest

from conftest import ptn_invar
from gems_b200 import PhyloTree, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def case(n, ncat, npat, seed, p_invar=0.0):
    rng = np.random.default_rng(seed)
    make = {4: synth.dna_gtr, 20: synth.protein, 61: synth.codon_gy}[n]
    model = make(rng, ncat, 0.5)
    model.p_invar = p_invar
    tree = synth.random_tree(14, 0.15, seed + 1)
    sites = 4 * npat + 64
    aln = synth.simulate(tree, model, sites, seed + 2, gap_frac=0.05)
    npat = min(npat, aln.npat)
    aln.patterns = np.ascontiguousarray(aln.patterns[:, :npat])
    aln.weights = aln.weights[:npat].copy()
    return tree, model, aln


def check(n, ncat, npat, seed, safe, precision="fp64", share=1, p_invar=0.0):
    tree, model, aln = case(n, ncat, npat, seed, p_invar)
    ot = orc.OracleTree(tree, model, aln, safe=safe, const_char=aln.const_char())
    gt = PhyloTree.from_case(tree, model, aln, precision=precision,
                             scaling="safe" if safe else "norm", invar=ptn_invar(model, aln))
    gt.session.set_newton_share(share)
    fp64 = precision == "fp64"
    tol = 1e-9 if fp64 else 1e-6
    lo, plo = ot.computeLikelihood(pattern_lh=True)
    lg, plg = gt.computeLikelihood(pattern_lh=True)
    assert abs(lg - lo) <= tol * abs(lo)
    assert np.allclose(plg, plo, rtol=tol, atol=1e-12 if fp64 else 1e-5)
    edges = list(zip(tree.eu.tolist(), tree.ev.tolist(), tree.length.tolist()))
    tip = next(e for e in edges if min(e[:2]) < tree.ntaxa)
    inner = next(e for e in edges if min(e[:2]) >= tree.ntaxa)
    for u, v, x in (tip, inner):
        fo, dfo = ot.computeFuncDerv(u, v, x, new_branch=True)
        fg, dfg = gt.computeFuncDerv(u, v, x, new_branch=True)
        dtol = (1e-9 if fp64 else 1e-5) * max(abs(dfo), abs(fo))
        assert abs(fg - fo) <= dtol and abs(dfg - dfo) <= dtol
        bo, bg = ot.computeLikelihoodFromBuffer(), gt.computeLikelihoodFromBuffer()
        assert abs(bg - bo) <= tol * abs(bo)
        ot.optimizeOneBranch(u, v)
        gt.optimizeOneBranch(u, v)
        a, b = ot.getBranchLength(u, v), gt.getBranchLength(u, v)
        assert abs(a - b) <= (1e-8 if fp64 else 1e-4) * max(a, 1e-2)
    gt.close()
    gt.session.close()


SIZES = [1, 15, 64, 65, 127, 129, 513]


@pytest.mark.parametrize("npat", SIZES)
@pytest.mark.parametrize("n,ncat,safe", [(4, 4, False), (4, 1, True), (4, 3, True), (20, 4, True),
                                         (61, 1, True), (61, 4, True)])
def test_pattern_counts(gpu, n, ncat, safe, npat):
    check(n, ncat, npat, 600 + npat, safe)


@pytest.mark.parametrize("ncat", [1, 2, 3, 4, 5, 6, 7, 8, 11, 16])
@pytest.mark.parametrize("safe", [False, True], ids=["norm", "safe"])
@pytest.mark.parametrize("n", [4, 20, 61])
def test_categories(gpu, n, ncat, safe):
    check(n, ncat, 90, 640 + ncat, safe, p_invar=0.1 if ncat == 4 else 0.0)


@pytest.mark.parametrize("n,ncat", [(4, 1), (4, 4), (4, 8), (20, 4), (61, 4)])
@pytest.mark.parametrize("safe", [False, True], ids=["norm", "safe"])
def test_mixed(gpu, n, ncat, safe):
    check(n, ncat, 130, 670 + ncat, safe, precision="mixed")


@pytest.mark.parametrize("n,ncat", [(4, 4), (4, 6), (20, 4), (61, 3), (61, 8)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_newton_reads_theta_again(gpu, n, ncat, precision):
    check(n, ncat, 2600, 690 + ncat, True, precision=precision, share=64)
