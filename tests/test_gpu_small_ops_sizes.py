"""Short op lists in a branch call's launch at the sizes where the launch changes: one and two
patterns of a pair, one block cluster of the Newton loop and several, rows beyond the registers',
streaming blocks on a share of the GPU, the largest pattern count and list that the rule takes and
the next ones.  Every call's list runs on stale partials, and the results, theta, partials and
counters have the bits of a session whose traversals are launches of their own (held to a launch
shape).  And a walk whose in-launch updates are shown to rescale."""
import numpy as np
import pytest

from gems_b200 import PhyloTree, synth
from gems_b200.api import GEMS_CHILD_PARTIAL, branch_struct, full_traversal

pytestmark = pytest.mark.gpu


def sessions(ntaxa, ncat, npat, precision, scaling, share, blen=0.2):
    rng = np.random.default_rng(77)
    model = synth.dna_gtr(rng, ncat, 0.5)
    tree = synth.random_tree(ntaxa, blen, 78)
    pats = rng.integers(0, 4, (ntaxa, npat)).astype(np.uint8)
    pats[rng.random((ntaxa, npat)) < 0.05] = synth.state_unknown(4)
    aln = synth.Alignment(ntaxa, 4, npat, pats, rng.integers(1, 9, npat).astype(float))
    out = []
    for separate in (False, True):
        s = PhyloTree.from_case(tree, model, aln, precision=precision, scaling=scaling).session
        s.set_newton_share(share)
        if separate:
            s.set_autotune(False, force_shape=0)
        out.append(s)
    return tree, out


def stretched(ops, br, f):
    return ([o[:5] + (o[5] * f, o[6] * f) for o in ops],
            branch_struct(br.dad_slot, br.node_kind, br.node_id, br.length * f))


def launches(s, call):
    n = s.launch_count()
    got = call(s)
    return got, s.launch_count() - n


@pytest.mark.parametrize("npat,ncat,share,precision,scaling", [
    (9_000, 4, 1, "fp64", "norm"),       # several clusters
    (18_501, 4, 1, "fp64", "safe"), (18_501, 4, 1, "mixed", "norm"),
    (18_501, 4, 4, "fp64", "norm"),      # rows beyond the registers', read again
    (18_501, 4, 16, "mixed", "safe"), (5_000, 16, 16, "fp64", "safe"),  # streaming blocks
    (2_600, 4, 64, "fp64", "norm"), (9_000, 2, 64, "mixed", "norm"),
    (30_000, 4, 1, "fp64", "safe"), (30_000, 4, 1, "mixed", "safe"),    # second patterns of pairs
    (32_768, 4, 1, "fp64", "norm"), (32_768, 2, 1, "mixed", "safe"),
])
def test_same_bits(gpu, npat, ncat, share, precision, scaling):
    tree, (a, b) = sessions(6, ncat, npat, precision, scaling, share)
    ops, br = full_traversal(tree)
    f = 1.0
    for call in (lambda s: s.branch_lnl(o, q, pattern_lh=True),
                 lambda s: s.branch_derv(o, q, df_frac=True),
                 lambda s: s.newton_branch(o, q, True, 1e-6, 10.0, 1e-6, 30),
                 lambda s: s.newton_branch(o, q, True, 1e-6, 10.0, 1e-6, 30)):
        f *= 1.17
        o, q = stretched(ops, br, f)
        (x, na), (y, nb) = launches(a, call), launches(b, call)
        assert na < nb
        for u, v in zip(x, y):
            np.testing.assert_array_equal(u, v)
        for slot in range(tree.ntaxa - 2):
            for u, v in zip(a.get_partial(slot), b.get_partial(slot)):
                np.testing.assert_array_equal(u, v)
        if call.__code__.co_names[0] != "branch_lnl":
            for u, v in zip(a.get_theta(), b.get_theta()):
                np.testing.assert_array_equal(u, v)
    for s in (a, b):
        s.close()


@pytest.mark.parametrize("ntaxa,ncat,npat,inside", [
    (18, 4, 333, True), (18, 2, 333, True),        # 16 updates: the longest list
    (19, 4, 333, False), (19, 2, 333, False),      # 17
    (18, 5, 333, False), (14, 5, 333, True),       # 80 and 60 rows of exponentials (64 at most)
    (6, 4, 32_768, True), (6, 4, 32_769, False),   # the largest pattern count and the next
    (6, 1, 333, False),                            # one category
])
def test_rule(gpu, ntaxa, ncat, npat, inside):
    tree, (a, b) = sessions(ntaxa, ncat, npat, "fp64", "safe", 1)
    o, q = full_traversal(tree)
    (x, na), (y, nb) = [launches(s, lambda s: s.branch_derv(o, q)) for s in (a, b)]
    assert x == y
    assert (na < nb) == inside and (na == 1) == inside
    for s in (a, b):
        s.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("scaling", ["norm", "safe"])
def test_updates_rescale(gpu, precision, scaling):
    tree, (a, b) = sessions(220, 4, 700, precision, scaling, 1, blen=1.5)
    ops, br = full_traversal(tree)
    for s in (a, b):
        s.traverse(ops)
    o, q = stretched(ops[-16:], br, 1.1)
    call = lambda s: s.branch_derv(o, q)
    (x, na), (y, nb) = launches(a, call), launches(b, call)
    assert x == y and na == 1 and nb > 1
    rescaled = 0
    for dst, lk, li, rk, ri, _, _ in o:
        u, v = a.get_partial(dst), b.get_partial(dst)
        np.testing.assert_array_equal(u[0], v[0])
        np.testing.assert_array_equal(u[1], v[1])
        below = sum(a.get_partial(i)[1].astype(int) for k, i in ((lk, li), (rk, ri))
                    if k == GEMS_CHILD_PARTIAL)
        rescaled += int(np.sum(u[1] > below))
    assert rescaled > 0
    for s in (a, b):
        s.close()
