"""Tip tables of the 61-state tensor-core traversal (FP64 mma) have the bits of the CUDA-core form's,
which sum in index order on FP64 FMA: a node of two tips is a product of one entry of each, in both
forms, so its partials are equal where both states are known, for every pair of states."""
import numpy as np
import pytest

from gems_b200 import Session, synth
from gems_b200.api import GEMS_CHILD_TIP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncat", [1, 3, 4, 8, 16])
def test_two_tips(gpu, ncat):
    rng = np.random.default_rng(300 + ncat)
    model = synth.codon_gy(rng, ncat, 0.5)
    a, b = np.divmod(np.arange(61 * 61), 61)
    tips = np.stack([a, b, a]).astype(np.uint8)
    got = []
    for tc in (True, False):
        s = Session(3, tips.shape[1], 61, ncat, 2, "mixed", "safe")
        s.upload_tips(tips)
        s.upload_patterns(np.ones(tips.shape[1]))
        s.set_model(model.eval, model.evec, model.inv_evec, model.rates, model.props)
        s.set_tensor_cores(tc)
        s.traverse([(0, GEMS_CHILD_TIP, 0, GEMS_CHILD_TIP, 1, 0.07, 0.9),
                    (1, GEMS_CHILD_TIP, 1, GEMS_CHILD_TIP, 2, 2.5, 1e-4)])
        got.append([s.get_partial(0), s.get_partial(1)])
        s.close()
    for x, y in zip(*got):
        np.testing.assert_array_equal(x[0], y[0])
        np.testing.assert_array_equal(x[1], y[1])
        assert x[0].max() > 0
