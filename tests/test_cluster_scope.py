"""Waits for data that another block of a cluster wrote (st.async, mapa addresses) acquire at
cluster scope: an mbarrier wait without a scope acquires within its own block only, which orders
copies and MMAs of that block but not what a neighbour sent.  Read from the sources: no GPU run
shows a missing acquire reliably."""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "gems_b200", "csrc")
BLOCK_WAITS = re.compile(r"\b(mbar_wait|mbar_try_wait|ws_wait)\s*\(")
CLUSTER_WAIT = "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64"


def code(path):
    txt = open(path).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", txt, flags=re.S))


def sources_that_send():
    return [p for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))
            if "st.async" in code(p) or "mapa." in code(p)]


def test_the_newton_exchange_is_covered():
    assert [os.path.basename(p) for p in sources_that_send()] == ["branch_kernels.cuh"]


@pytest.mark.parametrize("path", sources_that_send(), ids=os.path.basename)
def test_waits_acquire_at_cluster_scope(path):
    txt = code(path)
    assert not BLOCK_WAITS.search(txt), "a block-scope mbarrier wait beside cluster traffic"
    waits = re.findall(r"mbarrier\.(?:try_|test_)wait[\w.:]*", txt)
    assert waits and all(w == CLUSTER_WAIT for w in waits), waits
