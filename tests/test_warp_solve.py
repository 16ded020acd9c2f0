"""The tile-sparse column solve with one and two warps per eight lines against
the dense-block solve, bit for bit: every compiled order (one to five row tiles
per block), line counts that do not fill the last group of eight, one element
per column and several, and enough lines for one warp per group."""
import numpy as np
import pytest

import atum_b200 as A
import parity as PT
from atum_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(1, (3, 1, 2)), (2, (3, 1, 1)), (2, (5, 3, 4)), (3, (13, 9, 5)), (4, (3, 2, 3)),
                                 (5, (3, 1, 2)), (6, (3, 2, 2)), (7, (2, 1, 3)), (1, (37, 36, 2)), (4, (14, 14, 2))])
def test_equals_dense_blocks(monkeypatch, N, K):
    case = W.bubble_3d(N=N, K=K, steps=2)
    out = []
    for dense in ("1", "0"):
        monkeypatch.setenv("ATB_BAND_DENSE", dense)
        q = PT.to_dev(case.q0)
        s = A.ARK23(case.dg, case.lindg, q, case.dt, split_rhs=False)
        s.step(q, 2)
        out.append(PT.to_host(q))
        del s
    assert np.array_equal(out[0], out[1])
