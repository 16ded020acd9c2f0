"""Per-line banded solve from the stream of nonzero factor entries against the
solve that reads the full band, bit for bit: every compiled order, one element
per column and several, line counts that do not fill the last warp, and both
forms of the right-hand side (given whole; formed from stage tendencies)."""
import numpy as np
import pytest

import atum_b200 as A
import parity as PT
from atum_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split_rhs", [False, True])
@pytest.mark.parametrize("N,KV", [(1, 1), (1, 4), (2, 3), (4, 2), (5, 3), (6, 1), (7, 2)])
def test_stream_equals_band(monkeypatch, N, KV, split_rhs):
    case = W.sphere_zonal_flow(N=N, KH=1, KV=KV, steps=2)
    out = []
    for dense in ("1", "0"):
        monkeypatch.setenv("ATB_BAND_DENSE", dense)
        q = PT.to_dev(case.q0)
        s = A.ARK23(case.dg, case.lindg, q, case.dt, split_rhs=split_rhs)
        s.step(q, 2)
        out.append(PT.to_host(q))
        del s
    assert np.array_equal(out[0], out[1], equal_nan=True)
