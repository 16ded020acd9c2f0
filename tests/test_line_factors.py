"""What the solver holds per-line factors as -- the stream of nonzero entries, the
band without its zero blocks (what remains where the stream does not fit beside
it), the full band -- and that the solve reads the same bits from each, finite
ones: every compiled order, columns of one element and several."""
import ctypes as C

import numpy as np
import pytest

import atum_b200 as A
import parity as PT
from atum_b200 import workloads as W

pytestmark = pytest.mark.gpu

BAND, FACES, STREAM = 0, 1, 2


@pytest.mark.parametrize("split_rhs", [False, True])
@pytest.mark.parametrize("N,KV", [(1, 2), (2, 1), (3, 4), (4, 2), (5, 1), (6, 3), (7, 2)])
def test_factor_layouts(monkeypatch, N, KV, split_rhs):
    # (a second: the workload's own step, a hundred times the acoustic limit, overflows
    # on six columns)
    case = W.sphere_acoustic_wave(N=N, KH=1, KV=KV, steps=2, dt=1.0)
    out = []
    for env, kind in (("1", BAND), ("2", FACES), ("0", STREAM)):
        monkeypatch.setenv("ATB_BAND_DENSE", env)
        q = PT.to_dev(case.q0)
        s = A.ARK23(case.dg, case.lindg, q, case.dt, split_rhs=split_rhs)
        f = A._lib.lib().atb_detail_solver_lines
        f.argtypes = [C.c_void_p]
        assert f(s.h) == kind
        s.step(q, 2)
        out.append(PT.to_host(q))
        del s
    assert np.isfinite(out[0]).all()
    for o in out[1:]:
        assert np.array_equal(o, out[0])
