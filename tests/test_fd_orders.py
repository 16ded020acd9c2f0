"""Line kernels at the orders and surface fluxes that the operator tests leave out:
Kennedy-Gruber (3-D Euler-gravity) and shallow water (2-D) at every compiled order
against the oracle, their FP32-flux forms against FP64, and the fused ARK23 stage
with surface fluxes other than Rusanov's against two launches and the oracle."""
import numpy as np
import pytest

import atum_b200 as A
import parity as PT
import problems as P
from test_fp32flux_lines import apply, with_precision
from test_gpu_parity import FLUX, make_dg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("law,dim,form,sf,dirs", [("eg", 3, "kg", "rusanov", None), ("eg", 3, "kg", "matrix", (1, 3)),
                                                  ("sw_topo", 2, "ec", "rusanov", None), ("sw_topo", 2, "ec", "roe", None),
                                                  ("sw", 2, "ec", "ec", (2,)), ("sw_cor", 2, "ec", "central", None)])
def test_operator(orc, law, dim, form, sf, dirs, N):
    dg = make_dg(law, dim, N, 3, form, sf, "reflect" if law == "eg" else "periodic", dirs=dirs)
    q = PT.random_state(dg)
    want = np.zeros_like(q)
    orc.DGSEM(dg)(want, q, 0.0, increment=False)
    qd = PT.to_dev(q)
    got = PT.to_dev(np.zeros_like(q))
    dg(got, qd, 0.0, increment=False)
    # one operator application: the bound of the operator tests
    assert PT.rel_dof_error(PT.to_host(got), want) <= 1e-12
    # the FP32-flux form's own bound (test_precision.py)
    a, b = apply(with_precision(dg, "fp32flux"), qd), apply(with_precision(dg, "fp64"), qd)
    assert np.all(PT.field_rel_errors(PT.to_host(a), PT.to_host(b)) <= 1e-6)


@pytest.mark.parametrize("precision", ["fp64", "fp32flux"])
@pytest.mark.parametrize("N,sf,lin", [(2, "roe", "rusanov"), (3, "rusanov", "central"), (4, "matrix", "central"),
                                      (5, "ec", "rusanov"), (7, "roe", "rusanov")])
def test_fused_stage(orc, N, sf, lin, precision):
    c = P.bubble_3d(N=N, K=3, imex=True, steps=2)
    kw = dict(law=c.dg.law, grid=c.dg.grid, volume_form=c.dg.volume_form, surface_numericalflux=FLUX[sf])
    c.dg = A.DGSEM(precision=precision, **kw)
    c.lindg = A.DGSEM(law=c.lindg.law, grid=c.dg.grid, surface_numericalflux=FLUX[lin], directions=(3,))
    c.q0 = c.q0 * (1 + 1e-4 * np.random.default_rng(3).standard_normal(c.q0.shape))
    out = []
    for fuse in (True, False):
        q = PT.to_dev(c.q0)
        s = A.ARK23(c.dg, c.lindg, q, c.dt, split_rhs=False)
        s.fuse(fuse)
        s.step(q, 2)
        out.append(PT.to_host(q))
    # the bounds of the fused-stage tests
    d = np.max(np.abs(out[0] - out[1])) / np.max(np.abs(out[1]))
    assert d <= (1e-14 if precision == "fp64" else 1e-6), d
    if precision == "fp64":
        want, spread = PT.ulp_spread(orc, c, [2])
        PT.assert_parity(f"ARK23 N={N} {sf}/{lin}", out[0], want[0], 1e-12, spread[0])
