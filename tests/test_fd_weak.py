"""The weak form of 3-D Euler-gravity on the line-per-thread kernel against the
oracle: every compiled order, subsets of directions, tiles that the element
count does not fill, the pressure and density less the reference state
(pde_level_balance), Coriolis, the built-in and the run-time surface flux; and
the same bits for every elements-per-CTA count."""
import numpy as np
import pytest

import atum_b200 as A
import parity as PT
from test_fd_forms import contrast_state
from test_gpu_parity import make_dg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("law,N,sf,dirs", [("eg", 1, "rusanov", None), ("eg", 2, "rusanov", (1, 2)),
                                           ("eg", 3, "roe", None), ("eg", 4, "rusanov", (3,)),
                                           ("eg", 5, "central", None), ("eg", 6, "rusanov", None),
                                           ("eg", 7, "rusanov", None), ("eg_pde", 4, "rusanov", None),
                                           ("eg_pde", 6, "matrix", None), ("eg_cor", 1, "rusanov", (1, 3)),
                                           ("eg_cor", 7, "ec", None)])
def test_weak_matches_oracle(orc, law, N, sf, dirs):
    dg = make_dg(law, 3, N, 3, "weak", sf, "reflect", dirs=dirs)
    q = contrast_state(dg, 2.0)
    base = np.random.default_rng(4).standard_normal(q.shape)
    for inc in (False, True):
        want = base.copy()
        orc.DGSEM(dg)(want, q, 0.0, increment=inc)
        qd, got = PT.to_dev(q), PT.to_dev(base)
        dg(got, qd, 0.0, increment=inc)
        # one operator application: the bound of the operator tests
        assert PT.rel_dof_error(PT.to_host(got), want) <= 1e-12


@pytest.mark.parametrize("N", [1, 3, 4])
def test_launch_shape_does_not_change_results(N):
    dg = make_dg("eg", 3, N, 3, "weak", "rusanov")
    q = PT.to_dev(contrast_state(dg, 2.0))
    outs = []
    for E in [e for e in (1, 2, 3, 4, 8) if e * dg.grid.cell.Np <= 512]:
        A.batch.set_launch(dg, E)
        dq = q.clone()
        dg(dq, q, 0.0, increment=True)
        outs.append(dq)
    for o in outs[1:]:
        assert (o == outs[0]).all()
