"""The flux-differencing kernels' forms of the logarithmic means -- a line whose
densities and rho/p lie within a factor 1.2, within a factor 3, or further
apart takes another polynomial or the logarithms -- against the oracle, over
the orders' ends, the laws, subsets of directions and tiles that the element
count does not fill; and the same bits for every elements-per-CTA count."""
import numpy as np
import pytest

import atum_b200 as A
import parity as PT
from test_gpu_parity import make_dg

pytestmark = pytest.mark.gpu


def contrast_state(dg, contrast, seed=3):
    """Densities and pressures spread over a factor ``contrast`` in every element."""
    rng = np.random.default_rng(seed)
    law, shape = dg.law, (len(dg.grid), dg.grid.cell.Np)
    scale = 1e5 if dg.law.naux else 1.0
    rho = contrast ** rng.uniform(0, 1, shape)
    p = scale * contrast ** rng.uniform(0, 1, shape)
    m = [rho * np.sqrt(scale) * rng.uniform(-0.5, 0.5, shape) for _ in range(law.dim)]
    E = law.energy(rho, m, p, dg.auxstate_host()[0]) if law.naux else law.energy(rho, m, p)
    return np.stack([rho, *m, E])


@pytest.mark.parametrize("contrast", [1.05, 1.19, 1.25, 2.9, 12.0])
@pytest.mark.parametrize("law,dim,N,dirs", [("euler", 2, 1, None), ("euler", 2, 7, None), ("eg", 3, 1, None),
                                            ("eg", 3, 4, (1, 3)), ("eg", 3, 6, (2,)), ("eg", 3, 7, None),
                                            ("euler", 3, 3, None), ("eg", 2, 5, (2,))])
def test_mean_forms(orc, law, dim, N, dirs, contrast):
    dg = make_dg(law, dim, N, 3, "ec", "rusanov", "reflect", dirs=dirs)
    q = contrast_state(dg, contrast)
    want = np.zeros_like(q)
    orc.DGSEM(dg)(want, q, 0.0, increment=False)
    qd = PT.to_dev(q)
    got = PT.to_dev(np.zeros_like(q))
    dg(got, qd, 0.0, increment=False)
    # one operator application: the bound of the operator tests
    assert PT.rel_dof_error(PT.to_host(got), want) <= 1e-12


@pytest.mark.parametrize("precision", ["fp64", "fp32flux"])
@pytest.mark.parametrize("law,dim,N", [("euler", 2, 3), ("eg", 3, 2), ("eg", 3, 4), ("sw_topo", 2, 4)])
def test_launch_shape_does_not_change_results(law, dim, N, precision):
    dg = make_dg(law, dim, N, 5 if dim == 2 else 3, "ec", "rusanov")
    dg = A.DGSEM(law=dg.law, grid=dg.grid, volume_form=dg.volume_form, surface_numericalflux=dg.surface_numericalflux,
                 precision=precision)
    q = PT.to_dev(PT.random_state(dg) if law == "sw_topo" else contrast_state(dg, 2.0))
    outs = []
    for E in [e for e in (1, 2, 3, 7, 14) if e * dg.grid.cell.Np <= 512]:
        A.batch.set_launch(dg, E)
        dq = q.clone()
        dg(dq, q, 0.0, increment=True)
        outs.append(dq)
    for o in outs[1:]:
        assert (o == outs[0]).all()
