"""The line-per-thread flux-differencing kernels on curved elements: the orders
the operator tests leave out, both two-point volume fluxes with the built-in and
the run-time surface flux, every form of the logarithmic means (lines within a
factor 1.2, within a factor 3, further apart), subsets of directions, tiles that
the element count does not fill -- against the oracle; and the same bits for
every elements-per-CTA count."""
import numpy as np
import pytest

import atum_b200 as A
import parity as PT
from atum_b200 import workloads as W
from test_cubedsphere import _cell
from test_fd_forms import contrast_state

pytestmark = pytest.mark.gpu


def shell_dg(law, N, vflux, sflux, KV=3, directions=None):
    if law == "euler":
        g = A.cubedspheregrid(_cell(N), np.linspace(1.0, 2.0, KV + 1), 1)
        lw = A.EulerLaw(3, problem=A.ReflectiveWall())
    else:
        case = W.sphere_zonal_flow(N=N, KH=1, KV=KV)
        g, lw = case.dg.grid, case.dg.law
    kw = {} if directions is None else {"directions": directions}
    return A.DGSEM(law=lw, grid=g, volume_form=A.FluxDifferencingForm(vflux), surface_numericalflux=sflux, **kw)


def check(orc, dg, q):
    od = orc.DGSEM(dg)
    want, moved = np.zeros_like(q), np.zeros_like(q)
    od(want, q, 0.0, False)
    od(moved, PT.ulp_perturbed(q), 0.0, False)
    # the bound of the operator tests: the oracle's own one-ulp spread, at least 1e-12
    bound = np.maximum(1e-12, PT.SPREAD_FACTOR * PT.field_rel_errors(moved, want))
    qd = PT.to_dev(q)
    got = PT.to_dev(np.zeros_like(q))
    dg(got, qd, 0.0, increment=False)
    err = PT.field_rel_errors(PT.to_host(got), want)
    assert np.all(err <= bound), (err, bound)


@pytest.mark.parametrize("contrast", [1.1, 2.5, 12.0])
@pytest.mark.parametrize("N,dirs", [(1, None), (3, None), (4, (1, 3)), (5, None), (6, (2,)), (7, None)])
def test_mean_forms_on_a_shell(orc, N, dirs, contrast):
    dg = shell_dg("euler", N, A.EntropyConservativeFlux(), A.RusanovFlux(), directions=dirs)
    check(orc, dg, contrast_state(dg, contrast))


@pytest.mark.parametrize("law,vflux,sflux", [("euler", "kg", "rusanov"), ("euler", "ec", "roe"), ("eg", "kg", "rusanov"),
                                             ("eg", "kg", "matrix"), ("eg", "ec", "rusanov"), ("eg", "ec", "ec")])
@pytest.mark.parametrize("N", [1, 4, 6, 7])
def test_fluxes_on_a_shell(orc, law, vflux, sflux, N):
    vf = {"ec": A.EntropyConservativeFlux(), "kg": A.KennedyGruberFlux()}[vflux]
    sf = {"rusanov": A.RusanovFlux(), "roe": A.RoeFlux(), "matrix": A.MatrixFlux(),
          "ec": A.EntropyConservativeFlux()}[sflux]
    dg = shell_dg(law, N, vf, sf)
    check(orc, dg, PT.random_state(dg) if law == "eg" else contrast_state(dg, 1.5))


@pytest.mark.parametrize("N", [1, 2, 3, 4])
def test_launch_shape_does_not_change_results(N):
    dg = shell_dg("euler", N, A.EntropyConservativeFlux(), A.RusanovFlux())
    q = PT.to_dev(contrast_state(dg, 2.0))
    outs = []
    for E in [e for e in (1, 2, 3, 4, 18) if e * dg.grid.cell.Np <= 512]:
        A.batch.set_launch(dg, E)
        dq = q.clone()
        dg(dq, q, 0.0, increment=True)
        outs.append(dq)
    assert len(outs) > 1
    for o in outs[1:]:
        assert (o == outs[0]).all()
