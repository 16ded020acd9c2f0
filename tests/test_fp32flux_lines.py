"""The FP32-flux form with nearly uniform and high-contrast lines side by side in
one warp: the form a line takes depends on the line alone, so the same bits for
every elements-per-CTA count and for an instance packed with others or alone; and
the form's own bound against FP64 on either side of it."""
import numpy as np
import pytest

import atum_b200 as A
import parity as PT
from test_fd_forms import contrast_state
from test_gpu_parity import make_dg

pytestmark = pytest.mark.gpu


def with_precision(dg, precision):
    return A.DGSEM(law=dg.law, grid=dg.grid, volume_form=dg.volume_form, surface_numericalflux=dg.surface_numericalflux,
                   directions=dg.directions, precision=precision)


def mixed_state(dg, seed):
    """Elements in turn nearly uniform and with a contrast of 12 inside."""
    q, far = contrast_state(dg, 1.02, seed), contrast_state(dg, 12.0, seed + 1)
    q[:, ::2] = far[:, ::2]
    return q


def apply(dg, q):
    dq = q.clone()
    dg(dq, q, 0.0, increment=True)
    return dq


@pytest.mark.parametrize("contrast", [1.05, 1.19, 1.25, 2.9, 12.0])
@pytest.mark.parametrize("law,dim,N,sf", [("euler", 2, 1, "rusanov"), ("euler", 2, 7, "rusanov"), ("eg", 2, 6, "rusanov"),
                                          ("eg", 2, 3, "roe"), ("eg", 3, 1, "rusanov"), ("eg", 3, 4, "ec"),
                                          ("eg", 3, 7, "rusanov")])
def test_mean_forms(law, dim, N, sf, contrast):
    dg = make_dg(law, dim, N, 3, "ec", sf, "reflect")
    q = PT.to_dev(contrast_state(dg, contrast))
    a, b = apply(with_precision(dg, "fp32flux"), q), apply(with_precision(dg, "fp64"), q)
    assert np.all(PT.field_rel_errors(PT.to_host(a), PT.to_host(b)) <= 1e-6)


@pytest.mark.parametrize("sf", ["rusanov", "roe"])
@pytest.mark.parametrize("law,dim,N,K", [("euler", 2, 2, 5), ("eg", 2, 3, 4), ("eg", 3, 1, 4), ("eg", 3, 2, 3),
                                         ("eg", 3, 3, 3)])
def test_mixed_lines(law, dim, N, K, sf):
    dgs = [with_precision(make_dg(law, dim, N, k, "ec", sf, "reflect"), "fp32flux") for k in (K, K - 1)]
    qs = [PT.to_dev(mixed_state(dg, 7 + i)) for i, dg in enumerate(dgs)]
    alone = [apply(dg, q) for dg, q in zip(dgs, qs)]
    for E in (1, 2, 3, 5, 7):
        if E * dgs[0].grid.cell.Np > 512:
            break
        A.batch.set_launch(dgs[0], E)
        assert (apply(dgs[0], qs[0]) == alone[0]).all(), E
    packed = A.batch.PackedDGSEM(dgs)
    for a, b in zip(packed.unpack(apply(packed, packed.pack(qs))), alone):
        assert (a == b).all()
