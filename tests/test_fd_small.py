"""The line kernels' mode for grids of one wave (pairs and faces spread over the
threads of a CTA, the default on small grids) against one thread per line
(atb_op_set_launch): the same bits, over the orders, laws, two-point fluxes,
surface fluxes, precision forms, subsets of directions, every form of the
logarithmic means side by side, every epilogue of the steppers and the fused
ARK23 stage; and an instance packed with others on a grid too large for the mode."""
import numpy as np
import pytest

import atum_b200 as A
import parity as PT
import problems as P
from test_fd_forms import contrast_state
from test_fp32flux_lines import mixed_state, with_precision
from test_gpu_parity import make_dg

pytestmark = pytest.mark.gpu


def both(make, run):
    """``run`` on the operator of ``make()`` as created, and with one thread per line."""
    out = []
    for lines in (False, True):
        dg = make()
        if lines:
            A.batch.set_launch(dg, 1)
        out.append(run(dg))
    return out


def state(dg, kind):
    if kind == "mixed":
        q = mixed_state(dg, 3)
        q[:, ::3] = contrast_state(dg, 1.5, 8)[:, ::3]
        return q
    return PT.random_state(dg)


@pytest.mark.parametrize("precision", ["fp64", "fp32flux"])
@pytest.mark.parametrize("N", range(1, 8))
@pytest.mark.parametrize("law,dim,form,sf,dirs", [
    ("euler", 2, "ec", "rusanov", None), ("euler", 2, "ec", "roe", (2,)), ("euler", 3, "ec", "rusanov", None),
    ("eg", 2, "ec", "rusanov", None), ("eg", 2, "ec", "matrix", (1,)), ("eg", 3, "ec", "rusanov", None),
    ("eg", 3, "ec", "roe", (1, 3)), ("eg_cor", 3, "ec", "rusanov", None), ("eg", 3, "kg", "rusanov", (2, 3)),
    ("eg", 3, "kg", "ec", None), ("eg_pde", 3, "weak", "rusanov", None), ("eg", 3, "weak", "roe", (3,)),
    ("eg_pde", 3, "ec", "matrix", None)])
def test_operator(law, dim, form, sf, dirs, N, precision):
    if form == "weak" and precision != "fp64":
        pytest.skip("no FP32-flux weak form")
    dg = make_dg(law, dim, N, 3, form, sf, "reflect", dirs=dirs)
    for kind in ("smooth", "mixed"):
        q = PT.to_dev(state(dg, kind))
        base = PT.to_dev(np.random.default_rng(2).standard_normal(tuple(q.shape)))

        def run(d):
            dq = base.clone()
            d(dq, q, 0.0, increment=True)
            d(dq, q, 0.0, increment=False) if N % 2 else None
            return dq
        a, b = both(lambda: with_precision(dg, precision), run)
        assert (a == b).all(), (kind, float((a - b).abs().max()))


@pytest.mark.parametrize("precision", ["fp64", "fp32flux"])
@pytest.mark.parametrize("scheme,N", [("LSRK54", 2), ("LSRK54", 7), ("LSRK144", 4), ("RLSRK54", 3)])
def test_explicit_steps(scheme, N, precision):
    def make():
        return P.vortex_c1(N=N, K=5, precision=precision).dg

    c = P.vortex_c1(N=N, K=5, precision=precision)

    def run(dg):
        q = PT.to_dev(c.q0)
        getattr(A, scheme)(dg, q, c.dt).step(q, 3)
        return q
    a, b = both(make, run)
    assert (a == b).all()


@pytest.mark.parametrize("precision", ["fp64", "fp32flux"])
@pytest.mark.parametrize("N", range(1, 8))
def test_ark23_steps(N, precision):
    c = P.bubble_3d(N=N, K=3, imex=True, steps=2, precision=precision)
    out = []
    for lines in (False, True):
        for fuse in (True, False):
            cc = P.bubble_3d(N=N, K=3, imex=True, steps=2, precision=precision)
            if lines:
                A.batch.set_launch(cc.dg, 1)
            q = PT.to_dev(c.q0)
            s = A.ARK23(cc.dg, cc.lindg, q, c.dt, split_rhs=False)
            s.fuse(fuse)
            s.step(q, 2)
            out.append(q)
    assert (out[0] == out[2]).all() and (out[1] == out[3]).all()


@pytest.mark.parametrize("precision", ["fp64", "fp32flux"])
def test_packed_on_a_large_grid(precision):
    """One small instance among many: the pack takes one thread per line."""
    cs = [P.vortex_c1(N=5, K=k, precision=precision) for k in (7, 64, 64, 64)]
    qs = [PT.to_dev(c.q0) for c in cs]
    packed = A.batch.PackedDGSEM([c.dg for c in cs])
    q = packed.pack(qs)
    dq = q.clone()
    packed(dq, q, 0.0, increment=False)
    alone = qs[0].clone()
    cs[0].dg(alone, qs[0], 0.0, increment=False)
    assert (packed.unpack(dq)[0] == alone).all()
