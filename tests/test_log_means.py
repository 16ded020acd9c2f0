"""The logarithmic means of lines whose values lie more than a factor 3 apart: the
scalar function against 40 digits, and operators on states outside the positive
ones (densities or pressures of one negative sign, or of both signs) against the
oracle."""
import ctypes as C

import numpy as np
import pytest

import atum_b200 as A
import parity as PT
from test_curved_fd import shell_dg
from test_fd_forms import contrast_state
from test_gpu_parity import make_dg

pytestmark = pytest.mark.gpu


def device_math(fn, x, y):
    import torch
    f = A._lib.lib().atb_detail_math
    f.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]
    xd, yd = (torch.as_tensor(v, dtype=torch.float64, device="cuda").contiguous() for v in (x, y))
    out = torch.empty_like(xd)
    assert f(fn, xd.data_ptr(), yd.data_ptr(), out.data_ptr(), xd.numel(),
             torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


def test_log_mean_of_any_two_values():
    mp = pytest.importorskip("mpmath")
    rng = np.random.default_rng(1)
    # ratios about every rounding of the scale (powers of two times 1.5^(+-1)),
    # equal and nearly equal values, ratios up to 1e200, both signs
    near = np.concatenate([2.0 ** k * 1.5 ** s * (1 + d) for k in range(-4, 5) for s in (-1, 0, 1)
                           for d in (np.array([0.0, 1e-15, -1e-15, 1e-7, -1e-7, 1e-3, -1e-3]),)])
    ratio = np.concatenate([near, 10.0 ** rng.uniform(-3, 3, 1500), 1 + rng.uniform(-0.5, 0.5, 500),
                            10.0 ** rng.uniform(-200, 200, 200)])
    y = 10.0 ** rng.uniform(-8, 8, ratio.size) * np.where(rng.random(ratio.size) < 0.2, -1.0, 1.0)
    x = y * ratio
    got = device_math(0, x, y)
    with mp.workdps(40):
        want = [mp.mpf(a) if a == b else (mp.mpf(a) - mp.mpf(b)) / mp.log(mp.mpf(a) / mp.mpf(b)) for a, b in zip(x, y)]
        err = max(float(abs(mp.mpf(g) / w - 1)) for g, w in zip(got, want))
    # 2 f F(f^2) to 4 x 2^-53 of at most 0.406, in a logarithm of at least 0.287; its
    # sum, the difference, the reciprocal and the product: 8.5 x 2^-53 in all
    assert err <= 8.5 * 2.0 ** -53, err / 2.0 ** -53


def _states(dg):
    """(name, state): all densities negative; all pressures negative; pressures of
    both signs in every line."""
    q = contrast_state(dg, 12.0)
    law, dim = dg.law, dg.law.dim
    Phi = dg.auxstate_host()[0] if law.naux else 0.0
    ke = sum(q[1 + d] ** 2 for d in range(dim)) / (2 * q[0])
    inner = q[dim + 1] - ke - q[0] * Phi
    yield "rho < 0", -q
    sign = np.where(np.random.default_rng(9).random(q[0].shape) < 0.4, -1.0, 1.0)
    sign[:, ::2], sign[:, 1::2] = 1.0, -1.0
    for name, s in (("p < 0", -1.0), ("mixed", sign)):
        p = q.copy()
        p[dim + 1] = ke + q[0] * Phi + s * inner
        yield name, p


@pytest.mark.parametrize("law,dim,N", [("euler", 2, 3), ("euler", 2, 5), ("euler", 3, 3), ("eg", 3, 3), ("shell", 3, 3)])
def test_states_outside_the_positive(orc, law, dim, N):
    if law == "shell":
        dg = shell_dg("euler", N, A.EntropyConservativeFlux(), A.CentralFlux())
    else:
        dg = make_dg(law, dim, N, 3, "ec", "central", "reflect")
    od = orc.DGSEM(dg)
    for name, q in _states(dg):
        want, moved = np.zeros_like(q), np.zeros_like(q)
        od(want, q, 0.0, False)
        od(moved, PT.ulp_perturbed(q), 0.0, False)
        got = PT.to_dev(np.zeros_like(q))
        dg(got, PT.to_dev(q), 0.0, increment=False)
        got = PT.to_host(got)
        assert np.array_equal(np.isnan(got), np.isnan(want)), name
        assert np.isnan(want).any() == (name == "mixed"), name
        # the bound of the operator tests; p / rho of both signs cancel in B_1 + B_2,
        # so the oracle's own one-ulp spread counts too (as on curved elements)
        fin = np.isfinite(want) & np.isfinite(moved)
        want, moved, got = (np.where(fin, v, 0.0) for v in (want, moved, got))
        bound = np.maximum(1e-12, PT.SPREAD_FACTOR * PT.field_rel_errors(moved, want))
        err = PT.field_rel_errors(got, want)
        assert np.all(err <= bound), (name, err, bound)
