"""The marching y and z sweeps (meshes of at least a wave of columns) against the
CPU restatement, beyond the cubes that test_gpu_solver.py steps.

FP64: relative L1 <= 1e-11 per field against the field's own scale, the fixtures'
bound.  Mixed: 2e-5, FP32's 6e-8 through the fluxes of a step times the
cancellation of the random states' jumps (test_gpu_solver.py).
"""
import numpy as np
import pytest

from test_gpu_solver import GAMMA, _state

pytestmark = pytest.mark.gpu


def _check(d, o, n, precision):
    uo, bo = o.get_state()
    u, b = d.get_state()
    assert d.status() == 0
    tol = 1e-11 if precision == 2 else 2e-5
    for k in range(5):
        scale = np.abs(uo[..., 2:5]).max(-1).sum() if k >= 2 else np.abs(uo[..., k]).sum()
        assert np.abs(u[..., k] - uo[..., k]).sum() <= tol * scale, "field %d" % k
    own = np.s_[:, 2:n[2] + 2, 2:n[1] + 2, 2:n[0] + 2]
    assert np.abs(b[own] - bo[own]).sum() <= tol * np.abs(bo[own]).sum()


@pytest.mark.parametrize("precision", [2, 1])
def test_flat_block(precision):
    """A flat block whose (x, z) planes have rows times sites above 2^32, the bound
    of a quotient by one multiply-high without a shift; (x, y) planes stay below."""
    from kratos_b200 import Dynamics
    from oracle.kr_oracle import OracleMesh
    nb, n = (1, 1, 1), (29500, 4, 8)
    x_max = tuple(k / 8 for k in n)                       # cubic cells
    u0, b0 = _state(nb, n, "subsonic", 3)
    o = OracleMesh(True, nb, n, GAMMA, x_max=x_max)
    o.set_state(u0, b0)
    o.step(2)
    d = Dynamics(True, nb, n, gamma=GAMMA, precision=precision, x_max=x_max)
    d.set_state(u0, b0)
    d.step(2)
    _check(d, o, n, precision)
    d.close()


@pytest.mark.parametrize("integrator", [0, 1])
def test_not_a_number_spreads_no_further(integrator):
    """A cell without a velocity (NaN momentum) makes the same cells and faces NaN
    in the mixed step as in FP64: its neighbours' slopes, which it has a part in,
    are zero, so their other faces stay numbers."""
    from kratos_b200 import Dynamics
    nb, n = (1, 1, 1), (130, 131, 70)
    u0, b0 = _state(nb, n, "subsonic", 5)
    u0[0, 30, 60, 61, 3] = np.nan
    bad = []
    for precision in (2, 1):
        d = Dynamics(True, nb, n, gamma=GAMMA, precision=precision, integrator=integrator)
        d.set_state(u0, b0)
        d.step(1)
        u, b = d.get_state()
        bad.append((np.isnan(u).any(-1), np.isnan(b[:, 2:-2, 2:-2, 2:-2])))
        d.close()
    assert 0 < bad[0][0].sum() < 200
    for k in range(2):
        assert np.array_equal(bad[0][k], bad[1][k]), (bad[0][k].sum(), bad[1][k].sum())
