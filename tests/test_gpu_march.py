"""The marching y and z sweeps (meshes of at least a wave's worth of columns)
against the CPU restatement, and against the per-face sweeps that a smaller mesh
of the same blocks runs: solvers, integrators, physical sides, refined meshes and
the learned mode's stored choices.

FP64: relative L1 <= 1e-11 per field against the field's own scale, the fixtures'
bound.  Mixed: 2e-5, FP32's 6e-8 through the fluxes of a step times the
cancellation of the random states' jumps (test_gpu_solver.py).
"""
import numpy as np
import pytest

from test_gpu_solver import GAMMA, _state

pytestmark = pytest.mark.gpu


def _marches(n, axis, nblk):
    """The load from which the MHD sweep along `axis` marches (kr_march.cuh march_pays)."""
    import torch
    load = (n[0] + 2) * (n[3 - axis] + 2) / 32 * (n[axis] + 1) / 8 * nblk
    return load >= 32 * torch.cuda.get_device_properties(0).multi_processor_count


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


@pytest.mark.parametrize("precision", [2, 1])
@pytest.mark.parametrize("kinds", [("per", "per", "out", "fre", "fre", "out"), ("fre", "out", "per", "per", "out", "out")])
def test_beside_physical_sides(kinds, precision):
    from kratos_b200 import Dynamics
    from oracle.kr_oracle import OracleMesh
    nb, n = (2, 2, 2), (66, 61, 37)
    assert _marches(n, 1, 8) and _marches(n, 2, 8)
    u0, b0 = _state(nb, n, "subsonic", 9)
    o = OracleMesh(True, nb, n, GAMMA, kinds=kinds)
    o.set_state(u0, b0)
    o.step(2)
    d = Dynamics(True, nb, n, gamma=GAMMA, precision=precision, kinds=kinds)
    d.set_state(u0, b0)
    d.step(2)
    _check(d, o, n, precision)
    d.close()


@pytest.mark.parametrize("precision", [2, 1])
def test_refined_mesh(precision):
    """The refined z march: three levels, jumps across every axis, so that columns
    run beside sides whose neighbours are on another level (the ghost line's
    normal B out of the ring).  FP64: the larger of 1e-11 and ten times the
    restatement's own spread between builds with and without fused multiply-adds
    (test_gpu_smr_mhd.py); mixed as above."""
    from kratos_b200 import Dynamics
    from oracle.kr_oracle import OracleMesh
    import golden_io as G
    nb, n = (4, 4, 4), (18, 14, 16)
    regions = [(1, (0.0, 0.0, 0.0), (0.49, 1.0, 1.0)), (2, (0.2, 0.4, 0.4), (0.24, 0.45, 0.45))]
    ref = []
    for variant in ("", "fma"):
        o = OracleMesh(True, nb, n, GAMMA, regions=regions, variant=variant)
        o.init_problem("ot", 3)
        o.step(2)
        ref.append(o.get_state())
    d = Dynamics(True, nb, n, gamma=GAMMA, precision=precision, regions=regions)
    assert _marches(n, 2, d.nblk) and set(d.level) == {0, 1, 2}
    d.init_problem("ot", 3)
    d.step(2)
    u, b = d.get_state()
    assert d.status() == 0
    tol = 1e-11 if precision == 2 else 2e-5
    for k, (e, spread) in enumerate(zip(G.field_errors(u, ref[0][0]), G.field_errors(ref[1][0], ref[0][0]))):
        assert e <= max(tol, 10 * spread), "field %d" % k
    own = np.s_[:, 2:n[2] + 2, 2:n[1] + 2, 2:n[0] + 2]
    den = np.abs(ref[0][1][own]).sum()
    assert np.abs(b[own] - ref[0][1][own]).sum() <= max(tol, 10 * np.abs(ref[1][1][own] - ref[0][1][own]).sum() / den) * den
    d.close()


@pytest.mark.parametrize("kw", [dict(precision=2), dict(precision=1), dict(precision=2, riemann=1), dict(precision=1, riemann=1),
                                dict(precision=1, integrator=1), dict(precision=1, riemann=2, sel_period=4)])
def test_copies_of_a_block_step_as_the_block(kw):
    """A periodic block too small to march, and a mesh of 80 copies of it, which
    marches: every copy steps as the block does, to the rounding of the same
    operations in two kernels (1e-12 in FP64, 1e-6 in mixed precision, as batched
    launches against per-size ones).  In learned mode both take the choices of one
    evaluation at step 0, per face HLLE or HLLD, so a choice read for another face
    would show as the two fluxes' difference."""
    from kratos_b200 import Dynamics
    from kratos_b200 import selector as S
    n, nb = (34, 21, 18), (5, 4, 4)
    count = nb[0] * nb[1] * nb[2]
    assert _marches(n, 1, count) and _marches(n, 2, count) and not _marches(n, 1, 1) and not _marches(n, 2, 1)
    u0, b0 = _state((1, 1, 1), n, "subsonic", 21)
    small = Dynamics(True, (1, 1, 1), n, gamma=GAMMA, x_max=tuple(k / 16 for k in n), **kw)
    large = Dynamics(True, nb, n, gamma=GAMMA, x_max=tuple(k * m / 16 for k, m in zip(n, nb)), **kw)
    small.set_state(u0, b0)
    large.set_state(np.repeat(u0, count, axis=0), np.repeat(b0, count, axis=0))
    if kw.get("riemann") == 2:
        for d in (small, large):
            d.set_selector(S.init_params(5), 0.0)
    for d in (small, large):
        d.step(3)
        assert d.status() == 0
    if kw.get("riemann") == 2:
        (f0, c0), (f1, c1) = small.selector_stats(), large.selector_stats()
        assert f1 == count * f0 and c1 == count * c0 and 0.05 < c0 / f0 < 0.95, c0 / f0
    (u, b), (us, bs) = large.get_state(), small.get_state()
    tol = 1e-12 if kw["precision"] == 2 else 1e-6
    assert np.abs(u - us).sum() <= tol * count * np.abs(us).sum()
    own = np.s_[:, 2:n[2] + 2, 2:n[1] + 2, 2:n[0] + 2]
    assert np.abs(b[own] - bs[own]).sum() <= tol * count * np.abs(bs[own]).sum()
    small.close()
    large.close()
