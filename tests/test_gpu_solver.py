"""One step from random states against the CPU restatement: the regions of the
Riemann fan that smooth workloads do not reach (supersonic faces on both sides,
vanishing and tiny normal fields, degenerate star states, strong jumps of
density and pressure) and block shapes whose sites do not fill whole warps or
whose planes are too large to share a row of CTAs.

FP64: relative L1 <= 1e-11 per field against the field's own scale, as the
fixtures' bound.  Mixed: 2e-5, FP32's 6e-8 through the fluxes of one step, times
the face-to-face cancellation of jumps up to 50 (the field flux of a face is
small beside the products it is the difference of).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GAMMA = 5 / 3
FLOWS = {
    # velocity scale, field scale, field along z, spread of log density and pressure
    "subsonic": (0.2, 0.7, 0.3, 0.3),
    "supersonic": (8.0, 0.5, 0.2, 0.5),
    "no_normal_field": (0.5, 0.6, 0.0, 0.5),        # none along z, transverse ones on its faces
    "no_field": (0.5, 0.0, 0.0, 0.5),
    "tiny_normal_field": (0.5, 0.6, 1e-4, 0.5),
    "strong_field": (0.5, 4.0, 2.0, 1.0),
}


def _state(nb, n, flow, seed):
    """Random cell states and face fields B_a that do not depend on a."""
    rng = np.random.default_rng(seed)
    vs, bs, bz, spread = FLOWS[flow]
    nblk = nb[0] * nb[1] * nb[2]
    shape = [nb[a] * n[a] for a in range(3)]
    g = (shape[2], shape[1], shape[0])
    rho, p = np.exp(spread * rng.normal(size=g)), np.exp(spread * rng.normal(size=g))
    v = [vs * rng.normal(size=g) for _ in range(3)]
    b = [np.broadcast_to(bs * rng.normal(size=(g[0], g[1], 1)), g),
         np.broadcast_to(bs * rng.normal(size=(g[0], 1, g[2])), g),
         np.broadcast_to(bz * (1 + 0.5 * rng.normal(size=(1, g[1], g[2]))), g)]
    e = p / (GAMMA - 1) + 0.5 * rho * sum(q * q for q in v) + 0.5 * sum(q * q for q in b)
    u = np.stack([rho, e] + [rho * q for q in v] + b, axis=-1)
    hu = np.empty((nblk, n[2], n[1], n[0], 8))
    hb = np.zeros((nblk, n[2] + 5, n[1] + 5, n[0] + 5, 3))
    for k in range(nblk):
        r = (k % nb[0], (k // nb[0]) % nb[1], k // (nb[0] * nb[1]))
        sl = [slice(r[a] * n[a], (r[a] + 1) * n[a]) for a in range(3)]
        hu[k] = u[sl[2], sl[1], sl[0]]
        idx = [(np.arange(n[a] + 1) + r[a] * n[a]) % shape[a] for a in range(3)]
        for a in range(3):
            hb[k, 2:n[2] + 3, 2:n[1] + 3, 2:n[0] + 3, a] = b[a][np.ix_(idx[2], idx[1], idx[0])]
    return hu, hb


@pytest.mark.parametrize("precision", [2, 1])
@pytest.mark.parametrize("flow", sorted(FLOWS))
@pytest.mark.parametrize("nb,n", [((2, 2, 2), (8, 8, 8)), ((1, 2, 1), (33, 5, 19)), ((1, 1, 1), (260, 252, 4))])
def test_one_step_from_random_states(nb, n, flow, precision):
    from kratos_b200 import Dynamics
    from oracle.kr_oracle import OracleMesh
    u0, b0 = _state(nb, n, flow, 7)
    o = OracleMesh(True, nb, n, GAMMA)
    o.set_state(u0, b0)
    o.step(1)
    uo, bo = o.get_state()
    d = Dynamics(True, nb, n, gamma=GAMMA, precision=precision)
    d.set_state(u0, b0)
    d.step(1)
    u, b = d.get_state()
    assert d.status() == 0
    tol = 1e-11 if precision == 2 else 2e-5
    for k in range(5):
        scale = np.abs(uo[..., 2:5]).max(-1).sum() if k >= 2 else np.abs(uo[..., k]).sum()
        assert np.abs(u[..., k] - uo[..., k]).sum() <= tol * scale, "field %d" % k
    own = np.s_[:, 2:n[2] + 2, 2:n[1] + 2, 2:n[0] + 2]
    if flow == "no_field":
        assert not b[own].any() and not bo[own].any()
    else:
        assert np.abs(b[own] - bo[own]).sum() <= tol * np.abs(bo[own]).sum()
    d.close()


@pytest.mark.parametrize("precision", [2, 1])
@pytest.mark.parametrize("kw", [{}, {"integrator": 1}])
@pytest.mark.parametrize("nb,n", [((1, 1, 1), (130, 131, 70)), ((10, 10, 10), (9, 12, 17)), ((2, 1, 2), (300, 9, 101))])
def test_marching_sweeps(nb, n, kw, precision):
    """Meshes large enough for the y and z sweeps to march (columns that end in
    partial warps, one and many blocks, short and long runs of faces)."""
    from kratos_b200 import Dynamics
    from oracle.kr_oracle import OracleMesh
    u0, b0 = _state(nb, n, "subsonic", 11)
    o = OracleMesh(True, nb, n, GAMMA, **kw)
    o.set_state(u0, b0)
    o.step(2)
    uo, bo = o.get_state()
    d = Dynamics(True, nb, n, gamma=GAMMA, precision=precision, **kw)
    d.set_state(u0, b0)
    d.step(2)
    u, b = d.get_state()
    assert d.status() == 0
    tol = 1e-11 if precision == 2 else 2e-5
    for k in range(5):
        scale = np.abs(uo[..., 2:5]).max(-1).sum() if k >= 2 else np.abs(uo[..., k]).sum()
        assert np.abs(u[..., k] - uo[..., k]).sum() <= tol * scale, "field %d" % k
    own = np.s_[:, 2:n[2] + 2, 2:n[1] + 2, 2:n[0] + 2]
    assert np.abs(b[own] - bo[own]).sum() <= tol * np.abs(bo[own]).sum()
    d.close()
