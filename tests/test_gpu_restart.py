"""A march restarted from a snapshot carries on to the bit: 1/rho of a stored
state, formed anew at the restart, is the one that the running march holds.
A rounding that differs in one node of a million shows here only over many
node values, so the mesh is large (12 restarts of 409,600 nodes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def big_case(igr):
    basis = igr.DGBasis(3)
    mesh = igr.CartesianMesh2D(160, 160, 1.0, 1.0, basis)
    x, y = np.asarray(mesh.x), np.asarray(mesh.y)
    rho = 1.0 + 0.3 * np.sin(2 * np.pi * x) * np.cos(4 * np.pi * y) + 0.05 * np.sin(14 * np.pi * (x + y))
    u, v = 0.4 * np.sin(2 * np.pi * y), 0.3 * np.cos(2 * np.pi * (x - y))
    q0 = [np.asfortranarray(a) for a in (rho * u, rho * v, rho, 2.5 + 0.5 * rho * (u * u + v * v))]
    return basis, mesh, q0


@pytest.mark.parametrize("alpha", [0.0, 1e-5])
def test_restarts_from_snapshots_are_bitwise(igr, alpha):
    basis, mesh, q0 = big_case(igr)
    n, dt = 12, 1e-4
    T = dt * (n - 0.5)
    kw = dict(n_iter=3, solver="chebyshev")
    ctx = igr.default_context()
    whole, ns = igr.run_forward_store(*q0, dt, T, basis, mesh, 1.4, alpha, **kw)
    assert ns == n
    grad = igr.adjoint_conservative_ic(*q0, dt, T, basis, mesh, 1.4, alpha, **kw)
    assert ctx.last_adjoint_plan()["segments"] == 1
    ctx.set_tape_budget(8 * 5 * mesh.x.size * 11)  # room for 11 of the 13 snapshots
    try:
        steps, _ = igr.run_forward_store(*q0, dt, T, basis, mesh, 1.4, alpha, **kw)  # restarts after every step
        seg = igr.adjoint_conservative_ic(*q0, dt, T, basis, mesh, 1.4, alpha, **kw)
        assert ctx.last_adjoint_plan()["segments"] > 1
    finally:
        ctx.set_tape_budget(0)
    assert np.array_equal(steps.data, whole.data)
    for a, b in zip(seg, grad):
        assert np.array_equal(a, b)
