"""Launches of small grids (chained, with one shared-memory split) against those
of large ones: an instance alone, below the line of three tiles per SM, and the
same instance in a batch above it run the same arithmetic, so the results are
equal to the bit, also when calls follow one another without a pause."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# tiles of one instance: at most 456 (three per SM of 152); of three instances: more
@pytest.mark.parametrize("p,nx,ny", [(1, 77, 76), (2, 73, 75), (3, 84, 84), (4, 38, 80)])
@pytest.mark.parametrize("solver,n_iter", [("chebyshev", 5), ("pcg", 6)])
def test_small_grid_equals_its_part_of_a_large_one(igr, p, nx, ny, solver, n_iter):
    torch = pytest.importorskip("torch")
    host = lambda a: a.cpu().numpy() if isinstance(a, torch.Tensor) else np.asarray(a)
    basis = igr.DGBasis(p)
    mesh = igr.CartesianMesh2D(nx, ny, 1.0, 1.0, basis)
    x, y = (np.asarray(a).reshape(-1, order="F") for a in (mesh.x, mesh.y))
    q = []
    for k in range(3):
        rho = 1.0 + 0.2 * np.sin(2 * np.pi * (x + 0.1 * k)) * np.cos(2 * np.pi * y)
        u, v = 0.3 * np.sin(2 * np.pi * y), 0.2 * np.cos(2 * np.pi * (x + y))
        q.append(np.stack([rho * u, rho * v, rho, 2.5 + 0.5 * rho * (u * u + v * v)]))
    q0 = torch.from_numpy(np.stack(q)).cuda()
    g, al, dt = np.full(3, 1.4), np.full(3, 1e-4), np.full(3, 1e-4)
    kw = dict(objective="l2_pressure", device_arrays=True, n_iter=n_iter, solver=solver)
    whole = igr.adjoint_batch(q0, g, al, dt, 2, basis, mesh, **kw)
    for k in range(3):
        one = igr.adjoint_batch(q0[k:k + 1].contiguous(), g[:1], al[:1], dt[:1], 2, basis, mesh, **kw)
        for a, b in zip(whole, one):
            assert np.array_equal(host(a)[k], host(b)[0])
