"""The operator is odd to the bit, A(-x) = -A(x), as the FP64 contractions were:
the integer sums round symmetrically about zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_negated_operand_gives_the_negated_result(igr, p):
    basis = igr.DGBasis(p)
    mesh = igr.CartesianMesh2D(23, 17, 1.0, 0.7, basis)
    rng = np.random.default_rng(p)
    x = np.asfortranarray(rng.standard_normal(mesh.x.shape) * 2.0 ** rng.integers(-6, 6, mesh.x.shape))
    rho = np.asfortranarray(1.0 + rng.random(mesh.x.shape))
    y, z = np.zeros_like(x), np.zeros_like(x)
    igr.apply_sip_(y, x, rho, basis, mesh, 3e-3)
    igr.apply_sip_(z, np.asfortranarray(-x), rho, basis, mesh, 3e-3)
    assert np.array_equal(y, -z)
