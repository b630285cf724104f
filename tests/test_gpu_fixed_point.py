"""GPU side of the fixed-point line contractions, through the operator calls:
operands at the ends of the integer path's range and beyond it (where the FP64
chain runs), against the oracle. One operator application is held to the
operator bar, 1e-13 relative L2."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL_OP = 1e-13


def flat(a):
    return np.ascontiguousarray(np.asarray(a).reshape(-1, order="F"))


def rel(a, b, scale):
    a, b = flat(a) / scale, flat(b) / scale
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# 2^-890, 2^1000: the first and last decades of the integer path (its operator coefficients are O(1e-3 .. 1e2));
# 2^-1000, 2^1012: FP64 lines; 0: lines of zeros beside lines of data
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("power", [-1000, -890, 0, 1000, 1012])
@pytest.mark.parametrize("holes", [False, True])
def test_apply_sip_over_the_exponent_range(igr, oracle, p, power, holes):
    basis = igr.DGBasis(p)
    mesh = igr.CartesianMesh2D(5, 3, 1.0, 0.7, basis)
    G = oracle.Grid2D(p, 5, 3, 1.0, 0.7)
    rng = np.random.default_rng(100 + p)
    x = rng.standard_normal(mesh.x.shape)
    if holes:
        x[rng.random(x.shape) < 0.4] = 0.0
        x[:, 0, 1, 1] = 0.0
        x[:, :, 3, 2] = 0.0
    rho = 1.0 + 0.5 * rng.random(mesh.x.shape)
    s = 2.0 ** power
    y = np.zeros(mesh.x.shape, order="F")
    igr.apply_sip_(y, np.asfortranarray(x * s), np.asfortranarray(rho), basis, mesh, 3e-3)
    # power-of-two scaling commutes with the operator: the reference is taken at scale 1
    ref = oracle.apply_sip_2d(G, 3e-3, flat(x), flat(rho))
    assert rel(y, ref * s, s) <= RTOL_OP


@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_nonfinite_operand_stays_in_its_neighbourhood(igr, oracle, p, value):
    basis = igr.DGBasis(p)
    mesh = igr.CartesianMesh2D(6, 6, 1.0, 1.0, basis)
    rng = np.random.default_rng(7)
    x, rho = rng.standard_normal(mesh.x.shape), 1.0 + 0.5 * rng.random(mesh.x.shape)
    x[0, 0, 2, 3] = value
    y = np.zeros(mesh.x.shape, order="F")
    igr.apply_sip_(y, np.asfortranarray(x), np.asfortranarray(rho), basis, mesh, 3e-3)
    ref = oracle.apply_sip_2d(oracle.Grid2D(p, 6, 6, 1.0, 1.0), 3e-3, flat(x), flat(rho))
    got, ref = flat(y), flat(ref)
    bad = ~np.isfinite(ref)
    # the oracle multiplies by D's zero interior diagonal too (0 * inf = NaN): its non-finite set may be larger
    assert not np.any(~np.isfinite(got) & ~bad)
    assert np.count_nonzero(~np.isfinite(got)) > 0
    fine = ~bad
    assert np.linalg.norm(got[fine] - ref[fine]) <= RTOL_OP * np.linalg.norm(ref[fine])


# the hyperbolic right-hand side is homogeneous of degree one in (state, Sigma), so powers of two scale it; a gas at rest
# reaches the ends of the exponent range without squares of the momentum leaving it (1 / rho and the sound speed there
# take the IEEE operations)
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("power,moving", [(0, True), (-400, True), (400, True), (-890, False), (990, False), (-1000, False)])
def test_hyperbolic_rhs_over_the_exponent_range(igr, oracle, p, power, moving):
    basis = igr.DGBasis(p)
    mesh = igr.CartesianMesh2D(5, 3, 1.0, 0.7, basis)
    G = oracle.Grid2D(p, 5, 3, 1.0, 0.7)
    rng = np.random.default_rng(200 + p)
    sh = mesh.x.shape
    rho = 1.0 + 0.4 * rng.random(sh)
    mux, muy = [0.3 * rng.standard_normal(sh) if moving else np.zeros(sh) for _ in range(2)]
    E = 2.0 + rng.random(sh) + 0.5 * (mux ** 2 + muy ** 2) / rho
    S = 0.05 * rng.standard_normal(sh)
    s = 2.0 ** power
    out = [np.zeros(sh, order="F") for _ in range(4)]
    igr.compute_hyperbolic_rhs_(*out, *[np.asfortranarray(a * s) for a in (mux, muy, rho, E, S)], basis, mesh, 1.4)
    ref = oracle.hyperbolic_rhs_2d(G, 1.4, [flat(a) for a in (mux, muy, rho, E)], flat(S))
    for a, b in zip(out, ref):
        assert rel(a, flat(b) * s, s) <= RTOL_OP
