"""Whole operators, right-hand sides and gradients against long double: the
oracle's templates on the same double inputs, basis and constants
(tests/long_double.cpp), beside the FP64 oracle's own error.

Bounds. Operators and right-hand sides are sums of the same terms in another
order and with fewer roundings: at most twice the FP64 oracle's error. For P4
the kernels leave out D's interior diagonal, up to 1e-15 where a rounding is
1.1e-16: ten times. J and the parameter derivatives are sums over the mesh and
the steps with a cancellation of up to 1e6, which the oracle forms one after
the other: at most its error, in rms over four states. A mean error of a
fraction of a unit of the integer sums would add up there and show as several
times the oracle's."""
import ctypes as C
import os
import subprocess
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
GAMMA = 1.4
NDIR = 2


def ptr(a):
    assert a.dtype == np.float64 and a.flags["C_CONTIGUOUS"]
    return a.ctypes.data_as(C.POINTER(C.c_double))


def flat(a):
    return np.ascontiguousarray(np.asarray(a).reshape(-1, order="F"))


@pytest.fixture(scope="module")
def wide(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("ld") / "liblong_double.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-DDIRECTIONS=%d" % NDIR, "-o", out,
                    os.path.join(HERE, "long_double.cpp")], check=True, stderr=subprocess.DEVNULL)
    return C.CDLL(out)


def state(G, seed):
    """Pulses on a smooth moving gas with jumps between the elements; (q, dt, alpha)."""
    rng = np.random.default_rng(seed)
    x, y = G.coords()
    tx, ty = 2 * np.pi * x / G.Lx, 2 * np.pi * y / G.Ly
    jump = lambda: 1 + 0.01 * np.repeat(rng.uniform(-1, 1, G.N // G.np ** 2), G.np ** 2)  # noqa: E731
    rho = (1 + 0.15 * np.sin(tx + 2 * ty + rng.uniform(0, 6)) + 0.1 * np.sin(2 * tx - ty + rng.uniform(0, 6))) * jump()
    u = 0.3 * np.sin(tx + rng.uniform(0, 6)) * np.cos(ty + rng.uniform(0, 6)) * jump()
    v = 0.3 * np.cos(ty + rng.uniform(0, 6)) * np.sin(2 * tx + rng.uniform(0, 6)) * jump()
    P = np.full_like(x, 0.5)
    for _ in range(3):
        A, cx, cy = rng.uniform(1, 5), rng.uniform(0.2, 0.8), rng.uniform(0.2, 0.8) * G.Ly
        P = P + A * np.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * G.dx) ** 2)
    P = P * jump()
    q = np.stack([rho * u, rho * v, rho, P / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)])
    speed = max(np.max(np.abs(w) + np.sqrt(GAMMA * P / rho)) for w in (u, v))
    h = min(G.dx, G.dy)
    return q, 0.1 * h / ((2 * G.p + 1) * speed), 3 * h * h


CASES = [(1, 12, 10, "chebyshev", 5, 3), (2, 11, 12, "jacobi", 10, 3), (3, 12, 10, "chebyshev", 5, 3), (3, 12, 12, "pcg", 20, 2),
         (4, 9, 8, "pcg", 12, 2)]


@pytest.mark.parametrize("p,nx,ny,solver,n_iter,n_steps", CASES)
def test_errors_against_long_double(igr, oracle, wide, p, nx, ny, solver, n_iter, n_steps):
    basis = igr.DGBasis(p)
    mesh = igr.CartesianMesh2D(nx, ny, 1.0, ny / nx, basis)
    G = oracle.Grid2D(p, nx, ny, 1.0, ny / nx)
    N, sid = G.N, oracle.SOLVERS[solver]
    states = [state(G, 40 + s) for s in range(4)]
    prm, none = np.zeros(4), np.zeros((NDIR, 4, N))

    def exact(s):
        q, dt, alpha = s
        r = np.zeros((NDIR + 3, 2))
        wide.ld_gradient(*G.args(), C.c_double(GAMMA), C.c_double(alpha), C.c_int(n_steps), C.c_double(dt), C.c_int(n_iter),
                         C.c_int(sid), C.c_int(oracle.OBJECTIVES_2D["l2_pressure"]), ptr(prm), ptr(q), ptr(none), ptr(r))
        return r

    with ThreadPoolExecutor(4) as ex:
        refs = list(ex.map(exact, states))
    operators, sums = [], []
    for (q, dt, alpha), ref in zip(states, refs):
        f = [np.asfortranarray(a.reshape(mesh.x.shape, order="F")) for a in q]
        y, S = np.zeros_like(f[0]), np.zeros_like(f[0])
        dq = [np.zeros_like(f[0]) for _ in range(4)]
        igr.apply_sip_(y, f[3], f[2], basis, mesh, alpha)
        igr.compute_igr_euler_rhs_(*dq, *f, S, basis, mesh, GAMMA, alpha, n_iter=n_iter, solver=solver)
        dq64, S64 = oracle.igr_euler_rhs_2d(G, GAMMA, alpha, n_iter, solver, list(q), np.zeros(N))
        e = np.zeros((2, 6))
        one = np.zeros(2)
        cand = np.stack([flat(y), oracle.apply_sip_2d(G, alpha, q[3], q[2])])
        wide.ld_apply(*G.args(), C.c_double(alpha), ptr(q[3]), ptr(q[2]), C.c_int(2), ptr(cand), ptr(one))
        cand = np.stack([np.stack([flat(a) for a in (S, *dq)]), np.stack([S64, *dq64])])
        five = np.zeros((2, 5))
        wide.ld_rhs(*G.args(), C.c_double(GAMMA), C.c_double(alpha), C.c_int(n_iter), C.c_int(sid), ptr(q), ptr(np.zeros(N)),
                    C.c_int(2), ptr(cand), ptr(five))
        e[:, 0], e[:, 1:] = one, five
        operators.append(e)
        J, *_, dg, da = igr.enzyme_adjoint_ic(*f, n_steps, dt, basis, mesh, GAMMA, alpha, n_iter=n_iter, solver=solver,
                                              objective="l2_pressure", with_params=True)
        J64, _, dg64, da64 = oracle.adjoint_2d(G, GAMMA, alpha, n_steps, dt, n_iter, solver, "l2_pressure", list(q))
        r = ref[:3]
        off = lambda v: [(x - hi) - lo for x, (hi, lo) in zip(v, r)]  # noqa: E731
        sums.append([off((J, dg, da)), off((J64, dg64, da64))])
    operators, sums = (np.sqrt(np.mean(np.square(a), axis=0)) for a in (operators, sums))
    print("operators", operators, "sums", sums)
    assert np.all(operators[0] <= (10 if p == 4 else 2) * operators[1])
    assert np.all(sums[0] <= sums[1])
