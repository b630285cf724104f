"""Performance cases: what programs that use this package have it do.

A case is one call of a public entry point with its sizes and options. The
kinds cover both packages (2D and 1D) and every direction of the path:

  apply       apply_sip_                 one operator application (the smallest call)
  rhs         compute_igr_euler_rhs_     one right-hand side with its Sigma solve
  forward     run_forward                a forward trajectory
  gradient    enzyme_adjoint_ic          objective and its gradient by the discrete adjoint, one instance
  batch       adjoint_batch              the same for a batch; 2D: device arrays, 1D: mixed element counts
  tangent     sensitivity_batch / run_sensitivity   state and tangent together
  continuous  adjoint_conservative_batch forward store and backward adjoint PDE

All arithmetic is FP64, the only type that the entry points take. The host
arrays of the entry points are part of the call. States are Gaussian pressure
pulses (the benchmark's family, p_bg + sum A exp(-r^2/w^2)) on a smooth flow of
varying density and velocity, as a running simulation has them.

`exact` evaluates the same discretisation with torch in 64 bits (gradients by
autograd) for every kind but the tangent and the continuous adjoint, whose
reference equations are long; those are compared with earlier results alone.
"""
import math

import numpy as np
import torch

import igr_sensitivities_gb300 as igr
from igr_sensitivities_gb300 import igr1d

GAMMA = 1.4
CFL = 0.1


def listed():
    return [
        # one operator application on a small mesh: what a host-side solver or a unit study calls again and again
        dict(name="apply 2D 8x8 P3", kind="apply", dim=2, p=3, nx=8, ny=8, solver="pcg", iters=0, steps=0, batch=1),
        # one right-hand side on an odd mesh at another degree, the call of a host-side time integrator
        dict(name="rhs 2D 37x29 P2 jacobi", kind="rhs", dim=2, p=2, nx=37, ny=29, solver="jacobi", iters=20, steps=0,
             batch=1),
        # a P4 resolution of the blast refinement study (22 x 22, PCG 60): ragged against every tile
        dict(name="forward 2D 22x22 P4 pcg", kind="forward", dim=2, p=4, nx=22, ny=22, solver="pcg", iters=60, steps=10,
             batch=1),
        # the single forward of the 64 x 64 Chebyshev configuration
        dict(name="forward 2D 64x64 P3 cheb", kind="forward", dim=2, p=3, nx=64, ny=64, solver="chebyshev", iters=5,
             steps=40, batch=1),
        # the 128 x 128 PCG-60 forward configuration
        dict(name="forward 2D 128x128 P3 pcg", kind="forward", dim=2, p=3, nx=128, ny=128, solver="pcg", iters=60,
             steps=12, batch=1),
        # one 64 x 64 gradient, as an optimiser over initial conditions asks for
        dict(name="gradient 2D 64x64 P3 cheb", kind="gradient", dim=2, p=3, nx=64, ny=64, solver="chebyshev", iters=5,
             steps=30, batch=1),
        # the headline workload with fewer instances and steps: batched 128 x 128 gradients, device arrays
        dict(name="batch 2D 8x128x128 P3 cheb", kind="batch", dim=2, p=3, nx=128, ny=128, solver="chebyshev", iters=5,
             steps=8, batch=8),
        # batched tangents of the 256 x 256 PCG-60 parameter study
        dict(name="tangent 2D 2x256x256 P3 pcg", kind="tangent", dim=2, p=3, nx=256, ny=256, solver="pcg", iters=60,
             steps=1, batch=2),
        # batched continuous adjoints at the headline's mesh
        dict(name="continuous 2D 8x128x128 P3 cheb", kind="continuous", dim=2, p=3, nx=128, ny=128, solver="chebyshev",
             iters=5, steps=6, batch=8),
        # the 1D single-instance forward (N_e = 256, Jacobi 50)
        dict(name="forward 1D 256 P3 jacobi", kind="forward", dim=1, p=3, nx=256, ny=1, solver="jacobi", iters=50,
             steps=150, batch=1),
        # the 1D batch of gradients with N_e in 64..1024, PCG 102
        dict(name="batch 1D 256x64..1024 P3 pcg", kind="batch", dim=1, p=3, nx=1024, ny=1, solver="pcg", iters=102,
             steps=2, batch=256),
    ]


# A drawn case asks for no more than this much arithmetic in one pass (the
# model of work(); the 256 x 256 tangent and the 1D batch lie near it).
_MOST_FLOPS_2D, _MOST_FLOPS_1D = 2.5e10, 4.0e9
_MOST_SERIAL = 1500  # dependent solver iterations, what a small mesh's time goes by


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "rhs", "forward", "forward", "gradient", "gradient", "batch", "batch", "tangent",
                       "continuous"])
    dim = rng.choice([2, 2, 2, 1])
    p = rng.choice([1, 2, 3, 3, 3, 4])
    solver = rng.choice(["pcg", "chebyshev", "chebyshev", "jacobi"])
    iters = {"pcg": rng.choice([10, 30, 60]), "chebyshev": 5, "jacobi": rng.choice([10, 20, 50])}[solver]
    if kind == "apply":
        iters = 0
    batch = 1
    if dim == 2:
        nx = _log_int(rng, 4, 160)
        ny = nx if rng.random() < 0.4 else max(4, min(160, int(nx * rng.uniform(0.5, 2.0))))
        if kind in ("batch", "tangent", "continuous"):
            batch = _log_int(rng, 2, 16)
    else:
        nx, ny = _log_int(rng, 16, 2048), 1
        if kind in ("batch", "continuous"):
            batch = _log_int(rng, 2, 256)
    steps = 0 if kind in ("apply", "rhs") else _log_int(rng, 2, 40)
    case = dict(kind=kind, dim=dim, p=p, nx=nx, ny=ny, solver=solver, iters=iters, steps=steps, batch=batch)
    most = _MOST_FLOPS_2D if dim == 2 else _MOST_FLOPS_1D
    if dim == 1 and batch == 1:  # one instance is one cluster's work, and a thread's serial chain
        most = 4.0e8
    serial = (iters + 4) * {"forward": 1, "apply": 1, "rhs": 1}.get(kind, 3)
    case["steps"] = min(case["steps"], max(1, _MOST_SERIAL // serial))
    while case["steps"] > 1 and work(case)["flops"] > most:
        case["steps"] -= 1
    while case["batch"] > 2 and work(case)["flops"] > most:
        case["batch"] -= 1
    while case["nx"] > 8 and work(case)["flops"] > most:
        case["nx"] -= 1
    return case


def _element_counts(case):
    """Elements per instance; a 1D batch mixes nx, nx/2, .. nx/16 (at least 4)."""
    if case["dim"] == 2:
        return [case["nx"] * case["ny"]] * case["batch"]
    if case["kind"] in ("batch", "continuous"):
        return [max(4, case["nx"] >> (b * 7 % 5)) for b in range(case["batch"])]
    return [case["nx"]] * case["batch"]


def work(case):
    """Compulsory traffic (inputs read once, outputs written once) and the
    arithmetic of the discretisation: contractions with the differentiation
    matrix (2 n_p flops per node, field and direction) and pointwise terms."""
    dim, n_p = case["dim"], case["p"] + 1
    nodes = sum(_element_counts(case)) * n_p ** dim
    fields = dim + 2
    c = 2 * n_p * dim
    apply = 2 * c + 4 * dim + 2
    if case["kind"] == "apply":
        return {"bytes": 8 * 3 * nodes, "flops": apply * nodes}
    step = {"pcg": apply + 12, "jacobi": apply + 3, "chebyshev": apply + 7}[case["solver"]]
    first = 0 if case["solver"] == "jacobi" else apply
    stage = dim * c + c + 16 + first + case["iters"] * step + fields * c + 24 * dim + 5 * fields
    if case["kind"] == "rhs":
        return {"bytes": 8 * (2 * fields + 2) * nodes, "flops": stage * nodes}
    forward = 3 * stage * case["steps"] * nodes
    times = {"forward": 1, "tangent": 2, "continuous": 2, "gradient": 3, "batch": 3}[case["kind"]]
    arrays = {"forward": 2 * fields + 1, "tangent": 4 * fields + 2, "continuous": 2 * fields, "gradient": 2 * fields,
              "batch": 2 * fields}[case["kind"]]
    return {"bytes": 8 * arrays * nodes, "flops": times * forward}


# ----------------------------------------------------------------------------- inputs
def _mesh(case, basis, n_e=None):
    if case["dim"] == 2:
        return igr.CartesianMesh2D(case["nx"], case["ny"], 1.0, case["ny"] / case["nx"], basis)
    return igr.PeriodicMesh1D(n_e or case["nx"], 1.0, basis)


def _alpha(mesh, dim):
    return 3.0 * (min(mesh.dx, mesh.dy) if dim == 2 else mesh.dx) ** 2


def _state(rng, dim, xy, lengths, gamma, h, nodes):
    """(momenta, rho, E) on the nodes xy (flat CUDA tensors, Julia node order): pulses on a smooth moving gas."""
    th = [2 * np.pi * x / ln for x, ln in zip(xy, lengths)]
    rho = torch.ones_like(xy[0])
    for k in range(2):
        rho = rho + rng.uniform(0.05, 0.15) * torch.sin(sum((k + 1 + d) * t for d, t in enumerate(th))
                                                        + rng.uniform(0, 2 * np.pi))
    u = []
    for d in range(dim):
        v = torch.zeros_like(xy[0])
        for k in range(2):
            m = rng.uniform(0.1, 0.4) * torch.sin((k + 1) * th[d] + rng.uniform(0, 2 * np.pi))
            v = v + (m * torch.cos(th[1 - d] + rng.uniform(0, 2 * np.pi)) if dim == 2 else m)
        u.append(v)
    p = torch.full_like(xy[0], 0.5)
    width = max(0.04, 2.0 * h)
    for _ in range(3):
        A, c = rng.uniform(1.0, 5.0), [rng.uniform(0.2, 0.8) * ln for ln in lengths]
        p = p + A * torch.exp(-sum((x - cc) ** 2 for x, cc in zip(xy, c)) / width ** 2)
    # the jumps between elements that a discontinuous solution has (a continuous one would put every face at a tie
    # of its max() of two sides, where rounding decides)
    jump = lambda: 1 + 0.01 * torch.from_numpy(rng.uniform(-1, 1, rho.numel() // nodes)).to(rho).repeat_interleave(nodes)
    rho, p, u = rho * jump(), p * jump(), [v * jump() for v in u]
    kin = 0.5 * rho * sum(v * v for v in u)
    q = [rho * v for v in u] + [rho, p / (gamma - 1) + kin]
    speed = max(float((v.abs() + torch.sqrt(gamma * p / rho)).max()) for v in u)
    return torch.stack(q), speed


def _dt(case, mesh, speed):
    h = min(mesh.dx, mesh.dy) if case["dim"] == 2 else mesh.dx
    return CFL * h / ((2 * case["p"] + 1) * speed)


def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    dev = torch.device("cuda")
    dim = case["dim"]
    basis = igr.DGBasis(case["p"])
    counts = _element_counts(case)
    st = {"case": case, "basis": basis, "ctx": igr.default_context()}
    gammas, alphas, dts, states, meshes = [], [], [], [], {}
    for b in range(case["batch"]):
        n_e = counts[b] if dim == 1 else 0
        if n_e not in meshes:
            m = _mesh(case, basis, n_e)
            xy = [torch.from_numpy(np.ascontiguousarray(a.reshape(-1, order="F"))).to(dev)
                  for a in ((m.x, m.y) if dim == 2 else (m.x,))]
            meshes[n_e] = (m, xy)
        m, xy = meshes[n_e]
        g = GAMMA if case["batch"] == 1 else float(rng.uniform(1.3, 1.7))
        q, speed = _state(rng, dim, xy, (m.Lx, m.Ly) if dim == 2 else (m.L,), g, m.dx,
                          basis.n_p ** dim)
        gammas.append(g)
        alphas.append(_alpha(m, dim))
        dts.append(_dt(case, m, speed))
        states.append(q)
    st["mesh"] = meshes[counts[0] if dim == 1 else 0][0]
    if case["kind"] == "continuous":  # one number of steps for the whole batch
        dts = [min(dts)] * len(dts)
    st.update(gammas=np.array(gammas), alphas=np.array(alphas), dts=np.array(dts))
    st["T"] = (max(case["steps"], 1) - 0.5) * dts[0]
    if dim == 1 and case["kind"] in ("batch", "continuous"):
        st["n_e"] = np.array(counts, dtype=np.int32)
        st["states"] = [tuple(np.ascontiguousarray(v) for v in q.cpu().numpy()) for q in states]
    elif case["kind"] == "batch":
        st["q0"] = torch.stack(states).contiguous()  # the entry point takes device tensors
    elif case["kind"] in ("tangent", "continuous") and dim == 2:
        st["q0"] = np.ascontiguousarray(torch.stack(states).cpu().numpy())
    else:
        shape = st["mesh"].x.shape
        st["q"] = [np.asfortranarray(v.reshape(shape, order="F")) for v in states[0].cpu().numpy()]
    if case["kind"] == "tangent":  # a smooth direction of the initial state
        s = np.random.default_rng([seed, 78])
        if dim == 2:
            st["s0"] = np.ascontiguousarray(st["q0"] * s.uniform(0.1, 1.0, (case["batch"], 4, 1)))
        else:
            st["s"] = [v * float(s.uniform(0.1, 1.0)) for v in st["q"]]
    if case["kind"] == "apply":
        st["y"] = np.zeros(st["mesh"].x.shape, order="F")
    if case["kind"] == "rhs":
        st["dq"] = [np.zeros(st["mesh"].x.shape, order="F") for _ in range(dim + 2)]
    return st


# ----------------------------------------------------------------------------- one pass
def run(st):
    c = st["case"]
    M = igr if c["dim"] == 2 else igr1d
    basis, mesh, ctx = st["basis"], st["mesh"], st["ctx"]
    g, al, dt = float(st["gammas"][0]), float(st["alphas"][0]), float(st["dts"][0])
    kw = dict(n_iter=c["iters"], solver=c["solver"], ctx=ctx)
    kind = c["kind"]
    if kind == "apply":  # the energy as the operand
        M.apply_sip_(st["y"], st["q"][-1], st["q"][-2], basis, mesh, al, ctx=ctx)
        return st["y"]
    if kind == "rhs":
        S = np.zeros_like(st["q"][0])
        M.compute_igr_euler_rhs_(*st["dq"], *st["q"], S, basis, mesh, g, al, **kw)
        return [*st["dq"], S]
    if kind == "forward":
        return list(M.run_forward(*st["q"], dt, st["T"], basis, mesh, g, al, **kw))
    if c["dim"] == 2:
        if kind == "gradient":
            return list(igr.enzyme_adjoint_ic(*st["q"], c["steps"], dt, basis, mesh, g, al, objective="l2_pressure",
                                              with_params=True, **kw))
        if kind == "batch":
            return list(igr.adjoint_batch(st["q0"], st["gammas"], st["alphas"], st["dts"], c["steps"], basis, mesh,
                                          objective="l2_pressure", device_arrays=True, **kw))
        if kind == "tangent":
            return list(igr.sensitivity_batch(st["q0"], st["s0"], st["gammas"], st["alphas"], st["dts"], c["steps"], basis,
                                              mesh, s_gamma=1.0, **kw))
        return igr.adjoint_conservative_batch(st["q0"], st["gammas"], st["alphas"], st["dts"], st["T"], basis, mesh,
                                              objective="l2_density", **kw)
    if kind == "tangent":
        return list(igr1d.run_sensitivity(*st["q"], *st["s"], dt, st["T"], basis, mesh, g, al, s_gamma=1.0, **kw))
    if kind == "continuous":
        out = igr1d.adjoint_conservative_batch(st["states"], basis, st["n_e"], 1.0, st["gammas"], st["alphas"], st["dts"],
                                               st["T"], objective="l2_density", **kw)
        return np.concatenate([np.concatenate([np.ravel(v, order="F") for v in a]) for a in out])
    if kind == "gradient":
        J, dq, dg, da = igr1d.adjoint_batch([tuple(st["q"])], basis, [mesh.N_e], mesh.L, g, al, dt, c["steps"],
                                            objective="l2_pressure", **kw)
        return [J, *dq[0], dg, da]
    J, dq, dg, da = igr1d.adjoint_batch(st["states"], basis, st["n_e"], 1.0, st["gammas"], st["alphas"], st["dts"],
                                        c["steps"], objective="l2_pressure", **kw)
    return [J, np.concatenate([np.concatenate(a) for a in dq]), dg, da]


# ----------------------------------------------------------------------------- the same in torch
class _Torch:
    """The discretisation on B instances of one mesh: fields are (B, [N_ey,] N_ex, [n_p,] n_p), the x-node last."""

    def __init__(self, dim, basis, mesh, gamma, alpha):
        f = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")
        self.dim, self.n_p, self.p = dim, basis.n_p, basis.p
        self.D, self.w = f(basis.D), f(basis.w)
        self.h = [mesh.dx, mesh.dy] if dim == 2 else [mesh.dx]
        self.J = [x / 2 for x in self.h]
        self.g, self.a = gamma, alpha  # (B, 1, ..) tensors
        w = [self.w * j for j in self.J]
        self.W = w[0] if dim == 1 else w[1][:, None] * w[0][None, :]
        # quadrature weights along a face of direction d
        self.Wf = [torch.ones(1, dtype=torch.float64, device="cuda")] if dim == 1 else [w[1], w[0]]

    def der(self, d, v):  # sum_k D[i, k] v[k] along the nodes of direction d
        return v @ self.D.T if d == 0 else self.D @ v

    def der_t(self, d, v):
        return v @ self.D if d == 0 else self.D.T @ v

    def end(self, d, v, last):
        i = self.n_p - 1 if last else 0
        return v[..., i] if d == 0 else v[..., i, :]

    def at_ends(self, d, lo, hi):  # a field that is zero but at the end nodes of direction d
        z = torch.zeros_like(lo)
        return torch.stack([lo] + [z] * (self.n_p - 2) + [hi], dim=-1 if d == 0 else -2)

    def roll(self, d, v, by):  # face fields have one node axis fewer
        return torch.roll(v, by, dims=(-2 if d == 0 else -3) if self.dim == 2 else -1)

    def right(self, d, v):  # the first node of the next element
        return self.roll(d, self.end(d, v, False), -1)

    @staticmethod
    def larger(a, b):
        return torch.where(a >= b, a, b)

    def face(self, x):  # instance scalars against face fields
        return x[..., 0]

    def penalty(self, d, ir):
        return (self.p + 1) ** 2 * self.larger(self.end(d, ir, True), self.right(d, ir)) / self.h[d]

    def sip(self, x, ir):
        y = self.W * x * ir
        af = self.face(self.a)
        for d in range(self.dim):
            ij = 1 / self.J[d]
            gd = self.der(d, x)
            c = self.a * self.W * (ij * ij) * ir * gd
            jump = self.end(d, x, True) - self.right(d, x)
            irL, irR = self.end(d, ir, True), self.right(d, ir)
            avg = ij * (irL * self.end(d, gd, True) + irR * self.right(d, gd)) / 2
            F = af * self.Wf[d] * (self.penalty(d, ir) * jump - avg)
            s = -0.5 * ij * af * self.Wf[d] * jump
            c = c + self.at_ends(d, self.roll(d, s * irR, 1), s * irL)
            y = y + self.der_t(d, c) + self.at_ends(d, -self.roll(d, F, 1), F)
        return y

    def diagonal(self, ir):
        m = self.W * ir
        af = self.face(self.a)
        for d in range(self.dim):
            ij = 1 / self.J[d]
            c = self.a * self.W * (ij * ij) * ir
            D2 = self.D * self.D
            m = m + (c @ D2 if d == 0 else D2.T @ c)
            s = af * self.penalty(d, ir) * self.Wf[d]
            hi = s - af * ij * self.D[-1, -1] * self.end(d, ir, True) * self.Wf[d]
            lo = s + af * ij * self.D[0, 0] * self.right(d, ir) * self.Wf[d]
            m = m + self.at_ends(d, self.roll(d, lo, 1), hi)
        return m

    def source(self, u):
        gr = [[self.der(d, v) / self.J[d] for d in range(self.dim)] for v in u]
        div = sum(gr[d][d] for d in range(self.dim))
        R = div * div + sum(gr[i][k] * gr[k][i] for i in range(self.dim) for k in range(self.dim))
        return self.W * self.a * R

    def dot(self, a, b):
        return (a * b).sum(dim=tuple(range(1, a.dim())), keepdim=True)

    def solve(self, x, q, iters, solver):
        ir = 1 / q[-2]
        b, M = self.source([m * ir for m in q[:-2]]), self.diagonal(ir)
        if solver == "jacobi":
            for _ in range(iters):
                x = x + 2.0 / 3.0 * (b - self.sip(x, ir)) / M
            return x
        r = b - self.sip(x, ir)
        if solver == "pcg":
            z = r / M
            p, rz = z, self.dot(r, z)
            for _ in range(iters):
                Ap = self.sip(p, ir)
                a = rz / (self.dot(p, Ap) + 1e-30)
                x, r = x + a * p, r - a * Ap
                z = r / M
                new = self.dot(r, z)
                p, rz = z + new / (rz + 1e-30) * p, new
            return x
        lmax = (1.5, 2.0, 2.1, 2.2)[min(self.p, 4) - 1]
        theta, delta = (lmax + 1) / 2, (lmax - 1) / 2
        sigma = theta / delta
        rc = 1 / sigma
        for k in range(iters):
            z = r / M
            if k == 0:
                dd = z / theta
            else:
                rn = 1 / (2 * sigma - rc)
                dd = rn * rc * dd + 2 * rn / delta * z
                rc = rn
            x = x + dd
            if k + 1 < iters:
                r = b - self.sip(x, ir)
        return x

    def pressure(self, q):
        return (self.g - 1) * (q[-1] - sum(m * m for m in q[:-2]) / (2 * q[-2]))

    def rhs(self, q, S):
        P = self.pressure(q)
        out = [torch.zeros_like(v) for v in q]
        for d in range(self.dim):
            ij = 1 / self.J[d]
            u = q[d] / q[-2]
            f = [m * u for m in q[:-2]] + [q[d], (q[-1] + P + S) * u]
            f[d] = f[d] + P + S
            ws = u.abs() + torch.sqrt(self.g * P / q[-2])
            lam = self.larger(self.end(d, ws, True), self.right(d, ws))
            for v in range(len(q)):
                fL, fR = self.end(d, f[v], True), self.right(d, f[v])
                fs = (fL + fR) / 2 + lam * (self.end(d, q[v], True) - self.right(d, q[v])) / 2
                lift = self.at_ends(d, self.roll(d, (fs - fR) / self.w[0], 1), -(fs - fL) / self.w[-1])
                out[v] = out[v] - ij * self.der(d, f[v]) + ij * lift
        return out

    def step(self, q, S, dt, iters, solver):
        q0 = q
        for c0, c1 in ((0.0, 1.0), (0.75, 0.25), (1.0 / 3, 2.0 / 3)):
            S = self.solve(S, q, iters, solver)
            k = self.rhs(q, S)
            q = [c0 * a + c1 * b + c1 * dt * e for a, b, e in zip(q0, q, k)]
        return q, S


def _gradient(T, q, dt, case):
    """J, the gradient and (dJ/dgamma, dJ/dalpha) of every instance."""
    q = [v.detach().requires_grad_() for v in q]
    T.g, T.a = T.g.detach().requires_grad_(), T.a.detach().requires_grad_()
    x, S = q, torch.zeros_like(q[0])
    for _ in range(case["steps"]):
        x, S = T.step(x, S, dt, case["iters"], case["solver"])
    P = T.pressure(x)
    J = (T.W * P * P).sum(dim=tuple(range(1, P.dim())))
    grads = torch.autograd.grad(J.sum(), [*q, T.g, T.a])
    return J.detach(), grads[:-2], grads[-2].reshape(-1), grads[-1].reshape(-1)


def exact(case, seed):
    kind, dim = case["kind"], case["dim"]
    if kind in ("tangent", "continuous"):
        return None
    serial = case["steps"] * (case["iters"] + 4) * (3 if kind in ("gradient", "batch") else 1)
    per_group = 1 if dim == 1 else case["batch"]
    groups = len(set(_element_counts(case))) if dim == 1 else per_group
    if serial * groups > 9000 or work(case)["flops"] > 1e11:
        return None  # over 20 seconds of small torch operations
    st = prepare(case, seed)
    basis, n_p = st["basis"], st["basis"].n_p
    f = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device="cuda")

    def scalar(a):
        return f(a).reshape((-1,) + (1,) * (2 * dim))

    def fields(flat, mesh):  # (B, nodes) in the Julia order -> (B, [N_ey,] N_ex, [n_p,] n_p)
        return flat.reshape((-1,) + ((mesh.N_ey, mesh.N_ex, n_p, n_p) if dim == 2 else (mesh.N_e, n_p)))

    if kind == "batch":
        B = case["batch"]
        J, dg, da, dq = [None] * B, [None] * B, [None] * B, [None] * B
        counts = _element_counts(case)
        sets = [[b for b in range(B) if counts[b] == n] for n in sorted(set(counts))] if dim == 1 else [[b] for b in range(B)]
        for ids in sets:
            mesh = st["mesh"] if dim == 2 else igr.PeriodicMesh1D(counts[ids[0]], 1.0, basis)
            T = _Torch(dim, basis, mesh, scalar(st["gammas"][ids]), scalar(st["alphas"][ids]))
            if dim == 2:
                q = [fields(st["q0"][ids][:, v], mesh) for v in range(4)]
            else:
                q = [fields(f(np.stack([st["states"][b][v] for b in ids])), mesh) for v in range(3)]
            Jb, dqb, dgb, dab = _gradient(T, q, scalar(st["dts"][ids]), case)
            for k, b in enumerate(ids):
                J[b], dg[b], da[b] = Jb[k], dgb[k], dab[k]
                dq[b] = torch.stack([v[k].reshape(-1) for v in dqb])
        if dim == 2:
            return [torch.stack(J).cpu(), torch.stack(dq), torch.stack(dg).cpu(), torch.stack(da).cpu()]
        return [torch.stack(J).cpu().numpy(), torch.cat([v.reshape(-1) for v in dq]).cpu().numpy(),
                torch.stack(dg).cpu().numpy(), torch.stack(da).cpu().numpy()]

    mesh = st["mesh"]
    T = _Torch(dim, basis, mesh, scalar([st["gammas"][0]]), scalar([st["alphas"][0]]))
    q = [fields(f(v.reshape(-1, order="F"))[None], mesh) for v in st["q"]]
    host = lambda v: np.asfortranarray(v.detach().reshape(-1).cpu().numpy().reshape(mesh.x.shape, order="F"))
    if kind == "apply":
        return host(T.sip(q[-1], 1 / q[-2]))
    if kind == "rhs":
        S = T.solve(torch.zeros_like(q[0]), q, case["iters"], case["solver"])
        return [host(v) for v in T.rhs(q, S)] + [host(S)]
    if kind == "forward":
        n = math.ceil(st["T"] / float(st["dts"][0]))
        S = torch.zeros_like(q[0])
        for _ in range(n):
            q, S = T.step(q, S, st["T"] / n, case["iters"], case["solver"])
        return [host(v) for v in q] + [host(T.solve(S, q, case["iters"], case["solver"]))]
    J, dq, dg, da = _gradient(T, q, float(st["dts"][0]), case)
    if dim == 2:
        return [float(J[0]), *[host(v) for v in dq], float(dg[0]), float(da[0])]
    return [J.cpu().numpy(), *[v.reshape(-1).cpu().numpy() for v in dq], dg.cpu().numpy(), da.cpu().numpy()]
