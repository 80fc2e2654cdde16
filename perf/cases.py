"""Performance cases of the solve path: what a program built on this library has it do.

Each case is one pass through the public Python API (parallel_fem_codes_gb300.femgpu):

  transport  steady SUPG/CAU transport: device assembly, Diag set-up, one GMRES solve, the solution read back
  host       the same linear system through host buffers: element blocks in, Diag set-up, solve, solution out
  batch      many transport instances of uneven size assembled and solved together
  served     host-buffer requests answered by the request server (continuous batching)
  process    the nonlinear CAU fixed-point loop (assembly + solve per iteration), four iterations, where it has
             settled to about 1e-3
  euler      compressible Euler time loop (OBLIQUO): predictor / two corrections per step, BlockDiag GMRES(25)
  ns         one Navier-Stokes Picard system (jittered cavity, Re 1000): assembly, BlockDiag set-up, GMRES(50) cycles

Sizes are nodes per side of the unit square, 33 to 513 for transport (the batched workload's range), and the
Euler / Navier-Stokes meshes of the tests and the benchmark.  The workloads' tolerance is a relative residual of
1e-10; the mixed-precision cases ask for 1e-11, so that the solution itself, not only its residual, is good to 1e-9
over the whole range of conductivities.
"""
import math

import numpy as np
import torch

from parallel_fem_codes_gb300 import femgpu as fg
from parallel_fem_codes_gb300 import meshgen

MIXED_TOL = 1e-11
FP64_TOL = 1e-10
GAMMA = 0.0          # reaction of the transport problems
NONLINEAR = 4        # fixed-point iterations of the process cases (the drivers' 1e-3 stop takes 3 to 5 here)
BATCH_SEED = 4       # the batched workload's instance seed


def listed():
    return [
        # a single small solve, as an outer program asks for one after another: launches and latency
        dict(name="transport_33_fp64", kind="transport", n=33, k=1e-6, angle=30.0, precision=64),
        # the 129 x 129 steady configuration, served precision
        dict(name="transport_129_mixed", kind="transport", n=129, k=1e-6, angle=30.0, precision=32),
        # the same configuration entered as the reference's drivers do: element blocks and F on the host, FP64 GMRES(30)
        dict(name="host_129_fp64", kind="host", n=129, k=1e-6, angle=30.0, precision=64),
        # one large solve, convection-dominated, an odd size
        dict(name="transport_385_fp64", kind="transport", n=385, k=1e-5, angle=75.0, precision=64),
        # the largest single mesh of the batched workload, diffusive end of its range
        dict(name="transport_513_mixed", kind="transport", n=513, k=1e-3, angle=130.0, precision=32),
        # the batched workload (uneven sizes 33..513, mixed precision), 32 of its instances
        dict(name="batch_32_mixed", kind="batch", count=32, first=0, precision=32),
        # the plain method on a batch
        dict(name="batch_10_fp64", kind="batch", count=10, first=40, precision=64),
        # host-buffer requests through the server
        dict(name="served_16_mixed", kind="served", count=16, first=100, nmax=300, precision=32),
        # nonlinear shock-capturing loop, an odd size
        dict(name="process_97_fp64", kind="process", n=97, k=1e-6, angle=30.0, precision=64),
        # time loops: small FP64, and the larger one in served precision
        dict(name="euler_65_fp64", kind="euler", n=65, steps=4, precision=64),
        dict(name="euler_257_mixed", kind="euler", n=257, steps=3, precision=32),
        # GMRES(50) cycles on 3-dof blocks
        dict(name="ns_257_fp64", kind="ns", n=257, cycles=3, precision=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["transport", "transport", "host", "batch", "served", "process", "euler", "euler", "ns"])
    prec = rng.choice([32, 64])
    k = 10.0 ** rng.uniform(-8.0, -2.0)
    angle = rng.uniform(0.0, 360.0)
    if kind == "transport":
        return dict(kind=kind, n=_log_int(rng, 33, 513), k=k, angle=angle, precision=prec)
    if kind == "host":
        return dict(kind=kind, n=_log_int(rng, 33, 257), k=k, angle=angle, precision=prec)
    if kind == "batch":
        return dict(kind=kind, count=_log_int(rng, 2, 32 if prec == 32 else 10), first=rng.randrange(0, 200), precision=prec)
    if kind == "served":
        return dict(kind=kind, count=_log_int(rng, 2, 16), first=rng.randrange(0, 200), nmax=300, precision=32)
    if kind == "process":
        return dict(kind=kind, n=_log_int(rng, 33, 97), k=1e-6, angle=rng.uniform(20.0, 70.0), precision=64)
    if kind == "euler":
        return dict(kind=kind, n=_log_int(rng, 17, 257), steps=rng.randrange(1, 4), precision=prec)
    return dict(kind=kind, n=2 * _log_int(rng, 8, 128) + 1, cycles=rng.randrange(1, 4), precision=64)


# ---------------------------------------------------------------- inputs
def _transport(n, angle, k, rng):
    """A transport problem whose Dirichlet data and source are drawn from rng: smooth values around the workload's
    u = 1 on the inflow edges x = 0 and y = 0, 0 elsewhere on the boundary."""
    p = meshgen.transport_problem(n, angle_deg=angle, k=k)
    m = p.mesh
    a, b = rng.uniform(0.5, 1.5, 2), rng.uniform(0.0, 2.0 * math.pi, 2)
    on = (m.type == 0) & (p.upresc > 0)
    p.upresc = np.where(on, a[0] + 0.2 * a[1] * np.sin(5.0 * (m.x + m.y) + b[0]), 0.0)
    p.f = float(0.1 * np.cos(b[1]))
    p.gamma = GAMMA
    return p


def _batch_params(case):
    ns, angles, ks = meshgen.batch_transport_params(256, BATCH_SEED, 33, case.get("nmax", 513))
    idx = [(case["first"] + i) % 256 for i in range(case["count"])]
    return [(ns[i], angles[i], ks[i]) for i in idx]


def _problems(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    if case["kind"] in ("batch", "served"):
        return [_transport(n, a, k, rng) for n, a, k in _batch_params(case)]
    return [_transport(case["n"], case["angle"], case["k"], rng)]


def _elements(p, u=None):
    """Element matrices (nel, 3, 3) and loads (nel, 3) of the SUPG form with CAU shock capturing at u (free dofs)."""
    m = p.mesh
    U = np.where(m.type == 0, p.upresc, 0.0 if u is None else u[np.maximum(m.invp, 0)])
    X, Y, E = m.x[m.ien], m.y[m.ien], U[m.ien]
    b = np.stack([Y[:, 1] - Y[:, 2], Y[:, 2] - Y[:, 0], Y[:, 0] - Y[:, 1]], 1)
    c = np.stack([X[:, 2] - X[:, 1], X[:, 0] - X[:, 2], X[:, 1] - X[:, 0]], 1)
    two_a = c[:, 2] * b[:, 1] - c[:, 1] * b[:, 2]
    area, h = 0.5 * two_a, np.sqrt(np.abs(two_a))
    bx, by = p.beta
    adv = bx * b + by * c
    tau = 0.5 * h / math.hypot(bx, by)
    lap = (b[:, :, None] * b[:, None, :] + c[:, :, None] * c[:, None, :]) / (4.0 * area)[:, None, None]
    gx, gy = (b * E).sum(1) / two_a, (c * E).sum(1) / two_a
    ng = np.sqrt(gx * gx + gy * gy)
    bgu = bx * gx + by * gy
    res = np.abs(bgu + p.gamma * E.mean(1) - p.f)
    with np.errstate(divide="ignore", invalid="ignore"):
        nb = np.abs(bgu) / ng
        pe3 = (0.5 * h * nb / p.k) / 3.0
        eu = np.where(ng > 0, 0.5 * h * np.where(pe3 < 0.7, pe3, 0.7) * res / ng, 0.0)
    eu = eu if p.cau else np.zeros_like(eu)
    mass = (np.ones((3, 3)) + np.eye(3)) / 12.0
    K = (p.k + eu)[:, None, None] * lap
    K = K + adv[:, None, :] / 6.0                                                      # Galerkin advection
    K = K + (tau / (4.0 * area))[:, None, None] * adv[:, :, None] * adv[:, None, :]    # SUPG advection
    K = K + p.gamma * (area[:, None, None] * mass + tau[:, None, None] * adv[:, :, None] / 6.0)
    F = p.f * (area[:, None] / 3.0 + 0.5 * tau[:, None] * adv)
    return K, F


def _assemble(p, u=None):
    """(rows, cols, values, F): the linear system over the free dofs with the Dirichlet values moved to F."""
    m = p.mesh
    K, Fe = _elements(p, u)
    free = m.type[m.ien] != 0
    dof = np.where(free, m.invp[m.ien], 0)
    F = np.bincount(dof[free], weights=Fe[free], minlength=m.neq)
    lift = np.where(free[:, :, None] & ~free[:, None, :], K * p.upresc[m.ien][:, None, :], 0.0).sum(2)
    F = F - np.bincount(dof[free], weights=lift[free], minlength=m.neq)
    both = free[:, :, None] & free[:, None, :]
    r = np.broadcast_to(dof[:, :, None], K.shape)[both]
    c = np.broadcast_to(dof[:, None, :], K.shape)[both]
    return r, c, K[both], F


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return t.numpy(), t


def _host_system(p):
    """Element blocks and F (n + 1 slots) as a driver holds them on the host, in pinned memory."""
    K, _ = _elements(p)
    F = np.append(_assemble(p)[3], 0.0)
    return _pinned(K.reshape(p.mesh.nel, 9)), _pinned(F)


# ---------------------------------------------------------------- the cases
def _options(case):
    mixed = case["precision"] == 32
    return dict(tol=MIXED_TOL if mixed else FP64_TOL, precision=fg.FG_PREC_MIXED if mixed else fg.FG_PREC_FP64, lmax=2000)


def prepare(case, seed):
    kind = case["kind"]
    o = _options(case)
    if kind in ("transport", "process"):
        p = _problems(case, seed)[0]
        return dict(kind=kind, p=p, s=fg.transport_system(p), o=o)
    if kind == "host":
        p = _problems(case, seed)[0]
        (A, ka), (F, kf) = _host_system(p)
        return dict(kind=kind, s=fg.System(p.mesh), A=A, F=F, keep=(ka, kf), o=o)
    if kind == "batch":
        ps = _problems(case, seed)
        return dict(kind=kind, ps=ps, ss=[fg.transport_system(p) for p in ps], o=o)
    if kind == "served":
        ps = _problems(case, seed)
        bufs = [_host_system(p) for p in ps]
        return dict(kind=kind, ss=[fg.System(p.mesh) for p in ps], A=[b[0][0] for b in bufs], F=[b[1][0] for b in bufs],
                    keep=bufs, server=fg.Server(kmax=30, lmax=2000, tol=o["tol"], precision=o["precision"]))
    rng = np.random.Generator(np.random.PCG64(seed))
    if kind == "euler":
        p = meshgen.obliquo_problem(case["n"])
        m = p.mesh
        u0 = p.initial_state()
        # a smooth disturbance of the uniform initial state, a hundredth of it
        node = np.repeat(np.arange(m.nnodes), 4)[m.type != 0]
        w = np.sin(6.0 * m.x[node] + rng.uniform(0, 6)) * np.cos(5.0 * m.y[node] + rng.uniform(0, 6))
        u0 = u0 * (1.0 + 0.01 * w)
        t = fg.time_opts(stop_by_norm=0, max_corrections=2, final_time=case["steps"] * p.dt)
        o["lmax"] = 1000
        return dict(kind=kind, p=p, s=fg.euler_system(p), u0=u0, t=t, o=o)
    p = meshgen.cavity_problem(case["n"], reynolds=1000.0, jitter=0.2)
    m = p.mesh
    # a smooth state as after a few Picard iterations
    x, y = m.x, m.y
    a, b = rng.uniform(0.5, 1.0), rng.uniform(0.0, 0.3)
    psi = np.sin(math.pi * x) * np.sin(math.pi * y)
    v = np.stack([a * psi * np.cos(3 * y + b), -a * psi * np.cos(3 * x - b), 0.1 * np.cos(3 * x) * np.cos(2 * y)], 1).reshape(-1)
    o["lmax"] = case["cycles"]
    return dict(kind=kind, p=p, s=fg.ns_system(p), u=np.ascontiguousarray(v[m.type != 0]), o=o)


def run(st):
    kind = st["kind"]
    if kind == "transport":
        st["s"].transport_prepare(st["p"])
        fg.solve_resident([st["s"]], kmax=30, **st["o"])
        return st["s"].solution()
    if kind == "host":
        st["s"].set_blocks(st["A"])
        B = st["s"].precond_setup(fg.FG_PRECOND_DIAG, 0, st["F"])
        return st["s"].solve(B, kmax=30, F_true=st["F"], **st["o"]).x
    if kind == "batch":
        for s, p in zip(st["ss"], st["ps"]):
            s.transport_prepare(p)
        fg.solve_resident(st["ss"], kmax=30, **st["o"])
        return [s.solution() for s in st["ss"]]
    if kind == "served":
        srv = st["server"]
        Xs = [np.empty(s.n + 1) for s in st["ss"]]
        for i, s in enumerate(st["ss"]):
            srv.submit_host(s, st["A"][i], st["F"][i], Xs[i], i + 1)
        srv.wait(len(Xs), 120.0)
        srv.poll()
        return Xs
    if kind == "process":
        return st["s"].transport_process(st["p"], kmax=30, lmax=2000, tol=st["o"]["tol"], nonlinear_tol=1e-9,
                                         max_nonlinear=NONLINEAR, precision=st["o"]["precision"])[0]
    if kind == "euler":
        u, a, _ = st["s"].euler_predictor(st["p"], st["t"], u0=st["u0"], kmax=25, **st["o"])
        return [u, a]
    R = st["s"].ns_assemble(st["p"], st["u"])
    B = st["s"].precond_setup(fg.FG_PRECOND_BLOCKDIAG, 0, R)
    return [R, st["s"].solve(B, kmax=50, F_true=R, **st["o"]).x]


# ---------------------------------------------------------------- the least work
def _gmres(nodes, ndof, w, steps, kmax):
    """Bytes and operations of GMRES steps: the operator's nonzeros once and the basis once per step (about 7
    coupled nodes per node, kmax / 2 basis vectors on average), the new basis vector written."""
    nnz, n = 7.0 * nodes * ndof * ndof, float(nodes * ndof)
    return steps * (nnz * w + n * w * (0.5 * kmax + 1.0)), steps * (2.0 * nnz + 4.0 * n * 0.5 * kmax)


def _instance(n, w, solves=1):
    # about 15 n^0.72 steps to 1e-10 on this problem family; element blocks or geometry read, solution written
    nodes, nel = (n - 2) ** 2, 2 * (n - 1) ** 2
    b, f = _gmres(nodes, 1, w, 15.0 * n ** 0.72, 30)
    return solves * (b + nel * 72.0 + nodes * 16.0), solves * (f + nel * 150.0)


def work(case):
    w = 4.0 if case["precision"] == 32 else 8.0
    kind = case["kind"]
    if kind in ("batch", "served"):
        parts = [_instance(n, w) for n, _, _ in _batch_params(case)]
        return dict(bytes=sum(p[0] for p in parts), flops=sum(p[1] for p in parts))
    n = case["n"]
    if kind in ("transport", "host", "process"):
        b, f = _instance(n, w, NONLINEAR if kind == "process" else 1)
        return dict(bytes=b, flops=f)
    nodes, nel = n * n, 2 * (n - 1) ** 2
    if kind == "euler":
        # two corrections a step, about 14 GMRES steps each; 12 x 12 blocks formed once per correction
        c = 2 * case["steps"]
        b, f = _gmres(nodes, 4, w, 14.0 * c, 14)
        return dict(bytes=b + c * (nodes * 4 * 6 * 8.0 + nodes * 7 * 16 * 8.0), flops=f + c * nel * 4000.0)
    b, f = _gmres(nodes, 3, w, 49.0 * case["cycles"], 50)
    return dict(bytes=b + nodes * 3 * 4 * 8.0, flops=f + nel * 1500.0)


# ---------------------------------------------------------------- 64-bit reference
def _solve_exact(p, u=None):
    """The free-dof solution of the linear system at u by block-tridiagonal elimination over mesh rows."""
    r, c, v, F = _assemble(p, u)
    n = p.mesh.neq
    m = int(round(math.sqrt(n)))
    rb, order = r // m, np.argsort(r // m, kind="stable")
    r, c, v, rb = r[order], c[order], v[order], rb[order]
    at = np.searchsorted(rb, np.arange(m + 1))
    G, g = [], []
    for j in range(m):
        i = slice(at[j], at[j + 1])
        blk = np.bincount((r[i] - j * m) * (3 * m) + (c[i] - (j - 1) * m), weights=v[i], minlength=3 * m * m).reshape(m, 3 * m)
        L, D, U, f = blk[:, :m], blk[:, m:2 * m], blk[:, 2 * m:], F[j * m:(j + 1) * m]
        if j:
            D, f = D - L @ G[-1], f - L @ g[-1]
        s = np.linalg.solve(D, np.concatenate([U, f[:, None]], 1))
        G.append(s[:, :m].copy())
        g.append(s[:, m].copy())
    x = np.empty((m, m))
    x[m - 1] = g[m - 1]
    for j in range(m - 2, -1, -1):
        x[j] = g[j] - G[j] @ x[j + 1]
    return x.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("euler", "ns"):
        return None
    ps = _problems(case, seed)
    if kind == "process":
        u = np.zeros(ps[0].mesh.neq)
        for _ in range(NONLINEAR):
            u = _solve_exact(ps[0], u)
        return u
    if kind in ("batch", "served"):
        return [np.append(_solve_exact(p), 0.0) if p.mesh.neq <= 200 ** 2 else None for p in ps]
    return np.append(_solve_exact(ps[0]), 0.0)
