"""The on-chip restart cycle (csrc/cycle.cu) at the edges of its gangs: one
CTA, two, the largest gang whose CTAs sum all partials themselves and the next
one, many CTAs; restart lengths below and above the CTA's lane groups; a batch
that starts streaming and moves on chip as members converge.  FP64 solves
against the oracle's GMRES (solution 1e-9, iterations within two), mixed
precision against the same solution by its true residual.
"""
import numpy as np
import pytest

import oracle as O
from parallel_fem_codes_gb300 import meshgen as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fg():
    from parallel_fem_codes_gb300 import femgpu
    femgpu.lib()
    return femgpu


# 64 FP64 rows (256 FP32) a CTA: 64, 100, 256, 484, 529, 961, 1089, 4096 equations
@pytest.mark.parametrize("side,kmax", [(10, 30), (12, 30), (18, 30), (24, 30), (25, 30), (33, 30), (35, 30), (66, 30), (33, 3), (35, 33), (35, 60), (12, 60)])
def test_matches_the_oracle(fg, side, kmax):
    p = G.transport_problem(side, angle_deg=40.0, k=1e-3)
    m = p.mesh
    A, F = O.build_k_f_supg(p)
    lm = O.fill_lm(m)
    perm, inv, _ = O.permutation_of_lm(m)
    X0, it0, _, _, _ = O.ebe_diag_solve(lm, A, m.neq, F, perm, inv, kmax=kmax, lmax=3000, tol=1e-10)
    s = fg.System(m)
    s.set_blocks(A)
    B = s.precond_setup(fg.FG_PRECOND_DIAG, 0, F)
    r = s.solve(B, kmax=kmax, lmax=3000, tol=1e-10, F_true=F)
    assert r.stats["converged"] == 1 and r.stats["status"] == 0
    assert abs(r.stats["iterations"] - it0) <= 2
    n = np.linalg.norm
    assert n(r.x[:-1] - X0[:-1]) <= 1e-9 * n(X0[:-1])
    q = s.solve(B, kmax=kmax, lmax=3000, tol=1e-12, F_true=F, precision=fg.FG_PREC_MIXED)
    assert q.stats["converged"] == 1 and q.stats["true_rel_residual"] <= 1e-12
    assert n(q.x[:-1] - X0[:-1]) <= 1e-8 * n(X0[:-1])
    again = s.solve(B, kmax=kmax, lmax=3000, tol=1e-12, F_true=F, precision=fg.FG_PREC_MIXED)
    assert np.array_equal(again.x, q.x) and again.stats["iterations"] == q.stats["iterations"]


@pytest.mark.parametrize("precision", [64, 32])
def test_a_batch_moves_on_chip(fg, precision):
    # together more CTAs than are resident: the first cycles stream
    probs = [G.transport_problem(n, angle_deg=15.0 * n, k=10.0 ** -(2 + n % 5)) for n in (40, 300, 301, 45, 302, 120)]
    systems = [fg.transport_system(p) for p in probs]
    for s, p in zip(systems, probs):
        s.transport_prepare(p)
    st = fg.solve_resident(systems, tol=1e-11, lmax=3000, precision=precision)
    for s, p, q in zip(systems, probs, st):
        assert q["converged"] == 1 and q["status"] == 0
        x = s.solution()
        s.transport_prepare(p)
        F = s.transport_assemble(p)
        res = np.linalg.norm((F - s.matvec(x))[:-1]) / np.linalg.norm(F[:-1])
        assert res <= (1e-11 if precision == 32 else 1e-9)


def test_breakdown_and_zero_right_hand_side(fg):
    p = G.transport_problem(40, k=1e-2)
    s = fg.transport_system(p)
    F = s.transport_assemble(p)
    B = s.precond_setup(fg.FG_PRECOND_DIAG, 0, F)
    for prec in (64, 32):
        z = s.solve(np.zeros_like(B), F_true=np.zeros_like(F), precision=prec)
        assert z.stats["converged"] == 1 and not z.x.any()
        bad = B.copy()
        bad[7] = np.nan
        r = s.solve(bad, precision=prec)
        assert r.stats["converged"] == 0 and r.stats["status"] == fg.FG_ERR_BREAKDOWN
        ok = s.solve(B, F_true=F, precision=prec)
        assert ok.stats["converged"] == 1


@pytest.mark.parametrize("side,kmax,precision", [(370, 30, 64), (387, 30, 64), (560, 30, 32), (230, 60, 64)])
def test_a_system_beyond_shared_memory(fg, side, kmax, precision):
    # part of the basis in global memory; true residual by the element matvec
    p = G.transport_problem(side, angle_deg=40.0, k=1e-3)
    s = fg.transport_system(p)
    s.transport_prepare(p)
    st = fg.solve_resident([s], kmax=kmax, tol=1e-11, lmax=3000, precision=precision)[0]
    assert st["converged"] == 1 and st["status"] == 0
    x = s.solution()
    F = s.transport_assemble(p)
    assert np.linalg.norm((F - s.matvec(x))[:-1]) <= (1e-11 if precision == 32 else 1e-9) * np.linalg.norm(F[:-1])


# 376 x 376 equations fit 152 CTAs in FP64, 525 x 525 in FP32; up to four launches, then streaming
@pytest.mark.parametrize("sides,precision", [((380, 40, 300, 35), 64), ((200, 290, 210, 300, 220), 64), ((340, 350, 360, 365, 370), 64), ((378, 380, 382, 385, 387), 64),
                                             ((513, 37, 400), 32), ((530, 36), 32), ((500, 505, 510, 513, 37, 500), 32)])
def test_a_batch_in_several_launches(fg, sides, precision):
    probs = [G.transport_problem(n, angle_deg=11.0 * n, k=10.0 ** -(2 + n % 3)) for n in sides]
    systems = [fg.transport_system(p) for p in probs]
    for s, p in zip(systems, probs):
        s.transport_prepare(p)
    st = fg.solve_resident(systems, tol=1e-11, lmax=3000, precision=precision)
    for s, p, q in zip(systems, probs, st):
        assert q["converged"] == 1 and q["status"] == 0
        x = s.solution()
        F = s.transport_assemble(p)
        assert np.linalg.norm((F - s.matvec(x))[:-1]) <= (1e-11 if precision == 32 else 1e-9) * np.linalg.norm(F[:-1])


def test_streams_where_memory_for_the_gang_is_short(fg):
    # five systems too large for the chip stream one cycle and so have a basis; then no more may be allocated
    probs = [G.transport_problem(n, angle_deg=40.0, k=1e-2) for n in (380, 381, 382, 383, 384)]
    systems = [fg.transport_system(p) for p in probs]
    for s, p in zip(systems, probs):
        s.transport_prepare(p)
    fg.solve_resident(systems, tol=1e-11, lmax=1, precision=64)
    used = fg.memory_in_use()
    xs = []
    for limit in (used + 4096, 0):
        fg.set_memory_limit(limit)
        try:
            st = fg.solve_resident(systems[:1], tol=1e-11, lmax=3000, precision=64)[0]
        finally:
            fg.set_memory_limit(0)
        assert st["converged"] == 1 and st["status"] == 0
        assert (fg.memory_in_use() == used) == (limit > 0)
        xs.append(systems[0].solution())
    assert np.linalg.norm(xs[0] - xs[1]) <= 1e-8 * np.linalg.norm(xs[1])


@pytest.mark.parametrize("sides", [(381, 383, 385, 40, 120), (40, 381, 383, 385, 387, 120)])
def test_streaming_again_after_a_basis_was_lent(fg, sides):
    # odd counts of equations: the batch streams, then large members keep basis vectors where it streamed
    probs = [G.transport_problem(n, angle_deg=11.0 * n, k=10.0 ** -(2 + n % 3)) for n in sides]
    systems = [fg.transport_system(p) for p in probs]
    first = None
    for _ in range(3):
        for s, p in zip(systems, probs):
            s.transport_prepare(p)
        st = fg.solve_resident(systems, tol=1e-11, lmax=3000, precision=64)
        got = [(q["converged"], q["iterations"], s.solution()) for s, q in zip(systems, st)]
        first = first or got
        for a, b in zip(first, got):
            assert a[:2] == b[:2] and a[0] == 1
            assert np.array_equal(a[2], b[2]) and b[2][-1] == 0.0


@pytest.mark.parametrize("kmax,lmax", [(30, 2000), (2, 12)])
def test_every_memory_limit_solves_or_refuses(fg, kmax, lmax):
    # members stop at different cycles, so that the others' gangs grow; a limit in between must not strand a cycle
    probs = [G.transport_problem(n, angle_deg=40.0, k=k) for n, k in ((150, 1e-1), (210, 1e-3), (200, 1e-2), (60, 1e-1))]

    def solve(extra):
        systems = [fg.transport_system(p) for p in probs]
        for s, p in zip(systems, probs):
            s.transport_prepare(p)
        before = fg.memory_in_use()
        fg.set_memory_limit(before + extra if extra else 0)
        try:
            st = fg.solve_resident(systems, kmax=kmax, tol=1e-10, lmax=lmax, precision=64)
            return fg.memory_in_use() - before, [s.solution() for s in systems], st
        except fg.FemGpuError as e:
            assert extra and e.code == fg.FG_ERR_NOMEM
            return None
        finally:
            fg.set_memory_limit(0)

    need, ref, _ = solve(0)
    outcomes = []
    for short in (0, 1, 2, 3, 4, 6, 8, 12, 16, 32, 64, 256):
        got = solve(need - short * need // 1024)
        outcomes.append(got is not None)
        if got is None:
            continue
        for x, y, q in zip(ref, got[1], got[2]):
            assert q["status"] in (fg.FG_OK, fg.FG_ERR_NOTCONV)
            assert np.linalg.norm(x - y) <= 1e-7 * np.linalg.norm(x)
    assert outcomes[0] and not outcomes[-1]


@pytest.mark.parametrize("precision", [64, 32])
def test_wait_limit_times_out_and_recovers(fg, precision):
    # one poll an exchange: some CTA looks before its neighbour has published
    p = G.transport_problem(129, angle_deg=40.0, k=1e-3)
    s = fg.transport_system(p)
    s.transport_prepare(p)
    good = fg.solve_resident([s], tol=1e-10, precision=precision)[0]
    x = s.solution()
    try:
        fg.set_wait_limit(1)
        st = fg.solve_resident([s], tol=1e-10, precision=precision)[0]
    finally:
        fg.set_wait_limit()
    assert good["converged"] == 1 and st["converged"] == 0 and st["status"] == fg.FG_ERR_TIMEOUT
    again = fg.solve_resident([s], tol=1e-10, precision=precision)[0]
    assert again["converged"] == 1 and again["iterations"] == good["iterations"]
    assert np.array_equal(s.solution(), x)


def _multi_dof(fg, kind, n):
    if kind == "ns":
        p = G.cavity_problem(n, reynolds=1000.0, jitter=0.2)
        s = fg.ns_system(p)
        m = p.mesh
        v = np.stack([np.sin(3 * m.x) * m.y, np.cos(2 * m.y) * m.x, 0.1 * m.x * m.y], 1).reshape(-1)
        return s, s.ns_assemble(p, np.ascontiguousarray(v[m.type != 0]))
    # a transport operator for each dof, the dofs of a node coupled
    K, _ = O.build_k_f_supg(G.transport_problem(n, angle_deg=40.0, k=1e-2))
    m = G.multi_dof_mesh(n, kind, seed=1)
    A = np.einsum("eab,rq->earbq", K.reshape(m.nel, 3, 3), 0.9 * np.eye(kind) + 0.1)
    s = fg.System(m, reorder=False)
    s.set_blocks(np.ascontiguousarray(A.reshape(m.nel, -1)))
    return s, np.append(np.random.Generator(np.random.PCG64(9)).uniform(-1.0, 1.0, m.neq), 0.0)


# Bases beyond shared memory with 2 to 4 dofs a node, BlockDiag, GMRES(60): one
# system (a spilling gang) against four of them (which stream), one restart cycle
@pytest.mark.parametrize("kind,n,precision", [("ns", 181, 64), ("ns", 257, 32), (2, 221, 64), (4, 161, 64), (4, 231, 32)])
def test_spilling_and_streaming_agree(fg, kind, n, precision):
    systems, Bs, Fs = [], [], []
    for _ in range(4):
        s, F = _multi_dof(fg, kind, n)
        Bs.append(s.precond_setup(fg.FG_PRECOND_BLOCKDIAG, 0, F))
        Fs.append(F)
        systems.append(s)
    one = systems[0].solve(Bs[0], kmax=60, lmax=1, tol=1e-14, F_true=Fs[0], precision=precision)
    X, st = fg.solve_batch(systems, Bs, Fs, kmax=60, lmax=1, tol=1e-14, precision=precision)
    assert all(np.array_equal(X[0], x) for x in X[1:])
    assert one.stats["iterations"] == st[0]["iterations"] == 59
    # rounding over 59 steps, times 100 for the triangular system
    eps = 60 * 100 * (2.0 ** -53 if precision == 64 else 2.0 ** -24)
    assert np.linalg.norm(one.x - X[0]) <= eps * np.linalg.norm(X[0])
    a, b = one.stats["true_rel_residual"], st[0]["true_rel_residual"]
    assert abs(a - b) <= eps * max(a, 1e-3)
