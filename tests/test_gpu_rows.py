"""The assembled operator of the Krylov engine (csrc/rows.cu) on irregular
meshes: node degrees from 3 to 15, prescribed dofs scattered over the nodes,
unit counts around the slice length, 1 to 4 dofs per node.  Solves with random
diagonally dominant blocks against a dense solve of the same system; the
tolerance is the condition number times the relative residual asked for.
"""
import numpy as np
import pytest

from parallel_fem_codes_gb300 import meshgen as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fg():
    from parallel_fem_codes_gb300 import femgpu
    femgpu.lib()
    return femgpu


def _mesh(kind, ndof, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    if kind == "wheel":                       # a hub of 15 triangles (16 local colours at most)
        t = np.linspace(0.0, 2.0 * np.pi, 16)[:-1]
        X, Y = np.append(0.0, np.cos(t)), np.append(0.0, np.sin(t))
        ien = np.array([[0, 1 + i, 1 + (i + 1) % 15] for i in range(15)], dtype=np.int32)
    else:                                     # structured, every second quad with the other diagonal
        m, n = kind
        X, Y, ien = G.structured_mesh(m, n)
        for q in np.flatnonzero(rng.integers(0, 2, m * n)):
            a, b, d = ien[2 * q]
            c = ien[2 * q + 1, 2]
            ien[2 * q], ien[2 * q + 1] = (a, b, c), (b, d, c)
    ty = (rng.random(len(X) * ndof) > 0.15).astype(np.int32)
    ty[0] = 1
    invp, neq = G.number_dofs(ty)
    return G.Mesh(X, Y, ien, ndof, ty, invp, neq)


def _dense(m, A):
    S = 3 * m.ndof
    dof = (m.ien[:, :, None] * m.ndof + np.arange(m.ndof)).reshape(m.nel, S)
    dof = np.where(m.type[dof] != 0, m.invp[dof], m.neq)
    K = np.zeros((m.neq + 1, m.neq + 1))
    np.add.at(K, (np.repeat(dof, S, axis=1).reshape(-1), np.tile(dof, (1, S)).reshape(-1)), A.reshape(-1))
    K = K[:-1, :-1]
    free = np.flatnonzero(np.abs(K).sum(1) == 0)
    assert free.size == 0
    return K


@pytest.mark.parametrize("kind", [(1, 1), (4, 6), (5, 5), (31, 1), (13, 17), (23, 19), "wheel"])
@pytest.mark.parametrize("ndof,reorder", [(1, True), (1, False), (2, False), (3, False), (3, True), (4, False), (4, True)])
def test_solves_match_a_dense_solve(fg, kind, ndof, reorder):
    m = _mesh(kind, ndof, 3 + ndof)
    A = G.random_blocks(m.nel, 3 * ndof, seed=ndof, dominance=6.0 * ndof)
    K = _dense(m, A)
    rng = np.random.Generator(np.random.PCG64(9))
    F = np.append(rng.uniform(-1.0, 1.0, m.neq), 0.0)
    x = np.linalg.solve(K, F[:-1])
    s = fg.System(m, reorder=reorder)
    for pre in (fg.FG_PRECOND_NONE, fg.FG_PRECOND_DIAG, fg.FG_PRECOND_BLOCKDIAG):
        if pre == fg.FG_PRECOND_BLOCKDIAG and ndof == 1:
            continue
        s.set_blocks(A)
        B = s.precond_setup(pre, 0, F)
        for prec in (fg.FG_PREC_FP64, fg.FG_PREC_MIXED):
            r = s.solve(B, tol=1e-12, F_true=F, precision=prec)
            assert r.stats["converged"] == 1, r.stats
            tol = 10 * np.linalg.cond(K) * max(1e-12, r.stats["true_rel_residual"])
            assert np.linalg.norm(r.x[:-1] - x) <= tol * np.linalg.norm(x)
            assert r.x[-1] == 0.0


def test_new_blocks_are_assembled_again(fg):
    m = _mesh((6, 5), 1, 1)
    s = fg.System(m)
    F = np.append(np.ones(m.neq), 0.0)
    for seed in (1, 2):
        A = G.random_blocks(m.nel, 3, seed=seed, dominance=6.0)
        s.set_blocks(A)
        B = s.precond_setup(fg.FG_PRECOND_DIAG, 0, F)
        x = np.linalg.solve(_dense(m, A), F[:-1])
        for prec in (fg.FG_PREC_MIXED, fg.FG_PREC_FP64):
            r = s.solve(B, tol=1e-12, F_true=F, precision=prec)
            assert np.linalg.norm(r.x[:-1] - x) <= 1e-9 * np.linalg.norm(x)
        # the element matvec in FP32 sees the new blocks too
        y = s.matvec(r.x, precision=32)
        assert np.linalg.norm(y[:-1] - F[:-1]) <= 1e-5 * np.linalg.norm(F)


# Streaming sweeps (FP16 bases; a numbering too wide for the chip): rows in
# pairs (slices of one width), single rows (a wheel's hub, 2 dofs per node),
# columns within 2^15 units and beyond
@pytest.mark.parametrize("kind,ndof", [((4, 6), 1), ((5, 5), 1), ((31, 1), 1), ((13, 17), 1), ((40, 37), 1), ("wheel", 1),
                                       ((13, 17), 2), ("wheel", 2), ((32000, 1), 2), ((33000, 1), 2)])
def test_streamed_solves(fg, kind, ndof):
    m = _mesh(kind, ndof, 7)
    A = G.random_blocks(m.nel, 3 * ndof, seed=2, dominance=6.0 * ndof)
    F = np.append(np.random.Generator(np.random.PCG64(9)).uniform(-1.0, 1.0, m.neq), 0.0)
    s = fg.System(m, reorder=False)
    s.set_blocks(A)
    B = s.precond_setup(fg.FG_PRECOND_DIAG, 0, F)
    for prec in (fg.FG_PREC_MIXED16, fg.FG_PREC_MIXED, fg.FG_PREC_FP64):
        r = s.solve(B, tol=1e-11, F_true=F, precision=prec)
        assert r.stats["converged"] == 1, r.stats
        res = np.linalg.norm((F - s.matvec(r.x))[:-1]) / np.linalg.norm(F[:-1])
        assert res <= 1e-9, prec


# Operators and right-hand sides far from 1, by powers of two: the same solve but
# for the scale, on chip and streaming.  (The tolerance is the solves', 1e-11, times
# a condition below 100.)
@pytest.mark.parametrize("kind,ndof", [((23, 19), 1), ((33000, 1), 2)])
@pytest.mark.parametrize("precision,ea,ef", [(32, 50, 0), (32, -50, 0), (32, 0, 150), (32, -40, -150), (64, 400, 0), (64, -400, 0)])
def test_scaled_systems(fg, kind, ndof, precision, ea, ef):
    m = _mesh(kind, ndof, 7)
    A = G.random_blocks(m.nel, 3 * ndof, seed=2, dominance=6.0 * ndof)
    F = np.append(np.random.Generator(np.random.PCG64(9)).uniform(-1.0, 1.0, m.neq), 0.0)
    xs, its = [], []
    for a, f in ((0, 0), (ea, ef)):
        s = fg.System(m, reorder=False)
        s.set_blocks(A * 2.0 ** a)
        B = s.precond_setup(fg.FG_PRECOND_NONE, 0, F * 2.0 ** f)
        r = s.solve(B, tol=1e-11, F_true=F * 2.0 ** f, precision=precision)
        assert r.stats["converged"] == 1 and r.stats["true_rel_residual"] <= 1e-10, r.stats
        xs.append(r.x * 2.0 ** (a - f))
        its.append(r.stats["iterations"])
    assert its[0] == its[1]
    assert np.linalg.norm(xs[1] - xs[0]) <= 1e-9 * np.linalg.norm(xs[0])


# BlockDiag in the streaming matvec (a node's rows by shuffles): the meshes of
# test_streamed_solves with 2 to 4 dofs a node
@pytest.mark.parametrize("kind", [(1, 1), (13, 17), "wheel", (32000, 1), (33000, 1)])
@pytest.mark.parametrize("ndof", [2, 3, 4])
def test_streamed_block_diagonal(fg, kind, ndof):
    m = _mesh(kind, ndof, 7)
    A = G.random_blocks(m.nel, 3 * ndof, seed=2, dominance=6.0 * ndof)
    F = np.append(np.random.Generator(np.random.PCG64(9)).uniform(-1.0, 1.0, m.neq), 0.0)
    s = fg.System(m, reorder=False)
    s.set_blocks(A)
    B = s.precond_setup(fg.FG_PRECOND_BLOCKDIAG, 0, F)
    for prec in (fg.FG_PREC_MIXED16, fg.FG_PREC_MIXED, fg.FG_PREC_FP64):
        r = s.solve(B, tol=1e-11, F_true=F, precision=prec)
        assert r.stats["converged"] == 1, r.stats
        res = np.linalg.norm((F - s.matvec(r.x))[:-1]) / np.linalg.norm(F[:-1])
        assert res <= 1e-9, prec
