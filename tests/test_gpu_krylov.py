"""The Krylov solvers' vector kernels at the sizes where their tiles end: the
preconditioner's inner GMRES against the same iteration in numpy (basis sizes
around the 8-vector tile and the 32- and 64-column solve), and lockstep sets
on both forms of the Gram-Schmidt step (clusters up to 16,384 values and 12
systems, with and without basis vectors beyond their shared memory; three
launches of 1, 2 and 4 rows per thread) against numpy and against single solves."""
import numpy as np
import pytest

from mlfma_pmchwt_b200 import MLFMM, mesh as M, plane_wave

pytestmark = pytest.mark.gpu


def _near_matrix(op):
    sp = pytest.importorskip("scipy.sparse")
    z, N = op.near(), op.N
    t, s = z["target"].astype(np.int64), z["source"].astype(np.int64)
    rows = np.concatenate([t, t, t + N, t + N])
    cols = np.concatenate([s, s + N, s, s + N])
    val = np.concatenate([z["z11"], z["z12"], -z["z12"], z["z22"]])
    return sp.csr_matrix((val, (rows, cols)), shape=(2 * N, 2 * N))


class _Operator:
    """The FP64 apply as the right operand of @."""

    def __init__(self, op):
        self.op = op

    def __matmul__(self, x):
        return self.op.apply_ax(x)


def _gmres(Z, v, its):
    """its GMRES steps on Z z = v from zero; z and sum_j |y_j| |Z q_j|."""
    Q, W = [v / np.linalg.norm(v)], []
    H = np.zeros((its + 1, its), dtype=complex)
    for j in range(its):
        w = Z @ Q[j]
        W.append(np.linalg.norm(w))
        for _ in range(2):
            h = np.array([np.vdot(q, w) for q in Q])
            w = w - sum(c * q for c, q in zip(h, Q))
            H[:j + 1, j] += h
        H[j + 1, j] = np.linalg.norm(w)
        Q.append(w / H[j + 1, j])
    rhs = np.zeros(its + 1, dtype=complex)
    rhs[0] = np.linalg.norm(v)
    y = np.linalg.lstsq(H, rhs, rcond=None)[0]
    return sum(c * q for c, q in zip(y, Q)), float(np.abs(y) @ np.array(W))


@pytest.mark.parametrize("sub,inner", [(1, 1), (1, 7), (2, 8), (2, 9), (3, 16), (2, 33), (2, 63)])
def test_inner_gmres(sub, inner):
    """The residual of the device's z is that of the exact minimiser up to the
    complex64 products: each Z q_j is off by at most ~(ns + 2) eps32 |Z||q|,
    taken as 4e-6 |Z q_j| for the few hundred sources of a row, and enters the
    residual with the weight |y_j|; twice that bound is allowed."""
    torch = pytest.importorskip("torch")
    op = MLFMM(M.ellipsoid(sub, 0.13 * 2 ** sub, 0.11 * 2 ** sub, 0.09 * 2 ** sub), freq=3e8, eps_r=2.5 - 0.1j,
               leaf_coeff=0.25, device=0)
    Z = _near_matrix(op)
    rng = np.random.default_rng(inner)
    v = rng.standard_normal(op.n) + 1j * rng.standard_normal(op.n)
    vd = torch.from_numpy(v).cuda()
    zd = torch.empty_like(vd)
    torch.cuda.synchronize()
    op.near_precondition_device(inner, vd.data_ptr(), zd.data_ptr())
    z = zd.cpu().numpy()
    ref, weight = _gmres(Z, v, inner)
    got, best = np.linalg.norm(v - Z @ z), np.linalg.norm(v - Z @ ref)
    assert abs(got - best) <= 2 * 4e-6 * weight + 1e-12 * np.linalg.norm(v)


@pytest.mark.parametrize("R", [1, 10, 20])
def test_lockstep_rows_per_thread(R):
    """15,360 unknowns: 1 and 10 systems take clusters of two rows per thread, 20
    are 1,200 blocks of one row per thread and take three launches of four. Nine
    steps of GMRES orthonormal
    to rounding agree to ~k eps cond(H), below 1e-9 with cond(H) <= 1e5."""
    op = MLFMM(M.icosphere(4, 1.3), freq=3e8, eps_r=2.5 - 0.1j, leaf_coeff=0.25, device=0, tf_complex_argument=True)
    B = np.stack([op.compute_v_pmchwt(*plane_wave(90.0 * (j % 2), 9.0 * j, 20.0)) for j in range(R)])
    kw = dict(itr_max=9, mr=5, tol_abs=0.0, tol_rel=1e-12)
    X, _ = op.matrix_solver_batch(B, inner_its=0, **kw)
    for j in {0, R // 2, R - 1}:
        x, _ = op.matrix_solver(B[j], inner_its=0, **kw)
        assert np.linalg.norm(X[j] - x) <= 1e-9 * np.linalg.norm(x)


@pytest.mark.parametrize("inner", [12, 13, 33])
def test_inner_gmres_two_rows(inner):
    """As test_inner_gmres with two rows per thread of a cluster: a basis that its
    shared memory holds (12 vectors), and larger ones."""
    test_inner_gmres(4, inner)


def test_inner_gmres_long_vectors():
    """As test_inner_gmres past the clusters' range: three launches per step."""
    test_inner_gmres(5, 9)


def _sphere(sub):
    """15,360 (4) or 61,440 (5) unknowns."""
    return MLFMM(M.icosphere(sub, 1.3 * 2 ** (sub - 4)), freq=3e8, eps_r=2.5 - 0.1j, leaf_coeff=0.25, device=0,
                 tf_complex_argument=True)


def _incidences(op, R):
    return np.stack([op.compute_v_pmchwt(*plane_wave(90.0 * (j % 2), 9.0 * j, 20.0)) for j in range(R)])


@pytest.mark.parametrize("R", [1, 3])
def test_lockstep_long_vectors(R):
    """61,440 unknowns are past the clusters' range: 240 blocks of one row per
    thread, at three systems two rows. Five steps against the same in numpy on
    the operator's own apply, to the bound of test_lockstep_rows_per_thread, and
    the reported residual against the solution's own (two FP64 applies of
    ~1e-15 each)."""
    op = _sphere(5)
    B = _incidences(op, R)
    kw = dict(itr_max=5, mr=5, tol_abs=0.0, tol_rel=1e-12, inner_its=0)
    X, stats = op.matrix_solver_batch(B, **kw)
    for j in range(R):
        want = _gmres(_Operator(op), B[j], 5)[0]
        x, st = op.matrix_solver(B[j], **kw)
        for got, res in ((X[j], stats[j]["rel_residual"]), (x, st["rel_residual"])):
            assert np.linalg.norm(got - want) <= 1e-9 * np.linalg.norm(want)
            own = np.linalg.norm(B[j] - op.apply_ax(got)) / np.linalg.norm(B[j])
            assert abs(own - res) <= 1e-12


@pytest.mark.parametrize("R,its", [(8, 9), (12, 17)])
def test_lockstep_basis_beyond_the_clusters_memory(R, its):
    """15,360 unknowns, 8 systems and more: a cluster's shared memory holds 5
    vectors of the basis, the others come from global memory. As
    test_lockstep_long_vectors, for the first and last system."""
    op = _sphere(4)
    B = _incidences(op, R)
    X, _ = op.matrix_solver_batch(B, itr_max=its, mr=its, tol_abs=0.0, tol_rel=1e-12, inner_its=0)
    for j in (0, R - 1):
        want = _gmres(_Operator(op), B[j], its)[0]
        assert np.linalg.norm(X[j] - want) <= 1e-9 * np.linalg.norm(want)


@pytest.mark.parametrize("sub,R", [(4, 8), (4, 14), (4, 20), (5, 3)])
def test_lockstep_inner_steps(sub, R):
    """Three outer steps preconditioned by nine inner ones: clusters whose memory
    holds 5 of the 9 vectors (8 systems), and three launches of two (14), four
    (20) and, on 61,440 unknowns, two rows per thread. Against numpy with the
    FP64 near field: the 27 complex64 products are off by 4e-6 each
    (test_inner_gmres), at a condition of ten at most 1e-3 of the solution."""
    op = _sphere(sub)
    B = _incidences(op, R)
    X, _ = op.matrix_solver_batch(B, itr_max=3, mr=3, tol_abs=0.0, tol_rel=1e-12, inner_its=9)
    Z = _near_matrix(op)
    for j in (0, R - 1):
        V, D, H = [B[j] / np.linalg.norm(B[j])], [], np.zeros((4, 3), dtype=complex)
        for k in range(3):
            D.append(_gmres(Z, V[k], 9)[0])
            w = op.apply_ax(D[k])
            for _ in range(2):
                h = np.array([np.vdot(q, w) for q in V])
                w = w - sum(c * q for c, q in zip(h, V))
                H[:k + 1, k] += h
            H[k + 1, k] = np.linalg.norm(w)
            V.append(w / H[k + 1, k])
        y = np.linalg.lstsq(H, np.linalg.norm(B[j]) * np.eye(4)[0], rcond=None)[0]
        want = sum(c * d for c, d in zip(y, D))
        assert np.linalg.norm(X[j] - want) <= 1e-3 * np.linalg.norm(want)
