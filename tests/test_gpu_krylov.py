"""The Krylov solvers' vector kernels at the sizes where their tiles end: the
preconditioner's inner GMRES against the same iteration in numpy (basis sizes
around the 8-vector tile and the 32- and 64-column solve), and lockstep sets
of 1, 2 and 4 rows per thread against single solves."""
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
    """15,360 unknowns are 60 blocks of one row per thread: 1, 10 and 20
    systems take 1, 2 and 4 rows per thread. Nine steps of GMRES orthonormal
    to rounding agree to ~k eps cond(H), below 1e-9 with cond(H) <= 1e5."""
    op = MLFMM(M.icosphere(4, 1.3), freq=3e8, eps_r=2.5 - 0.1j, leaf_coeff=0.25, device=0, tf_complex_argument=True)
    B = np.stack([op.compute_v_pmchwt(*plane_wave(90.0 * (j % 2), 9.0 * j, 20.0)) for j in range(R)])
    kw = dict(itr_max=9, mr=5, tol_abs=0.0, tol_rel=1e-12)
    X, _ = op.matrix_solver_batch(B, inner_its=0, **kw)
    for j in {0, R // 2, R - 1}:
        x, _ = op.matrix_solver(B[j], inner_its=0, **kw)
        assert np.linalg.norm(X[j] - x) <= 1e-9 * np.linalg.norm(x)


def test_inner_gmres_two_rows():
    """As test_inner_gmres with two rows per thread of a cluster and a basis
    larger than its shared memory (5 vectors)."""
    test_inner_gmres(4, 12)


@pytest.mark.parametrize("R", [1, 3])
def test_lockstep_long_vectors(R):
    """61,440 unknowns are past the clusters' range: 240 blocks of one row per
    thread, at three systems two rows. The bound of test_lockstep_rows_per_thread;
    one system against its own residual, which GMRES reports."""
    op = MLFMM(M.icosphere(5, 2.6), freq=3e8, eps_r=2.5 - 0.1j, leaf_coeff=0.25, device=0, tf_complex_argument=True)
    B = np.stack([op.compute_v_pmchwt(*plane_wave(90.0 * (j % 2), 9.0 * j, 20.0)) for j in range(R)])
    kw = dict(itr_max=5, mr=5, tol_abs=0.0, tol_rel=1e-12)
    X, _ = op.matrix_solver_batch(B, inner_its=0, **kw)
    for j in range(R):
        x, res = op.matrix_solver(B[j], inner_its=0, **kw)
        assert np.linalg.norm(X[j] - x) <= 1e-9 * np.linalg.norm(x)
        assert np.linalg.norm(B[j] - op.apply_ax(x)) < np.linalg.norm(B[j])
