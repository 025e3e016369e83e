"""The near-field products of the preconditioner and of the public entry
point against the read-out entries in numpy, at row and source counts around
the kernels' tiles (a box of a few RWGs to hundreds, lists of sources longer
than the piece that the box kernel stages at a time), and the lockstep
product for 1 to 9 systems through one inner step."""
import numpy as np
import pytest

from mlfma_pmchwt_b200 import MLFMM, mesh as M

pytestmark = pytest.mark.gpu

BODIES = {"few": (2, 0.9, 0.12), "ordinary": (3, 1.0, 0.25), "crowded": (4, 0.8, 0.4), "one list": (2, 0.2, 0.3)}


def _near(op, x):
    z, N = op.near(), op.N
    t, s = z["target"], z["source"]
    J, Mc = x[:N][s], x[N:][s]
    w = np.zeros(2 * N, dtype=complex)
    np.add.at(w, t, z["z11"] * J + z["z12"] * Mc)
    np.add.at(w, t + N, z["z22"] * Mc - z["z12"] * J)
    mag = np.zeros(2 * N)
    np.add.at(mag, t, abs(z["z11"] * J) + abs(z["z12"] * Mc))
    np.add.at(mag, t + N, abs(z["z22"] * Mc) + abs(z["z12"] * J))
    return w, mag, int(np.bincount(t).max())


@pytest.mark.parametrize("body", BODIES)
def test_near_product(body):
    """FP64: a row's error is below (2 ns + 4) eps of the sum of its terms' magnitudes."""
    sub, radius, leaf = BODIES[body]
    _check_near(MLFMM(M.ellipsoid(sub, radius, 0.9 * radius, 0.8 * radius), freq=3e8, eps_r=2.5 - 0.1j, leaf_coeff=leaf,
                      device=0))


def _check_near(op):
    torch = pytest.importorskip("torch")
    g = np.random.default_rng(1)
    x = g.standard_normal(op.n) + 1j * g.standard_normal(op.n)
    want, mag, ns = _near(op, x)
    xd = torch.from_numpy(x).cuda()
    wd = torch.full_like(xd, float("nan"))
    torch.cuda.synchronize()
    op.apply_near_device(xd.data_ptr(), wd.data_ptr())
    torch.cuda.synchronize()
    assert np.all(np.abs(wd.cpu().numpy() - want) <= (2 * ns + 4) * 2.3e-16 * mag)


@pytest.mark.parametrize("body", BODIES)
@pytest.mark.parametrize("R", [1, 2, 3, 4, 5, 8, 9])
def test_lockstep_near_product(body, R):
    """One outer step with two inner steps: z, and so x, lies in span{b, Z b} of
    the FP64 entries up to the rounding of the first product.
    Complex64: a row is off by at most (2 ns + 4) eps32 of
    its terms' magnitudes."""
    sub, radius, leaf = BODIES[body]
    op = MLFMM(M.ellipsoid(sub, radius, 0.9 * radius, 0.8 * radius), freq=3e8, eps_r=2.5 - 0.1j, leaf_coeff=leaf,
               device=0)
    g = np.random.default_rng(R)
    B = g.standard_normal((R, op.n)) + 1j * g.standard_normal((R, op.n))
    X, _ = op.matrix_solver_batch(B, itr_max=1, mr=1, tol_abs=0.0, tol_rel=1e-14, inner_its=2)
    one = [op.matrix_solver(B[j], itr_max=1, mr=1, tol_abs=0.0, tol_rel=1e-14, inner_its=2)[0] for j in range(R)]
    for j in range(R):
        _, mag, ns = _near(op, B[j] / np.linalg.norm(B[j]))
        want, _, _ = _near(op, B[j] / np.linalg.norm(B[j]))
        # x is in span{b, Z b}: its components outside are the products' rounding
        Q, _ = np.linalg.qr(np.stack([B[j], want], axis=1))
        for x in (X[j], one[j]):
            off = np.linalg.norm(x - Q @ (Q.conj().T @ x)) / np.linalg.norm(x)
            assert off <= 2 * (2 * ns + 4) * 6e-8 * np.linalg.norm(mag) / np.linalg.norm(want)


def _long_lists(precision):
    """Lists of up to 3,718 sources: three pieces of the shared memory that the
    box kernel stages them in (1,536 in FP64, 3,072 in complex64: two)."""
    op = MLFMM(M.ellipsoid(4, 0.7, 0.63, 0.56), freq=3e8, eps_r=2.5 - 0.1j, leaf_coeff=0.4, device=0,
               precision=precision)
    assert 3 * 1536 > int(np.bincount(op.near(values=False)["target"]).max()) > 3072
    return op


def test_near_product_of_long_lists():
    """As test_near_product."""
    _check_near(_long_lists("fp64"))


def test_complex64_near_product_of_long_lists():
    """The complex64 operator's near rows against the FP64 operator: a lane's ~120
    terms are off by a few 6e-8 of their size each: 1e-5, as the other
    comparisons of the two operators."""
    op = _long_lists("mixed")
    x = M.unit_disk_vector(op.n, 2)
    w = op.apply_ax(x)
    assert np.linalg.norm(op.apply_ax_mixed(x) - w) <= 1e-5 * np.linalg.norm(w)


@pytest.mark.parametrize("sub,radius,leaf", [(3, 1.0, 0.1), (4, 1.3, 0.4)])
def test_near_product_by_rows(sub, radius, leaf):
    """As test_near_product where a warp takes each row: a thousand boxes of two
    RWGs, and 226 MB of entries."""
    op = MLFMM(M.icosphere(sub, radius), freq=3e8, eps_r=2.5 - 0.1j, leaf_coeff=leaf, device=0)
    boxes = len(op.leaf_rwgs()[0]) - 1
    assert boxes > 592 and op.N < 3 * boxes or 48 * op.info.near_pairs > 2e8
    _check_near(op)


def test_complex64_near_product_by_rows():
    """As test_complex64_near_product_of_long_lists on boxes of two RWGs."""
    op = MLFMM(M.icosphere(3, 1.0), freq=3e8, eps_r=2.5 - 0.1j, leaf_coeff=0.1, device=0, precision="mixed")
    assert len(op.leaf_rwgs()[0]) - 1 > 592
    x = M.unit_disk_vector(op.n, 2)
    w = op.apply_ax(x)
    assert np.linalg.norm(op.apply_ax_mixed(x) - w) <= 1e-5 * np.linalg.norm(w)
