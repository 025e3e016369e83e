"""The bistatic far-field kernel at the ends of its tiles (4 angles, pairs and
32 solutions, 256 RWGs or 64, 8 slices, 512 angles per launch) and for triangles
wider than its phase series covers, against the single-solution entry point;
both batched far fields with every triangle rule on a body off the origin."""
import dataclasses

import numpy as np
import pytest

from mlfma_pmchwt_b200 import MLFMM, mesh as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sub,radius,R,angles", [(2, 0.5, 1, 1), (2, 0.5, 2, 3), (3, 1.0, 3, 5), (1, 0.6, 5, 8),
                                                 (4, 1.2, 32, 4), (2, 0.5, 33, 7), (2, 0.5, 66, 513)])
def test_far_field_tiles(sub, radius, R, angles):
    """Sums of 2N products of order one in a different order: 1e-12 of the
    largest field, as the other far-field comparisons."""
    torch = pytest.importorskip("torch")
    op = MLFMM(M.icosphere(sub, radius), freq=3e8, eps_r=2.5, leaf_coeff=0.25, device=0)
    g = np.random.default_rng(R)
    I = g.standard_normal((R, op.n)) + 1j * g.standard_normal((R, op.n))
    th, ph = g.uniform(0, 180, angles), g.uniform(0, 360, angles)
    th[0] = 0.0
    Id = torch.from_numpy(I).cuda()
    F = torch.full((R, angles, 3), float("nan"), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    op.calculate_rcs_batch_device(R, Id.data_ptr(), th, ph, F.data_ptr())
    torch.cuda.synchronize()
    got = F.cpu().numpy()
    for r in {0, R // 2, R - 1}:
        want, _ = op.calculate_rcs_pmchwt(I[r], th, ph)
        np.testing.assert_allclose(got[r], want, rtol=0, atol=1e-12 * np.abs(want).max())


@pytest.mark.parametrize("rule", [1, 3, 4, 6, 7, 12, 13, 16])
def test_far_field_rules(rule):
    """A body 20 wavelengths from the origin: phases of up to 130 rad, each
    rounded to ~4 eps of that (1.2e-13), RWG vectors of a tenth of a
    wavelength as differences of positions (3e-14): 1e-12 of the largest field.
    Coordinates of a point that miss 1 by 1e-12 (the centroid of the rules of 1
    and 4 points) must not move the points: that is 1e-10 here."""
    torch = pytest.importorskip("torch")
    m = M.icosphere(2, 0.5)
    m = dataclasses.replace(m, points=m.points + np.array([12.0, -12.0, 11.0]))
    op = MLFMM(m, freq=3e8, eps_r=2.5, leaf_coeff=0.25, gauss_points=rule, device=0)
    g = np.random.default_rng(rule)
    I = g.standard_normal((3, op.n)) + 1j * g.standard_normal((3, op.n))
    th, ph = g.uniform(0, 180, 3), g.uniform(0, 360, 3)
    Id = torch.from_numpy(I).cuda()
    F = torch.full((3, 3, 3), float("nan"), dtype=torch.complex128, device="cuda")
    Fm = torch.full((3, 3), float("nan"), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    op.calculate_rcs_batch_device(3, Id.data_ptr(), th, ph, F.data_ptr())
    op.calculate_rcs_mono_device(3, Id.data_ptr(), th, ph, Fm.data_ptr())
    torch.cuda.synchronize()
    got, mono = F.cpu().numpy(), Fm.cpu().numpy()
    for r in range(3):
        want, _ = op.calculate_rcs_pmchwt(I[r], th, ph)
        np.testing.assert_allclose(got[r], want, rtol=0, atol=1e-12 * np.abs(want).max())
        np.testing.assert_allclose(mono[r], want[r], rtol=0, atol=1e-12 * np.abs(want).max())


@pytest.mark.parametrize("sub", [1, 2, 3])
def test_far_field_of_a_solution_alone_and_among_others(sub):
    """A solution's field has the same bits whatever number of solutions and
    angles share the call (the kernels split their sums by both; few solutions
    of many angles or of a small body take a kernel of their own)."""
    torch = pytest.importorskip("torch")
    op = MLFMM(M.icosphere(sub, 0.125 * 2 ** sub), freq=3e8, eps_r=2.5, leaf_coeff=0.25, device=0)
    g = np.random.default_rng(5)
    I = torch.from_numpy(g.standard_normal((33, op.n)) + 1j * g.standard_normal((33, op.n))).cuda()
    th, ph = g.uniform(0, 180, 150), g.uniform(0, 360, 150)

    def field(lo, hi, n):
        F = torch.full((hi - lo, n, 3), float("nan"), dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        op.calculate_rcs_batch_device(hi - lo, I[lo:hi].data_ptr(), th[:n], ph[:n], F.data_ptr())
        torch.cuda.synchronize()
        return F.cpu().numpy()

    every = field(0, 33, 150)
    for r in (0, 1, 32):
        np.testing.assert_array_equal(field(r, r + 1, 150)[0], every[r])
        np.testing.assert_array_equal(field(r, r + 1, 3)[0], every[r, :3])
    for R in (2, 3, 4, 5, 7, 8, 9, 16, 17, 32):
        np.testing.assert_array_equal(field(0, R, 150), every[:R])
        np.testing.assert_array_equal(field(0, R, 9), every[:R, :9])
