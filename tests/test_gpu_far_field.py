"""The bistatic far-field kernel at the ends of its tiles (4 angles, pairs and
32 solutions, 256 RWGs, 8 slices, 512 angles per launch) and for triangles
wider than its phase series covers, against the single-solution entry point."""
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
