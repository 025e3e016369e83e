"""The GPU path against the committed golden fixtures (outputs of the reference
compiled from its sources, tests/golden/make_golden.py), which need no
reference sources: matvec, excitation, GMRES history and RCS of two spheres."""
import numpy as np
import pytest

from conftest import FREQ, ROOT, needs_lib, rel

pytestmark = [pytest.mark.gpu, needs_lib]


@pytest.mark.parametrize("name", ["sphere_s2", "sphere_s3"])
def test_reference_outputs(name):
    """The bounds of the parity suite: matvec 1e-10, excitation 1e-12, GMRES
    history 1e-5 per entry, RCS 0.01 dB."""
    from mlfma_pmchwt_b200 import MLFMM, plane_wave
    from mlfma_pmchwt_b200 import mesh as M
    g = dict(np.load(ROOT / "tests" / "golden" / f"{name}.npz"))
    op = MLFMM(M.icosphere(int(g["sub"]), float(g["radius"])), freq=FREQ, eps_r=complex(g["eps_r"]),
               leaf_coeff=float(g["leaf"]), device=0)
    assert op.N == int(g["N"]) and op.max_level == int(g["max_level"])
    assert rel(op.apply_ax(g["x"]), g["w"]) < 1e-10
    V = op.compute_v_pmchwt(*plane_wave(0.0, 0.0, 0.0))
    assert rel(V, g["V"]) < 1e-12
    _, st = op.matrix_solver(g["V"], itr_max=60, mr=30, tol_abs=1e-8, tol_rel=1e-6)
    np.testing.assert_allclose(st["history"], g["gmres_history"], rtol=1e-5)
    _, db = op.calculate_rcs_pmchwt(g["gmres_x"], g["rcs_theta"], np.zeros_like(g["rcs_theta"]))
    np.testing.assert_allclose(db, g["rcs_db"], rtol=0, atol=0.01)
    op.close()
