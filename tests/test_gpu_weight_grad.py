"""The weight-gradient kernel of the learned preconditioner where its row
split changes: fewer rows than one CTA's two tiles, ragged ends, and so many
rows that a CTA takes more than two tiles. Against the float64 oracle with the
tolerances of the other gradient tests (FP32 sums)."""
import numpy as np
import pytest

from conftest import FREQ, needs_lib, rel
from learned_util import oracle_graph

pytestmark = [pytest.mark.gpu, needs_lib]


@pytest.mark.parametrize("sub,axes", [(1, (0.5, 0.4, 0.3)), (2, (0.6, 0.5, 0.4)), (5, (2.0, 1.6, 1.2))])
def test_weight_gradient_row_splits(sub, axes):
    import torch
    from mlfma_pmchwt_b200 import MLFMM, mesh as M
    from oracle import learned_precond as LP
    m, eps = M.ellipsoid(sub, *axes), 3.0 - 0.1j
    op = MLFMM(m, freq=FREQ, eps_r=eps, leaf_coeff=0.25, device=0)
    rng = np.random.default_rng(sub)
    c = lambda: rng.normal(size=op.n) + 1j * rng.normal(size=op.n)
    v, z, e = c(), c(), c()
    th = (LP.init_params(sub) + 0.05 * rng.normal(size=LP.param_count())).astype(np.float32)
    V, Z, E, T = (torch.from_numpy(a).cuda() for a in (v, z, e, th))
    Y, G = torch.empty_like(V), torch.zeros_like(T)
    L = torch.zeros(1, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    op.lp_loss_grad_device(T.data_ptr(), V.data_ptr(), Z.data_ptr(), E.data_ptr(), Y.data_ptr(), G.data_ptr(),
                           L.data_ptr())
    torch.cuda.synchronize()
    _, want, _ = LP.loss_grad(th, oracle_graph(op, m, eps), v, z, e)
    assert rel(G.cpu().numpy().astype(np.float64), want) < 1e-4
