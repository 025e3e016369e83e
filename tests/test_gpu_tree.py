"""The tree passes level by level against the same sums in numpy, on the stage
arrays and tables an operator reads out: interpolation by pairs of parent
rows, translation by box pairs, anterpolation by pairs of child rows. Grids
of odd and even theta counts, a lossy body, grids so fine that an
anterpolation band holds a single child row, and launches of few and of many
warps (the translation shares a pair's list among its warps below 740)."""
import numpy as np
import pytest

from mlfma_pmchwt_b200 import MLFMM, mesh as M

pytestmark = pytest.mark.gpu

BODIES = {"deep": lambda: dict(mesh=M.ellipsoid(3, 1.0, 0.8, 0.7), eps_r=2.5 - 0.1j, leaf_coeff=0.12),
          "shallow": lambda: dict(mesh=M.icosphere(3, 1.0), eps_r=4.0, leaf_coeff=0.25),
          "split lists": lambda: dict(mesh=M.ellipsoid(2, 0.7, 0.6, 0.5), eps_r=4.0, leaf_coeff=0.2),
          "fine grids": lambda: dict(mesh=M.icosphere(1, 1.0), eps_r=360.0, leaf_coeff=0.25)}


def _close(got, want):
    """Sums of a few hundred products: 1e-12 of the array's largest value."""
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("body", BODIES)
def test_tree_levels(body):
    op = MLFMM(freq=3e8, device=0, **BODIES[body]())
    assert op.max_level > 2
    x = M.unit_disk_vector(op.n, 3)
    op.apply_ax(x)
    odd, single = set(), False
    for m, k in ((1, op.k1), (2, op.k2)):
        S = {l: op.stage("S", m, l) for l in op.levels()}
        B = {l: op.stage("B", m, l) for l in op.levels()}
        mats = {}
        for l in range(op.max_level - 1, 1, -1):  # parent l, child l + 1
            g, gc, q = op.grid(m, l), op.grid(m, l + 1), op.interp(m, l)
            odd.add(g["L"] % 2)
            single = single or 2944 // (6 * 2 * g["L"]) <= 1
            T, F = np.zeros((g["L"], gc["L"])), np.zeros((2 * g["L"], 2 * gc["L"]))
            for i in range(3):
                np.add.at(T, (np.arange(len(T)), q["tidx"][:, i]), q["lt"][:, i])
                np.add.at(F, (np.arange(len(F)), q["pidx"][:, i]), q["lp"][:, i])
            th, ph = np.meshgrid(g["theta"], g["phi"], indexing="ij")
            kh = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)]).reshape(3, -1)
            (cp, xp), (cc, xc) = op.level(l), op.level(l + 1)
            at = {int(c): i for i, c in enumerate(cp)}
            par = np.array([at[int(c) >> 3] for c in cc])
            up = np.exp(-1j * k * ((xp[par] - xc) @ kh))
            dn = np.exp(-1j * k * ((xc - xp[par]) @ kh))
            c = S[l + 1].reshape(len(cc), 6, gc["L"], 2 * gc["L"])
            want = np.zeros_like(S[l])
            np.add.at(want, par, (T @ c @ F.T).reshape(len(cc), 6, -1) * up[:, None])
            _close(S[l], want)
            mats[l] = (T, F, dn, par)
        for l in op.levels():
            g, lst = op.grid(m, l), op.level_lists(l)
            tf, off = op.transfer(m, l)
            tf = tf * (np.repeat(g["wtheta"], 2 * g["L"]) * g["wphi"])
            row = {(int(a) + 3) * 49 + (int(b) + 3) * 7 + int(c) + 3: i for i, (a, b, c) in enumerate(off)}
            want = np.zeros_like(B[l])
            for b in range(len(want)):
                for e in range(lst["far_ptr"][b], lst["far_ptr"][b + 1]):
                    want[b] += tf[row[int(lst["far_off"][e])]] * S[l][lst["far_idx"][e]]
            if l > 2:
                T, F, dn, par = mats[l - 1]
                p = (B[l - 1][par] * dn[:, None]).reshape(len(par), 6, T.shape[0], F.shape[0])
                want += (T.T @ p @ F).reshape(want.shape)
            _close(B[l], want)
    assert odd == {0, 1} or body != "deep"
    assert single or body != "fine grids"


@pytest.mark.parametrize("body", BODIES)
def test_profiled_apply_has_the_same_bits(body):
    """Stage timing runs one stage after another, with the same launches: the
    translation's sums follow the number of warps of a launch."""
    op = MLFMM(freq=3e8, device=0, **BODIES[body]())
    x = M.unit_disk_vector(op.n, 4)
    plain = op.apply_ax(x)
    op.profile(True)
    timed = op.apply_ax(x)
    assert op.stage_times()[1] == 1
    op.profile(False)
    np.testing.assert_array_equal(timed, plain)


@pytest.mark.parametrize("R", [1, 3])
def test_batched_large_tree(R):
    """Trees above 116 MB per right-hand side run slot after slot. Rows against
    the FP64 operator: an entry is a sum of ~1e4 complex64 products taken in
    chunks, each entry rounded to 6e-8, so 1e-6 of the row's norm is allowed."""
    torch = pytest.importorskip("torch")
    op = MLFMM(M.icosphere(5, 2.5), freq=3e8, eps_r=4.0, leaf_coeff=0.25, device=0, precision="mixed")
    levels = op.max_level - 1
    assert sum(op.info.boxes[l] * 96 * (op.info.K_k1[l] + op.info.K_k2[l]) for l in range(levels)) > 116 << 20
    X = torch.from_numpy(np.stack([M.unit_disk_vector(op.n, 40 + j) for j in range(R)])).cuda()
    W = torch.full_like(X, float("nan"))
    torch.cuda.synchronize()
    op.apply_batch_mixed_device(R, X.data_ptr(), W.data_ptr())
    torch.cuda.synchronize()
    for x, w in zip(X.cpu().numpy(), W.cpu().numpy()):
        ref = op.apply_ax(x)
        assert np.linalg.norm(w - ref) <= 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("sub,radius,default", [(3, 1.0, 1), (5, 2.5, 0)])
def test_batch_tree_variant_selects_the_passes(sub, radius, default):
    """batch_tree.variant starts with the size's choice, and each value runs
    what it names at every size: one anterpolation launch per level pair and
    medium, for each of the three rows (0) or once for all (1)."""
    torch = pytest.importorskip("torch")
    from torch.profiler import ProfilerActivity, profile
    op = MLFMM(M.icosphere(sub, radius), freq=3e8, eps_r=4.0, leaf_coeff=0.25, device=0, precision="mixed")
    assert op.get_tuning("batch_tree.variant") == default
    X = torch.from_numpy(np.stack([M.unit_disk_vector(op.n, 40 + j) for j in range(3)])).cuda()
    rows = []
    for v in (0, 1):
        op.set_tuning("batch_tree.variant", v)
        assert op.get_tuning("batch_tree.variant") == v
        W = torch.full_like(X, float("nan"))
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            op.apply_batch_mixed_device(3, X.data_ptr(), W.data_ptr())
            torch.cuda.synchronize()
        names = [e.name for e in p.events()]
        if not any("_kernel" in n for n in names):
            pytest.skip("no kernel records on this machine")
        launches = sum("l2l_sep_kernel" in n for n in names)
        assert launches == 2 * (op.max_level - 2) * (1 if v else 3)
        rows.append(W.cpu().numpy())
    np.testing.assert_allclose(rows[1], rows[0], rtol=0, atol=1e-12 * np.abs(rows[0]).max())


def test_batched_apply_reserves_what_its_passes_use():
    """A first batched apply slot after slot takes the leaf level's arrays of 16
    slots; selecting the passes over all slots takes those of the levels above,
    at once, and no more later. 128 MB beside that for the right-hand sides,
    the heap's chunk and the loading of kernels."""
    torch = pytest.importorskip("torch")
    op = MLFMM(M.icosphere(5, 2.5), freq=3e8, eps_r=4.0, leaf_coeff=0.25, device=0, precision="mixed")
    level = [16 * 96 * op.info.boxes[l] * (op.info.K_k1[l] + op.info.K_k2[l]) for l in range(op.max_level - 1)]
    leaf, upper = level[-1], sum(level[:-1])
    assert op.get_tuning("batch_tree.variant") == 0 and upper > 1 << 30
    X = torch.from_numpy(np.stack([M.unit_disk_vector(op.n, j) for j in range(2)])).cuda()
    W = torch.empty_like(X)
    torch.cuda.synchronize()
    free = [torch.cuda.mem_get_info()[0]]

    def step(what):
        what()
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
        return free[-2] - free[-1]

    run = lambda: op.apply_batch_mixed_device(2, X.data_ptr(), W.data_ptr())
    assert leaf <= step(run) <= leaf + (128 << 20)
    assert upper <= step(lambda: op.set_tuning("batch_tree.variant", 1)) <= upper + (128 << 20)
    assert step(run) <= 128 << 20
    assert step(lambda: [op.set_tuning("batch_tree.variant", v) for v in (0, 1)]) == 0
