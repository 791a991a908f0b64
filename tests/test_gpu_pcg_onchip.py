"""The one-kernel PCG of small systems against the graph of sweeps and the
oracle, bit for bit, where its split can go wrong: fewer rows than a warp, the
edges of a 128-row unit and a 1024-row tile, more units than SMs, rows of
uneven length (with and without row patterns), row lengths that leave the
matrix to the graph, iteration caps and every start vector."""
import numpy as np
import pytest

from cel_v3_b200 import synth
from oracle import celref as R
from tests.helpers import random_csr, spd_from_pattern

pytestmark = pytest.mark.gpu


def grid(nx, ny, nz):
    _, k = synth.lognormal_faces(np.random.default_rng(nx), nx, ny, nz)
    return synth.diffusion7(nx, ny, nz, *k)


def rand(n, **kw):
    return spd_from_pattern(*random_csr(n, np.random.default_rng(n), **kw))


def wide_band(n):
    """Symmetric, diagonally dominant, 1 to 5 entries a row, no row patterns."""
    i = np.arange(n - 700)
    i = i[np.random.default_rng(1).random(i.size) < 0.8]
    j = i + 1 + (i * 2654435761) % 600
    u = 0.5 + np.random.default_rng(2).random(i.size)
    import scipy.sparse as sp
    A = sp.coo_matrix((u, (i, j)), shape=(n, n))
    A = A + A.T
    A = (sp.diags(np.asarray(A.sum(axis=1)).ravel() + 0.1) - A).tocsr()
    A.sort_indices()
    return A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data


CASES = {
    "one_row": lambda: grid(1, 1, 1),
    "31_rows": lambda: grid(31, 1, 1),
    "129_rows": lambda: grid(43, 3, 1),
    "one_tile": lambda: grid(16, 8, 8),
    "tile_and_a_row": lambda: grid(41, 25, 1),
    "values_partly_cached": lambda: grid(75, 70, 64),
    "wide_few_tiles": lambda: grid(95, 90, 89),
    "wide_ragged": lambda: grid(113, 112, 111),
    "wide_most_tiles": lambda: grid(128, 128, 128),
    "wide_uneven_rows": lambda: wide_band(760003),
    "too_many_rows": lambda: grid(131, 129, 127),
    "uneven_rows": lambda: rand(1023, max_len=9),
    "uneven_rows_many_units": lambda: rand(20011, max_len=12),
    "some_long_rows": lambda: rand(4099, max_len=5, long_rows=40, long_len=300),
    "rows_too_long_to_slice": lambda: rand(2049, max_len=3, long_rows=2, long_len=1500),
}


def solve(celgpu, h, torch, m, b, x0, **kw):
    x = torch.from_numpy(x0.copy()).cuda()
    i = h.pcg_jacobi(m, b.data_ptr(), x.data_ptr(), history=True, **kw)
    torch.cuda.synchronize()
    return x.cpu().numpy(), i


@pytest.mark.parametrize("name", sorted(CASES))
def test_onchip_equals_graph_and_oracle(gpu, name, monkeypatch):
    celgpu, h, torch = gpu
    rp, ci, v = CASES[name]()
    n = rp.size - 1
    rng = np.random.default_rng(7)
    b, x0 = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    bd = torch.from_numpy(b).cuda()
    m = h.matrix_from_csr(rp, ci, v).jacobi()
    cap = 2000 if n < 500000 else 25
    runs = [dict(x0_mode=celgpu.X0_ZERO, eps_rel=1e-9, iter_max=cap), dict(x0_mode=celgpu.X0_USER, iter_max=3),
            dict(x0_mode=celgpu.X0_REF_ONES, eps_rel=0.0, eps_abs=1e-3, iter_max=cap), dict(iter_max=0)]
    if n < 5000:
        runs.append(dict(precision=celgpu.PREC_FP32_IR, eps_rel=1e-9, inner_eps_rel=1e-3))
    for kw in runs:
        monkeypatch.setenv("CELG_ONCHIP_ROWS", "0")
        xg, ig = solve(celgpu, h, torch, m, bd, x0, **kw)
        monkeypatch.delenv("CELG_ONCHIP_ROWS")
        for _ in range(2):
            xo, io = solve(celgpu, h, torch, m, bd, x0, **kw)
            assert np.array_equal(xg, xo) and np.array_equal(ig.history, io.history)
            for f in ("iter_done", "status", "final_norm2", "bnorm", "verified_relres", "arnoldi_steps"):
                assert io[f] == ig[f], f
    xr, ir = R.pcg_jacobi(R.Matrix(rp, ci, v), R.jacobi(R.diag(rp, ci, v)), b, eps_rel=1e-9, iter_max=cap,
                          red=R.RED_TREE)
    x, i = solve(celgpu, h, torch, m, bd, x0, **runs[0])
    assert i.iter_done == ir["iter_done"] and np.array_equal(x, xr)
    m.destroy()


def test_onchip_scaled_matrix_and_breakdown(gpu, monkeypatch):
    """Scaling after a solve rewrites the values the kernel keeps a copy of;
    solves that end before their first step end alike on both paths."""
    celgpu, h, torch = gpu
    rp, ci, v = grid(13, 11, 9)
    n = rp.size - 1
    b = np.random.default_rng(1).uniform(-1, 1, n)
    bd = torch.from_numpy(b).cuda()
    m = h.matrix_from_csr(rp, ci, v).jacobi()
    solve(celgpu, h, torch, m, bd, np.zeros(n), iter_max=500)
    m.scale_diagonal()
    x, i = solve(celgpu, h, torch, m, bd, np.zeros(n), iter_max=500)
    fresh = h.matrix_from_csr(rp, ci, v).jacobi().scale_diagonal()
    y, j = solve(celgpu, h, torch, fresh, bd, np.zeros(n), iter_max=500)
    assert i.iter_done == j.iter_done and np.array_equal(x, y)
    m.destroy()
    fresh.destroy()
    # alpha = r.Jr = 0 stops both paths before the first step; A p = 0 breaks down
    for vals, status in (([1.0, 0.0, 0.0, -1.0], celgpu.OK), ([1.0, -1.0, -1.0, 1.0], celgpu.ERR_BREAKDOWN)):
        two = h.matrix_from_csr(np.array([0, 2, 4], np.int32), np.array([0, 1, 0, 1], np.int32),
                                np.array(vals)).jacobi()
        ones = torch.ones(2, dtype=torch.float64).cuda()
        x, i = solve(celgpu, h, torch, two, ones, np.zeros(2), iter_max=10)
        monkeypatch.setenv("CELG_ONCHIP_ROWS", "0")
        y, j = solve(celgpu, h, torch, two, ones, np.zeros(2), iter_max=10)
        monkeypatch.delenv("CELG_ONCHIP_ROWS")
        assert i.status == j.status == status and i.iter_done == j.iter_done == 0
        assert np.all(x == 0.0) and np.all(y == 0.0)
        two.destroy()
