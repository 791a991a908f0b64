"""Bytes per iteration that celg_elm_performance reports, for every form a
matrix is read in, against the arrays that the iteration's kernels touch."""
import numpy as np
import pytest

from cel_v3_b200 import synth
from tests.helpers import random_csr, spd_from_pattern

pytestmark = pytest.mark.gpu


def poisson():  # row table, one Jacobi value
    return synth.poisson7(16, 15, 14)


def diffusion():  # row patterns
    _, k = synth.lognormal_faces(np.random.default_rng(1), 16, 15, 14, 0.5)
    return synth.diffusion7(16, 15, 14, *k)


def offsets():  # rows of 11 entries: 1-byte offsets
    import scipy.sparse as sp
    off = list(range(-5, 6))
    A = sp.diags([np.full(3000 - abs(o), -0.5 if o else 8.0) for o in off], off).tocsr()
    A.sort_indices()
    return A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data


def columns():  # int32 columns
    return spd_from_pattern(*random_csr(3000, np.random.default_rng(3), max_len=9))


def stored(n, nnz, vt):
    return {"poisson": n, "diffusion": vt * nnz + n + 4 * (n + 1), "offsets": (vt + 1) * nnz + 4 * (n + 1),
            "columns": (vt + 4) * nnz + 4 * (n + 1)}


@pytest.mark.parametrize("kind", [poisson, diffusion, offsets, columns])
def test_reported_bytes(gpu, kind, monkeypatch):
    celgpu, h, torch = gpu
    rp, ci, v = kind()
    n, nnz, name = rp.size - 1, int(rp[-1]), kind.__name__
    m = h.matrix_from_csr(rp, ci, v).jacobi()
    b = torch.ones(n, 8, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    kw = dict(eps_rel=1e-6, iter_max=50, x0_mode=celgpu.X0_ZERO, inner_eps_rel=1e-2)
    uni = name == "poisson"

    def single(**k):
        h.pcg_jacobi(m, b.data_ptr(), x.data_ptr(), **kw, **k)
        return h.elm_performance()[2]

    monkeypatch.setenv("CELG_ONCHIP_ROWS", "0")
    assert single() == stored(n, nnz, 8)[name] + (92 - 16 * uni) * n
    for prec in (celgpu.PREC_FP32_RU, celgpu.PREC_FP32_IR):
        assert single(precision=prec) == stored(n, nnz, 4)[name] + (46 - 8 * uni) * n
    monkeypatch.delenv("CELG_ONCHIP_ROWS")
    # in one kernel: p, and what of the matrix does not stay on chip
    assert single() == 16 * n + (0 if name in ("poisson", "diffusion") else 12 * nnz)
    m.to_jad()
    jad = stored(n, nnz, 8)["diffusion" if uni else name]
    assert single(fmt=celgpu.FMT_JAD) == jad + 96 * n
    h.pcg_multirhs(m, 8, b.data_ptr(), x.data_ptr(), **kw)
    vec = h.tuned_config(celgpu.TUNE_SPMM)[0] >= 10 and name in ("poisson", "diffusion")
    assert h.elm_performance()[2] == stored(n, nnz, 8)[name if vec else "columns"] + 76 * n * 8 + 16 * n
    for prec in (celgpu.PREC_FP32_RU, celgpu.PREC_FP32_IR):
        h.pcg_multirhs(m, 8, b.data_ptr(), x.data_ptr(), **kw, precision=prec)
        form = name if name in ("poisson", "diffusion") else "columns"
        assert h.elm_performance()[2] == stored(n, nnz, 4)[form] + 40 * n * 8 + 8 * n
    m.destroy()


def test_reported_bytes_of_the_wide_kernel(gpu):
    celgpu, h, torch = gpu
    for build, matrix in ((synth.poisson7, lambda n, nnz: n), (None, lambda n, nnz: 8 * nnz + n)):
        if build:
            rp, ci, v = build(96)
        else:
            _, k = synth.lognormal_faces(np.random.default_rng(1), 96, 96, 96, 0.5)
            rp, ci, v = synth.diffusion7(96, 96, 96, *k)
        n, nnz = rp.size - 1, int(rp[-1])
        m = h.matrix_from_csr(rp, ci, v).jacobi()
        b = torch.ones(n, dtype=torch.float64, device="cuda")
        x = torch.zeros_like(b)
        h.pcg_jacobi(m, b.data_ptr(), x.data_ptr(), eps_rel=1e-3, iter_max=20, x0_mode=celgpu.X0_ZERO)
        assert h.elm_performance()[2] == matrix(n, nnz) + (48 if build else 64) * n
        m.destroy()
