"""The 16-byte-gather SpMM on the row table (constant-coefficient rows read
through one byte each) against the multi-RHS mirror, bit for bit: fewer rows
than a tile, one row past a tile, row groups without rows in the last tile,
more tiles than resident CTAs (a CTA then reads its next tile's bytes ahead,
in either tile order), the smallest and largest column counts."""
import numpy as np
import pytest

from cel_v3_b200 import synth
from tests.test_gpu_multirhs import dev, mirror, mirror_ru

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [10, 11, 12, 13, 14])
@pytest.mark.parametrize("dims,k,iters", [((11, 10, 9), 32, 2000), ((41, 25, 1), 2, 2000),
                                          ((20, 21, 22), 6, 2000), ((101, 89, 70), 2, 3)])
def test_table_spmm_bitexact(gpu, cfg, dims, k, iters, monkeypatch):
    celgpu, h, torch = gpu
    monkeypatch.setenv("CELG_SPMM_CFG", str(cfg))
    rp, ci, v = synth.poisson7(*dims)
    n = rp.size - 1
    B = np.random.default_rng(23).uniform(-1.0, 1.0, (n, k))
    m = h.matrix_from_csr(rp, ci, v).jacobi()
    Bd, Xd = dev(torch, B), dev(torch, np.zeros((n, k)))
    infos = h.pcg_multirhs(m, k, Bd.data_ptr(), Xd.data_ptr(), eps_rel=1e-10, iter_max=iters)
    Xo, ito, _ = mirror(rp, ci, v, B, 1e-10, iters)
    m.destroy()
    assert np.array_equal(Xd.cpu().numpy(), Xo)
    assert [i.iter_done for i in infos] == list(ito)


@pytest.mark.parametrize("cfg32", range(5))
@pytest.mark.parametrize("dims,k", [((11, 10, 9), 32), ((41, 25, 1), 4)])
def test_table_spmm_fp32_bitexact(gpu, cfg32, dims, k, monkeypatch):
    celgpu, h, torch = gpu
    monkeypatch.setenv("CELG_SPMM32_CFG", str(cfg32))
    rp, ci, v = synth.poisson7(*dims)
    n = rp.size - 1
    B = np.random.default_rng(29).uniform(-1.0, 1.0, (n, k))
    m = h.matrix_from_csr(rp, ci, v).jacobi()
    Bd, Xd = dev(torch, B), dev(torch, np.zeros((n, k)))
    infos = h.pcg_multirhs(m, k, Bd.data_ptr(), Xd.data_ptr(), eps_rel=1e-10, iter_max=3000,
                           precision=celgpu.PREC_FP32_RU, inner_eps_rel=1e-2)
    Xo, its, _, _ = mirror_ru(rp, ci, v, B, 1e-10, 1e-2, 3000)
    m.destroy()
    assert np.array_equal(Xd.cpu().numpy(), Xo)
    assert [i.iter_done for i in infos] == its
