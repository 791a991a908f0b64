"""A matrix whose rows are scaled after it has been solved with: whatever was
derived from its old values (FP32 copies, the concatenated copies of a batch)
has to follow, so that the next solve gives the bits of a matrix that was
scaled before its first one."""
import numpy as np
import pytest

from cel_v3_b200 import synth

pytestmark = pytest.mark.gpu


def constant(q):
    return synth.poisson7(q, q - 1, q - 2)


def variable(q):
    _, k = synth.lognormal_faces(np.random.default_rng(q), q, q - 1, q - 2, 0.5)
    return synth.diffusion7(q, q - 1, q - 2, *k)


@pytest.mark.parametrize("kind", [constant, variable])
@pytest.mark.parametrize("precision", ["fp64", "fp32_ru", "fp32_ir"])
@pytest.mark.parametrize("columns", [1, 8])
def test_scaled_after_a_solve(gpu, kind, precision, columns):
    celgpu, h, torch = gpu
    rp, ci, v = kind(14)
    n = rp.size - 1
    prec = {"fp64": celgpu.PREC_FP64, "fp32_ru": celgpu.PREC_FP32_RU, "fp32_ir": celgpu.PREC_FP32_IR}[precision]
    b = torch.from_numpy(np.random.default_rng(3).uniform(-1, 1, (n, columns))).cuda()
    kw = dict(eps_rel=1e-9, iter_max=2000, x0_mode=celgpu.X0_ZERO, precision=prec, inner_eps_rel=1e-2)

    def solve(m):
        x = torch.zeros_like(b)
        if columns == 1:
            i = [h.pcg_jacobi(m, b.data_ptr(), x.data_ptr(), **kw)]
        else:
            i = h.pcg_multirhs(m, columns, b.data_ptr(), x.data_ptr(), **kw)
        torch.cuda.synchronize()
        return x.cpu().numpy(), [(q.iter_done, q.arnoldi_steps, q.final_norm2) for q in i]

    m = h.matrix_from_csr(rp, ci, v).jacobi()
    solve(m)
    m.scale_diagonal()
    fresh = h.matrix_from_csr(rp, ci, v).jacobi().scale_diagonal()
    got, want = solve(m), solve(fresh)
    assert got[1] == want[1] and np.array_equal(got[0], want[0])
    m.destroy()
    fresh.destroy()


@pytest.mark.parametrize("precision", ["fp64", "fp32_ru", "fp32_ir"])
def test_scaled_between_batches(gpu, precision, monkeypatch):
    """The common sweeps read concatenated copies of the systems."""
    celgpu, h, torch = gpu
    prec = {"fp64": celgpu.PREC_FP64, "fp32_ru": celgpu.PREC_FP32_RU, "fp32_ir": celgpu.PREC_FP32_IR}[precision]
    kw = dict(eps_rel=1e-9, iter_max=2000, x0_mode=celgpu.X0_ZERO, precision=prec, inner_eps_rel=1e-2)
    monkeypatch.setenv("CELG_ONCHIP_ROWS", "0")
    mats = [h.matrix_from_csr(*variable(q)).jacobi() for q in (9, 14, 11)]
    b = [torch.from_numpy(np.random.default_rng(m.n).uniform(-1, 1, m.n)).cuda() for m in mats]
    x = [torch.zeros_like(t) for t in b]

    def batch():
        i = h.pcg_batched(mats, [t.data_ptr() for t in b], [t.data_ptr() for t in x], **kw)
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in x], i

    batch()
    mats[1].scale_diagonal()
    got, info = batch()
    for k, m in enumerate(mats):
        y = torch.zeros_like(b[k])
        one = h.pcg_jacobi(m, b[k].data_ptr(), y.data_ptr(), **kw)
        torch.cuda.synchronize()
        assert info[k].iter_done == one.iter_done and np.array_equal(got[k], y.cpu().numpy()), k
    for m in mats:
        m.destroy()
