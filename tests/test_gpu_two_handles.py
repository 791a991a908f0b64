"""Two handles of one process: a matrix that another handle multiplies with is
destroyed while that handle's stream still has work (its memory must not go to
the next matrix before)."""
import numpy as np
import pytest

from cel_v3_b200 import synth

pytestmark = pytest.mark.gpu


def grid(q):
    _, k = synth.lognormal_faces(np.random.default_rng(q), q, q, q, 0.5)
    return synth.diffusion7(q, q, q, *k)


@pytest.mark.parametrize("how", ["other_handle", "captured"])
def test_matrix_destroyed_under_another_stream(gpu, how):
    celgpu, _, torch = gpu
    s2 = torch.cuda.Stream()
    h1 = celgpu.Handle(0, torch.cuda.current_stream().cuda_stream)
    h2 = celgpu.Handle(0, s2.cuda_stream)
    rp, ci, v = grid(60)
    n = rp.size - 1
    x = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, n)).cuda()
    want, y = torch.zeros_like(x), torch.zeros_like(x)
    other = [torch.from_numpy(a).cuda() for a in (rp, ci, -v)]
    m = h1.matrix_from_csr(rp, ci, v)
    h1.spmv(m, x.data_ptr(), want.data_ptr())
    torch.cuda.synchronize()
    if how == "captured":
        side = torch.cuda.Stream()
        hc = celgpu.Handle(0, side.cuda_stream)
        mc = hc.matrix_from_csr(rp, ci, v)
        hc.spmv(mc, x.data_ptr(), y.data_ptr())
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side, capture_error_mode="relaxed"):
            for _ in range(100):
                hc.spmv(mc, x.data_ptr(), y.data_ptr())
        with torch.cuda.stream(s2):
            for _ in range(20):
                g.replay()
        y_last, mat, own = y, mc, hc
    else:
        with torch.cuda.stream(s2):
            for _ in range(2000):
                h2.spmv(m, x.data_ptr(), y.data_ptr())
        y_last, mat, own = y, m, h1
    mat.destroy()
    m2 = own.matrix_from_csr_device(n, int(rp[-1]), *[t.data_ptr() for t in other])
    torch.cuda.synchronize()
    assert torch.equal(y_last, want)
    z = torch.zeros_like(x)
    own.spmv(m2, x.data_ptr(), z.data_ptr())
    torch.cuda.synchronize()
    assert torch.equal(z, -want)
    m2.destroy()
    if how == "captured":
        del g
        m.destroy()
        hc.close()
    h1.close()
    h2.close()
