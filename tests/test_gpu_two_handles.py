"""Two handles of one process: a matrix that another handle multiplies with is
destroyed while that handle's stream still has work (its memory must not go to
the next matrix before), and solves on chip at the same time from two threads."""
import threading

import numpy as np
import pytest

from cel_v3_b200 import synth
from tests.helpers import random_csr, spd_from_pattern

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


def test_solves_from_two_threads(gpu):
    celgpu, _, torch = gpu
    band = spd_from_pattern(*random_csr(30011, np.random.default_rng(5), max_len=9))
    systems = [[grid(33), band, grid(24)], [band, grid(41), grid(20)]]
    out, errors = [[], []], []

    def work(w, reps):
        try:
            stream = torch.cuda.Stream()
            h = celgpu.Handle(0, stream.cuda_stream)
            with torch.cuda.stream(stream):
                mats = [h.matrix_from_csr(*s).jacobi() for s in systems[w]]
                b = [torch.linspace(-1, 1, m.n, dtype=torch.float64, device="cuda") for m in mats]
                x = [torch.zeros_like(t) for t in b]
                for _ in range(reps):
                    res = []
                    for m, r, s in zip(mats, b, x):
                        kw = dict(eps_rel=1e-9, iter_max=400, x0_mode=celgpu.X0_ZERO)
                        i = h.pcg_jacobi(m, r.data_ptr(), s.data_ptr(), **kw)
                        res.append((i.iter_done, s.cpu().numpy()))
                        i = h.gmres_jacobi(m, r.data_ptr(), s.data_ptr(), restart=12, **kw)
                        res.append((i.arnoldi_steps, s.cpu().numpy()))
                    i = h.pcg_batched(mats, [t.data_ptr() for t in b], [t.data_ptr() for t in x], **kw)
                    res += [(q.iter_done, s.cpu().numpy()) for q, s in zip(i, x)]
                    out[w].append(res)
                    fresh = h.matrix_from_csr(*systems[w][2])  # blocks come and go meanwhile
                    fresh.destroy()
                for m in mats:
                    m.destroy()
            h.close()
        except BaseException as e:  # noqa: BLE001 - reported by the test
            errors.append(e)

    for w in (0, 1):  # each alone
        work(w, 1)
    alone = [out[0].pop(), out[1].pop()]
    threads = [threading.Thread(target=work, args=(w, 6)) for w in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for w in (0, 1):
        assert len(out[w]) == 6
        for res in out[w]:
            for (i, a), (j, c) in zip(res, alone[w]):
                assert i == j and np.array_equal(a, c)
