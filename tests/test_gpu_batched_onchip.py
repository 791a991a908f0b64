"""Batched FP64 solves in kernels of their own, side by side on shares of the
SMs, against the common sweeps and the single solves, bit for bit: systems of
every share (one row to 912k), unstructured ones, an empty one, one matrix
used twice, every start vector; repeated, and after another batch."""
import numpy as np
import pytest

from cel_v3_b200 import synth
from tests.helpers import random_csr, spd_from_pattern

pytestmark = pytest.mark.gpu


def grid(q):
    _, k = synth.lognormal_faces(np.random.default_rng(q), q, q, q, 0.5)
    return synth.diffusion7(q, q, q, *k)


@pytest.mark.parametrize("x0", ["zero", "ones", "user"])
def test_batched_kernels_equal_sweeps_and_singles(gpu, x0, monkeypatch):
    celgpu, h, torch = gpu
    sides = [20, 59, 1, 80, 33, 97, 41, 62] if x0 == "zero" else [20, 59, 1, 33, 82]
    mats = [h.matrix_from_csr(*grid(q)).jacobi() for q in sides]
    mats.append(h.matrix_from_csr(*spd_from_pattern(*random_csr(20011, np.random.default_rng(5), max_len=9))).jacobi())
    mats.append(h.matrix_from_csr(np.zeros(1, np.int32), np.zeros(0, np.int32), np.zeros(0)).jacobi())
    mats.append(mats[0])
    rng = np.random.default_rng(1)
    sizes = [m.n for m in mats]
    b = [torch.from_numpy(rng.uniform(-1, 1, max(n, 1))).cuda() for n in sizes]
    start = [torch.from_numpy(rng.uniform(-1, 1, max(n, 1))).cuda() for n in sizes]
    kw = dict(eps_rel=1e-9, iter_max=60, x0_mode={"zero": celgpu.X0_ZERO, "ones": celgpu.X0_REF_ONES,
                                                  "user": celgpu.X0_USER}[x0])

    def solve():
        x = [s.clone() for s in start]
        info = h.pcg_batched(mats, [t.data_ptr() for t in b], [t.data_ptr() for t in x], **kw)
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in x], info

    monkeypatch.setenv("CELG_ONCHIP_ROWS", "0")
    xs, si = solve()
    monkeypatch.delenv("CELG_ONCHIP_ROWS")
    for _ in range(2):
        xo, oi = solve()
        for k in range(len(mats)):
            assert np.array_equal(xs[k], xo[k]), k
            for f in ("iter_done", "final_norm2", "bnorm", "verified_relres", "status"):
                assert si[k][f] == oi[k][f], (k, f)
        h.pcg_batched(mats[:2], [t.data_ptr() for t in b[:2]], [t.clone().data_ptr() for t in start[:2]], **kw)
    for k in (0, 1, len(sides)):
        x = start[k].clone()
        i = h.pcg_jacobi(mats[k], b[k].data_ptr(), x.data_ptr(), **kw)
        torch.cuda.synchronize()
        assert np.array_equal(x.cpu().numpy(), xo[k]) and i.iter_done == oi[k].iter_done
    for m in mats[:-1]:
        m.destroy()
