"""A process that has fewer SMs at its disposal than the device reports: the
driver refuses cooperative grids that cannot all be resident, and the solves
then take the sweeps.  The handle is told that the device has more SMs than it
has, which makes the same grids too large."""
import ctypes

import numpy as np
import pytest

from cel_v3_b200 import synth

pytestmark = pytest.mark.gpu


def pretend(celgpu, h, sms):
    """celg_handle::sms (celg_internal.h), found by its value."""
    at = ctypes.c_int.from_address(h.ptr.value + 32)
    assert at.value == h.sm_count() and at.value > 100
    at.value = sms
    assert h.sm_count() == sms


def grid(nx, ny, nz):
    _, k = synth.lognormal_faces(np.random.default_rng(nx), nx, ny, nz, 0.5)
    return synth.diffusion7(nx, ny, nz, *k)


def test_refused_grids_leave_the_solve_to_the_sweeps(gpu):
    celgpu, _, torch = gpu
    rp, ci, v = grid(60, 60, 57)  # 201 tiles: more CTAs than SMs at 296
    n = rp.size - 1
    b = torch.linspace(-1, 1, n, dtype=torch.float64, device="cuda")
    kw = dict(eps_rel=1e-9, iter_max=300, x0_mode=celgpu.X0_ZERO)
    got = []
    for sms in (None, 296):
        h = celgpu.Handle(0, torch.cuda.current_stream().cuda_stream)
        if sms:
            pretend(celgpu, h, sms)
        m = h.matrix_from_csr(rp, ci, v).jacobi()
        x = torch.zeros_like(b)
        i = h.pcg_jacobi(m, b.data_ptr(), x.data_ptr(), **kw)
        y = torch.zeros_like(b)
        j = h.gmres_jacobi(m, b.data_ptr(), y.data_ptr(), restart=10, **kw)
        got.append((i.iter_done, x.cpu().numpy(), j.arnoldi_steps, y.cpu().numpy()))
        m.destroy()
        h.close()
    for p, q in zip(*got):
        assert np.array_equal(p, q)


def test_batch_refused_after_its_first_system(gpu):
    """Of two systems the larger needs the smaller grid (140 and 155 CTAs with
    160 SMs): nothing may have run when the second is refused."""
    celgpu, _, torch = gpu
    systems = [grid(100, 100, 100), grid(100, 100, 95)]
    b = [torch.linspace(-1, 1, s[0].size - 1, dtype=torch.float64, device="cuda") for s in systems]
    start = [t.cos() for t in b]
    kw = dict(eps_rel=1e-6, iter_max=40, x0_mode=celgpu.X0_USER)
    got = []
    for sms in (None, 160):
        h = celgpu.Handle(0, torch.cuda.current_stream().cuda_stream)
        if sms:
            pretend(celgpu, h, sms)
        mats = [h.matrix_from_csr(*s).jacobi() for s in systems]
        x = [t.clone() for t in start]
        i = h.pcg_batched(mats, [t.data_ptr() for t in b], [t.data_ptr() for t in x], **kw)
        got.append(([q.iter_done for q in i], [t.cpu().numpy() for t in x]))
        for m in mats:
            m.destroy()
        h.close()
    assert got[0][0] == got[1][0]
    for p, q in zip(got[0][1], got[1][1]):
        assert np.array_equal(p, q)
