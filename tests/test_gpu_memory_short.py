"""Calls with little device memory left: what is only kept for speed (sliced
copies, exchange words, row forms, spare blocks) gives way, and the call does
what it did without it; an ELM assembly that failed can be repeated."""
import numpy as np
import pytest

from cel_v3_b200 import synth

pytestmark = pytest.mark.gpu

MB = 1 << 20


class Filled:
    """Holds all device memory but about `leave` bytes."""

    def __init__(self, torch, leave):
        self.torch, self.held = torch, []
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        for _ in range(40):
            extra = torch.cuda.mem_get_info()[0] - leave
            if extra < 24 * MB:
                break
            try:
                self.held.append(torch.empty(extra, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                self.held.append(torch.empty(extra * 3 // 4, dtype=torch.uint8, device="cuda"))
        assert torch.cuda.mem_get_info()[0] < leave + 24 * MB

    def release(self):
        self.held = []
        self.torch.cuda.empty_cache()


def handle(celgpu, torch):
    return celgpu.Handle(0, torch.cuda.current_stream().cuda_stream)


def band(n, half):
    """Dense band: 2 half + 1 entries a row, no row patterns."""
    import scipy.sparse as sp
    off = list(range(-half, half + 1))
    A = sp.diags([np.full(n - abs(o), -1.0 / (1 + abs(o)) if o else 8.0) for o in off], off).tocsr()
    A.sort_indices()
    return A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data


def test_pcg_without_room_for_the_sliced_copy(gpu, monkeypatch):
    celgpu, _, torch = gpu
    h = handle(celgpu, torch)
    m = h.matrix_from_csr(*band(600000, 10)).jacobi()
    b = torch.linspace(-1, 1, m.n, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    kw = dict(eps_rel=1e-9, iter_max=400, x0_mode=celgpu.X0_ZERO)
    monkeypatch.setenv("CELG_ONCHIP_ROWS", "0")
    i = h.pcg_jacobi(m, b.data_ptr(), x.data_ptr(), **kw)
    want = x.cpu().numpy()
    monkeypatch.delenv("CELG_ONCHIP_ROWS")
    f = Filled(torch, 64 * MB)
    try:
        j = h.pcg_jacobi(m, b.data_ptr(), x.data_ptr(), **kw)
        got = x.cpu().numpy()
    finally:
        f.release()
    assert j.status == celgpu.OK and j.iter_done == i.iter_done and np.array_equal(got, want)
    j = h.pcg_jacobi(m, b.data_ptr(), x.data_ptr(), **kw)  # and on chip once there is room
    assert j.iter_done == i.iter_done and np.array_equal(x.cpu().numpy(), want)
    m.destroy()
    h.close()


def test_batch_without_room_for_its_kernels(gpu, monkeypatch):
    celgpu, _, torch = gpu
    h = handle(celgpu, torch)
    mats = [h.matrix_from_csr(*band(n, 10)).jacobi() for n in (600000, 20000)]
    b = [torch.linspace(-1, 1, m.n, dtype=torch.float64, device="cuda") for m in mats]
    x = [torch.zeros_like(t) for t in b]
    kw = dict(eps_rel=1e-9, iter_max=400, x0_mode=celgpu.X0_ZERO)

    def batch():
        i = h.pcg_batched(mats, [t.data_ptr() for t in b], [t.data_ptr() for t in x], **kw)
        return [q.iter_done for q in i], [t.cpu().numpy() for t in x]

    monkeypatch.setenv("CELG_ONCHIP_ROWS", "0")
    want = batch()
    monkeypatch.delenv("CELG_ONCHIP_ROWS")
    f = Filled(torch, 64 * MB)
    try:
        got = batch()
    finally:
        f.release()
    assert got[0] == want[0] and all(np.array_equal(p, q) for p, q in zip(got[1], want[1]))
    for m in mats:
        m.destroy()
    h.close()


def test_matrix_without_room_for_its_row_forms(gpu):
    celgpu, _, torch = gpu
    h = handle(celgpu, torch)
    n = 48 * MB
    rp = torch.arange(n + 1, dtype=torch.int32, device="cuda")
    v = torch.full((n,), 3.0, dtype=torch.float64, device="cuda")
    x = torch.linspace(-1, 1, n, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)
    f = Filled(torch, 16 * n + 4 * MB)  # the CSR block, not the byte a row
    try:
        m = h.matrix_from_csr_device(n, n, rp.data_ptr(), rp.data_ptr(), v.data_ptr())
        form = m.column_form()
        h.spmv(m, x.data_ptr(), y.data_ptr())
        torch.cuda.synchronize()
    finally:
        f.release()
    assert form == celgpu.COLS_INT32
    assert torch.equal(y, 3.0 * x)
    m.destroy()
    h.close()


def test_spare_blocks_give_way(gpu, monkeypatch):
    """Work vectors of a solve when what is left is held as spare blocks."""
    celgpu, _, torch = gpu
    h = handle(celgpu, torch)
    monkeypatch.setenv("CELG_ONCHIP_ROWS", "0")
    big = h.matrix_from_csr(*synth.poisson7(128)).jacobi()
    b = torch.ones(big.n, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    spare = [h.matrix_from_csr(*synth.poisson7(68)) for _ in range(3)]
    for m in spare:
        m.destroy()  # about 28 MB each
    f = Filled(torch, 32 * MB)
    try:
        i = h.pcg_jacobi(big, b.data_ptr(), x.data_ptr(), eps_rel=1e-3, iter_max=100, x0_mode=celgpu.X0_ZERO)
    finally:
        f.release()
    assert i.status == celgpu.ERR_NOCONV and i.iter_done == 100  # the cap, not an allocation
    big.destroy()
    h.close()


def elm_system():
    _, k = synth.lognormal_faces(np.random.default_rng(1), 90, 88, 86, 0.5)
    rp, ci, v = synth.diffusion7(90, 88, 86, *k)
    return rp.astype(np.int64), ci + 1, v


@pytest.mark.parametrize("scaling", [False, True])
def test_elm_completion_can_be_repeated(gpu, scaling):
    celgpu, _, torch = gpu
    rp, ci, v = elm_system()
    n = rp.size - 1
    b = np.random.default_rng(2).uniform(-1, 1, n)
    p = celgpu.params(eps_rel=1e-8, iter_max=60, fmt=celgpu.FMT_JAD)
    got = []
    for short in (False, True):
        h = handle(celgpu, torch)
        h.elm_init(n)
        h.elm_set_solver(celgpu.SOLVER_PCG, p, diag_scaling=scaling)
        h.elm_insert_rows(1, rp, ci, v)
        if short:
            f = Filled(torch, 32 * MB)
            try:
                with pytest.raises(celgpu.CelgError) as e:
                    h.elm_matrix_completed()
                assert e.value.status == celgpu.ERR_CUDA
            finally:
                f.release()
            h.elm_row_start(5)
            h.elm_reinsert(5, 40.0)  # the rows can still be changed
        else:
            w = v.copy()
            w[rp[4] + np.nonzero(ci[rp[4]:rp[5]] == 5)[0][0]] = 40.0
            h.elm_destroy()
            h.elm_init(n)
            h.elm_set_solver(celgpu.SOLVER_PCG, p, diag_scaling=scaling)
            h.elm_insert_rows(1, rp, ci, w)
        h.elm_matrix_completed()
        got.append((h.elm_doit(b)[1], h.elm_collect_solution(n)))
        h.elm_destroy()
        h.close()
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])


def test_elm_hint_is_no_device_memory(gpu):
    celgpu, _, torch = gpu
    rp, ci, v = elm_system()
    n = rp.size - 1
    h = handle(celgpu, torch)
    h.elm_init(n, nnz_hint=(300, 0))  # 2.4 GB if all of it were taken
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    h.elm_insert_rows(1, rp[:30001], ci[:rp[30000]], v[:rp[30000]])
    assert before - torch.cuda.mem_get_info()[0] < 64 * MB
    h.elm_insert_rows(30001, rp[30000:], ci[rp[30000]:], v[rp[30000]:])
    assert before - torch.cuda.mem_get_info()[0] < 256 * MB
    h.elm_matrix_completed()
    h.elm_destroy()
    h.close()


def test_elm_rows_without_room_on_the_device(gpu):
    """They wait on the host, as rows that come entry by entry do."""
    celgpu, _, torch = gpu
    rp, ci, v = elm_system()
    n = rp.size - 1
    b = np.random.default_rng(2).uniform(-1, 1, n)
    got = []
    for short in (False, True):
        h = handle(celgpu, torch)
        h.elm_init(n, nnz_hint=(0, 0))
        h.elm_set_solver(celgpu.SOLVER_PCG, celgpu.params(eps_rel=1e-6, iter_max=300))
        if short:
            h.elm_insert_rows(1, rp[:2001], ci[:rp[2000]], v[:rp[2000]])
            f = Filled(torch, 8 * MB)
            try:
                h.elm_insert_rows(2001, rp[2000:], ci[rp[2000]:], v[rp[2000]:])
            finally:
                f.release()
        else:
            h.elm_insert_rows(1, rp, ci, v)
        h.elm_matrix_completed()
        got.append((h.elm_doit(b)[1:], h.elm_collect_solution(n)))
        h.elm_destroy()
        h.close()
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
