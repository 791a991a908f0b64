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
