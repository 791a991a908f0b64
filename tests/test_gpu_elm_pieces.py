"""ELM rows in pieces, short ones among them: the same matrix as from one call,
without a sort (the rows are in order) and without taking entries back from the
device."""
import numpy as np
import pytest

from cel_v3_b200 import synth

pytestmark = pytest.mark.gpu


def device_work(torch, fn):
    """Names of the kernels and copies that fn runs on the GPU."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    return [e.name for e in prof.events()]


@pytest.mark.parametrize("pieces", ["long_short", "short_long", "thousands", "all_short", "with_empty", "gap"])
def test_pieces_equal_one_call(gpu, pieces):
    celgpu, h, torch = gpu
    _, k = synth.lognormal_faces(np.random.default_rng(1), 19, 18, 17, 0.5)
    rp, ci, v = synth.diffusion7(19, 18, 17, *k)
    rp, ci = rp.astype(np.int64), ci + 1
    n = rp.size - 1
    b = np.random.default_rng(2).uniform(-1, 1, n)
    cuts = {"long_short": [0, n - 3, n], "short_long": [0, 5, n], "thousands": list(range(0, n, 1000)) + [n],
            "all_short": list(range(0, n, 37)) + [n], "with_empty": [0, 0, 700, 700, 2900, 2900, n, n],
            "gap": [0, 2000, 2010, n]}[pieces]

    def insert(cuts):
        for a, e in zip(cuts[:-1], cuts[1:]):
            if pieces == "gap" and a == 2000:
                h.elm_insert_rows(a + 1, np.arange(11), np.arange(2001, 2011), np.full(10, 2.0))
            else:
                h.elm_insert_rows(a + 1, rp[a:e + 1], ci[rp[a]:rp[e]], v[rp[a]:rp[e]])

    def assemble(cuts):
        h.elm_init(n)
        h.elm_set_solver(celgpu.SOLVER_PCG, celgpu.params(eps_rel=1e-10, iter_max=500))
        insert(cuts)
        h.elm_matrix_completed()

    names = device_work(torch, lambda: assemble(cuts))
    assert any("row_sets" in s for s in names), names  # the profiler sees the assembly
    assert not any("Sort" in s for s in names) and not any("DtoH" in s and "Pageable" in s for s in names), names
    _, niter, ftol = h.elm_doit(b)
    x = h.elm_collect_solution(n)
    h.elm_destroy()
    # the same entries, one by one
    h.elm_init(n)
    h.elm_set_solver(celgpu.SOLVER_PCG, celgpu.params(eps_rel=1e-10, iter_max=500))
    for r in range(n):
        h.elm_row_start(r + 1)
        if pieces == "gap" and 2000 <= r < 2010:
            h.elm_insert(r + 1, 2.0)
            continue
        for q in range(rp[r], rp[r + 1]):
            h.elm_insert(int(ci[q]), float(v[q]))
    h.elm_matrix_completed()
    assert h.elm_doit(b)[1:] == (niter, ftol) and np.array_equal(h.elm_collect_solution(n), x)
    h.elm_destroy()


def test_pieces_then_changes(gpu):
    """A re-inserted diagonal and an inserted entry after short pieces, some of
    which have not gone to the device."""
    celgpu, h, torch = gpu
    rp, ci, v = synth.poisson7(12)
    rp, ci = rp.astype(np.int64), ci + 1
    n = rp.size - 1
    b = np.random.default_rng(2).uniform(-1, 1, n)
    out = []
    for pieces in (True, False):
        h.elm_init(n)
        h.elm_set_solver(celgpu.SOLVER_PCG, celgpu.params(eps_rel=1e-10, iter_max=500))
        if pieces:
            for a, e in ((0, 900), (900, 901), (901, 1000), (1000, n - 1)):
                h.elm_insert_rows(a + 1, rp[a:e + 1], ci[rp[a]:rp[e]], v[rp[a]:rp[e]])
        else:
            for r in range(n - 1):
                h.elm_row_start(r + 1)
                for q in range(rp[r], rp[r + 1]):
                    h.elm_insert(int(ci[q]), float(v[q]))
        h.elm_row_start(n)
        h.elm_insert(n, 6.5)
        h.elm_row_start(950)
        h.elm_reinsert(950, 40.0)
        h.elm_row_start(3)
        h.elm_reinsert(3, 50.0)
        h.elm_matrix_completed()
        out.append((h.elm_doit(b)[1:], h.elm_collect_solution(n)))
        h.elm_destroy()
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])
