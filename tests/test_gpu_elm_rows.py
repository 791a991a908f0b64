"""ELM assembly by whole rows (copied straight into the matrix) against the
same entries inserted one by one: all rows at once, in pieces, with rows left
out, out of order, with unsorted columns, then changed entry by entry."""
import numpy as np
import pytest

from cel_v3_b200 import synth

pytestmark = pytest.mark.gpu


def system():
    _, k = synth.lognormal_faces(np.random.default_rng(1), 17, 16, 15, 0.5)
    rp, ci, v = synth.diffusion7(17, 16, 15, *k)
    return rp.astype(np.int64), ci + 1, v


def solve(celgpu, h, n, b):
    h.elm_set_solver(celgpu.SOLVER_PCG, celgpu.params(eps_rel=1e-10, iter_max=500))
    h.elm_matrix_completed()
    _, niter, ftol = h.elm_doit(b)
    x = h.elm_collect_solution(n)
    h.elm_destroy()
    return x, niter, ftol


def entries(h, rp, ci, v, rows):
    for r in rows:
        h.elm_row_start(int(r) + 1)
        for k in range(rp[r], rp[r + 1]):
            h.elm_insert(int(ci[k]), float(v[k]))


@pytest.mark.parametrize("how", ["at_once", "pieces", "pieces_then_entries", "gap", "swapped", "unsorted", "reinsert",
                                 "too_small_hint", "offset_row_ptr"])
def test_rows_equal_entries(gpu, how):
    celgpu, h, torch = gpu
    rp, ci, v = system()
    n = rp.size - 1
    b = np.random.default_rng(2).uniform(-1, 1, n)
    rows = np.arange(n)
    cuts = [0, 1500, 1501, 3000, n]
    hint = (1, 0) if how == "too_small_hint" else (7, 0)

    def piece(a, e):
        lo, hi = rp[a], rp[e]
        off = 5 if how == "offset_row_ptr" else 0
        h.elm_insert_rows(a + 1, rp[a:e + 1] - lo + off, ci[lo:hi], v[lo:hi])

    vv = v.copy()
    h.elm_init(n, nnz_hint=hint)
    if how in ("at_once", "offset_row_ptr"):
        piece(0, n)
    elif how in ("pieces", "too_small_hint"):
        for a, e in zip(cuts[:-1], cuts[1:]):
            piece(a, e)
    elif how == "pieces_then_entries":
        piece(0, 2000)
        entries(h, rp, ci, v, range(2000, n))
    elif how == "gap":  # rows 2000..2009 have nothing but their diagonal, inserted last
        piece(0, 2000)
        piece(2010, n)
        rows = np.concatenate([np.arange(2000), np.arange(2010, n)])
    elif how == "swapped":
        piece(2000, n)
        piece(0, 2000)
    elif how == "unsorted":
        c2, v2 = ci.copy(), v.copy()
        for r in range(0, n, 3):
            c2[rp[r]:rp[r + 1]] = c2[rp[r]:rp[r + 1]][::-1]
            v2[rp[r]:rp[r + 1]] = v2[rp[r]:rp[r + 1]][::-1]
        h.elm_insert_rows(1, rp, c2, v2)
    elif how == "reinsert":
        piece(0, n)
        h.elm_row_start(78)
        h.elm_reinsert(78, 50.0)
        vv[rp[77] + np.nonzero(ci[rp[77]:rp[78]] == 78)[0][0]] = 50.0
    if how == "gap":
        entries(h, np.arange(n + 1), np.arange(1, n + 1), np.full(n, 2.0), range(2000, 2010))
    got = solve(celgpu, h, n, b)
    h.elm_init(n, nnz_hint=hint)
    entries(h, rp, ci, vv, rows)
    if how == "gap":
        entries(h, np.arange(n + 1), np.arange(1, n + 1), np.full(n, 2.0), range(2000, 2010))
    want = solve(celgpu, h, n, b)
    assert got[1:] == want[1:] and np.array_equal(got[0], want[0])


def test_rows_rejected_as_before(gpu):
    celgpu, h, torch = gpu
    rp, ci, v = system()
    n = rp.size - 1
    h.elm_init(n)
    bad = ci.copy()
    bad[4000] = n + 1
    with pytest.raises(celgpu.CelgError):
        h.elm_insert_rows(1, rp, bad, v)
    with pytest.raises(celgpu.CelgError):
        h.elm_insert_rows(2, rp, ci, v)  # one row too many
    back = rp.copy()
    back[9] = back[11]
    with pytest.raises(celgpu.CelgError):
        h.elm_insert_rows(1, back, ci, v)
    h.elm_destroy()
