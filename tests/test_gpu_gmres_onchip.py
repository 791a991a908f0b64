"""GMRES(m) with the orthogonalisation in one kernel per Arnoldi step against
the sweeps, bit for bit: fewer rows than a tile, tile edges, one to fourteen
tiles per CTA (the last two not staged), restarts of one vector and of many,
both formats, the reference's literal rotations, the iteration cap."""
import numpy as np
import pytest

from cel_v3_b200 import synth
from tests.helpers import random_csr, spd_from_pattern

pytestmark = pytest.mark.gpu


def grid(nx, ny, nz):
    _, k = synth.lognormal_faces(np.random.default_rng(nx), nx, ny, nz, 0.5)
    return synth.diffusion7(nx, ny, nz, *k)


CASES = {
    "one_row": (lambda: grid(1, 1, 1), 2, 3),
    "129_rows": (lambda: grid(43, 3, 1), 5, 4),
    "one_tile": (lambda: grid(16, 8, 8), 1, 6),
    "tile_and_a_row": (lambda: grid(41, 25, 1), 7, 3),
    "uneven_rows": (lambda: spd_from_pattern(*random_csr(20011, np.random.default_rng(5), max_len=9)), 30, 1),
    "two_tiles_a_cta": (lambda: grid(60, 61, 62), 12, 1),
    "odd_tiles_a_cta": (lambda: grid(95, 97, 99), 6, 1),
    "last_tiles_not_staged": (lambda: grid(127, 128, 127), 5, 1),
    "more_than_fit": (lambda: grid(131, 129, 127), 3, 1),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_onchip_orthogonalisation_equals_sweeps(gpu, name, monkeypatch):
    celgpu, h, torch = gpu
    make, restart, iters = CASES[name]
    rp, ci, v = make()
    n = rp.size - 1
    m = h.matrix_from_csr(rp, ci, v).jacobi()
    m.to_jad()
    b = torch.from_numpy(np.random.default_rng(2).uniform(-1, 1, n)).cuda()
    runs = [dict(), dict(fmt=celgpu.FMT_JAD)] + ([dict(literal_ref_bugs=1)] if n < 30000 else [])
    for kw in runs:
        got = []
        for rows in ("0", None):
            if rows is None:
                monkeypatch.delenv("CELG_ONCHIP_ROWS")
            else:
                monkeypatch.setenv("CELG_ONCHIP_ROWS", rows)
            x = torch.zeros(n, dtype=torch.float64).cuda()
            # iter_max 0: the outer loop ends after the first m + 1 restarts
            i = h.gmres_jacobi(m, b.data_ptr(), x.data_ptr(), restart=restart, iter_max=0 if iters == 1 else iters,
                               eps_rel=1e-9, history=4000, **kw)
            torch.cuda.synchronize()
            got.append((x.cpu().numpy(), i))
        (xs, s), (xo, o) = got
        assert np.array_equal(s.history, o.history) and len(o.history) > 1
        assert np.array_equal(xs, xo, equal_nan=True)
        for f in ("iter_done", "arnoldi_steps", "status", "bnorm"):
            assert s[f] == o[f], f
        assert s.final_norm2 == o.final_norm2 or (np.isnan(s.final_norm2) and np.isnan(o.final_norm2))
    m.destroy()
