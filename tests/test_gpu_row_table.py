"""Row-table sweeps (constant-coefficient rows read through one byte each)
against the oracle, bit for bit: few rows, the edges of a tile, systems large
enough for the staged window (with ragged ends, several clusters of offsets,
an x the bulk copies cannot start on), values that stop repeating late, rows
that differ in a sign of zero only, rescaled values."""
import numpy as np
import pytest

from cel_v3_b200 import synth
from oracle import celref as R

pytestmark = pytest.mark.gpu


def band(n, offsets, values):
    """Rows i with entries (i + o, value) for the offsets that fall inside."""
    i = np.arange(n)
    keep = np.stack([(i + o >= 0) & (i + o < n) for o in offsets], 1)
    ci = (i[:, None] + np.array(offsets)[None, :])[keep].astype(np.int32)
    v = np.broadcast_to(np.array(values, float), keep.shape)[keep]
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    return rp, ci, np.ascontiguousarray(v)


def late_change():
    rp, ci, v = synth.poisson7(30, 40, 50)
    v[-400:] += np.arange(400) * 1e-3
    return rp, ci, v


def signed_zero():
    rp, ci, v = band(3000, (-1, 0, 1), (0.0, 2.0, -1.0))
    v[rp[700]] = -0.0
    return rp, ci, v


CASES = {
    "one_row": lambda: synth.poisson7(1, 1, 1),
    "tile_edge": lambda: synth.poisson7(41, 25, 1),
    "poisson": lambda: synth.poisson7(20, 21, 22),
    "window_ragged": lambda: synth.poisson7(85, 83, 67),
    "window_wide_planes": lambda: synth.poisson7(131, 127, 31),
    "window_five_clusters": lambda: band(500003, (-70001, -3000, -5, 0, 7, 2500, 90000),
                                         (0.5, -1.0, 0.25, 8.0, -0.125, 3.0, 1.5)),
    "pairs_ragged": lambda: band(7400003, (-39597, -201, -1, 0, 1, 201, 39597),
                                 (-1.0, -2.0, -3.0, 12.5, -3.0, -2.0, -1.0)),
    "too_many_clusters": lambda: band(480001, (-70000, -50000, -30000, -10000, 0, 20000, 40000, 60000),
                                      (1.0, 2.0, 3.0, 40.0, 5.0, 6.0, 7.0, 8.0)),
    "values_change_late": late_change,
    "signed_zero": signed_zero,
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_spmv_forms_bitexact(gpu, name):
    celgpu, h, torch = gpu
    rp, ci, v = CASES[name]()
    n = rp.size - 1
    x = np.random.default_rng(3).standard_normal(n)
    want = R.spmv_csr(rp, ci, v, x)
    m = h.matrix_from_csr(rp, ci, v)
    assert m.column_form() == celgpu.COLS_PATTERN
    m.to_jad()
    buf = torch.zeros(n + 1, dtype=torch.float64).cuda()
    for shift in (0, 1):  # 1: x starts on an odd 8 bytes
        buf[shift:shift + n] = torch.from_numpy(x).cuda()
        y = torch.full((n,), 3.0, dtype=torch.float64).cuda()
        h.spmv(m, buf.data_ptr() + 8 * shift, y.data_ptr(), fmt=celgpu.FMT_JAD)
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy(), want)
        h.spmv(m, buf.data_ptr() + 8 * shift, y.data_ptr(), accumulate=True)
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy(), want + want)
    x32 = torch.from_numpy(x.astype(np.float32)).cuda()
    y32 = torch.zeros(n, dtype=torch.float32).cuda()
    m.make_fp32()
    h.spmv_f32(m, x32.data_ptr(), y32.data_ptr())
    torch.cuda.synchronize()
    want32 = np.zeros(n, np.float32)
    lens = np.diff(rp)
    for k in range(int(lens.max())):
        rows = np.nonzero(lens > k)[0]
        e = rp[rows] + k
        want32[rows] += v[e].astype(np.float32) * x.astype(np.float32)[ci[e]]
    assert np.array_equal(y32.cpu().numpy(), want32)
    m.destroy()


@pytest.mark.parametrize("name,precision", [("window_ragged", "fp64"), ("window_ragged", "fp32_ru"),
                                            ("window_ragged", "fp32_ir"), ("poisson", "fp64")])
def test_pcg_same_bits_with_and_without_repeating_values(gpu, name, precision, monkeypatch):
    """The same system with one more, uncoupled, row whose value no other row
    has reads its values from the matrix when 256 of them differ; with fewer
    it keeps the row table.  Both equal the oracle / each other."""
    celgpu, h, torch = gpu
    monkeypatch.setenv("CELG_ONCHIP_ROWS", "0")
    rp, ci, v = CASES[name]()
    n, extra = rp.size - 1, 300
    rp2 = np.concatenate([rp, rp[-1] + 1 + np.arange(extra)]).astype(np.int32)
    ci2 = np.concatenate([ci, n + np.arange(extra)]).astype(np.int32)
    v2 = np.concatenate([v, 1.0 + np.arange(extra)])
    b = np.random.default_rng(5).uniform(-1, 1, n)
    out = []
    prec = {"fp64": celgpu.PREC_FP64, "fp32_ru": celgpu.PREC_FP32_RU, "fp32_ir": celgpu.PREC_FP32_IR}[precision]
    for rows in ((rp, ci, v, b), (rp2, ci2, v2, np.concatenate([b, np.zeros(extra)]))):
        m = h.matrix_from_csr(*rows[:3]).jacobi()
        x = torch.zeros(rows[3].size, dtype=torch.float64).cuda()
        i = h.pcg_jacobi(m, torch.from_numpy(rows[3]).cuda().data_ptr(), x.data_ptr(), eps_rel=1e-9, iter_max=25,
                         precision=prec, outer_max=2, inner_iter_max=25,
                         inner_eps_rel=1e-2 if precision == "fp32_ru" else 1e-4)
        torch.cuda.synchronize()
        out.append((x.cpu().numpy()[:n], i.iter_done, i.arnoldi_steps))
        m.destroy()
    # (the extra rows start a tile of their own or fill the last one with
    # zeros: every partial sum is the same)
    assert out[0][1:] == out[1][1:] and np.array_equal(out[0][0], out[1][0])
    if precision == "fp64":
        xr, ir = R.pcg_jacobi(R.Matrix(rp, ci, v), R.jacobi(R.diag(rp, ci, v)), b, eps_rel=1e-9, iter_max=25,
                              red=R.RED_TREE)
        assert np.array_equal(out[0][0], xr)


def test_scaling_rebuilds_the_table(gpu):
    celgpu, h, torch = gpu
    rp, ci, v = CASES["poisson"]()
    n = rp.size - 1
    x = np.random.default_rng(3).standard_normal(n)
    m = h.matrix_from_csr(rp, ci, v).jacobi()
    m.scale_diagonal()
    vs = v / np.sqrt(np.repeat(np.abs(R.diag(rp, ci, v)), np.diff(rp)))
    y = torch.zeros(n, dtype=torch.float64).cuda()
    h.spmv(m, torch.from_numpy(x).cuda().data_ptr(), y.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), R.spmv_csr(rp, ci, vs, x))
    m.destroy()
