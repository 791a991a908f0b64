"""What celg_tuned_config reports after each kind of batched solve: the path
(systems in kernels of their own, or common sweeps) and the shape that the
last batch's sweeps really ran with."""
import pytest

from cel_v3_b200 import synth

pytestmark = pytest.mark.gpu


def test_reported_shape_is_the_last_batchs(gpu, monkeypatch):
    celgpu, _, torch = gpu
    h = celgpu.Handle(0, torch.cuda.current_stream().cuda_stream)
    with pytest.raises(celgpu.CelgError) as e:
        h.tuned_config(celgpu.TUNE_BATCH_PATH)
    assert e.value.status == celgpu.ERR_STATE
    mats = [h.matrix_from_csr(*synth.poisson7(q)).jacobi() for q in (20, 24)]
    b = [torch.ones(m.n, dtype=torch.float64, device="cuda") for m in mats]
    x = [torch.zeros_like(t) for t in b]
    shapes = [(0, 8), (0, 6), (0, 4), (2, 8), (2, 4), (1, 8)]

    def batch(prec):
        h.pcg_batched(mats, [t.data_ptr() for t in b], [t.data_ptr() for t in x], eps_rel=1e-8, iter_max=500,
                      precision=prec, inner_eps_rel=1e-2)

    batch(celgpu.PREC_FP64)
    assert h.tuned_config(celgpu.TUNE_BATCH_PATH) == (celgpu.BATCH_KERNELS, 0)
    monkeypatch.setenv("CELG_BATCH_SHAPE", "3")
    batch(celgpu.PREC_FP32_RU)
    assert h.tuned_config(celgpu.TUNE_BATCH) == shapes[3]
    assert h.tuned_config(celgpu.TUNE_BATCH_PATH) == (celgpu.BATCH_SWEEPS, 0)
    batch(celgpu.PREC_FP64)  # a shape asked for: the sweeps
    assert h.tuned_config(celgpu.TUNE_BATCH) == shapes[3]
    assert h.tuned_config(celgpu.TUNE_BATCH_PATH) == (celgpu.BATCH_SWEEPS, 0)
    monkeypatch.delenv("CELG_BATCH_SHAPE")
    batch(celgpu.PREC_FP64)
    assert h.tuned_config(celgpu.TUNE_BATCH_PATH) == (celgpu.BATCH_KERNELS, 0)
    assert h.tuned_config(celgpu.TUNE_BATCH) == shapes[0]  # documented: no shape in use
    for prec in (celgpu.PREC_FP32_IR, celgpu.PREC_FP32_RU):
        batch(prec)
        assert h.tuned_config(celgpu.TUNE_BATCH) == shapes[3]  # the batch's copy keeps its shape
    torch.cuda.synchronize()
    for m in mats:
        m.destroy()
    h.close()


def test_tuners_pick_is_reported_after_common_sweeps(gpu, monkeypatch):
    """Without a forced shape and without kernels of their own the tuner runs."""
    celgpu, _, torch = gpu
    h = celgpu.Handle(0, torch.cuda.current_stream().cuda_stream)
    monkeypatch.setenv("CELG_ONCHIP_ROWS", "0")
    mats = [h.matrix_from_csr(*synth.poisson7(q)).jacobi() for q in (20, 24, 31)]
    b = [torch.ones(m.n, dtype=torch.float64, device="cuda") for m in mats]
    x = [torch.zeros_like(t) for t in b]
    h.pcg_batched(mats, [t.data_ptr() for t in b], [t.data_ptr() for t in x], eps_rel=1e-8, iter_max=500)
    assert h.tuned_config(celgpu.TUNE_BATCH_PATH) == (celgpu.BATCH_SWEEPS, 0)
    assert h.tuned_config(celgpu.TUNE_BATCH) in [(0, 8), (0, 6), (0, 4), (2, 8), (2, 4), (1, 8)]
    torch.cuda.synchronize()
    for m in mats:
        m.destroy()
    h.close()
