"""A host batch that is cut into pieces and counts cells runs on the shapes of a batch of its size, with the counts and
results of a small one."""
import ctypes

import numpy as np
import pytest

from bsbolt_gb300 import _lib, autotune, extend, synth

pytestmark = pytest.mark.gpu


def test_shapes_and_counts(gpu_ctx):
    few, seq = synth.ksw_jobs(1 << 14, seed=5)
    mat, n = synth.fill_scmat(1, 4), 1 << 20
    want, cells = extend.ksw_extend2_batch(gpu_ctx, few, seq, mat, 6, 1, 6, 1, 100, want_cells=True)
    got, counted = extend.ksw_extend2_batch(gpu_ctx, np.resize(few, n), seq, mat, 6, 1, 6, 1, 100, want_cells=True)
    ms = (ctypes.c_float * _lib.BSB_NUM_TILES)()
    gpu_ctx.L.bsb_last_tile_ms(gpu_ctx.handle, ms, _lib.BSB_NUM_TILES)
    shapes = {s for t, s in enumerate(autotune.shapes()) if ms[t] > 0}
    assert {(4, 8), (4, 20), (4, 24), (4, 28), (4, 32), (8, 18)} <= shapes, shapes
    assert np.array_equal(got, np.tile(want, (n // len(few), 1))) and np.array_equal(counted, np.tile(cells, n // len(few)))


@pytest.mark.parametrize("device", [False, True], ids=["host", "device"])
@pytest.mark.parametrize("past", [0, 1])
def test_line_for_batches_that_count(gpu_ctx, device, past):
    """450 jobs an SM take the map of smaller batches, one more the default."""
    torch = pytest.importorskip("torch")
    few, seq = synth.ksw_jobs(1 << 14, seed=5)
    mat, n = synth.fill_scmat(1, 4), 450 * torch.cuda.get_device_properties(0).multi_processor_count + past
    want, cells = extend.ksw_extend2_batch(gpu_ctx, few, seq, mat, 6, 1, 6, 1, 100, want_cells=True)
    jobs = np.resize(few, n)
    if device:
        dj, ds = torch.from_numpy(jobs.view(np.uint8).copy()).cuda(), torch.from_numpy(seq).cuda()
        do, dc = torch.zeros((n, 6), dtype=torch.int32, device="cuda"), torch.zeros(n, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        extend.ksw_extend2_device(gpu_ctx, dj.data_ptr(), n, ds.data_ptr(), len(seq),
                                  extend.make_param(mat, 6, 1, 6, 1, 100), do.data_ptr(), dc.data_ptr())
        _lib.check(gpu_ctx.handle, gpu_ctx.L.bsb_sync(gpu_ctx.handle))
        got, counted = do.cpu().numpy(), dc.cpu().numpy()
    else:
        got, counted = extend.ksw_extend2_batch(gpu_ctx, jobs, seq, mat, 6, 1, 6, 1, 100, want_cells=True)
    ms = (ctypes.c_float * _lib.BSB_NUM_TILES)()
    gpu_ctx.L.bsb_last_tile_ms(gpu_ctx.handle, ms, _lib.BSB_NUM_TILES)
    shapes = {s for t, s in enumerate(autotune.shapes()) if ms[t] > 0}
    assert ((4, 32) in shapes) == bool(past), shapes
    assert np.array_equal(got, np.resize(want, (n, 6))) and np.array_equal(counted, np.resize(cells, n))
