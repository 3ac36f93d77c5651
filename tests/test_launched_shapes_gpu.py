"""What bsb_sync reads back are the marks of the shapes that ran: no error stays behind on scorings that leave the ring
out, and every shape's time, the cut rings' among them, is reported."""
import ctypes

import numpy as np
import pytest

import oracle
from bsbolt_gb300 import _lib, extend, synth

pytestmark = pytest.mark.gpu


def run_device(torch, ctx, jobs, seq, scoring):
    """(tuples, ms of the batch, ms by shape) of one batch through the device entry and bsb_sync."""
    a, b, o_del, e_del, o_ins, e_ins, zdrop = scoring
    dj, ds = torch.from_numpy(jobs.view(np.uint8).copy()).cuda(), torch.from_numpy(seq).cuda()
    do = torch.zeros((len(jobs), 6), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    extend.ksw_extend2_device(ctx, dj.data_ptr(), len(jobs), ds.data_ptr(), len(seq),
                              extend.make_param(synth.fill_scmat(a, b), o_del, e_del, o_ins, e_ins, zdrop), do.data_ptr())
    _lib.check(ctx.handle, ctx.L.bsb_sync(ctx.handle))
    ms = (ctypes.c_float * _lib.BSB_NUM_TILES)()
    assert ctx.L.bsb_last_tile_ms(ctx.handle, ms, _lib.BSB_NUM_TILES) == 0
    return do.cpu().numpy(), ctx.last_kernel_ms(), list(ms)


# scores above 15, gaps above 8000, gap extensions above 500: 32-bit cells, no ring
@pytest.mark.parametrize("scoring", [(20, 30, 60, 10, 50, 5, 400), (1, 4, 9000, 1, 6, 1, 100), (1, 4, 6, 501, 6, 1, 100)],
                         ids=["scores", "gap-opens", "gap-extensions"])
def test_device_batches_on_a_fresh_context_with_32_bit_cells(scoring):
    torch = pytest.importorskip("torch")
    a, b, o_del, e_del, o_ins, e_ins, zdrop = scoring
    ctx = extend.Context(0)
    try:
        for k in range(3):
            jobs, seq = synth.ksw_jobs(700 + k, seed=k, qmin=1, qmax=400)
            got, _, _ = run_device(torch, ctx, jobs, seq, scoring)
            ref, _ = oracle.ksw_batch(jobs, seq, synth.fill_scmat(a, b), o_del, e_del, o_ins, e_ins, zdrop, n_threads=8)
            assert np.array_equal(got, ref), f"batch {k}"
    finally:
        ctx.close()


def test_shape_times_add_up_with_the_cut_rings(gpu_ctx):
    """From 2^20 jobs on the shapes run one after the other, so their times and the scheduling make up the batch's."""
    torch = pytest.importorskip("torch")
    few, seq = synth.ksw_jobs(1 << 16, seed=5, qmin=10, qmax=300)
    jobs = np.tile(few, 16)
    scoring = (1, 4, 6, 1, 6, 1, 100)
    run_device(torch, gpu_ctx, jobs, seq, scoring)
    _, total, ms = run_device(torch, gpu_ctx, jobs, seq, scoring)
    G, C = (ctypes.c_int32 * _lib.BSB_NUM_TILES)(), (ctypes.c_int32 * _lib.BSB_NUM_TILES)()
    gpu_ctx.L.bsb_tile_shapes(G, C, _lib.BSB_NUM_TILES)
    by = {(G[t], C[t]): ms[t] for t in range(_lib.BSB_NUM_TILES)}
    assert all(by[32, c] > 0 for c in (7, 9, 11)), [by[32, c] for c in (7, 9, 11)]
    assert 0.75 * total < sum(ms) <= total * 1.01, (sum(ms), total)
