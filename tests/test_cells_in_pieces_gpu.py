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
