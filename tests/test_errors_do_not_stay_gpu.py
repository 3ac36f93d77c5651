"""A CUDA error that one call has reported is not met again by the next calls of the thread."""
import ctypes

import numpy as np
import pytest

import oracle
from bsbolt_gb300 import _lib, extend, index, matesw, synth

pytestmark = pytest.mark.gpu

MAT = synth.fill_scmat(1, 4)


def extension(ctx, tmp_path):
    jobs, seq = synth.ksw_jobs(200, seed=2)
    out = extend.ksw_extend2_batch(ctx, jobs, seq, MAT, 6, 1, 6, 1, 100)
    assert np.array_equal(out, oracle.ksw_batch(jobs, seq, MAT, 6, 1, 6, 1, 100)[0])


def rescue(ctx, tmp_path):
    jobs = np.zeros(3, matesw.JOB_DTYPE)
    jobs["qlen"], jobs["tlen"], jobs["xtra"] = 40, 90, matesw.matesw_xtra(40)
    matesw.align2_batch(ctx, jobs, np.zeros(90, np.uint8), MAT, 6, 1, 6, 1)


def build(ctx, tmp_path):
    synth.write_fasta(str(tmp_path / "r.fa"), synth.bs_genome(1, 5000, 0.4, 0.01, seed=1))
    index.build_index(str(tmp_path / "r.fa"), str(tmp_path / "r"), ctx=ctx)


@pytest.mark.parametrize("after", [extension, rescue, build], ids=lambda f: f.__name__)
def test_after_an_allocation_that_does_not_fit(tmp_path, after):
    """A sequence buffer of 2^45 bytes, of which the jobs use the first few (nothing behind them is read)."""
    ctx = extend.Context(0)
    try:
        jobs, seq = synth.ksw_jobs(4, seed=1)
        out, p = np.zeros((4, 6), np.int32), extend.make_param(MAT, 6, 1, 6, 1, 100)
        assert ctx.L.bsb_extend_batch(ctx.handle, ctypes.byref(p), jobs.ctypes.data, 4, seq.ctypes.data, 1 << 45,
                                      out.ctypes.data, None) == _lib.BSB_ENOMEM
        after(ctx, tmp_path)
    finally:
        ctx.close()
