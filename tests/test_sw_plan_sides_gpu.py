"""ksw_align2 batches on both sides of the line between the lists made on the host and on the device: the same results,
the same refusals."""
import numpy as np
import pytest

import oracle
from bsbolt_gb300 import _lib, matesw, synth

from test_sw_forms_gpu import BYTE, START, STOP, SUBO, golden_data, make_jobs

pytestmark = pytest.mark.gpu

MAT = synth.fill_scmat(1, 4)


@pytest.fixture(scope="module")
def mixed():
    """Jobs of every list: packed byte and word lanes, one-lane byte (over 256 bases) and word jobs (over 320)."""
    jobs, seq = make_jobs(np.random.Generator(np.random.PCG64(5)), 241, [1, 16, 40, 128, 129, 250, 256, 257, 320, 321, 500],
                          [0, 19, 40], [BYTE | SUBO | START, SUBO | START, BYTE | START, BYTE | STOP, SUBO, 0])
    want = oracle.align2_batch(jobs.view(golden_data.SW_JOB_DTYPE), seq, MAT, 6, 1, 6, 1, n_threads=8)
    return jobs, seq, want


@pytest.mark.parametrize("n", [1, 2, 8191, 8192, 8193, 20_000])
def test_same_results(gpu_ctx, mixed, n):
    jobs, seq, want = mixed
    got = matesw.align2_batch(gpu_ctx, np.resize(jobs, n), seq, MAT, 6, 1, 6, 1)
    for f in ("score", "te", "qe", "score2", "te2", "tb", "qb"):
        assert np.array_equal(got[f], np.resize(want[f], n)), f


@pytest.mark.parametrize("n", [8192, 8193])
@pytest.mark.parametrize("field,value,code", [("qoff", -1, "EINVAL"), ("toff", 1 << 40, "EINVAL"), ("tlen", -1, "EINVAL"),
                                              ("qlen", 1025, "ETOOLONG")])
def test_same_refusals(gpu_ctx, mixed, n, field, value, code):
    jobs, seq, _ = mixed
    for at in (0, 5000, n - 1):
        bad = np.resize(jobs, n)
        bad["qoff"] = bad["toff"] = 0                   # (so that only the field given is at fault)
        bad[field][at:] = value
        with pytest.raises(_lib.BsbError, match=f"job {at}:") as e:
            matesw.align2_batch(gpu_ctx, bad, seq, MAT, 6, 1, 6, 1)
        assert e.value.code == getattr(_lib, "BSB_" + code)
