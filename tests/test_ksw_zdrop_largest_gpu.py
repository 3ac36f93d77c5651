"""The largest z-drop, as good as none: the diagonal still answers its jobs (the time of a batch it decides whole), and
the results are the oracle's."""
import numpy as np
import pytest

import oracle
from bsbolt_gb300 import extend, synth

pytestmark = pytest.mark.gpu

MAT = synth.fill_scmat(1, 4)
LARGEST = 2**31 - 1


@pytest.mark.parametrize("zdrop", [LARGEST - 1, LARGEST])
def test_results(gpu_ctx, zdrop):
    jobs, seq = synth.ksw_jobs(20_000, seed=4, qmin=1, qmax=300, sub=0.02)
    want, _ = oracle.ksw_batch(jobs, seq, MAT, 6, 1, 6, 1, zdrop, n_threads=16)
    assert np.array_equal(extend.ksw_extend2_batch(gpu_ctx, jobs, seq, MAT, 6, 1, 6, 1, zdrop), want)


def test_exact_copies_are_answered_from_the_diagonal(gpu_ctx):
    few, seq = synth.ksw_jobs(1000, seed=4, qmin=100, qmax=140, sub=0.0, indel=0.0, unrelated=0.0)
    jobs = np.resize(few, 200_000)

    def ms(zdrop):
        t = []
        for _ in range(4):
            extend.ksw_extend2_batch(gpu_ctx, jobs, seq, MAT, 6, 1, 6, 1, zdrop)
            t.append(gpu_ctx.last_kernel_ms())
        return min(t)

    usual, largest = ms(100), ms(LARGEST)
    assert largest < 2 * usual, f"{largest:.3f} ms against {usual:.3f}"
