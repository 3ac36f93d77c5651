"""ksw_align2 with a matrix of positive entries only: byte-lane jobs run on the packed kernels like any others, with the
oracle's results (every H stays 0 there) and in their time."""
import time

import numpy as np
import pytest

from bsbolt_gb300 import matesw, synth

from test_sw_forms_gpu import BYTE, START, STOP, SUBO, check, make_jobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mat", [synth.fill_scmat(2, 3) + 4, synth.fill_scmat(60, 5) + 8, np.full(25, 127), np.full(25, 1),
                                 np.arange(25) + 100], ids=["min-1", "min-3", "all-127", "all-1", "100-124"])
@pytest.mark.parametrize("minsc", [[0], [0, 1, 19, 254, 255]])
def test_results(gpu_ctx, mat, minsc):
    rng = np.random.Generator(np.random.PCG64(7))
    jobs, seq = make_jobs(rng, 300, [1, 16, 17, 40, 100, 150, 249, 256, 257, 300], minsc,
                          [BYTE | SUBO | START, BYTE | START, BYTE | STOP, BYTE, SUBO | START])
    check(gpu_ctx, jobs, seq, np.asarray(mat).astype(np.int8), 6, 1, 6, 1)


def test_time(gpu_ctx):
    """40k mates of 150 bases: the one-lane kernels take 3.0 ms with such a matrix, the packed ones 0.6 (and 1.3 with the
    usual one, where H is not always 0)."""
    few, seq = make_jobs(np.random.Generator(np.random.PCG64(7)), 500, [150], [19], [BYTE | SUBO | START])
    jobs = np.resize(few, 40_000)

    def best(mat):
        t = []
        for _ in range(5):
            t0 = time.perf_counter()
            matesw.align2_batch(gpu_ctx, jobs, seq, np.asarray(mat, np.int8), 6, 1, 6, 1)
            t.append(time.perf_counter() - t0)
        return min(t)

    usual, positive = best(synth.fill_scmat(1, 4)), best(synth.fill_scmat(2, 3) + 4)
    print(f"{usual * 1e3:.2f} ms, {positive * 1e3:.2f} with positive entries only")
    assert positive < 1.5 * usual, f"{positive * 1e3:.2f} ms against {usual * 1e3:.2f}"
