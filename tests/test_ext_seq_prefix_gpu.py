"""A host batch copies the part of the sequence buffer its jobs use, whatever the buffer's size: the time of a batch does
not grow with what lies behind."""
import time

import numpy as np
import pytest

from bsbolt_gb300 import extend, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["in-order", "shuffled"])
def test_unused_rest_of_the_buffer_costs_nothing(gpu_ctx, order):
    n = 300_000
    few, seq = synth.ksw_jobs(4096, seed=3)
    jobs = np.resize(few, n)
    if order == "shuffled":
        np.random.Generator(np.random.PCG64(1)).shuffle(jobs)
    wide = np.zeros(2000 * n, np.uint8)
    wide[:len(seq)] = seq
    mat = synth.fill_scmat(1, 4)

    def run(s):
        t = []
        for _ in range(6):
            t0 = time.perf_counter()
            out = extend.ksw_extend2_batch(gpu_ctx, jobs, s, mat, 6, 1, 6, 1, 100)
            t.append(time.perf_counter() - t0)
        return out, min(t)

    want, exact = run(seq)
    got, whole = run(wide)
    assert np.array_equal(got, want)
    # (600 MB take 2.5 ms and more on the way to the device, the jobs themselves 1.7)
    assert whole < 1.8 * exact, f"{whole * 1e3:.1f} ms with the buffer's rest, {exact * 1e3:.1f} without"
