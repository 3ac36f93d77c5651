"""Alignments in bands of 61 cost what their cells do: at most twice the time of bands of 20 (three times the cells, beside
what all jobs pay; their directions written a byte at a time took two and a half times as long)."""
import time

import numpy as np
import pytest

from bsbolt_gb300 import cigar

from test_global_bands_gpu import loaded  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


def test_time_of_a_wide_band(loaded):  # noqa: F811
    ctx, bi = loaded
    codes, n, length = bi.pac_codes(), 20_000, 250
    rng = np.random.Generator(np.random.PCG64(2))
    jobs = np.zeros(n, cigar.JOB_DTYPE)
    jobs["rb"] = rng.integers(10, len(codes) - 600, n)
    jobs["re"], jobs["l_query"] = jobs["rb"] + length + rng.integers(0, 6, n), length
    jobs["qoff"] = jobs["ooff"] = np.arange(n) * length
    q = codes[jobs["rb"][:, None] + np.arange(length)]
    q = np.where(rng.random(q.shape) < 0.03, rng.integers(0, 4, q.shape), q).astype(np.uint8).reshape(-1)

    def best(w):
        jobs["w"] = w
        t = []
        for _ in range(5):
            t0 = time.perf_counter()
            cigar.gen_cigar_batch(ctx, jobs, q, q, bi.crick_l)
            t.append(time.perf_counter() - t0)
        return min(t)

    narrow, wide = best(20), best(60)
    print(f"{narrow * 1e3:.2f} ms, {wide * 1e3:.2f} wide")
    assert wide < 2 * narrow, f"{wide * 1e3:.2f} ms against {narrow * 1e3:.2f}"
