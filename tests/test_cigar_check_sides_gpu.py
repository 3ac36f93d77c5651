"""bwa_gen_cigar2 batches on both sides of the line between jobs checked on the host and on the device: the same records,
the same refusals."""
import numpy as np
import pytest

import oracle
from bsbolt_gb300 import _lib, cigar, synth

from test_job_checks_gpu import loaded  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


def make(bi, n):
    codes = bi.pac_codes()
    rng = np.random.Generator(np.random.PCG64(n))
    jobs = np.zeros(n, cigar.JOB_DTYPE)
    jobs["rb"] = rng.integers(20, 5000, n)
    jobs["re"], jobs["l_query"], jobs["w"] = jobs["rb"] + 50 + rng.integers(-3, 4, n), 50, rng.integers(3, 30, n)
    jobs["qoff"] = jobs["ooff"] = np.arange(n) * 50
    q = codes[jobs["rb"][:, None] + np.arange(50)]
    return jobs, np.where(rng.random(q.shape) < 0.02, rng.integers(0, 4, q.shape), q).astype(np.uint8).reshape(-1)


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097])
def test_same_records(loaded, n):  # noqa: F811
    ctx, bi = loaded
    jobs, q = make(bi, n)
    out, blob = cigar.gen_cigar_batch(ctx, jobs, q, q, bi.crick_l)
    want, wblob = oracle.gen_cigar_batch(synth.fill_scmat(1, 4), 6, 1, 6, 1, bi.l_pac, bi.pac, bi.opac, bi.crick_l, jobs, q, q)
    for f in ("score", "n_cigar", "NM", "status"):
        assert np.array_equal(out[f], want[f]), f
    assert np.array_equal(blob, wblob)


@pytest.mark.parametrize("n", [4096, 4097])
@pytest.mark.parametrize("field,value,code", [("qoff", -1, "EINVAL"), ("ooff", 1 << 40, "EINVAL"), ("l_query", 1025, "ETOOLONG"),
                                              ("w", -1, "EINVAL")])
def test_same_refusals(loaded, n, field, value, code):  # noqa: F811
    ctx, bi = loaded
    jobs, q = make(bi, n)
    q = np.concatenate([q, np.zeros(2000, np.uint8)])
    for at in (0, 2000, n - 1):
        bad = jobs.copy()
        bad[field][at:] = value
        with pytest.raises(_lib.BsbError, match=f"job {at}:") as e:
            cigar.gen_cigar_batch(ctx, bad, q, q, bi.crick_l)
        assert e.value.code == getattr(_lib, "BSB_" + code)
