"""Batches whose jobs are checked on the device: every kind of unfit job is refused with its code, the first one is
named, nothing is written, and the batch without it gives the oracle's records."""
import numpy as np
import pytest

import oracle
from bsbolt_gb300 import _lib, cigar, index, matesw, seed, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def loaded(gpu_ctx, tmp_path_factory):
    d = tmp_path_factory.mktemp("checks")
    fa = str(d / "ref.fa")
    rng = np.random.Generator(np.random.PCG64(9))
    synth.write_fasta(fa, [("c1", rng.integers(0, 4, 6000).astype(np.uint8))])
    prefix = str(d / "ref")
    index.build_index(fa, prefix)
    seed.load_index(gpu_ctx, prefix)
    return gpu_ctx, index.BwaIndex(prefix)


CIGAR_FAULTS = [("qoff", -1, "EINVAL"), ("qoff", 17000 - 49, "EINVAL"), ("ooff", -1, "EINVAL"),
                ("ooff", 17000 - 49, "EINVAL"), ("l_query", 1025, "ETOOLONG"), ("w", -1, "EINVAL"),
                ("re", 3000 + 1025, "ETOOLONG")]


@pytest.mark.parametrize("field,value,code", CIGAR_FAULTS)
@pytest.mark.parametrize("at", [0, 150, 299])
def test_cigar_jobs(loaded, field, value, code, at):
    ctx, bi = loaded
    codes = bi.pac_codes()
    jobs = np.zeros(300, cigar.JOB_DTYPE)
    jobs["rb"] = np.arange(300) * 10 + 20
    jobs["re"], jobs["l_query"], jobs["w"] = jobs["rb"] + 50, 50, np.arange(300) % 7
    jobs["qoff"] = jobs["ooff"] = np.arange(300) * 50
    qbuf = np.concatenate([codes[b:b + 50] for b in jobs["rb"]] + [codes[:2000]]).astype(np.uint8)
    bad = jobs.copy()
    if field == "re":
        bad["rb"][at:] = 3000
    bad[field][at:] = value                      # the jobs behind it are unfit too
    with pytest.raises(_lib.BsbError, match=f"job {at}:") as e:
        cigar.gen_cigar_batch(ctx, bad, qbuf, qbuf, bi.crick_l)
    assert e.value.code == getattr(_lib, "BSB_" + code)
    out, blob = cigar.gen_cigar_batch(ctx, jobs, qbuf, qbuf, bi.crick_l)
    want, wblob = oracle.gen_cigar_batch(synth.fill_scmat(1, 4), 6, 1, 6, 1, bi.l_pac, bi.pac, bi.opac, bi.crick_l,
                                         jobs, qbuf, qbuf)
    assert np.array_equal(out["score"], want["score"]) and np.array_equal(blob, wblob)


@pytest.mark.parametrize("field,value,code", [("qoff", -1, "EINVAL"), ("qoff", 30000 - 59, "EINVAL"),
                                              ("toff", -1, "EINVAL"), ("toff", 30000 - 149, "EINVAL"),
                                              ("qlen", -1, "EINVAL"), ("tlen", -1, "EINVAL"),
                                              ("qlen", 1025, "ETOOLONG")])
@pytest.mark.parametrize("at", [0, 150, 299])
def test_mate_rescue_jobs(gpu_ctx, field, value, code, at):
    rng = np.random.Generator(np.random.PCG64(at))
    seq = rng.integers(0, 4, 30000).astype(np.uint8)
    jobs = np.zeros(300, matesw.JOB_DTYPE)
    jobs["qoff"], jobs["toff"], jobs["qlen"], jobs["tlen"] = np.arange(300) * 60, np.arange(300) * 60, 60, 150
    jobs["xtra"] = np.where(np.arange(300) % 3, matesw.matesw_xtra(60), matesw.KSW_XSTART)
    bad = jobs.copy()
    bad[field][at:] = value
    with pytest.raises(_lib.BsbError, match=f"job {at}:") as e:
        matesw.align2_batch(gpu_ctx, bad, seq, synth.fill_scmat(1, 4), 6, 1, 6, 1)
    assert e.value.code == getattr(_lib, "BSB_" + code)
    got = matesw.align2_batch(gpu_ctx, jobs, seq, synth.fill_scmat(1, 4), 6, 1, 6, 1)
    want = oracle.align2_batch(jobs, seq, synth.fill_scmat(1, 4), 6, 1, 6, 1)
    for f in want.dtype.names:
        if f in got.dtype.names:
            assert np.array_equal(got[f], want[f]), f


@pytest.mark.parametrize("field,value,code", [("qoff", -1, "EINVAL"), ("toff", 1 << 40, "EINVAL"), ("qlen", -1, "EINVAL"),
                                              ("qlen", 1024, "ETOOLONG"), ("tlen", -1, "EINVAL"), ("w", -1, "EINVAL"),
                                              ("h0", 0, "EINVAL"), ("h0", (1 << 20) + 1, "EINVAL"), ("flags", 1, "EINVAL")])
@pytest.mark.parametrize("n", [4095, 4096])              # checked on the host, on the device
def test_extension_jobs(gpu_ctx, field, value, code, n):
    from bsbolt_gb300 import extend
    jobs, seq = synth.ksw_jobs(n, seed=3, qmin=1, qmax=300)
    mat = synth.fill_scmat(1, 4)
    for at in (0, 1000, n - 1):
        bad = jobs.copy()
        bad[field][at:] = value
        with pytest.raises(_lib.BsbError, match=f"job {at}:") as e:
            extend.ksw_extend2_batch(gpu_ctx, bad, np.concatenate([seq, np.zeros(2000, np.uint8)]), mat, 6, 1, 6, 1, 100)
        assert e.value.code == getattr(_lib, "BSB_" + code)
    want, _ = oracle.ksw_batch(jobs, seq, mat, 6, 1, 6, 1, 100, n_threads=8)
    assert np.array_equal(extend.ksw_extend2_batch(gpu_ctx, jobs, seq, mat, 6, 1, 6, 1, 100), want)
    # a buffer of which the jobs use a small part
    wide = np.concatenate([seq, np.zeros(4096 * 2048 + (1 << 20), np.uint8)])
    assert np.array_equal(extend.ksw_extend2_batch(gpu_ctx, jobs, wide, mat, 6, 1, 6, 1, 100), want)
