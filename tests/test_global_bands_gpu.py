"""The global alignment's band forms (ksw_global.cuh) at the widths where they change, against the oracle."""
import numpy as np
import pytest

import oracle
from bsbolt_gb300 import cigar, index, seed, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def loaded(gpu_ctx, tmp_path_factory):
    d = tmp_path_factory.mktemp("bands")
    fa = str(d / "ref.fa")
    rng = np.random.Generator(np.random.PCG64(3))
    synth.write_fasta(fa, [("c1", rng.integers(0, 4, 20000).astype(np.uint8))])
    prefix = str(d / "ref")
    index.build_index(fa, prefix)
    seed.load_index(gpu_ctx, prefix)
    return gpu_ctx, index.BwaIndex(prefix)


# both sides of 2w + 1 = 64 and 128, the narrowest band, lengths around 32 and the staging limit of 256
@pytest.mark.parametrize("w", [1, 15, 31, 32, 63, 64, 90])
@pytest.mark.parametrize("length", [1, 31, 33, 256, 257, 420])
def test_bands_equal_the_oracle(loaded, w, length):
    ctx, bi = loaded
    rng = np.random.Generator(np.random.PCG64(1000 * w + length))
    codes, lp = bi.pac_codes(), bi.l_pac
    both = np.concatenate([codes, 3 - codes[::-1]]).astype(np.uint8)
    jobs, qs, at = [], [], 0
    for k in range(40):
        rb = int(rng.integers(10, lp - length - 300)) + (lp if k & 1 else 0)
        q = both[rb:rb + length].copy()
        mut = rng.random(length) < 0.03
        q[mut] = rng.integers(0, 5, int(mut.sum()))
        for _ in range(int(rng.integers(0, 4))):                  # gaps of either kind, up to the band
            p, g = int(rng.integers(0, len(q) + 1)), int(rng.integers(1, max(2, min(w, length // 3) + 1)))
            q = np.concatenate([q[:p], rng.integers(0, 4, g).astype(np.uint8), q[p:]]) if rng.random() < 0.5 else \
                np.concatenate([q[:p], q[p + g:]])
        if len(q) == 0:
            q = both[rb:rb + 1].copy()
        jobs.append((rb, rb + length + int(rng.integers(0, 3)), at, at, len(q), w))
        qs.append(q)
        at += len(q)
    jobs, qbuf = np.array(jobs, cigar.JOB_DTYPE), np.concatenate(qs)
    out, blob = cigar.gen_cigar_batch(ctx, jobs, qbuf, qbuf, bi.crick_l)
    want, wblob = oracle.gen_cigar_batch(synth.fill_scmat(1, 4), 6, 1, 6, 1, lp, bi.pac, bi.opac, bi.crick_l, jobs,
                                         qbuf, qbuf)
    for f in want.dtype.names:
        if f != "pad_":
            assert np.array_equal(out[f], want[f]), f
    assert np.array_equal(blob, wblob)
