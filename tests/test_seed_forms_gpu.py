"""Seeding over the options and read shapes its kernels branch on, against the oracle: reads up to
the longest accepted, N at every place, tiny and repetitive references, seed lengths from 1 up,
re-seed thresholds, and batches from one read to more than a warp's worth."""
import numpy as np
import pytest

import oracle
from bsbolt_gb300 import extend, index, seed, synth

pytestmark = pytest.mark.gpu


def references():
    rng = np.random.Generator(np.random.PCG64(3))
    tiny = rng.integers(0, 4, 150).astype(np.uint8)
    unit = rng.integers(0, 4, 37).astype(np.uint8)
    tandem = np.concatenate([rng.integers(0, 4, 500), np.tile(unit, 40), np.zeros(300), rng.integers(0, 4, 700)])
    three = np.array([0, 2, 3, 3], np.uint8)[rng.integers(0, 4, 60_000)]
    three[30_000:36_000] = three[1000:7000]
    return {"tiny": tiny, "tandem": tandem.astype(np.uint8), "three-letter": three}


@pytest.fixture(scope="module", params=["tiny", "tandem", "three-letter"])
def loaded(request, tmp_path_factory):
    d = tmp_path_factory.mktemp("forms")
    fa, prefix = str(d / "ref.fa"), str(d / "ref")
    synth.write_fasta(fa, [("c", references()[request.param])])
    index.build_index(fa, prefix)
    ctx = extend.Context(0)
    seed.load_index(ctx, prefix)
    bi = index.BwaIndex(prefix)
    yield ctx, bi, oracle.OracleBwt(bi.primary, bi.L2[1:], bi.bwt, bi.sa, bi.sa_intv)
    ctx.close()


def reads_of(pac, n, longest, rng):
    out = []
    for k in range(n):
        L = int(rng.integers(1, longest + 1)) if k % 4 else longest
        L = min(L, len(pac) - 1)
        st = int(rng.integers(0, len(pac) - L))
        r = pac[st:st + L].copy()
        if k % 2:
            r = (3 - r[::-1]).astype(np.uint8)
        if k % 3 == 0:
            e = rng.random(L) < 0.03
            r[e] = rng.integers(0, 5, int(e.sum()))
        if k % 7 == 0:
            r[(np.arange(L) + k) % (11 + k % 20) == 0] = 4
        if k % 5 == 0 and L > 60:              # two pieces from different places
            r[L // 2:] = pac[:L - L // 2] if k % 2 else rng.integers(0, 4, L - L // 2)
        out.append(r.astype(np.uint8))
    return out


@pytest.mark.parametrize("n,longest", [(1, 100), (33, 1024), (700, 150)])
@pytest.mark.parametrize("msl,width,intv", [(19, 10, 20), (1, 3, 20), (11, 10, 0), (12, 40, 20), (13, 0, 5)])
def test_seeds_equal_the_oracle(loaded, n, longest, msl, width, intv):
    ctx, bi, ob = loaded
    rng = np.random.Generator(np.random.PCG64(100 * n + msl))
    reads = reads_of(bi.pac_codes(), n, longest, rng)
    offs = np.zeros(len(reads) + 1, np.int64)
    offs[1:] = np.cumsum([len(r) for r in reads])
    seqs = np.concatenate(reads)
    want, woff = ob.collect_intv(seqs, offs, min_seed_len=msl, split_width=width, max_mem_intv=intv, n_threads=8)
    lens = np.diff(offs)
    got, off = seed.seed_batch(ctx, seqs, offs, min_seed_len=msl, split_width=width, max_mem_intv=intv)
    for r in range(n):
        exp = want[woff[r]:woff[r + 1]] if lens[r] >= msl else want[:0]
        assert np.array_equal(got[off[r]:off[r + 1]], exp), f"read {r} of {lens[r]} bases"
