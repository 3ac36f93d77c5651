"""Batches of 4096 reads of 600-1023 bases, whose chains' first extensions run as batches on the widest shapes, against
the oracle: exact only at one end or in the middle, so that an extension takes the read's whole length, on both strands
and up to the largest score that 16-bit cells hold (1023 bases, match score 1)."""
import os

import numpy as np
import pytest

import oracle
from bsbolt_gb300 import _lib, extend, index, seed, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def loaded(tmp_path_factory):
    rng = np.random.Generator(np.random.PCG64(41))
    g = rng.integers(0, 4, 400_000).astype(np.uint8)
    for k in range(12):                                    # a few copies, with differences
        c = g[3000:4500].copy()
        m = rng.random(len(c)) < 0.03
        c[m] = rng.integers(0, 4, int(m.sum()))
        g[20_000 + 9000 * k:20_000 + 9000 * k + len(c)] = c
    d = tmp_path_factory.mktemp("long")
    synth.write_fasta(str(d / "ref.fa"), [("a", g[:150_000]), ("b", g[150_000:])])
    index.build_index(str(d / "ref.fa"), str(d / "ref"))
    ctx = extend.Context(0)
    seed.load_index(ctx, str(d / "ref"))
    yield ctx, index.BwaIndex(str(d / "ref"))
    ctx.close()


def make_reads(pac, n, rng):
    out = []
    for k in range(n):
        L = 1023 if k % 5 == 0 else int(rng.integers(600, 1024))
        st = int(rng.integers(0, len(pac) - L - 20)) if k % 4 else 20_000 + 9000 * (k // 4 % 12)
        r = pac[st:st + L + 20].copy()
        e = rng.random(len(r)) < rng.choice([0.03, 0.06, 0.10])
        at = (0, L - 40, int(rng.integers(0, L - 40)))[k % 3]          # the stretch that stays exact
        e[at:at + 40] = False
        r[e] = rng.integers(0, 5, int(e.sum()))
        for _ in range(int(rng.integers(0, 4))):                     # gaps, outside that stretch
            p, gap = int(rng.integers(1, L)), int(rng.integers(1, 9))
            if not at - gap <= p <= at + 40:
                r = np.delete(r, np.s_[p:p + gap]) if rng.random() < 0.5 else \
                    np.insert(r, p, rng.integers(0, 4, gap).astype(np.uint8))
        if k % 7 == 0:                                               # the far half is something else
            h = slice(L // 2, None) if at < L // 2 else slice(0, L // 2)
            r[h] = rng.integers(0, 4, len(r[h]))
        r = r[:L].astype(np.uint8)
        out.append((np.where(r < 4, 3 - r, 4)[::-1] if k % 2 else r).astype(np.uint8))
    return out


@pytest.mark.parametrize("changes", [{}, {"pen_clip5": 30, "pen_clip3": 30, "zdrop": 40}, {"w": 30, "zdrop": 0}],
                         ids=lambda c: ",".join(c) or "defaults")
def test_regions_equal_the_oracle(loaded, changes):
    ctx, bi = loaded
    reads = make_reads(bi.pac_codes(), 4096, np.random.Generator(np.random.PCG64(43)))
    offs = np.zeros(len(reads) + 1, np.int64)
    offs[1:] = np.cumsum([len(r) for r in reads])
    assert np.diff(offs).max() == 1023 and np.diff(offs).min() >= 590
    seqs = np.concatenate(reads)
    opt, oo = _lib.AlignOpt.bwa_defaults(), oracle.Opt.from_list([1, 4, 6, 1, 6, 1, 100, 100, 5, 5, 19, 500, 10, 20, 10000])
    for k, v in changes.items():
        setattr(opt, k, v)
        setattr(oo, k, v)
    ob = oracle.OracleBwt(bi.primary, bi.L2[1:], bi.bwt, bi.sa, bi.sa_intv)
    anns = np.array([(a.offset, a.len, 0) for a in bi.anns], dtype=oracle.ANN_DTYPE)
    want = oracle.align_regs(ob, anns, bi.pac, bi.l_pac, oo, seqs, offs, n_threads=os.cpu_count() or 8)
    regs, roff = seed.align_regs(ctx, seqs, offs, opt)
    assert np.array_equal(roff, want["regs_off"])
    for f in want["regs"].dtype.names:
        bad = np.nonzero(regs[f] != want["regs"][f])[0]
        assert len(bad) == 0, f"reg.{f} at {bad[:5]}: {regs[bad[:5]]} vs {want['regs'][bad[:5]]}"
    assert len(seed.last_read_order(ctx, 4096)) < 4096       # the first extensions did run ahead
