"""Chaining by a warp per read and, where chains start at the same place, by the reference's tree:
alignment regions against the oracle for reads that hold one reference stretch twice, further apart
than the band (so that a second chain starts where the first does), reads with few and with many
SA rows (beyond the rows kept in shared memory), chains of equal weight, and the chain options."""
import numpy as np
import pytest

import oracle
from bsbolt_gb300 import _lib, extend, index, seed, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def loaded(tmp_path_factory):
    rng = np.random.Generator(np.random.PCG64(5))
    g = rng.integers(0, 4, 60_000).astype(np.uint8)
    unit = rng.integers(0, 4, 400).astype(np.uint8)
    for k in range(70):                                   # a family of near-identical copies
        c = unit.copy()
        m = rng.random(len(c)) < 0.01 * (k % 4)
        c[m] = rng.integers(0, 4, int(m.sum()))
        g[500 + 800 * k:900 + 800 * k] = c
    d = tmp_path_factory.mktemp("chains")
    synth.write_fasta(str(d / "ref.fa"), [("a", g[:35_000]), ("b", g[35_000:])])
    index.build_index(str(d / "ref.fa"), str(d / "ref"))
    ctx = extend.Context(0)
    seed.load_index(ctx, str(d / "ref"))
    bi = index.BwaIndex(str(d / "ref"))
    yield ctx, bi
    ctx.close()


def make_reads(pac, rng):
    out = []
    for k in range(400):
        st = int(rng.integers(0, len(pac) - 700))
        kind = k % 5
        if kind == 0:                                     # one stretch twice, 110-200 bases apart
            a = pac[st:st + int(rng.integers(25, 60))]
            r = np.concatenate([a, rng.integers(0, 4, int(rng.integers(110, 200))), a])
            if k % 2:
                r = np.concatenate([r, pac[st + 300:st + 340], rng.integers(0, 4, 120), a[:24], pac[st + 300:st + 330]])
        elif kind == 1:                                   # inside the family: many rows
            r = pac[520 + 800 * (k % 60):][: int(rng.integers(100, 350))]
        elif kind == 2:                                   # many short pieces: chains of equal weight
            r = np.concatenate([pac[s:s + 22] for s in rng.integers(0, len(pac) - 30, 8)])
        else:
            r = pac[st:st + int(rng.integers(30, 400))]
        r = np.array(r, np.uint8)
        if k % 3 == 0:
            r = (3 - r[::-1]).astype(np.uint8)
        e = rng.random(len(r)) < 0.01
        r[e] = rng.integers(0, 5, int(e.sum()))
        out.append(r)
    return out


@pytest.mark.parametrize("changes", [{}, {"w": 20, "max_chain_gap": 60}, {"max_occ": 20},
                                     {"min_chain_weight": 25}, {"max_chain_extend": 2}],
                         ids=lambda c: ",".join(c) or "defaults")
def test_regions_equal_the_oracle(loaded, changes):
    ctx, bi = loaded
    reads = make_reads(bi.pac_codes(), np.random.Generator(np.random.PCG64(9)))
    offs = np.zeros(len(reads) + 1, np.int64)
    offs[1:] = np.cumsum([len(r) for r in reads])
    seqs = np.concatenate(reads)
    o = [1, 4, 6, 1, 6, 1, 100, 100, 5, 5, 19, 500, 10, 20, 10000]
    opt = _lib.AlignOpt.bwa_defaults()
    oo = oracle.Opt.from_list(o)
    for k, v in changes.items():
        setattr(opt, k, v)
        setattr(oo, k, v)
    ob = oracle.OracleBwt(bi.primary, bi.L2[1:], bi.bwt, bi.sa, bi.sa_intv)
    anns = np.array([(a.offset, a.len, 0) for a in bi.anns], dtype=oracle.ANN_DTYPE)
    want = oracle.align_regs(ob, anns, bi.pac, bi.l_pac, oo, seqs, offs, n_threads=8)
    regs, roff = seed.align_regs(ctx, seqs, offs, opt)
    assert np.array_equal(roff, want["regs_off"])
    for f in want["regs"].dtype.names:
        assert np.array_equal(regs[f], want["regs"][f]), f"reg.{f}"


@pytest.mark.parametrize("changes", [{}, {"pen_clip5": 30, "pen_clip3": 30, "zdrop": 20}, {"w": 6, "zdrop": 0},
                                     {"a": 2, "b": 3, "o_del": 4, "e_del": 2}, {"o_ins": 9000}],
                         ids=lambda c: ",".join(c) or "defaults")
def test_large_batches_equal_small_ones(loaded, changes):
    """From 4096 reads on the chains' first extensions run as batches of their own (on 16-bit cells;
    scorings that need 32-bit ones stay with the read's warp); the regions are those of small batches."""
    ctx, bi = loaded
    pac = bi.pac_codes()
    rng = np.random.Generator(np.random.PCG64(21))
    reads = []
    for k in range(11):
        reads += make_reads(pac, rng)
    offs = np.zeros(len(reads) + 1, np.int64)
    offs[1:] = np.cumsum([len(r) for r in reads])
    seqs = np.concatenate(reads)
    opt = _lib.AlignOpt.bwa_defaults(a=changes.get("a", 1), b=changes.get("b", 4))
    for k, v in changes.items():
        setattr(opt, k, v)
    assert len(reads) >= 4096
    regs, roff = seed.align_regs(ctx, seqs, offs, opt)
    for lo in range(0, len(reads), 2000):
        hi = min(lo + 2000, len(reads))
        part, poff = seed.align_regs(ctx, seqs[offs[lo]:offs[hi]], offs[lo:hi + 1] - offs[lo], opt)
        assert np.array_equal(roff[lo:hi + 1] - roff[lo], poff)
        assert regs[roff[lo]:roff[hi]].tobytes() == part.tobytes()


@pytest.mark.parametrize("redun,gap", [(0.95, 10000), (0.5, 10000), (0.95, 60)])
def test_dedup_equals_the_oracle(loaded, redun, gap):
    """mem_sort_dedup_patch on reads with one to more than 64 regions, many of them with equal ends or
    equal scores and starts."""
    ctx, bi = loaded
    reads = make_reads(bi.pac_codes(), np.random.Generator(np.random.PCG64(13)))
    offs = np.zeros(len(reads) + 1, np.int64)
    offs[1:] = np.cumsum([len(r) for r in reads])
    seqs = np.concatenate(reads)
    opt = _lib.AlignOpt.bwa_defaults(max_chain_gap=gap)
    oo = oracle.Opt.from_list([1, 4, 6, 1, 6, 1, 100, 100, 5, 5, 19, 500, 10, 20, gap])
    opt.mask_level_redun = oo.mask_level_redun = redun
    regs, roff = seed.align_regs(ctx, seqs, offs, opt)
    n = np.diff(roff)
    assert n.max() > 64 and (n == 1).any() and (n == 2).any()
    want, woff = oracle.sort_dedup_batch(oo, bi.l_pac, bi.pac, seqs, offs, regs, roff)
    got, goff = seed.align_regs(ctx, seqs, offs, opt, dedup=True)
    assert np.array_equal(goff, woff)
    for f in want.dtype.names:
        assert np.array_equal(got[f], want[f]), f"reg.{f}"
