"""Reads that are left to the tree (two chains start at one place) are spread over the warps: thirty-two that take about
as long as one another alone take about that long together, and give the oracle's regions."""
import numpy as np
import pytest

import oracle
from bsbolt_gb300 import _lib, extend, index, seed, synth

pytestmark = pytest.mark.gpu


def test_reads_of_one_base(tmp_path):
    rng = np.random.Generator(np.random.PCG64(3))
    g = rng.integers(0, 4, 60_000).astype(np.uint8)
    g[10_000:50_000] = 0
    synth.write_fasta(str(tmp_path / "r.fa"), [("c", g)])
    index.build_index(str(tmp_path / "r.fa"), str(tmp_path / "r"))
    bi = index.BwaIndex(str(tmp_path / "r"))
    reads = []
    for k in range(40):
        r = np.zeros(100, np.uint8)
        e = rng.random(100) < 0.05
        r[e] = rng.integers(0, 4, int(e.sum()))
        reads.append(r.astype(np.uint8))
    ctx = extend.Context(0)
    try:
        seed.load_index(ctx, str(tmp_path / "r"))

        def run(some):
            offs, seqs = np.arange(len(some) + 1, dtype=np.int64) * 100, np.concatenate(some)
            ms = []
            for _ in range(3):
                regs, roff = seed.align_regs(ctx, seqs, offs, _lib.AlignOpt.bwa_defaults(w=20))
                ms.append(seed.last_stage_ms(ctx)["chains"])
            return seqs, offs, regs, roff, min(ms)

        ms = np.array([run([r])[4] for r in reads])
        at = np.argsort(ms)
        lo = min(range(len(reads) - 31), key=lambda k: ms[at[k + 31]] / ms[at[k]])        # the 32 most alike
        reads, alone = [reads[k] for k in at[lo:lo + 32]], float(ms[at[lo + 31]])
        seqs, offs, regs, roff, together = run(reads)
        ob = oracle.OracleBwt(bi.primary, bi.L2[1:], bi.bwt, bi.sa, bi.sa_intv)
        anns = np.array([(a.offset, a.len, 0) for a in bi.anns], dtype=oracle.ANN_DTYPE)
        oo = oracle.Opt.from_list([1, 4, 6, 1, 6, 1, 20, 100, 5, 5, 19, 500, 10, 20, 10000])
        want = oracle.align_regs(ob, anns, bi.pac, bi.l_pac, oo, seqs, offs, n_threads=8)
        assert np.array_equal(roff, want["regs_off"]) and np.diff(roff).max() > 64
        for f in want["regs"].dtype.names:
            assert np.array_equal(regs[f], want["regs"][f]), f"reg.{f}"
        print(f"{ms[at[lo]]:.2f} to {alone:.2f} ms alone, {together:.2f} for 32")
        assert together < 2 * alone, f"{together:.2f} ms for 32 reads, {alone:.2f} for one"
    finally:
        ctx.close()
