"""The packed ksw_align2 passes where their groups, lane widths and scorings meet, against the oracle."""
import os
import sys

import numpy as np
import pytest

import oracle
from bsbolt_gb300 import matesw, synth

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
import golden_data  # noqa: E402

pytestmark = pytest.mark.gpu


def make_jobs(rng, n, qlens, minsc, flags):
    """Mates against windows with a mutated copy, jobs of different lengths next to one another."""
    jobs, parts, at = np.zeros(n, matesw.JOB_DTYPE), [], 0
    for k in range(n):
        ql = int(rng.choice(qlens))
        q = rng.integers(0, 4, ql).astype(np.uint8)
        copy = q.copy()
        mut = rng.random(ql) < rng.choice([0.0, 0.02, 0.15])
        copy[mut] = rng.integers(0, 5, int(mut.sum()))
        if ql > 8 and rng.random() < 0.4:
            p, g = int(rng.integers(1, ql - 1)), int(rng.integers(1, 7))
            copy = np.concatenate([copy[:p], copy[p + g:]]) if rng.random() < 0.5 else \
                np.concatenate([copy[:p], rng.integers(0, 4, g).astype(np.uint8), copy[p:]])
        sides = [rng.integers(0, 4, int(rng.integers(0, 90))).astype(np.uint8) for _ in range(2)]
        t = np.concatenate([sides[0], copy, sides[1]] + ([copy] if rng.random() < 0.3 else []))
        jobs[k] = (at, at + ql, ql, len(t), int(rng.choice(flags)) | int(rng.choice(minsc)), 0)
        parts += [q, t]
        at += ql + len(t)
    return jobs, np.concatenate(parts)


def check(ctx, jobs, seq, mat, o_del, e_del, o_ins, e_ins):
    got = matesw.align2_batch(ctx, jobs, seq, mat, o_del, e_del, o_ins, e_ins)
    want = oracle.align2_batch(jobs.view(golden_data.SW_JOB_DTYPE), seq, mat, o_del, e_del, o_ins, e_ins, n_threads=8)
    for f in ("score", "te", "qe", "score2", "te2", "tb", "qb"):
        bad = np.nonzero(got[f] != want[f])[0]
        assert len(bad) == 0, f"{f} differs at jobs {bad[:6]}: {got[f][bad[:6]]} vs {want[f][bad[:6]]}"


BYTE, STOP, SUBO, START = matesw.KSW_XBYTE, 0x20000, matesw.KSW_XSUBO, matesw.KSW_XSTART


# every bucket's edges in one list, both lane widths; thresholds of 0, of the usual size and above 16 bits' half;
# batches that leave groups of the last warp empty
@pytest.mark.parametrize("n", [1, 3, 5, 400])
@pytest.mark.parametrize("flags", [[BYTE | SUBO | START], [SUBO | START], [BYTE | START, BYTE | STOP, SUBO, BYTE, 0]])
def test_mixed_lengths(gpu_ctx, n, flags):
    rng = np.random.Generator(np.random.PCG64(n))
    jobs, seq = make_jobs(rng, n, [1, 15, 16, 17, 32, 33, 64, 65, 127, 128, 129, 192, 249, 256, 257, 320, 321],
                          [0, 19, 40, 0xffff], flags)
    check(gpu_ctx, jobs, seq, synth.fill_scmat(1, 4), 6, 1, 6, 1)


# scores that meet the byte lanes' ceiling, matrices whose smallest entry is 0 or above, penalties beyond every
# score, at the word lanes' limit, of gaps that open for nothing
@pytest.mark.parametrize("mat,pen", [
    (synth.fill_scmat(3, 2), (4, 1, 4, 1)), (synth.fill_scmat(100, 90), (6, 1, 6, 1)),
    (np.maximum(synth.fill_scmat(2, 3), 0), (6, 1, 6, 1)), (synth.fill_scmat(2, 3) + 4, (6, 1, 6, 1)),
    (synth.fill_scmat(100, 100), (300, 50, 32000, 700)), (synth.fill_scmat(1, 4), (32000, 767, 1, 32766)),
    (synth.fill_scmat(1, 4), (0, 0, 0, 0)), (synth.fill_scmat(1, 128), (0, 1, 0, 3))])
def test_scorings(gpu_ctx, mat, pen):
    rng = np.random.Generator(np.random.PCG64(7))
    jobs, seq = make_jobs(rng, 300, [16, 40, 100, 150, 249, 300], [0, 19], [BYTE | SUBO | START, SUBO | START])
    check(gpu_ctx, jobs, seq, np.asarray(mat, np.int8), *pen)
