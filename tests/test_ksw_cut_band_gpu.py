"""Jobs whose band is cut (cut_band, ksw_core.cuh) in batches large enough for it, against the oracle: losses along the
main diagonal on both sides of each ring's reach, few bases ahead of them (low h0), gaps and better paths beside the
diagonal, targets that end at or just behind the query, z-drops and bands near the cut."""
import numpy as np
import pytest

import oracle
from bsbolt_gb300 import extend, synth

pytestmark = pytest.mark.gpu


def make(rng, n, lengths, a, b):
    rows, parts, at = [], [], 0
    for k in range(n):
        ql = int(rng.choice(lengths))
        unit = rng.integers(0, 4, int(rng.choice([2, 3, 7, 400])))       # repeats: other diagonals match as well
        q = np.resize(unit, ql).astype(np.uint8)
        t = q.copy()
        for p in rng.integers(0, ql, int(rng.integers(1, 11))):
            t[p] = rng.integers(0, 5)
        if rng.random() < 0.2:
            q[int(rng.integers(0, ql))] = 4
        if rng.random() < 0.4:                                          # a gap soon made good by another, or not
            c, g = int(rng.integers(0, ql)), int(rng.integers(1, 8))
            t = np.concatenate([t[:c], rng.integers(0, 4, g).astype(np.uint8), t[c:]])
            if rng.random() < 0.6:
                c = min(len(t) - g, c + int(rng.integers(1, 40)))
                t = np.concatenate([t[:c], t[c + g:]])
        kind = int(rng.integers(0, 4))
        if kind == 0:
            t = t[:ql + int(rng.integers(-1, 3))]
        elif kind == 1:
            t = np.concatenate([t, q[-30:], rng.integers(0, 4, 60).astype(np.uint8)])   # the query's end again
        elif kind == 2:
            t = np.concatenate([t, rng.integers(0, 4, int(rng.integers(0, 100))).astype(np.uint8)])
        rows.append((at, at + ql, ql, len(t), int(rng.choice([5, 12, 20, 35, 60, 100])),
                     int(rng.choice([8, 11, 12, 20, 24, 47, 48, 100])), int(rng.choice([0, 5, 30])), 0))
        parts += [q, t]
        at += ql + len(t)
    return np.array(rows, dtype=synth.JOB_DTYPE), np.concatenate(parts)


@pytest.mark.parametrize("scoring", [(1, 4, 6, 1, 6, 1, 100), (1, 4, 6, 1, 6, 1, 25), (2, 3, 5, 2, 8, 1, 0),
                                     (1, 1, 0, 1, 2, 1, 100), (1, 2, 12, 3, 4, 2, 60)],
                         ids=["bwa", "small-zdrop", "asymmetric", "cheap-gaps", "dear-deletions"])
@pytest.mark.parametrize("per_sm,lengths", [(1301, [64, 65, 80, 96, 97, 120, 140, 143, 144, 145, 200, 300]),
                                            (120, [143, 144, 145, 180, 224, 300, 500, 990, 991, 992])],
                         ids=["first-map", "second-map"])
def test_cut_bands(gpu_ctx, scoring, per_sm, lengths):
    torch = pytest.importorskip("torch")
    a, b, o_del, e_del, o_ins, e_ins, zdrop = scoring
    few, seq = make(np.random.Generator(np.random.PCG64(17)), 4000, lengths, a, b)
    mat = synth.fill_scmat(a, b)
    ref, _ = oracle.ksw_batch(few, seq, mat, o_del, e_del, o_ins, e_ins, zdrop, n_threads=16)
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    times = (n + len(few) - 1) // len(few)
    jobs = np.tile(few, times)
    out = extend.ksw_extend2_batch(gpu_ctx, jobs, seq, mat, o_del, e_del, o_ins, e_ins, zdrop)
    for k in range(times):
        part = out[k * len(few):(k + 1) * len(few)]
        if not np.array_equal(part, ref):
            bad = np.nonzero([x != y for x, y in zip(part.tolist(), ref.tolist())])[0]
            raise AssertionError(f"jobs {bad[:5]}: {part[bad[:5]]} vs {ref[bad[:5]]}, {few[bad[:5]]}")
