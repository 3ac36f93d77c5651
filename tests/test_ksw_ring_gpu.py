"""Long queries whose registers move along with a narrow band (ksw_tiles.cuh, the ring): both sides of each of its
limits, with and without cell counts, host and device entry, against the oracle."""
import numpy as np
import pytest

import oracle
from bsbolt_gb300 import extend, synth

pytestmark = pytest.mark.gpu


def long_jobs(seed, n=700):
    """Queries around the ring's width, a multiple of its columns, and its longest; targets with substitutions, Ns and
    gaps up to the band, too short, unrelated halfway or with a flank; bands on both sides of the widest that fits."""
    rng = np.random.Generator(np.random.PCG64(seed))
    parts, rows, base = [], [], 0
    lengths = [200, 222, 223, 224, 225, 238, 239, 255, 256, 257, 264, 300, 336, 448, 449, 600, 700, 1008, 1009, 1010, 1015, 1016, 1023]
    for k in range(n):
        qlen = int(lengths[k % len(lengths)])
        w = int(rng.choice([0, 1, 7, 13, 14, 15, 60, 100, 103, 104, 105, 123, 124, 200]))
        q = rng.integers(0, 4, qlen).astype(np.uint8)
        q[rng.random(qlen) < 0.01] = 4
        t = q.copy()
        mut = rng.random(qlen) < rng.choice([0.0, 0.01, 0.1])
        t[mut] = rng.integers(0, 5, int(mut.sum()))
        for _ in range(int(rng.integers(0, 5))):
            c, g = int(rng.integers(0, len(t))), int(rng.integers(1, max(2, w + 2)))
            t = np.concatenate([t[:c], t[c + g:]]) if rng.random() < 0.5 else \
                np.concatenate([t[:c], rng.integers(0, 4, g).astype(np.uint8), t[c:]])
        kind = int(rng.integers(0, 5))
        if kind == 0:
            t = t[:max(1, int(rng.integers(0, len(t) + 1)))]
        elif kind == 1:
            t = np.concatenate([t, q[-60:], rng.integers(0, 4, 100).astype(np.uint8)])
        elif kind == 2:
            c = len(t) // 2
            t = np.concatenate([t[:c], rng.integers(0, 4, qlen).astype(np.uint8)])
        h0 = int(rng.choice([1, 19, 60, 300, 800, 1500]))
        rows.append((base, base + qlen, qlen, len(t), h0, w, int(rng.choice([0, 5, 30])), 0))
        parts += [q, t]
        base += qlen + len(t)
    return np.array(rows, dtype=synth.JOB_DTYPE), np.concatenate(parts)


@pytest.mark.parametrize("scoring", [(1, 4, 6, 1, 6, 1, 100), (1, 4, 6, 1, 6, 1, 0), (1, 2, 3, 2, 9, 1, 40),
                                     (1, 1, 0, 1, 0, 1, 100), (2, 3, 300, 30, 5, 2, 200)],
                         ids=["bwa", "no-zdrop", "asymmetric", "no-gap-open", "dear-deletions"])
@pytest.mark.parametrize("times", [1, 12], ids=["warp-a-job", "two-a-warp"])
def test_ring_equals_the_oracle(gpu_ctx, scoring, times):
    torch = pytest.importorskip("torch")
    a, b, o_del, e_del, o_ins, e_ins, zdrop = scoring
    jobs, seq = long_jobs(11)
    jobs = np.tile(jobs, times)
    mat = synth.fill_scmat(a, b)
    ref, rcells = oracle.ksw_batch(jobs, seq, mat, o_del, e_del, o_ins, e_ins, zdrop, n_threads=16)
    for lo in (0, 1, len(jobs) - 1):                                       # a full batch, and ends that leave groups without a job
        out = extend.ksw_extend2_batch(gpu_ctx, jobs[lo:], seq, mat, o_del, e_del, o_ins, e_ins, zdrop)
        assert np.array_equal(out, ref[lo:])
    out, cells = extend.ksw_extend2_batch(gpu_ctx, jobs, seq, mat, o_del, e_del, o_ins, e_ins, zdrop, want_cells=True)
    assert np.array_equal(out, ref) and np.array_equal(cells, rcells)
    dj, ds = torch.from_numpy(jobs.view(np.uint8).copy()).cuda(), torch.from_numpy(seq).cuda()
    do = torch.zeros((len(jobs), 6), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    extend.ksw_extend2_device(gpu_ctx, dj.data_ptr(), len(jobs), ds.data_ptr(), len(seq),
                              extend.make_param(mat, o_del, e_del, o_ins, e_ins, zdrop), do.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(do.cpu().numpy(), ref)
