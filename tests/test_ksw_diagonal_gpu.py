"""Extension jobs answered from their main diagonal, and rows left out once no result can
change (ksw_core.cuh): without cell counts both are in use, with them neither, and both forms
give the oracle's tuples."""
import numpy as np
import pytest

import oracle
from bsbolt_gb300 import extend, synth

pytestmark = pytest.mark.gpu


def edge_jobs(a, limit, seed):
    """Queries around the 32-column step; targets equal to the query up to a few substitutions
    and Ns (losses on both sides of `limit`), one base short, exact, or with a flank that
    repeats the query's end; h0 down to 1 and narrow bands."""
    rng = np.random.Generator(np.random.PCG64(seed))
    parts, rows, base = [], [], 0
    for qlen in [1, 2, 3, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 140, 255, 256, 300] * 60:
        q = rng.integers(0, 4, qlen).astype(np.uint8)
        q[rng.random(qlen) < 0.02] = 4
        t = q.copy()
        at = rng.integers(0, qlen, int(rng.integers(0, 4)))
        if rng.random() < 0.3:
            at = np.concatenate([at, [0, qlen - 1][: int(rng.integers(1, 3))]])
        t[at] = rng.integers(0, 5, len(at))
        kind = int(rng.integers(0, 5))
        if kind == 0:
            t = t[:-1]
        elif kind == 1:
            t = np.concatenate([t, q[-min(qlen, 20):], rng.integers(0, 4, 60).astype(np.uint8)])
        elif kind == 2:
            t = np.concatenate([t, rng.integers(0, 4, 100).astype(np.uint8)])
        elif kind == 3 and qlen > 4:
            c = int(rng.integers(1, qlen - 1))
            t = np.concatenate([t[:c], rng.integers(0, 4, int(rng.integers(1, 4))).astype(np.uint8), t[c:]])
        h0 = int(rng.choice([1, 2, max(1, limit - a), max(1, limit - a + 1), limit, 19, 60, 2100]))
        rows.append((base, base + len(q), len(q), len(t), h0, int(rng.choice([0, 1, 5, 100])),
                     int(rng.choice([0, 5, 30])), 0))
        parts += [q, t]
        base += len(q) + len(t)
    return np.array(rows, dtype=synth.JOB_DTYPE), np.concatenate(parts)


@pytest.mark.parametrize("scoring", [(1, 4, 6, 1, 6, 1, 100), (1, 4, 6, 1, 6, 1, 3), (2, 3, 4, 2, 9, 1, 0),
                                     (1, 1, 0, 1, 0, 1, 100), (20, 30, 60, 10, 50, 5, 400)],
                         ids=["bwa", "small-zdrop", "asymmetric", "no-gap-open", "32-bit-cells"])
def test_diagonal_jobs_and_left_out_rows(gpu_ctx, scoring):
    a, b, o_del, e_del, o_ins, e_ins, zdrop = scoring
    jobs, seq = edge_jobs(a, min(o_del + e_del, o_ins + e_ins), 7)
    mat = synth.fill_scmat(a, b)
    ref, rcells = oracle.ksw_batch(jobs, seq, mat, o_del, e_del, o_ins, e_ins, zdrop, n_threads=8)
    out = extend.ksw_extend2_batch(gpu_ctx, jobs, seq, mat, o_del, e_del, o_ins, e_ins, zdrop)
    assert np.array_equal(out, ref)
    out, cells = extend.ksw_extend2_batch(gpu_ctx, jobs, seq, mat, o_del, e_del, o_ins, e_ins, zdrop, want_cells=True)
    assert np.array_equal(out, ref) and np.array_equal(cells, rcells)


@pytest.mark.parametrize("per_sm", [50, 90, 1300])
@pytest.mark.parametrize("past", [0, 1])
@pytest.mark.parametrize("device", [False, True], ids=["host", "device"])
def test_built_in_maps_by_batch_size(gpu_ctx, per_sm, past, device):
    """Both sides of each line between two built-in tile maps, host and device entry."""
    torch = pytest.importorskip("torch")
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + past
    jobs, seq = synth.ksw_jobs(n, seed=n, qmin=1, qmax=300)
    mat = synth.fill_scmat(1, 4)
    ref, _ = oracle.ksw_batch(jobs, seq, mat, 6, 1, 6, 1, 100, n_threads=16)
    if not device:
        out = extend.ksw_extend2_batch(gpu_ctx, jobs, seq, mat, 6, 1, 6, 1, 100)
    else:
        dj, ds = torch.from_numpy(jobs.view(np.uint8).copy()).cuda(), torch.from_numpy(seq).cuda()
        do = torch.zeros((n, 6), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        extend.ksw_extend2_device(gpu_ctx, dj.data_ptr(), n, ds.data_ptr(), len(seq),
                                  extend.make_param(mat, 6, 1, 6, 1, 100), do.data_ptr())
        torch.cuda.synchronize()
        out = do.cpu().numpy()
    assert np.array_equal(out, ref)
