"""The diagonal test's word loads: every alignment of query, target and buffer, jobs at both ends of the buffer,
losses of every size around the limit, matrices whose matches do not all score alike."""
import numpy as np
import pytest

import oracle
from bsbolt_gb300 import extend, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("uneven", [False, True], ids=["plain-matrix", "uneven-matches"])
def test_alignments(gpu_ctx, shift, uneven):
    torch = pytest.importorskip("torch")
    rng = np.random.Generator(np.random.PCG64(shift))
    rows, parts, at = [], [], 0
    for k in range(1200):
        ql = int(rng.integers(1, 80))
        q = rng.integers(0, 4, ql).astype(np.uint8)
        t = q.copy()
        for p in rng.integers(0, ql, int(rng.integers(0, 4))):
            t[p] = rng.integers(0, 5)
        if rng.random() < 0.1:
            q[int(rng.integers(0, ql))] = 4
        t = np.concatenate([t, rng.integers(0, 4, int(rng.integers(0, 3))).astype(np.uint8)])
        rows.append((at, at + ql, ql, len(t), int(rng.choice([1, 5, 30])), 100, 5, 0))
        parts += [q, t]
        at += ql + len(t)
    jobs, seq = np.array(rows, dtype=synth.JOB_DTYPE), np.concatenate(parts)
    mat = synth.fill_scmat(2, 3).copy()
    if uneven:
        mat[6], mat[18] = 1, 2
    ref, _ = oracle.ksw_batch(jobs, seq, mat, 6, 1, 6, 1, 100, n_threads=8)
    buf = torch.zeros(len(seq) + shift, dtype=torch.uint8, device="cuda")
    buf[shift:] = torch.from_numpy(seq).cuda()
    dj, do = torch.from_numpy(jobs.view(np.uint8).copy()).cuda(), torch.zeros((len(jobs), 6), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    extend.ksw_extend2_device(gpu_ctx, dj.data_ptr(), len(jobs), buf.data_ptr() + shift, len(seq),
                              extend.make_param(mat, 6, 1, 6, 1, 100), do.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(do.cpu().numpy(), ref)
