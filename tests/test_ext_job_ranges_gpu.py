"""Extension jobs whose offset plus length passes the largest 64-bit number, and sequence buffers of negative size, are
refused by every entry as any other range outside the buffer is."""
import ctypes

import numpy as np
import pytest

import oracle
from bsbolt_gb300 import _lib, cost_model, extend, synth

pytestmark = pytest.mark.gpu

FAR = [2**63 - 1, 2**63 - 20, 2**62]
MAT = synth.fill_scmat(1, 4)


@pytest.mark.parametrize("field", ["qoff", "toff"])
@pytest.mark.parametrize("n", [40, 4096, 1 << 20])        # checked on the host, on the device, by several host threads
def test_host_entry(gpu_ctx, field, n):
    few, seq = synth.ksw_jobs(64, seed=9)
    jobs = np.resize(few, n)
    for far in FAR:
        jobs[field][n - 3] = far
        with pytest.raises(_lib.BsbError, match=f"job {n - 3}: sequence range") as e:
            extend.ksw_extend2_batch(gpu_ctx, jobs, seq, MAT, 6, 1, 6, 1, 100)
        assert e.value.code == _lib.BSB_EINVAL


@pytest.mark.parametrize("n", [40, 4096])
def test_negative_buffer_size(gpu_ctx, n):
    few, seq = synth.ksw_jobs(64, seed=9)
    jobs, out = np.resize(few, n), np.zeros((n, 6), np.int32)
    p = extend.make_param(MAT, 6, 1, 6, 1, 100)
    for size in (-1, -257, -2**63):
        rc = gpu_ctx.L.bsb_extend_batch(gpu_ctx.handle, ctypes.byref(p), ctypes.c_void_p(jobs.ctypes.data), n,
                                        ctypes.c_void_p(seq.ctypes.data), size, ctypes.c_void_p(out.ctypes.data), None)
        assert rc == _lib.BSB_EINVAL and not out.any()


def test_device_entry_and_features(gpu_ctx):
    torch = pytest.importorskip("torch")
    jobs, seq = synth.ksw_jobs(500, seed=9)
    want, _ = oracle.ksw_batch(jobs, seq, MAT, 6, 1, 6, 1, 100)
    bad = jobs.copy()
    at = [0, 100, 200, 300, 400, 499]
    for k, r in enumerate(at):
        bad["qoff" if k % 2 else "toff"][r] = FAR[k // 2]
    dj, ds = torch.from_numpy(bad.view(np.uint8).copy()).cuda(), torch.from_numpy(seq).cuda()
    do = torch.full((500, 6), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    extend.ksw_extend2_device(gpu_ctx, dj.data_ptr(), 500, ds.data_ptr(), len(seq),
                              extend.make_param(MAT, 6, 1, 6, 1, 100), do.data_ptr())
    with pytest.raises(_lib.BsbError, match="6 extension jobs"):
        _lib.check(gpu_ctx.handle, gpu_ctx.L.bsb_sync(gpu_ctx.handle))
    want[at] = -7
    assert np.array_equal(do.cpu().numpy(), want)
    feat = cost_model.CostModel(gpu_ctx).features(dj, 500, ds, len(seq)).cpu().numpy()
    assert np.isfinite(feat).all()
