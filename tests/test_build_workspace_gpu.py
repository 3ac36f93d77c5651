"""The workspace that a context keeps between builds of small texts: 4 GB at most, and given back where memory is
needed."""
import ctypes

import numpy as np
import pytest

from bsbolt_gb300 import _lib, extend, index, seed, synth

pytestmark = pytest.mark.gpu

GB = 1 << 30


def build(ctx, n, chunk=0):
    pac = np.random.Generator(np.random.PCG64(n)).integers(0, 256, (n + 3) // 4, dtype=np.uint8)
    bwt, sa = np.empty((2 * n + 15) // 16, np.uint32), np.empty((2 * n + 32) // 32, np.uint64)
    primary = ctypes.c_uint64()
    _lib.check(ctx.handle, ctx.L.bsb_build_bwt(ctx.handle, pac.ctypes.data, n, 32, chunk, bwt.ctypes.data,
                                               ctypes.byref(primary), sa.ctypes.data))


@pytest.mark.parametrize("how", ["upload", "full-sa", "suffix-array", "chunks", "no-room", "close"])
def test_kept_workspace(tmp_path, how):
    torch = pytest.importorskip("torch")
    synth.write_fasta(str(tmp_path / "r.fa"), synth.bs_genome(1, 5000, 0.4, 0.01, seed=1))
    index.build_index(str(tmp_path / "r.fa"), str(tmp_path / "r"))
    ctx = extend.Context(0)
    free = lambda: torch.cuda.mem_get_info()[0]                           # noqa: E731
    try:
        if how == "full-sa":
            seed.load_index(ctx, str(tmp_path / "r"))
            _lib.check(ctx.handle, ctx.L.bsb_index_full_sa(ctx.handle, 0))
        before = free()
        build(ctx, 57_000_000)
        kept = before - free()
        assert 3.5 * GB < kept <= 4 * GB + (64 << 20), kept / GB
        if how == "upload":
            seed.load_index(ctx, str(tmp_path / "r"))
        elif how == "full-sa":
            _lib.check(ctx.handle, ctx.L.bsb_index_full_sa(ctx.handle, 1))
        elif how == "suffix-array":
            pac, sa = np.zeros(25, np.uint8), np.zeros(201, np.int64)
            _lib.check(ctx.handle, ctx.L.bsb_build_suffix_array(ctx.handle, pac.ctypes.data, 100, sa.ctypes.data))
        elif how == "chunks":
            build(ctx, 100_000, chunk=50_000)
        elif how == "no-room":                        # 2^45 bytes of sequences never fit
            jobs, seq = synth.ksw_jobs(4, seed=1)
            out, p = np.zeros((4, 6), np.int32), extend.make_param(synth.fill_scmat(1, 4), 6, 1, 6, 1, 100)
            assert ctx.L.bsb_extend_batch(ctx.handle, ctypes.byref(p), jobs.ctypes.data, 4, seq.ctypes.data, 1 << 45,
                                          out.ctypes.data, None) == _lib.BSB_ENOMEM
        else:
            ctx.close()
        assert before - free() < GB, (before - free()) / GB
    finally:
        ctx.close()
