"""A context whose map was read and put back, or that the autotuner has measured on, runs as one that never had a map:
on the built-in maps for the batch's size, with the cut rings (seen by their times)."""
import numpy as np
import pytest

from bsbolt_gb300 import autotune, extend, synth

from test_launched_shapes_gpu import run_device

pytestmark = pytest.mark.gpu

SCORING = (1, 4, 6, 1, 6, 1, 100)


def shapes_run(ctx, jobs, seq):
    torch = pytest.importorskip("torch")
    sl = autotune.shapes(ctx.L)
    return {sl[t] for t, ms in enumerate(run_device(torch, ctx, jobs, seq, SCORING)[2]) if ms > 0}


@pytest.mark.parametrize("how", ["get-set", "default-set", "tune"])
def test_built_in_maps_again(how):
    few, seq = synth.ksw_jobs(1 << 12, seed=5, qmin=10, qmax=300)
    ctx = extend.Context(0)
    try:
        sizes = [64, 1 << 13, 1 << 18]
        before = [shapes_run(ctx, np.resize(few, n), seq) for n in sizes]
        assert len({frozenset(b) for b in before}) == 3 and {(32, 7), (32, 9)} <= before[2]
        if how == "get-set":
            autotune.set_map(ctx, autotune.get_map(ctx))
        elif how == "default-set":
            m = autotune.default_map()
            m[0] = 3                                     # (unused)
            autotune.set_map(ctx, m)
        else:
            autotune.tune(ctx, few, seq, extend.make_param(synth.fill_scmat(1, 4), 6, 1, 6, 1, 100), min_jobs=100, reps=1)
        assert [shapes_run(ctx, np.resize(few, n), seq) for n in sizes] == before
        other = autotune.default_map()
        other[1:9] = autotune.shapes().index((32, 6))
        autotune.set_map(ctx, other)                     # another map is used as it is
        assert not {(32, 7), (32, 9)} & shapes_run(ctx, np.resize(few, 1 << 18), seq)
        autotune.set_map(ctx, None)
        assert shapes_run(ctx, np.resize(few, 1 << 18), seq) == before[2]
    finally:
        ctx.close()
