"""The autotuner's map is at least as fast as the context's on all the jobs: shapes that win band by band are not
returned where the map they make is slower (the built-in maps have more than their shapes)."""
import numpy as np
import pytest

from bsbolt_gb300 import _lib, autotune, extend, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("whole,returned", [(2.0, False), (0.5, True)])
def test_map_slower_as_a_whole_is_not_returned(gpu_ctx, monkeypatch, whole, returned):
    """Times as given: another shape wins every band by half, the map takes `whole` of the current one's."""
    jobs, seq = synth.ksw_jobs(6000, seed=77)
    base = autotune.default_map()
    real = autotune._run

    def run(ctx, param, j, s):
        changed = not np.array_equal(autotune.get_map(ctx), base)
        return real(ctx, param, j, s)[0], (whole if changed else 1.0) if len(j) == len(jobs) else 0.5 if changed else 1.0

    monkeypatch.setattr(autotune, "_run", run)
    p = extend.make_param(synth.fill_scmat(1, 4), 6, 1, 6, 1, 100)
    tmap, report = autotune.tune(gpu_ctx, jobs, seq, p, min_jobs=100, reps=1)
    assert report and all(r["best"] != r["current"] and r["kept"] == returned for r in report)
    assert np.array_equal(tmap[1:], base[1:]) != returned
    assert np.array_equal(autotune.get_map(gpu_ctx), base)


def test_tuned_map_is_not_slower(gpu_ctx):
    """As measured: queries that take the rings and cut bands of the built-in maps."""
    jobs, seq = synth.ksw_jobs(1 << 17, seed=5, qmin=200, qmax=400)
    p = extend.make_param(synth.fill_scmat(1, 4), 6, 1, 6, 1, 100)
    tmap, _ = autotune.tune(gpu_ctx, jobs, seq, p, min_jobs=2000, max_jobs=4000, reps=1)

    def ms():
        return min(autotune._run(gpu_ctx, p, jobs, seq)[1] for _ in range(4))

    usual = ms()
    try:
        autotune.set_map(gpu_ctx, tmap)
        tuned = ms()
    finally:
        autotune.set_map(gpu_ctx, None)
    assert tuned < 1.1 * usual, f"{tuned:.3f} ms against {usual:.3f}"
