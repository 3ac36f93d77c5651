"""bsb_build_bwt where its groups of equal prefixes change hands (sa_build.cu): copies on both sides of the largest
small group, more open suffixes than the small groups' list holds, mixtures of both, texts around the first key's
length, against the host's suffix order."""
import ctypes

import numpy as np
import pytest

from bsbolt_gb300 import _lib, index

pytestmark = pytest.mark.gpu


def check(ctx, b, intv=8):
    l_pac = len(b)
    pac = np.zeros((l_pac + 3) // 4, np.uint8)
    np.bitwise_or.at(pac, np.arange(l_pac) >> 2, (b << ((~np.arange(l_pac) & 3) << 1)).astype(np.uint8))
    text = np.concatenate([b, 3 - b[::-1]]).astype(np.uint8)
    n = len(text)
    sa = index.suffix_array(text).astype(np.int64)
    sym = text[sa[sa != 0] - 1].astype(np.uint32)
    sym = np.concatenate([sym, np.zeros((-len(sym)) % 16, np.uint32)]).reshape(-1, 16)
    want = np.zeros(len(sym), np.uint32)
    for j in range(16):
        want |= sym[:, j] << np.uint32((15 - j) * 2)
    bwt, samples, pr = np.empty((n + 15) // 16, np.uint32), np.empty((n + intv) // intv, np.uint64), ctypes.c_uint64()
    _lib.check(ctx.handle, ctx.L.bsb_build_bwt(ctx.handle, pac.ctypes.data_as(ctypes.c_void_p), l_pac, intv, 0,
                                               bwt.ctypes.data_as(ctypes.c_void_p), ctypes.byref(pr),
                                               samples.ctypes.data_as(ctypes.c_void_p)))
    assert pr.value == int(np.nonzero(sa == 0)[0][0])
    assert np.array_equal(bwt, want)
    assert np.array_equal(samples, sa[::intv].astype(np.uint64))


@pytest.mark.parametrize("copies", [2, 3, 31, 32, 33, 64, 70])
@pytest.mark.parametrize("unit,changed", [(25, 0.0), (700, 0.0), (700, 0.003)])
def test_copies_of_a_unit(gpu_ctx, copies, unit, changed):
    """Copies apart from one another in a random text: few open suffixes; and nothing but copies: nearly all open."""
    rng = np.random.Generator(np.random.PCG64(copies * 1000 + unit))
    u = rng.integers(0, 4, unit).astype(np.uint8)
    for spacing in (0, 3 * unit):
        parts = []
        for _ in range(copies):
            v = u.copy()
            e = rng.random(unit) < changed
            v[e] = rng.integers(0, 4, int(e.sum()))
            parts += [v, rng.integers(0, 4, int(rng.integers(0, spacing + 1))).astype(np.uint8)]
        check(gpu_ctx, np.concatenate(parts))


@pytest.mark.parametrize("base", [0, 3])
def test_short_texts(gpu_ctx, base):
    """Every suffix shorter than the first key, or just not; ends that the padding equals."""
    rng = np.random.Generator(np.random.PCG64(2))
    for l_pac in list(range(1, 14)) + [15, 16, 17, 20, 21, 32, 33]:
        check(gpu_ctx, np.full(l_pac, base, np.uint8), 1)
        b = rng.integers(0, 4, l_pac).astype(np.uint8)
        b[: l_pac // 2] = 3 - base                                # the text ends in a run of `base`
        check(gpu_ctx, b, 1)


def test_mixed_sizes(gpu_ctx):
    """Long runs, tandem repeats, pairs of long copies and random text in one."""
    rng = np.random.Generator(np.random.PCG64(4))
    copy = rng.integers(0, 4, 9000).astype(np.uint8)
    parts = [np.zeros(3000, np.uint8), rng.integers(0, 4, 20000).astype(np.uint8), copy,
             np.resize(rng.integers(0, 4, 11), 5000).astype(np.uint8), copy, np.full(800, 2, np.uint8), 3 - copy[::-1],
             rng.choice([0, 2, 3], 30000, p=[0.3, 0.2, 0.5]).astype(np.uint8)]
    parts += [np.concatenate([copy[:300], rng.integers(0, 4, 50).astype(np.uint8)]) for _ in range(60)]
    check(gpu_ctx, np.concatenate(parts))
