"""The order alignment batches take reads in, as bsb_last_read_order gives it: by the caller's keys, by the model's
prediction, by chains; over all reads of small and logged batches, over the reads that need further extensions from
4096 reads on.  The order changes no region."""
import numpy as np
import pytest

from bsbolt_gb300 import _lib, seed

from test_chain_forms_gpu import loaded, make_reads  # noqa: F401  (loaded: the fixture)

pytestmark = pytest.mark.gpu


def bins(key):
    """key_bin (chain.cu): half octaves, larger keys first."""
    k = np.asarray(key, np.int64)
    msb = np.floor(np.log2(np.maximum(k, 1))).astype(np.int64)
    return np.where(k <= 0, 63, 63 - np.minimum(2 * msb + np.where(msb > 0, k >> np.maximum(msb - 1, 0) & 1, 0), 63))


@pytest.mark.parametrize("n", [1, 700, 4096, 4400])
def test_reads_are_taken_in_the_order_asked_for(loaded, n):  # noqa: F811
    torch = pytest.importorskip("torch")
    from bsbolt_gb300 import cost_model
    ctx, bi = loaded
    rng = np.random.Generator(np.random.PCG64(31))
    reads = sum((make_reads(bi.pac_codes(), rng) for _ in range((n + 399) // 400)), [])[:n]
    offs = np.zeros(n + 1, np.int64)
    offs[1:] = np.cumsum([len(r) for r in reads])
    seqs = np.concatenate(reads)
    opt = _lib.AlignOpt.bwa_defaults()
    seed.read_cost_log(ctx, True)
    try:
        regs, roff = seed.align_regs(ctx, seqs, offs, opt)
        feat, _ = seed.last_read_costs(ctx, n)
        assert sorted(seed.last_read_order(ctx, n)) == list(range(n))
    finally:
        seed.read_cost_log(ctx, False)
    chains = np.minimum(np.rint(np.expm1(4 * feat[:, 1].astype(np.float64))), 63)
    keys = (1 << rng.integers(0, 30, n)).astype(np.int64)
    model = cost_model.CostModel(ctx, seed=5)
    want = {"chains": -chains, "keys": bins(keys), "model": bins(model.forward(torch.from_numpy(feat).cuda(), True)[1]
                                                                 .cpu().numpy())}
    taken = None
    for how, first in want.items():
        if how == "keys":
            seed.set_read_order_keys(ctx, keys)
        if how == "model":
            seed.set_read_cost_model(ctx, model)
        try:
            got, goff = seed.align_regs(ctx, seqs, offs, opt)
            order = seed.last_read_order(ctx, n)
        finally:
            seed.set_read_cost_model(ctx, None)
        assert np.array_equal(goff, roff) and got.tobytes() == regs.tobytes()
        assert len(set(order.tolist())) == len(order) and (len(order) == n if n < 4096 else n // 50 < len(order) < n)
        assert taken is None or set(order.tolist()) == taken      # which reads are left does not depend on the order
        taken = set(order.tolist())
        assert (np.diff(first[order]) >= 0).all(), f"by {how}: {first[order][:40]}"


def test_read_order_errors(gpu_ctx):
    ctx = type(gpu_ctx)(0)
    try:
        with pytest.raises(_lib.BsbError) as e:
            seed.last_read_order(ctx, 5)
        assert e.value.code == _lib.BSB_EINVAL
    finally:
        ctx.close()
