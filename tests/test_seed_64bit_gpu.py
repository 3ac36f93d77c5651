"""The 64-bit form of the seeding kernels, their table and lists, which an index takes from 2^32 - 2 rows on, forced on
small ones beside the 32-bit form: the reference's own seed lists, the oracle's over the options and read shapes of
test_seed_forms_gpu, and a text that holds two bases only."""
import os
import sys

import numpy as np
import pytest

import oracle
from bsbolt_gb300 import _lib, extend, index, seed, synth

from test_seed_forms_gpu import reads_of, references

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
sys.path.insert(0, GOLDEN)
import golden_data  # noqa: E402

TABLE = 1 << 24                                          # entries of 16 or 32 bytes


def texts():
    rng = np.random.Generator(np.random.PCG64(8))
    two = np.where(rng.random(20_000) < 0.5, 0, 3).astype(np.uint8)
    return {**references(), "two-letter": two}


@pytest.fixture(scope="module", params=["tiny", "tandem", "three-letter", "two-letter"])
def indexed(request, tmp_path_factory):
    d = tmp_path_factory.mktemp("wide")
    synth.write_fasta(str(d / "ref.fa"), [("c", texts()[request.param])])
    index.build_index(str(d / "ref.fa"), str(d / "ref"))
    bi = index.BwaIndex(str(d / "ref"))
    return str(d / "ref"), bi, oracle.OracleBwt(bi.primary, bi.L2[1:], bi.bwt, bi.sa, bi.sa_intv)


@pytest.fixture(params=["0", "1"], ids=["32-bit", "64-bit"])
def form(request, monkeypatch):
    """A function that gives a context with the index loaded in this form."""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("BSB_SEED_64BIT", request.param)
    ctx = extend.Context(0)

    def load(prefix):
        before = torch.cuda.mem_get_info()[0]
        seed.load_index(ctx, prefix)
        taken = before - torch.cuda.mem_get_info()[0]
        assert (taken >= 32 * TABLE) == (request.param == "1"), taken      # the form's own table
        return ctx

    yield load
    ctx.close()


@pytest.mark.parametrize("n,longest", [(1, 100), (33, 1024), (700, 150)])
@pytest.mark.parametrize("msl,width,intv", [(19, 10, 20), (1, 3, 20), (11, 10, 0), (12, 40, 20), (13, 0, 5)])
def test_seeds_equal_the_oracle(form, indexed, n, longest, msl, width, intv):
    prefix, bi, ob = indexed
    ctx = form(prefix)
    rng = np.random.Generator(np.random.PCG64(100 * n + msl))
    reads = reads_of(bi.pac_codes(), n, longest, rng)
    offs = np.zeros(len(reads) + 1, np.int64)
    offs[1:] = np.cumsum([len(r) for r in reads])
    seqs = np.concatenate(reads)
    want, woff = ob.collect_intv(seqs, offs, min_seed_len=msl, split_width=width, max_mem_intv=intv, n_threads=8)
    lens = np.diff(offs)
    got, off = seed.seed_batch(ctx, seqs, offs, min_seed_len=msl, split_width=width, max_mem_intv=intv)
    for r in range(n):
        exp = want[woff[r]:woff[r + 1]] if lens[r] >= msl else want[:0]
        assert np.array_equal(got[off[r]:off[r + 1]], exp), f"read {r} of {lens[r]} bases"


@pytest.mark.parametrize("name", ["L5", "L30"])
def test_seeds_match_the_reference(form, tmp_path, name):
    synth.write_fasta(str(tmp_path / "ref.fa"), golden_data.golden_genome())
    index.build_index(str(tmp_path / "ref.fa"), str(tmp_path / "ref"))
    d = np.load(os.path.join(GOLDEN, f"reads_{name}.npz"))
    o = d["opts"]
    got, off = seed.seed_batch(form(str(tmp_path / "ref")), d["reads"], d["read_off"], min_seed_len=int(o[10]),
                               split_width=int(o[12]), max_mem_intv=int(o[13]))
    ref, roff = d["smem"], d["smem_off"]
    lens = np.diff(d["read_off"])
    for r in range(len(lens)):
        exp = ref[roff[r]:roff[r + 1]] if lens[r] >= int(o[10]) else ref[0:0]
        assert np.array_equal(got[off[r]:off[r + 1]], exp), f"read {r}: seeds differ"


def test_suffix_array_rows(form, indexed):
    """Every row through the full suffix array and through the walk."""
    prefix, bi, _ = indexed
    ctx = form(prefix)
    pac = bi.pac_codes()
    full = index.suffix_array(np.concatenate([pac, 3 - pac[::-1]]).astype(np.uint8)).astype(np.int64)
    want = np.where(full == 2 * len(pac), -1, full)
    rows = np.arange(len(full)).astype(np.uint64)
    for resident in (1, 0):
        _lib.check(ctx.handle, ctx.L.bsb_index_full_sa(ctx.handle, resident))
        assert np.array_equal(seed.sa_batch(ctx, rows).astype(np.int64), want)
