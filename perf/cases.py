"""The work a user of this framework has it do, case by case, for timing.

Every case goes through the entry points a program calls: the batched ``ksw_extend2``
(host numpy buffers, or device buffers), SMEM seeding, the whole of ``mem_align1_core`` for a
batch of reads (seeds, SA rows, chains, extensions, dedup), ``bwa_gen_cigar2`` and ``ksw_align2``
batches, and the index's suffix sort.  The calls that return a varying number of records are
made as the aligner makes them: through the C interface, into buffers the caller owns and
reuses, sized for the batch (returned whole, the unused tail as it was).  Inputs are synthetic, with the shapes and distributions of
the workloads the repository is built for (directional bisulfite reads from a reference with
thinned CpG; three-letter extension jobs; mate-rescue windows).  Host-buffer entry points take
host arrays here too, as the aligner calls them, and the copies count.

Every output is a whole number (scores, coordinates, suffix intervals, CIGAR words, text bytes;
the one float field of a region, ``frac_rep``, is returned as its bits), so ``exact`` has nothing
to say: the results have to be equal.
"""
import ctypes
import math
import os
import tempfile

import numpy as np
import torch

from bsbolt_gb300 import _lib, cigar, extend, index, matesw, seed as seeding, synth

BASES_PER_BATCH = 10_000_000        # one -K batch of the aligner


def listed():
    return [
        # A handful of extension calls, as an aligner's last, nearly empty batch or an interactive
        # caller makes them: launches and synchronisations are all there is.
        {"name": "extend_64", "kind": "extend", "n": 64, "qmin": 10, "qmax": 140, "bonus": 5, "device": False},
        # One 64k-job batch from host arrays: the extension jobs of a few thousand reads.
        {"name": "extend_64k", "kind": "extend", "n": 65_536, "qmin": 10, "qmax": 140, "bonus": 5, "device": False},
        # Throughput: 2M jobs already in device memory (the headline distribution, q 10-140).
        {"name": "extend_2m_device", "kind": "extend", "n": 2_000_000, "qmin": 10, "qmax": 140, "bonus": 5,
         "device": True},
        # Long flanks of long reads, with the aligner's default clipping penalty as end bonus.
        {"name": "extend_long", "kind": "extend", "n": 50_000, "qmin": 100, "qmax": 600, "bonus": 30,
         "device": False},
        # SMEM seeding alone, of quality-trimmed reads (every length from 36 to 250).
        {"name": "seeds_ragged", "kind": "seed", "mb": 2, "reads": 20_000, "lo": 36, "hi": 250},
        # The end of a file: a batch of a few reads through the whole of mem_align1_core.
        {"name": "align_64", "kind": "align", "mb": 2, "reads": 64, "lo": 100, "hi": 100, "rrbs": False, "clip": 5},
        # 20k directional pairs 2x100 on a 2 Mb reference without repeats: a bacterium, a panel.
        {"name": "align_2mb_pe100", "kind": "align", "mb": 2, "reads": 40_000, "lo": 100, "hi": 100, "rrbs": False,
         "clip": 5},
        # One -K batch of whole-genome pairs 2x150, 100 Mb reference with 15 % repeats.
        {"name": "align_100mb_pe150", "kind": "align", "mb": 100, "reads": 66_666, "lo": 150, "hi": 150,
         "rrbs": False, "clip": 5},
        # One -K batch of RRBS reads (75 and 100 bases, few start positions), bsbolt's clipping penalty.
        {"name": "align_100mb_rrbs", "kind": "align", "mb": 100, "reads": 114_000, "lo": 75, "hi": 100,
         "rrbs": True, "clip": 30},
        # CIGAR, MD and methylation strings of a batch's best regions.
        {"name": "cigar_40k", "kind": "cigar", "mb": 2, "reads": 40_000, "lo": 100, "hi": 100},
        # Mate rescue of a batch: 40k windows, mates of 30-250 bases.
        {"name": "rescue_40k", "kind": "rescue", "n": 40_000, "qmin": 30, "qmax": 250},
        # Index building: BWT and sampled suffix array of a 10 Mb converted text and its reverse complement.
        {"name": "index_10mb", "kind": "index", "bases": 10_000_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["extend", "extend", "seed", "align", "align", "align", "cigar", "rescue", "index"])
    if kind == "extend":
        qmax = _log_int(rng, 40, 600)
        qmin = rng.randint(5, qmax)
        most = min(2_000_000, int(2_000_000 * (150 / (qmin + qmax)) ** 2.2))
        return {"kind": kind, "n": _log_int(rng, 33, most), "qmin": qmin, "qmax": qmax,
                "bonus": rng.choice([0, 5, 30]), "device": rng.random() < 0.5}
    if kind == "rescue":
        qmax = rng.randint(60, 300)
        return {"kind": kind, "n": _log_int(rng, 17, 40_000), "qmin": rng.randint(20, qmax), "qmax": qmax}
    if kind == "index":
        return {"kind": kind, "bases": _log_int(rng, 20_001, 10_000_000)}
    hi = rng.choice([rng.randint(36, 120), rng.randint(100, 250), rng.randint(150, 500)])
    lo = rng.choice([hi, rng.randint(30, hi)])
    case = {"kind": kind, "mb": rng.choice([2, 100]), "reads": 2 * _log_int(rng, 20, BASES_PER_BATCH // hi // 2),
            "lo": lo, "hi": hi}
    if kind == "align":
        case["rrbs"] = hi <= 150 and rng.random() < 0.3
        case["clip"] = rng.choice([5, 30])
        if case["rrbs"]:
            case["mb"] = 100            # a 2 Mb reference holds too few MspI fragments
    return case


# ------------------------------------------------------------------ references and reads

_refs = {}


def _reference(mb):
    """(contigs, BwaIndex) of a seeded synthetic reference, built once per process: 2 Mb of four
    i.i.d. contigs, or 100 Mb with 15 % interspersed repeats."""
    if mb not in _refs:
        contigs = synth.bs_genome(4, mb * 250_000, gc=0.41, cpg_frac=0.01, seed=20261203)
        if mb > 10:
            synth.add_repeats(contigs, 0.15, seed=20261203)
        with tempfile.TemporaryDirectory() as d:
            fasta, prefix = os.path.join(d, "ref.fa"), os.path.join(d, "ref")
            synth.write_fasta(fasta, contigs)
            ctx = extend.Context(0)
            index.build_index(fasta, prefix, ctx=ctx)
            ctx.close()
            _refs[mb] = contigs, index.BwaIndex(prefix)
    return _refs[mb]


def _loaded(bi):
    """A context with the index in device memory, handed over as the aligner does (the arrays
    bwa_idx_load read)."""
    ctx = extend.Context(0)
    off = np.array([a.offset for a in bi.anns], np.int64)
    ln = np.array([a.len for a in bi.anns], np.int32)
    v = _lib.IndexView(primary=bi.primary, bwt=bi.bwt.ctypes.data, bwt_size=len(bi.bwt), sa=bi.sa.ctypes.data,
                       n_sa=bi.n_sa, sa_intv=bi.sa_intv, pac=bi.pac.ctypes.data, l_pac=bi.l_pac,
                       n_seqs=len(bi.anns), ann_offset=off.ctypes.data, ann_len=ln.ctypes.data)
    for i in range(5):
        v.L2[i] = int(bi.L2[i])
    _lib.check(ctx.handle, ctx.L.bsb_index_upload(ctx.handle, ctypes.byref(v)))
    cigar.upload_opac(ctx, bi.opac, bi.l_pac)
    return ctx


def _reads(contigs, case, seed):
    """(converted reads, offsets, reads as sequenced) of a batch: directional pairs, read 1 C->T and
    read 2 G->A, trimmed to lengths between lo and hi; or single-end RRBS reads, C->T."""
    n, lo, hi = case["reads"], case["lo"], case["hi"]
    if case.get("rrbs"):
        orig, offs = synth.rrbs_reads_se(contigs, n, (lo, hi), seed=seed)
        return synth.bs_convert(orig, g2a=False), offs, orig
    r1, r2 = synth.bs_reads_pe_block(contigs, n // 2, hi, max(300, 2 * hi + 100), 40, seed=seed)
    orig = np.stack([r1, r2], axis=1).reshape(-1, hi)
    conv = np.stack([synth.bs_convert(r1, g2a=False), synth.bs_convert(r2, g2a=True)], axis=1).reshape(-1, hi)
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    lens = rng.integers(lo, hi + 1, len(orig))
    keep = np.arange(hi)[None, :] < lens[:, None]
    offs = np.zeros(len(orig) + 1, np.int64)
    offs[1:] = np.cumsum(lens)
    return conv[keep], offs, orig[keep]


def _cigar_jobs(regs, roff, offs, opt):
    """One bwa_gen_cigar2 job per aligned read -- its best region, with the first band mem_reg2aln
    tries (infer_bw, bwamem.c:796-803)."""
    has = np.nonzero(roff[1:] > roff[:-1])[0]
    best = np.array([roff[r] + int(np.argmax(regs["score"][roff[r]:roff[r + 1]])) for r in has], np.int64)
    g = regs[best]
    l1, l2, sc = (x.astype(np.int64) for x in (g["qe"] - g["qb"], g["re"] - g["rb"], g["truesc"]))
    w = np.trunc((np.minimum(l1, l2) * opt.a - sc - opt.o_del) / opt.e_del + 2.0).astype(np.int64)
    w = np.maximum(w, np.abs(l1 - l2))
    w[(l1 == l2) & (l1 * opt.a - sc < 2 * (opt.o_del + opt.e_del - opt.a))] = 0
    jobs = np.zeros(len(best), cigar.JOB_DTYPE)
    jobs["rb"], jobs["re"] = g["rb"], g["re"]
    jobs["qoff"], jobs["ooff"] = offs[has] + g["qb"], offs[has]
    jobs["l_query"] = l1
    jobs["w"] = np.minimum(np.where(w > opt.w, np.minimum(w, g["w"]), w), opt.w << 2)
    return jobs


# ------------------------------------------------------------------ alignment jobs

def _rand(g, n):
    return torch.rand(n, device="cuda", generator=g)


def _bases(g, n, p):
    """n base codes 0..4 with the probabilities p."""
    edges = torch.cumsum(torch.tensor(p, device="cuda", dtype=torch.float32), 0)
    return torch.bucketize(_rand(g, n), edges / edges[-1], right=True).clamp_(max=4).to(torch.uint8)


def _between(g, lo, hi, n):
    """n whole numbers in [lo, hi]; hi may be a tensor."""
    return lo + (_rand(g, n) * (hi - lo + 1)).to(torch.int64)


def _pairs(g, qlen, before, after, sub, indel, unrelated, p):
    """Queries, and per query a target: `before` random bases, a copy of the query with
    substitutions at the job's rate and at most one 1-5-base indel, `after` random bases; where
    `unrelated`, the copy is random too.  Returns (sequence bytes, qoff, toff, tlen)."""
    n = len(qlen)
    qoff = torch.cumsum(qlen, 0) - qlen
    qtot = int(qlen.sum())
    q = _bases(g, qtot, p)
    at = (_rand(g, n) * qlen).to(torch.int64)
    size = torch.where(_rand(g, n) < indel, _between(g, 1, 5, n), 0)
    dele = _rand(g, n) < 0.5
    size = torch.where(dele, torch.minimum(size, qlen - at - 1).clamp(min=0), size)
    body = qlen + torch.where(dele, -size, size)
    tlen = before + body + after
    toff = torch.cumsum(tlen, 0) - tlen
    job = torch.repeat_interleave(torch.arange(n, device="cuda", dtype=torch.int32), tlen)
    k = torch.arange(len(job), device="cuda") - toff[job] - before[job]
    a, s, d = at[job], size[job], dele[job]
    src = torch.where(k < a, k, torch.where(d, k + s, torch.where(k < a + s, -1, k - s)))
    copied = (k >= 0) & (k < body[job]) & (src >= 0) & ~unrelated[job] & (_rand(g, len(job)) >= sub[job])
    t = _bases(g, len(job), p)
    t = torch.where(copied, q[(src.clamp(min=0) + qoff[job]).clamp(max=qtot - 1)], t)
    return torch.cat([q, t]), qoff, qtot + toff, tlen


def _extend_jobs(case, seed):
    """ksw_extend2 jobs in the converted alphabet (A/G/T 30/20/50 %, 1 % N): 1 % substitutions, 0.1 %
    indels, 100 bases of flank, a fifth of the targets unrelated, h0 of 19-100, w = 100."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"]
    qlen = _between(g, case["qmin"], case["qmax"], n)
    zero = torch.zeros_like(qlen)
    seq, qoff, toff, tlen = _pairs(g, qlen, zero, zero + 100, torch.full((n,), 0.01, device="cuda"),
                                   1 - 0.999 ** qlen.float(), _rand(g, n) < 0.2, [0.30, 0.0, 0.20, 0.50, 0.01])
    jobs = np.zeros(n, synth.JOB_DTYPE)
    for name, v in (("qoff", qoff), ("toff", toff), ("qlen", qlen), ("tlen", tlen), ("h0", _between(g, 19, 100, n))):
        jobs[name] = v.cpu().numpy()
    jobs["w"], jobs["end_bonus"] = 100, case["bonus"]
    return jobs, seq


def _rescue_jobs(case, seed):
    """ksw_align2 jobs as mem_matesw makes them: a mate against a window of its length plus 20-700
    bases, which in four of five jobs holds a copy with 0-15 % substitutions."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"]
    qlen = _between(g, case["qmin"], case["qmax"], n)
    extra = _between(g, 20, 700, n)
    before = (_rand(g, n) * extra).to(torch.int64)
    sub = torch.tensor([0.0, 0.01, 0.05, 0.15], device="cuda")[_between(g, 0, 3, n)]
    seq, qoff, toff, tlen = _pairs(g, qlen, before, extra - before, sub, torch.full((n,), 0.5, device="cuda"),
                                   _rand(g, n) < 0.2, [0.25, 0.25, 0.25, 0.25, 0.01])
    jobs = np.zeros(n, matesw.JOB_DTYPE)
    for name, v in (("qoff", qoff), ("toff", toff), ("qlen", qlen), ("tlen", tlen)):
        jobs[name] = v.cpu().numpy()
    jobs["xtra"] = [matesw.matesw_xtra(int(x)) for x in jobs["qlen"]]
    return jobs, seq


# ------------------------------------------------------------------ the case interface

def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "extend":
        jobs, seq = _extend_jobs(case, seed)
        s.update(ctx=extend.Context(0), mat=synth.fill_scmat(1, 4), device=case["device"])
        if case["device"]:
            s.update(jobs=torch.from_numpy(jobs.view(np.uint8)).cuda(), n=len(jobs), seq=seq,
                     out=torch.zeros((len(jobs), 6), dtype=torch.int32, device="cuda"),
                     param=extend.make_param(s["mat"], 6, 1, 6, 1, 100))
            torch.cuda.synchronize()
        else:
            s.update(jobs=jobs, seq=seq.cpu().numpy())
    elif kind == "rescue":
        jobs, seq = _rescue_jobs(case, seed)
        s.update(ctx=extend.Context(0), mat=synth.fill_scmat(1, 4), jobs=jobs, seq=seq.cpu().numpy())
    elif kind == "index":
        rng = np.random.Generator(np.random.PCG64(seed))
        n = case["bases"]
        # a converted text: three letters, with copies of earlier stretches as repeats have
        text = np.array([0, 2, 3, 3], np.uint8)[rng.integers(0, 4, n)]
        for _ in range(max(1, n // 50_000)):
            ln = int(rng.integers(300, 6000))
            a, b = (int(x) for x in rng.integers(0, n - ln, 2))
            text[b:b + ln] = text[a:a + ln].copy()
        pad = np.concatenate([text, np.zeros(-n % 4, np.uint8)]).reshape(-1, 4)
        s.update(ctx=extend.Context(0), n=n,
                 pac=(pad[:, 0] << 6 | pad[:, 1] << 4 | pad[:, 2] << 2 | pad[:, 3]).astype(np.uint8))
    else:
        contigs, bi = _reference(case["mb"])
        reads, offs, orig = _reads(contigs, case, seed)
        s.update(ctx=_loaded(bi), reads=reads, offs=offs)
        n = case["reads"]
        s.update(n=n, off=np.zeros(n + 1, np.int64))
        if kind == "seed":
            s.update(opt=_lib.SeedOpt(19, 1.5, 10, 20), out=np.zeros((64 * n + 1000, 4), np.int64))
        if kind == "align":
            s.update(opt=_lib.AlignOpt.bwa_defaults(pen_clip5=case["clip"], pen_clip3=case["clip"]),
                     out=np.zeros(16 * n + 1000, seeding.REG_DTYPE))
        if kind == "cigar":
            opt = _lib.AlignOpt.bwa_defaults()
            regs, roff = seeding.align_regs(s["ctx"], reads, offs, opt, dedup=True)
            s.update(jobs=np.resize(_cigar_jobs(regs, roff, offs, opt), n), orig=orig, crick_l=bi.crick_l, opt=opt,
                     out=np.zeros(n, cigar.OUT_DTYPE), blob=np.zeros((96 + 5 * case["hi"]) * n, np.uint8))
    return s


def _ints(a):
    """A table of records as whole numbers (float fields as their bits)."""
    return a.view(np.int32).reshape(len(a), -1)


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "extend":
        if s["device"]:
            extend.ksw_extend2_device(ctx, s["jobs"].data_ptr(), s["n"], s["seq"].data_ptr(), s["seq"].numel(),
                                      s["param"], s["out"].data_ptr())
            return s["out"]
        return extend.ksw_extend2_batch(ctx, s["jobs"], s["seq"], s["mat"], 6, 1, 6, 1, 100)
    if kind == "rescue":
        return _ints(matesw.align2_batch(ctx, s["jobs"], s["seq"], s["mat"], 6, 1, 6, 1))
    if kind == "index":
        n, intv = s["n"], 32
        bwt, sa = np.empty((2 * n + 15) // 16, np.uint32), np.empty((2 * n + intv) // intv, np.uint64)
        primary = ctypes.c_uint64()
        _lib.check(ctx.handle, ctx.L.bsb_build_bwt(ctx.handle, s["pac"].ctypes.data, n, intv, 0, bwt.ctypes.data,
                                                   ctypes.byref(primary), sa.ctypes.data))
        return bwt.view(np.int32), sa.view(np.int64), int(primary.value)
    L, n, out, off = ctx.L, s["n"], s["out"], s["off"]
    opt, reads = ctypes.byref(s["opt"]), s["reads"].ctypes.data
    if kind == "seed":
        _lib.check(ctx.handle, L.bsb_seed_batch(ctx.handle, opt, n, reads, s["offs"].ctypes.data, out.ctypes.data,
                                                len(out), off.ctypes.data))
        return out, off
    if kind == "align":
        _lib.check(ctx.handle, L.bsb_mem_align1_batch(ctx.handle, opt, n, reads, s["offs"].ctypes.data,
                                                      out.ctypes.data, len(out), off.ctypes.data))
        return _ints(out), off
    used, blob = ctypes.c_int64(), s["blob"]
    _lib.check(ctx.handle, L.bsb_gen_cigar_batch(ctx.handle, opt, s["crick_l"], n, s["jobs"].ctypes.data, reads,
                                                 len(s["reads"]), s["orig"].ctypes.data, len(s["orig"]),
                                                 out.ctypes.data, blob.ctypes.data, len(blob), ctypes.byref(used)))
    return _ints(out), blob, int(used.value)


def work(case):
    """Bytes only: the path is integer work on sequences, with no floating-point operations, and
    how many cells or index steps a job needs depends on its data.  Counted are the job records and
    sequences a call reads and the records it writes."""
    kind = case["kind"]
    if kind == "extend":
        return {"bytes": case["n"] * (40 + case["qmin"] + case["qmax"] + 100 + 24), "flops": 0}
    if kind == "rescue":
        return {"bytes": case["n"] * (32 + case["qmin"] + case["qmax"] + 360 + 28), "flops": 0}
    if kind == "index":
        return {"bytes": case["bases"] / 4 + case["bases"] / 2 + case["bases"] / 2, "flops": 0}
    bases = (case["lo"] + case["hi"]) / 2
    if kind == "seed":          # a read, its offset, and around eight 32-byte intervals
        return {"bytes": case["reads"] * (bases + 16 + 8 * 32), "flops": 0}
    if kind == "align":         # a read, its offsets, and one 56-byte region
        return {"bytes": case["reads"] * (bases + 16 + 56), "flops": 0}
    # a job, both forms of the read, two 2-bit stretches of reference, a record of about 60 bytes
    return {"bytes": case["reads"] * (40 + 2 * bases + bases / 2 + 48 + 60), "flops": 0}


def exact(case, seed):
    return None                 # whole numbers throughout: equality is the measure
