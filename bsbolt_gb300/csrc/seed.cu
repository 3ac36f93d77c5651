// seed.cu -- SMEM seeding (mem_collect_intv) and suffix-array lookups on sm_103a.
//
// mem_collect_intv (bsbolt/External/BWA/bwamem.c:118-166) runs three passes:
//   pass 1  bwt_smem1 from every x (bwt.c:289-356), keep SMEMs >= min_seed_len;
//   pass 2  re-seed from the middle of SMEMs >= split_len with <= split_width hits;
//   pass 3  bwt_seed_strategy1 (bwt.c:358-379) from every x;
// then sorts each read's seeds by info.  Equal info means the same substring and so the same
// interval, so the sort needs no tie rule and the order seeds are found in does not matter.
//
// What bounds it is the chain of dependent sector fetches: an interval can be extended by its next
// base only once its two occurrence sectors have arrived.  bwt_smem1 keeps its matches in lock step
// (all forward matches from x, then one round over all of them per base to the left), which makes
// the chain of a read several hundred extensions long.  The matches are independent, though.  A
// match [x, e) that the forward phase pushed can be extended to the left on its own until it has
// fewer than min_intv occurrences, say to [b, e); it is an SMEM exactly if it cannot be extended
// to the right there either, which is one extension more and asked only of matches long enough to be
// seeds.  (bwt_smem1 emits the first match that fails in a round, and nothing for those behind it:
// a shorter match [x, e') never stops before a longer one, b(e') <= b(e), and stops at the same b
// exactly if [b, e') can still grow to the right.  Matches it drops for having the size of a longer
// one are of the second kind.  It emits nothing but the longest match where the base left of x is
// missing or an N.)
//
// So a warp takes a few reads: a lane each for the forward phases, every lane with one extension a
// step, and the pushed matches go to a list of the warp; then the lanes take matches from the
// list, one after the other, each extending its own to the left.  The re-seeds of pass 2 are
// a second launch of the same two phases, with their threshold on the occurrences; pass 3 is a forward
// phase of its own.  Against the lock-step form, a state machine with one thread per read and pass
// (11-13 of 32 lanes active; now 20), one GB300, seeding stage of a batch with its copies: 64 reads
// 0.76 -> 0.14 ms, 40k reads of 100 bases on a 2 Mb reference 1.51 -> 0.57, 67k of 150 on 100 Mb
// 3.6 -> 1.73, 114k RRBS reads 3.2 -> 1.6; 15 % more extensions.
//
// bwt_sa (bwt.c:86-96) is one thread per suffix-array row: one load from the full
// suffix array when it is resident, else LF steps until a sampled row, each step
// one 32-byte sector.

#include <algorithm>

#include "bsb_internal.cuh"
#include "fm_index.cuh"
#include "scan.cuh"

namespace {

constexpr int kSeedBlock = 128, kSeedWarps = kSeedBlock / 32;
constexpr int kSeedRho = 16;            // most reads (re-seeds) a warp takes at once

struct SeedOpt {
    int min_seed_len, split_len, split_width, max_mem_intv;
};

// A bi-interval (bwtintv_t without info) in the width the index needs: 32 bits below
// 2^32 - 2 rows, else 64.
template <class P>
struct Iv {
    P x0, x1, x2;
};
constexpr uint64_t kNarrowRows = 0xfffffffdull;

// A match on a warp's list: its interval, and slot of the read << 21 | start << 11 | end (reads
// have at most 1024 bases, so a start is below 2^10 and an end below 2^11).
struct alignas(16) Match32 {
    uint32_t x0, x1, x2, pos;
};
struct alignas(16) Match64 {
    uint64_t x0, x1, x2;
    uint32_t pos, pad;
};
template <class P> struct MatchOf;
template <> struct MatchOf<uint32_t> { using type = Match32; };
template <> struct MatchOf<uint64_t> { using type = Match64; };
static_assert(BSB_SEED_MAX_LEN <= 1024, "match positions are packed");

template <class P>
__device__ __forceinline__ Iv<P> set_intv(const DevFM &F, int c)   // bwt.h:80
{
    Iv<P> r;
    r.x0 = l2_at<P>(F, c) + 1;
    r.x1 = l2_at<P>(F, 3 - c) + 1;
    r.x2 = l2_at<P>(F, c + 1) - l2_at<P>(F, c);
    return r;
}

// bwt_extend (bwt.c:262-275) of ik by the single base c: the reference computes all
// four extensions and its callers keep ok[c] only, so only that one is formed here.
template <class P>
__device__ __forceinline__ Iv<P> extend_one(const DevFM &F, const Iv<P> &ik, bool is_back, int c)
{
    const P xf = is_back ? ik.x0 : ik.x1;     // x[!is_back]
    const P xb = is_back ? ik.x1 : ik.x0;     // x[is_back]
    P kge, kgt, lge, lgt;
    occ_cumulative<P>(F, sym_row<P>(F, xf - 1), c, kge, kgt);
    occ_cumulative<P>(F, sym_row<P>(F, xf - 1 + ik.x2), c, lge, lgt);
    const P fw = l2_at<P>(F, c) + 1 + (kge - kgt);
    const P bk = xb + (xf <= (P)F.primary && xf + ik.x2 - 1 >= (P)F.primary) + (lgt - kgt);   // bases > c come first
    Iv<P> o;
    o.x0 = is_back ? fw : bk;
    o.x1 = is_back ? bk : fw;
    o.x2 = (lge - lgt) - (kge - kgt);
    return o;
}

// Launch control words: [0] next chunk of the first launch, [1] overflow (read + 1),
// [2] pass-2 items queued, [3] next chunk of the second launch, [4..5] the bwt_extend
// calls of both launches (uint64; each is one bwt_2occ4, two occurrence queries).
enum { kCtrlNext1 = 0, kCtrlOverflow = 1, kCtrlQueued = 2, kCtrlNext2 = 3, kCtrlExt = 4, kCtrlWords = 8 };

// A pass-2 item: bwt_smem1 of read r from x with min_intv occurrences.
struct Reseed {
    int r, x;
    int64_t min_intv;
};

// out holds, per read r, mult * (2*len(r) + 32) slots starting at mult * (2*(offs[r]-offs[0]) +
// 32*r): the first part_cap0(len, mult) for passes 1-2 (filled in any order through an atomic
// count), the last part_cap1(len) (len/2 + 8: pass 3 finds at most one seed per
// min_seed_len + 1 >= 2 bases) for pass 3; count[2r + part] counts each part.  Passes 1-2
// have no such bound (every re-seed of a repeat can add SMEMs): a batch in which a read
// overflows runs again with mult doubled.
__device__ __host__ __forceinline__ int part_cap1(int len) { return len / 2 + 8; }
__device__ __host__ __forceinline__ int part_cap0(int len, int mult) { return mult * (2 * len + 32) - part_cap1(len); }
__device__ __host__ __forceinline__ int64_t part_base(int64_t rel_off, int r, int mult)
{
    return (int64_t)mult * (2 * rel_off + 32 * (int64_t)r);
}

// What the emission of a seed needs, apart from the seed.
struct SeedOut {
    DevIntv *out;
    int *count, *ctrl;
    Reseed *queue;
    int queue_cap, mult;
    const int64_t *offs;
};

// Passes 1-2: one SMEM [b, e) of read r; from pass 1 a long, rare one is queued for pass 2.
template <class P, int Pass>
__device__ __noinline__ void emit_smem(const SeedOpt &opt, const SeedOut &S, int r, int len, int b, int e, Iv<P> v)
{
    const int slot = atomicAdd(&S.count[2 * r], 1);
    if (slot < part_cap0(len, S.mult)) {
        DevIntv d;
        d.x0 = v.x0, d.x1 = v.x1, d.x2 = v.x2;
        d.info = (uint64_t)(uint32_t)b << 32 | (uint32_t)e;
        S.out[part_base(S.offs[r] - S.offs[0], r, S.mult) + slot] = d;
    } else {
        atomicMax(S.ctrl + kCtrlOverflow, r + 1);
    }
    if (Pass == 1 && e - b >= opt.split_len && (uint64_t)v.x2 <= (uint64_t)(int64_t)opt.split_width) {
        const int q = atomicAdd(S.ctrl + kCtrlQueued, 1);
        if (q < S.queue_cap) S.queue[q] = Reseed{r, (b + e) >> 1, (int64_t)v.x2 + 1};
        else atomicMax(S.ctrl + kCtrlOverflow, r + 1);
    }
}

// The reads of a warp's chunk.
struct ChunkRead {
    const uint8_t *q;
    int len, r;
    int64_t min_intv;
};

// Pass 3 of read r by one lane of a converged warp (has: the lane has a read).
template <class P>
__device__ __forceinline__ unsigned pass3(const DevFM &F, const SeedOpt &opt, const SeedOut &S, bool has, int r, int len,
                                          const uint8_t *q)
{
    DevIntv *dst = nullptr;
    int cap = 0, n = 0, i = 0, x = 0;
    if (has) {
        dst = S.out + part_base(S.offs[r] - S.offs[0], r, S.mult) + part_cap0(len, S.mult);
        cap = part_cap1(len);
    }
    bool in = false;
    Iv<P> ik;
    ik.x0 = ik.x1 = ik.x2 = 0;
    int qc = has && i < len ? q[i] : 4;
    unsigned n_ext = 0;
    while (__any_sync(BSB_FULL_MASK, has && i < len)) {
        const bool act = has && i < len;
        const int qn = act && i + 1 < len ? q[i + 1] : 4;      // for the next step, under this one's fetches
        if (act && in && qc < 4) {
            const Iv<P> ok = extend_one<P>(F, ik, false, 3 - qc);
            ++n_ext;
            ik = ok;
            if (ok.x2 < (P)opt.max_mem_intv && i - x >= opt.min_seed_len) {
                if (ok.x2 > 0) {                               // an empty interval is not kept (bwamem.c:160)
                    if (n < cap) {
                        DevIntv d;
                        d.x0 = ok.x0, d.x1 = ok.x1, d.x2 = ok.x2;
                        d.info = (uint64_t)(uint32_t)x << 32 | (uint32_t)(i + 1);
                        dst[n] = d;
                    }
                    ++n;
                }
                in = false;
            }
        } else if (act) {
            in = qc < 4;
            if (in) ik = set_intv<P>(F, qc), x = i;
        }
        ++i;
        qc = qn;
    }
    if (has) {
        if (n > cap) atomicMax(S.ctrl + kCtrlOverflow, r + 1);
        S.count[2 * r + 1] = n < cap ? n : cap;
    }
    return n_ext;
}

// Mode 0: chunks of rho reads for pass 1, then chunks of 32 reads for pass 3.  Mode 1: chunks of
// the queued re-seeds of pass 2, as many a chunk as spread them over all warps (at most rho).
// matches: region_cap entries per warp.  A read (a re-seed) pushes at most one match per end
// position, so rho * (max_len + 1) entries always hold a chunk.
template <class P, int Mode>
__global__ void __launch_bounds__(kSeedBlock, sizeof(P) == 4 ? 7 : 5)
seed_kernel(DevFM F, SeedOpt opt, int n_reads, int max_len, const uint8_t *__restrict__ seqs, SeedOut S,
            typename MatchOf<P>::type *__restrict__ matches, int region_cap, int rho)
{
    using Match = typename MatchOf<P>::type;
    __shared__ ChunkRead chunk_reads[kSeedWarps][32];
    const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    ChunkRead *const CR = chunk_reads[wb];
    Match *const list = matches + (size_t)(blockIdx.x * kSeedWarps + wb) * region_cap;
    const int64_t *const offs = S.offs;
    int *const next = S.ctrl + (Mode ? kCtrlNext2 : kCtrlNext1);
    const int n_items = Mode ? min(*(volatile int *)(S.ctrl + kCtrlQueued), S.queue_cap) : n_reads;
    if (Mode) {
        const int warps = gridDim.x * kSeedWarps;
        rho = min(rho, max(1, (n_items + warps - 1) / warps));
    }
    const int n1 = (n_items + rho - 1) / rho;
    const int n_chunks = n1 + (Mode == 0 && opt.max_mem_intv > 0 ? (n_reads + 31) / 32 : 0);
    unsigned n_ext = 0;
    for (;;) {
        int ch = 0;
        if (lane == 0) ch = atomicAdd(next, 1);
        ch = __shfl_sync(BSB_FULL_MASK, ch, 0);
        if (ch >= n_chunks) break;
        // ---- the chunk's reads, a lane each
        const bool p3 = Mode == 0 && ch >= n1;
        const int item = p3 ? (ch - n1) * 32 + lane : ch * rho + lane;
        bool act = item < n_items && (p3 || lane < rho);
        int r = 0, len = 0, x = 0;
        P mi = 1;
        const uint8_t *q = seqs;
        if (act) {
            r = item;
            if (Mode) {
                const Reseed it = S.queue[item];
                r = it.r, x = it.x, mi = (P)it.min_intv;
            }
            const int64_t o = offs[r], l = offs[r + 1] - o;
            q = seqs + o;
            len = (int)l;
            if (l < 0 || l > max_len) {                 // outside what the launch was sized for: refuse
                atomicMax(S.ctrl + kCtrlOverflow, r + 1);
                act = false;
            } else if (len < opt.min_seed_len) {        // mem_chain returns before seeding (bwamem.c:266)
                act = false;
            }
        }
        if (p3) {
            n_ext += pass3<P>(F, opt, S, act, r, len, q);
            continue;
        }
        __syncwarp();
        CR[lane] = ChunkRead{q, len, r, (int64_t)mi};
        __syncwarp();
        // ---- forward (bwt.c:300-319): every lane one extension a step, matches pushed when their
        // size is about to change.  lb: the leftmost base a match from x can reach (no N before x)
        int total = 0;
        {
            int i = 0, lb = 0;
            bool in = false;
            Iv<P> ik;
            ik.x0 = ik.x1 = ik.x2 = 0;
            if (Mode && act) {
                if (q[x] > 3) act = false;              // bwt_smem1 returns at once: no SMEM
                else {
                    ik = set_intv<P>(F, q[x]);
                    lb = x == 0 || q[x - 1] > 3 ? x : 0;
                    in = true;
                    i = x + 1;
                }
            }
            int qc = act && i < len ? q[i] : 4;
            while (__any_sync(BSB_FULL_MASK, act)) {
                const int qn = act && i + 1 < len ? q[i + 1] : 4;
                const bool ext = act && in && qc < 4;
                Iv<P> ok = ik;
                if (ext) ok = extend_one<P>(F, ik, false, 3 - qc);
                n_ext += ext;
                bool push = false, stop = false;
                if (act && in) {
                    push = qc > 3 || ok.x2 != ik.x2;      // an N or the read's end stops the match
                    stop = qc > 3 || (push && ok.x2 < mi);
                }
                const Iv<P> pv = ik;
                const int px = x, pe = i;
                const bool enq = push && px > lb && pe - lb >= opt.min_seed_len;
                // nothing to the left of x: only the longest match, and it is an SMEM
                const bool seed = push && stop && px == lb && pe - px >= opt.min_seed_len;
                if (act) {
                    if (ext && !stop) ik = ok;
                    if (!in || stop) {
                        in = qc < 4 && !(Mode && stop);
                        if (in) ik = set_intv<P>(F, qc), x = i;
                        else lb = i + 1;
                        if (i >= len || (Mode && stop)) act = false;
                    }
                    ++i;
                }
                qc = qn;
                const unsigned m = __ballot_sync(BSB_FULL_MASK, enq);
                if (enq) {
                    const int slot = total + __popc(m & below);
                    Match e;
                    e.x0 = pv.x0, e.x1 = pv.x1, e.x2 = pv.x2;
                    e.pos = (uint32_t)lane << 21 | (uint32_t)px << 11 | (uint32_t)pe;
                    if (slot < region_cap) list[slot] = e;
                }
                total += __popc(m);
                if (seed) emit_smem<P, Mode + 1>(opt, S, r, len, px, pe, pv);
            }
            total = min(total, region_cap);
        }
        __syncwarp();
        // ---- backward: the lanes take the list's matches, the next one loaded ahead
        int taken = 0;
        bool have = false, spare = false, right = false;
        Iv<P> v;
        v.x0 = v.x1 = v.x2 = 0;
        Match sp;
        sp.x0 = sp.x1 = sp.x2 = 0, sp.pos = 0;
        int i = 0, e = 0, c = 4, slot = 0;
        q = seqs, len = 0, mi = 1;
        for (;;) {
            if (!have && spare) {
                v.x0 = sp.x0, v.x1 = sp.x1, v.x2 = sp.x2;
                slot = (int)(sp.pos >> 21);
                i = (int)(sp.pos >> 11 & 1023u) - 1, e = (int)(sp.pos & 2047u);
                q = CR[slot].q, len = CR[slot].len, mi = (P)CR[slot].min_intv;
                c = q[i];                               // x > lb: there is a base to the left
                have = true, spare = right = false;
            }
            if (taken < total) {
                const unsigned m = __ballot_sync(BSB_FULL_MASK, !spare);
                const int k = taken + __popc(m & below);
                if (!spare && k < total) sp = list[k], spare = true;
                taken += __popc(m);
            }
            if (!__any_sync(BSB_FULL_MASK, have || spare)) break;
            if (!have) continue;
            const int qn = !right && i > 0 ? q[i - 1] : 4;
            const bool ext = right || c < 4;
            Iv<P> ok = v;
            if (ext) ok = extend_one<P>(F, v, !right, right ? 3 - c : c);
            n_ext += ext;
            const bool grows = ext && ok.x2 >= mi;
            if (right) {                                // asked whether [i + 1, e) can grow to the right
                have = false;
                if (!grows) emit_smem<P, Mode + 1>(opt, S, CR[slot].r, len, i + 1, e, v);
            } else if (grows) {
                v = ok;
                --i;
                c = i >= 0 ? qn : 4;
            } else if (e - (i + 1) >= opt.min_seed_len) {   // [i + 1, e) is as long as it gets to the left
                c = e < len ? q[e] : 4;
                right = true;
            } else {
                have = false;
            }
        }
        __syncwarp();
    }
    if (n_ext) atomicAdd((unsigned long long *)(S.ctrl + kCtrlExt), (unsigned long long)n_ext);
}

// Seeds of read r in the two parts of its padded region (a part that overflowed holds
// its capacity; the launch reports the overflow).
__device__ __forceinline__ void part_counts(const int *__restrict__ count, const int64_t *__restrict__ offs, int r,
                                            int mult, int &na, int &nb)
{
    const int len = (int)(offs[r + 1] - offs[r]);
    na = min(count[2 * r], part_cap0(len, mult));
    nb = min(count[2 * r + 1], part_cap1(len));
}

// Seeds each read keeps (both parts, clamped to their caps), for the offset scan.
__global__ void read_totals(const int *__restrict__ count, const int64_t *__restrict__ offs, int n, int mult,
                            int *__restrict__ tot)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        int na, nb;
        part_counts(count, offs, r, mult, na, nb);
        tot[r] = na + nb;
    }
}

// Each read's seeds, sorted by info into the compact output (one block per read): an
// element's place is the number of elements with a smaller info, plus the number of
// equal ones before it (ks_introsort with intv_lt, bwamem.c:92-93; elements with equal
// info are equal, so the tie rule cannot show).
constexpr int kSortStage = 256, kCompactWarps = 4;
// One warp per read: the read's two parts merged into info order by rank (keys staged in
// the warp's slice of shared memory when they fit).
__global__ void __launch_bounds__(kCompactWarps * 32)
compact_seeds(const DevIntv *__restrict__ padded, const int64_t *__restrict__ offs, int n_reads, int mult,
              const int *__restrict__ count, const int64_t *__restrict__ out_off, DevIntv *__restrict__ out)
{
    __shared__ uint64_t keys[kCompactWarps][kSortStage];
    const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
    uint64_t *key = keys[wb];
    const int64_t base_off = offs[0];
    for (int r = blockIdx.x * kCompactWarps + wb; r < n_reads; r += gridDim.x * kCompactWarps) {
        const int len = (int)(offs[r + 1] - offs[r]);
        const DevIntv *a = padded + part_base(offs[r] - base_off, r, mult);
        const DevIntv *b = a + part_cap0(len, mult);
        int na, nb;
        part_counts(count, offs, r, mult, na, nb);
        const int m = na + nb;
        DevIntv *dst = out + out_off[r];
        const bool staged = m <= kSortStage;
        __syncwarp();
        if (staged)
            for (int i = lane; i < m; i += 32) key[i] = (i < na ? a[i] : b[i - na]).info;
        __syncwarp();
        for (int i = lane; i < m; i += 32) {
            const DevIntv v = i < na ? a[i] : b[i - na];
            int rank = 0;
            for (int j = 0; j < m; ++j) {
                const uint64_t w = staged ? key[j] : (j < na ? a[j] : b[j - na]).info;
                rank += w < v.info || (w == v.info && j < i);
            }
            dst[rank] = v;
        }
    }
}

// Longest LF walk between sampled rows accepted: a valid index needs a few hundred
// steps at most (rows are sampled every sa_intv by row number); a corrupt one must not
// loop forever.
constexpr uint64_t kMaxWalk = 1ull << 20;

// bwt_sa: LF-walk to the nearest sampled row (bwt.c:53-59, 86-96), or one load when
// the full suffix array is resident.  Rows beyond seq_len are answered with
// (uint64_t)-2 and never walked; a walk longer than kMaxWalk with (uint64_t)-3.
__global__ void sa_kernel(DevFM F, const uint64_t *__restrict__ rows, int64_t n, uint64_t *__restrict__ pos)
{
    const uint64_t mask = (1ull << F.sa_shift) - 1;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint64_t k = rows[i], steps = 0;
        if (k > F.seq_len) {
            pos[i] = ~(uint64_t)1;
            continue;
        }
        if (F.sa_full) {
            pos[i] = __ldg(F.sa_full + k);
            continue;
        }
        while ((k & mask) && steps < kMaxWalk) {
            ++steps;
            k = lf_step(F, k);
        }
        pos[i] = (k & mask) ? ~(uint64_t)2 : steps + __ldg(F.sa + (k >> F.sa_shift));
    }
}

// The full suffix array from the sampled one: sampled row s holds its sample, and the
// rows LF(s), LF^2(s), ... up to the next sampled row hold sa(s) - 1, sa(s) - 2, ...
// (bwt_sa's own walk, read backwards: every row's walk ends at the sampled row this
// fill starts from, so each row gets the value bwt_sa gives it).  Row 0 answers BWA's
// sample, (uint64_t)-1; the rows after it count down from seq_len.
__global__ void sa_fill_kernel(DevFM F, int64_t n_sa, uint64_t *__restrict__ full, int *__restrict__ failed)
{
    const uint64_t mask = (1ull << F.sa_shift) - 1;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_sa; t += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t s = (uint64_t)t << F.sa_shift;
        if (s > F.seq_len) continue;
        const uint64_t sv = F.sa[t];
        full[s] = sv;
        uint64_t v = s == 0 ? F.seq_len : sv, k = s;
        for (uint64_t step = 0;; ++step) {
            if (step >= kMaxWalk) {                      // not a valid index: the walk is kept
                atomicExch(failed, 1);
                break;
            }
            k = lf_step(F, k);
            if (!(k & mask)) break;                     // the next sampled row starts its own run
            full[k] = --v;
        }
    }
}

}  // namespace

static bool seed_narrow(uint64_t seq_len) { return seq_len < kNarrowRows; }

// The launch shape of a batch: warps that are resident at once, reads a chunk of pass 1 takes, and
// the match list each warp needs.
// rho: as few reads a warp as still occupy every warp, so that the matches of a read spread over the
// warp's lanes, and at most kSeedRho (67k reads of 150 bases: 2.5 ms at 2, 1.93 at 4, 1.73 at 8 and
// 16, 1.86 at 24, 2.1 at 32, where the forward phases fill the lanes but half the warps stay empty).
SeedPlan seed_plan(int n_sm, int max_len, int n_reads, uint64_t seq_len)
{
    const bool narrow = seed_narrow(seq_len);
    static int resident[2] = {0, 0};
    if (!resident[narrow]) {
        int b = 0, b2 = 0;
        const cudaError_t e =
            narrow ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, seed_kernel<uint32_t, 0>, kSeedBlock, 0)
                   : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, seed_kernel<uint64_t, 0>, kSeedBlock, 0);
        const cudaError_t e2 =
            narrow ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b2, seed_kernel<uint32_t, 1>, kSeedBlock, 0)
                   : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b2, seed_kernel<uint64_t, 1>, kSeedBlock, 0);
        b = std::min(b, b2);
        if (e != cudaSuccess || e2 != cudaSuccess || b < 1) b = 4;
        resident[narrow] = b;
    }
    SeedPlan p;
    const int64_t warps = (int64_t)n_sm * resident[narrow] * kSeedWarps;
    p.rho = (int)std::min<int64_t>(kSeedRho, std::max<int64_t>(1, (n_reads + warps - 1) / warps));
    const size_t entry = narrow ? sizeof(Match32) : sizeof(Match64);
    const size_t budget = (size_t)1 << 30;              // long reads: fewer reads a warp
    const size_t fit = budget / ((size_t)warps * (size_t)(max_len + 1) * entry);
    if ((size_t)p.rho > fit) p.rho = (int)std::max<size_t>(1, fit);
    // no more warps than the first launch has chunks (pass 1 and pass 3) or the second can use
    const int64_t chunks = (n_reads + p.rho - 1) / p.rho + (n_reads + 31) / 32;
    p.blocks = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)n_sm * resident[narrow],
                                                           std::max<int64_t>((chunks + kSeedWarps - 1) / kSeedWarps,
                                                                             std::min<int64_t>(n_reads, n_sm))));
    p.region_cap = p.rho * (max_len + 1);
    p.list_bytes = (size_t)p.blocks * kSeedWarps * (size_t)p.region_cap * entry;
    return p;
}

// Pass-2 work items a batch can queue: at most one per SMEM of pass 1, i.e. per read
// position.
size_t seed_queue_bytes(int64_t total_bases, int n_reads, int mult, int64_t *entries)
{
    *entries = (int64_t)mult * (total_bases + n_reads) + 64;
    return (size_t)*entries * sizeof(Reseed);
}

size_t seed_padded_entries(int64_t total_bases, int n_reads, int mult)
{
    return (size_t)mult * (2 * (size_t)total_bases + 32 * (size_t)n_reads);
}

template <class P>
static void seed_passes(const DevFM &F, const SeedOpt &o, int n_reads, int max_len, const uint8_t *d_seqs,
                        const SeedOut &S, void *d_lists, const SeedPlan &p, cudaStream_t st)
{
    using Match = typename MatchOf<P>::type;
    seed_kernel<P, 0><<<p.blocks, kSeedBlock, 0, st>>>(F, o, n_reads, max_len, d_seqs, S, (Match *)d_lists,
                                                       p.region_cap, p.rho);
    seed_kernel<P, 1><<<p.blocks, kSeedBlock, 0, st>>>(F, o, n_reads, max_len, d_seqs, S, (Match *)d_lists,
                                                       p.region_cap, p.rho);
}

cudaError_t seed_launch(const DevFM &F, int min_seed_len, float split_factor, int split_width, int max_mem_intv,
                        int n_reads, const uint8_t *d_seqs, const int64_t *d_offs, int max_len,
                        void *d_padded, int *d_count, int64_t *d_out_off, void *d_out,
                        void *d_lists, int *d_ctrl, void *d_queue, int64_t queue_cap, int *d_tot,
                        int64_t *d_scan_tmp, int mult, int n_sm, cudaStream_t st)
{
    SeedOpt o;
    o.min_seed_len = min_seed_len;
    o.split_len = (int)(min_seed_len * split_factor + .499);    // bwamem.c:122
    o.split_width = split_width;
    o.max_mem_intv = max_mem_intv;
    cudaError_t e = cudaMemsetAsync(d_ctrl, 0, kCtrlWords * sizeof(int), st);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(d_count, 0, sizeof(int) * 2 * (size_t)n_reads, st);
    if (e != cudaSuccess) return e;
    SeedOut S;
    S.out = (DevIntv *)d_padded;
    S.count = d_count, S.ctrl = d_ctrl;
    S.queue = (Reseed *)d_queue;
    S.queue_cap = (int)(queue_cap < 0x7fffffff ? queue_cap : 0x7fffffff);
    S.mult = mult;
    S.offs = d_offs;
    const SeedPlan p = seed_plan(n_sm, max_len, n_reads, F.seq_len);
    if (seed_narrow(F.seq_len)) seed_passes<uint32_t>(F, o, n_reads, max_len, d_seqs, S, d_lists, p, st);
    else seed_passes<uint64_t>(F, o, n_reads, max_len, d_seqs, S, d_lists, p, st);
    read_totals<<<n_sm * 4, 256, 0, st>>>(d_count, d_offs, n_reads, mult, d_tot);
    e = scan_i32_i64(d_tot, n_reads, d_out_off, d_scan_tmp, st);
    if (e != cudaSuccess) return e;
    const int cb = (int)((n_reads + kCompactWarps - 1) / kCompactWarps);
    compact_seeds<<<cb < n_sm * 16 ? cb : n_sm * 16, kCompactWarps * 32, 0, st>>>(
        (const DevIntv *)d_padded, d_offs, n_reads, mult, d_count, d_out_off, (DevIntv *)d_out);
    return cudaGetLastError();
}

cudaError_t sa_full_build(const DevFM &F, int64_t n_sa, uint64_t *full, int *failed, int n_sm, cudaStream_t st)
{
    const int64_t want = (n_sa + 255) / 256;
    const int blocks = (int)(want < (int64_t)n_sm * 32 ? want : (int64_t)n_sm * 32);
    sa_fill_kernel<<<blocks > 0 ? blocks : 1, 256, 0, st>>>(F, n_sa, full, failed);
    return cudaGetLastError();
}

cudaError_t sa_launch(const DevFM &F, const uint64_t *d_rows, int64_t n, uint64_t *d_pos, int n_sm, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    const int64_t want = (n + 255) / 256;
    const int blocks = (int)(want < (int64_t)n_sm * 16 ? want : (int64_t)n_sm * 16);
    sa_kernel<<<blocks, 256, 0, st>>>(F, d_rows, n, d_pos);
    return cudaGetLastError();
}
