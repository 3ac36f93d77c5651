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
// So pass 1 is two kernels: forward phases, 32 reads a warp, one extension a step for every lane
// (pass 3 is a forward phase of its own, in the same launch), which list their matches; then
// warps whose lanes take matches from the lists, one after the other, each extending its own to the
// left.  The re-seeds of pass 2 run both phases in one kernel, a few a warp, with their threshold on
// the occurrences.  A table of the bi-intervals of all 12-base strings stands in for the first 11
// extensions of every forward phase and of every short match.  One GB300, seeding stage of a batch
// with its copies: 64 reads 0.76 -> 0.165 ms, 40k reads of 100 bases on a 2 Mb reference 1.51 -> 0.38,
// 67k of 150 on 100 Mb 3.6 -> 1.24, 114k RRBS reads 3.2 -> 1.2 (the lock-step form, a state machine
// with one thread per read and pass and 11-13 of 32 lanes active, against this one; with both phases
// in one kernel and no table 0.14, 0.57, 1.73 and 1.6).  Of the 39M extensions of the third a
// forward step runs at 3.5 TB/s of DRAM, half the device's copy rate; the rest waits for sectors
// (L2 serves 24-37 %) with 20 of 64 warps per SM and 22 of 32 lanes.
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

struct SeedOpt {
    int min_seed_len, split_len, split_width, max_mem_intv;
};

// A bi-interval (bwtintv_t without info) in the width the index needs: 32 bits below
// 2^32 - 2 rows, else 64.
template <class P>
struct Iv {
    P x0, x1, x2;
};

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
// four extensions and its callers keep ok[c] only, so only that one is formed here.  In two
// halves, around the load of the two rows' sectors (wk, wl): extend_rows and extend_with.
template <class P>
__device__ __forceinline__ void extend_rows(const DevFM &F, const Iv<P> &ik, bool is_back, P &kk, P &ll)
{
    const P xf = is_back ? ik.x0 : ik.x1;     // x[!is_back]
    kk = sym_row<P>(F, xf - 1);
    ll = sym_row<P>(F, xf - 1 + ik.x2);
}
template <class P>
__device__ __forceinline__ Iv<P> extend_with(const DevFM &F, const Iv<P> &ik, bool is_back, int c, P kk, P ll,
                                             const uint32_t (&wk)[8], const uint32_t (&wl)[8])
{
    const P xf = is_back ? ik.x0 : ik.x1, xb = is_back ? ik.x1 : ik.x0;
    P kge, kgt, lge, lgt;
    occ_cumulative<P>(F, wk, kk, c, kge, kgt);
    occ_cumulative<P>(F, wl, ll, c, lge, lgt);
    const P fw = l2_at<P>(F, c) + 1 + (kge - kgt);
    const P bk = xb + (xf <= (P)F.primary && xf + ik.x2 - 1 >= (P)F.primary) + (lgt - kgt);   // bases > c come first
    Iv<P> o;
    o.x0 = is_back ? fw : bk;
    o.x1 = is_back ? bk : fw;
    o.x2 = (lge - lgt) - (kge - kgt);
    return o;
}

// Entry `code` of the k-mer table out of its 32 bytes.
template <class P>
__device__ __forceinline__ const uint4 *kmer_at(const DevFM &F, uint32_t code)
{
    return F.kmers + (sizeof(P) == 4 ? (code & ~1u) : 2 * (uint64_t)code);
}
template <class P>
__device__ __forceinline__ Iv<P> kmer_of(const uint32_t (&w)[8], uint32_t code)
{
    Iv<P> r;
    if (sizeof(P) == 4) {
        const bool odd = code & 1;
        r.x0 = odd ? w[4] : w[0], r.x1 = odd ? w[5] : w[1], r.x2 = odd ? w[6] : w[2];
    } else {
        r.x0 = (P)((uint64_t)w[1] << 32 | w[0]), r.x1 = (P)((uint64_t)w[3] << 32 | w[2]);
        r.x2 = (P)((uint64_t)w[5] << 32 | w[4]);
    }
    return r;
}

// The k-mer table, one thread per string of kKmer - 2 bases and the 16 strings it starts.
template <class P>
__device__ __forceinline__ Iv<P> extend_one(const DevFM &F, const Iv<P> &ik, int base)
{
    P kk, ll;
    uint32_t wk[8], wl[8];
    extend_rows<P>(F, ik, false, kk, ll);
    load32(sector_of<P>(F, kk), wk);
    load32(sector_of<P>(F, ll), wl);
    return extend_with<P>(F, ik, false, 3 - base, kk, ll, wk, wl);
}
template <class P>
__global__ void kmer_kernel(DevFM F, uint4 *__restrict__ out)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= kKmers / 16) return;
    Iv<P> v = set_intv<P>(F, (int)(t >> (2 * kKmer - 6)) & 3);
    for (int k = kKmer - 4; k >= 0; --k) v = extend_one<P>(F, v, (int)(t >> (2 * k)) & 3);
    for (int a = 0; a < 4; ++a) {
        const Iv<P> va = extend_one<P>(F, v, a);
        for (int b = 0; b < 4; ++b) {
            const Iv<P> e = extend_one<P>(F, va, b);
            const uint32_t code = t << 4 | a << 2 | b;
            if (sizeof(P) == 4) {
                out[code] = make_uint4((uint32_t)e.x0, (uint32_t)e.x1, (uint32_t)e.x2, 0u);
            } else {
                const uint64_t x0 = e.x0, x1 = e.x1, x2 = e.x2;
                out[2 * (uint64_t)code] = make_uint4((uint32_t)x0, (uint32_t)(x0 >> 32), (uint32_t)x1, (uint32_t)(x1 >> 32));
                out[2 * (uint64_t)code + 1] = make_uint4((uint32_t)x2, (uint32_t)(x2 >> 32), 0u, 0u);
            }
        }
    }
}

// Control words: [1] overflow (read + 1), [2] pass-2 items queued, [3] next chunk of pass 2, [4..5]
// the bwt_extend calls of the batch (uint64; each is one bwt_2occ4, two occurrence queries).
enum { kCtrlOverflow = 1, kCtrlQueued = 2, kCtrlNext = 3, kCtrlExt = 4, kCtrlWords = 8 };

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

// The reads of a warp's chunk, beside their packed bases.
struct ChunkRead {
    int len, r;
    int64_t min_intv;
};

// Passes 1-2: the first n (<= 32) SMEMs of a warp's buffer go out, a lane each, so that the wait for
// a read's slot counter is paid once for 32 of them; from pass 1 the long, rare ones are queued for
// pass 2.
template <class P, int Pass>
__device__ __forceinline__ void flush_smems(const SeedOpt &opt, const SeedOut &S, const ChunkRead *CR,
                                            const typename MatchOf<P>::type *buf, int n, int lane)
{
    bool again = false;
    Reseed rs;
    rs.r = rs.x = 0, rs.min_intv = 0;
    if (lane < n) {
        const typename MatchOf<P>::type v = buf[lane];
        const int k = (int)(v.pos >> 21 & 31u), b = (int)(v.pos >> 11 & 1023u), e = (int)(v.pos & 2047u);
        const int r = CR[k].r;
        const int slot = atomicAdd(&S.count[2 * r], 1);
        if (slot < part_cap0(CR[k].len, S.mult)) {
            DevIntv d;
            d.x0 = v.x0, d.x1 = v.x1, d.x2 = v.x2;
            d.info = (uint64_t)(uint32_t)b << 32 | (uint32_t)e;
            S.out[part_base(S.offs[r] - S.offs[0], r, S.mult) + slot] = d;
        } else {
            atomicMax(S.ctrl + kCtrlOverflow, r + 1);
        }
        again = Pass == 1 && e - b >= opt.split_len && (uint64_t)v.x2 <= (uint64_t)(int64_t)opt.split_width;
        rs.r = r, rs.x = (b + e) >> 1, rs.min_intv = (int64_t)v.x2 + 1;
    }
    if (Pass == 1) {
        const unsigned m = __ballot_sync(BSB_FULL_MASK, again);
        if (m) {
            int at = 0;
            if (lane == 0) at = atomicAdd(S.ctrl + kCtrlQueued, __popc(m));
            at = __shfl_sync(BSB_FULL_MASK, at, 0) + __popc(m & ((1u << lane) - 1u));
            if (again) {
                if (at < S.queue_cap) S.queue[at] = rs;
                else atomicMax(S.ctrl + kCtrlOverflow, rs.r + 1);
            }
        }
    }
}

// The reads of a warp's chunk, in shared memory: per read nw words of 16 bases (first base in the
// top bits, 0 for an N) and nm words of N bits (first base in bit 0; set from the read's end on),
// both strides odd so that the lanes' reads lie in different banks.
__host__ __device__ __forceinline__ int chunk_words(int max_len) { return (max_len / 16 + 2) | 1; }
__host__ __device__ __forceinline__ int chunk_masks(int max_len) { return (max_len / 32 + 2) | 1; }

struct PackedReads {
    const uint32_t *w, *m;
    int nw, nm;
    // base i of read k, 4 for an N and past the end
    __device__ __forceinline__ int base(int k, int i) const
    {
        const uint32_t v = w[k * nw + (i >> 4)], n = m[k * nm + (i >> 5)];
        return (n >> (i & 31) & 1u) ? 4 : (int)(v >> (30 - 2 * (i & 15)) & 3u);
    }
    // the code of the kKmer bases from i on; false where an N or the read's end is among them
    __device__ __forceinline__ bool kmer(int k, int i, uint32_t &code) const
    {
        const uint32_t *p = w + k * nw + (i >> 4), *q = m + k * nm + (i >> 5);
        code = __funnelshift_l(p[1], p[0], 2 * (i & 15)) >> (32 - 2 * kKmer);
        return !(__funnelshift_r(q[0], q[1], i & 31) & ((1u << kKmer) - 1u));
    }
};

// Packs the chunk's reads (lane k < n holds read k's bytes and length; a lane without a read: 0),
// 16 bases a lane and step.
__device__ __forceinline__ void pack_reads(uint32_t *w, uint32_t *m, int nw, int nm, int n, const uint8_t *q, int len,
                                           int lane)
{
    const int per = 2 * nm;                             // 16-bit halves of a read's N bits, at least nw
    for (int t0 = 0; t0 < n * per; t0 += 32) {
        const int t = t0 + lane, k = min(t / per, 31), word = t - t / per * per;
        const uint8_t *p = (const uint8_t *)__shfl_sync(BSB_FULL_MASK, (unsigned long long)q, k);
        const int l = __shfl_sync(BSB_FULL_MASK, len, k) - word * 16;
        uint32_t b[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) b[j] = j < l ? __ldg(p + word * 16 + j) : 4u;
        uint32_t v = 0, none = 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            v |= (b[j] < 4 ? b[j] : 0u) << (30 - 2 * j);
            none |= (uint32_t)(b[j] > 3) << j;
        }
        if (t < n * per) {
            if (word < nw) w[k * nw + word] = v;
            ((uint16_t *)m)[k * per + word] = (uint16_t)none;
        }
    }
}

// Pass 3 of read r, packed read k, by one lane of a converged warp (has: the lane has a read).
template <class P>
__device__ __forceinline__ unsigned pass3(const DevFM &F, const SeedOpt &opt, const SeedOut &S, bool has, int r, int len,
                                          const PackedReads &R, int k, bool tab)
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
    unsigned n_ext = 0;
    while (__any_sync(BSB_FULL_MASK, has && i < len)) {
        const bool act = has && i < len;
        const int qc = act ? R.base(k, i) : 4;
        uint32_t code = 0;
        const bool jump = act && !in && tab && R.kmer(k, i, code), ext = act && in && qc < 4;
        if (jump || ext) {
            P kk = 0, ll = 0;
            uint32_t wk[8], wl[8];
            if (ext) extend_rows<P>(F, ik, false, kk, ll);
            load32(jump ? kmer_at<P>(F, code) : sector_of<P>(F, kk), wk);
            load32(jump ? kmer_at<P>(F, code) : sector_of<P>(F, ll), wl);
            if (jump) {
                ik = kmer_of<P>(wk, code);
                in = true, x = i;
                i += kKmer - 1;
            } else {
                ik = extend_with<P>(F, ik, false, 3 - qc, kk, ll, wk, wl);
                ++n_ext;
                if (ik.x2 < (P)opt.max_mem_intv && i - x >= opt.min_seed_len) {
                    if (ik.x2 > 0) {                           // an empty interval is not kept (bwamem.c:160)
                        if (n < cap) {
                            DevIntv d;
                            d.x0 = ik.x0, d.x1 = ik.x1, d.x2 = ik.x2;
                            d.info = (uint64_t)(uint32_t)x << 32 | (uint32_t)(i + 1);
                            dst[n] = d;
                        }
                        ++n;
                    }
                    in = false;
                }
            }
        } else if (act) {
            in = qc < 4;
            if (in) ik = set_intv<P>(F, qc), x = i;
        }
        ++i;
    }
    if (has) {
        if (n > cap) atomicMax(S.ctrl + kCtrlOverflow, r + 1);
        S.count[2 * r + 1] = n < cap ? n : cap;
    }
    return n_ext;
}

// With a k-mer table (and min_seed_len >= kKmer) a match of fewer than kKmer bases is never formed:
// the forward phase starts at length kKmer, and what would be the matches [x, e) with e < x + kKmer
// is one record of x (a fan); such a match to the left has to reach [e - kKmer, e) to become a
// seed, so it starts from that string's entry.  (An end whose size does not change there is tried
// too; its match can grow to the right, so it is not emitted.)  Where the string from x has fewer
// than min_intv occurrences the forward phase goes base by base, and the short matches it lists are
// marked kTable to start the same way.  kSeed: the match is an SMEM as it stands.
constexpr uint32_t kTable = 1u << 31, kSeed = 1u << 30;
constexpr int kFan = kKmer - 1;

// The forward phases of bwt_smem1 (bwt.c:300-319) for the reads of a warp's chunk, a lane each, one
// extension a step; matches are listed when their size is about to change.  Reseed false: all
// matches of a read, the next one from where the longest ended; true: one from x with mi
// occurrences.  Matches go to list[0 ..), fans to list[cap - 1], list[cap - 2] ..: together at most one
// per read and end position, so a cap of the reads' bases and one more each always holds them.
template <class P, bool Reseed>
__device__ __forceinline__ unsigned forward_phase(const DevFM &F, const SeedOpt &opt, const PackedReads &R, bool act,
                                                  int len, int x, P mi, bool tab, typename MatchOf<P>::type *list, int cap,
                                                  int lane, int &n_list, int &n_fans)
{
    using Match = typename MatchOf<P>::type;
    const unsigned below = (1u << lane) - 1u;
    int i = Reseed ? x : 0, lb = 0;       // lb: the leftmost base a match from x can reach (no N before x)
    bool in = false, slow = false;        // slow: this match base by base from its start
    Iv<P> ik;
    ik.x0 = ik.x1 = ik.x2 = 0;
    unsigned n_ext = 0;
    n_list = n_fans = 0;
    if (Reseed && act) {
        act = R.base(lane, x) < 4;        // bwt_smem1 returns at once: no SMEM
        lb = x == 0 || R.base(lane, x - 1) > 3 ? x : 0;
    }
    while (__any_sync(BSB_FULL_MASK, act)) {
        const int qc = act ? R.base(lane, i) : 4;
        uint32_t code = 0;
        const bool jump = act && !in && !slow && tab && R.kmer(lane, i, code), ext = act && in && qc < 4;
        Iv<P> ok = ik;
        if (jump || ext) {
            P kk = 0, ll = 0;
            uint32_t wk[8], wl[8];
            if (ext) extend_rows<P>(F, ik, false, kk, ll);
            load32(jump ? kmer_at<P>(F, code) : sector_of<P>(F, kk), wk);
            load32(jump ? kmer_at<P>(F, code) : sector_of<P>(F, ll), wl);
            ok = jump ? kmer_of<P>(wk, code) : extend_with<P>(F, ik, false, 3 - qc, kk, ll, wk, wl);
        }
        n_ext += ext;
        const bool push = act && in && (qc > 3 || ok.x2 != ik.x2);    // an N or the read's end stops the match
        const bool stop = push && (qc > 3 || ok.x2 < mi);
        // nothing to the left of x: only the longest match, and it is an SMEM
        const bool seed = stop && x == lb;
        const bool put = (seed || (push && x > lb)) && i - lb >= opt.min_seed_len;
        const unsigned m = __ballot_sync(BSB_FULL_MASK, put);
        if (put) {
            const int slot = n_list + __popc(m & below);
            Match e;
            e.x0 = ik.x0, e.x1 = ik.x1, e.x2 = ik.x2;
            e.pos = (uint32_t)lane << 21 | (uint32_t)x << 11 | (uint32_t)i;
            if (seed) e.pos |= kSeed;
            else if (tab && i - x < kKmer) e.pos |= kTable;
            if (slot < cap) list[slot] = e;
        }
        n_list += __popc(m);
        const bool hit = jump && ok.x2 >= mi, fan = hit && i > lb && i + kKmer - 1 >= lb + opt.min_seed_len;
        const unsigned mf = __ballot_sync(BSB_FULL_MASK, fan);
        if (fan) {
            const int slot = cap - 1 - n_fans - __popc(mf & below);
            if (slot >= 0)
                list[slot].pos = (uint32_t)lane << 21 | (uint32_t)i << 11 | (uint32_t)max(i + 1, lb + opt.min_seed_len);
        }
        n_fans += __popc(mf);
        if (hit) {
            in = true, x = i, ik = ok, i += kKmer;
        } else if (jump) {
            slow = true;
        } else if (act) {
            if (Reseed && stop) {
                act = false;
            } else if (stop && tab && qc < 4) {           // a new match from i, which is looked up first
                in = slow = false;
            } else {
                if (!in || stop) {
                    in = qc < 4, slow = false;
                    if (in) ik = set_intv<P>(F, qc), x = i;
                    else lb = i + 1, act = i < len;
                } else {
                    ik = ok;
                }
                ++i;
            }
        }
    }
    n_list = min(n_list, cap);
    n_fans = min(n_fans, cap);
    return n_ext;
}

// The listed matches to the left (bwt.c:320-353): the lanes take them one after the other, the next
// one loaded ahead; of the units k = 32 * (j * stride + first) + l (fans first, kFan each) for all
// j and l.  buf: 64 SMEMs of shared memory.
template <class P, bool Reseed>
__device__ __forceinline__ unsigned backward_phase(const DevFM &F, const SeedOpt &opt, const SeedOut &S,
                                                   const PackedReads &R, const ChunkRead *CR, bool tab,
                                                   const typename MatchOf<P>::type *list, int cap, int n_list, int n_fans,
                                                   int first, int stride, typename MatchOf<P>::type *buf, int lane)
{
    using Match = typename MatchOf<P>::type;
    const unsigned below = (1u << lane) - 1u;
    const int fans = n_fans * kFan, total = fans + n_list;
    unsigned n_ext = 0;
    int taken = 0, n_buf = 0;
    bool have = false, spare = false, right = false, jump = false, done = false;
    Iv<P> v;
    v.x0 = v.x1 = v.x2 = 0;
    Match sp;
    sp.x0 = sp.x1 = sp.x2 = 0, sp.pos = 0;
    int i = 0, e = 0, slot = 0;
    P mi = 1;
    bool more = 32 * first < total;
    for (;;) {
        if (!have && spare) {
            v.x0 = sp.x0, v.x1 = sp.x1, v.x2 = sp.x2;
            slot = (int)(sp.pos >> 21 & 31u);
            e = (int)(sp.pos & 2047u);
            jump = sp.pos & kTable, done = sp.pos & kSeed;
            i = jump ? e - kKmer : (int)(sp.pos >> 11 & 1023u) - 1;
            if (Reseed) mi = (P)CR[slot].min_intv;
            have = true, spare = right = false;
        }
        if (more) {
            const unsigned m = __ballot_sync(BSB_FULL_MASK, !spare);
            const int t = taken + __popc(m & below), k = ((t >> 5) * stride + first) * 32 + (t & 31);
            if (!spare && k < total) {
                if (k < fans) {                         // end x + 1 + k % kFan of fan k / kFan
                    const uint32_t f = list[cap - 1 - k / kFan].pos;
                    const uint32_t end = (f >> 11 & 1023u) + 1 + (uint32_t)(k % kFan);
                    sp.pos = (f & ~2047u) | kTable | end;
                    spare = end >= (f & 2047u);
                } else {
                    sp = list[k - fans], spare = true;
                }
            }
            taken += __popc(m);
            more = ((taken >> 5) * stride + first) * 32 < total;
        }
        if (!__any_sync(BSB_FULL_MASK, have || spare || more)) break;
        uint32_t code = 0;
        if (have && jump && !R.kmer(slot, i, code)) have = jump = false;   // an N among the last kKmer bases: too short
        bool put = have && done;
        if (have && !done) {
            const int c = jump || (!right && i < 0) ? 4 : R.base(slot, right ? e : i);
            const bool ext = c < 4;
            Iv<P> ok = v;
            if (jump || ext) {
                P kk = 0, ll = 0;
                uint32_t wk[8], wl[8];
                if (ext) extend_rows<P>(F, v, !right, kk, ll);
                load32(jump ? kmer_at<P>(F, code) : sector_of<P>(F, kk), wk);
                load32(jump ? kmer_at<P>(F, code) : sector_of<P>(F, ll), wl);
                ok = jump ? kmer_of<P>(wk, code) : extend_with<P>(F, v, !right, right ? 3 - c : c, kk, ll, wk, wl);
            }
            n_ext += ext;
            const bool grows = (jump || ext) && ok.x2 >= mi;
            if (right) {                                // asked whether [i + 1, e) can grow to the right
                have = false, put = !grows;
            } else if (grows) {
                v = ok;
                --i;
            } else if (!jump && e - (i + 1) >= opt.min_seed_len) {   // [i + 1, e) is as long as it gets to the left
                right = true;
            } else {
                have = false;
            }
            jump = false;
        }
        const unsigned mp = __ballot_sync(BSB_FULL_MASK, put);
        if (mp) {
            if (put) {
                Match o;
                o.x0 = v.x0, o.x1 = v.x1, o.x2 = v.x2;
                o.pos = (uint32_t)slot << 21 | (uint32_t)(i + 1) << 11 | (uint32_t)e;
                buf[n_buf + __popc(mp & below)] = o;
                have = false;
            }
            n_buf += __popc(mp);
            if (n_buf >= 32) {
                __syncwarp();
                flush_smems<P, Reseed ? 2 : 1>(opt, S, CR, buf, 32, lane);
                n_buf -= 32;
                Match o = sp;
                if (lane < n_buf) o = buf[32 + lane];
                __syncwarp();
                if (lane < n_buf) buf[lane] = o;
            }
        }
    }
    __syncwarp();
    flush_smems<P, Reseed ? 2 : 1>(opt, S, CR, buf, n_buf, lane);
    __syncwarp();
    return n_ext;
}

// The warp's share of a block's dynamic shared memory: packed reads, then 64 SMEMs.
template <class P>
__device__ __forceinline__ typename MatchOf<P>::type *warp_smem(uint32_t *smem, int slots, int max_len, int wb,
                                                                uint32_t *&pw, uint32_t *&pm, PackedReads &R)
{
    using Match = typename MatchOf<P>::type;
    R.nw = chunk_words(max_len), R.nm = chunk_masks(max_len);
    Match *const bufs = (Match *)smem;
    uint32_t *const reads = (uint32_t *)(bufs + 64 * kSeedWarps) + (size_t)wb * slots * (R.nw + R.nm);
    pw = reads, pm = reads + slots * R.nw;
    R.w = pw, R.m = pm;
    return bufs + 64 * wb;
}

__device__ __forceinline__ void count_extensions(const SeedOut &S, unsigned n_ext, int lane)
{
    n_ext = __reduce_add_sync(BSB_FULL_MASK, n_ext);
    if (lane == 0 && n_ext) atomicAdd((unsigned long long *)(S.ctrl + kCtrlExt), (unsigned long long)n_ext);
}

// The list of reads r0 .. r1 - 1 among pass 1's: an entry per base and one more per read, from their
// first base's place on; kept inside the list_cap entries whatever the offsets say.
__device__ __forceinline__ int list_of(const SeedOut &S, int r0, int r1, int slots, int max_len, int64_t list_cap,
                                       int64_t &at)
{
    at = S.offs[r0] - S.offs[0] + r0;
    int64_t cap = min(S.offs[r1] - S.offs[r0], (int64_t)slots * max_len) + (r1 - r0);
    cap = min(cap, list_cap - at);
    if (at < 0 || cap < 0) at = cap = 0;
    return (int)cap;
}

// A lane's read of a chunk: false where there is none or mem_chain returns before seeding it
// (bwamem.c:266); a length the launch was not sized for is refused.
__device__ __forceinline__ bool chunk_read(const SeedOut &S, const SeedOpt &opt, const uint8_t *seqs, int r, int max_len,
                                           const uint8_t *&q, int &len)
{
    const int64_t o = S.offs[r], l = S.offs[r + 1] - o;
    q = seqs + o;
    len = 0;
    if (l < 0 || l > max_len) {
        atomicMax(S.ctrl + kCtrlOverflow, r + 1);
        return false;
    }
    if (l < opt.min_seed_len) return false;
    len = (int)l;
    return true;
}

// Pass 1's forward phases (a warp each for reads 32c ..) and pass 3 (the warps after these, `slots`
// reads each).  A warp's list: as many entries as its reads have bases, and one more per read.
// counts[c]: its matches and fans.
template <class P>
__global__ void __launch_bounds__(kSeedBlock, sizeof(P) == 4 ? 8 : 6)
seed_forward_kernel(DevFM F, SeedOpt opt, int n_reads, int max_len, int slots, const uint8_t *__restrict__ seqs,
                    SeedOut S, typename MatchOf<P>::type *__restrict__ lists, int64_t list_cap,
                    int2 *__restrict__ counts)
{
    extern __shared__ __align__(16) uint32_t smem[];
    const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
    const bool tab = F.kmers != nullptr && opt.min_seed_len >= kKmer;
    const int n1 = (n_reads + slots - 1) / slots;
    int c = blockIdx.x * kSeedWarps + wb;
    const bool p3 = c >= n1;
    if (p3) c -= n1;
    if (c >= n1 || (p3 && opt.max_mem_intv <= 0)) return;
    uint32_t *pw, *pm;
    PackedReads R;
    warp_smem<P>(smem, slots, max_len, wb, pw, pm, R);
    const int r = c * slots + lane;
    const uint8_t *q = seqs;
    int len = 0;
    const bool act = lane < slots && r < n_reads && chunk_read(S, opt, seqs, r, max_len, q, len);
    pack_reads(pw, pm, R.nw, R.nm, slots, q, len, lane);
    __syncwarp();
    unsigned n_ext;
    if (p3) {
        n_ext = pass3<P>(F, opt, S, act, r, len, R, lane, tab);
    } else {
        int64_t b0;
        const int cap = list_of(S, c * slots, min((c + 1) * slots, n_reads), slots, max_len, list_cap, b0);
        int n_list, n_fans;
        n_ext = forward_phase<P, false>(F, opt, R, act, len, 0, (P)1, tab, lists + b0, cap, lane, n_list, n_fans);
        if (lane == 0) counts[c] = make_int2(n_list, n_fans);
    }
    count_extensions(S, n_ext, lane);
}

// Pass 1's backward phases: `split` warps share a list.
template <class P>
__global__ void __launch_bounds__(kSeedBlock, sizeof(P) == 4 ? 8 : 6)
seed_backward_kernel(DevFM F, SeedOpt opt, int n_reads, int max_len, int slots, int split,
                     const uint8_t *__restrict__ seqs, SeedOut S, const typename MatchOf<P>::type *__restrict__ lists,
                     int64_t list_cap, const int2 *__restrict__ counts)
{
    extern __shared__ __align__(16) uint32_t smem[];
    __shared__ ChunkRead chunk_reads[kSeedWarps][32];
    const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
    const bool tab = F.kmers != nullptr && opt.min_seed_len >= kKmer;
    const int u = blockIdx.x * kSeedWarps + wb, c = u / split;
    if (c * slots >= n_reads) return;
    const int2 n = counts[c];
    if (32 * (u - c * split) >= n.x + n.y * kFan) return;
    uint32_t *pw, *pm;
    PackedReads R;
    typename MatchOf<P>::type *const buf = warp_smem<P>(smem, slots, max_len, wb, pw, pm, R);
    const int r = c * slots + lane;
    const uint8_t *q = seqs;
    int len = 0;
    if (lane < slots && r < n_reads) chunk_read(S, opt, seqs, r, max_len, q, len);
    chunk_reads[wb][lane] = ChunkRead{len, r, 1};
    pack_reads(pw, pm, R.nw, R.nm, slots, q, len, lane);
    __syncwarp();
    int64_t b0;
    const int cap = list_of(S, c * slots, min((c + 1) * slots, n_reads), slots, max_len, list_cap, b0);
    const unsigned n_ext = backward_phase<P, false>(F, opt, S, R, chunk_reads[wb], tab, lists + b0, cap, n.x, n.y,
                                                    u - c * split, split, buf, lane);
    count_extensions(S, n_ext, lane);
}

// Pass 2: chunks of the queued re-seeds, as many a chunk as spread them over all warps (at most
// slots), both phases; lists of slots * (max_len + 1) entries per warp.
template <class P>
__global__ void __launch_bounds__(kSeedBlock, sizeof(P) == 4 ? 8 : 5)
seed_again_kernel(DevFM F, SeedOpt opt, int max_len, int slots, const uint8_t *__restrict__ seqs, SeedOut S,
                  typename MatchOf<P>::type *__restrict__ lists)
{
    extern __shared__ __align__(16) uint32_t smem[];
    __shared__ ChunkRead chunk_reads[kSeedWarps][32];
    const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
    const bool tab = F.kmers != nullptr && opt.min_seed_len >= kKmer;
    ChunkRead *const CR = chunk_reads[wb];
    uint32_t *pw, *pm;
    PackedReads R;
    typename MatchOf<P>::type *const buf = warp_smem<P>(smem, slots, max_len, wb, pw, pm, R);
    const int cap = slots * (max_len + 1);
    typename MatchOf<P>::type *const list = lists + (size_t)(blockIdx.x * kSeedWarps + wb) * cap;
    const int n_items = min(*(volatile int *)(S.ctrl + kCtrlQueued), S.queue_cap);
    const int warps = gridDim.x * kSeedWarps;
    const int per = min(slots, max(1, (n_items + warps - 1) / warps));
    unsigned n_ext = 0;
    for (;;) {
        int ch = 0;
        if (lane == 0) ch = atomicAdd(S.ctrl + kCtrlNext, 1);
        ch = __shfl_sync(BSB_FULL_MASK, ch, 0);
        if ((int64_t)ch * per >= n_items) break;
        const int item = ch * per + lane;
        bool act = lane < per && item < n_items;
        Reseed it;
        it.r = it.x = 0, it.min_intv = 1;
        const uint8_t *q = seqs;
        int len = 0;
        if (act) {
            it = S.queue[item];
            act = chunk_read(S, opt, seqs, it.r, max_len, q, len);
        }
        CR[lane] = ChunkRead{len, it.r, it.min_intv};
        pack_reads(pw, pm, R.nw, R.nm, per, q, len, lane);
        __syncwarp();
        int n_list, n_fans;
        n_ext += forward_phase<P, true>(F, opt, R, act, len, it.x, (P)it.min_intv, tab, list, cap, lane, n_list, n_fans);
        __syncwarp();
        n_ext += backward_phase<P, true>(F, opt, S, R, CR, tab, list, cap, n_list, n_fans, 0, 1, buf, lane);
    }
    count_extensions(S, n_ext, lane);
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
template <class P>
__global__ void sa_kernel(DevFM F, const uint64_t *__restrict__ rows, int64_t n, uint64_t *__restrict__ pos)
{
    const uint64_t mask = (1ull << F.sa_shift) - 1;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t row = rows[i];
        if (row > F.seq_len) {
            pos[i] = ~(uint64_t)1;
            continue;
        }
        if (F.sa_full) {
            pos[i] = __ldg(F.sa_full + row);
            continue;
        }
        P k = (P)row;
        uint64_t steps = 0;
        while ((k & (P)mask) && steps < kMaxWalk) {
            ++steps;
            k = lf_step<P>(F, k);
        }
        pos[i] = (k & (P)mask) ? ~(uint64_t)2 : steps + __ldg(F.sa + (k >> F.sa_shift));
    }
}

// The full suffix array from the sampled one: sampled row s holds its sample, and the
// rows LF(s), LF^2(s), ... up to the next sampled row hold sa(s) - 1, sa(s) - 2, ...
// (bwt_sa's own walk, read backwards: every row's walk ends at the sampled row this
// fill starts from, so each row gets the value bwt_sa gives it).  Row 0 answers BWA's
// sample, (uint64_t)-1; the rows after it count down from seq_len.
template <class P>
__global__ void sa_fill_kernel(DevFM F, int64_t n_sa, uint64_t *__restrict__ full, int *__restrict__ failed)
{
    const uint64_t mask = (1ull << F.sa_shift) - 1;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_sa; t += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t s = (uint64_t)t << F.sa_shift;
        if (s > F.seq_len) continue;
        const uint64_t sv = F.sa[t];
        full[s] = sv;
        uint64_t v = s == 0 ? F.seq_len : sv;
        P k = (P)s;
        for (uint64_t step = 0;; ++step) {
            if (step >= kMaxWalk) {                      // not a valid index: the walk is kept
                atomicExch(failed, 1);
                break;
            }
            k = lf_step<P>(F, k);
            if (!(k & (P)mask)) break;                     // the next sampled row starts its own run
            full[k] = --v;
        }
    }
}

}  // namespace

// Builds the k-mer table of an index (kmer_bytes(F.wide) bytes) on the stream.
size_t kmer_bytes(bool wide) { return (size_t)kKmers * (wide ? 32 : 16); }
cudaError_t kmer_build(const DevFM &F, void *out, cudaStream_t st)
{
    const unsigned blocks = kKmers / 16 / 128;
    if (F.wide) kmer_kernel<uint64_t><<<blocks, 128, 0, st>>>(F, (uint4 *)out);
    else kmer_kernel<uint32_t><<<blocks, 128, 0, st>>>(F, (uint4 *)out);
    return cudaGetLastError();
}

template <class P>
static int again_blocks_per_sm(size_t smem)
{
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, seed_again_kernel<P>, kSeedBlock, smem) != cudaSuccess || b < 1)
        b = 4;
    return b;
}

// The launch shape of a batch.  slots: reads a warp packs and runs side by side (32, 16 where that
// would take more than 48 KB of shared memory a block).  split: warps that share a list of pass 1
// matches: enough to fill the GPU, and at least four, which even out the lists (67k reads of 150
// bases, seeding stage: 1.28 ms at 2, 1.30 at 3, 1.24 at 4, 1.26 at 6 and 8).  32 warps per SM at 64
// registers: 40 at 48 registers 1.29, 48 at 40 2.1.  The lists of pass 1 and 2 share the memory.
SeedPlan seed_plan(int n_sm, int64_t total_bases, int max_len, int n_reads, bool wide)
{
    const bool narrow = !wide;
    const size_t entry = narrow ? sizeof(Match32) : sizeof(Match64);
    SeedPlan p;
    p.slots = max_len <= 512 ? 32 : 16;
    p.smem = kSeedWarps * (64 * entry + sizeof(uint32_t) * (size_t)p.slots *
                                            (size_t)(chunk_words(max_len) + chunk_masks(max_len)));
    const int64_t lists = (n_reads + p.slots - 1) / p.slots, warps = (int64_t)n_sm * 32;
    p.split = (int)std::min<int64_t>(32, std::max<int64_t>(4, (warps + lists - 1) / lists));
    // pass 2: no more warps than there are re-seeds to expect (a few a read), fewer for long reads,
    // whose lists would take more than 1 GB
    const size_t per_block = (size_t)kSeedWarps * p.slots * (size_t)(max_len + 1) * entry, budget = (size_t)1 << 30;
    int64_t blocks = (int64_t)n_sm * (narrow ? again_blocks_per_sm<uint32_t>(p.smem) : again_blocks_per_sm<uint64_t>(p.smem));
    blocks = std::min<int64_t>(blocks, std::max<int64_t>(1, (int64_t)(budget / per_block)));
    p.again_blocks = (int)std::max<int64_t>(1, std::min<int64_t>(blocks, n_reads));
    p.counts_bytes = sizeof(int2) * (size_t)lists;
    p.list_entries = total_bases + n_reads;
    p.list_bytes = std::max((size_t)p.again_blocks * per_block, (size_t)p.list_entries * entry);
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
                        const SeedOut &S, void *d_lists, int2 *d_counts, const SeedPlan &p, cudaStream_t st)
{
    using Match = typename MatchOf<P>::type;
    const int lists = (n_reads + p.slots - 1) / p.slots;
    const auto blocks = [](int64_t warps) { return (unsigned)((warps + kSeedWarps - 1) / kSeedWarps); };
    seed_forward_kernel<P><<<blocks(2 * (int64_t)lists), kSeedBlock, p.smem, st>>>(F, o, n_reads, max_len, p.slots, d_seqs,
                                                                                   S, (Match *)d_lists, p.list_entries, d_counts);
    seed_backward_kernel<P><<<blocks((int64_t)lists * p.split), kSeedBlock, p.smem, st>>>(
        F, o, n_reads, max_len, p.slots, p.split, d_seqs, S, (const Match *)d_lists, p.list_entries, d_counts);
    seed_again_kernel<P><<<p.again_blocks, kSeedBlock, p.smem, st>>>(F, o, max_len, p.slots, d_seqs, S, (Match *)d_lists);
}

cudaError_t seed_launch(const DevFM &F, int min_seed_len, float split_factor, int split_width, int max_mem_intv,
                        int n_reads, const uint8_t *d_seqs, const int64_t *d_offs, int max_len,
                        void *d_padded, int *d_count, int64_t *d_out_off, void *d_out,
                        const SeedPlan &p, void *d_lists, void *d_list_counts, int *d_ctrl, void *d_queue, int64_t queue_cap, int *d_tot,
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
    int2 *const d_counts = (int2 *)d_list_counts;
    if (F.wide) seed_passes<uint64_t>(F, o, n_reads, max_len, d_seqs, S, d_lists, d_counts, p, st);
    else seed_passes<uint32_t>(F, o, n_reads, max_len, d_seqs, S, d_lists, d_counts, p, st);
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
    (F.wide ? sa_fill_kernel<uint64_t> : sa_fill_kernel<uint32_t>)<<<blocks > 0 ? blocks : 1, 256, 0, st>>>(F, n_sa, full, failed);
    return cudaGetLastError();
}

cudaError_t sa_launch(const DevFM &F, const uint64_t *d_rows, int64_t n, uint64_t *d_pos, int n_sm, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    const int64_t want = (n + 255) / 256;
    const int blocks = (int)(want < (int64_t)n_sm * 16 ? want : (int64_t)n_sm * 16);
    (F.wide ? sa_kernel<uint64_t> : sa_kernel<uint32_t>)<<<blocks, 256, 0, st>>>(F, d_rows, n, d_pos);
    return cudaGetLastError();
}
