// fm_index.cuh -- device view of the FM-index and the occurrence primitives.
//
// The occurrence array holds the reference's information (bwt.h:70-78,
// bwtindex.c:151-173: per 128 BWT symbols four uint64 cumulative counts and
// eight uint32 words of 2-bit symbols) re-cut at upload (occ_sectors_kernel) into one
// 32-byte sector per 64 symbols, so an occurrence query reads one sector: two 16-byte
// loads of one transaction, at the reference's density (0.5 byte per row).
//
// What a query wants is not a base's count alone: bwt_extend by base c needs the
// occurrences of c and, for the other strand's interval, of the bases above c.  Both follow
// from two cumulative counts, the symbols >= c and the symbols > c, so a sector holds the
// counts of symbols > A, > C and > G before it, and its symbols as two bit planes (lo, hi; the
// first symbol in bit 0): "symbol >= k" is one expression of the planes, and each cumulative
// count two population counts.  Against 32-symbol sectors with a count per base and symbols two
// bits apart: half the bytes (more of the index in L2), 8 population counts an extension
// instead of 12, and no 64-bit arithmetic for an index below 2^32 rows.
#pragma once

#include <stdint.h>

struct DevFM {
    const uint4 *blk;        // 32-byte occurrence sectors
    const uint64_t *sb;      // symbols > A, > C, > G before each 2^32-row superblock
    const uint4 *kmers;      // bi-interval of every kKmer-base string (KmerOf<P>), or NULL
    const uint64_t *sa;      // sampled suffix array, sa[0] = (uint64_t)-1
    const uint64_t *sa_full; // every row's bwt_sa value (seq_len + 1 entries), or NULL
    uint64_t primary;
    uint64_t seq_len;
    uint64_t L2[5];
    int sa_shift;            // log2(sa_intv)
    int wide;                // seeding and its table in 64 bits
};

// An index below this many rows is seeded in 32 bits.
constexpr uint64_t kNarrowRows = 0xfffffffdull;

struct DevIntv {             // bwtintv_t (bwt.h:60-62)
    uint64_t x0, x1, x2, info;
};

// Sector s: {symbols > A, > C, > G in the rows of its superblock before it, 0},
// {lo plane of symbols 0-31, lo of 32-63, hi of 0-31, hi of 32-63}.
constexpr int kSectorSyms = 64;

// The table of bi-intervals (x0, x1, x2) by string, the first base in the code's highest bits: 16
// bytes an entry (0.27 GB) for an index below 2^32 rows, else 32.
constexpr int kKmer = 12;
constexpr uint32_t kKmers = 1u << (2 * kKmer);

// 32 bytes in one transaction.
__device__ __forceinline__ void load32(const uint4 *p, uint32_t (&v)[8])
{
    asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "l"(p));
}

// Counts of A, C, G among the first n (0..16) symbols of x, a word of the reference's array (most
// significant pair first).
__device__ __forceinline__ void word_counts(uint32_t x, int n, uint32_t &a, uint32_t &c, uint32_t &g)
{
    const uint32_t keep = n >= 16 ? 0xffffffffu : ~(0xffffffffu >> (2 * n));
    const uint32_t hi = (x >> 1) & 0x55555555u, lo = x & 0x55555555u;
    a += __popc(~(hi | lo) & 0x55555555u & keep);
    c += __popc(lo & ~hi & keep);
    g += __popc(hi & ~lo & keep);
}

// F.L2[i] for i = 0..4, indexed with constants only (a dynamic index would copy the
// kernel parameter to local memory).
template <class P = uint64_t>
__device__ __forceinline__ P l2_at(const DevFM &F, int i)
{
    return i == 0   ? (P)F.L2[0]
           : i == 1 ? (P)F.L2[1]
           : i == 2 ? (P)F.L2[2]
           : i == 3 ? (P)F.L2[3]
                    : (P)F.L2[4];
}

// Row k of the BWT as a position of its $-free array (bwt_occ4's adjustment, bwt.c:176), held inside
// the array: k is at most seq_len on a valid index, so the clamp then changes nothing.
template <class P>
__device__ __forceinline__ P sym_row(const DevFM &F, P k)
{
    k -= k >= (P)F.primary;
    return k < (P)F.seq_len ? k : (P)F.seq_len - 1;
}

template <class P>
__device__ __forceinline__ const uint4 *sector_of(const DevFM &F, P kk)
{
    return F.blk + (uint64_t)(kk >> 6) * 2;
}

// Symbols >= c and > c in rows [0, kk] of the $-free BWT (bwt_occ4, bwt.c:169-187), w the sector of
// kk.  P: uint32_t for an index below 2^32 rows, which has one superblock, else uint64_t.
template <class P>
__device__ __forceinline__ void occ_cumulative(const DevFM &F, const uint32_t (&w)[8], P kk, int c, P &ge, P &gt)
{
    const uint4 v = make_uint4(w[0], w[1], w[2], w[3]), s = make_uint4(w[4], w[5], w[6], w[7]);
    const uint64_t keep = ~0ull >> (63 - (int)(kk & 63));
    const uint32_t k0 = (uint32_t)keep, k1 = (uint32_t)(keep >> 32);
    // [symbol >= t] = (hi | lo & x) & (lo | y): hi|lo for t = 1, hi for 2, hi&lo for 3
    const uint32_t xe = c == 1 ? ~0u : 0u, ye = c <= 2 ? ~0u : 0u;       // t = c (c = 0 counts every symbol)
    const uint32_t xg = c == 0 ? ~0u : 0u, yg = c <= 1 ? ~0u : 0u;       // t = c + 1 (c = 3 counts none)
    const uint32_t ne = __popc((s.z | (s.x & xe)) & (s.x | ye) & k0) + __popc((s.w | (s.y & xe)) & (s.y | ye) & k1);
    const uint32_t ng = __popc((s.z | (s.x & xg)) & (s.x | yg) & k0) + __popc((s.w | (s.y & xg)) & (s.y | yg) & k1);
    P be = c == 1 ? v.x : c == 2 ? v.y : v.z, bg = c == 0 ? v.x : c == 1 ? v.y : v.z;
    if (sizeof(P) == 8) {
        const uint64_t *b = F.sb + 3 * ((uint64_t)kk >> 32);
        be += (P)__ldg(b + (c == 0 ? 0 : c - 1));
        bg += (P)__ldg(b + (c == 3 ? 2 : c));
    }
    ge = c == 0 ? kk + 1 : be + ne;
    gt = c == 3 ? 0 : bg + ng;
}

// One LF step of bwt_sa (bwt_invPsi, bwt.c:53-59): the row of the suffix one text
// position earlier; the primary row steps to row 0 (BWA's "$" convention).
template <class P>
__device__ __forceinline__ P lf_step(const DevFM &F, P k)
{
    if (k == (P)F.primary) return 0;
    // the symbol row (bwt_invPsi uses k > primary, bwt.c:55) equals the counted row here
    const P kk = sym_row<P>(F, k);
    uint32_t w[8];
    load32(sector_of<P>(F, kk), w);
    const int n = (int)(kk & 31);
    const uint32_t lo = (kk & 32) ? w[5] : w[4], hi = (kk & 32) ? w[7] : w[6];
    const int c = (int)(lo >> n & 1u) | (int)(hi >> n & 1u) << 1;
    P ge, gt;
    occ_cumulative<P>(F, w, kk, c, ge, gt);
    return l2_at<P>(F, c) + ge - gt;
}
