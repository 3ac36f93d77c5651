// sw_pack.cuh -- ksw_align2's striped passes (bsbolt/External/BWA/ksw.c:111-327) with two
// SIMD lanes per thread, for sm_103a.
//
// The reference's results depend on its SSE2 striping (the query cut into slen segments of P
// lanes, column j + l*slen in lane l of segment j; F carried along a lane's stripe in the first
// pass, E and the row maximum taken from that pass, the lazy-F loop fixing H for the next row).
// Here thread t of a group of P/2 plays SIMD lanes t (low 16 bits) and t + P/2 (high 16 bits):
//   P = 16, byte lanes (ksw_u8), for matrices with an entry <= 0: then shift = -min, and a score that the
//     reference's bytes would clip puts the row's maximum at 255 - shift or above, where the pass ends with
//     score 255 whatever the rest of the row holds.  So signed scores in 16 bits, without a clip, are exact.
//     (Matrices without one leave every H at 0: sw.cu hands in scores that do.)
//   P = 8, word lanes (ksw_i16): the same instructions, for jobs whose scores
//     cannot reach the reference's 16-bit saturation (qlen * max score <= 32640) and whose
//     penalties stay below 32768, so that 16-bit arithmetic without saturation is exact.
// A job's H and E vectors and its query-profile selectors are register arrays sized by its
// segment count's bucket (below); the row's scores come from two profile words of its
// target base by one byte permute per pair of cells.  The lazy-F loop runs in closed form (see
// pack_pass).  The groups of a warp take consecutive jobs of a list sorted by segment count and go through
// their rows in step, so that every exchange and vote is the whole warp's.
#pragma once

#include <cstdint>

#include "bsb_internal.cuh"

namespace bsbsw {

constexpr int kXByte = 0x10000, kXStop = 0x20000, kXSubo = 0x40000, kXStart = 0x80000;
constexpr int kPackBlock = 128;
constexpr int kPackMaxSeg8 = 16;    // byte lanes: queries of up to 256 bases
constexpr int kPackMaxSeg16 = 40;   // word lanes: queries of up to 320 bases
// counter block of one lane width: [0..3] queues, [kRcnt + s] reverse passes of s segments,
// [kRcur + s] their scatter cursors
constexpr int kRcnt = 64, kRcur = 128, kCtrInts = 192;

struct PassOut {
    int score, te, qe, score2, te2;
};

struct PackParams {
    // per target base: the scores of query bases 0..3 (x), and of base 4 and the padding column, whose
    // score is 0 (y), as signed bytes; the last for rows past a target's end: every score 0
    uint2 prof[6];
    uint32_t npe_del, npoe_del, npe_ins, npoe_ins;         // negated penalties in both halves
    int shift, qmax, pe_ins;
};

// A pass's query and target: forward (qe = te = -1) or the reverse pass of ksw_align2
// (ksw.c:350): query[0..qe] reversed, target[0..te] reversed and the rest as is.
struct SwSeq {
    const uint8_t *q, *t;
    int qe, te;
    __device__ __forceinline__ int qc(int c) const { return qe < 0 ? q[c] : q[qe - c]; }
    __device__ __forceinline__ int tc(int i) const { return t[i <= te ? te - i : i]; }
};

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel)   // bit 3 of a nibble: sign fill
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

__host__ __device__ __forceinline__ uint32_t neg2(int v) { return (uint32_t)(uint16_t)(-v) * 0x10001u; }

constexpr unsigned kAll = 0xffffffffu;

template <int G>
__device__ __forceinline__ uint32_t lane_up(uint32_t x, int tid)   // _mm_slli_si128 by one lane
{
    const uint32_t r = __shfl_sync(kAll, x, (tid + G - 1) & (G - 1), G);
    return prmt(r, 0u, tid ? 0x3210u : 0x1044u);
}

// maximum / minimum over the group's threads (G of them)
template <int G>
__device__ __forceinline__ int grp_max(int v)
{
#pragma unroll
    for (int d = G / 2; d > 0; d >>= 1) v = max(v, __shfl_xor_sync(kAll, v, d, G));
    return v;
}

template <int G>
__device__ __forceinline__ int grp_min(int v)
{
#pragma unroll
    for (int d = G / 2; d > 0; d >>= 1) v = min(v, __shfl_xor_sync(kAll, v, d, G));
    return v;
}

// Segment counts per pass instance: a bucket of B consecutive counts (SLMAX - B, SLMAX] shares
// one instance, the exact count sl a runtime value: the striping uses sl, segments at and past
// sl are skipped (only the last B - 1 of the instance's segments test it).  Eight byte-lane and
// four word-lane instances keep the code the SMs run at one time small: with one instance per
// count, instruction fetch was the kernel's main stall.
template <int P>
constexpr int kSegBucket = P == 16 ? 2 : 8;

// The ksw_u8 (P = 16) or ksw_i16 (P = 8) passes of a warp's groups of P/2 threads, each on its own job of sl
// segments, SLMAX - kSegBucket < sl <= SLMAX (a group without one: qlen = tlen = 0).  hm: the thread's Hmax slots
// (stride kPackBlock); bbuf: the suboptimal rows (KSW_XSUBO only).
//
// Bound by the integer pipe, which takes a warp's instruction every second clock (81 % busy, 117 of its
// instructions a row of 10 segments).  Hence: no clip and no relu that another instruction implies (7 instructions
// a segment, 9 before); the groups in step, since an exchange or vote under a group's own mask is carried out
// group by group with a synchronisation each (40 instructions a row went there); the row's maximum only compared,
// and reduced where it matters; and registers for the widest instance without spills (4 blocks an SM; at 5, 6 and 7
// the call below takes 2.08, 2.21 and 2.31 ms).  40k mates of 30-250 bases against 500-base windows, forward
// passes: 1.76 ms before, 1.22 now, the word-lane mates beside them 1.21 and 0.80; the call 2.72 and 2.00.
template <int P, int SLMAX>
__device__ __noinline__ PassOut pack_pass(const PackParams &S, const uint2 *prof, int sl, int qlen, int tlen,
                                          const SwSeq &a, int xtra, uint32_t *hm, int2 *bbuf, int tid)
{
    constexpr bool U8 = P == 16;
    constexpr int G = P / 2, SLMIN = SLMAX - kSegBucket<P> + 1;    // segments below SLMIN always exist
    const uint32_t npe_del = S.npe_del, npoe_del = S.npoe_del, npe_ins = S.npe_ins, npoe_ins = S.npoe_ins;
    const uint32_t oe_ins = neg2((int)(int16_t)(npoe_ins & 0xffffu));
    const int shift = S.shift, pe_ins = S.pe_ins;
    const uint32_t npe_one = 0u - (uint32_t)pe_ins * 0x10001u;     // one e_ins less in both halves of -j * e_ins, j >= 1
    uint32_t sel[SLMAX], H[SLMAX], E[SLMAX];
#pragma unroll
    for (int j = 0; j < SLMAX; ++j) {              // ksw_qinit's striping; the vectors start at zero
        const int c0 = j + tid * sl, c1 = j + (tid + G) * sl;
        const bool in = j < sl;
        const uint32_t x = in && c0 < qlen ? (uint32_t)a.qc(c0) : 5u, y = in && c1 < qlen ? (uint32_t)a.qc(c1) : 5u;
        sel[j] = x | (x | 8u) << 4 | y << 8 | (y | 8u) << 12;      // bytes: score(x), its sign, score(y), its sign
        H[j] = 0, E[j] = 0;
        hm[j * kPackBlock] = 0;
    }
    const int minsc = (xtra & kXSubo) ? xtra & 0xffff : 0x10000;
    const int endsc = (xtra & kXStop) ? xtra & 0xffff : 0x10000;
    int gmax = 0, te = -1, n_b = 0, last_row = -2, last_sc = 0;
    // rows whose maximum is above lim (in both halves) are looked at: min(gmax, minsc - 1)
    const int low = min(minsc, 0x8000) - 1;
    uint32_t lim = (uint32_t)(uint16_t)min(gmax, low) * 0x10001u;
    uint32_t hlast = 0;                            // H of segment sl - 1 in the previous row
    // the lazy F's scan: what a lane's G loses on the way o lanes up (a thread without a lane there: all of it),
    // and from the last low lane to this thread's high one
    const int d = pe_ins * sl;
    uint32_t up[3];
#pragma unroll
    for (int o = 1, k = 0; o < G; o <<= 1, ++k) up[k] = tid >= o ? neg2(min(o * d, 32767)) : 0x80008000u;
    const uint32_t low_up = neg2(min(d * (tid + 1), 32767)) & 0xffff0000u;
    const unsigned my_group = ((1u << G) - 1u) << (threadIdx.x & 31 & ~(G - 1));
    int tmax = __reduce_max_sync(kAll, tlen);
    int tb = tid < tlen ? a.tc(tid) : 5;           // a row's base, one a thread for G rows
    uint2 pr = prof[__shfl_sync(kAll, tb, 0, G)];
    int i = 0;
    while (i < tmax) {
        int tn = i + G + tid < tlen ? a.tc(i + G + tid) : 5;
#pragma unroll 1
        for (int r = 0; r < G && i < tmax; ++r, ++i) {
            const uint32_t xlo = pr.x, xhi = pr.y;
            pr = prof[__shfl_sync(kAll, r + 1 < G ? tb : tn, (r + 1) & (G - 1), G)];
            uint32_t h = lane_up<G>(hlast, tid), F = oe_ins, mx = 0;     // H(i-1, -1), ksw.c:141-142
            // H = max(a, E, f), a = the diagonal plus the score (ksw.c:149-153); the next f is
            // max(relu(f - e_ins), relu(H - oe_ins)) = relu(max(f - e_ins, max(a, E) - oe_ins)), as
            // relu(f - oe_ins) <= relu(f - e_ins).  F = f + oe_ins, not held at zero (H is): one instruction a
            // segment, and one for H
#pragma unroll
            for (int j = 0; j < SLMAX; ++j)
                if (j < SLMIN || j < sl) {
                    const uint32_t ae = __viaddmax_s16x2(h, prmt(xlo, xhi, sel[j]), E[j]);
                    const uint32_t hv = __viaddmax_s16x2_relu(F, npoe_ins, ae);
                    F = __viaddmax_s16x2(F, npe_ins, ae);
                    if (j < SLMIN && (j & 1)) mx = __vimax3_s16x2_relu(mx, hv, H[j - 1]);
                    else if (j >= SLMIN - (SLMIN & 1)) mx = __vimax_s16x2_relu(mx, hv);
                    E[j] = __viaddmax_s16x2(E[j], npe_del, __viaddmax_s16x2(hv, npoe_del, 0u));
                    h = H[j];
                    H[j] = hv;
                }
            {   // lazy F (ksw.c:166-177, 284-295).  The reference shifts f up one lane per round and
                // sweeps the segments until no lane can raise an H any more.  The sweep raises H(l, j)
                // to relu(G(l) - j*e_ins) at most, where G(l) is the F arriving at lane l's first
                // column: G(0) = 0, G(l) = max(x(l), relu(G(l-1) - sl*e_ins)), x(l) the f leaving lane
                // l-1; its early exit (Farrar's) leaves out only updates that change nothing.  So: the
                // reference's own first test, and where a lane fails it, G as a max-plus scan over its group's
                // lanes (the group's threads, then the low lanes into the high ones) and one max per
                // segment, without a vote per segment.  (Segments past sl take values nothing reads.)
                const uint32_t x = lane_up<G>(__viaddmax_s16x2(F, npoe_ins, 0u), tid);
                const uint32_t h0 = __vimax_s16x2_relu(H[0], x);
                const uint32_t hh = __viaddmax_s16x2(h0, npoe_ins, 0u), fn = __viaddmax_s16x2(x, npe_ins, 0u);
                H[0] = h0;
                const unsigned fail = __ballot_sync(kAll, __vimax_s16x2_relu(fn, hh) != hh);
                if (fail) {
                    uint32_t g = x;
#pragma unroll
                    for (int o = 1, k = 0; o < G; o <<= 1, ++k)
                        g = __viaddmax_s16x2(__shfl_up_sync(kAll, g, o, G), up[k], g);
                    g = __viaddmax_s16x2(__shfl_sync(kAll, g, G - 1, G) << 16, low_up, g);
                    if (!(fail & my_group)) g = 0;       // a group without a failing lane keeps its H as they are
                    H[0] = __vimax_s16x2_relu(H[0], g);
                    if (U8) {                            // at most 15 * 255 down
                        uint32_t down = npe_ins;
#pragma unroll
                        for (int j = 1; j < SLMAX; ++j) {
                            H[j] = __viaddmax_s16x2(g, down, H[j]);
                            down += npe_one;
                        }
                    } else {
#pragma unroll
                        for (int j = 1; j < SLMAX; ++j) {
                            g = __viaddmax_s16x2(g, npe_ins, 0u);
                            H[j] = __vimax_s16x2_relu(H[j], g);
                        }
                    }
                }
            }
            hlast = H[SLMIN - 1];
#pragma unroll
            for (int j = SLMIN; j < SLMAX; ++j)
                if (j == sl - 1) hlast = H[j];
            if (__any_sync(kAll, __viaddmax_s16x2(mx, 0u, lim) != lim)) {
#pragma unroll
                for (int d = G / 2; d > 0; d >>= 1) mx = __vimax_s16x2_relu(mx, __shfl_xor_sync(kAll, mx, d, G));
                const int imax = max((int)(mx & 0xffffu), (int)(mx >> 16));
                bool ends = false;
                if (i < tlen) {
                    if (imax >= minsc) {              // the rows of the suboptimal score (ksw.c:182-189)
                        if (n_b == 0 || last_row + 1 != i) {
                            if (tid == 0) bbuf[n_b] = make_int2(imax, i);
                            ++n_b, last_row = i, last_sc = imax;
                        } else if (last_sc < imax) {
                            if (tid == 0) bbuf[n_b - 1] = make_int2(imax, i);
                            last_row = i, last_sc = imax;
                        }
                    }
                    if (imax > gmax) {
                        gmax = imax, te = i;
                        lim = (uint32_t)(uint16_t)min(gmax, low) * 0x10001u;
#pragma unroll
                        for (int j = 0; j < SLMAX; ++j) hm[j * kPackBlock] = H[j];
                        ends = (U8 && gmax + shift >= 255) || gmax >= endsc;
                    }
                } else {                             // past this group's target
                    lim = 0x7fff7fffu;
                }
                if (ends) tlen = i + 1, tb = tn = 5;
                if (__any_sync(kAll, ends)) tmax = __reduce_max_sync(kAll, tlen);
            }
        }
        tb = tn;
    }
    __syncwarp();
    PassOut r;
    r.score = U8 ? (gmax + shift < 255 ? gmax : 255) : gmax;
    r.te = te, r.qe = -1, r.score2 = -1, r.te2 = -1;
    const bool whole = !U8 || r.score != 255;
    int best = -1, col = 0x7fffffff;              // the smallest column holding the best Hmax value
#pragma unroll 1
    for (int j = 0; j < sl; ++j) {
        const uint32_t v = hm[j * kPackBlock];
        const int v0 = (int)(v & 0xffffu), v1 = (int)(v >> 16), c0 = j + tid * sl, c1 = j + (tid + G) * sl;
        if (v0 > best || (v0 == best && c0 < col)) best = v0, col = c0;
        if (v1 > best || (v1 == best && c1 < col)) best = v1, col = c1;
    }
    __syncwarp();
    const int gbest = grp_max<G>(best), qe = grp_min<G>(best == gbest ? col : 0x7fffffff);
    if (whole) r.qe = qe;
    if (__any_sync(kAll, n_b != 0)) {              // ksw.c:218-225: the best row outside te +- d
        const int reach = (r.score + S.qmax - 1) / S.qmax, lo = te - reach, hi = te + reach;
        int bs = -1, bk = 0x7fffffff;
#pragma unroll 1
        for (int k = tid; k < n_b; k += G) {
            const int2 e = bbuf[k];
            if ((e.y < lo || e.y > hi) && e.x > bs) bs = e.x, bk = k;
        }
        __syncwarp();
        const int gbs = grp_max<G>(bs);
        const int gk = grp_min<G>(bs == gbs ? bk : 0x7fffffff);
        if (whole && n_b && gbs > r.score2 && gk != 0x7fffffff) r.score2 = gbs, r.te2 = bbuf[gk].y;
    }
    return r;
}

// pack_pass of the bucket ending at hi (the same in the whole warp), for buckets ending at SLMAX..HI (step
// kSegBucket<P>).  Each instance is a function of its own, so a kernel's registers are those of its largest.
template <int P, int SLMAX, int HI>
__device__ __forceinline__ PassOut pack_range(int hi, const PackParams &S, const uint2 *prof, int sl, int qlen,
                                              int tlen, const SwSeq &a, int xtra, uint32_t *hm, int2 *bbuf, int tid)
{
    if constexpr (SLMAX >= HI) {
        return pack_pass<P, HI>(S, prof, sl, qlen, tlen, a, xtra, hm, bbuf, tid);
    } else {
        if (hi <= SLMAX) return pack_pass<P, SLMAX>(S, prof, sl, qlen, tlen, a, xtra, hm, bbuf, tid);
        return pack_range<P, SLMAX + kSegBucket<P>, HI>(hi, S, prof, sl, qlen, tlen, a, xtra, hm, bbuf, tid);
    }
}

// Jobs of LO..HI segments of P lanes (MAXS: the largest segment count of the lane width).
// REV = false: forward passes of list[0..n_fwd) (rsl[id] = the segment count of the reversed
// query when the job wants start positions, else 0; ctr[kRcnt + s] counts them).  REV = true:
// reverse passes of the jobs of list (grouped by segment count, the largest first, by
// sw_rev_scatter) whose reversed query has LO..HI segments, completing tb and qb.  Each warp
// takes 64/P consecutive jobs of its list at a time; q is the queue counter.
template <int P, bool REV, int LO, int HI, int MAXS>
__global__ void __launch_bounds__(kPackBlock, P == 16 ? 4 : 1)
sw_pack_kernel(PackParams S, const bsb_sw_job_t *__restrict__ jobs, const uint8_t *__restrict__ seq,
               const int32_t *__restrict__ list, int n_fwd, const int64_t *__restrict__ boff,
               int2 *__restrict__ bscratch, bsb_kswr_t *__restrict__ out, uint8_t *__restrict__ rsl,
               int *__restrict__ ctr, int *__restrict__ q)
{
    constexpr int G = P / 2, NG = 32 / G, B = kSegBucket<P>;
    __shared__ uint32_t hmax_s[HI * kPackBlock];
    __shared__ uint2 prof[6];
    if (threadIdx.x == 0) {
#pragma unroll
        for (int c = 0; c < 6; ++c) prof[c] = S.prof[c];
    }
    __syncthreads();
    int total = n_fwd;
    if (REV) {                                   // this range's part of the reverse list
        int skip = 0;
        total = 0;
        for (int s = MAXS; s > HI; --s) skip += ctr[kRcnt + s];
        for (int s = HI; s >= LO; --s) total += ctr[kRcnt + s];
        list += skip;
    }
    const int wl = threadIdx.x & 31, g = wl / G, tid = wl % G;
    uint32_t *hm = hmax_s + threadIdx.x;
    for (;;) {
        int base = 0;
        if (wl == 0) base = atomicAdd(q, NG);
        base = __shfl_sync(kAll, base, 0);
        if (base >= total) break;
        const int k = base + g;
        int id = 0, left = 0, qlen = 0, tlen = 0, xtra = 0;        // left: the segments of a job still to be run
        SwSeq a{seq, seq, -1, -1};
        int2 *bbuf = nullptr;
        bsb_kswr_t o{};
        if (k < total) {
            id = list[k];
            const bsb_sw_job_t jb = jobs[id];
            a.q += jb.qoff, a.t += jb.toff;
            tlen = jb.tlen;
            if (!REV) {
                qlen = jb.qlen, xtra = jb.xtra, bbuf = bscratch + boff[id];
            } else {
                o = out[id];
                a.qe = o.qe, a.te = o.te;
                qlen = o.qe + 1, xtra = kXStop | o.score;
            }
            left = (qlen + P - 1) / P;
        }
        // a list sorted by segment count gives a warp jobs of one bucket but at the buckets' borders
        for (int top; (top = __reduce_max_sync(kAll, left)) > 0;) {
            const int hi = LO + B - 1 + (top - LO) / B * B;
            const bool mine = left > hi - B;
            const PassOut r = pack_range<P, LO + B - 1, HI>(hi, S, prof, mine ? left : hi, mine ? qlen : 0,
                                                            mine ? tlen : 0, a, mine ? xtra : 0, hm, bbuf, tid);
            if (mine && tid == 0) {
                if (!REV) {
                    const bool start = (xtra & kXStart) && !((xtra & kXSubo) && r.score < (xtra & 0xffff));
                    o.score = r.score, o.te = r.te, o.qe = r.qe, o.score2 = r.score2, o.te2 = r.te2;
                    o.tb = -1, o.qb = -1;
                    out[id] = o;
                    // a saturated byte pass leaves qe at -1, where the reference would profile no columns
                    const int sl = start && r.qe >= 0 ? (r.qe + P) / P : 0;
                    rsl[id] = (uint8_t)sl;
                    if (sl) atomicAdd(&ctr[kRcnt + sl], 1);
                } else if (r.score == o.score) {
                    out[id].tb = o.te - r.te, out[id].qb = o.qe - r.qe;
                }
            }
            if (mine) left = 0;
        }
        __syncwarp();
    }
}

// Lists the jobs of list[0..n) that want a reverse pass, grouped by its segment count (the
// largest first).
template <int MAXS>
__global__ void sw_rev_scatter(const int32_t *__restrict__ list, int n, const uint8_t *__restrict__ rsl,
                               int *__restrict__ ctr, int32_t *__restrict__ rlist)
{
    __shared__ int off[MAXS + 1];
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int s = MAXS; s >= 1; --s) off[s] = acc, acc += ctr[kRcnt + s];
    }
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int id = list[i], s = rsl[id];
        if (s) rlist[off[s] + atomicAdd(&ctr[kRcur + s], 1)] = id;
    }
}

// One sw_pack_kernel launch on st: the forward passes of list[0..n) or (rev) the reverse passes
// of this range.  ctr: the lane width's counter block; ctr[q] the queue.
template <int P, int LO, int HI, int MAXS>
cudaError_t sw_pack_run(bool rev, const PackParams &S, const bsb_sw_job_t *jobs, const uint8_t *seq,
                        const int32_t *list, int n, const int64_t *boff, int2 *bscratch, bsb_kswr_t *out,
                        uint8_t *rsl, int *ctr, int q, int n_sm, cudaStream_t st)
{
    static int resident[2] = {};
    if (!resident[0]) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident[0], sw_pack_kernel<P, false, LO, HI, MAXS>,
                                                      kPackBlock, 0);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident[1], sw_pack_kernel<P, true, LO, HI, MAXS>,
                                                      kPackBlock, 0);
        resident[0] = resident[0] > 0 ? resident[0] : 1, resident[1] = resident[1] > 0 ? resident[1] : 1;
    }
    const int per_block = kPackBlock * 2 / P;              // jobs in flight per block
    const int64_t want = ((int64_t)n + per_block - 1) / per_block, cap = (int64_t)n_sm * resident[rev ? 1 : 0];
    const int grid = (int)(want < cap ? want : cap);
    if (grid <= 0) return cudaSuccess;
    if (rev)
        sw_pack_kernel<P, true, LO, HI, MAXS><<<grid, kPackBlock, 0, st>>>(S, jobs, seq, list, 0, boff, bscratch,
                                                                           out, rsl, ctr, ctr + q);
    else
        sw_pack_kernel<P, false, LO, HI, MAXS><<<grid, kPackBlock, 0, st>>>(S, jobs, seq, list, n, boff, bscratch,
                                                                            out, rsl, ctr, ctr + q);
    return cudaGetLastError();
}

// The word-lane ranges, each in a translation unit of its own (sw_pack16a.cu: 1..16 segments,
// sw_pack16b.cu: 17..40) so that they compile side by side.
cudaError_t sw_pack16_run_lo(bool rev, const PackParams &S, const bsb_sw_job_t *jobs, const uint8_t *seq,
                             const int32_t *list, int n, const int64_t *boff, int2 *bscratch, bsb_kswr_t *out,
                             uint8_t *rsl, int *ctr, int q, int n_sm, cudaStream_t st);
cudaError_t sw_pack16_run_hi(bool rev, const PackParams &S, const bsb_sw_job_t *jobs, const uint8_t *seq,
                             const int32_t *list, int n, const int64_t *boff, int2 *bscratch, bsb_kswr_t *out,
                             uint8_t *rsl, int *ctr, int q, int n_sm, cudaStream_t st);

}  // namespace bsbsw
