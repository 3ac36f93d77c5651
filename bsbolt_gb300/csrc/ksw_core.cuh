// ksw_core.cuh -- the warp-cooperative, bit-exact ksw_extend2 (ksw.c:380-479).
//
// Shared by the batched extension kernels (ksw_extend.cu) and the per-read
// chain extension (chain.cu).  See ksw_extend.cu for the design notes.
#pragma once

#include <climits>

#include "bsb_internal.cuh"

struct KswResult {
    int score, qle, tle, gtle, gscore, max_off;
    long long cells;
};

// Sign-extended byte of x chosen by a prmt selector (bit 3 of each selector
// nibble replicates the sign of the chosen byte, PTX ISA prmt.b32 default mode).
__device__ __forceinline__ int prmt_sext(uint32_t x, uint32_t sel)
{
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(x), "r"(sel));
    return (int)r;
}

// Scores of target bases 0..3 against query base qc, one per byte:
// mat[c*5 + qc] for c = 0..3.  The matrix is only indexed with constants
// (selecting on qc), which keeps the kernel parameters out of local memory.
__device__ __forceinline__ uint32_t profile_word(const KswParams &P, int qc)
{
    uint32_t w[5];
#pragma unroll
    for (int b = 0; b < 5; ++b)
        w[b] = (uint32_t)(uint8_t)P.mat[b] | (uint32_t)(uint8_t)P.mat[5 + b] << 8 |
               (uint32_t)(uint8_t)P.mat[10 + b] << 16 | (uint32_t)(uint8_t)P.mat[15 + b] << 24;
    return qc == 0 ? w[0] : qc == 1 ? w[1] : qc == 2 ? w[2] : qc == 3 ? w[3] : w[4];
}

// mat[20 + qc]: the score of an N in the target against query base qc.
__device__ __forceinline__ int profile_n(const KswParams &P, int qc)
{
    return qc == 0 ? P.mat[20] : qc == 1 ? P.mat[21] : qc == 2 ? P.mat[22] : qc == 3 ? P.mat[23] : P.mat[24];
}

__device__ __forceinline__ uint32_t sext_selector(int byte)
{
    const uint32_t b = (uint32_t)byte, r = b | 8u;
    return b | r << 4 | r << 8 | r << 12;
}

// A job's query or target: bytes, or for the jobs of an alignment batch (Packed, see KswParams) the
// read's bytes and places of the forward-reverse text, either of them run backwards.
template <bool Packed> struct JobText;
template <> struct JobText<false> {
    const uint8_t *p = nullptr;
    __device__ __forceinline__ int byte(int i) const { return p[i]; }
    __device__ __forceinline__ uint32_t base(const KswParams &, int i) const { return p[i]; }
};
template <> struct JobText<true> {
    int64_t at = 0;
    int back = 0;
    __device__ __forceinline__ int byte(int i) const { return *(const uint8_t *)(at + (back ? -i : i)); }
    __device__ __forceinline__ uint32_t base(const KswParams &P, int i) const
    {
        return (uint32_t)packed_text_base(P.pac, P.l_pac, at + (back ? -i : i));
    }
};
template <bool Packed>
__device__ __forceinline__ JobText<Packed> job_query(const uint8_t *seq, const bsb_ext_job_t &jb)
{
    JobText<Packed> t;
    if constexpr (Packed) t.at = (int64_t)(seq + jb.qoff), t.back = jb.flags & kExtBack;
    else t.p = seq + jb.qoff;
    return t;
}
template <bool Packed>
__device__ __forceinline__ JobText<Packed> job_target(const uint8_t *seq, const bsb_ext_job_t &jb)
{
    JobText<Packed> t;
    if constexpr (Packed) t.at = jb.toff, t.back = jb.flags & kExtBack;
    else t.p = seq + jb.toff;
    return t;
}

// The scoring matrix as a shared table, score of target base t against query base q at
// t << 3 | q (bases above 4 are N, as in profile_word).
constexpr int kScoreTable = 40;
__device__ __forceinline__ void load_score_table(const KswParams &P, int8_t *tab)
{
    if (threadIdx.x < 25) {
        int v = 0;
#pragma unroll
        for (int k = 0; k < 25; ++k) v = (int)threadIdx.x == k ? P.mat[k] : v;
        tab[(threadIdx.x / 5) << 3 | threadIdx.x % 5] = (int8_t)v;
    }
}

// The loss a job's main diagonal must stay below for its result to be known without the DP
// (ksw_diagonal), 0 when the scoring never allows it.
__device__ __forceinline__ int diagonal_limit(const KswParams &P, int h0)
{
    int lim = min(P.o_del + P.e_del, P.o_ins + P.e_ins);
    if (P.zdrop > 0 && P.zdrop < lim) lim = P.zdrop + 1;         // (zdrop + 1 may not exist)
    return P.mat_max > 0 ? min(lim, h0 + P.mat_max) : 0;
}

// ksw_extend2 of a job whose query lies on its target's main diagonal with little loss, in one
// pass over the diagonal and no DP.  Let a = max(mat), D(i) = h0 + a(i+1) - L(i) the score of the
// diagonal through row i, L(i) what its columns lose against a.  Every other cell (i, j) pays at
// least one gap: H(i,j) <= h0 + a(min(i,j)+1) - (o + e|i-j|).  So while L stays below o + e of
// both gaps, D(i) is the strict maximum of row i (no tie), the band (which follows the non-zero
// cells) holds it, max_off stays 0, no row after the query's end and no other row's last column
// reaches D(qlen-1), and with L below h0 + a no D(i) is 0 and with L <= zdrop none drops far
// enough to stop: score is the diagonal's best prefix (the first one, since later ones have to
// exceed it), gscore = D(qlen-1) at row qlen-1.  Needs tlen >= qlen >= 1.  Returns false where the
// diagonal loses too much.  A group of G lanes takes a job, 32 columns a step (column k*G + lane of
// the group in slot k); all lanes of the warp call it, the groups with a job each (lim <= 0: none).
template <int G, class Acc>
__device__ __forceinline__ bool ksw_diagonal(const int8_t *tab, int a, int lim, int qlen, int tlen, int h0,
                                             const Acc &acc, int lane, int &best, int &best_j, int &last)
{
    constexpr int K = 32 / G;
    const int gl = lane & (G - 1), g0 = lane & ~(G - 1);
    bool on = lim > 0 && qlen >= 1 && tlen >= qlen;
    int loss = 0;
    best = h0, best_j = -1;
    for (int c0 = 0; __any_sync(BSB_FULL_MASK, on && c0 < qlen); c0 += 32) {
        int l[K];
        unsigned m = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int j = c0 + k * G + gl;
            l[k] = on && j < qlen ? a - tab[min(acc.t(j), 4) << 3 | min(acc.q(j), 4)] : 0;
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const unsigned v = __ballot_sync(BSB_FULL_MASK, l[k] != 0);
            m |= G == 32 ? v : ((v >> g0) & ((1u << (G & 31)) - 1)) << (k * G & 31);
        }
        while (__any_sync(BSB_FULL_MASK, m != 0)) {          // the columns that lose, in order
            const int b = m ? __ffs(m) - 1 : 0;
            int x = l[0];
#pragma unroll
            for (int k = 1; k < K; ++k) x = b / G == k ? l[k] : x;
            x = __shfl_sync(BSB_FULL_MASK, x, b & (G - 1), G);
            if (m) {
                const int v = h0 + a * (c0 + b) - loss;      // the diagonal just before this column
                if (v > best) best = v, best_j = c0 + b - 1;
                loss += x;
                on = loss < lim;
                m = on ? m & (m - 1) : 0;
            }
        }
    }
    last = h0 + a * qlen - loss;
    if (last > best) best = last, best_j = qlen - 1;
    return on;
}

// ksw_diagonal for jobs of a byte buffer, 8 lanes a job: a lane takes 4 columns side by side as one word of each
// sequence (two aligned loads, both inside the buffer, else bytes), and where the words agree on bases 0..3 that
// score `a` on themselves (plain) nothing is lost and nothing looked up.  Losses are never negative, so the job is on
// while the total is below lim, and the diagonal's best prefix is the largest of its values just before the
// columns that lose and at its end, the first of equals.  loss: the whole diagonal's (where the job is on); lowest: the
// smallest of h0 and the diagonal's values just behind the columns that lose.
__device__ __forceinline__ uint32_t word_at(const uint8_t *p)
{
    const uint32_t *const w = (const uint32_t *)((uintptr_t)p & ~(uintptr_t)3);
    return __funnelshift_r(w[0], w[1], 8 * (unsigned)((uintptr_t)p & 3));
}
__device__ __forceinline__ bool ksw_diagonal_words(const int8_t *tab, int a, bool plain, int lim, int qlen, int tlen,
                                                   int h0, const uint8_t *q, const uint8_t *t, const uint8_t *buf,
                                                   const uint8_t *buf_end, int lane, int &best, int &best_j, int &last,
                                                   int &loss, int &lowest)
{
    const int gl = lane & 7;
    bool on = lim > 0 && qlen >= 1 && tlen >= qlen;
    int low = h0, key = 0;                       // key: the best prefix above h0 so far, << 11, and 2047 less its length
    loss = 0;
    for (int c0 = 0; __any_sync(BSB_FULL_MASK, on && c0 < qlen); c0 += 32) {
        const int j = c0 + 4 * gl;
        int l[4] = {0, 0, 0, 0};
        if (on && j < qlen) {
            uint32_t x = 0, y = 0;
            const int n = min(qlen - j, 4);
            if (((max((uintptr_t)q, (uintptr_t)t) + j) | 3) + 4 < (uintptr_t)buf_end &&
                ((min((uintptr_t)q, (uintptr_t)t) + j) & ~(uintptr_t)3) >= (uintptr_t)buf) {
                x = word_at(q + j), y = word_at(t + j);
            } else {
                for (int k = 0; k < n; ++k) x |= (uint32_t)q[j + k] << 8 * k, y |= (uint32_t)t[j + k] << 8 * k;
            }
            const uint32_t in = n == 4 ? 0xffffffffu : (1u << 8 * n) - 1u;
            if (!plain || (((x ^ y) | (x & 0xfcfcfcfcu)) & in)) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (k < n) l[k] = a - tab[min(y >> 8 * k & 255u, 4u) << 3 | min(x >> 8 * k & 255u, 4u)];
            }
        }
        const int sum = l[0] + l[1] + l[2] + l[3];
        if (!__any_sync(BSB_FULL_MASK, sum != 0)) continue;
        int incl = sum;
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) {
            const int v = __shfl_up_sync(BSB_FULL_MASK, incl, d, 8);
            if (gl >= d) incl += v;
        }
        int before = loss + incl - sum;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int v = a * (j + k) - before;
            if (l[k] && v > 0) key = max(key, v << 11 | (2047 - (j + k)));
            before += l[k];
            if (l[k]) low = min(low, h0 + a * (j + k + 1) - before);
        }
        loss += __shfl_sync(BSB_FULL_MASK, incl, 7, 8);
        on = on && loss < lim;
    }
    {
        const int v = a * qlen - loss;
        if (v > 0) key = max(key, v << 11 | (2047 - qlen));
    }
#pragma unroll
    for (int d = 4; d > 0; d >>= 1) {
        key = max(key, __shfl_xor_sync(BSB_FULL_MASK, key, d, 8));
        low = min(low, __shfl_xor_sync(BSB_FULL_MASK, low, d, 8));
    }
    lowest = low;
    best = h0 + (key >> 11), best_j = key ? 2047 - (key & 2047) - 1 : -1;
    last = h0 + a * qlen - loss;
    return on;
}

// How far a job's band can be cut without changing its result.  Notation and bound of ksw_diagonal: with L the whole
// diagonal's loss and D such that o + e(D+1) > L for both gaps, a path that leaves the 2D + 1 diagonals around the main
// one is worth less than the main diagonal in the same row or column from there on.  So it is never a row's maximum
// (nor ties with it), and never the last column's best, up to row qlen-1; behind it nothing but those diagonals can
// reach D(qlen-1) in the last column, and they end by row qlen-1+D.  A cell of those diagonals whose value comes
// from such a path is itself below the main diagonal, and so are the cells it leads to.  What is left is that the
// reference computes all 2D + 1 diagonals in every row, whatever its band w >= D (the band follows the non-zero cells: so
// the main diagonal has to exceed o + eD everywhere, which keeps the gaps from it non-zero that far), and that no
// row up to qlen-1+D ends the job: it is non-zero by the same condition, and its drop is at most L + o_del + e_del D.
// Then every band from D on gives the same six results.  Returns D, or -1 where the conditions do not hold.
__device__ __forceinline__ int cut_band(const KswParams &P, int loss, int lowest)
{
    const int D = max(0, max((loss - P.o_del) / P.e_del, (loss - P.o_ins) / P.e_ins));
    if (lowest <= max(P.o_del + P.e_del * D, P.o_ins + P.e_ins * D)) return -1;
    if (P.zdrop > 0 && loss + P.o_del + P.e_del * D > P.zdrop) return -1;
    return D;
}

// Rows that can no longer change a result.  After row i every cell of a later row is reached from
// H(i, j-1) or E(i+1, j) of some column j (stale cells beyond the band included: the band can grow
// back over them), gaining at most a = max(mat) per remaining column, and from nothing where both
// are 0.  So with U the largest max(H, E) + a(qlen - j) over the non-zero columns, U < gscore means
// that no later row can raise gscore, tie with it (a tie moves gtle) or raise the score, which is
// at least gscore: the six results are final and only the cell count would go on.  The test costs
// a pass over the columns, so a row runs it only when its own maximum m at mj does not already
// show a larger U.  Of a job that aligns to its end this leaves out the target's flank: 100 of
// about 175 rows of the batched jobs.
__device__ __forceinline__ bool rows_may_be_done(int gscore, int m, int mj, int qlen, int a)
{
    return gscore > 0 && (mj == qlen - 1 || m + a * (qlen - 1 - mj) < gscore);
}

// Extends one job with the calling warp (every lane returns the same tuple).
// All control values are warp-uniform.  Acc supplies query base j and target
// base i (q(j), t(i)), so jobs can read a byte buffer or the 2-bit reference.
//
// Register state per lane, columns j = lane*C + s:
//   Hs[s] = eh[j].h = H(i-1, j-1),  Es[s] = eh[j].e = E(i, j)   (ksw.c:376-378)
// Invariant: every column left of the band (j < beg) holds H = E = 0.  The
// reference never reads those cells again (beg only grows), and with them at
// zero the F scan and the row maximum need no left-edge masks: a dead column
// has M = 0, T = 0, V = e_ins*(j+1), F = 0 and H = 0.  The shrink step only
// moves beg over cells that are already zero; when the band edge i-w moves
// beg instead, the cells it passes are zeroed explicitly.
template <int C, class Acc>
__device__ __forceinline__ KswResult ksw_warp(const KswParams &P, int qlen, int tlen, int h0, int w_in,
                                              int end_bonus, const Acc &acc, int lane, bool count_cells)
{
    const int o_del = P.o_del, e_del = P.e_del, o_ins = P.o_ins, e_ins = P.e_ins;
    const int oe_del = o_del + e_del, oe_ins = o_ins + e_ins;
    const int base = lane * C;

    // query profile: byte c of prof[s] = mat[c*5 + q[j]] for target bases 0..3;
    // the N row (target base 4) is kept apart in profN, four slots per word.
    uint32_t prof[C];
    uint32_t profN[(C + 3) / 4];
    int Hs[C], Es[C];
#pragma unroll
    for (int s = 0; s < (C + 3) / 4; ++s) profN[s] = 0;
    const int h1run = max(h0 - oe_ins, 0);
#pragma unroll
    for (int s = 0; s < C; ++s) {
        const int j = base + s;
        const int qc = j < qlen ? acc.q(j) : 0;
        prof[s] = profile_word(P, qc);
        profN[s >> 2] |= (uint32_t)(uint8_t)profile_n(P, qc) << ((s & 3) * 8);
        // first row: h0, then an insertion run clipped at zero (ksw.c:395-397)
        Hs[s] = j == 0 ? h0 : (j <= qlen ? max(h1run - e_ins * (j - 1), 0) : 0);
        Es[s] = 0;
    }

    // band clamp (ksw.c:399-407)
    int w = w_in;
    {
        int max_ins = band_cap(qlen * P.mat_max + end_bonus - o_ins, e_ins);
        max_ins = max_ins > 1 ? max_ins : 1;
        w = w < max_ins ? w : max_ins;
        int max_del = band_cap(qlen * P.mat_max + end_bonus - o_del, e_del);
        max_del = max_del > 1 ? max_del : 1;
        w = w < max_del ? w : max_del;
    }

    int best = h0, best_i = -1, best_j = -1, max_ie = -1, gscore = -1, max_off = 0;
    int beg = 0, end = qlen;
    long long ncell = 0;
    const int q_lane = qlen / C, q_slot = qlen % C;   // owner of column qlen

    // target bases arrive 32 rows at a time, one byte per lane, next chunk prefetched
    uint32_t tch = lane < tlen ? (uint32_t)acc.t(lane) : 4u;
    uint32_t tnext = 32 + lane < tlen ? (uint32_t)acc.t(32 + lane) : 4u;

    for (int i = 0; i < tlen; ++i) {
        const int tc = (int)__shfl_sync(BSB_FULL_MASK, tch, i & 31);
        if ((i & 31) == 31) {
            tch = tnext;
            const int ti = i + 33 + lane;
            tnext = ti < tlen ? (uint32_t)acc.t(ti) : 4u;
        }
        // band of this row (ksw.c:416-419)
        if (beg < i - w) {
            beg = i - w;
#pragma unroll
            for (int s = 0; s < C; ++s)
                if (base + s < beg) Hs[s] = 0, Es[s] = 0;
        }
        if (end > i + w + 1) end = i + w + 1;
        if (end > qlen) end = qlen;
        // H(i,-1) (ksw.c:421-424)
        const int h1_init = beg == 0 ? max(h0 - (o_del + e_del * (i + 1)), 0) : 0;

        if (beg >= end) {
            // empty band: the reference's loop does not run, eh[end] gets {h1,0},
            // the query-end test sees j == beg, and the zero row max stops it.
            if (beg == qlen) {
                max_ie = gscore > h1_init ? max_ie : i;
                gscore = gscore > h1_init ? gscore : h1_init;
            }
            break;
        }

        // ---- pass 1: M, next-row E, and the F-scan operand V = T(j) + e_ins*(j+1)
        int Mv[C], En[C], Pf[C];
        int run = 0;
        if (tc < 4) {
            const uint32_t sel = sext_selector(tc);
#pragma unroll
            for (int s = 0; s < C; ++s) {
                const int j = base + s;
                const int sc = prmt_sext(prof[s], sel);
                const int Hp = Hs[s];
                const int M = Hp ? Hp + sc : 0;
                const int Ti = __viaddmax_s32(M, -oe_ins, 0);
                En[s] = __viaddmax_s32(Es[s], -e_del, __viaddmax_s32(M, -oe_del, 0));
                run = max(run, Ti + e_ins * (j + 1));
                Pf[s] = run;
                Mv[s] = M;
            }
        } else {
#pragma unroll
            for (int s = 0; s < C; ++s) {
                const int j = base + s;
                const int sc = prmt_sext(profN[s >> 2], sext_selector(s & 3));
                const int Hp = Hs[s];
                const int M = Hp ? Hp + sc : 0;
                const int Ti = __viaddmax_s32(M, -oe_ins, 0);
                En[s] = __viaddmax_s32(Es[s], -e_del, __viaddmax_s32(M, -oe_del, 0));
                run = max(run, Ti + e_ins * (j + 1));
                Pf[s] = run;
                Mv[s] = M;
            }
        }

        // ---- warp exclusive prefix max of the lane totals (lane 0 starts from 0 = F at column 0)
        int incl = run;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) incl = max(incl, __shfl_up_sync(BSB_FULL_MASK, incl, d));
        const int excl = __shfl_up_sync(BSB_FULL_MASK, incl, 1);
        const int carry = lane == 0 ? 0 : excl;

        // ---- pass 2: H, the row-max key (H << 10 | j), and the new eh[] (H shifted one column)
        int kmax = -1, prevH = 0;
        uint32_t nzb = 0;
#pragma unroll
        for (int s = 0; s < C; ++s) {
            const int j = base + s;
            const int G = s == 0 ? carry : max(carry, Pf[s - 1]);
            const int F = G - e_ins * j;
            const int H = __vimax3_s32(Mv[s], Es[s], F);
            const bool lt = j < end;
            if (lt) kmax = max(kmax, H * 1024 + j);     // ties keep the later column (ksw.c:437)
            const int nE = lt ? En[s] : 0;     // E beyond end is 0 at every row (ksw_group16.cuh, pass 2)
            Es[s] = nE;
            if (s > 0) {
                const int nH = j <= end ? prevH : Hs[s];
                Hs[s] = nH;
                if (j <= end && (nH | nE) != 0) nzb |= 1u << s;
            }
            prevH = H;
        }
        {
            int Hleft = __shfl_up_sync(BSB_FULL_MASK, prevH, 1);
            if (lane == 0) Hleft = h1_init;
            const int nH = base <= end ? Hleft : Hs[0];
            Hs[0] = nH;
            if (base <= end && (nH | Es[0]) != 0) nzb |= 1u;
        }

        ncell += end - beg;
        const int kw = __reduce_max_sync(BSB_FULL_MASK, kmax);
        const int m = kw >> 10, mj = kw & 1023;

        if (end == qlen) {          // reached the query end: eh[qlen].h == H(i,qlen-1) (ksw.c:450-453)
            int hsel = 0;
#pragma unroll
            for (int s = 0; s < C; ++s) hsel = s == q_slot ? Hs[s] : hsel;
            const int h1 = __shfl_sync(BSB_FULL_MASK, hsel, q_lane);
            max_ie = gscore > h1 ? max_ie : i;
            gscore = gscore > h1 ? gscore : h1;
        }
        if (m == 0) break;                             // ksw.c:454
        if (m > best) {
            best = m, best_i = i, best_j = mj;
            const int d = mj > i ? mj - i : i - mj;
            max_off = max_off > d ? max_off : d;
        } else if (P.zdrop > 0) {                      // ksw.c:458-464
            const int di = i - best_i, dj = mj - best_j;
            if (di > dj) {
                if (best - m - (di - dj) * e_del > P.zdrop) break;
            } else {
                if (best - m - (dj - di) * e_ins > P.zdrop) break;
            }
        }
        if (!count_cells && rows_may_be_done(gscore, m, mj, qlen, P.mat_max)) {
            int U = 0;
#pragma unroll
            for (int s = 0; s < C; ++s) {
                const int X = max(Hs[s], Es[s]);
                if (X > 0) U = max(U, X + P.mat_max * (qlen - base - s));
            }
            if (__reduce_max_sync(BSB_FULL_MASK, U) < gscore) break;
        }
        // shrink to the non-zero cells (ksw.c:466-469); columns left of beg are zero
        const int lfirst = nzb ? base + __ffs(nzb) - 1 : INT_MAX;
        const int llast = nzb ? base + 31 - __clz(nzb) : -1;
        const int fnz = __reduce_min_sync(BSB_FULL_MASK, lfirst);
        const int lnz = __reduce_max_sync(BSB_FULL_MASK, llast);
        if (fnz < end) {
            beg = fnz;
            end = lnz + 2 < qlen ? lnz + 2 : qlen;
        } else {
            const int jj = lnz == end ? end : end - 1;
            beg = end;
            end = jj + 2 < qlen ? jj + 2 : qlen;
        }
    }
    KswResult r;
    r.score = best; r.qle = best_j + 1; r.tle = best_i + 1;
    r.gtle = max_ie + 1; r.gscore = gscore; r.max_off = max_off;
    r.cells = ncell;
    return r;
}

