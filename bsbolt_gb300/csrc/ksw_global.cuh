// ksw_global.cuh -- the DP of ksw_global2 (bsbolt/External/BWA/ksw.c:504-582) on one warp,
// shared by bwa_gen_cigar2 (cigar.cu) and mem_patch_reg's score-only call (chain.cu).
#pragma once

#include <cstdint>

#include "bsb_internal.cuh"

constexpr int kNegInf = -0x40000000;        // MINUS_INF, ksw.c:490

struct GlobalPen {
    int o_del, e_del, o_ins, e_ins;
};

// The DP rows of ksw_global2 (ksw.c:519-582) on staged sequences (qs, ts after the strand
// flip), one warp: row i is processed 32 columns at a time, one column per lane.  At the
// start of cell j the reference holds eh[j] = {H(i-1, j-1), E(i, j)} and f = F(i, j); F
// depends only on the row's M values (F(i, j+1) = max(M(i, j) - oe_ins, F(i, j) - e_ins),
// F(i, beg) = -inf), so the lanes get it from a max-plus prefix scan -- max commutes with
// subtracting a constant, so the values are the reference's exactly -- and everything
// else in a cell is local.  H / E: qlen + 1 entries each (the reference's eh); Z: tlen
// rows of `stride` direction bytes, or NULL for the score alone (ksw_global2 without a
// CIGAR); ts[i]: target base i.  Returns the score on every lane.
template <class TS>
__device__ __forceinline__ int global_rows_warp(const GlobalPen &P, const int8_t *smat, const uint8_t *qs, int qlen,
                                                const TS &ts, int tlen, int w, int stride, int32_t *H, int32_t *E,
                                                uint8_t *Z, int lane)
{
    const int oe_del = P.o_del + P.e_del, oe_ins = P.o_ins + P.e_ins, e_ins = P.e_ins;
    for (int j = lane; j <= qlen; j += 32) {
        H[j] = j == 0 ? 0 : j <= w ? -(P.o_ins + e_ins * j) : kNegInf;
        E[j] = kNegInf;
    }
    __syncwarp();
    for (int i = 0; i < tlen; ++i) {
        const int8_t *srow = smat + ts[i] * 5;
        const int beg = i > w ? i - w : 0, end = i + w + 1 < qlen ? i + w + 1 : qlen;
        int32_t f_carry = kNegInf;                                        // F(i, j0)
        int32_t h_carry = beg == 0 ? -(P.o_del + P.e_del * (i + 1)) : kNegInf;   // H(i, j0 - 1)
        uint8_t *zrow = Z ? Z + (size_t)i * stride : nullptr;
        if (beg >= end && lane == 0) H[end] = h_carry, E[end] = kNegInf;     // an empty row (not reached: w > |tlen - qlen|)
        for (int j0 = beg; j0 < end; j0 += 32) {
            const int j = j0 + lane;
            const bool on = j < end;
            int32_t m = kNegInf, e = kNegInf;
            if (on) m = H[j] + srow[qs[j]], e = E[j];
            // out_L = F(i, j0+L+1) = max(m_L - oe_ins, out_{L-1} - e_ins), out_{-1} = f_carry;
            // with b_L = m_L - oe_ins + L*e_ins it is an inclusive max-scan shifted back
            int32_t sc = on ? m - oe_ins + lane * e_ins : INT32_MIN / 2;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int32_t v = __shfl_up_sync(BSB_FULL_MASK, sc, d);
                if (lane >= d) sc = sc > v ? sc : v;
            }
            const int32_t c0 = f_carry - e_ins;                          // out_{-1}, normalised at L = -1
            const int32_t out = (sc > c0 ? sc : c0) - lane * e_ins;      // F(i, j + 1)
            int32_t f = __shfl_up_sync(BSB_FULL_MASK, out, 1);          // F(i, j)
            if (lane == 0) f = f_carry;
            int32_t h, t;
            uint32_t dir;
            if (m >= e) h = m, dir = 0;
            else h = e, dir = 1;
            if (h < f) h = f, dir = 2;
            t = m - oe_del;
            e -= P.e_del;
            if (e > t) dir |= 1 << 2;
            else e = t;
            t = m - oe_ins;
            if (f - e_ins > t) dir |= 2 << 4;
            int32_t hprev = __shfl_up_sync(BSB_FULL_MASK, h, 1);        // H(i, j - 1)
            if (lane == 0) hprev = h_carry;
            if (on) {
                H[j] = hprev;
                E[j] = e;
                if (zrow) zrow[j - beg] = (uint8_t)dir;
                if (j == end - 1) H[end] = h, E[end] = kNegInf;
            }
            f_carry = __shfl_sync(BSB_FULL_MASK, out, 31);
            h_carry = __shfl_sync(BSB_FULL_MASK, h, 31);
        }
        __syncwarp();
    }
    return H[qlen];
}

// The same cells with the band's diagonals over the lanes, C neighbours to a lane: cell (i, d), j = i + d - w,
// takes H from its own diagonal's row before, E from diagonal d + 1's row before and F from diagonal d - 1's
// same row.  Lane k does row s - k in step s: F comes from the lane below's step before, E of a lane's last
// diagonal from the lane above's first in the same step, so a step is one exchange each way and C cells whose
// only chain is F's, and a job takes tlen + band / C steps.  H, E and F stay in registers (a diagonal's first
// H is the border's value; a cell outside leaves E and F at -inf), and scores are fetched a step ahead.
// Needs 2w + 1 < 32 C, Z and stride multiples of 4.  The lanes' rows differ, so every byte of directions is a sector of
// its own to write: of four a lane makes one word where they lie side by side (5000 alignments of 250 bases in bands of
// 61, the call: 1.42 ms by bytes, 0.82 by words; in rows 1.17).  Two to a lane stay bytes: most such bands hold theirs
// in shared memory, and the words' branch costs more (40000 alignments of 100 bases: 120 us by bytes, 129 by words).
template <int C, class TS>
__device__ __forceinline__ int global_diagonals_warp(const GlobalPen &P, const int8_t *smat, const uint8_t *qs,
                                                     int qlen, const TS &ts, int tlen, int w, int stride, uint8_t *Z,
                                                     int lane)
{
    const int oe_del = P.o_del + P.e_del, oe_ins = P.o_ins + P.e_ins, e_ins = P.e_ins;
    const int d0 = lane * C, last = 2 * w;
    int32_t h[C], e[C], f_out = kNegInf;
    int sc[C], q[C];                              // this step's scores; the next step's query bases
    int i = -lane, t = 0;                         // this step's row; the next row's base
    const auto base_q = [&](int j) { return (unsigned)j < (unsigned)qlen ? (int)qs[j] : 0; };
    const auto base_t = [&](int r) { return (unsigned)r < (unsigned)tlen ? (int)ts[r] : 0; };
    t = base_t(i);
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const int j = d0 + c - w;
        h[c] = j > 0 ? -(P.o_ins + e_ins * j) : j < 0 ? -(P.o_del - P.e_del * j) : 0;
        e[c] = kNegInf;
        sc[c] = smat[t * 5 + base_q(i + j)];
        q[c] = base_q(i + j + 1);
    }
    t = base_t(i + 1);
    const int steps = tlen + last / C;
    for (int s = 0; s < steps; ++s, ++i) {
        int next[C];
#pragma unroll
        for (int c = 0; c < C; ++c) next[c] = smat[t * 5 + q[c]];
        const int j0 = i + d0 - w;
        t = base_t(i + 2);
#pragma unroll
        for (int c = 0; c < C - 1; ++c) q[c] = q[c + 1];
        q[C - 1] = base_q(j0 + C + 1);
        int32_t f = __shfl_up_sync(BSB_FULL_MASK, f_out, 1);
        if (lane == 0) f = kNegInf;
        const bool row = (unsigned)i < (unsigned)tlen;
        const int z_at = i * stride + (i >= w ? d0 : j0);
        uint32_t dirs = 0;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int32_t e_in = c == C - 1 ? __shfl_down_sync(BSB_FULL_MASK, e[0], 1) : e[c + 1];
            const bool on = row && (unsigned)(j0 + c) < (unsigned)qlen && d0 + c <= last;
            const int32_t m = h[c] + sc[c];
            int32_t best = m;
            uint32_t dir = 0;
            if (m < e_in) best = e_in, dir = 1;
            if (best < f) best = f, dir = 2;
            const int32_t td = m - oe_del, ed = e_in - P.e_del;
            if (ed > td) dir |= 1 << 2;
            const int32_t ti = m - oe_ins, fi = f - e_ins;
            if (fi > ti) dir |= 2 << 4;
            e[c] = on ? (ed > td ? ed : td) : kNegInf;
            f = on ? (fi > ti ? fi : ti) : kNegInf;
            if (on) {
                h[c] = best;
                if (C == 2 && Z) Z[z_at + c] = (uint8_t)dir;
            }
            dirs |= dir << 8 * c;
            sc[c] = next[c];
        }
        if (C == 4 && Z && row) {
            if (i >= w && j0 >= 0 && j0 + C <= qlen && d0 + C - 1 <= last) {
                *(uint32_t *)(Z + z_at) = dirs;
            } else {
#pragma unroll
                for (int c = 0; c < C; ++c)
                    if ((unsigned)(j0 + c) < (unsigned)qlen && d0 + c <= last) Z[z_at + c] = (uint8_t)(dirs >> 8 * c);
            }
        }
        f_out = f;
    }
    __syncwarp();
    const int d = qlen - tlen + w;                // the last cell's diagonal
    int32_t score = h[0];
#pragma unroll
    for (int c = 1; c < C; ++c)
        if (d % C == c) score = h[c];
    return __shfl_sync(BSB_FULL_MASK, score, d / C);
}

// Which form: the diagonals' wherever they fit four to a lane, two to a lane where that suffices (half the cells
// a step).  A row at a time costs a five-step scan and four exchanges per 32 columns one after the other, some
// 2000 clocks a row for a band of 65 columns against 150 here: bwa_gen_cigar2's kernel on 40k reads of 100 bases
// 204 us -> 124, and a merge's 150-row alignment in mem_patch_reg 180 us -> 15.  Rows are left for wider bands.
template <class TS>
__device__ __forceinline__ int global_warp(const GlobalPen &P, const int8_t *smat, const uint8_t *qs, int qlen,
                                           const TS &ts, int tlen, int w, int stride, int32_t *H, int32_t *E,
                                           uint8_t *Z, int lane)
{
    const int diagonals = 2 * w + 1;
    if (diagonals < 64) return global_diagonals_warp<2>(P, smat, qs, qlen, ts, tlen, w, stride, Z, lane);
    if (diagonals < 128) return global_diagonals_warp<4>(P, smat, qs, qlen, ts, tlen, w, stride, Z, lane);
    return global_rows_warp(P, smat, qs, qlen, ts, tlen, w, stride, H, E, Z, lane);
}
