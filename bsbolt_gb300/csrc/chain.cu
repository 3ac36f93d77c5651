// chain.cu -- seeds -> chains -> filtered chains -> alignment regions, on sm_103a.
//
// The pre-dedup part of mem_align1_core (bsbolt/External/BWA/bwamem.c:1157-1180)
// after seeding:
//   rows_count / rows_fill  the SA rows mem_chain samples per seed interval
//                           (bwamem.c:280-283), then sa_kernel (seed.cu) maps them
//                           to reference positions;
//   chain_warp_kernel       one warp per read: mem_chain, mem_chain_weight and
//                           mem_chain_flt with ks_introsort's exact order;
//   chain_kernel            the same by one thread, with the reference's B-tree of
//                           chains (kbtree.h, t = 5), for reads where two chains start
//                           at the same place and the tree's nodes decide;
//   chain2aln_plain         one warp per read: mem_chain2aln (bwamem.c:636-790) for the reads whose
//                           extensions were all run as batches before
//   chain2aln_kernel        one warp per read: mem_chain2aln (bwamem.c:636-790),
//                           each ksw_extend2 run by the warp (ksw_core.cuh) on the
//                           read and the device 2-bit reference directly, so no
//                           reversed copies or target windows are materialised.

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <vector>

#include "bsb_internal.cuh"
#include "ksw_global.cuh"
#include "fm_index.cuh"
#include "ksw_core.cuh"
#include "scan.cuh"

size_t seed_padded_entries(int64_t total_bases, int n_reads, int mult);   // seed.cu

namespace {

constexpr int kBT = 5;                  // kbtree order for 40-byte keys in 512-byte nodes
constexpr int kBTMax = 2 * kBT - 1;

struct BtNode {
    int n, internal;
    int key[kBTMax];
    int child[kBTMax + 1];
};

struct ChainRec {                       // a chain while it is being built
    int64_t pos;                        // first seed's rbeg (the tree key)
    int64_t first_rbeg, last_rbeg;
    int first_qbeg, last_qbeg, last_len;
    int n, rid;
};

struct DevSeed {                        // mem_seed_t (bwamem.c:171-174)
    int64_t rbeg;
    int32_t qbeg, len, score, pad;
};

struct DevChain {                       // a kept chain, in mem_chain_flt's order
    int32_t n, rid, w, kept;
    int32_t seed_off, first;
    float frac_rep;
    int32_t pad;
};

struct AlnOpt {
    int a, o_del, e_del, o_ins, e_ins, w, zdrop, pen_clip5, pen_clip3;
    int min_seed_len, max_occ, max_chain_gap, min_chain_weight, max_chain_extend;
    float mask_level, drop_ratio;
};

struct DevBns {
    const int64_t *ann_offset;
    const int32_t *ann_len;
    int n_seqs;
    int64_t l_pac;
    const uint8_t *pac;
};

// ---------------------------------------------------------------- bns lookups

__device__ int pos2rid(const DevBns &B, int64_t pos_f)              // bntseq.c:364-379
{
    int left = 0, mid = 0, right = B.n_seqs;
    if (pos_f >= B.l_pac) return -1;
    while (left < right) {
        mid = (left + right) >> 1;
        if (pos_f >= B.ann_offset[mid]) {
            if (mid == B.n_seqs - 1) break;
            if (pos_f < B.ann_offset[mid + 1]) break;
            left = mid + 1;
        } else right = mid;
    }
    return mid;
}

__device__ __forceinline__ int64_t depos(const DevBns &B, int64_t pos, int &is_rev)
{
    is_rev = pos >= B.l_pac;
    return is_rev ? (B.l_pac << 1) - 1 - pos : pos;
}

__device__ int intv2rid(const DevBns &B, int64_t rb, int64_t re)    // bntseq.c:381-389
{
    int is_rev;
    if (rb < B.l_pac && re > B.l_pac) return -2;
    const int rid_b = pos2rid(B, depos(B, rb, is_rev));
    const int rid_e = rb < re ? pos2rid(B, depos(B, re - 1, is_rev)) : rid_b;
    return rid_b == rid_e ? rid_b : -1;
}

// base at position p of the forward-reverse text (bns_get_seq, bntseq.c:414-434)
__device__ __forceinline__ int text_base(const DevBns &B, int64_t p)
{
    if (p < B.l_pac) return __ldg(B.pac + (p >> 2)) >> ((~p & 3) << 1) & 3;
    p = (B.l_pac << 1) - 1 - p;
    return 3 - (__ldg(B.pac + (p >> 2)) >> ((~p & 3) << 1) & 3);
}

// ---------------------------------------------------------------- SA rows

__device__ __forceinline__ int rows_of(uint64_t x2, int max_occ, uint64_t &step)
{
    step = x2 > (uint64_t)max_occ ? x2 / (uint64_t)max_occ : 1;
    const uint64_t n = (x2 + step - 1) / step;                       // k = 0, step, ... < x2
    return (int)(n < (uint64_t)max_occ ? n : (uint64_t)max_occ);
}

__global__ void rows_count(const DevIntv *__restrict__ seeds, int64_t n, int max_occ, int *__restrict__ cnt)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint64_t step;
        cnt[i] = rows_of(seeds[i].x2, max_occ, step);
    }
}

__global__ void rows_fill(const DevIntv *__restrict__ seeds, int64_t n, int max_occ, const int64_t *__restrict__ roff,
                          uint64_t *__restrict__ rows)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint64_t step;
        const int m = rows_of(seeds[i].x2, max_occ, step);
        uint64_t *dst = rows + roff[i];
        for (int c = 0; c < m; ++c) dst[c] = seeds[i].x0 + (uint64_t)c * step;
    }
}

// ---------------------------------------------------------------- chaining

struct Bt {
    BtNode *nodes;
    int n_nodes, root;
    const ChainRec *ch;
    __device__ int64_t key(int c) const { return ch[c].pos; }
    __device__ int fresh()
    {
        BtNode &x = nodes[n_nodes];
        x.n = 0;
        x.internal = 0;
        return n_nodes++;
    }
    // lower bound stepped back unless equal (kbtree.h:116-130); r = 0 when equal
    __device__ int find(const BtNode &x, int64_t k, int &r) const
    {
        int begin = 0, end = x.n;
        if (x.n == 0) return -1;
        while (begin < end) {
            const int mid = (begin + end) >> 1;
            if (key(x.key[mid]) < k) begin = mid + 1;
            else end = mid;
        }
        if (begin == x.n) { r = 1; return x.n - 1; }
        const int64_t kb = key(x.key[begin]);
        r = k < kb ? -1 : (k > kb ? 1 : 0);
        if (r < 0) --begin;
        return begin;
    }
    __device__ int lower(int64_t k) const                             // kb_intervalp
    {
        int lo = -1, xi = root;
        for (;;) {
            const BtNode &x = nodes[xi];
            int r = 0;
            const int i = find(x, k, r);
            if (i >= 0 && r == 0) return x.key[i];
            if (i >= 0) lo = x.key[i];
            if (!x.internal) return lo;
            xi = x.child[i + 1];
        }
    }
    __device__ void split(int xi, int i, int yi)                      // kbtree.h:173-190
    {
        const int zi = fresh();
        BtNode &x = nodes[xi], &y = nodes[yi], &z = nodes[zi];
        z.internal = y.internal;
        z.n = kBT - 1;
        for (int j = 0; j < kBT - 1; ++j) z.key[j] = y.key[kBT + j];
        if (y.internal)
            for (int j = 0; j < kBT; ++j) z.child[j] = y.child[kBT + j];
        y.n = kBT - 1;
        for (int j = x.n; j >= i + 1; --j) x.child[j + 1] = x.child[j];
        x.child[i + 1] = zi;
        for (int j = x.n - 1; j >= i; --j) x.key[j + 1] = x.key[j];
        x.key[i] = y.key[kBT - 1];
        ++x.n;
    }
    __device__ void insert(int c)                                     // kbtree.h:191-223
    {
        const int64_t k = key(c);
        if (nodes[root].n == kBTMax) {
            const int si = fresh();
            nodes[si].internal = 1;
            nodes[si].child[0] = root;
            root = si;
            split(si, 0, nodes[si].child[0]);
        }
        int xi = root;
        for (;;) {
            BtNode &x = nodes[xi];
            int r;
            if (!x.internal) {
                const int i = find(x, k, r);
                for (int j = x.n - 1; j > i; --j) x.key[j + 1] = x.key[j];
                x.key[i + 1] = c;
                ++x.n;
                return;
            }
            int i = find(x, k, r) + 1;
            if (nodes[x.child[i]].n == kBTMax) {
                split(xi, i, x.child[i]);
                if (k > key(nodes[xi].key[i])) ++i;
            }
            xi = nodes[xi].child[i];
        }
    }
};

// ks_introsort (ksort.h:146-226) over an index array with the comparison lt(x, y):
// restated step for step, since records that compare equal keep the order it leaves.
template <class Lt>
struct KsSort {
    int *a;
    Lt lt;
    __device__ void insertsort(int s, int t)
    {
        for (int i = s + 1; i < t; ++i)
            for (int j = i; j > s && lt(a[j], a[j - 1]); --j) { int tmp = a[j]; a[j] = a[j - 1]; a[j - 1] = tmp; }
    }
    __device__ void combsort(int s, size_t n)
    {
        const double shrink_factor = 1.2473309501039786540366528676643;
        int do_swap;
        size_t gap = n;
        do {
            if (gap > 2) {
                gap = (size_t)(gap / shrink_factor);
                if (gap == 9 || gap == 10) gap = 11;
            }
            do_swap = 0;
            for (size_t i = 0; i + gap < n; ++i) {
                const int ii = s + (int)i, jj = ii + (int)gap;
                if (lt(a[jj], a[ii])) { int tmp = a[ii]; a[ii] = a[jj]; a[jj] = tmp; do_swap = 1; }
            }
        } while (do_swap || gap > 2);
        if (gap != 1) insertsort(s, s + (int)n);
    }
    __device__ void sort(int n, int *stk_l, int *stk_r, int *stk_d)
    {
        if (n < 1) return;
        if (n == 2) {
            if (lt(a[1], a[0])) { int tmp = a[0]; a[0] = a[1]; a[1] = tmp; }
            return;
        }
        int d;
        for (d = 2; 1ul << d < (unsigned long)n; ++d) ;
        int top = 0, s = 0, t = n - 1;
        d <<= 1;
        for (;;) {
            if (s < t) {
                if (--d == 0) {
                    combsort(s, (size_t)(t - s + 1));
                    t = s;
                    continue;
                }
                int i = s, j = t, k = i + ((j - i) >> 1) + 1;
                if (lt(a[k], a[i])) {
                    if (lt(a[k], a[j])) k = j;
                } else k = lt(a[j], a[i]) ? i : j;
                const int rp = a[k];
                if (k != t) { int tmp = a[k]; a[k] = a[t]; a[t] = tmp; }
                for (;;) {
                    do ++i; while (lt(a[i], rp));
                    do --j; while (i <= j && lt(rp, a[j]));
                    if (j <= i) break;
                    int tmp = a[i]; a[i] = a[j]; a[j] = tmp;
                }
                { int tmp = a[i]; a[i] = a[t]; a[t] = tmp; }
                if (i - s > t - i) {
                    if (i - s > 16) { stk_l[top] = s; stk_r[top] = i - 1; stk_d[top] = d; ++top; }
                    s = t - i > 16 ? i + 1 : t;
                } else {
                    if (t - i > 16) { stk_l[top] = i + 1; stk_r[top] = t; stk_d[top] = d; ++top; }
                    t = i - s > 16 ? i - 1 : s;
                }
            } else {
                if (top == 0) {
                    insertsort(0, n);
                    return;
                }
                --top;
                s = stk_l[top]; t = stk_r[top]; d = stk_d[top];
            }
        }
    }
};

// mem_chain_flt's order: chain weight, descending (bwamem.c:328-329)
struct FltLt {
    const int *w;
    __device__ bool operator()(int x, int y) const { return w[x] > w[y]; }
};

// The reads that chain_warp_kernel leaves (two chains start at the same place, so their order
// follows the tree's nodes): one thread per read, with the tree itself.  Per-read scratch is carved
// from arrays sized by the read's SA-row count R (a read never has more chains, seeds or tree nodes
// than rows).  Outputs the kept chains in mem_chain_flt's order and their seeds (in insertion
// order) at the read's row offset.
__global__ void __launch_bounds__(128)
chain_kernel(AlnOpt opt, DevBns B, const int *__restrict__ list, const int *__restrict__ n_list,
             const int64_t *__restrict__ read_off, const DevIntv *__restrict__ seeds,
             const int64_t *__restrict__ seed_off, const int64_t *__restrict__ row_off_of_seed,
             const uint64_t *__restrict__ pos, ChainRec *__restrict__ chains, BtNode *__restrict__ nodes,
             int *__restrict__ row_chain, int *__restrict__ iwork, DevSeed *__restrict__ out_seeds,
             DevChain *__restrict__ out_chains, int *__restrict__ n_chains)
{
    // As few reads a warp as the list allows, one where there are no more reads than warps: the lanes' trees take different
    // paths, one after the other.  4096 reads of 100 bases, a quarter of them from tandem repeats (up to 2000 chains each),
    // the chaining stage: 1.02 s with 32 reads a warp, 0.38 with one.
    const int n = *n_list, warps = (int)(gridDim.x * blockDim.x) >> 5, per = min(32, (n + warps - 1) / warps);
    const int lane = threadIdx.x & 31;
    if (lane >= per) return;
    for (int t = ((int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per + lane; t < n; t += warps * per) {
        const int r = list[t];
        const int len = (int)(read_off[r + 1] - read_off[r]);
        const int64_t s0 = seed_off[r], s1 = seed_off[r + 1];
        const int64_t R0 = row_off_of_seed[s0], R = row_off_of_seed[s1] - R0;
        n_chains[r] = 0;
        if (len < opt.min_seed_len || R == 0) continue;
        ChainRec *ch = chains + R0;
        BtNode *nd = nodes + R0;
        int *rc = row_chain + R0;
        // frac_rep (bwamem.c:271-278)
        int b = 0, e = 0, l_rep = 0;
        for (int64_t i = s0; i < s1; ++i) {
            const int sb = (int)(seeds[i].info >> 32), se = (int)(uint32_t)seeds[i].info;
            if (seeds[i].x2 <= (uint64_t)opt.max_occ) continue;
            if (sb > e) l_rep += e - b, b = sb, e = se;
            else e = e > se ? e : se;
        }
        l_rep += e - b;
        const float frac_rep = (float)l_rep / len;
        // mem_chain (bwamem.c:279-305)
        Bt bt;
        bt.nodes = nd;
        bt.n_nodes = 0;
        bt.ch = ch;
        bt.root = bt.fresh();
        int n_chn = 0;
        for (int64_t i = s0; i < s1; ++i) {
            const DevIntv p = seeds[i];
            const int slen = (int)((uint32_t)p.info - (uint32_t)(p.info >> 32));
            const int qbeg = (int)(p.info >> 32);
            const int64_t rlo = row_off_of_seed[i] - R0, rhi = row_off_of_seed[i + 1] - R0;
            for (int64_t k = rlo; k < rhi; ++k) {
                const int64_t rbeg = (int64_t)pos[R0 + k];
                rc[k] = -1;
                const int rid = intv2rid(B, rbeg, rbeg + slen);
                if (rid < 0) continue;
                bool to_add = true;
                if (n_chn > 0) {
                    const int lo = bt.lower(rbeg);
                    if (lo >= 0) {                               // test_and_merge (bwamem.c:203-227)
                        ChainRec &c = ch[lo];
                        const int64_t qend = c.last_qbeg + c.last_len, rend = c.last_rbeg + c.last_len;
                        if (rid != c.rid) {
                        } else if (qbeg >= c.first_qbeg && qbeg + slen <= qend && rbeg >= c.first_rbeg &&
                                   rbeg + slen <= rend) {
                            to_add = false;                      // contained: the seed is dropped
                        } else if ((c.last_rbeg < B.l_pac || c.first_rbeg < B.l_pac) && rbeg >= B.l_pac) {
                        } else {
                            const int64_t x = qbeg - c.last_qbeg, y = rbeg - c.last_rbeg;
                            if (y >= 0 && x - y <= opt.w && y - x <= opt.w && x - c.last_len < opt.max_chain_gap &&
                                y - c.last_len < opt.max_chain_gap) {
                                c.last_qbeg = qbeg; c.last_rbeg = rbeg; c.last_len = slen;
                                ++c.n;
                                rc[k] = lo;
                                to_add = false;
                            }
                        }
                    }
                }
                if (to_add) {
                    ChainRec &c = ch[n_chn];
                    c.pos = rbeg; c.first_rbeg = c.last_rbeg = rbeg;
                    c.first_qbeg = c.last_qbeg = qbeg; c.last_len = slen;
                    c.n = 1; c.rid = rid;
                    rc[k] = n_chn;
                    bt.insert(n_chn);
                    ++n_chn;
                }
            }
        }
        if (n_chn == 0) continue;
        // iwork layout (R ints each): order | seed start | weight | sort stack (3 x 64)
        int *order = iwork + R0 * 3, *sstart = order + R, *wgt = order + 2 * R;
        // in-order traversal (__kb_traverse); a t = 5 B-tree over < 2^31 keys is < 16 levels deep
        {
            int n_ord = 0;
            int stk_x[40], stk_i[40];
            int sp = 0;
            stk_x[0] = bt.root; stk_i[0] = 0;
            for (;;) {
                while (stk_x[sp] >= 0 && stk_i[sp] <= nd[stk_x[sp]].n) {
                    const BtNode &x = nd[stk_x[sp]];
                    stk_x[sp + 1] = x.internal ? x.child[stk_i[sp]] : -1;
                    stk_i[sp + 1] = 0;
                    ++sp;
                }
                --sp;
                if (sp >= 0) {
                    const int xi = stk_x[sp];
                    if (xi >= 0 && stk_i[sp] < nd[xi].n) order[n_ord++] = nd[xi].key[stk_i[sp]];
                    ++stk_i[sp];
                } else break;
            }
        }
        // seeds grouped by chain in insertion order: chain c's seeds start at sstart[c]
        for (int c = 0; c < n_chn; ++c) sstart[c] = 0;
        for (int64_t k = 0; k < R; ++k) if (rc[k] >= 0) ++sstart[rc[k]];
        {
            int acc = 0;
            for (int c = 0; c < n_chn; ++c) { const int v = sstart[c]; sstart[c] = acc; acc += v; }
        }
        DevSeed *sd = out_seeds + R0;
        {
            // place seeds; wgt[] counts per chain while placing
            for (int c = 0; c < n_chn; ++c) wgt[c] = 0;
            for (int64_t i = s0; i < s1; ++i) {
                const DevIntv p = seeds[i];
                const int slen = (int)((uint32_t)p.info - (uint32_t)(p.info >> 32));
                const int64_t rlo = row_off_of_seed[i] - R0, rhi = row_off_of_seed[i + 1] - R0;
                for (int64_t k = rlo; k < rhi; ++k) {
                    const int c = rc[k];
                    if (c < 0) continue;
                    DevSeed s;
                    s.rbeg = (int64_t)pos[R0 + k];
                    s.qbeg = (int)(p.info >> 32);
                    s.len = s.score = slen;
                    s.pad = 0;
                    sd[sstart[c] + wgt[c]++] = s;
                }
            }
        }
        // mem_chain_weight (bwamem.c:229-250) per chain, indexed by tree order
        for (int c = 0; c < n_chn; ++c) {
            const DevSeed *s = sd + sstart[c];
            const int n = ch[c].n;
            int64_t end = 0;
            int w = 0, tmp;
            for (int j = 0; j < n; ++j) {
                if (s[j].qbeg >= end) w += s[j].len;
                else if (s[j].qbeg + s[j].len > end) w += (int)(s[j].qbeg + s[j].len - end);
                end = end > s[j].qbeg + s[j].len ? end : s[j].qbeg + s[j].len;
            }
            tmp = w; w = 0; end = 0;
            for (int j = 0; j < n; ++j) {
                if (s[j].rbeg >= end) w += s[j].len;
                else if (s[j].rbeg + s[j].len > end) w += (int)(s[j].rbeg + s[j].len - end);
                end = end > s[j].rbeg + s[j].len ? end : s[j].rbeg + s[j].len;
            }
            w = w < tmp ? w : tmp;
            wgt[c] = w < (1 << 30) ? w : (1 << 30) - 1;
        }
        // mem_chain_flt (bwamem.c:331-389): drop light chains, sort by weight, mark kept
        int n = 0;
        for (int k = 0; k < n_chn; ++k)
            if (wgt[order[k]] >= opt.min_chain_weight) order[n++] = order[k];
        if (n == 0) continue;
        {
            int stk_l[64], stk_r[64], stk_d[64];
            KsSort<FltLt> fs{order, FltLt{wgt}};
            fs.sort(n, stk_l, stk_r, stk_d);
        }
        DevChain *oc = out_chains + R0;              // working copy, compacted at the end
        for (int k = 0; k < n; ++k) {
            const int c = order[k];
            oc[k].n = ch[c].n; oc[k].rid = ch[c].rid; oc[k].w = wgt[c];
            oc[k].kept = 0; oc[k].first = -1; oc[k].seed_off = sstart[c];
            oc[k].frac_rep = frac_rep; oc[k].pad = 0;
        }
        {
            // kept chain indices reuse rc[] (rows are no longer needed)
            int *kept = rc, n_kept = 0;
            oc[0].kept = 3;
            kept[n_kept++] = 0;
            for (int i = 1; i < n; ++i) {
                int large_ovlp = 0, k;
                const DevSeed *si = sd + oc[i].seed_off;
                const int bi = si[0].qbeg, ei = si[oc[i].n - 1].qbeg + si[oc[i].n - 1].len;
                for (k = 0; k < n_kept; ++k) {
                    const int j = kept[k];
                    const DevSeed *sj = sd + oc[j].seed_off;
                    const int bj = sj[0].qbeg, ej = sj[oc[j].n - 1].qbeg + sj[oc[j].n - 1].len;
                    const int b_max = bj > bi ? bj : bi, e_min = ej < ei ? ej : ei;
                    if (e_min > b_max) {                  // no ALT contigs: the is_alt test always passes
                        const int li = ei - bi, lj = ej - bj, min_l = li < lj ? li : lj;
                        if (e_min - b_max >= min_l * opt.mask_level && min_l < opt.max_chain_gap) {
                            large_ovlp = 1;
                            if (oc[j].first < 0) oc[j].first = i;
                            if (oc[i].w < oc[j].w * opt.drop_ratio && oc[j].w - oc[i].w >= opt.min_seed_len << 1)
                                break;
                        }
                    }
                }
                if (k == n_kept) {
                    kept[n_kept++] = i;
                    oc[i].kept = large_ovlp ? 2 : 3;
                }
            }
            for (int i = 0; i < n_kept; ++i)
                if (oc[kept[i]].first >= 0) oc[oc[kept[i]].first].kept = 1;
            int i, k = 0;
            for (i = 0; i < n; ++i) {
                if (oc[i].kept == 0 || oc[i].kept == 3) continue;
                if (++k >= opt.max_chain_extend) break;
            }
            for (; i < n; ++i)
                if (oc[i].kept < 3) oc[i].kept = 0;
            for (i = k = 0; i < n; ++i)
                if (oc[i].kept != 0) oc[k++] = oc[i];
            n_chains[r] = k;
        }
    }
}

// ---------------------------------------------------------------- chaining, a warp per read

// mem_chain, mem_chain_weight and mem_chain_flt with a warp per read.  The tree serves two
// purposes, the chain with the largest pos at or before a row, and the chains in order of pos; while
// no two chains of a read have the same pos neither depends on the tree's nodes.  A read where a
// second chain would start at a pos that another one has (a seed that fails test_and_merge against
// the chain it found there) goes to chain_kernel.
//
// chain_fast, up to kFastRows rows and 64 chains (of the 100 Mb workload's reads all but a few in a
// thousand): the chains' places lie sorted over the lanes' registers, two a lane, so a row's
// chain is one ballot and an insertion one shuffle; the chains' fields lie in shared memory.  Rows are
// taken in order, one after the other (each sees the chains of those before), but their seed, contig
// and place are found 32 at a time.  ks_introsort: a partition step's swaps follow from two
// ballots over its segment, and the closing insertion sort is a stable sort, i.e. ranks.
// mem_chain_flt: one step per kept chain, all others compared with it at once, in place of one
// step per chain.
// chain_general, any size: the same on arrays in the read's slices of the scratch, the sort on one lane.
//
// One thread per read walking the tree in global memory took 2.27 ms for 67k reads of 150 bases (36
// rows, 20 chains a read), some 20,000 cycles a row; a warp per read with chain_general on shared
// memory 1.03 ms (75,000 cycles a read: 960 a row, 12,500 the sort, 14,800 the filter); this 0.63 ms
// (114k RRBS reads 1.78 -> 0.74 ms, 64 reads 78 -> 19 us), 6000 instructions a read with the issue
// slots 71 % busy; with the longest reads first (order_hist_rows) and chain_general's filter by kept chains 0.50
// and 0.51.  40 warps per SM (48 registers): 24 at 80 registers 0.68, 32 at 64 0.65.
constexpr int kFastRows = 128, kFastChains = 64, kChainWarps = 4;

struct FastChain {
    int64_t pos, last_rbeg;             // first seed's rbeg, last seed's
    int rid, first_qbeg, last_q, n;     // last_q: last seed's qbeg << 16 | len
};
struct ChainSmem {
    FastChain ch[kFastChains];
    int row[kFastRows], row_q[kFastRows];           // chain << 16 | place in it, or -1; qbeg << 16 | len
    int order[kFastChains], weight[kFastChains], start[kFastChains];
};

// ks_introsort (ksort.h:146-226) of order[0 .. n), n <= 64, by weight[] (of the same places),
// descending: the permutation it leaves, ties included.
__device__ __forceinline__ void sort_places(int *order, int *weight, int n, int lane)
{
    const auto swap2 = [&](int x, int y) {
        const int c = order[x], w = weight[x];
        order[x] = order[y], weight[x] = weight[y];
        order[y] = c, weight[y] = w;
    };
    if (n > 2) {
        int d, top = 0, s = 0, t = n - 1;
        int stk[8];                                     // s | t << 8 | d << 16; segments of more than 16 only
        for (d = 2; 1 << d < n; ++d) ;
        d <<= 1;
        for (;;) {
            if (s < t) {
                if (--d == 0) {                         // the reference's combsort
                    if (lane == 0) {
                        const double shrink_factor = 1.2473309501039786540366528676643;
                        const int m = t - s + 1;
                        int swapped, gap = m;
                        do {
                            if (gap > 2) {
                                gap = (int)(gap / shrink_factor);
                                if (gap == 9 || gap == 10) gap = 11;
                            }
                            swapped = 0;
                            for (int i = s; i + gap < s + m; ++i)
                                if (weight[i + gap] > weight[i]) swap2(i, i + gap), swapped = 1;
                        } while (swapped || gap > 2);
                        if (gap != 1)
                            for (int i = s + 1; i < s + m; ++i)
                                for (int j = i; j > s && weight[j] > weight[j - 1]; --j) swap2(j, j - 1);
                    }
                    __syncwarp();
                    t = s;
                    continue;
                }
                int k = s + ((t - s) >> 1) + 1;
                const int ws = weight[s], wt = weight[t], wm = weight[k];
                if (wm > ws) {
                    if (wm > wt) k = t;
                } else {
                    k = wt > ws ? s : t;
                }
                const int wp = weight[k];
                __syncwarp();
                if (lane == 0 && k != t) swap2(k, t);
                __syncwarp();
                // from the left the places not above the pivot, from the right those not below it
                const int w0 = lane < n ? weight[lane] : 0, w1 = lane + 32 < n ? weight[lane + 32] : 0;
                const uint64_t in = (~0ull >> (63 - t)) & (~0ull << s);
                uint64_t L = in & ((uint64_t)__ballot_sync(BSB_FULL_MASK, w1 <= wp) << 32 |
                                   __ballot_sync(BSB_FULL_MASK, w0 <= wp));
                const uint64_t Rm = in & ((uint64_t)__ballot_sync(BSB_FULL_MASK, w1 >= wp) << 32 |
                                          __ballot_sync(BSB_FULL_MASK, w0 >= wp));
                int i = s, j = t, x = -1, y = -1;       // lane q swaps the q-th pair
                for (int q = 0;; ++q) {
                    i = __ffsll((long long)(L & (~0ull << i << 1))) - 1;         // t is among them
                    const uint64_t below = Rm & ((1ull << j) - 1ull);
                    const int p = 63 - __clzll((long long)below);               // -1: none
                    if (p <= i) break;
                    j = p;
                    L |= 1ull << j;                     // it takes place i's, which is not above the pivot
                    if (lane == q) x = i, y = j;
                }
                __syncwarp();
                if (x >= 0) swap2(x, y);
                __syncwarp();
                if (lane == 0) swap2(i, t);
                __syncwarp();
                if (i - s > t - i) {
                    if (i - s > 16) stk[top++] = s | (i - 1) << 8 | d << 16;
                    s = t - i > 16 ? i + 1 : t;
                } else {
                    if (t - i > 16) stk[top++] = (i + 1) | t << 8 | d << 16;
                    t = i - s > 16 ? i - 1 : s;
                }
            } else {
                if (top == 0) break;
                --top;
                s = stk[top] & 255, t = stk[top] >> 8 & 255, d = stk[top] >> 16;
            }
        }
    }
    // insertion sort: stable
    int c[2], w[2], rank[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int k = lane + 32 * h;
        c[h] = k < n ? order[k] : 0, w[h] = k < n ? weight[k] : 0, rank[h] = 0;
    }
    for (int e = 0; e < n; ++e) {
        const int u = weight[e];
#pragma unroll
        for (int h = 0; h < 2; ++h) rank[h] += u > w[h] || (u == w[h] && e < lane + 32 * h);
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (lane + 32 * h < n) order[rank[h]] = c[h], weight[rank[h]] = w[h];
    __syncwarp();
}

// -1: more than 64 chains (chain_general takes the read); 0: left to chain_kernel; 1: done, n_out
// kept chains.
__device__ __forceinline__ int chain_fast(const AlnOpt &opt, const DevBns &B, float frac_rep, const DevIntv *seeds, int ns,
                                          const int64_t *roff, int64_t R0, int R, const uint64_t *pos, ChainSmem &S,
                                          DevSeed *sd, DevChain *oc, int lane, int &n_out)
{
    constexpr int64_t kNone = INT64_MAX;
    n_out = 0;
    // mem_chain (bwamem.c:279-305).  p[h], c[h]: the chain with the (lane + 32 h)-th smallest pos
    int64_t p[2] = {kNone, kNone};
    int c[2] = {0, 0}, n = 0;
    for (int base = 0; base < R; base += 32) {
        const int k = base + lane;
        int64_t rb = 0;
        int q = 0, rid = -1;
        // the seed of row k: the last with roff <= R0 + k, 32 seeds at a time over the lanes
        int at = 0;
        for (int s0 = 0; s0 < ns; s0 += 32) {
            const int first = s0 + lane < ns ? (int)min(roff[s0 + lane] - R0, (int64_t)INT_MAX) : INT_MAX;
            int lo = 0, hi = 32;                        // seeds of these that start at or before k
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                const int mid = (lo + hi) >> 1, f = __shfl_sync(BSB_FULL_MASK, first, min(mid, 31));
                if (lo < hi) {
                    if (f <= k) lo = mid + 1;
                    else hi = mid;
                }
            }
            at += lo;
            if (__all_sync(BSB_FULL_MASK, lo < 32 || k >= R)) break;
        }
        if (k < R) {
            const uint64_t info = seeds[at - 1].info;
            const int qb = (int)(info >> 32), sl = (int)(uint32_t)info - qb;
            q = qb << 16 | sl;
            rb = (int64_t)pos[R0 + k];
            rid = intv2rid(B, rb, rb + sl);
            S.row[k] = -1;
            S.row_q[k] = q;
        }
        __syncwarp();
        for (unsigned todo = __ballot_sync(BSB_FULL_MASK, rid >= 0); todo; todo &= todo - 1) {
            const int j = __ffs(todo) - 1;
            const int64_t rbeg = __shfl_sync(BSB_FULL_MASK, rb, j);
            const int id = __shfl_sync(BSB_FULL_MASK, rid, j), qs = __shfl_sync(BSB_FULL_MASK, q, j);
            const int qbeg = qs >> 16, slen = qs & 0xffff;
            int below = __popc(__ballot_sync(BSB_FULL_MASK, p[0] <= rbeg));
            if (n > 32) below += __popc(__ballot_sync(BSB_FULL_MASK, p[1] <= rbeg));
            if (below) {                                // test_and_merge (bwamem.c:203-227)
                const int e = below - 1, ci = __shfl_sync(BSB_FULL_MASK, e < 32 ? c[0] : c[1], e & 31);
                const FastChain f = S.ch[ci];
                const int lq = f.last_q >> 16, ll = f.last_q & 0xffff;
                const int64_t y = rbeg - f.last_rbeg;
                const int x = qbeg - lq;
                bool add = true;
                if (id != f.rid) {
                } else if (qbeg >= f.first_qbeg && qbeg + slen <= lq + ll && rbeg >= f.pos && y + slen <= ll) {
                    add = false;                        // contained: the seed is dropped
                } else if ((f.last_rbeg < B.l_pac || f.pos < B.l_pac) && rbeg >= B.l_pac) {
                } else if (y >= 0 && x - y <= opt.w && y - x <= opt.w && x - ll < opt.max_chain_gap &&
                           y - ll < opt.max_chain_gap) {
                    __syncwarp();
                    if (lane == 0) {
                        S.ch[ci].last_rbeg = rbeg, S.ch[ci].last_q = qs, S.ch[ci].n = f.n + 1;
                        S.row[base + j] = ci << 16 | f.n;
                    }
                    add = false;
                }
                if (!add) {
                    __syncwarp();
                    continue;
                }
                if (f.pos == rbeg) return 0;
            }
            if (n == kFastChains) return -1;
            if (lane == 0) {
                FastChain f;
                f.pos = f.last_rbeg = rbeg;
                f.rid = id, f.first_qbeg = qbeg, f.last_q = qs, f.n = 1;
                S.ch[n] = f;
                S.row[base + j] = n << 16;
            }
            if (n >= 32) {
                const int64_t up = __shfl_up_sync(BSB_FULL_MASK, p[1], 1), over = __shfl_sync(BSB_FULL_MASK, p[0], 31);
                const int cu = __shfl_up_sync(BSB_FULL_MASK, c[1], 1), co = __shfl_sync(BSB_FULL_MASK, c[0], 31);
                if (lane + 32 > below) p[1] = lane ? up : over, c[1] = lane ? cu : co;
                else if (lane + 32 == below) p[1] = rbeg, c[1] = n;
            }
            if (below < 32) {
                const int64_t up = __shfl_up_sync(BSB_FULL_MASK, p[0], 1);
                const int cu = __shfl_up_sync(BSB_FULL_MASK, c[0], 1);
                if (lane > below) p[0] = up, c[0] = cu;
                else if (lane == below) p[0] = rbeg, c[0] = n;
            }
            ++n;
            __syncwarp();
        }
    }
    if (n == 0) return 1;
    // where the chains' seeds start, in order of pos; the seeds
    int acc = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const bool has = lane + 32 * h < n;
        const int v = has ? S.ch[c[h]].n : 0;
        int incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(BSB_FULL_MASK, incl, d);
            if (lane >= d) incl += u;
        }
        if (has) S.start[c[h]] = acc + incl - v;
        acc += __shfl_sync(BSB_FULL_MASK, incl, 31);
    }
    __syncwarp();
    for (int k = lane; k < R; k += 32) {
        const int t = S.row[k];
        if (t < 0) continue;
        DevSeed s;
        s.rbeg = (int64_t)pos[R0 + k];
        s.qbeg = S.row_q[k] >> 16;
        s.len = s.score = S.row_q[k] & 0xffff;
        s.pad = 0;
        sd[S.start[t >> 16] + (t & 0xffff)] = s;
    }
    __syncwarp();
    // mem_chain_weight (bwamem.c:229-250); mem_chain_flt (bwamem.c:331-389): light chains dropped
    int m = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        int w = -1;
        if (lane + 32 * h < n) {
            const DevSeed *s = sd + S.start[c[h]];
            const int cn = S.ch[c[h]].n;
            int64_t qe = 0, re = 0;
            int wq = 0, wr = 0;
            for (int j = 0; j < cn; ++j) {
                const DevSeed t = s[j];
                if (t.qbeg >= qe) wq += t.len;
                else if (t.qbeg + t.len > qe) wq += (int)(t.qbeg + t.len - qe);
                qe = qe > t.qbeg + t.len ? qe : t.qbeg + t.len;
                if (t.rbeg >= re) wr += t.len;
                else if (t.rbeg + t.len > re) wr += (int)(t.rbeg + t.len - re);
                re = re > t.rbeg + t.len ? re : t.rbeg + t.len;
            }
            w = wr < wq ? wr : wq;
        }
        const bool heavy = lane + 32 * h < n && w >= opt.min_chain_weight;
        const unsigned hm = __ballot_sync(BSB_FULL_MASK, heavy);
        if (heavy) {
            const int at = m + __popc(hm & ((1u << lane) - 1u));
            S.order[at] = c[h], S.weight[at] = w;
        }
        m += __popc(hm);
    }
    n = m;
    if (n == 0) return 1;
    __syncwarp();
    if (n > 1) sort_places(S.order, S.weight, n, lane);
    // the kept chains one after the other (each the first that none before it dropped), all chains
    // behind it at once
    int b[2], e[2], w[2], mark[2] = {0, 0}, first[2] = {-1, -1};      // mark: 1 overlaps a kept chain, 2 is a first
    bool alive[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int k = lane + 32 * h;
        alive[h] = k < n;
        c[h] = k < n ? S.order[k] : 0, w[h] = k < n ? S.weight[k] : 0;
        b[h] = S.ch[c[h]].first_qbeg;
        const int lq = S.ch[c[h]].last_q;
        e[h] = (lq >> 16) + (lq & 0xffff);
    }
    for (int j = 0; j < n;) {
        const int jl = j & 31, bj = __shfl_sync(BSB_FULL_MASK, j < 32 ? b[0] : b[1], jl);
        const int ej = __shfl_sync(BSB_FULL_MASK, j < 32 ? e[0] : e[1], jl);
        const int wj = __shfl_sync(BSB_FULL_MASK, j < 32 ? w[0] : w[1], jl);
        uint64_t over = 0, live = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            bool ovl = false;
            if (alive[h] && lane + 32 * h > j) {
                const int b_max = bj > b[h] ? bj : b[h], e_min = ej < e[h] ? ej : e[h];
                if (e_min > b_max) {                     // no ALT contigs: the is_alt test always passes
                    const int li = e[h] - b[h], lj = ej - bj, min_l = li < lj ? li : lj;
                    if (e_min - b_max >= min_l * opt.mask_level && min_l < opt.max_chain_gap) {
                        ovl = true;
                        mark[h] |= 1;
                        if (w[h] < wj * opt.drop_ratio && wj - w[h] >= opt.min_seed_len << 1) alive[h] = false;
                    }
                }
            }
            over |= (uint64_t)__ballot_sync(BSB_FULL_MASK, ovl) << (32 * h);
            live |= (uint64_t)__ballot_sync(BSB_FULL_MASK, alive[h]) << (32 * h);
        }
        const int f = __ffsll((long long)over) - 1;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (lane + 32 * h == j) first[h] = f;
            if (lane + 32 * h == f) mark[h] |= 2;
        }
        const uint64_t rest = j == 63 ? 0ull : live & (~0ull << (j + 1));
        j = rest ? __ffsll((long long)rest) - 1 : n;
    }
    int kept[2];
    uint64_t weak = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        kept[h] = mark[h] & 2 ? 1 : !alive[h] ? 0 : mark[h] & 1 ? 2 : 3;
        weak |= (uint64_t)__ballot_sync(BSB_FULL_MASK, kept[h] == 1 || kept[h] == 2) << (32 * h);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int k = lane + 32 * h;
        // from the max_chain_extend-th of these on, only the strongest stay
        if (kept[h] < 3 && __popcll(weak & (~0ull >> (63 - k))) >= opt.max_chain_extend) kept[h] = 0;
        const unsigned km = __ballot_sync(BSB_FULL_MASK, kept[h] != 0);
        if (kept[h] != 0) {
            DevChain d;
            d.n = S.ch[c[h]].n, d.rid = S.ch[c[h]].rid, d.w = w[h];
            d.kept = kept[h], d.first = first[h], d.seed_off = S.start[c[h]];
            d.frac_rep = frac_rep, d.pad = 0;
            oc[n_out + __popc(km & ((1u << lane) - 1u))] = d;
        }
        n_out += __popc(km);
    }
    return 1;
}

struct ChainArrays {                    // of one read; R entries each
    int64_t *pos, *last_rbeg;           // per chain: first seed's rbeg, last seed's
    int *rid, *first_qbeg, *last_qbeg, *last_len, *n;
    int *row_chain, *row_at, *row_q;    // per row: its chain (-1: none), place in it, qbeg << 16 | len
    int *order, *start, *weight;        // per chain
};

// frac_rep (bwamem.c:271-278): only seeds with more than max_occ hits count.
__device__ __forceinline__ float repeat_share(const AlnOpt &opt, int len, const DevIntv *seeds, int ns, int lane)
{
    int l_rep = 0;
    bool many = false;
    for (int i = lane; i < ns; i += 32) many |= seeds[i].x2 > (uint64_t)opt.max_occ;
    if (__any_sync(BSB_FULL_MASK, many)) {
        int b = 0, e = 0;
        for (int i = 0; i < ns; ++i) {
            const int sb = (int)(seeds[i].info >> 32), se = (int)(uint32_t)seeds[i].info;
            if (seeds[i].x2 <= (uint64_t)opt.max_occ) continue;
            if (sb > e) l_rep += e - b, b = sb, e = se;
            else e = e > se ? e : se;
        }
        l_rep += e - b;
    }
    return (float)l_rep / len;
}

// Chains as weight << 20 | place, descending weight.
struct PackedWeightLt {
    __device__ bool operator()(int x, int y) const { return x >> 20 > y >> 20; }
};

// False: left to chain_kernel.  n_out: kept chains.
__device__ __noinline__ bool chain_general(const AlnOpt &opt, const DevBns &B, float frac_rep, const DevIntv *seeds,
                                           int ns, const int64_t *roff, int64_t R0, int R, const uint64_t *pos,
                                           ChainArrays A, DevSeed *sd, DevChain *oc, int lane, int *n_kept_out)
{
    const unsigned below = (1u << lane) - 1u;
    int n_out = 0;
    *n_kept_out = 0;
    // mem_chain (bwamem.c:279-305)
    int n_chn = 0;
    for (int base = 0; base < R; base += 32) {
        const int k = base + lane;
        int64_t rb = 0;
        int qb = 0, sl = 0, rid = -1;
        if (k < R) {
            int lo = 0, hi = ns - 1;                     // the seed of row k: the last with roff <= R0 + k
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (roff[mid] <= R0 + k) lo = mid;
                else hi = mid - 1;
            }
            const uint64_t info = seeds[lo].info;
            qb = (int)(info >> 32), sl = (int)(uint32_t)info - qb;
            rb = (int64_t)pos[R0 + k];
            rid = intv2rid(B, rb, rb + sl);
            A.row_chain[k] = -1;
            A.row_q[k] = qb << 16 | sl;
        }
        __syncwarp();
        const int rows = min(32, R - base);
        for (int j = 0; j < rows; ++j) {
            const int id = __shfl_sync(BSB_FULL_MASK, rid, j);
            if (id < 0) continue;
            const int64_t rbeg = __shfl_sync(BSB_FULL_MASK, rb, j);
            const int qbeg = __shfl_sync(BSB_FULL_MASK, qb, j), slen = __shfl_sync(BSB_FULL_MASK, sl, j);
            // the chain with the largest pos <= rbeg: high words first, then low words among the highest
            int64_t bp = -1;
            int bc = -1;
            for (int c = lane; c < n_chn; c += 32) {
                const int64_t p = A.pos[c];
                if (p <= rbeg && p > bp) bp = p, bc = c;
            }
            const int hi = (int)(bp >> 32), mh = __reduce_max_sync(BSB_FULL_MASK, hi);
            bool add = true;
            if (mh >= 0) {
                const uint32_t lw = hi == mh ? (uint32_t)bp : 0u, ml = __reduce_max_sync(BSB_FULL_MASK, lw);
                const unsigned m = __ballot_sync(BSB_FULL_MASK, hi == mh && (uint32_t)bp == ml);
                const int c = __shfl_sync(BSB_FULL_MASK, bc, __ffs(m) - 1);
                // test_and_merge (bwamem.c:203-227)
                const int64_t first_rbeg = A.pos[c], last_rbeg = A.last_rbeg[c];
                const int lq = A.last_qbeg[c], ll = A.last_len[c];
                const int64_t qend = lq + ll, rend = last_rbeg + ll;
                if (id != A.rid[c]) {
                } else if (qbeg >= A.first_qbeg[c] && qbeg + slen <= qend && rbeg >= first_rbeg && rbeg + slen <= rend) {
                    add = false;                         // contained: the seed is dropped
                } else if ((last_rbeg < B.l_pac || first_rbeg < B.l_pac) && rbeg >= B.l_pac) {
                } else {
                    const int64_t x = qbeg - lq, y = rbeg - last_rbeg;
                    if (y >= 0 && x - y <= opt.w && y - x <= opt.w && x - ll < opt.max_chain_gap &&
                        y - ll < opt.max_chain_gap) {
                        const int at = A.n[c];
                        __syncwarp();
                        if (lane == 0) {
                            A.last_qbeg[c] = qbeg, A.last_rbeg[c] = rbeg, A.last_len[c] = slen;
                            A.n[c] = at + 1;
                            A.row_chain[base + j] = c, A.row_at[base + j] = at;
                        }
                        add = false;
                    }
                }
                if (add && first_rbeg == rbeg) return false;
            }
            if (add) {
                if (lane == 0) {
                    A.pos[n_chn] = A.last_rbeg[n_chn] = rbeg;
                    A.first_qbeg[n_chn] = A.last_qbeg[n_chn] = qbeg, A.last_len[n_chn] = slen;
                    A.n[n_chn] = 1, A.rid[n_chn] = id;
                    A.row_chain[base + j] = n_chn, A.row_at[base + j] = 0;
                }
                ++n_chn;
            }
            __syncwarp();
        }
    }
    if (n_chn == 0) return true;
    // the chains in order of pos, and where their seeds start
    for (int c = lane; c < n_chn; c += 32) {
        const int64_t p = A.pos[c];
        int rank = 0;
        for (int d = 0; d < n_chn; ++d) rank += A.pos[d] < p;
        A.order[rank] = c;
    }
    for (int base = 0, acc = 0; base < n_chn; base += 32) {
        const int c = base + lane, v = c < n_chn ? A.n[c] : 0;
        int incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(BSB_FULL_MASK, incl, d);
            if (lane >= d) incl += u;
        }
        if (c < n_chn) A.start[c] = acc + incl - v;
        acc += __shfl_sync(BSB_FULL_MASK, incl, 31);
    }
    __syncwarp();
    for (int k = lane; k < R; k += 32) {
        const int c = A.row_chain[k];
        if (c < 0) continue;
        DevSeed s;
        s.rbeg = (int64_t)pos[R0 + k];
        s.qbeg = A.row_q[k] >> 16;
        s.len = s.score = A.row_q[k] & 0xffff;
        s.pad = 0;
        sd[A.start[c] + A.row_at[k]] = s;
    }
    __syncwarp();
    // mem_chain_weight (bwamem.c:229-250)
    for (int c = lane; c < n_chn; c += 32) {
        const DevSeed *s = sd + A.start[c];
        const int n = A.n[c];
        int64_t qe = 0, re = 0;
        int wq = 0, wr = 0;
        for (int j = 0; j < n; ++j) {
            const DevSeed t = s[j];
            if (t.qbeg >= qe) wq += t.len;
            else if (t.qbeg + t.len > qe) wq += (int)(t.qbeg + t.len - qe);
            qe = qe > t.qbeg + t.len ? qe : t.qbeg + t.len;
            if (t.rbeg >= re) wr += t.len;
            else if (t.rbeg + t.len > re) wr += (int)(t.rbeg + t.len - re);
            re = re > t.rbeg + t.len ? re : t.rbeg + t.len;
        }
        const int w = wr < wq ? wr : wq;
        A.weight[c] = w < (1 << 30) ? w : (1 << 30) - 1;
    }
    __syncwarp();
    // mem_chain_flt (bwamem.c:331-389): drop light chains, sort by weight, mark kept
    int n = 0;
    for (int base = 0; base < n_chn; base += 32) {
        const int k = base + lane, c = k < n_chn ? A.order[k] : 0;
        const bool heavy = k < n_chn && A.weight[c] >= opt.min_chain_weight;
        const unsigned m = __ballot_sync(BSB_FULL_MASK, heavy);
        if (heavy) A.order[n + __popc(m & below)] = c;
        n += __popc(m);
        __syncwarp();
    }
    if (n == 0) return true;
    if (n > 1) {
        // by weight, descending: ranks where the weights differ, ks_introsort's steps where some
        // are equal.  (row_at and row_chain are free from here on.)
        bool equal = false;
        for (int k = lane; k < n; k += 32) {
            const int c = A.order[k], w = A.weight[c];
            int rank = 0;
            for (int d = 0; d < n; ++d) {
                const int u = A.weight[A.order[d]];
                rank += u > w;
                equal |= u == w && d != k;
            }
            A.row_at[rank] = c;
        }
        equal = __any_sync(BSB_FULL_MASK, equal);
        __syncwarp();
        if (!equal) {
            for (int k = lane; k < n; k += 32) A.order[k] = A.row_at[k];
        } else {
            // one word for weight and chain where they fit (a weight is at most the read's length): a comparison
            // is then one load
            bool fits = n_chn <= 1 << 20;
            for (int k = lane; k < n; k += 32) fits &= A.weight[A.order[k]] < 1 << 11;
            fits = __all_sync(BSB_FULL_MASK, fits);
            if (fits) {
                for (int k = lane; k < n; k += 32) A.order[k] |= A.weight[A.order[k]] << 20;
                __syncwarp();
            }
            if (lane == 0) {
                int stk_l[64], stk_r[64], stk_d[64];
                if (fits) KsSort<PackedWeightLt>{A.order, PackedWeightLt{}}.sort(n, stk_l, stk_r, stk_d);
                else KsSort<FltLt>{A.order, FltLt{A.weight}}.sort(n, stk_l, stk_r, stk_d);
            }
            __syncwarp();
            if (fits)
                for (int k = lane; k < n; k += 32) A.order[k] &= (1 << 20) - 1;
        }
        __syncwarp();
    }
    // the kept chains one after the other, as in chain_fast: all chains behind one at once.  kept: first the marks
    // (1 overlaps a kept chain, 2 is a first, 4 dropped)
    int *const kept = A.row_chain, *const first = A.row_at;
    for (int k = lane; k < n; k += 32) kept[k] = 0, first[k] = -1;
    __syncwarp();
    for (int j = 0; j < n;) {
        const int cj = A.order[j], wj = A.weight[cj];
        const int bj = A.first_qbeg[cj], ej = A.last_qbeg[cj] + A.last_len[cj];
        int f = -1, next = n;
        for (int base = (j + 1) & ~31; base < n; base += 32) {
            const int k = base + lane;
            bool ovl = false, live = false;
            if (k > j && k < n && !(kept[k] & 4)) {
                live = true;
                const int ck = A.order[k], wk = A.weight[ck];
                const int bk = A.first_qbeg[ck], ek = A.last_qbeg[ck] + A.last_len[ck];
                const int b_max = bj > bk ? bj : bk, e_min = ej < ek ? ej : ek;
                if (e_min > b_max) {                     // no ALT contigs: the is_alt test always passes
                    const int lk = ek - bk, lj = ej - bj, min_l = lk < lj ? lk : lj;
                    if (e_min - b_max >= min_l * opt.mask_level && min_l < opt.max_chain_gap) {
                        ovl = true;
                        live = !(wk < wj * opt.drop_ratio && wj - wk >= opt.min_seed_len << 1);
                        kept[k] |= live ? 1 : 5;
                    }
                }
            }
            const unsigned mo = __ballot_sync(BSB_FULL_MASK, ovl), ml = __ballot_sync(BSB_FULL_MASK, live);
            if (mo && f < 0) f = base + __ffs(mo) - 1;
            if (ml && next == n) next = base + __ffs(ml) - 1;
        }
        __syncwarp();
        if (lane == 0 && f >= 0) first[j] = f, kept[f] |= 2;
        __syncwarp();
        j = next;
    }
    for (int k = lane; k < n; k += 32) {
        const int m = kept[k];
        kept[k] = m & 2 ? 1 : m & 4 ? 0 : m & 1 ? 2 : 3;
    }
    __syncwarp();
    if (n >= opt.max_chain_extend) {
        if (lane == 0) {
            int i, k = 0;
            for (i = 0; i < n; ++i) {
                if (kept[i] == 0 || kept[i] == 3) continue;
                if (++k >= opt.max_chain_extend) break;
            }
            for (; i < n; ++i)
                if (kept[i] < 3) kept[i] = 0;
        }
        __syncwarp();
    }
    for (int base = 0; base < n; base += 32) {
        const int i = base + lane;
        const bool keep = i < n && kept[i] != 0;
        const unsigned m = __ballot_sync(BSB_FULL_MASK, keep);
        if (keep) {
            const int c = A.order[i];
            DevChain d;
            d.n = A.n[c], d.rid = A.rid[c], d.w = A.weight[c];
            d.kept = kept[i], d.first = first[i], d.seed_off = A.start[c];
            d.frac_rep = frac_rep, d.pad = 0;
            oc[n_out + __popc(m & below)] = d;
        }
        n_out += __popc(m);
    }
    *n_kept_out = n_out;
    return true;
}

__global__ void __launch_bounds__(kChainWarps * 32, 10)
chain_warp_kernel(AlnOpt opt, DevBns B, int n_reads, const int64_t *__restrict__ read_off,
                  const DevIntv *__restrict__ seeds, const int64_t *__restrict__ seed_off,
                  const int64_t *__restrict__ row_off_of_seed, const uint64_t *__restrict__ pos,
                  ChainRec *__restrict__ chains, BtNode *__restrict__ nodes, int *__restrict__ row_chain,
                  int *__restrict__ iwork, DevSeed *__restrict__ out_seeds, DevChain *__restrict__ out_chains,
                  int *__restrict__ n_chains, int *__restrict__ left, int *__restrict__ n_left,
                  const int *__restrict__ order)
{
    __shared__ ChainSmem sm[kChainWarps];
    const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
    int r = blockIdx.x * kChainWarps + wb;
    if (r >= n_reads) return;
    if (order) r = order[r];
    const int len = (int)(read_off[r + 1] - read_off[r]);
    const int64_t s0 = seed_off[r], s1 = seed_off[r + 1];
    const int64_t R0 = row_off_of_seed[s0];
    const int R = (int)(row_off_of_seed[s1] - R0);
    int n_out = 0;
    bool done = true;
    if (len >= opt.min_seed_len && R > 0) {
        DevSeed *const sd = out_seeds + R0;
        DevChain *const oc = out_chains + R0;
        const int ns = (int)(s1 - s0);
        const float frac_rep = repeat_share(opt, len, seeds + s0, ns, lane);
        int how = -1;
        if (R <= kFastRows)
            how = chain_fast(opt, B, frac_rep, seeds + s0, ns, row_off_of_seed + s0, R0, R, pos, sm[wb], sd, oc, lane, n_out);
        done = how != 0;
        if (how < 0) {
            static_assert(sizeof(ChainRec) >= 2 * 8 + 5 * 4 && sizeof(BtNode) >= 2 * 4, "the read's scratch slices");
            ChainArrays A;
            A.pos = (int64_t *)(chains + R0), A.last_rbeg = A.pos + R;
            int *const ai = (int *)(A.last_rbeg + R);
            A.rid = ai, A.first_qbeg = ai + R, A.last_qbeg = ai + 2 * (int64_t)R, A.last_len = ai + 3 * (int64_t)R;
            A.n = ai + 4 * (int64_t)R;
            A.row_chain = row_chain + R0;
            A.row_at = (int *)(nodes + R0), A.row_q = A.row_at + R;
            A.order = iwork + R0 * 3, A.start = A.order + R, A.weight = A.order + 2 * (int64_t)R;
            __syncwarp();
            done = chain_general(opt, B, frac_rep, seeds + s0, ns, row_off_of_seed + s0, R0, R, pos, A, sd, oc, lane, &n_out);
        }
    }
    if (lane == 0) {
        n_chains[r] = n_out;
        if (!done) left[atomicAdd(n_left, 1)] = r;
    }
}

// ---------------------------------------------------------------- chain2aln

// Query base j and target base i of one extension: q(j) = read[q0 + qdir*j],
// t(i) = text base at t0 + tdir*i.  Left extensions run on both reversed,
// as the reference's reversed copies do (bwamem.c:721-724).
struct ReadRefAcc {
    const uint8_t *read;
    int q0, qdir;
    int64_t t0;
    int tdir;
    DevBns B;
    __device__ __forceinline__ int q(int j) const { return read[q0 + qdir * j]; }
    __device__ __forceinline__ int t(int i) const { return text_base(B, t0 + (int64_t)tdir * i); }
};

__device__ __forceinline__ int cal_max_gap(const AlnOpt &o, int qlen)         // bwamem.c:625-632
{
    const int l_del = band_cap(qlen * o.a - o.o_del, o.e_del);
    const int l_ins = band_cap(qlen * o.a - o.o_ins, o.e_ins);
    int l = l_del > l_ins ? l_del : l_ins;
    l = l > 1 ? l : 1;
    return l < o.w << 1 ? l : o.w << 1;
}

template <int C>
__device__ KswResult run_ext(const KswParams &P, int qlen, int tlen, int h0, int w, int eb, const ReadRefAcc &acc,
                             int lane, bool count_cells)
{
    return ksw_warp<C>(P, qlen, tlen, h0, w, eb, acc, lane, count_cells);
}

// A warp tile (C columns per lane) that holds qlen + 1 columns; a kernel compiled for
// reads of at most 32 * MaxC - 1 bases only instantiates C <= MaxC.
template <int MaxC>
__device__ KswResult extend_any(const KswParams &P, const int8_t *tab, int qlen, int tlen, int h0, int w, int eb,
                                const ReadRefAcc &acc, int lane, bool count_cells)
{
    // most extensions of a read are its own bases with a mismatch at most: no DP (ksw_core.cuh)
    if (!count_cells) {
        int best, best_j, last;
        if (ksw_diagonal<32>(tab, P.mat_max, diagonal_limit(P, h0), qlen, tlen, h0, acc, lane, best, best_j, last)) {
            KswResult r;
            r.score = best, r.qle = r.tle = best_j + 1, r.gtle = qlen, r.gscore = last, r.max_off = 0, r.cells = 0;
            return r;
        }
    }
    // One width per kernel where it can be: each width is a fully unrolled copy of the
    // DP, and the warps of an SM run extensions of every length at once, so extra copies
    // cost more in instruction-cache misses than the columns a tighter fit saves
    // (measured on GB300: one 8-column copy beat {1, 2, 4, 8} by 20 % on a 100 Mb
    // reference with repeats and 2x150 reads, and by 2 % on a 2 Mb one with 2x100).
    const int need = (qlen + 32) >> 5;
    if constexpr (MaxC <= 8) {
        return run_ext<MaxC>(P, qlen, tlen, h0, w, eb, acc, lane, count_cells);
    } else if constexpr (MaxC <= 16) {
        if (need <= 8) return run_ext<8>(P, qlen, tlen, h0, w, eb, acc, lane, count_cells);
        return run_ext<16>(P, qlen, tlen, h0, w, eb, acc, lane, count_cells);
    } else {                 // reads of 512-1023 bases: extensions past 511 columns need 32 per lane
        if (need <= 8) return run_ext<8>(P, qlen, tlen, h0, w, eb, acc, lane, count_cells);
        if (need <= 16) return run_ext<16>(P, qlen, tlen, h0, w, eb, acc, lane, count_cells);
        return run_ext<32>(P, qlen, tlen, h0, w, eb, acc, lane, count_cells);
    }
}

// The target span of a chain's extensions: the widest that any seed can use (bwamem.c:646-661),
// clipped to the contig of the first seed as bns_fetch_seq does (bntseq.c:436-461).
__device__ __forceinline__ void chain_window(const AlnOpt &opt, const DevBns &B, int l_query, const DevSeed *cs, int n,
                                             int64_t &rmax0, int64_t &rmax1)
{
    const int64_t l_pac = B.l_pac;
    rmax0 = l_pac << 1, rmax1 = 0;
    for (int i = 0; i < n; ++i) {
        const DevSeed t = cs[i];
        const int64_t b = t.rbeg - (t.qbeg + cal_max_gap(opt, t.qbeg));
        const int64_t e = t.rbeg + t.len + ((l_query - t.qbeg - t.len) + cal_max_gap(opt, l_query - t.qbeg - t.len));
        rmax0 = rmax0 < b ? rmax0 : b;
        rmax1 = rmax1 > e ? rmax1 : e;
    }
    rmax0 = rmax0 > 0 ? rmax0 : 0;
    rmax1 = rmax1 < l_pac << 1 ? rmax1 : l_pac << 1;
    if (rmax0 < l_pac && l_pac < rmax1) {
        if (cs[0].rbeg < l_pac) rmax1 = l_pac;
        else rmax0 = l_pac;
    }
    int is_rev;
    const int rid = pos2rid(B, depos(B, cs[0].rbeg, is_rev));
    int64_t far_beg = B.ann_offset[rid], far_end = far_beg + B.ann_len[rid];
    if (is_rev) {
        const int64_t t = far_beg;
        far_beg = (l_pac << 1) - far_end;
        far_end = (l_pac << 1) - t;
    }
    rmax0 = rmax0 > far_beg ? rmax0 : far_beg;
    rmax1 = rmax1 < far_end ? rmax1 : far_end;
}

// ---------------------------------------------------------------- the chains' first extensions, batched

// mem_chain2aln takes a chain's seeds from the highest score down, and most chains are one seed, or
// one whose region then covers the others.  So the extensions of every chain's first seed are nearly
// all there are, and they need nothing of the read's other chains: they run as two batches of the
// job-parallel extension (ksw_extend.cu: the main diagonal first, then 4 to 32 lanes a job on 16-bit
// cells), left ends and then right ends, whose h0 is the left ends' score.  chain2aln_kernel takes the
// results where it comes to such a seed; what it passes over (a seed inside an earlier region) was
// extended for nothing.  A warp per extension of a few dozen rows took 8,100 warp instructions a
// region.  One GB300, everything from the read order to the regions: 114k RRBS reads (450k regions)
// 4.62 -> 1.68 ms; 67k reads of 150 bases 2.21 -> 1.05; 40k of 100 on 2 Mb 0.46 -> 0.39.  (With the jobs'
// bytes written out first, and chain2aln_kernel alone behind them, RRBS 2.54 against 1.98.)
struct PreChain {
    int64_t rmax0, rmax1;
    int seed, pad;                      // the first seed to extend
};
struct PreResults {                     // chains: NULL where there are none
    const PreChain *chains;
    const int64_t *off;                 // per read, its first chain's place
    const bsb_ext_out_t *left, *right;  // score < 0: not run
};

// One thread per kept chain: its window, its first seed and the two jobs, on the reads and the 2-bit
// reference as they lie.  Rows from qlen + w + 1 on are never reached (the band is then right of the
// query), so targets end there.
__global__ void pre_plan_kernel(AlnOpt opt, DevBns B, int64_t n_chains, int n_reads,
                                const int64_t *__restrict__ chain_off, const int64_t *__restrict__ read_off,
                                const int64_t *__restrict__ seed_off, const int64_t *__restrict__ row_off_of_seed,
                                const DevSeed *__restrict__ seeds, const DevChain *__restrict__ chains,
                                PreChain *__restrict__ pre, bsb_ext_job_t *__restrict__ left,
                                bsb_ext_job_t *__restrict__ right)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n_chains) return;
    int lo = 0, hi = n_reads - 1;                     // the chain's read: the last with chain_off <= t
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (chain_off[mid] <= t) lo = mid;
        else hi = mid - 1;
    }
    const int64_t R0 = row_off_of_seed[seed_off[lo]];
    const int l_query = (int)(read_off[lo + 1] - read_off[lo]);
    const DevChain c = chains[R0 + (t - chain_off[lo])];
    const DevSeed *cs = seeds + R0 + c.seed_off;
    PreChain p;
    bsb_ext_job_t L, R;
    memset(&p, 0, sizeof p);
    memset(&L, 0, sizeof L);
    L.flags = kExtNone;
    R = L;
    if (c.n > 0) {
        chain_window(opt, B, l_query, cs, c.n, p.rmax0, p.rmax1);
        for (int i = 1; i < c.n; ++i)
            if (cs[i].score >= cs[p.seed].score) p.seed = i;
        const DevSeed s = cs[p.seed];
        const int qe = s.qbeg + s.len;
        L.qlen = s.qbeg, R.qlen = l_query - qe;
        L.tlen = (int)min(s.rbeg - p.rmax0, (int64_t)L.qlen + opt.w + 1);
        R.tlen = (int)min(p.rmax1 - (s.rbeg + s.len), (int64_t)R.qlen + opt.w + 1);
        L.qoff = read_off[lo] + s.qbeg - 1, L.toff = s.rbeg - 1;
        R.qoff = read_off[lo] + qe, R.toff = s.rbeg + s.len;
        L.h0 = R.h0 = s.len * opt.a;
        L.w = R.w = opt.w;
        L.end_bonus = opt.pen_clip5, R.end_bonus = opt.pen_clip3;
        L.flags = L.qlen < 1 ? kExtNone : kExtBack, R.flags = R.qlen < 1 ? kExtNone : 0;
    }
    pre[t] = p;
    left[t] = L;
    right[t] = R;
}

// A result that mem_chain2aln would take without trying a wider band (bwamem.c:727,756).
__device__ __forceinline__ bool pre_usable(const AlnOpt &opt, const bsb_ext_out_t &x)
{
    return x.score >= 0 && x.max_off < (opt.w >> 1) + (opt.w >> 2);
}

__device__ __forceinline__ bool pre_result(const AlnOpt &opt, const bsb_ext_out_t &o, KswResult &x)
{
    x.score = o.score, x.qle = o.qle, x.tle = o.tle, x.gtle = o.gtle, x.gscore = o.gscore, x.max_off = o.max_off;
    x.cells = 0;
    return pre_usable(opt, o);
}

// The right ends' h0, or no job where the left end is not decided.
__global__ void pre_right_kernel(AlnOpt opt, int64_t n_chains, const bsb_ext_job_t *__restrict__ left,
                                 const bsb_ext_out_t *__restrict__ left_out, bsb_ext_job_t *__restrict__ right)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n_chains || (left[t].flags & kExtNone)) return;       // no left end: h0 as planned
    const bsb_ext_out_t x = left_out[t];
    if (pre_usable(opt, x)) right[t].h0 = x.score;
    else right[t].flags |= kExtNone;
}

// Is seed s (almost) contained in region p of its read (bwamem.c:675-690)?
struct RegSpan {
    int64_t rb, re;
    int qb, qe, w, seedlen0;
};
__device__ __forceinline__ bool seed_in_region(const AlnOpt &opt, int l_query, const RegSpan &p, int64_t rbeg, int qbeg,
                                               int len)
{
    if (rbeg < p.rb || rbeg + len > p.re || qbeg < p.qb || qbeg + len > p.qe) return false;
    if (len - p.seedlen0 > .1 * l_query) return false;
    int qd = qbeg - p.qb;
    int64_t rd = rbeg - p.rb;
    int max_gap = cal_max_gap(opt, qd < rd ? qd : (int)rd);
    int w = max_gap < p.w ? max_gap : p.w;
    if (qd - rd < w && rd - qd < w) return true;
    qd = p.qe - (qbeg + len);
    rd = p.re - (rbeg + len);
    max_gap = cal_max_gap(opt, qd < rd ? qd : (int)rd);
    w = max_gap < p.w ? max_gap : p.w;
    return qd - rd < w && rd - qd < w;
}

// Can seed s, contained in a region, lead elsewhere because of seed t, extended before it (bwamem.c:691-707)?
__device__ __forceinline__ bool seeds_part(int64_t s_rbeg, int s_qbeg, int s_len, int64_t t_rbeg, int t_qbeg, int t_len)
{
    if (t_len < s_len * .95) return false;
    return (s_qbeg <= t_qbeg && s_qbeg + s_len - t_qbeg >= s_len >> 2 && t_qbeg - s_qbeg != t_rbeg - s_rbeg) ||
           (t_qbeg <= s_qbeg && t_qbeg + t_len - s_qbeg >= s_len >> 2 && s_qbeg - t_qbeg != s_rbeg - t_rbeg);
}

// The ends of seed s's region from its extensions (bwamem.c:736-775; left has no part where the seed starts the read,
// right none where it ends it).
__device__ __forceinline__ void left_end(const AlnOpt &opt, const DevSeed &s, const KswResult &x, bsb_reg_t &a)
{
    if (x.gscore <= 0 || x.gscore <= a.score - opt.pen_clip5) {
        a.qb = s.qbeg - x.qle, a.rb = s.rbeg - x.tle;
        a.truesc = a.score;
    } else {
        a.qb = 0, a.rb = s.rbeg - x.gtle;
        a.truesc = x.gscore;
    }
}
__device__ __forceinline__ void right_end(const AlnOpt &opt, int l_query, const DevSeed &s, const KswResult &x, int sc0,
                                          bsb_reg_t &a)
{
    if (x.gscore <= 0 || x.gscore <= a.score - opt.pen_clip3) {
        a.qe = s.qbeg + s.len + x.qle, a.re = s.rbeg + s.len + x.tle;
        a.truesc += a.score - sc0;
    } else {
        a.qe = l_query, a.re = s.rbeg + s.len + x.gtle;
        a.truesc += x.gscore - sc0;
    }
}

// The learned order: reads by predicted cost, most expensive first, in 64 bins of half an
// octave of the predicted cells (key).
__device__ __forceinline__ int key_bin(int32_t key)
{
    if (key <= 0) return 63;
    const uint32_t k = (uint32_t)key;
    const int msb = 31 - __clz(k);
    const int half = 2 * msb + (msb > 0 ? (int)(k >> (msb - 1) & 1u) : 0);
    return 63 - (half < 63 ? half : 63);
}

// The order chain2aln_kernel takes reads in: by the keys given, or else (key NULL) most chains first (reads are
// independent, so the order changes no result; it shortens the tail a few repeat-laden reads would otherwise set).
// Where chain2aln_plain has gone before, only the reads it left.
constexpr int kOrderBins = 64, kOrderThreads = 256;
__device__ __forceinline__ int read_bin(const int32_t *key, const int *n_chains, int r)
{
    return key ? key_bin(key[r]) : kOrderBins - 1 - min(n_chains[r], kOrderBins - 1);
}

// mem_chain2aln for the reads whose extensions are all known (PreResults), a warp a read: 32 chains at a time, each lane
// one chain's first seed, its region and its record; then the chains in order, the seed of each against the regions so
// far over the lanes, and the chain's other seeds over the lanes, which must all be contained in a region and not part
// from the chain's first.  A read where one would be extended, or with more than kPlainRegs regions, gets n_regs -1:
// it is left for chain2aln_kernel, in the read order, and counted in its bin of that (cnt; key as in read_bin).  That
// kernel's loads follow one another chain by chain, on 16 warps an SM (it holds the DP).
// 114k RRBS reads (450k regions): 617 us -> 199 and 175 for the reads left; 67k of 150 bases 292 -> 89 and 86.  At 10
// blocks an SM, or a block for every four reads in place of 8 an SM: 20-80 us more.
constexpr int kPlainWarps = 4, kPlainRegs = 64;
__global__ void __launch_bounds__(kPlainWarps * 32, 8)
chain2aln_plain(AlnOpt opt, int n_reads, const int64_t *__restrict__ read_off, const int64_t *__restrict__ seed_off,
                const int64_t *__restrict__ row_off_of_seed, const DevSeed *__restrict__ seeds,
                const DevChain *__restrict__ chains, const int *__restrict__ n_chains, bsb_reg_t *__restrict__ regs,
                int *__restrict__ n_regs, PreResults pre, const int32_t *__restrict__ key, int *__restrict__ cnt)
{
    __shared__ RegSpan sm[kPlainWarps][kPlainRegs];
    const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
    RegSpan *const list = sm[wb];
    for (int r = blockIdx.x * kPlainWarps + wb; r < n_reads; r += gridDim.x * kPlainWarps) {
        const int nc = n_chains[r];
        const int64_t R0 = row_off_of_seed[seed_off[r]], P0 = pre.off[r];
        const int l_query = (int)(read_off[r + 1] - read_off[r]);
        const DevSeed *const sd = seeds + R0;
        int nav = 0;
        bool ok = true;
        __syncwarp();
        for (int base = 0; base < nc && ok; base += 32) {
            const int ci = base + lane;
            DevChain c;
            c.n = 0;
            if (ci < nc) c = chains[R0 + ci];
            DevSeed s;
            s.rbeg = 0, s.qbeg = s.len = s.score = 0;
            bsb_reg_t a;
            memset(&a, 0, sizeof a);
            bool known = true;
            int first = 0;
            if (c.n > 0) {
                first = pre.chains[P0 + ci].seed;
                s = sd[c.seed_off + first];
                a.w = opt.w, a.rid = c.rid, a.seedlen0 = s.len, a.frac_rep = c.frac_rep;
                KswResult x;
                if (s.qbeg) {
                    known = pre_result(opt, pre.left[P0 + ci], x);
                    a.score = x.score;
                    left_end(opt, s, x, a);
                } else {
                    a.score = a.truesc = s.len * opt.a, a.qb = 0, a.rb = s.rbeg;
                }
                if (s.qbeg + s.len != l_query) {
                    const int sc0 = a.score;
                    known = pre_result(opt, pre.right[P0 + ci], x) && known;
                    a.score = x.score;
                    right_end(opt, l_query, s, x, sc0, a);
                } else {
                    a.qe = l_query, a.re = s.rbeg + s.len;
                }
                for (int i = 0; i < c.n; ++i) {          // seedcov (bwamem.c:779-783)
                    const DevSeed t = c.n == 1 ? s : sd[c.seed_off + i];
                    if (t.qbeg >= a.qb && t.qbeg + t.len <= a.qe && t.rbeg >= a.rb && t.rbeg + t.len <= a.re)
                        a.seedcov += t.len;
                }
            }
            int slot = -1;
            for (unsigned todo = __ballot_sync(BSB_FULL_MASK, c.n > 0); todo; todo &= todo - 1) {
                const int j = __ffs(todo) - 1;
                const int64_t rbeg = __shfl_sync(BSB_FULL_MASK, s.rbeg, j);
                const int qbeg = __shfl_sync(BSB_FULL_MASK, s.qbeg, j), len = __shfl_sync(BSB_FULL_MASK, s.len, j);
                bool in = false;
                for (int i = lane; i < nav; i += 32) in |= seed_in_region(opt, l_query, list[i], rbeg, qbeg, len);
                const bool fresh = !__any_sync(BSB_FULL_MASK, in);
                if (fresh) {
                    ok = __shfl_sync(BSB_FULL_MASK, known, j) && nav < kPlainRegs;
                    if (!ok) break;
                    if (lane == j) list[nav] = RegSpan{a.rb, a.re, a.qb, a.qe, a.w, a.seedlen0}, slot = nav;
                    ++nav;
                    __syncwarp();
                }
                const int n = __shfl_sync(BSB_FULL_MASK, c.n, j);
                if (n > 1) {
                    const int f = __shfl_sync(BSB_FULL_MASK, first, j);
                    const DevSeed *const cs = sd + __shfl_sync(BSB_FULL_MASK, c.seed_off, j);
                    // (the reference marks an excluded seed by key 0, which a seed 0 of score 0 has in any case)
                    const bool stands = fresh && (f != 0 || __shfl_sync(BSB_FULL_MASK, s.score, j) != 0);
                    bool extends = false;
                    for (int i = lane; i < n; i += 32) {
                        if (i == f) continue;
                        const DevSeed t = cs[i];
                        bool held = false;
                        for (int x = 0; x < nav && !held; ++x)
                            held = seed_in_region(opt, l_query, list[x], t.rbeg, t.qbeg, t.len);
                        extends |= !held || (stands && seeds_part(t.rbeg, t.qbeg, t.len, rbeg, qbeg, len));
                    }
                    ok = !__any_sync(BSB_FULL_MASK, extends);
                    if (!ok) break;
                }
            }
            if (ok && slot >= 0) regs[R0 + slot] = a;
        }
        if (lane == 0) {
            n_regs[r] = ok ? nav : -1;
            if (!ok) atomicAdd(&cnt[read_bin(key, n_chains, r)], 1);
        }
    }
}

// One warp per read, the *n_list reads of `order`.  regs: the read's region slots start at its row offset.
// MaxC = 4, 5, 8 serve batches whose reads are at most 127, 159, 255 bases long (one DP
// copy of that width), 16 every read the batch accepts; the 4- and 5-column variants are
// held to 4 blocks (16 warps) per SM, the 8-column one to 3.
template <int MaxC>
__global__ void __launch_bounds__(128, MaxC <= 5 ? 4 : MaxC <= 8 ? 3 : 1)
chain2aln_kernel(AlnOpt opt, KswParams P, DevBns B, const uint8_t *__restrict__ reads,
                 const int64_t *__restrict__ read_off, const int64_t *__restrict__ seed_off,
                 const int64_t *__restrict__ row_off_of_seed, const DevSeed *__restrict__ seeds,
                 const DevChain *__restrict__ chains, const int *__restrict__ n_chains, uint64_t *__restrict__ srt_buf,
                 bsb_reg_t *__restrict__ regs, int *__restrict__ n_regs, int *__restrict__ next,
                 const int *__restrict__ order, const int *__restrict__ n_list, int64_t *__restrict__ read_cells,
                 PreResults pre)
{
    const int n_reads = *n_list;
    __shared__ int8_t tab[kScoreTable];
    load_score_table(P, tab);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (;;) {
        int k = 0;
        if (lane == 0) k = atomicAdd(next, 1);
        k = __shfl_sync(BSB_FULL_MASK, k, 0);
        if (k >= n_reads) break;
        const int r = order[k];
        const int64_t R0 = row_off_of_seed[seed_off[r]];
        const int nc = n_chains[r];
        const int l_query = (int)(read_off[r + 1] - read_off[r]);
        const uint8_t *query = reads + read_off[r];
        const DevSeed *sd = seeds + R0;
        const DevChain *chn = chains + R0;
        bsb_reg_t *av = regs + R0;
        uint64_t *srt = srt_buf + R0;
        int nav = 0;
        long long cells = 0;           // DP cells of the read's ksw_extend2 calls, band retries included
        const int64_t l_pac = B.l_pac;
        for (int ci = 0; ci < nc; ++ci) {
            const DevChain c = chn[ci];
            const DevSeed *cs = sd + c.seed_off;
            if (c.n == 0) continue;
            int64_t rmax0, rmax1;
            if (pre.chains) rmax0 = pre.chains[pre.off[r] + ci].rmax0, rmax1 = pre.chains[pre.off[r] + ci].rmax1;
            else chain_window(opt, B, l_query, cs, c.n, rmax0, rmax1);
            // seeds by (score, index) ascending; keys are distinct, so ranks give ks_introsort_64's order
            for (int i = lane; i < c.n; i += 32) {
                const uint64_t ki = (uint64_t)(uint32_t)cs[i].score << 32 | (uint32_t)i;
                int rank = 0;
                for (int j = 0; j < c.n; ++j)
                    rank += ((uint64_t)(uint32_t)cs[j].score << 32 | (uint32_t)j) < ki;
                srt[rank] = ki;
            }
            __syncwarp();
            for (int k = c.n - 1; k >= 0; --k) {
                const DevSeed s = cs[(uint32_t)srt[k]];
                // is the seed (almost) contained in a region of this read already? (bwamem.c:675-690)
                int hit = nav;
                for (int i0 = 0; i0 < nav && hit == nav; i0 += 32) {
                    const int i = i0 + lane;
                    bool ok = false;
                    if (i < nav) {
                        const bsb_reg_t p = av[i];
                        ok = seed_in_region(opt, l_query, RegSpan{p.rb, p.re, p.qb, p.qe, p.w, p.seedlen0}, s.rbeg, s.qbeg,
                                            s.len);
                    }
                    const unsigned m = __ballot_sync(BSB_FULL_MASK, ok);
                    if (m) hit = i0 + __ffs(m) - 1;
                }
                if (hit < nav) {   // contained: extend only if an overlapping seed may lead elsewhere (bwamem.c:691-707)
                    int found = c.n;
                    for (int i0 = k + 1; i0 < c.n && found == c.n; i0 += 32) {
                        const int i = i0 + lane;
                        bool ok = false;
                        if (i < c.n && srt[i] != 0) {
                            const DevSeed t = cs[(uint32_t)srt[i]];
                            ok = seeds_part(s.rbeg, s.qbeg, s.len, t.rbeg, t.qbeg, t.len);
                        }
                        const unsigned m = __ballot_sync(BSB_FULL_MASK, ok);
                        if (m) found = i0 + __ffs(m) - 1;
                    }
                    if (found == c.n) {
                        __syncwarp();
                        if (lane == 0) srt[k] = 0;
                        __syncwarp();
                        continue;
                    }
                }
                bsb_reg_t a;
                memset(&a, 0, sizeof a);
                int aw0 = opt.w, aw1 = opt.w;
                a.w = opt.w;
                a.score = a.truesc = -1;
                a.rid = c.rid;
                const bool first_seed = pre.chains && k == c.n - 1;
                if (s.qbeg) {      // left extension (bwamem.c:715-748)
                    ReadRefAcc acc{query, s.qbeg - 1, -1, s.rbeg - 1, -1, B};
                    const int tlen = (int)(s.rbeg - rmax0);
                    KswResult x;
                    const bool known = first_seed && pre_result(opt, pre.left[pre.off[r] + ci], x);
                    if (known) a.score = x.score;
                    for (int i = 0; i < 2 && !known; ++i) {
                        const int prev = a.score;
                        aw0 = opt.w << i;
                        x = extend_any<MaxC>(P, tab, s.qbeg, tlen, s.len * opt.a, aw0, opt.pen_clip5, acc, lane,
                                             read_cells != nullptr);
                        cells += x.cells;
                        a.score = x.score;
                        if (a.score == prev || x.max_off < (aw0 >> 1) + (aw0 >> 2)) break;
                    }
                    left_end(opt, s, x, a);
                } else a.score = a.truesc = s.len * opt.a, a.qb = 0, a.rb = s.rbeg;
                if (s.qbeg + s.len != l_query) {   // right extension (bwamem.c:750-775)
                    const int qe = s.qbeg + s.len, sc0 = a.score;
                    const int re = (int)(s.rbeg + s.len - rmax0);
                    ReadRefAcc acc{query, qe, 1, rmax0 + re, 1, B};
                    const int tlen = (int)(rmax1 - rmax0 - re);
                    KswResult x;
                    // (the right end's job started from the left end's score where that was known)
                    const bool known = first_seed && pre_result(opt, pre.right[pre.off[r] + ci], x);
                    if (known) a.score = x.score;
                    for (int i = 0; i < 2 && !known; ++i) {
                        const int prev = a.score;
                        aw1 = opt.w << i;
                        x = extend_any<MaxC>(P, tab, l_query - qe, tlen, sc0, aw1, opt.pen_clip3, acc, lane,
                                             read_cells != nullptr);
                        cells += x.cells;
                        a.score = x.score;
                        if (a.score == prev || x.max_off < (aw1 >> 1) + (aw1 >> 2)) break;
                    }
                    right_end(opt, l_query, s, x, sc0, a);
                } else a.qe = l_query, a.re = s.rbeg + s.len;
                int cov = 0;      // seedcov (bwamem.c:779-783)
                for (int i = lane; i < c.n; i += 32) {
                    const DevSeed t = cs[i];
                    if (t.qbeg >= a.qb && t.qbeg + t.len <= a.qe && t.rbeg >= a.rb && t.rbeg + t.len <= a.re) cov += t.len;
                }
                a.seedcov = __reduce_add_sync(BSB_FULL_MASK, cov);
                a.w = aw0 > aw1 ? aw0 : aw1;
                a.seedlen0 = s.len;
                a.frac_rep = c.frac_rep;
                if (lane == 0) av[nav] = a;
                ++nav;
                __syncwarp();
            }
        }
        if (lane == 0) {
            n_regs[r] = nav;
            if (read_cells) read_cells[r] = cells;
        }
    }
}

// ---------------------------------------------------------------- mem_flt_chained_seeds

// mem_flt_chained_seeds (bwamem.c:602-619) for the reads whose length makes it run
// (min_hsp[r] >= 0; the host evaluates the reference's double and float thresholds):
// each seed of each kept chain gets mem_seed_sw's score (bwamem.c:574-598) -- ksw_align2
// with KSW_XSTART over windows of 50 bases around the seed, on the GPU's ksw_align2 --
// and the chain keeps the seeds with no Smith-Waterman or a score of at least min_hsp,
// rescored.  seed_sw_window is mem_seed_sw up to its ksw_align2 call, with bns_fetch_seq's
// clip to the contig of the window's middle (bntseq.c:436-461); false: no SW, score -1.
constexpr int kSeedSwShortLen = 200, kSeedSwExt = 50;     // MEM_SHORT_LEN, MEM_SHORT_EXT

__device__ bool seed_sw_window(const DevBns &B, int l_query, const DevSeed &s, int &qb, int &qe, int64_t &rb,
                               int64_t &re)
{
    const int64_t l_pac = B.l_pac;
    if (s.len >= kSeedSwShortLen) return false;
    qb = s.qbeg, qe = s.qbeg + s.len;
    rb = s.rbeg, re = s.rbeg + s.len;
    const int64_t mid = (rb + re) >> 1;
    qb -= kSeedSwExt; qb = qb > 0 ? qb : 0;
    qe += kSeedSwExt; qe = qe < l_query ? qe : l_query;
    rb -= kSeedSwExt; rb = rb > 0 ? rb : 0;
    re += kSeedSwExt; re = re < l_pac << 1 ? re : l_pac << 1;
    if (rb < l_pac && l_pac < re) {
        if (mid < l_pac) re = l_pac;
        else rb = l_pac;
    }
    if (qe - qb >= kSeedSwShortLen || re - rb >= kSeedSwShortLen) return false;
    int is_rev;
    const int rid = pos2rid(B, depos(B, mid, is_rev));
    int64_t far_beg = B.ann_offset[rid], far_end = far_beg + B.ann_len[rid];
    if (is_rev) {
        const int64_t t = far_beg;
        far_beg = (l_pac << 1) - far_end;
        far_end = (l_pac << 1) - t;
    }
    rb = rb > far_beg ? rb : far_beg;
    re = re < far_end ? re : far_end;
    return true;
}

// Per read (thread per read): the Smith-Waterman jobs its seeds need and their bytes.
__global__ void seed_sw_count(DevBns B, int n_reads, const int *__restrict__ min_hsp,
                              const int64_t *__restrict__ read_off, const int64_t *__restrict__ seed_off,
                              const int64_t *__restrict__ row_off_of_seed, const DevSeed *__restrict__ seeds,
                              const DevChain *__restrict__ chains, const int *__restrict__ n_chains,
                              int *__restrict__ n_jobs, int64_t *__restrict__ n_bytes)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_reads; r += gridDim.x * blockDim.x) {
        int nj = 0;
        int64_t nb = 0;
        if (min_hsp[r] >= 0) {
            const int64_t R0 = row_off_of_seed[seed_off[r]];
            const int l_query = (int)(read_off[r + 1] - read_off[r]);
            for (int ci = 0; ci < n_chains[r]; ++ci) {
                const DevChain c = chains[R0 + ci];
                for (int i = 0; i < c.n; ++i) {
                    int qb, qe;
                    int64_t rb, re;
                    if (seed_sw_window(B, l_query, seeds[R0 + c.seed_off + i], qb, qe, rb, re))
                        ++nj, nb += (qe - qb) + (re - rb);
                }
            }
        }
        n_jobs[r] = nj;
        n_bytes[r] = nb;
    }
}

// The jobs (ksw_align2(qe-qb, query+qb, re-rb, rseq, ..., KSW_XSTART, 0)) and their bytes at
// each read's offsets, in chain and seed order.
__global__ void seed_sw_fill(DevBns B, int n_reads, const int *__restrict__ min_hsp,
                             const uint8_t *__restrict__ reads, const int64_t *__restrict__ read_off,
                             const int64_t *__restrict__ seed_off, const int64_t *__restrict__ row_off_of_seed,
                             const DevSeed *__restrict__ seeds, const DevChain *__restrict__ chains,
                             const int *__restrict__ n_chains, const int64_t *__restrict__ job_off,
                             const int64_t *__restrict__ byte_off, bsb_sw_job_t *__restrict__ jobs,
                             uint8_t *__restrict__ bytes)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_reads; r += gridDim.x * blockDim.x) {
        if (min_hsp[r] < 0) continue;
        const int64_t R0 = row_off_of_seed[seed_off[r]];
        const int l_query = (int)(read_off[r + 1] - read_off[r]);
        const uint8_t *q = reads + read_off[r];
        int64_t j = job_off[r], b = byte_off[r];
        for (int ci = 0; ci < n_chains[r]; ++ci) {
            const DevChain c = chains[R0 + ci];
            for (int i = 0; i < c.n; ++i) {
                int qb, qe;
                int64_t rb, re;
                if (!seed_sw_window(B, l_query, seeds[R0 + c.seed_off + i], qb, qe, rb, re)) continue;
                bsb_sw_job_t jb;
                jb.qoff = b, jb.qlen = qe - qb;
                for (int x = qb; x < qe; ++x) bytes[b++] = q[x];
                jb.toff = b, jb.tlen = (int32_t)(re - rb);
                for (int64_t x = rb; x < re; ++x) bytes[b++] = (uint8_t)text_base(B, x);
                jb.xtra = 0x80000;                                   // KSW_XSTART
                jb.pad_ = 0;
                jobs[j++] = jb;
            }
        }
    }
}

// The filter itself (bwamem.c:608-617): seeds keep their order, a seed without SW scores
// len * a, and chains shrink in place.
__global__ void seed_sw_apply(AlnOpt opt, DevBns B, int n_reads, const int *__restrict__ min_hsp,
                              const int64_t *__restrict__ read_off, const int64_t *__restrict__ seed_off,
                              const int64_t *__restrict__ row_off_of_seed, DevSeed *__restrict__ seeds,
                              DevChain *__restrict__ chains, const int *__restrict__ n_chains,
                              const int64_t *__restrict__ job_off, const int *__restrict__ score)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_reads; r += gridDim.x * blockDim.x) {
        const int mh = min_hsp[r];
        if (mh < 0) continue;
        const int64_t R0 = row_off_of_seed[seed_off[r]];
        const int l_query = (int)(read_off[r + 1] - read_off[r]);
        int64_t j = job_off[r];
        for (int ci = 0; ci < n_chains[r]; ++ci) {
            DevChain &c = chains[R0 + ci];
            DevSeed *cs = seeds + R0 + c.seed_off;
            int k = 0;
            for (int i = 0; i < c.n; ++i) {
                DevSeed sd = cs[i];
                int qb, qe;
                int64_t rb, re;
                const int sc = seed_sw_window(B, l_query, sd, qb, qe, rb, re) ? score[j++] : -1;
                if (sc < 0 || sc >= mh) {
                    sd.score = sc < 0 ? sd.len * opt.a : sc;
                    cs[k++] = sd;
                }
            }
            c.n = k;
        }
    }
}

// ---------------------------------------------------------------- learned read order

// Eight features per read for the learned extension-cost model (no reference counterpart:
// they only order the read queue of chain2aln_kernel), from the kept chains after the seed
// filter -- the inputs mem_chain2aln works from (bwamem.c:636-790):
//   f0 read length / 256          f1 log1p(kept chains) / 4     f2 log1p(their seeds) / 6
//   f3 best chain weight / length f4 mean seed offset / length  f5 chains on the reverse half
//   f6 C+G fraction of the read   f7 log2(1 + plain bound of the extension cells) / 24
// where the plain bound sums, over the seeds, the bases left and right of the seed times the
// band they are extended in (2w + 1).
__global__ void read_features_kernel(AlnOpt opt, DevBns B, int n_reads, const uint8_t *__restrict__ reads,
                                     const int64_t *__restrict__ read_off, const int64_t *__restrict__ seed_off,
                                     const int64_t *__restrict__ row_off_of_seed, const DevSeed *__restrict__ seeds,
                                     const DevChain *__restrict__ chains, const int *__restrict__ n_chains,
                                     float *__restrict__ feat)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_reads; r += gridDim.x * blockDim.x) {
        const int L = (int)(read_off[r + 1] - read_off[r]);
        const uint8_t *q = reads + read_off[r];
        const int64_t R0 = row_off_of_seed[seed_off[r]];
        int ns = 0, wmax = 0, nrev = 0, kept = 0, cg = 0;
        double qsum = 0., bound = 0.;
        for (int ci = 0; ci < n_chains[r]; ++ci) {
            const DevChain c = chains[R0 + ci];
            if (c.n == 0) continue;
            ++kept;
            wmax = c.w > wmax ? c.w : wmax;
            for (int i = 0; i < c.n; ++i) {
                const DevSeed sd = seeds[R0 + c.seed_off + i];
                ++ns;
                qsum += sd.qbeg;
                bound += (double)(L - sd.len) * (2 * opt.w + 1);
                nrev += sd.rbeg >= B.l_pac;
            }
        }
        for (int i = 0; i < L; ++i) cg += q[i] == 1 || q[i] == 2;
        float *f = feat + (int64_t)r * 8;
        const float l = L > 0 ? (float)L : 1.f;
        f[0] = L / 256.f;
        f[1] = log1pf((float)kept) / 4.f;
        f[2] = log1pf((float)ns) / 6.f;
        f[3] = wmax / l;
        f[4] = ns ? (float)(qsum / ns) / l : 0.f;
        f[5] = ns ? (float)nrev / ns : 0.f;
        f[6] = cg / l;
        f[7] = (float)(log2(1.0 + bound) / 24.0);
    }
}

// Counting sort into 64 bins in two kernels: the bins' sizes, then the places (bin -1: the read gets none; n_placed,
// optional: how many did).  A block counts in shared memory and touches each global counter once (one global atomic
// per read on a few busy counters took 84 us for 67k reads, the two kernels together).
template <class Bin>
__device__ __forceinline__ void order_count(int n_reads, int *__restrict__ cnt, Bin bin)
{
    __shared__ int sh[kOrderBins];
    if (threadIdx.x < kOrderBins) sh[threadIdx.x] = 0;
    __syncthreads();
    for (int r = blockIdx.x * kOrderThreads + threadIdx.x; r < n_reads; r += gridDim.x * kOrderThreads)
        atomicAdd(&sh[bin(r)], 1);
    __syncthreads();
    if (threadIdx.x < kOrderBins && sh[threadIdx.x]) atomicAdd(&cnt[threadIdx.x], sh[threadIdx.x]);
}
template <class Bin>
__device__ __forceinline__ void order_place(int n_reads, const int *__restrict__ cnt, int *__restrict__ cur,
                                            int *__restrict__ order, int *__restrict__ n_placed, Bin bin)
{
    __shared__ int off[kOrderBins], sh[kOrderBins];
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int b = 0; b < kOrderBins; ++b) off[b] = acc, acc += cnt[b];
        if (n_placed && blockIdx.x == 0) *n_placed = acc;
    }
    for (int base = blockIdx.x * kOrderThreads; base < n_reads; base += gridDim.x * kOrderThreads) {
        if (threadIdx.x < kOrderBins) sh[threadIdx.x] = 0;
        __syncthreads();
        const int r = base + threadIdx.x, b = r < n_reads ? bin(r) : -1;
        const int at = b < 0 ? 0 : atomicAdd(&sh[b], 1);
        __syncthreads();
        if (threadIdx.x < kOrderBins && sh[threadIdx.x])
            sh[threadIdx.x] = off[threadIdx.x] + atomicAdd(&cur[threadIdx.x], sh[threadIdx.x]);
        __syncthreads();
        if (b >= 0) order[sh[b] + at] = r;
        __syncthreads();
    }
}

// Not where chain2aln_plain has gone before, which counts.
__global__ void __launch_bounds__(kOrderThreads)
order_hist(const int32_t *__restrict__ key, const int *__restrict__ n_chains, int n_reads, int *__restrict__ cnt)
{
    order_count(n_reads, cnt, [=](int r) { return read_bin(key, n_chains, r); });
}
// n_regs: chain2aln_plain's (below 0: the read was left), or NULL.
__global__ void __launch_bounds__(kOrderThreads)
order_scatter(const int32_t *__restrict__ key, const int *__restrict__ n_chains, const int *__restrict__ n_regs, int n_reads,
              const int *__restrict__ cnt, int *__restrict__ cur, int *__restrict__ order, int *__restrict__ n_placed)
{
    order_place(n_reads, cnt, cur, order, n_placed,
                [=](int r) { return n_regs && n_regs[r] >= 0 ? -1 : read_bin(key, n_chains, r); });
}

// The order chain_warp_kernel takes a large batch's reads in: most rows first, in steps of four.  A read on
// chain_general takes up to 0.25 ms, and a few such among 67k reads, met anywhere in the batch, set the end of the
// kernel; and the four reads of a block then take about as long as one another.  67k reads of 150 bases 0.64 -> 0.50
// ms, 114k RRBS reads 0.74 -> 0.51, the sort 11 us of it.
__device__ __forceinline__ int rows_bin(const int64_t *__restrict__ seed_off, const int64_t *__restrict__ row_off_of_seed,
                                        int r)
{
    const int64_t q = (row_off_of_seed[seed_off[r + 1]] - row_off_of_seed[seed_off[r]]) >> 2;
    return kOrderBins - 1 - (int)(q < kOrderBins - 1 ? q : kOrderBins - 1);
}
constexpr int kRowOrderReads = 2048;    // smaller batches fit the GPU at once
__global__ void __launch_bounds__(kOrderThreads)
order_hist_rows(const int64_t *__restrict__ seed_off, const int64_t *__restrict__ row_off_of_seed, int n_reads,
                int *__restrict__ cnt)
{
    order_count(n_reads, cnt, [=](int r) { return rows_bin(seed_off, row_off_of_seed, r); });
}
__global__ void __launch_bounds__(kOrderThreads)
order_scatter_rows(const int64_t *__restrict__ seed_off, const int64_t *__restrict__ row_off_of_seed, int n_reads,
                   const int *__restrict__ cnt, int *__restrict__ cur, int *__restrict__ order)
{
    order_place(n_reads, cnt, cur, order, nullptr, [=](int r) { return rows_bin(seed_off, row_off_of_seed, r); });
}

// One warp per read (reads hold a few regions each).
__global__ void compact_regs(const bsb_reg_t *__restrict__ regs, const int64_t *__restrict__ seed_off,
                             const int64_t *__restrict__ row_off_of_seed, int n_reads, const int *__restrict__ n_regs,
                             const int64_t *__restrict__ out_off, bsb_reg_t *__restrict__ out)
{
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < n_reads; r += gridDim.x * wpb) {
        const bsb_reg_t *src = regs + row_off_of_seed[seed_off[r]];
        for (int i = lane; i < n_regs[r]; i += 32) out[out_off[r] + i] = src[i];
    }
}

// ---------------------------------------------------------------- mem_sort_dedup_patch

struct RegReLt {                      // alnreg_slt2 (bwamem.c:395): by end
    const bsb_reg_t *r;
    __device__ bool operator()(int x, int y) const { return r[x].re < r[y].re; }
};

struct RegScoreLt {                   // alnreg_slt (bwamem.c:398): score down, then rb, qb up
    const bsb_reg_t *r;
    __device__ bool operator()(int x, int y) const
    {
        const bsb_reg_t &a = r[x], &b = r[y];
        return a.score > b.score || (a.score == b.score && (a.rb < b.rb || (a.rb == b.rb && a.qb < b.qb)));
    }
};

struct DedupOpt {
    int w, max_chain_gap;
    float mask_level_redun;
    GlobalPen pen;
    int8_t mat[25];
};

constexpr int kDedupWarps = 4, kDedupFew = 64;

struct DedupSmem {                    // one warp's orders, and its global alignment of mem_patch_reg
    int *order, *weight;              // kDedupFew entries
    int32_t *H, *E;                   // max_len + 1 entries
    uint8_t *q;                       // max_len entries
};
__host__ __device__ __forceinline__ int dedup_warp_bytes(int max_len)
{
    return 4 * (2 * kDedupFew + 2 * (max_len + 1)) + ((max_len + 3) & ~3);
}

// dst[k] = src[ix ? ix[k] : k] for k < n by the warp, 4 bytes a lane; one_comp: with n_comp = 1.
__device__ __forceinline__ void copy_regs(bsb_reg_t *dst, const bsb_reg_t *src, const int *ix, int n, bool one_comp,
                                          int lane)
{
    constexpr int kWords = sizeof(bsb_reg_t) / 4, kComp = offsetof(bsb_reg_t, n_comp) / 4;
    for (int t = lane; t < n * kWords; t += 32) {
        const int k = t / kWords, f = t - k * kWords;
        const int v = ((const int *)(src + (ix ? ix[k] : k)))[f];
        ((int *)dst)[t] = one_comp && f == kComp ? 1 : v;
    }
}

// Target base i of [rb, re) after bwa_gen_cigar2's flip (bwa.c:216-221): read backwards on the
// reverse strand.
struct PatchText {
    DevBns B;
    int64_t rb, re;
    bool rev;
    __device__ __forceinline__ int operator[](int i) const { return text_base(B, rev ? re - 1 - i : rb + i); }
};

// mem_patch_reg's tests before its alignment (bwamem.c:413-428).
__device__ __forceinline__ bool patch_candidate(const DedupOpt &O, int64_t l_pac, const bsb_reg_t &a, const bsb_reg_t &b)
{
    if (a.rb < l_pac && b.rb >= l_pac) return false;                   // different strands
    if (a.qb >= b.qb || a.qe >= b.qe || a.re >= b.re) return false;   // not colinear
    int w = (int)((a.re - b.rb) - (a.qe - b.qb));
    w = w > 0 ? w : -w;
    const bool apart = a.re < b.rb || a.qe < b.qb;
    if (w > (apart ? O.w << 1 : O.w << 2)) return false;
    double r = __dsub_rn(__ddiv_rn((double)(a.re - b.rb), (double)(b.re - a.rb)),
                         __ddiv_rn((double)(a.qe - b.qb), (double)(b.qe - a.qb)));
    r = r > 0. ? r : -r;
    return !(r >= (apart ? (double)0.05f : (double)(0.05f * 2)));     // PATCH_MAX_R_BW
}

// The rest of mem_patch_reg (bwamem.c:410-439) on the warp: every lane takes the same steps; the global
// alignment of its bwa_gen_cigar2 call (score only, bwa.c:211-244) runs on the whole warp.  The
// reference's double expressions are evaluated as written (no fused multiply-adds).
__device__ __noinline__ int patch_reg_warp(const DedupOpt &O, const int8_t *smat, const DevBns &B, const uint8_t *read,
                                           const bsb_reg_t &a, const bsb_reg_t &b, int *w_out, const DedupSmem &S,
                                           int lane)
{
    const int64_t l_pac = B.l_pac;
    int w = (int)((a.re - b.rb) - (a.qe - b.qb));
    w = w > 0 ? w : -w;
    w += a.w + b.w;
    w = w < O.w << 2 ? w : O.w << 2;
    // bwa_gen_cigar2(..., w, l_pac, pac, pac, b.qe - a.qb, query + a.qb, a.rb, b.re, &score, 0, ...)
    const int lq = b.qe - a.qb;
    const int64_t rb = a.rb, re = b.re;
    const int sc2 = b.score + a.score;
    const int q_s = (int)__dadd_rn(__dmul_rn(__ddiv_rn((double)(b.qe - a.qb), (double)((b.qe - b.qb) + (a.qe - a.qb))),
                                             (double)sc2), .499);
    const int r_s = (int)__dadd_rn(__dmul_rn(__ddiv_rn((double)(b.re - a.rb), (double)((b.re - b.rb) + (a.re - a.rb))),
                                             (double)sc2), .499);
    int score = 0;
    if (!(lq <= 0 || rb >= re || (rb < l_pac && re > l_pac)) && rb >= 0 && re <= l_pac << 1) {
        const bool rev = rb >= l_pac;
        const int rlen = (int)(re - rb);
        for (int j = lane; j < lq; j += 32) S.q[j] = read[rev ? b.qe - 1 - j : a.qb + j];
        __syncwarp();
        const PatchText T{B, rb, re, rev};
        const int dl = rlen > lq ? rlen - lq : lq - rlen;
        if (lq == rlen && w == 0) {                                     // without gaps (bwa.c:222-230)
            int part = 0;
            for (int j = lane; j < lq; j += 32) part += smat[T[j] * 5 + S.q[j]];
            score = __reduce_add_sync(BSB_FULL_MASK, part);
        } else {                                                       // the band of bwa.c:232-240
            const int half = ((lq + 1) >> 1) * smat[0];
            const int max_ins = (int)__dadd_rn(__ddiv_rn((double)(half - O.pen.o_ins), (double)O.pen.e_ins), 1.);
            const int max_del = (int)__dadd_rn(__ddiv_rn((double)(half - O.pen.o_del), (double)O.pen.e_del), 1.);
            int max_gap = max_ins > max_del ? max_ins : max_del;
            max_gap = max_gap > 1 ? max_gap : 1;
            int bw = (max_gap + dl + 1) >> 1;
            bw = bw < w ? bw : w;
            bw = bw > dl + 3 ? bw : dl + 3;
            score = global_warp(O.pen, smat, S.q, lq, T, rlen, bw, 0, S.H, S.E, nullptr, lane);
        }
        __syncwarp();
    }
    if (__ddiv_rn((double)score, (double)(q_s > r_s ? q_s : r_s)) < (double)0.90f) return 0;   // PATCH_MIN_SC_RATIO
    *w_out = w;
    return score;
}

// mem_sort_dedup_patch (bwamem.c:441-493) per read, one warp per read.  in: the read's
// pre-dedup regions at reg_off[r]; a: scratch of the same size (the sorted copy that the scan
// edits); ix: index scratch; out: the kept regions at reg_off[r], n_out[r] of them.  The two
// ks_introsort orders: each region's count of regions that come before it decides every comparison, so
// up to 64 regions are sort_places' integers (more: lane 0 on the records).  The redundancy and
// merge scan is taken by every lane in step (lane 0 writes), so that the warp can run a merge's global
// alignment, and only at regions that reach the one before.
// Both sorts on one lane with the records in global memory, all regions scanned: 0.50 ms for 114k RRBS
// reads (450k regions), 0.20 ms for 67k of 150 bases; as here 0.25 and 0.12.  Time is a warp's own chain
// (10k clocks a read), so warps resident count up to where registers spill: at 6, 8, 10 and 12 blocks an SM the
// stage takes 0.315, 0.288, 0.287, 0.350 ms on the RRBS reads and 0.190, 0.181, 0.207, 0.237 on the others.
__global__ void __launch_bounds__(kDedupWarps * 32, 8)
dedup_kernel(DedupOpt O, DevBns B, int n_reads, const uint8_t *__restrict__ reads,
             const int64_t *__restrict__ read_off, const int64_t *__restrict__ reg_off,
             const bsb_reg_t *__restrict__ in, bsb_reg_t *a_all, int *ix_all, bsb_reg_t *__restrict__ out,
             int *__restrict__ n_out, int max_len)
{
    extern __shared__ __align__(16) char dedup_smem[];
    __shared__ int8_t smat[25];
    if (threadIdx.x < 25) smat[threadIdx.x] = O.mat[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
    DedupSmem S;
    S.order = (int *)(dedup_smem + wb * dedup_warp_bytes(max_len)), S.weight = S.order + kDedupFew;
    S.H = (int32_t *)(S.weight + kDedupFew), S.E = S.H + max_len + 1;
    S.q = (uint8_t *)(S.E + max_len + 1);
    for (int r = blockIdx.x * kDedupWarps + wb; r < n_reads; r += gridDim.x * kDedupWarps) {
        const int64_t o0 = reg_off[r];
        const int n = (int)(reg_off[r + 1] - o0);
        const bsb_reg_t *a_in = in + o0;
        bsb_reg_t *a = a_all + o0, *dst = out + o0;
        int *ix = ix_all + o0;
        if (n <= 1) {                                    // bwamem.c:444: returned as they are
            if (n == 1) copy_regs(dst, a_in, nullptr, 1, false, lane);
            if (lane == 0) n_out[r] = n;
            continue;
        }
        const bool few = n <= kDedupFew;
        // which regions the scan has to look at: those that reach the one before (neither its contig and end
        // nor a region's own start changes before the scan comes to it)
        uint64_t near = ~0ull;
        if (few) {                                       // sort by end (bwamem.c:445)
            int64_t re[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) re[h] = lane + 32 * h < n ? a_in[lane + 32 * h].re : 0;
            int less[2] = {0, 0};
            for (int e = 0; e < n; ++e) {
                const int64_t x = __shfl_sync(BSB_FULL_MASK, e < 32 ? re[0] : re[1], e & 31);
                less[0] += x < re[0], less[1] += x < re[1];
            }
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (lane + 32 * h < n) S.order[lane + 32 * h] = lane + 32 * h, S.weight[lane + 32 * h] = -less[h];
            __syncwarp();
            sort_places(S.order, S.weight, n, lane);
            near = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = lane + 32 * h;
                bool reach = false;
                if (k >= 1 && k < n) {
                    const bsb_reg_t &p = a_in[S.order[k]], &q = a_in[S.order[k - 1]];
                    reach = p.rid == q.rid && p.rb < q.re + O.max_chain_gap;
                }
                near |= (uint64_t)__ballot_sync(BSB_FULL_MASK, reach) << (32 * h);
            }
            if (near) copy_regs(a, a_in, S.order, n, true, lane);
            __syncwarp();
        } else {
            if (lane == 0) {
                int stk_l[64], stk_r[64], stk_d[64];
                for (int k = 0; k < n; ++k) ix[k] = k;
                KsSort<RegReLt>{ix, RegReLt{a_in}}.sort(n, stk_l, stk_r, stk_d);
            }
            __syncwarp();
            copy_regs(a, a_in, ix, n, true, lane);
            __syncwarp();
        }
        const uint8_t *read = reads + read_off[r];
        for (int i = 1; i < n; ++i) {                    // bwamem.c:447-474
            if (few) {
                const uint64_t rest = i < 64 ? near >> i : 0ull;
                if (!rest) break;
                i += __ffsll((long long)rest) - 1;
            }
            bsb_reg_t p = a[i];
            if (p.rid != a[i - 1].rid || p.rb >= a[i - 1].re + O.max_chain_gap) continue;
            // The reference goes down from i - 1 until a region is out of reach; here 32 at a time, the lanes
            // finding what each would do: end the scan, exclude region j, exclude region i and end, or try to
            // merge.  Exclusions of j change nothing for the others, so only the last two are taken one by one;
            // a merge changes p, and the regions below it are looked at again.
            bool ended = false;
            for (int top = i - 1; top >= 0 && !ended;) {
                const int j = top - lane;
                bool out = false, drop_j = false, drop_i = false, merge = false;
                if (j >= 0) {
                    const bsb_reg_t q = a[j];
                    out = p.rid != q.rid || p.rb >= q.re + O.max_chain_gap;
                    if (!out && q.qe != q.qb) {                  // (else a[j] has been excluded)
                        const int64_t or_ = q.re - p.rb;
                        const int64_t oq = q.qb < p.qb ? q.qe - p.qb : p.qe - q.qb;
                        const int64_t mr = q.re - q.rb < p.re - p.rb ? q.re - q.rb : p.re - p.rb;
                        const int64_t mq = q.qe - q.qb < p.qe - p.qb ? q.qe - q.qb : p.qe - p.qb;
                        // float, as the reference's float option times an int64
                        if ((float)or_ > __fmul_rn(O.mask_level_redun, (float)mr) &&
                            (float)oq > __fmul_rn(O.mask_level_redun, (float)mq)) {
                            drop_i = p.score < q.score;
                            drop_j = !drop_i;
                        } else {
                            merge = q.rb < p.rb && patch_candidate(O, B.l_pac, q, p);
                        }
                    }
                }
                const unsigned mo = __ballot_sync(BSB_FULL_MASK, out || j < 0);
                unsigned events = __ballot_sync(BSB_FULL_MASK, drop_i || merge);
                const unsigned reach = mo ? (1u << (__ffs(mo) - 1)) - 1u : 0xffffffffu;
                events &= reach;
                int next = mo ? -1 : top - 32, done = 0;        // lanes below `done` have been taken
                bool again = false;
                while (!again) {
                    const int e = events ? __ffs(events) - 1 : 32;
                    if (drop_j && lane >= done && lane < e && (reach >> lane & 1u)) a[j].qe = a[j].qb;
                    __syncwarp();
                    if (e == 32) break;
                    done = e + 1;
                    events &= events - 1;
                    if (__shfl_sync(BSB_FULL_MASK, drop_i, e)) {
                        if (lane == 0) a[i].qe = p.qb;
                        next = -1;
                        break;
                    }
                    const bsb_reg_t q = a[top - e];
                    int w = 0;
                    const int score = patch_reg_warp(O, smat, B, read, q, p, &w, S, lane);
                    if (score > 0) {                             // merge q into p
                        if (lane == 0) {
                            bsb_reg_t u = p;
                            u.n_comp += q.n_comp + 1;
                            u.seedcov = u.seedcov > q.seedcov ? u.seedcov : q.seedcov;
                            u.qb = q.qb, u.rb = q.rb;
                            u.truesc = u.score = score;
                            u.w = w;
                            a[i] = u;
                            a[top - e].qb = q.qe;
                        }
                        __syncwarp();
                        p = a[i];
                        next = top - e - 1;
                        again = true;
                    }
                }
                __syncwarp();
                ended = next < 0;
                top = next;
            }
        }
        __syncwarp();
        if (few) {                                       // bwamem.c:475-492
            // the regions in order: a's, or where the scan had nothing to do the given ones through S.order
            const bsb_reg_t *const from_regs = near ? a : a_in;
            int m = 0, first_reg = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = lane + 32 * h, c = k >= n ? 0 : near ? k : S.order[k];
                if (h == 0) first_reg = __shfl_sync(BSB_FULL_MASK, c, 0);
                const bool keep = k < n && from_regs[c].qe > from_regs[c].qb;
                const unsigned km = __ballot_sync(BSB_FULL_MASK, keep);
                if (keep) S.order[m + __popc(km & ((1u << lane) - 1u))] = c;
                m += __popc(km);
            }
            __syncwarp();
            int cnt = 1;
            if (m == 0) {                                // the reference then returns its first region
                if (lane == 0) S.order[0] = first_reg;
                __syncwarp();
                copy_regs(dst, from_regs, S.order, 1, !near, lane);
            } else {
                // by (score down, rb up, qb up); identical ones once
                int sc[2], qb[2], less[2] = {0, 0};
                int64_t rb[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const bsb_reg_t &x = from_regs[S.order[lane + 32 * h < m ? lane + 32 * h : 0]];
                    sc[h] = x.score, rb[h] = x.rb, qb[h] = x.qb;
                }
                for (int e = 0; e < m; ++e) {
                    const int es = __shfl_sync(BSB_FULL_MASK, e < 32 ? sc[0] : sc[1], e & 31);
                    const int eq = __shfl_sync(BSB_FULL_MASK, e < 32 ? qb[0] : qb[1], e & 31);
                    const int64_t er = __shfl_sync(BSB_FULL_MASK, e < 32 ? rb[0] : rb[1], e & 31);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        less[h] += es > sc[h] || (es == sc[h] && (er < rb[h] || (er == rb[h] && eq < qb[h])));
                }
                __syncwarp();
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (lane + 32 * h < m) S.weight[lane + 32 * h] = -less[h];
                __syncwarp();
                if (m > 1) sort_places(S.order, S.weight, m, lane);
                cnt = 0;
                int at[2], from[2];
                bool out_[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int k = lane + 32 * h;
                    out_[h] = k < m && (k == 0 || S.weight[k] != S.weight[k - 1]);
                    from[h] = k < m ? S.order[k] : 0;
                    const unsigned om = __ballot_sync(BSB_FULL_MASK, out_[h]);
                    at[h] = cnt + __popc(om & ((1u << lane) - 1u));
                    cnt += __popc(om);
                }
                __syncwarp();
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (out_[h]) S.order[at[h]] = from[h];
                __syncwarp();
                copy_regs(dst, from_regs, S.order, cnt, !near, lane);
            }
            if (lane == 0) n_out[r] = cnt;
            __syncwarp();
            continue;
        }
        if (lane == 0) {
            int m = 0;
            for (int k = 0; k < n; ++k)
                if (a[k].qe > a[k].qb) ix[m++] = k;
            int cnt;
            if (m == 0) {                                // the reference then returns its first region
                dst[0] = a[0];
                cnt = 1;
            } else {
                int stk_l[64], stk_r[64], stk_d[64];
                KsSort<RegScoreLt>{ix, RegScoreLt{a}}.sort(m, stk_l, stk_r, stk_d);
                dst[0] = a[ix[0]];
                cnt = 1;
                for (int k = 1; k < m; ++k) {
                    const bsb_reg_t &x = a[ix[k]], &y = a[ix[k - 1]];
                    if (!(x.score == y.score && x.rb == y.rb && x.qb == y.qb)) dst[cnt++] = x;
                }
            }
            n_out[r] = cnt;
        }
        __syncwarp();
    }
}

__global__ void compact_kept(const bsb_reg_t *__restrict__ regs, const int64_t *__restrict__ in_off, int n_reads,
                             const int *__restrict__ n_kept, const int64_t *__restrict__ out_off,
                             bsb_reg_t *__restrict__ out)
{
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < n_reads; r += gridDim.x * wpb) {
        const bsb_reg_t *src = regs + in_off[r];
        for (int i = lane; i < n_kept[r]; i += 32) out[out_off[r] + i] = src[i];
    }
}

}  // namespace

// ---------------------------------------------------------------- host driver

struct AlignScratch {
    int *rcnt;                   // per seed interval: SA rows
    int64_t *roff;               // n_seeds + 1
    uint64_t *rows, *pos;
    ChainRec *chains;
    BtNode *nodes;
    int *row_chain, *iwork;
    DevSeed *cseeds;
    DevChain *cchains;
    uint64_t *srt;
    bsb_reg_t *regs;
    int *n_chains, *n_regs, *ctrl;
    int64_t *reg_off;
};

static size_t al(size_t x) { return (x + 255) & ~(size_t)255; }

// dedup: also run mem_sort_dedup_patch per read (the regions mem_align1_core returns).
// The seed-level Smith-Waterman filter of the batch (mem_flt_chained_seeds) between chain_kernel
// and chain2aln_kernel, for the reads with h_min_hsp[r] >= 0: jobs and their bytes are built on
// the device, run through ksw_align2 on the GPU (bsb_align2_run, with staging of its own: d_in
// and d_out hold the batch meanwhile), and the scores go back to the chains on the device.
static int seed_sw_filter(bsb_ctx *ctx, const bsb_align_opt_t *o, const DevBns &B, int n_reads,
                          const int *h_min_hsp, const uint8_t *d_reads, const int64_t *d_read_off,
                          const int64_t *d_seed_off, const int64_t *roff, DevSeed *cseeds, DevChain *cchains,
                          const int *n_chains, const AlnOpt &ao)
{
    int rc;
    cudaStream_t st = ctx->stream;
    const size_t nr = (size_t)n_reads;
    const size_t head = al(4 * nr) + al(4 * nr) + al(8 * nr) + 2 * al(8 * (nr + 1));
    if ((rc = bsb_ensure(ctx, &ctx->flt_dev, &ctx->flt_dev_bytes, head + 256, "seed SW filter"))) return rc;
    char *D = (char *)ctx->flt_dev;
    int *d_mh = (int *)D, *d_nj = (int *)(D + al(4 * nr));
    int64_t *d_nb = (int64_t *)(D + 2 * al(4 * nr));
    int64_t *d_joff = (int64_t *)(D + 2 * al(4 * nr) + al(8 * nr)), *d_boff = d_joff + al(8 * (nr + 1)) / 8;
    const int grid = (int)std::min<int64_t>((n_reads + 127) / 128, (int64_t)ctx->n_sm * 8);
    std::vector<int> nj(nr);
    std::vector<int64_t> nbytes(nr), joff(nr + 1), boff(nr + 1);
    if ((rc = bsb_cuda(ctx, cudaMemcpyAsync(d_mh, h_min_hsp, 4 * nr, cudaMemcpyHostToDevice, st), "H2D min_hsp")))
        return rc;
    seed_sw_count<<<grid, 128, 0, st>>>(B, n_reads, d_mh, d_read_off, d_seed_off, roff, cseeds, cchains, n_chains,
                                        d_nj, d_nb);
    if ((rc = bsb_cuda(ctx, cudaMemcpyAsync(nj.data(), d_nj, 4 * nr, cudaMemcpyDeviceToHost, st), "D2H SW jobs")) ||
        (rc = bsb_cuda(ctx, cudaMemcpyAsync(nbytes.data(), d_nb, 8 * nr, cudaMemcpyDeviceToHost, st), "D2H SW bytes")) ||
        (rc = bsb_cuda(ctx, cudaStreamSynchronize(st), "seed SW count")))
        return rc;
    joff[0] = boff[0] = 0;
    for (size_t r = 0; r < nr; ++r) joff[r + 1] = joff[r] + nj[r], boff[r + 1] = boff[r] + nbytes[r];
    const int64_t NJ = joff[nr], NB = boff[nr];
    std::vector<int> score((size_t)NJ + 1);
    if (NJ > 0) {
        const size_t need = head + al(sizeof(bsb_sw_job_t) * (size_t)NJ) + al((size_t)NB) + al(4 * (size_t)NJ);
        if ((rc = bsb_ensure(ctx, &ctx->flt_dev, &ctx->flt_dev_bytes, need + 256, "seed SW filter"))) return rc;
        D = (char *)ctx->flt_dev;        // (re)allocated: recompute the views
        d_mh = (int *)D;
        d_joff = (int64_t *)(D + 2 * al(4 * nr) + al(8 * nr)), d_boff = d_joff + al(8 * (nr + 1)) / 8;
        bsb_sw_job_t *d_jobs = (bsb_sw_job_t *)(D + head);
        uint8_t *d_bytes = (uint8_t *)(D + head + al(sizeof(bsb_sw_job_t) * (size_t)NJ));
        if ((rc = bsb_cuda(ctx, cudaMemcpyAsync(d_mh, h_min_hsp, 4 * nr, cudaMemcpyHostToDevice, st), "H2D min_hsp")) ||
            (rc = bsb_cuda(ctx, cudaMemcpyAsync(d_joff, joff.data(), 8 * (nr + 1), cudaMemcpyHostToDevice, st), "H2D")) ||
            (rc = bsb_cuda(ctx, cudaMemcpyAsync(d_boff, boff.data(), 8 * (nr + 1), cudaMemcpyHostToDevice, st), "H2D")))
            return rc;
        seed_sw_fill<<<grid, 128, 0, st>>>(B, n_reads, d_mh, d_reads, d_read_off, d_seed_off, roff, cseeds, cchains,
                                           n_chains, d_joff, d_boff, d_jobs, d_bytes);
        std::vector<bsb_sw_job_t> jobs((size_t)NJ);
        std::vector<uint8_t> bytes((size_t)NB + 1);
        std::vector<bsb_kswr_t> res((size_t)NJ);
        if ((rc = bsb_cuda(ctx, cudaMemcpyAsync(jobs.data(), d_jobs, sizeof(bsb_sw_job_t) * NJ, cudaMemcpyDeviceToHost,
                                                st), "D2H SW jobs")) ||
            (rc = bsb_cuda(ctx, cudaMemcpyAsync(bytes.data(), d_bytes, NB, cudaMemcpyDeviceToHost, st), "D2H SW bytes")) ||
            (rc = bsb_cuda(ctx, cudaStreamSynchronize(st), "seed SW jobs")))
            return rc;
        bsb_ext_param_t p;
        memset(&p, 0, sizeof p);
        memcpy(p.mat, o->mat, 25);
        p.o_del = o->o_del, p.e_del = o->e_del, p.o_ins = o->o_ins, p.e_ins = o->e_ins, p.zdrop = o->zdrop;
        if ((rc = bsb_align2_run(ctx, &p, jobs.data(), NJ, bytes.data(), NB, res.data(), &ctx->flt_in,
                                 &ctx->flt_in_bytes, &ctx->flt_out, &ctx->flt_out_bytes)))
            return rc;
        for (int64_t i = 0; i < NJ; ++i) score[(size_t)i] = res[(size_t)i].score;
    }
    int *d_score = (int *)(D + head + al(sizeof(bsb_sw_job_t) * (size_t)NJ) + al((size_t)NB));
    if (NJ > 0 &&
        (rc = bsb_cuda(ctx, cudaMemcpyAsync(d_score, score.data(), 4 * (size_t)NJ, cudaMemcpyHostToDevice, st), "H2D")))
        return rc;
    seed_sw_apply<<<grid, 128, 0, st>>>(ao, B, n_reads, d_mh, d_read_off, d_seed_off, roff, cseeds, cchains, n_chains,
                                        d_joff, d_score);
    if ((rc = bsb_cuda(ctx, cudaGetLastError(), "seed SW filter"))) return rc;
    // the host vectors above must outlive the copies that read them
    return bsb_cuda(ctx, cudaStreamSynchronize(st), "seed SW filter");
}

// Batches of fewer reads run their extensions inside chain2aln_kernel: it then has warps to spare,
// and the batches' some 20 launches would take longer.
constexpr int kPreReads = 4096;

// The extensions of every chain's first seed as two batches (pre_plan_kernel); chain_off receives the
// offsets of the reads' chains.  Leaves pre empty where the scoring or the reads' length need 32-bit
// cells.
static int first_extensions(bsb_ctx *ctx, const bsb_align_opt_t *o, const AlnOpt &ao, const DevBns &B,
                            const KswParams &P, int n_reads, int max_len, const uint8_t *d_reads,
                            const int64_t *d_read_off, const int64_t *d_seed_off, const int64_t *roff,
                            const DevSeed *cseeds, const DevChain *cchains, const int *n_chains, int64_t *chain_off,
                            int64_t *scan_tmp, PreResults *pre)
{
    cudaStream_t st = ctx->stream;
    int rc;
    for (int k = 0; k < 25; ++k)
        if (o->mat[k] > 63 || o->mat[k] < -63) return 0;
    if (!ksw_pack16(P) || o->w > 4096 || (int64_t)max_len * (o->a + P.mat_max) > ksw_pack16_max()) return 0;
    int64_t T = 0;
    if ((rc = bsb_cuda(ctx, scan_i32_i64(n_chains, n_reads, chain_off, scan_tmp, st), "chain offsets")) ||
        (rc = bsb_cuda(ctx, cudaMemcpyAsync(&T, chain_off + n_reads, 8, cudaMemcpyDeviceToHost, st), "chain total")) ||
        (rc = bsb_cuda(ctx, cudaStreamSynchronize(st), "chain total")))
        return rc;
    if (T == 0 || T > 0x7fffffff) return 0;
    size_t off = 0;
    const size_t o_pre = off; off += al(sizeof(PreChain) * T);
    const size_t o_left = off; off += al(sizeof(bsb_ext_job_t) * T);
    const size_t o_right = off; off += al(sizeof(bsb_ext_job_t) * T);
    const size_t o_out = off; off += al(sizeof(bsb_ext_out_t) * 2 * T);
    const size_t o_scr = off; off += al(ksw_scratch_bytes(T));
    if (bsb_ensure(ctx, &ctx->pre_buf, &ctx->pre_bytes, off, "chain extensions")) {
        cudaGetLastError();              // no room: chain2aln_kernel extends every seed itself
        return 0;
    }
    char *const D = (char *)ctx->pre_buf;
    PreChain *const pc = (PreChain *)(D + o_pre);
    bsb_ext_job_t *const left = (bsb_ext_job_t *)(D + o_left), *const right = (bsb_ext_job_t *)(D + o_right);
    bsb_ext_out_t *const out = (bsb_ext_out_t *)(D + o_out);
    const unsigned tb = (unsigned)((T + 127) / 128);
    pre_plan_kernel<<<tb, 128, 0, st>>>(ao, B, T, n_reads, chain_off, d_read_off, d_seed_off, roff, cseeds, cchains, pc,
                                        left, right);
    if ((rc = bsb_cuda(ctx, cudaMemsetAsync(out, 0x80, sizeof(bsb_ext_out_t) * 2 * T, st), "chain extensions"))) return rc;
    KswParams Q = P;
    Q.pac = B.pac, Q.l_pac = B.l_pac;
    const int builtin = ksw_builtin(T, ctx->n_sm, false);
    const uint8_t *const map = ksw_builtin_tile_map(builtin);
    uint64_t tiles = 0;
    for (int need = 1; need <= max_len + 1 && need < BSB_TILE_MAP_LEN; ++need) tiles |= 1ull << map[need];
    for (int side = 0; side < 2; ++side) {
        if (side) pre_right_kernel<<<tb, 128, 0, st>>>(ao, T, left, out, right);
        if ((rc = bsb_cuda(ctx, ksw_launch(Q, side ? right : left, T, 0, d_reads, nullptr, nullptr, builtin, tiles,
                                           out + side * T, nullptr, D + o_scr, ctx->n_sm, st, nullptr, nullptr, nullptr,
                                           nullptr, &ctx->ms, true), "chain extensions")))
            return rc;
    }
    pre->chains = pc, pre->off = chain_off, pre->left = out, pre->right = out + T;
    return 0;
}

static int bsb_align_regs_run(bsb_ctx *ctx, const bsb_align_opt_t *o, int n_reads, const uint8_t *d_reads,
                       const int64_t *d_read_off, const bsb_intv_t *d_seeds, const int64_t *d_seed_off,
                       int64_t n_seeds, int max_len, bool dedup, bsb_reg_t **d_regs_out, int64_t **d_reg_off_out,
                       int64_t *n_regs_total, const int *h_min_hsp)
{
    int rc;
    cudaStream_t st = ctx->stream;
    const int nb = ctx->n_sm * 4;
    // rows per seed interval and their offsets
    const int64_t scan_n = n_seeds > n_reads ? n_seeds : n_reads;
    size_t need = al(sizeof(int) * (n_seeds + 1)) + al(sizeof(int64_t) * (n_seeds + 1)) +
                  al(sizeof(int64_t) * scan_tmp_words(scan_n));
    if ((rc = bsb_ensure(ctx, &ctx->arena0, &ctx->arena0_bytes, need, "chain scratch (rows)"))) return rc;
    int *rcnt = (int *)ctx->arena0;
    int64_t *roff = (int64_t *)((char *)ctx->arena0 + al(sizeof(int) * (n_seeds + 1)));
    int64_t *scan_tmp = (int64_t *)((char *)roff + al(sizeof(int64_t) * (n_seeds + 1)));
    if (n_seeds > 0) {
        rows_count<<<nb, 256, 0, st>>>((const DevIntv *)d_seeds, n_seeds, o->max_occ, rcnt);
    }
    if ((rc = bsb_cuda(ctx, scan_i32_i64(rcnt, n_seeds, roff, scan_tmp, st), "row offsets"))) return rc;
    int64_t R = 0;
    if ((rc = bsb_cuda(ctx, cudaMemcpyAsync(&R, roff + n_seeds, 8, cudaMemcpyDeviceToHost, st), "row total"))) return rc;
    if ((rc = bsb_cuda(ctx, cudaStreamSynchronize(st), "row count"))) return rc;
    // per-row arrays (all sized by R)
    const size_t Rb = (size_t)(R > 0 ? R : 1);
    size_t off = 0;
    const size_t o_rows = off; off += al(8 * Rb);
    const size_t o_pos = off; off += al(8 * Rb);
    const size_t o_chains = off; off += al(sizeof(ChainRec) * Rb);
    const size_t o_nodes = off; off += al(sizeof(BtNode) * (Rb + 2));
    const size_t o_rowc = off; off += al(sizeof(int) * Rb);
    const size_t o_iwork = off; off += al(sizeof(int) * 3 * Rb);
    const size_t o_cseeds = off; off += al(sizeof(DevSeed) * Rb);
    const size_t o_cchains = off; off += al(sizeof(DevChain) * Rb);
    const size_t o_srt = off; off += al(8 * Rb);
    const size_t o_regs = off; off += al(sizeof(bsb_reg_t) * Rb);
    const size_t o_nch = off; off += al(sizeof(int) * (n_reads + 1));
    const size_t o_nreg = off; off += al(sizeof(int) * (n_reads + 1));
    const size_t o_ctrl = off; off += al(sizeof(int) * 4);
    const size_t o_regoff = off; off += al(sizeof(int64_t) * (n_reads + 1));
    const size_t o_out = off; off += al(sizeof(bsb_reg_t) * Rb);
    const size_t o_by_rows = off; off += al(sizeof(int) * (size_t)n_reads);
    const size_t o_order = off; off += al(sizeof(int) * (n_reads + 1)) + al(sizeof(int) * 2 * kOrderBins);
    const size_t o_dtmp = off; off += dedup ? al(sizeof(bsb_reg_t) * Rb) : 0;
    const size_t o_dn = off; off += dedup ? al(sizeof(int) * (n_reads + 1)) : 0;
    const size_t o_doff = off; off += dedup ? al(sizeof(int64_t) * (n_reads + 1)) : 0;
    if ((rc = bsb_ensure(ctx, &ctx->arena1, &ctx->arena1_bytes, off, "chain scratch"))) return rc;
    char *A = (char *)ctx->arena1;
    uint64_t *rows = (uint64_t *)(A + o_rows), *pos = (uint64_t *)(A + o_pos);
    ChainRec *chains = (ChainRec *)(A + o_chains);
    BtNode *nodes = (BtNode *)(A + o_nodes);
    int *row_chain = (int *)(A + o_rowc), *iwork = (int *)(A + o_iwork);
    DevSeed *cseeds = (DevSeed *)(A + o_cseeds);
    DevChain *cchains = (DevChain *)(A + o_cchains);
    uint64_t *srt = (uint64_t *)(A + o_srt);
    bsb_reg_t *regs = (bsb_reg_t *)(A + o_regs), *regs_out = (bsb_reg_t *)(A + o_out);
    int *n_chains = (int *)(A + o_nch), *n_regs = (int *)(A + o_nreg), *ctrl = (int *)(A + o_ctrl);
    int64_t *reg_off = (int64_t *)(A + o_regoff);
    if ((rc = bsb_cuda(ctx, cudaMemsetAsync(ctrl, 0, sizeof(int) * 4, st), "ctrl"))) return rc;
    if (n_seeds > 0 && R > 0) {
        rows_fill<<<nb, 256, 0, st>>>((const DevIntv *)d_seeds, n_seeds, o->max_occ, roff, rows);
        cudaError_t e = bsb_sa_launch_ctx(ctx, rows, R, pos);
        if (e != cudaSuccess) return bsb_cuda(ctx, e, "SA rows");
    }
    if ((rc = bsb_cuda(ctx, cudaEventRecord(ctx->stage_ev[2], st), "stage mark"))) return rc;
    AlnOpt ao;
    ao.a = o->a; ao.o_del = o->o_del; ao.e_del = o->e_del; ao.o_ins = o->o_ins; ao.e_ins = o->e_ins;
    ao.w = o->w; ao.zdrop = o->zdrop; ao.pen_clip5 = o->pen_clip5; ao.pen_clip3 = o->pen_clip3;
    ao.min_seed_len = o->min_seed_len; ao.max_occ = o->max_occ; ao.max_chain_gap = o->max_chain_gap;
    ao.min_chain_weight = o->min_chain_weight; ao.max_chain_extend = o->max_chain_extend;
    ao.mask_level = o->mask_level; ao.drop_ratio = o->drop_ratio;
    DevBns B;
    B.ann_offset = (const int64_t *)ctx->idx_ann_off;
    B.ann_len = (const int32_t *)ctx->idx_ann_len;
    B.n_seqs = ctx->n_seqs;
    B.l_pac = ctx->l_pac;
    B.pac = (const uint8_t *)ctx->idx_pac;
    KswParams P;
    memcpy(P.mat, o->mat, 25);
    P.o_del = o->o_del; P.e_del = o->e_del; P.o_ins = o->o_ins; P.e_ins = o->e_ins; P.zdrop = o->zdrop;
    int mx = 0;
    for (int i = 0; i < 25; ++i) mx = mx > o->mat[i] ? mx : o->mat[i];
    P.mat_max = mx;
    P.pack16 = 0;
    int *const left = (int *)(A + o_order);                  // reads for chain_kernel (the read order comes after)
    int *by_rows = nullptr;
    if (n_reads >= kRowOrderReads) {
        int *const cnt = (int *)(A + o_order + al(sizeof(int) * (n_reads + 1)));
        by_rows = (int *)(A + o_by_rows);
        const int ob = std::min((n_reads + kOrderThreads - 1) / kOrderThreads, ctx->n_sm * 4);
        if ((rc = bsb_cuda(ctx, cudaMemsetAsync(cnt, 0, sizeof(int) * 2 * kOrderBins, st), "read order"))) return rc;
        order_hist_rows<<<ob, kOrderThreads, 0, st>>>(d_seed_off, roff, n_reads, cnt);
        order_scatter_rows<<<ob, kOrderThreads, 0, st>>>(d_seed_off, roff, n_reads, cnt, cnt + kOrderBins, by_rows);
    }
    chain_warp_kernel<<<(n_reads + kChainWarps - 1) / kChainWarps, kChainWarps * 32, 0, st>>>(
        ao, B, n_reads, d_read_off, (const DevIntv *)d_seeds, d_seed_off, roff, pos, chains, nodes, row_chain, iwork,
        cseeds, cchains, n_chains, left, ctrl, by_rows);
    chain_kernel<<<ctx->n_sm * 4, 128, 0, st>>>(ao, B, left, ctrl, d_read_off, (const DevIntv *)d_seeds, d_seed_off, roff, pos,
                                            chains, nodes, row_chain, iwork, cseeds, cchains, n_chains);
    if (h_min_hsp &&
        (rc = seed_sw_filter(ctx, o, B, n_reads, h_min_hsp, d_reads, d_read_off, d_seed_off, roff, cseeds, cchains,
                             n_chains, ao)))
        return rc;
    if ((rc = bsb_cuda(ctx, cudaEventRecord(ctx->stage_ev[3], st), "stage mark"))) return rc;
    int *const order = (int *)(A + o_order);
    int *const n_list = ctrl + 2, *const ocnt = (int *)(A + o_order + al(sizeof(int) * (n_reads + 1)));
    const bool logging = ctx->read_log != 0;
    // per-read features / extension cells for the learned read order (kept for bsb_last_read_costs)
    float *d_feat = nullptr;
    int64_t *d_rcells = nullptr;
    int32_t *d_rkey = nullptr;
    const bool keyed = !ctx->order_keys.empty() && (int64_t)ctx->order_keys.size() == n_reads;
    if (!keyed) ctx->order_keys.clear();          // keys for another batch size are dropped
    const bool learned = ctx->read_model != nullptr && !keyed;
    if (learned || logging || keyed) {
        const size_t nr = (size_t)n_reads;
        if ((rc = bsb_ensure(ctx, &ctx->rc_buf, &ctx->rc_bytes, al(32 * nr) + al(8 * nr) + al(4 * nr) + 256,
                             "read costs")))
            return rc;
        d_feat = (float *)ctx->rc_buf;
        d_rcells = (int64_t *)((char *)ctx->rc_buf + al(32 * nr));
        d_rkey = (int32_t *)((char *)ctx->rc_buf + al(32 * nr) + al(8 * nr));
        const int fb = (int)std::min<int64_t>((n_reads + 127) / 128, (int64_t)ctx->n_sm * 8);
        if (learned || logging)
            read_features_kernel<<<fb, 128, 0, st>>>(ao, B, n_reads, d_reads, d_read_off, d_seed_off, roff, cseeds,
                                                     cchains, n_chains, d_feat);
        ctx->rc_n = logging ? n_reads : 0;
    }
    const int32_t *key = nullptr;
    if (keyed) {             // the caller's keys, once (the copy is done before they are cleared)
        if ((rc = bsb_cuda(ctx, cudaMemcpyAsync(d_rkey, ctx->order_keys.data(), sizeof(int32_t) * (size_t)n_reads,
                                                cudaMemcpyHostToDevice, st), "read order keys")) ||
            (rc = bsb_cuda(ctx, cudaStreamSynchronize(st), "read order keys")))
            return rc;
        ctx->order_keys.clear();
        key = d_rkey;
    } else if (learned) {    // predicted cells of every read
        if ((rc = bsb_mlp_forward(ctx, (const bsb_mlp_weights_t *)ctx->read_model, d_feat, n_reads, nullptr, d_rkey)))
            return rc;
        key = d_rkey;
    }
    if ((rc = bsb_cuda(ctx, cudaMemsetAsync(ocnt, 0, sizeof(int) * 2 * kOrderBins, st), "read order"))) return rc;
    PreResults pre{};
    if (!logging && n_reads >= kPreReads &&
        (rc = first_extensions(ctx, o, ao, B, P, n_reads, max_len, d_reads, d_read_off, d_seed_off, roff, cseeds, cchains,
                               n_chains, reg_off, scan_tmp, &pre)))
        return rc;
    const int ob = std::min((n_reads + kOrderThreads - 1) / kOrderThreads, ctx->n_sm * 4);
    if (pre.chains) {           // the reads that need no other extension than their chains' first
        const int pb = std::min((n_reads + kPlainWarps - 1) / kPlainWarps, ctx->n_sm * 8);
        chain2aln_plain<<<pb, kPlainWarps * 32, 0, st>>>(ao, n_reads, d_read_off, d_seed_off, roff, cseeds, cchains,
                                                         n_chains, regs, n_regs, pre, key, ocnt);
    } else {
        order_hist<<<ob, kOrderThreads, 0, st>>>(key, n_chains, n_reads, ocnt);
    }
    order_scatter<<<ob, kOrderThreads, 0, st>>>(key, n_chains, pre.chains ? n_regs : nullptr, n_reads, ocnt,
                                                ocnt + kOrderBins, order, n_list);
    ctx->queue_reads = order, ctx->queue_count = n_list;
    int64_t *const rcells_out = logging ? d_rcells : nullptr;
    // every extension of these reads fits (max_len + 1) columns: the narrowest variant that holds them
    if (max_len <= 127)
        chain2aln_kernel<4><<<ctx->n_sm * 8, 128, 0, st>>>(ao, P, B, d_reads, d_read_off, d_seed_off, roff,
                                                            cseeds, cchains, n_chains, srt, regs, n_regs, ctrl + 1, order, n_list, rcells_out, pre);
    else if (max_len <= 159)
        chain2aln_kernel<5><<<ctx->n_sm * 8, 128, 0, st>>>(ao, P, B, d_reads, d_read_off, d_seed_off, roff,
                                                            cseeds, cchains, n_chains, srt, regs, n_regs, ctrl + 1, order, n_list, rcells_out, pre);
    else if (max_len <= 255)
        chain2aln_kernel<8><<<ctx->n_sm * 8, 128, 0, st>>>(ao, P, B, d_reads, d_read_off, d_seed_off, roff,
                                                            cseeds, cchains, n_chains, srt, regs, n_regs, ctrl + 1, order, n_list, rcells_out, pre);
    else if (max_len <= 511)
        chain2aln_kernel<16><<<ctx->n_sm * 4, 128, 0, st>>>(ao, P, B, d_reads, d_read_off, d_seed_off, roff,
                                                             cseeds, cchains, n_chains, srt, regs, n_regs, ctrl + 1, order, n_list, rcells_out, pre);
    else
        chain2aln_kernel<32><<<ctx->n_sm * 2, 128, 0, st>>>(ao, P, B, d_reads, d_read_off, d_seed_off, roff,
                                                             cseeds, cchains, n_chains, srt, regs, n_regs, ctrl + 1, order, n_list, rcells_out, pre);
    if ((rc = bsb_cuda(ctx, cudaEventRecord(ctx->stage_ev[4], st), "stage mark")) ||
        (rc = bsb_cuda(ctx, scan_i32_i64(n_regs, n_reads, reg_off, scan_tmp, st), "region offsets")))
        return rc;
    const int cgrid = (int)((n_reads + 3) / 4) < ctx->n_sm * 16 ? (int)((n_reads + 3) / 4) : ctx->n_sm * 16;
    compact_regs<<<cgrid, 128, 0, st>>>(regs, d_seed_off, roff, n_reads, n_regs, reg_off, regs_out);
    if (dedup) {
        // mem_sort_dedup_patch: regs_out (pre-dedup, at reg_off) -> regs (kept, at reg_off,
        // n_kept per read) -> regs_out again, compacted at the new offsets
        DedupOpt D;
        D.w = o->w, D.max_chain_gap = o->max_chain_gap, D.mask_level_redun = o->mask_level_redun;
        D.pen = GlobalPen{o->o_del, o->e_del, o->o_ins, o->e_ins};
        memcpy(D.mat, o->mat, 25);
        bsb_reg_t *dtmp = (bsb_reg_t *)(A + o_dtmp);
        int *n_kept = (int *)(A + o_dn);
        int64_t *kept_off = (int64_t *)(A + o_doff);
        const int db = (int)((n_reads + kDedupWarps - 1) / kDedupWarps);
        dedup_kernel<<<db, kDedupWarps * 32, kDedupWarps * dedup_warp_bytes(max_len), st>>>(
            D, B, n_reads, d_reads, d_read_off, reg_off, regs_out, dtmp, iwork, regs, n_kept, max_len);
        if ((rc = bsb_cuda(ctx, scan_i32_i64(n_kept, n_reads, kept_off, scan_tmp, st), "kept offsets"))) return rc;
        compact_kept<<<cgrid, 128, 0, st>>>(regs, reg_off, n_reads, n_kept, kept_off, regs_out);
        reg_off = kept_off;
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return bsb_cuda(ctx, e, "chain/extension launch");
    if ((rc = bsb_cuda(ctx, cudaEventRecord(ctx->stage_ev[5], st), "stage mark")) ||
        (rc = bsb_cuda(ctx, cudaMemcpyAsync(n_regs_total, reg_off + n_reads, 8, cudaMemcpyDeviceToHost, st), "reg total")))
        return rc;
    if ((rc = bsb_cuda(ctx, cudaStreamSynchronize(st), "chain/extension"))) return rc;
    *d_regs_out = regs_out;
    *d_reg_off_out = reg_off;
    return 0;
}

static int align_batch(bsb_ctx *ctx, const bsb_align_opt_t *o, int32_t n_reads, const uint8_t *seqs,
                       const int64_t *offs, bsb_reg_t *regs, int64_t max_regs, int64_t *regs_off, bool dedup)
{
    if (!ctx) return BSB_EINVAL;
    if (!ctx->has_index || !ctx->idx_pac || !ctx->idx_ann_off)
        return bsb_fail(ctx, BSB_ENOINDEX, "no index with pac and contig table loaded");
    if (!o || !offs || n_reads < 0 || (n_reads > 0 && (!seqs || !regs || !regs_off)))
        return bsb_fail(ctx, BSB_EINVAL, "NULL argument");
    if (o->e_del < 1 || o->e_ins < 1 || o->o_del < 0 || o->o_ins < 0 || o->a < 1 || o->w < 0 || o->max_occ < 1 ||
        o->min_seed_len < 1 || o->max_chain_extend < 1)
        return bsb_fail(ctx, BSB_EINVAL, "unsupported options");
    if (n_reads == 0) {
        regs_off[0] = 0;
        return 0;
    }
    int max_len = 0;
    // mem_flt_chained_seeds (bwamem.c:602-606): per read length, its min_HSP_score when the
    // seed-level SW filter runs for that length, else -1 (the reference returns early)
    int hsp_of_len[BSB_ALIGN_MAX_LEN + 1];
    for (int l = 0; l <= BSB_ALIGN_MAX_LEN; ++l) {
        const double min_l = o->min_chain_weight ? 1.1f * o->min_chain_weight : 5.5f * log((double)l);
        hsp_of_len[l] = l > 0 && !(min_l > 0.05f * l) ? (int)(o->a * min_l + .499) : -1;
    }
    std::vector<int> min_hsp((size_t)n_reads);
    bool any_filter = false;
    for (int r = 0; r < n_reads; ++r) {
        const int64_t l = offs[r + 1] - offs[r];
        if (l < 0) return bsb_fail(ctx, BSB_EINVAL, "read %d: negative length", r);
        if (l > BSB_ALIGN_MAX_LEN) return bsb_fail(ctx, BSB_ETOOLONG, "read %d: length %lld > %d", r, (long long)l, BSB_ALIGN_MAX_LEN);
        min_hsp[(size_t)r] = hsp_of_len[l];
        any_filter |= hsp_of_len[l] >= 0;
        if (l > max_len) max_len = (int)l;
    }
    const int64_t total = offs[n_reads] - offs[0];
    int rc;
    if ((rc = bsb_cuda(ctx, cudaSetDevice(ctx->device), "cudaSetDevice"))) return rc;
    const size_t off_b = sizeof(int64_t) * ((size_t)n_reads + 1);
    const size_t seq_b = al((size_t)total);
    if ((rc = bsb_ensure(ctx, &ctx->d_in, &ctx->d_in_bytes, seq_b + 2 * al(off_b) + 256, "align input staging")))
        return rc;
    uint8_t *d_reads = (uint8_t *)ctx->d_in;
    int64_t *d_offs = (int64_t *)((char *)ctx->d_in + seq_b);
    int64_t *d_seed_off = (int64_t *)((char *)d_offs + al(off_b));
    std::vector<int64_t> rel(n_reads + 1);
    for (int r = 0; r <= n_reads; ++r) rel[r] = offs[r] - offs[0];
    ctx->stage_valid = false;
    ctx->queue_reads = ctx->queue_count = nullptr;
    cudaEvent_t *const sev = ctx->stage_ev;
    if ((rc = bsb_cuda(ctx, cudaEventRecord(sev[0], ctx->stream), "stage mark")) ||
        (rc = bsb_cuda(ctx, cudaMemcpyAsync(d_reads, seqs + offs[0], total, cudaMemcpyHostToDevice, ctx->stream), "H2D reads")))
        return rc;
    if ((rc = bsb_cuda(ctx, cudaMemcpyAsync(d_offs, rel.data(), off_b, cudaMemcpyHostToDevice, ctx->stream), "H2D offsets")))
        return rc;
    bsb_seed_opt_t so;
    so.min_seed_len = o->min_seed_len; so.split_factor = o->split_factor;
    so.split_width = o->split_width; so.max_mem_intv = o->max_mem_intv;
    // a read whose passes 1-2 overflow its seed slots: seeding again with twice the slots
    bsb_intv_t *d_seeds = nullptr;
    int64_t n_seeds = 0;
    for (int mult = 1;; mult *= 2) {
        const size_t seeds_b = al(seed_padded_entries(total, n_reads, mult) * sizeof(bsb_intv_t));
        if ((rc = bsb_ensure(ctx, &ctx->d_out, &ctx->d_out_bytes, seeds_b + 256, "align seed buffer"))) return rc;
        d_seeds = (bsb_intv_t *)ctx->d_out;
        if ((rc = bsb_seed_batch_device_m(ctx, &so, n_reads, d_reads, d_offs, total, max_len, d_seeds, d_seed_off,
                                          mult)) ||
            (rc = bsb_cuda(ctx, cudaEventRecord(sev[1], ctx->stream), "stage mark")))
            return rc;
        int ctrl[2] = {0, 0};
        if ((rc = bsb_cuda(ctx, cudaMemcpyAsync(&n_seeds, d_seed_off + n_reads, 8, cudaMemcpyDeviceToHost, ctx->stream),
                           "seed total")) ||
            (rc = bsb_cuda(ctx, cudaMemcpyAsync(ctrl, ctx->seed_ctrl, sizeof ctrl, cudaMemcpyDeviceToHost, ctx->stream),
                           "seed ctrl")) ||
            (rc = bsb_cuda(ctx, cudaStreamSynchronize(ctx->stream), "seeding")))
            return rc;
        if (!ctrl[1]) break;
        if (mult >= kSeedSlotMultMax)
            return bsb_fail(ctx, BSB_ETOOLONG, "read %d produced more seeds than %d times its buffer holds",
                            ctrl[1] - 1, mult);
        ++ctx->seed_regrown;
    }
    bsb_reg_t *d_regs = nullptr;
    int64_t *d_reg_off = nullptr, n_regs = 0;
    if ((rc = bsb_align_regs_run(ctx, o, n_reads, d_reads, d_offs, d_seeds, d_seed_off, n_seeds, max_len, dedup, &d_regs,
                                 &d_reg_off, &n_regs, any_filter ? min_hsp.data() : nullptr)))
        return rc;
    if ((rc = bsb_cuda(ctx, cudaMemcpyAsync(regs_off, d_reg_off, off_b, cudaMemcpyDeviceToHost, ctx->stream), "D2H offsets")))
        return rc;
    if (n_regs > max_regs) {
        // the offsets still go back: regs_off[n_reads] tells the caller the size to call again with
        if ((rc = bsb_cuda(ctx, cudaStreamSynchronize(ctx->stream), "align batch"))) return rc;
        return bsb_fail(ctx, BSB_ECAPACITY, "%lld regions do not fit max_regs %lld", (long long)n_regs,
                        (long long)max_regs);
    }
    if (n_regs > 0 &&
        (rc = bsb_cuda(ctx, cudaMemcpyAsync(regs, d_regs, sizeof(bsb_reg_t) * n_regs, cudaMemcpyDeviceToHost, ctx->stream),
                       "D2H regions")))
        return rc;
    if ((rc = bsb_cuda(ctx, cudaEventRecord(sev[BSB_ALIGN_STAGES], ctx->stream), "stage mark")) ||
        (rc = bsb_cuda(ctx, cudaStreamSynchronize(ctx->stream), "align batch")))
        return rc;
    ctx->stage_valid = true;
    return 0;
}

extern "C" int bsb_align_regs_batch(bsb_ctx *ctx, const bsb_align_opt_t *o, int32_t n_reads, const uint8_t *seqs,
                                    const int64_t *offs, bsb_reg_t *regs, int64_t max_regs, int64_t *regs_off)
{
    return align_batch(ctx, o, n_reads, seqs, offs, regs, max_regs, regs_off, false);
}

extern "C" int bsb_mem_align1_batch(bsb_ctx *ctx, const bsb_align_opt_t *o, int32_t n_reads, const uint8_t *seqs,
                                    const int64_t *offs, bsb_reg_t *regs, int64_t max_regs, int64_t *regs_off)
{
    if (!ctx) return BSB_EINVAL;
    if (o && !(o->mask_level_redun >= 0.f && o->mask_level_redun <= 1.f))
        return bsb_fail(ctx, BSB_EINVAL, "mask_level_redun must lie in [0, 1]");
    return align_batch(ctx, o, n_reads, seqs, offs, regs, max_regs, regs_off, true);
}

extern "C" int bsb_last_stage_ms(const bsb_ctx *ctx, float *ms, int n)
{
    if (!ctx || !ms || n < 0 || !ctx->stage_valid) return BSB_EINVAL;
    for (int k = 0; k < BSB_ALIGN_STAGES && k < n; ++k)
        if (cudaEventElapsedTime(&ms[k], ctx->stage_ev[k], ctx->stage_ev[k + 1]) != cudaSuccess) return BSB_ECUDA;
    return 0;
}

extern "C" int bsb_read_cost_log(bsb_ctx *ctx, int enable)
{
    if (!ctx) return BSB_EINVAL;
    ctx->read_log = enable != 0;
    ctx->rc_n = 0;
    return 0;
}

extern "C" int bsb_last_read_costs(bsb_ctx *ctx, int32_t n_reads, float *feat, int64_t *cells)
{
    if (!ctx) return BSB_EINVAL;
    if (!ctx->read_log || ctx->rc_n == 0) return bsb_fail(ctx, BSB_EINVAL, "no logged batch (bsb_read_cost_log)");
    if (n_reads != ctx->rc_n) return bsb_fail(ctx, BSB_EINVAL, "the logged batch has %d reads, not %d", ctx->rc_n, n_reads);
    int rc;
    if ((rc = bsb_cuda(ctx, cudaSetDevice(ctx->device), "cudaSetDevice"))) return rc;
    const size_t nr = (size_t)n_reads;
    const char *b = (const char *)ctx->rc_buf;
    if (feat && (rc = bsb_cuda(ctx, cudaMemcpyAsync(feat, b, 32 * nr, cudaMemcpyDeviceToHost, ctx->stream), "D2H")))
        return rc;
    if (cells && (rc = bsb_cuda(ctx, cudaMemcpyAsync(cells, b + al(32 * nr), 8 * nr, cudaMemcpyDeviceToHost,
                                                     ctx->stream), "D2H")))
        return rc;
    return bsb_cuda(ctx, cudaStreamSynchronize(ctx->stream), "read costs");
}

extern "C" int bsb_last_read_order(bsb_ctx *ctx, int32_t *reads, int32_t max, int32_t *n)
{
    if (!ctx) return BSB_EINVAL;
    if (!n || max < 0 || (max > 0 && !reads)) return bsb_fail(ctx, BSB_EINVAL, "read order: NULL or negative count");
    if (!ctx->queue_reads) return bsb_fail(ctx, BSB_EINVAL, "no alignment batch on this context");
    int rc;
    if ((rc = bsb_cuda(ctx, cudaSetDevice(ctx->device), "cudaSetDevice")) ||
        (rc = bsb_cuda(ctx, cudaMemcpyAsync(n, ctx->queue_count, sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream),
                       "read order")) ||
        (rc = bsb_cuda(ctx, cudaStreamSynchronize(ctx->stream), "read order")))
        return rc;
    const size_t got = std::min(*n, max);
    if (got && ((rc = bsb_cuda(ctx, cudaMemcpyAsync(reads, ctx->queue_reads, sizeof(int32_t) * got, cudaMemcpyDeviceToHost,
                                                    ctx->stream), "read order")) ||
                (rc = bsb_cuda(ctx, cudaStreamSynchronize(ctx->stream), "read order"))))
        return rc;
    return 0;
}

extern "C" int bsb_set_read_cost_model(bsb_ctx *ctx, const bsb_mlp_weights_t *d_w)
{
    if (!ctx) return BSB_EINVAL;
    ctx->read_model = d_w;
    return 0;
}

extern "C" int bsb_set_read_order_keys(bsb_ctx *ctx, const int32_t *keys, int32_t n)
{
    if (!ctx) return BSB_EINVAL;
    if (n < 0 || (n > 0 && !keys)) return bsb_fail(ctx, BSB_EINVAL, "read order keys: NULL or negative count");
    ctx->order_keys.assign(keys, keys + (n > 0 ? n : 0));
    return 0;
}
