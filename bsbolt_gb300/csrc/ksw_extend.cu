// ksw_extend.cu -- batched ksw_extend2 for sm_103a: the scheduler.
//
// Bit-exact restatement of the reference banded extension
// (bsbolt/External/BWA/ksw.c:380-479).  The DP itself is ksw_group.cuh: a
// group of G lanes runs one job row by row, 32/G jobs per warp.
//
// Why row-parallel and not an anti-diagonal wavefront: the reference decides
// each row's band [beg,end) from the complete previous row (the shrink to
// non-zero cells, ksw.c:466-469), stops on a zero row (ksw.c:454) and tests
// z-drop per target row (ksw.c:458-464).  A wavefront would have to run rows
// whose band is not known yet.  Instead a group computes a whole row at once:
//   * lane L of the group owns query columns [L*C, L*C+C) in registers;
//   * M and E depend only on the previous row and are computed per cell;
//   * F(i,j+1) = max(F(i,j) - e_ins, max(M(i,j) - oe_ins, 0)) is a max-plus
//     recurrence along the row: each lane runs it over its own columns, and
//     a group scan of the lane maps x -> max(x - e_ins*C, F_lane) supplies
//     every lane's carry-in (one __shfl_up_sync ladder per row);
//   * the row maximum, its last column, and the first/last non-zero cell of
//     the shrink are group reductions.
// The register file holds the reference's whole eh[] array, including cells
// outside the current band: the band may grow back over them and read stale
// values, exactly as the reference does.
//
// Scheduling (the plain schedule): each job gets the tile shape the tile map
// assigns to its query length (ksw_tiles.cuh), and within a shape jobs are
// issued longest-bound-first (qlen x min(tlen, qlen+w), or a caller supplied
// cost key); each shape runs as a persistent kernel whose groups pull jobs
// from a device counter.  Shapes with an even C run their jobs on 16-bit cells,
// two per register (ksw_group16.cuh); a job whose scores could leave 16 bits
// (h0 + qlen * max(mat) > kPack16MaxH) is binned last in its shape and runs on
// the 32-bit kernel.  Results never depend on the shape, the cell width or the
// order.  Long queries with a narrow band run on registers that move along with the band
// (ksw_ring16.cu) where the scheduler's own maps are in use; so do, in large batches, jobs whose band can be cut
// (cut_band, ksw_core.cuh).

#include <climits>
#include <cstdio>

#include "ksw_group16.cuh"
#include "ksw_tiles.cuh"

__constant__ KswTileMap c_tile_maps[kBuiltinMaps] = {kBuiltinTileMaps[0], kBuiltinTileMaps[1], kBuiltinTileMaps[2],
                                                     kBuiltinTileMaps[3], kBuiltinTileMaps[4]};

namespace {

constexpr int kClasses = 128;           // cost classes within a tile shape; the last one holds the
                                        // jobs that need 32-bit cells
constexpr int kWideClass = kClasses - 1;

__device__ __forceinline__ int cost_class(uint32_t key)
{
    // 4 classes per power of two; class 0 = cheapest
    if (key == 0) return 0;
    const int msb = 31 - __clz(key);
    const int frac = msb >= 2 ? (int)((key >> (msb - 2)) & 3) : (int)((key << (2 - msb)) & 3);
    const int c = msb * 4 + frac;
    return c < kWideClass ? c : kWideClass - 1;
}

// Shapes with a 16-bit kernel (tile_has_pack16), as a bit set.
constexpr uint64_t pack16_tiles()
{
    uint64_t m = 0;
    for (int t = 0; t < kNumTiles; ++t)
        if (tile_has_pack16(kTileList[t].C)) m |= 1ull << t;
    return m;
}
constexpr uint64_t kPack16Tiles = pack16_tiles();

// Histogram of (tile, class) keys.  Tiles are major; within a tile, classes
// are laid out most expensive first so an ascending scan issues longest-first.
// A job that fails the preconditions (the host entry checks them; the device
// entry cannot) gets the reject key kRejectKey: it is counted, never issued,
// and its output is left untouched.
constexpr int kRejectKey = kNumTiles * kClasses;
constexpr int kHistSlots = kNumTiles * kClasses + 1;
constexpr int kScanThreads = 1024;

// A job as ksw_diagonal reads it.
template <bool Packed>
struct JobAcc {
    const KswParams &P;
    JobText<Packed> qs, ts;
    __device__ __forceinline__ int q(int j) const { return qs.byte(j); }
    __device__ __forceinline__ int t(int i) const { return (int)ts.base(P, i); }
};

// A job's band as ksw.c:399-407 cuts it.
__device__ __forceinline__ int clamped_band(const KswParams &P, const bsb_ext_job_t &j)
{
    const int mi = band_cap(j.qlen * P.mat_max + j.end_bonus - P.o_ins, P.e_ins);
    const int md = band_cap(j.qlen * P.mat_max + j.end_bonus - P.o_del, P.e_del);
    return min(min(j.w, max(mi, 1)), max(md, 1));
}

// Keys and their histogram; and, unless cells are counted, the jobs whose result the main
// diagonal decides (ksw_diagonal): these are answered here, get the key kDoneKey and are never
// issued.  A warp takes `per` jobs at a time: a lane each for the checks and the key, then four
// diagonals at once, eight lanes each (2M jobs of 10-140 bases: 0.38 ms, 26 us without the
// diagonals; one diagonal after the other by the whole warp 0.52 ms; 64 jobs 9 against 46 us).
// Half of those jobs end here: with the rows left out (ksw_core.cuh) the batch takes 7.9 ms
// instead of 23.4, and 6.8 with the others' bands cut (ksw_tiles.cuh).
constexpr int32_t kDoneKey = -1;
constexpr int kHistThreads = 256;
template <bool Packed>
__global__ void __launch_bounds__(kHistThreads)
ksw_sched_hist(KswParams P, const bsb_ext_job_t *__restrict__ jobs, int n, long long seq_bytes,
               const uint8_t *__restrict__ seq, const int32_t *__restrict__ cost, const uint8_t *__restrict__ map,
               int builtin, int ring, int diagonals, int cuts, int per, bsb_ext_out_t *__restrict__ out, int *__restrict__ hist,
               int32_t *__restrict__ key_out)
{
    __shared__ int sh[kHistSlots];
    __shared__ int8_t tab[kScoreTable];
    for (int i = threadIdx.x; i < kHistSlots; i += blockDim.x) sh[i] = 0;
    load_score_table(P, tab);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int warps = (int)(gridDim.x * blockDim.x) >> 5;
    const bool plain = tab[0] == P.mat_max && tab[9] == P.mat_max && tab[18] == P.mat_max && tab[27] == P.mat_max;
    for (long long i0 = (long long)((int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per; i0 < n;
         i0 += (long long)warps * per) {
        const int i = (int)(i0 + lane);
        const bool in = lane < per && i0 + lane < n;
        bsb_ext_job_t jb;
        jb.qoff = jb.toff = 0, jb.qlen = jb.tlen = jb.h0 = jb.w = jb.end_bonus = jb.flags = 0;
        if (in) jb = jobs[i];
        const bool ok = in && jb.qlen >= 0 && jb.qlen < kMaxNeed && jb.tlen >= 0 && jb.w >= 0 && jb.h0 > 0 &&
                        jb.h0 <= (1 << 20) &&
                        (Packed ? !(jb.flags & kExtNone)
                                : jb.flags == 0 && span_inside(jb.qoff, jb.qlen, seq_bytes) &&
                                      span_inside(jb.toff, jb.tlen, seq_bytes));
        int key;
        if (!ok) {
            key = kRejectKey;
        } else {
            const int need = jb.qlen + 1;
            const int t = !Packed && ring && ksw_ring_fits(P, jb, ring_of(builtin)) ? kRingTile
                          : map ? map[need] : c_tile_maps[builtin].tile[need];
            uint32_t k;
            if (cost) k = (uint32_t)max(cost[i], 0);
            else {
                const long long span = min((long long)jb.tlen, (long long)jb.qlen + jb.w);
                const long long c = (long long)jb.qlen * max(span, 0LL);
                k = (uint32_t)min(c, (long long)0x7fffffff);
            }
            const bool wide = P.pack16 && (kPack16Tiles >> t & 1) &&
                              (long long)jb.h0 + (long long)jb.qlen * P.mat_max > kPack16MaxH;
            key = t >= kNumTiles ? kRejectKey
                  : wide         ? t * kClasses + kWideClass
                                 : t * kClasses + (kWideClass - 1 - cost_class(k));
        }
        if (diagonals) {
            const int lim = key != kRejectKey && in ? diagonal_limit(P, jb.h0) : 0;
            // the widest ring a job's query pays for, and how far its diagonal is followed for that
            int cut = -1, band = 0, far = lim;
            if (!Packed && cuts && lim > 0 && key % kClasses != kWideClass) {
                band = clamped_band(P, jb);
#pragma unroll
                for (int c = 0; c < kCutRings; ++c)
                    if (cuts >> c & 1 && jb.qlen + 1 >= cut_from(c, builtin) && band > cut_width(c)) cut = c;
                if (jb.qlen + 32 >= 1024) cut = -1;
                if (cut >= 0)
                    far = max(lim, min(P.o_del + P.e_del * (cut_width(cut) + 1), P.o_ins + P.e_ins * (cut_width(cut) + 1)));
            }
            const JobText<Packed> qt = job_query<Packed>(seq, jb), tt = job_target<Packed>(seq, jb);
            for (int r = 0; r < per; r += 4) {
                const int b = r + (lane >> 3);
                JobAcc<Packed> acc{P, qt, tt};
                if constexpr (Packed) {
                    acc.qs.at = __shfl_sync(BSB_FULL_MASK, qt.at, b), acc.ts.at = __shfl_sync(BSB_FULL_MASK, tt.at, b);
                    acc.qs.back = acc.ts.back = __shfl_sync(BSB_FULL_MASK, qt.back, b);
                } else {
                    acc.qs.p = (const uint8_t *)__shfl_sync(BSB_FULL_MASK, (unsigned long long)qt.p, b);
                    acc.ts.p = (const uint8_t *)__shfl_sync(BSB_FULL_MASK, (unsigned long long)tt.p, b);
                }
                const int qlen = __shfl_sync(BSB_FULL_MASK, jb.qlen, b), tlen = __shfl_sync(BSB_FULL_MASK, jb.tlen, b);
                const int h0 = __shfl_sync(BSB_FULL_MASK, jb.h0, b), lm = __shfl_sync(BSB_FULL_MASK, lim, b);
                int best, best_j, last;
                bool known;
                int cls = 0;
                if constexpr (Packed) {
                    known = ksw_diagonal<8>(tab, P.mat_max, lm, qlen, tlen, h0, acc, lane, best, best_j, last);
                } else {
                    const int fr = __shfl_sync(BSB_FULL_MASK, far, b), most = __shfl_sync(BSB_FULL_MASK, cut, b);
                    int loss, lowest;
                    const bool followed = ksw_diagonal_words(tab, P.mat_max, plain, fr, qlen, tlen, h0, acc.qs.p, acc.ts.p,
                                                             seq, seq + seq_bytes, lane, best, best_j, last, loss, lowest);
                    known = followed && loss < lm;
                    if (followed && !known && most >= 0) {
                        const int D = cut_band(P, loss, lowest);
                        if (D >= 0) {
#pragma unroll
                            for (int c = kCutRings - 1; c >= 0; --c)
                                if (c <= most && cuts >> c & 1 && D <= cut_width(c)) cls = c + 1;
                        }
                    }
                }
                if (known && (lane & 7) == 0) {
                    bsb_ext_out_t o;
                    o.score = best; o.qle = o.tle = best_j + 1;
                    o.gtle = qlen; o.gscore = last; o.max_off = 0;
                    out[i0 + b] = o;
                }
                if constexpr (!Packed) {
                    const unsigned c0 = __ballot_sync(BSB_FULL_MASK, cls & 1), c1 = __ballot_sync(BSB_FULL_MASK, cls & 2);
                    if (lane >= r && lane < r + 4) {
                        const int c = (int)(c0 >> ((lane - r) * 8) & 1u) | (int)(c1 >> ((lane - r) * 8) & 1u) << 1;
                        if (c) key = cut_tile(c - 1) * kClasses + key % kClasses;
                    }
                }
                const unsigned done = __ballot_sync(BSB_FULL_MASK, known);
                if (lane >= r && lane < r + 4 && (done >> ((lane - r) * 8) & 1)) key = kDoneKey;
            }
        }
        if (in) {
            key_out[i] = key;
            if (key != kDoneKey) atomicAdd(&sh[key], 1);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kHistSlots; i += blockDim.x)
        if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// Exclusive scan of the histogram (one block: a contiguous chunk per thread,
// then a scan of the chunk totals) -> cursors and, per tile t, the ranges of its
// launches: ranges[6t ..] = {start, wide start | wide start, end | start, end}
// (the 16-bit kernel, the 32-bit kernel for the wide class, or one 32-bit kernel
// for the whole tile).  rejected[0] counts the rejected jobs.
constexpr int kRangeInts = 6;
__global__ void __launch_bounds__(kScanThreads)
ksw_sched_scan(const int *__restrict__ hist, int *__restrict__ cursor, int32_t *__restrict__ ranges,
               int *__restrict__ rejected)
{
    constexpr int kChunk = (kHistSlots + kScanThreads - 1) / kScanThreads;
    __shared__ int tot[kScanThreads];
    const int t = threadIdx.x, lo = t * kChunk;
    int v[kChunk];
    int s = 0;
#pragma unroll
    for (int k = 0; k < kChunk; ++k) {
        v[k] = lo + k < kHistSlots ? hist[lo + k] : 0;
        s += v[k];
    }
    tot[t] = s;
    __syncthreads();
    for (int d = 1; d < kScanThreads; d <<= 1) {      // inclusive Hillis-Steele scan of the totals
        const int add = t >= d ? tot[t - d] : 0;
        __syncthreads();
        tot[t] += add;
        __syncthreads();
    }
    int acc = t ? tot[t - 1] : 0;
#pragma unroll
    for (int k = 0; k < kChunk; ++k) {
        const int i = lo + k;
        if (i < kHistSlots) {
            cursor[i] = acc;
            const int tile = i / kClasses, cls = i % kClasses;
            if (cls == 0) {
                if (tile < kNumTiles) ranges[kRangeInts * tile] = ranges[kRangeInts * tile + 4] = acc;
                if (tile > 0) ranges[kRangeInts * (tile - 1) + 3] = ranges[kRangeInts * (tile - 1) + 5] = acc;
            }
            if (cls == kWideClass && tile < kNumTiles)
                ranges[kRangeInts * tile + 1] = ranges[kRangeInts * tile + 2] = acc;
            if (i == kRejectKey) rejected[0] = tot[kScanThreads - 1] - acc;
        }
        acc += v[k];
    }
}

__global__ void ksw_sched_scatter(const int32_t *__restrict__ key, int n, int *__restrict__ cursor,
                                  int32_t *__restrict__ order)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int k = key[i];
        if (k == kDoneKey) continue;
        order[atomicAdd(&cursor[k], 1)] = i;
    }
}

// The same for large batches: a block counts its tile's keys in shared memory and takes each key's places
// with one atomic, in place of one global atomic per job on a few hundred busy counters (the 500k
// extensions of an RRBS batch: 97 -> 9 us).
constexpr int kScatterThreads = 512, kScatterItems = 8, kScatterTile = kScatterThreads * kScatterItems;
__global__ void __launch_bounds__(kScatterThreads)
ksw_sched_scatter_tiles(const int32_t *__restrict__ key, int n, int *__restrict__ cursor, int32_t *__restrict__ order)
{
    __shared__ int sh[kHistSlots];
    for (int i = threadIdx.x; i < kHistSlots; i += kScatterThreads) sh[i] = 0;
    __syncthreads();
    const long long base = (long long)blockIdx.x * kScatterTile;
    int k[kScatterItems], at[kScatterItems];
#pragma unroll
    for (int u = 0; u < kScatterItems; ++u) {
        const long long i = base + u * kScatterThreads + threadIdx.x;
        k[u] = i < n ? key[i] : kDoneKey;
        if (k[u] != kDoneKey) at[u] = atomicAdd(&sh[k[u]], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kHistSlots; i += kScatterThreads)
        if (sh[i]) sh[i] = atomicAdd(&cursor[i], sh[i]);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kScatterItems; ++u)
        if (k[u] != kDoneKey) order[sh[k[u]] + at[u]] = (int32_t)(base + u * kScatterThreads + threadIdx.x);
}

__global__ void __launch_bounds__(256)
ksw_scan_kernel(KswParams P, const bsb_ext_job_t *__restrict__ jobs, int64_t n, int64_t seq_bytes,
                const uint8_t *__restrict__ map, int builtin, ExtScan *__restrict__ out)
{
    const int lane = threadIdx.x & 31, ring = ring_of(builtin);
    unsigned long long bad = 0, need = 0;
    unsigned lo = 0, hi = 0;
    for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; i0 < n; i0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = i0 + lane;
        if (i >= n) continue;
        const bsb_ext_job_t j = jobs[i];
        if (!ext_job_ok(j, seq_bytes, kMaxNeed - 1)) {
            bad = max(bad, (unsigned long long)(n - i));
            continue;
        }
        const int t = map ? map[j.qlen + 1]
                      : P.pack16 && ksw_ring_fits(P, j, ring) ? kRingTile : c_tile_maps[builtin].tile[j.qlen + 1];
        if (t < 32) lo |= 1u << t;
        else hi |= 1u << (t - 32);
        need = max(need, (unsigned long long)max(j.qoff + j.qlen, j.toff + j.tlen));
    }
    lo = __reduce_or_sync(BSB_FULL_MASK, lo), hi = __reduce_or_sync(BSB_FULL_MASK, hi);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        bad = max(bad, __shfl_xor_sync(BSB_FULL_MASK, bad, d));
        need = max(need, __shfl_xor_sync(BSB_FULL_MASK, need, d));
    }
    if (lane == 0) {
        if (bad) atomicMax(&out->bad, bad);
        atomicOr(&out->tiles, (unsigned long long)hi << 32 | lo);
        atomicMax(&out->need, need);
    }
}

}  // namespace

static_assert(kRejectKey % kClasses == 0, "the reject slot starts a bin");

// scratch layout (int32 words): counter[3*kNumTiles] | rejected[1] | hist[kHistSlots] |
//   cursor[kHistSlots] | ranges[kRangeInts*kNumTiles] | (256-byte aligned) key[n] | order[n]
static size_t fixed_bytes()
{
    size_t fixed = sizeof(int) * (3 * kNumTiles + 1 + 2 * kHistSlots + kRangeInts * kNumTiles);
    return (fixed + 255) & ~(size_t)255;
}

size_t ksw_scratch_bytes(int64_t n) { return fixed_bytes() + sizeof(int32_t) * 2 * (size_t)n + 256; }

int ksw_max_qlen() { return kMaxNeed - 1; }

int64_t ksw_concurrent_below() { return (int64_t)1 << 20; }

int *ksw_rejected_counter(void *scratch) { return (int *)scratch + 3 * kNumTiles; }

int ksw_pack16_max() { return kPack16MaxH; }

bool ksw_pack16(const KswParams &P)
{
    return P.o_del + P.e_del <= 8000 && P.o_ins + P.e_ins <= 8000 && P.e_del <= 500 && P.e_ins <= 500 &&
           P.mat_max <= kPack16MaxScore;
}

int ksw_builtin(int64_t n, int n_sm, bool counting) { return ksw_builtin_of(n, n_sm, counting); }

const uint8_t *ksw_builtin_tile_map(int builtin) { return kBuiltinTileMaps[builtin].tile; }

const uint8_t *ksw_default_tile_map() { return kDefaultTileMap.tile; }

int ksw_tile_shape(int t, int *G, int *C)
{
    if (t < 0 || t >= kNumTiles) return -1;
    *G = kTileList[t].G;
    *C = kTileList[t].C;
    return 0;
}

uint64_t ksw_map_tiles(const uint8_t *map)
{
    uint64_t m = 0;
    for (int need = 1; need <= kMaxNeed; ++need) m |= 1ull << map[need];
    return m;
}

uint64_t ksw_builtin_tiles(int builtin) { return ksw_map_tiles(kBuiltinTileMaps[builtin].tile) | 1ull << kRingTile; }

cudaError_t ksw_scan_jobs(const KswParams &P, const bsb_ext_job_t *d_jobs, int64_t n, int64_t seq_bytes,
                          const uint8_t *d_map, int builtin, ExtScan *out, int n_sm, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof *out, st);
    if (e != cudaSuccess) return e;
    ksw_scan_kernel<<<(int)min((n + 255) / 256, (int64_t)n_sm * 2), 256, 0, st>>>(P, d_jobs, n, seq_bytes, d_map, builtin,
                                                                                  out);
    return cudaGetLastError();
}

int ksw_ring_from(int builtin) { return ring_cols(ring_of(builtin)); }

bool ksw_takes_ring(const KswParams &P, const bsb_ext_job_t &j, int builtin)
{
    return P.pack16 && ksw_ring_fits(P, j, ring_of(builtin));
}

int ksw_ring_tile() { return kRingTile; }

namespace {

// What the head of the scratch holds behind the counters.
constexpr size_t kZeroedBytes = sizeof(int) * (3 * kNumTiles + 1 + kHistSlots);
struct SchedScratch {
    int *rejected, *hist, *cursor;
    int32_t *ranges;
    explicit SchedScratch(void *scratch)
        : rejected((int *)scratch + 3 * kNumTiles), hist(rejected + 1), cursor(hist + kHistSlots), ranges(cursor + kHistSlots)
    {
    }
};

}  // namespace

cudaError_t ksw_load_kernels(void *scratch, cudaStream_t st)
{
    const SchedScratch s(scratch);
    KswParams P{};
    P.e_del = P.e_ins = P.pack16 = 1;
    cudaError_t e = cudaMemsetAsync(scratch, 0, kZeroedBytes, st);
    if (e != cudaSuccess) return e;
    ksw_sched_hist<false><<<1, kHistThreads, 0, st>>>(P, nullptr, 0, 0, nullptr, nullptr, nullptr, 0, 0, 0, 0, 4, nullptr,
                                                      s.hist, nullptr);
    ksw_sched_scan<<<1, kScanThreads, 0, st>>>(s.hist, s.cursor, s.ranges, s.rejected);
    ksw_sched_scatter<<<1, 256, 0, st>>>(nullptr, 0, s.cursor, nullptr);
    ksw_sched_scatter_tiles<<<1, kScatterThreads, 0, st>>>(nullptr, 0, s.cursor, nullptr);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const auto run = [&](KswTileLaunch f) {
        return f ? f(P, nullptr, nullptr, nullptr, s.ranges, (int *)scratch, nullptr, nullptr, -1, st) : cudaSuccess;
    };
    uint64_t tiles = 0;
    for (int b = 0; b < kBuiltinMaps; ++b) tiles |= ksw_map_tiles(kBuiltinTileMaps[b].tile);
    for (int t = 0; t < kNumTiles; ++t)
        if (tiles >> t & 1 &&
            ((e = run(ksw_tile_launcher(t))) != cudaSuccess || (e = run(ksw_tile16_launcher(t))) != cudaSuccess))
            return e;
    for (int r = 0; r < (int)(sizeof(kRings) / sizeof(kRings[0])); ++r)
        if ((e = run(ksw_ring16(r))) != cudaSuccess) return e;
    return cudaSuccess;
}

cudaError_t ksw_launch(const KswParams &P, const bsb_ext_job_t *d_jobs, int64_t n, int64_t seq_bytes,
                       const uint8_t *d_seq, const int32_t *d_cost, const uint8_t *d_map, int builtin, uint64_t tiles,
                       bsb_ext_out_t *d_out, int64_t *d_cells, void *scratch, int n_sm, cudaStream_t st,
                       cudaEvent_t ev0, cudaEvent_t ev1, const cudaEvent_t *tile_ev, uint64_t *launched,
                       const KswStreams *ms, bool all_narrow)
{
    if (launched) *launched = 0;
    int *const counter = (int *)scratch;    // 3 per tile: 16-bit range, wide range, whole tile
    const SchedScratch sched(scratch);
    int *const rejected = sched.rejected, *const hist = sched.hist, *const cursor = sched.cursor;
    int32_t *const ranges = sched.ranges, *const key = (int32_t *)((char *)scratch + fixed_bytes()), *const order = key + n;
    // 16-bit cells need every value of the packed arithmetic inside 16 bits: penalties
    // and their multiples by a lane's column count stay small, and scores at most
    // kPack16MaxScore (h0 + qlen * max score is checked per job)
    KswParams Q = P;
    Q.pack16 = ksw_pack16(P);
    const bool ring = !d_map && !Q.pac && Q.pack16 && (tiles >> kRingTile & 1);
    if (!d_map && !ring) tiles &= ~(1ull << kRingTile);
    // the rings for cut bands that queries of the batch's shapes are wide enough for
    int cuts = 0;
    if (!d_map && !Q.pac && Q.pack16 && !d_cells && builtin <= 1) {
        for (int t = 0; t < kNumTiles; ++t)
            for (int c = 0; c < kCutRings; ++c)
                if (tiles >> t & 1 && (t == kRingTile || kTileList[t].G * kTileList[t].C >= cut_from(c, builtin))) cuts |= 1 << c;
        for (int c = 0; c < kCutRings; ++c)
            if (cuts >> c & 1) tiles |= 1ull << cut_tile(c);
    }
    cudaError_t e;
    if (ev0) cudaEventRecord(ev0, st);
    e = cudaMemsetAsync(scratch, 0, kZeroedBytes, st);
    if (e != cudaSuccess) return e;
    if (n > 0) {
        const int nb = (int)min((int64_t)n_sm * 8, (n + 255) / 256);
        // jobs a warp takes at a time: 32, or 4 where that still leaves warps free (the diagonals of
        // a warp's jobs are a chain of dependent loads, four at a time)
        const int per = n >= (int64_t)n_sm * 8 * (kHistThreads / 32) * 4 ? 32 : 4;
        const int hb = (int)min((int64_t)n_sm * 8, (n + per * (kHistThreads / 32) - 1) / (per * (kHistThreads / 32)));
        const auto hist_kernel = Q.pac ? ksw_sched_hist<true> : ksw_sched_hist<false>;
        hist_kernel<<<hb, kHistThreads, 0, st>>>(Q, d_jobs, (int)n, (long long)seq_bytes, d_seq, d_cost, d_map, builtin,
                                                 ring, d_cells == nullptr, cuts, per, d_out, hist, key);
        ksw_sched_scan<<<1, kScanThreads, 0, st>>>(hist, cursor, ranges, rejected);
        if (n >= 8 * kScatterTile)
            ksw_sched_scatter_tiles<<<(unsigned)((n + kScatterTile - 1) / kScatterTile), kScatterThreads, 0, st>>>(
                key, (int)n, cursor, order);
        else
            ksw_sched_scatter<<<nb, 256, 0, st>>>(key, (int)n, cursor, order);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        // Small batches: the shapes run on four streams, so the next shape's blocks fill
        // the SMs a finishing shape leaves during its tail.  Large batches keep one stream
        // (the tails are a small part of them, and each shape is timed alone).
        const bool conc = ms && n < ksw_concurrent_below();
        if (conc) {
            cudaEventRecord(ms->fork, st);
            for (int a = 0; a < BSB_AUX_STREAMS; ++a) cudaStreamWaitEvent(ms->aux[a], ms->fork, 0);
        }
        int k = 0;
        for (int t = 0; t < kNumTiles; ++t) {
            if (!(tiles >> t & 1)) continue;
            KswTileLaunch f = ksw_tile_launcher(t), f16 = Q.pack16 ? ksw_tile16_launcher(t) : nullptr;
            if (Q.pac) f16 = Q.pack16 && all_narrow ? ksw_packed16_launcher(t) : nullptr;   // 16-bit cells only
            if (!f || (Q.pac && !f16)) return cudaErrorInvalidValue;
            const int lane = k++ % (BSB_AUX_STREAMS + 1);
            cudaStream_t s = conc && lane ? ms->aux[lane - 1] : st;
            const int32_t *r = ranges + kRangeInts * t;
            if (tile_ev) cudaEventRecord(tile_ev[2 * t], s);
            int cut = -1;
            for (int c = 0; c < kCutRings; ++c)
                if (cuts >> c & 1 && t == cut_tile(c)) cut = c;
            if ((ring && t == kRingTile) || cut >= 0) {
                e = ksw_ring16(cut >= 0 ? kFirstCut + cut : ring_of(builtin))(Q, d_jobs, d_seq, order, r + 4, counter + 3 * t, d_out, d_cells, n_sm, s);
            } else if (f16) {
                // the wide class is rare (very large h0): one block per SM drains it
                e = f16(Q, d_jobs, d_seq, order, r, counter + 3 * t, d_out, d_cells, n_sm, s);
                if (e == cudaSuccess && !all_narrow)
                    e = f(Q, d_jobs, d_seq, order, r + 2, counter + 3 * t + 1, d_out, d_cells, -n_sm, s);
            } else {
                e = f(Q, d_jobs, d_seq, order, r + 4, counter + 3 * t + 2, d_out, d_cells, n_sm, s);
            }
            if (e != cudaSuccess) return e;
            if (tile_ev) cudaEventRecord(tile_ev[2 * t + 1], s);
            if (launched) *launched |= 1ull << t;
        }
        if (conc) {
            for (int a = 0; a < BSB_AUX_STREAMS; ++a) {
                cudaEventRecord(ms->join[a], ms->aux[a]);
                cudaStreamWaitEvent(st, ms->join[a], 0);
            }
        }
    }
    if (ev1) cudaEventRecord(ev1, st);
    return cudaSuccess;
}
