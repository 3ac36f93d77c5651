// ksw_tiles.cuh -- the tile shapes of the batched extension and the map that
// assigns one to every query length.
//
// A tile is G lanes per job (32/G jobs per warp) x C query columns per lane;
// it holds queries of up to G*C - 1 bases (columns 0..qlen).  Every shape in
// kTileList is compiled (ksw_tiles_g*.cu); a tile map picks, for each
// need = qlen + 1, the shape its jobs run on.  The default map below was
// chosen by timing every candidate shape per query-length band on a GB300;
// bsb_set_tile_map installs another one (e.g. the autotuner's) per context.
// The shape never changes a result, only the time.
#pragma once

#include "bsb_internal.cuh"

struct KswTile {
    int G, C;
};

constexpr KswTile kTileList[] = {
    {4, 1},   {4, 2},   {4, 3},   {4, 4},   {4, 5},   {4, 6},   {4, 7},   {4, 8},      //  0..7
    {4, 9},   {4, 10},  {4, 11},  {4, 12},  {4, 13},  {4, 14},  {4, 15},  {4, 16},     //  8..15
    {8, 6},   {8, 7},   {8, 8},   {8, 9},   {8, 10},  {8, 11},  {8, 12},  {8, 13},     // 16..23
    {8, 14},  {8, 15},  {8, 16},  {8, 17},  {8, 18},                                    // 24..28
    {16, 5},  {16, 6},  {16, 7},  {16, 8},  {16, 9},  {16, 10}, {16, 11}, {16, 12},    // 29..36
    {16, 13}, {16, 14}, {16, 15}, {16, 16},                                             // 37..40
    {32, 5},  {32, 6},  {32, 7},  {32, 8},  {32, 9},  {32, 10}, {32, 11}, {32, 12},    // 41..48
    {32, 13}, {32, 14}, {32, 15}, {32, 16},                                             // 49..52
    {32, 20}, {32, 24}, {32, 28}, {32, 32},                                             // 53..56
    {4, 20},  {4, 24},  {4, 28},  {4, 32}};                                             // 57..60
constexpr int kNumTiles = sizeof(kTileList) / sizeof(kTileList[0]);
constexpr int kMaxNeed = BSB_TILE_MAP_LEN - 1;    // columns 0..qlen with qlen <= 1023
constexpr int kKswBlock = 128;                      // threads per block (4 warps)
constexpr int kPack16MaxH = 2047;                   // the largest H of the 16-bit cells (ksw_group16.cuh)

static_assert(kNumTiles == BSB_NUM_TILES, "tile list and public header disagree");
static_assert(kNumTiles <= 64, "tile sets are 64-bit masks");

// Shapes with a 16-bit two-columns-per-register kernel: an even C (every shape has C <= 32:
// a lane's non-zero columns are one 32-bit mask, and the 16-bit row-maximum key keeps a
// column index in 4 bits per half).
constexpr bool tile_has_pack16(int C) { return C % 2 == 0 && C <= 32; }

constexpr int tile_index(int G, int C)
{
    for (int t = 0; t < kNumTiles; ++t)
        if (kTileList[t].G == G && kTileList[t].C == C) return t;
    return -1;
}

struct KswTileMap {
    uint8_t tile[kMaxNeed + 1];    // [0] unused
};

// 4 lanes up to 128 columns (even C up to 16, then 20, 24, 28, 32), 8 lanes up to
// 144, 16 up to 256, then 32; the narrowest even C that holds the query within each
// group size (even C runs on 16-bit cells, two per register: cheaper than the
// next-narrower odd C).  Measured on GB300 with the autotuner on the 4M-job
// distribution: 4x20..4x32 beat 8x10..8x16 by 1.11-1.23x on the bands they hold (fewer
// lanes per job amortise a row's fixed work over more columns).
constexpr int even_up(int c) { return c + (c & 1); }
constexpr KswTileMap make_default_tile_map()
{
    KswTileMap m{};
    for (int need = 1; need <= kMaxNeed; ++need) {
        int t = 0;
        if (need <= 64) t = tile_index(4, even_up((need + 3) / 4));
        else if (need <= 128) t = tile_index(4, ((need + 15) / 16) * 4);
        else if (need <= 144) t = tile_index(8, even_up((need + 7) / 8 < 9 ? 9 : (need + 7) / 8));
        else if (need <= 256) t = tile_index(16, even_up((need + 15) / 16 < 10 ? 10 : (need + 15) / 16));
        else if (need <= 512) t = tile_index(32, even_up((need + 31) / 32 < 9 ? 9 : (need + 31) / 32));
        else if (need <= 640) t = tile_index(32, 20);
        else if (need <= 768) t = tile_index(32, 24);
        else if (need <= 896) t = tile_index(32, 28);
        else t = tile_index(32, 32);
        m.tile[need] = (uint8_t)t;
    }
    return m;
}

constexpr KswTileMap kDefaultTileMap = make_default_tile_map();

// The built-in maps by batch size.  The default map fills the GPU with 4-lane groups only from a
// few hundred thousand jobs on; a smaller batch is bound by the rows of its longest jobs, one after
// the other, and a row takes the fewer cycles the more lanes share it (a 4x32 group about 1600, a
// 32x6 warp 600).  So the fewer jobs, the wider the groups, and few shapes, so that few launches
// follow one another.  Jobs of 10-140 bases, us (default map in brackets): 64 jobs 129 (328), 3000
// 181 (490), 10,000 220 (537), 30,000 300 (586), 130,000 774 (792), 260,000 1362 (1349).
// Queries beyond the bands given here keep the default's shapes.
constexpr int kBuiltinMaps = 5;
constexpr KswTileMap with_band(KswTileMap m, int lo, int hi, int G, int C)
{
    for (int need = lo; need <= hi; ++need) m.tile[need] = (uint8_t)tile_index(G, C);
    return m;
}
constexpr KswTileMap kBuiltinTileMaps[kBuiltinMaps] = {
    kDefaultTileMap,
    with_band(with_band(kDefaultTileMap, 1, 64, 4, 16), 65, 144, 8, 18),
    with_band(kDefaultTileMap, 1, 160, 16, 10),
    with_band(with_band(kDefaultTileMap, 1, 192, 32, 6), 193, 256, 32, 8),
    with_band(with_band(kDefaultTileMap, 1, 192, 32, 6), 193, 256, 32, 8),     // (with the other ring, below)
};
// The built-in map of a batch of n jobs (lines between the measured sizes where two maps meet).  Counting cells means
// computing all of them, with twice the jobs and more rows: such batches fill the GPU sooner (100,000 jobs of 10-140 bases
// through the device entry 1.41 ms on the default map, 1.65 on the next; 45,000 0.96 and 0.85).
inline int ksw_builtin_of(int64_t n, int n_sm, bool counting)
{
    const int64_t per = n / n_sm + (n % n_sm != 0);
    return per <= 30 ? 4 : per <= 50 ? 3 : per <= 90 ? 2 : per <= (counting ? 450 : 1300) ? 1 : 0;
}

// Queries wider than a ring's columns whose band is narrower run on it (ksw_group16.cuh): registers for G*C columns
// that move along with the band.  Taken on the built-in maps only (an installed map's shapes are the caller's);
// their jobs are listed, and their time is reported, under a shape no built-in map uses.  A row costs what its
// lanes hold, so a 600-base query with a band of 201 pays for 224 columns instead of 640, two jobs a warp:
// 50k jobs of 500-600 bases 14.4 ms -> 6.7, 50k of 100-600 6.9 -> 4.3, 20k of 230-300 1.68 -> 1.44; 16x16, 8x30 and
// 8x32 rings 4.6, 4.6 and 4.6 where 16x14 takes 4.3.  The smallest batches are bound by the rows one after the
// other, where a warp a job is faster: 64 jobs of 300-600 bases 0.77 ms -> 0.54 (16x14 0.64), 3000 of 100-600 1.05
// -> 0.76 (0.95), but 7500 of 300-600 1.34 (1.16), 10,000 of 300-400 1.55 -> 1.38 (1.12).
constexpr KswTile kRings[] = {{16, 14}, {32, 8}, {4, 8}, {4, 16}, {4, 32}};
__host__ __device__ __forceinline__ constexpr int ring_of(int builtin) { return builtin == kBuiltinMaps - 1 ? 1 : 0; }
__host__ __device__ __forceinline__ constexpr int ring_cols(int ring) { return ring ? 32 * 8 : 16 * 14; }
__host__ __device__ __forceinline__ constexpr int ring_block(int ring) { return ring ? 8 : 14; }
static_assert(ring_cols(0) == kRings[0].G * kRings[0].C && ring_cols(1) == kRings[1].G * kRings[1].C &&
              ring_block(0) == kRings[0].C && ring_block(1) == kRings[1].C, "the rings' sizes");
// Jobs whose band can be cut (cut_band, ksw_core.cuh: most of those with a few mismatches) run on rings of their own, by
// the band they need, where the query is wider than its ring pays for: 4 lanes of 8, 16 and 32 columns, eight jobs a
// warp.  Only in batches that come near to filling the GPU with 4-lane groups (the first two built-in maps; on the
// second, beyond its 8 x 18 shape: 64k jobs of 10-140 bases 658 us, 674 with the shorter ones cut), on byte jobs, and not
// where cells are counted.  2M jobs of 10-140 bases 7.92 ms -> 6.84, 50k of 100-600 4.03 -> 3.30 (half of them cut).
constexpr int kCutRings = 3, kFirstCut = 2;
__host__ __device__ __forceinline__ constexpr int cut_from(int c, int builtin)          // query + 1
{
    return builtin == 1 || c == 2 ? 145 : c == 1 ? 97 : 65;
}
__host__ __device__ __forceinline__ constexpr int cut_width(int c) { return c == 0 ? 11 : c == 1 ? 23 : 47; }
static_assert(2 * cut_width(0) + 8 + 1 <= 32 && 2 * cut_width(1) + 16 + 1 <= 64 && 2 * cut_width(2) + 32 + 1 <= 128,
              "the cut rings' bands");
constexpr int kRingTile = tile_index(32, 5);
constexpr int kCutTile0 = tile_index(32, 7), kCutTile1 = tile_index(32, 9), kCutTile2 = tile_index(32, 11);
__host__ __device__ __forceinline__ constexpr int cut_tile(int c)
{
    return c == 0 ? kCutTile0 : c == 1 ? kCutTile1 : kCutTile2;
}
constexpr bool ring_tile_is_free()
{
    for (int b = 0; b < kBuiltinMaps; ++b)
        for (int need = 1; need <= kMaxNeed; ++need)
            if (kBuiltinTileMaps[b].tile[need] == kRingTile || kBuiltinTileMaps[b].tile[need] == kCutTile0 ||
                kBuiltinTileMaps[b].tile[need] == kCutTile1 || kBuiltinTileMaps[b].tile[need] == kCutTile2)
                return false;
    return true;
}
static_assert(ring_tile_is_free(), "a built-in map uses the ring's place");
// The job's cells fit 16 bits, no column passes the row-maximum key's 10 bits, and a block of columns beside
// the band of a row (w as ksw.c:399-407 cuts it) holds all columns that row and the next write.
__host__ __device__ __forceinline__ bool ksw_ring_fits(const KswParams &P, const bsb_ext_job_t &j, int ring)
{
    const int cols = ring_cols(ring), block = ring_block(ring);
    if (j.qlen < cols || j.qlen + block >= 1024 ||
        (long long)j.h0 + (long long)j.qlen * P.mat_max > kPack16MaxH)
        return false;
    const int mi = band_cap(j.qlen * P.mat_max + j.end_bonus - P.o_ins, P.e_ins);
    const int md = band_cap(j.qlen * P.mat_max + j.end_bonus - P.o_del, P.e_del);
    int w = j.w;
    w = w < mi ? w : mi > 1 ? mi : 1;
    w = w < md ? w : md > 1 ? md : 1;
    return 2 * (long long)w + block + 1 <= cols;
}

// Launches the persistent kernel of one tile shape over a range of the scheduled
// order: the jobs order[range[0] .. range[1]), drawn through *counter.
typedef cudaError_t (*KswTileLaunch)(const KswParams &P, const bsb_ext_job_t *jobs, const uint8_t *seq,
                                     const int32_t *order, const int32_t *range, int *counter,
                                     bsb_ext_out_t *out, int64_t *cells, int n_sm, cudaStream_t st);

KswTileLaunch ksw_tiles_g4(int C);
KswTileLaunch ksw_tiles_g8(int C);
KswTileLaunch ksw_tiles_g16(int C);
KswTileLaunch ksw_tiles_g32(int C);
KswTileLaunch ksw_tiles16_g4(int C);
KswTileLaunch ksw_tiles16_g8(int C);
KswTileLaunch ksw_tiles16_g16(int C);
KswTileLaunch ksw_tiles16_g32(int C);

// The kernels of an alignment batch's jobs exist for the shapes of the built-in maps.
KswTileLaunch ksw_packed16_g4(int C);
KswTileLaunch ksw_packed16_wide(int G, int C);
KswTileLaunch ksw_ring16(int ring);
inline KswTileLaunch ksw_packed16_launcher(int t)
{
    if (t < 0 || t >= kNumTiles) return nullptr;
    return kTileList[t].G == 4 ? ksw_packed16_g4(kTileList[t].C) : ksw_packed16_wide(kTileList[t].G, kTileList[t].C);
}

// The 32-bit cell kernel of tile t (every shape has one).
inline KswTileLaunch ksw_tile_launcher(int t)
{
    if (t < 0 || t >= kNumTiles) return nullptr;
    const KswTile s = kTileList[t];
    switch (s.G) {
    case 4: return ksw_tiles_g4(s.C);
    case 8: return ksw_tiles_g8(s.C);
    case 16: return ksw_tiles_g16(s.C);
    case 32: return ksw_tiles_g32(s.C);
    default: return nullptr;
    }
}

// The 16-bit two-columns-per-register kernel of tile t (tile_has_pack16), or NULL.
inline KswTileLaunch ksw_tile16_launcher(int t)
{
    if (t < 0 || t >= kNumTiles || !tile_has_pack16(kTileList[t].C)) return nullptr;
    const KswTile s = kTileList[t];
    switch (s.G) {
    case 4: return ksw_tiles16_g4(s.C);
    case 8: return ksw_tiles16_g8(s.C);
    case 16: return ksw_tiles16_g16(s.C);
    case 32: return ksw_tiles16_g32(s.C);
    default: return nullptr;
    }
}
