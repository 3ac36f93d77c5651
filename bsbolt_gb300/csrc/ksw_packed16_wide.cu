// ksw_packed16_wide.cu -- the 16-bit extension kernels of an alignment batch's jobs, 8 to 32 lanes per
// job.
#include "ksw_tiles_impl.cuh"

KswTileLaunch ksw_packed16_wide(int G, int C)
{
    switch (G << 8 | C) {
    case 8 << 8 | 18: return ksw_packed16_launch<9, 8>;
    case 16 << 8 | 10: return ksw_packed16_launch<5, 16>;
    case 16 << 8 | 12: return ksw_packed16_launch<6, 16>;
    case 16 << 8 | 14: return ksw_packed16_launch<7, 16>;
    case 16 << 8 | 16: return ksw_packed16_launch<8, 16>;
    case 32 << 8 | 6: return ksw_packed16_launch<3, 32>;
    case 32 << 8 | 8: return ksw_packed16_launch<4, 32>;
    case 32 << 8 | 10: return ksw_packed16_launch<5, 32>;
    case 32 << 8 | 12: return ksw_packed16_launch<6, 32>;
    case 32 << 8 | 14: return ksw_packed16_launch<7, 32>;
    case 32 << 8 | 16: return ksw_packed16_launch<8, 32>;
    case 32 << 8 | 20: return ksw_packed16_launch<10, 32>;
    case 32 << 8 | 24: return ksw_packed16_launch<12, 32>;
    case 32 << 8 | 28: return ksw_packed16_launch<14, 32>;
    case 32 << 8 | 32: return ksw_packed16_launch<16, 32>;
    default: return nullptr;
    }
}
