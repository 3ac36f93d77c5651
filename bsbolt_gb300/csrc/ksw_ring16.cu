// ksw_ring16.cu -- the extension kernel of long queries with a narrow band (ksw_group16.cuh, Ring).
#include "ksw_tiles_impl.cuh"

namespace {

template <int C2, int G>
__global__ void __launch_bounds__(kKswBlock, ksw16_min_blocks(C2, G))
ksw_ring16_kernel(KswParams P, const bsb_ext_job_t *__restrict__ jobs, const uint8_t *__restrict__ seq,
                  const int32_t *__restrict__ order, const int32_t *__restrict__ range, int *__restrict__ counter,
                  bsb_ext_out_t *__restrict__ out, int64_t *__restrict__ cells)
{
    __shared__ uint8_t queries[kKswBlock / G][kMaxNeed];
    __shared__ uint2 words[5];
    if (threadIdx.x < 5)
        words[threadIdx.x] = make_uint2(profile_word(P, threadIdx.x), (uint8_t)profile_n(P, threadIdx.x));
    __syncthreads();
    ksw_group16_run<C2, G, false, true>(P, jobs, seq, order, range[0], range[1], counter, out, cells,
                                        queries[threadIdx.x / G], words);
}

template <int R>
cudaError_t ksw_ring16_launch(const KswParams &P, const bsb_ext_job_t *jobs, const uint8_t *seq, const int32_t *order,
                              const int32_t *range, int *counter, bsb_ext_out_t *out, int64_t *cells, int n_sm,
                              cudaStream_t st)
{
    static int blocks_per_sm = 0;
    return ksw_launch_wave(ksw_ring16_kernel<kRings[R].C / 2, kRings[R].G>, blocks_per_sm, P, jobs, seq, order, range, counter,
                           out, cells, n_sm, st);
}

}  // namespace

KswTileLaunch ksw_ring16(int ring)
{
    switch (ring) {
    case 0: return ksw_ring16_launch<0>;
    case 1: return ksw_ring16_launch<1>;
    case 2: return ksw_ring16_launch<2>;
    case 3: return ksw_ring16_launch<3>;
    default: return ksw_ring16_launch<4>;
    }
}
