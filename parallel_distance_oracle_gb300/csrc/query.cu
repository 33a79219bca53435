// query.cu -- exact 2-hop distance queries on a device-resident label set: a
// warp per pair (the per-pair code and its derivation are in
// query_device.cuh), grid-stride over the batch.
//
// What bounds it: the chain of dependent loads of a pair (endpoints, ranks,
// offsets and BP distances, then sets and lists), hidden by other warps, so
// residency decides: 64 warps per SM, which is why the kernel is held to 32
// registers, counts its bytes only in the profiling instance and keeps pair
// numbers in 32 bits (10M uniform pairs on R-MAT s20, K = 64: 5.05 ms with 8
// blocks of 256 threads per SM, 5.65 ms with 6).  Reading a pair's lists in
// one round instead of block by block, and the BP sets of the deciding roots
// only, took the same batch from 7.08 ms; 1M weighted pairs (s16) from 285 us
// to 215 us.

#include "query_device.cuh"

namespace pado {
namespace {

// Pairs per launch: pair numbers fit 32 bits with room for the grid stride.
constexpr uint64_t MAX_LAUNCH_PAIRS = 1ull << 31;

template <bool COUNT>
__global__ void __launch_bounds__(256, 8) query_unw_kernel(IndexView v, uint32_t k, const uint32_t *__restrict__ qa,
                                                           const uint32_t *__restrict__ qb, uint8_t *__restrict__ out)
{
    __shared__ QueryScratch qs[8];
    const int lane = threadIdx.x & 31;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    unsigned long long bytes = 0;
    for (uint32_t p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < k; p += nwarps) {
        bytes += 9;  // endpoints, result
        const uint8_t d = query_unw_pair(v, qa[p], qb[p], lane, qs[threadIdx.x >> 5], bytes);
        if (lane == 0) out[p] = d;
    }
    if (COUNT && lane == 0 && bytes) atomicAdd(&v.work[W_Q_UNW], bytes);
}

template <bool COUNT>
__global__ void __launch_bounds__(256) query_w_kernel(IndexView v, uint32_t k, const uint32_t *__restrict__ qa,
                                                      const uint32_t *__restrict__ qb, int16_t *__restrict__ out)
{
    __shared__ QueryScratch qs[8];
    const int lane = threadIdx.x & 31;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    unsigned long long bytes = 0;
    for (uint32_t p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < k; p += nwarps) {
        bytes += 10;
        const int16_t d = query_w_pair(v, qa[p], qb[p], lane, qs[threadIdx.x >> 5], bytes);
        if (lane == 0) out[p] = d;
    }
    if (COUNT && lane == 0 && bytes) atomicAdd(&v.work[W_Q_W], bytes);
}

// Calls launch(pairs done before, pairs of this launch) over the batch.
template <typename F>
void in_launches(uint64_t k, F &&launch)
{
    for (uint64_t at = 0; at < k; at += MAX_LAUNCH_PAIRS) launch(at, (uint32_t)std::min(MAX_LAUNCH_PAIRS, k - at));
}

}  // namespace

void launch_query_unw(const IndexView &v0, uint64_t k, const uint32_t *a, const uint32_t *b, uint8_t *out,
                      cudaStream_t s)
{
    IndexView v = v0;
    v.work = work_counters();
    in_launches(k, [&](uint64_t at, uint32_t n) {
        const unsigned grid = grid_for((uint64_t)n * 32, 256, 152u * 64u);
        PADO_LAUNCH("query_unw_kernel", s,
                    (v.work ? query_unw_kernel<true> : query_unw_kernel<false>)<<<grid, 256, 0, s>>>(
                        v, n, a + at, b + at, out + at));
    });
}

void launch_query_w(const IndexView &v0, uint64_t k, const uint32_t *a, const uint32_t *b, int16_t *out,
                    cudaStream_t s)
{
    IndexView v = v0;
    v.work = work_counters();
    in_launches(k, [&](uint64_t at, uint32_t n) {
        const unsigned grid = grid_for((uint64_t)n * 32, 256, 152u * 64u);
        PADO_LAUNCH("query_w_kernel", s,
                    (v.work ? query_w_kernel<true> : query_w_kernel<false>)<<<grid, 256, 0, s>>>(
                        v, n, a + at, b + at, out + at));
    });
}

}  // namespace pado
