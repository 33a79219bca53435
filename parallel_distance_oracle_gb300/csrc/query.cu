// query.cu -- exact 2-hop distance queries on a device-resident label set: a
// warp per pair (the per-pair code and its derivation are in
// query_device.cuh), grid-stride over the batch.
//
// What bounds it: on label sets larger than L2 the pair's reads (10M uniform pairs
// on R-MAT s20, K = 64), else the instructions of a pair and the chain of its
// dependent loads (endpoints, ranks, offsets; BP distances and hubs; sets), hidden
// by other warps, so residency decides: 64 warps per SM, which is why the kernel is
// held to 32 registers, counts its bytes only in the profiling instance and keeps
// pair numbers in 32 bits.  In a large batch a warp takes a group of consecutive
// pairs: its lanes read the heads (ranks, offsets, lengths) of all of them at
// once, and the results leave in one store.
//   10M uniform pairs, s20, K = 64:  7.16 ms at first; 5.05 with the BP sets of the
//     deciding roots only and the lists in one round; 4.62 with lists of up to 32
//     compared in registers and no reads for empty ones; 4.35 in groups
//   2M pairs, s12, K = 50:  460 -> 526 -> 424 -> 367 us; Zipf endpoints 371 -> 471 -> 396 -> 319 us
//   2M weighted pairs, s16:  567 -> 409 -> 377 -> 331 us

#include "query_device.cuh"

namespace pado {
namespace {

// Pairs per launch: pair numbers fit 32 bits with room for the grid stride.
constexpr uint64_t MAX_LAUNCH_PAIRS = 1ull << 31;

// Pairs whose heads a warp reads together, a lane each.
constexpr uint32_t MAX_GROUP = 32;

template <bool COUNT, bool ONE>
__global__ void __launch_bounds__(256, 8) query_unw_kernel(IndexView v, uint32_t k, uint32_t group,
                                                           const uint32_t *__restrict__ qa,
                                                           const uint32_t *__restrict__ qb, uint8_t *__restrict__ out)
{
    __shared__ QueryScratch qs[8];
    __shared__ PairHead heads[8][ONE ? 1 : MAX_GROUP];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t step = ((gridDim.x * blockDim.x) >> 5) * group;
    unsigned long long bytes = 0;
    for (uint32_t p = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * group; p < k; p += step) {
        if (ONE) {
            const uint8_t d = query_unw_pair<true>(v, pair_head(v, qa[p], qb[p], U8_INF), lane, qs[warp], bytes);
            if (lane == 0) out[p] = d;
            bytes += 9;
            continue;
        }
        const uint32_t cnt = min(group, k - p);
        __syncwarp();
        if ((uint32_t)lane < cnt) heads[warp][lane] = pair_head(v, qa[p + lane], qb[p + lane], U8_INF);
        __syncwarp();
        uint8_t mine = 0;
        for (uint32_t j = 0; j < cnt; ++j) {
            const uint8_t d = query_unw_pair<false>(v, heads[warp][j], lane, qs[warp], bytes);
            if ((uint32_t)lane == j) mine = d;
        }
        bytes += 9ull * cnt;  // endpoints, results
        if ((uint32_t)lane < cnt) out[p + lane] = mine;
    }
    if (COUNT && lane == 0 && bytes) atomicAdd(&v.work[W_Q_UNW], bytes);
}

template <bool COUNT, bool ONE>
__global__ void __launch_bounds__(256) query_w_kernel(IndexView v, uint32_t k, uint32_t group,
                                                           const uint32_t *__restrict__ qa,
                                                           const uint32_t *__restrict__ qb, int16_t *__restrict__ out)
{
    __shared__ QueryScratch qs[8];
    __shared__ PairHead heads[8][ONE ? 1 : MAX_GROUP];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t step = ((gridDim.x * blockDim.x) >> 5) * group;
    unsigned long long bytes = 0;
    for (uint32_t p = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * group; p < k; p += step) {
        if (ONE) {
            const int16_t d = query_w_pair<true>(v, pair_head(v, qa[p], qb[p], I16_INF), lane, qs[warp], bytes);
            if (lane == 0) out[p] = d;
            bytes += 10;
            continue;
        }
        const uint32_t cnt = min(group, k - p);
        __syncwarp();
        if ((uint32_t)lane < cnt) heads[warp][lane] = pair_head(v, qa[p + lane], qb[p + lane], I16_INF);
        __syncwarp();
        int16_t mine = 0;
        for (uint32_t j = 0; j < cnt; ++j) {
            const int16_t d = query_w_pair<false>(v, heads[warp][j], lane, qs[warp], bytes);
            if ((uint32_t)lane == j) mine = d;
        }
        bytes += 10ull * cnt;  // endpoints, results
        if ((uint32_t)lane < cnt) out[p + lane] = mine;
    }
    if (COUNT && lane == 0 && bytes) atomicAdd(&v.work[W_Q_W], bytes);
}

// Pairs per warp and turn: doubled while every resident warp still gets four
// groups (4 against 16: 0.7M uniform pairs on s20 385 us against 351, 2M pairs on s12 367
// against 374; with one group a warp 0.2M pairs on s20 take 147 us, not 134).
// Groups of one keep the head in registers (20,000 pairs: 10.3 us, through shared memory 11.4).
uint32_t pair_group(uint64_t k)
{
    uint32_t g = 1;
    while (g < MAX_GROUP && k >= (uint64_t)g * 2 * 4 * 152 * 64) g *= 2;
    return g;
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
        const uint32_t group = pair_group(n);
        const unsigned grid = grid_for(((uint64_t)n + group - 1) / group * 32, 256, 152u * 64u);
        PADO_LAUNCH("query_unw_kernel", s,
                    (v.work ? group == 1 ? query_unw_kernel<true, true> : query_unw_kernel<true, false>
                     : group == 1 ? query_unw_kernel<false, true> : query_unw_kernel<false, false>)<<<grid, 256, 0, s>>>(
                        v, n, group, a + at, b + at, out + at));
    });
}

void launch_query_w(const IndexView &v0, uint64_t k, const uint32_t *a, const uint32_t *b, int16_t *out,
                    cudaStream_t s)
{
    IndexView v = v0;
    v.work = work_counters();
    in_launches(k, [&](uint64_t at, uint32_t n) {
        const uint32_t group = pair_group(n);
        const unsigned grid = grid_for(((uint64_t)n + group - 1) / group * 32, 256, 152u * 64u);
        PADO_LAUNCH("query_w_kernel", s,
                    (v.work ? group == 1 ? query_w_kernel<true, true> : query_w_kernel<true, false>
                     : group == 1 ? query_w_kernel<false, true> : query_w_kernel<false, false>)<<<grid, 256, 0, s>>>(
                        v, n, group, a + at, b + at, out + at));
    });
}

}  // namespace pado
