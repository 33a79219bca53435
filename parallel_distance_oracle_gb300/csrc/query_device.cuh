// query_device.cuh -- one exact 2-hop distance query per warp, shared by the
// plain query kernels (query.cu) and the serving loop's mixed-batch kernel
// (serve.cu).
//
// Restates query_distance (reference includes/pado_unw_unv_unp.h:1312-1445;
// weighted includes/pado_weighted_unv_unp.h:1782-1900):
//   d = INF; for each BP root i: td = bpd_a[i] + bpd_b[i]; if td-2 <= d then
//   td -= 2 / 1 / 0 by the S^-1 / S^0 intersections and d = min(d, td);
//   then d = min over common hubs h of dist_a(h) + dist_b(h); saturate.
// Lane i evaluates BP roots i and i+32 (K <= 64); the sets S^-1 / S^0, 16 of a
// root's 17 bytes per vertex, are read only for the roots that can decide the
// minimum (see query_unw_pair).  The two hub-sorted label
// lists are intersected 32 x 32 entries at a time: each lane binary-searches
// its a-hub among the b-block with warp shuffles, and the block whose last
// hub is smaller advances.  The result is a warp
// min-reduction.  Everything is integer arithmetic with the reference's
// unsigned comparisons, so results are bit-exact.
#pragma once

#include "pado_internal.cuh"

namespace pado {
namespace {

constexpr unsigned FULL = 0xffffffffu;

// Entries of the longer label list that are searched at once, per warp in
// shared memory.
constexpr uint32_t QWIN = 128;

// A warp's scratch in shared memory.
struct QueryScratch {
    uint32_t win[QWIN];
    uint16_t root[MAX_BP];
};

// Starts the copy of list entries [0, min(n, QWIN)) into the warp's window,
// padded with a value above every hub (no registers are held meanwhile).
__device__ __forceinline__ void stage_window(uint32_t *win, const uint32_t *__restrict__ h, uint32_t n, int lane)
{
#pragma unroll
    for (uint32_t q = 0; q < QWIN; q += 32) {
        const uint32_t j = q + lane;
        if (j < n)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(win + j)),
                         "l"(h + j)
                         : "memory");
        else
            win[j] = 0xffffffffu;
    }
}

__device__ __forceinline__ void window_ready()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
}

// Minimum of da(h) + db(h) over hubs h common to the two sorted lists, and d;
// la <= lb, the window holds (or awaits) b's first entries and `av` a's first
// hubs.  32 hubs of a at a time are searched in the window (7 steps in shared
// memory); whichever side ends at the lower hub moves on.
template <typename D>
__device__ __forceinline__ uint32_t intersect_min(uint32_t *win, uint32_t av, const uint32_t *__restrict__ ha,
                                                  const D *__restrict__ da, uint32_t la,
                                                  const uint32_t *__restrict__ hb, const D *__restrict__ db,
                                                  uint32_t lb, uint32_t d, int lane)
{
    window_ready();
    if (la == 0) return d;
    uint32_t ia = 0, ib = 0;
    for (;;) {
        uint32_t lo = 0;
#pragma unroll
        for (uint32_t step = QWIN / 2; step > 0; step >>= 1)
            if (win[lo + step - 1] < av) lo += step;
        if (ia + lane < la && win[lo] == av) d = min(d, (uint32_t)(int32_t)da[ia + lane] + (uint32_t)(int32_t)db[ib + lo]);
        const uint32_t amax = __shfl_sync(FULL, av, (int)(min(la - ia, 32u) - 1));
        if (lb - ib > QWIN && amax > win[QWIN - 1]) {
            ib += QWIN;
            __syncwarp();
            stage_window(win, hb + ib, lb - ib, lane);
            window_ready();
        } else {
            ia += 32;
            if (ia >= la) return d;
            av = ia + lane < la ? __ldg(ha + ia + lane) : 0xfffffffeu;
        }
    }
}

// Distance between original ids x and y on an unweighted index (every lane
// returns it).  `bytes` accumulates the algorithmic bytes read (lane 0 only).
__device__ __forceinline__ uint8_t query_unw_pair(const IndexView &v, uint32_t x, uint32_t y, int lane, QueryScratch &qs,
                                                  unsigned long long &bytes)
{
    if (x >= v.n || y >= v.n) return (x == y) ? 0 : U8_INF;
    uint32_t rx = v.rank ? v.rank[x] : x;
    uint32_t ry = v.rank ? v.rank[y] : y;
    uint64_t oa = v.off[rx], ob = v.off[ry];
    uint32_t la = (uint32_t)(v.off[rx + 1] - oa), lb = (uint32_t)(v.off[ry + 1] - ob);
    // BP part: lane i takes roots i and i + 32.  A root takes part when
    // 2 <= td <= 257 (the unsigned td - 2 <= 255) and gives td, td - 1 or
    // td - 2.  With mt the least taking-part td, a root of td >= mt + 2 gives at least
    // mt and cannot lower the minimum that a root of td = mt gives, so the
    // sets are read only where td <= mt + 1 -- for no root at all when either
    // vertex reaches none.  They are loaded together with the first block of
    // the label lists, whose addresses became known at the same time.
    const uint8_t *pdx = v.bpd + (uint64_t)rx * v.K, *pdy = v.bpd + (uint64_t)ry * v.K;
    const uint32_t i0 = lane, i1 = lane + 32;
    const uint32_t t0 = i0 < v.K ? (uint32_t)pdx[i0] + (uint32_t)pdy[i0] : 0u;
    const uint32_t t1 = i1 < v.K ? (uint32_t)pdx[i1] + (uint32_t)pdy[i1] : 0u;
    const bool p0 = t0 - 2u <= (uint32_t)U8_INF, p1 = t1 - 2u <= (uint32_t)U8_INF;
    const uint32_t mt = __reduce_min_sync(FULL, min(p0 ? t0 : 0xffffu, p1 ? t1 : 0xffffu));
    // the roots to read, packed to the front (td << 6 | root): one per lane
    // and round, which needs half the registers of a lane's two roots at once
    const bool n0 = p0 && t0 <= mt + 1u, n1 = p1 && t1 <= mt + 1u;
    const uint32_t m0 = __ballot_sync(FULL, n0), m1 = __ballot_sync(FULL, n1);
    const uint32_t below = (1u << lane) - 1u, c0 = __popc(m0), cnt = c0 + __popc(m1);
    __syncwarp();  // the previous pair's list and window are done with
    if (n0) qs.root[__popc(m0 & below)] = (uint16_t)(t0 << 6 | i0);
    if (n1) qs.root[c0 + __popc(m1 & below)] = (uint16_t)(t1 << 6 | i1);
    bytes += (v.rank ? 8 : 0) + 32 + 2ull * v.K + 5ull * (la + lb) + 32ull * cnt;
    const uint64_t kx = (uint64_t)rx * v.K, ky = (uint64_t)ry * v.K;
    if (la > lb) {
        const uint64_t o = oa;
        const uint32_t l = la;
        oa = ob, la = lb;
        ob = o, lb = l;
    }
    stage_window(qs.win, v.hub + ob, lb, lane);
    const uint32_t av = (uint32_t)lane < la ? __ldg(v.hub + oa + lane) : 0xfffffffeu;
    __syncwarp();
    uint32_t d = U8_INF;
#pragma unroll 1
    for (uint32_t c = lane; c < cnt; c += 32) {
        const uint32_t i = qs.root[c] & 63u, td = qs.root[c] >> 6;
        const ulonglong2 sx = reinterpret_cast<const ulonglong2 *>(v.bps)[kx + i];
        const ulonglong2 sy = reinterpret_cast<const ulonglong2 *>(v.bps)[ky + i];
        d = min(d, td - ((sx.x & sy.x) ? 2u : (((sx.x & sy.y) | (sx.y & sy.x)) ? 1u : 0u)));
    }
    d = intersect_min<uint8_t>(qs.win, av, v.hub + oa, v.dist8 + oa, la, v.hub + ob, v.dist8 + ob, lb, d, lane);
    d = __reduce_min_sync(FULL, d);
    return (uint8_t)(d >= (uint32_t)(U8_INF - 2) ? U8_INF : d);
}

// Same on a weighted index (int16 distances, I16_INF = unreachable).
__device__ __forceinline__ int16_t query_w_pair(const IndexView &v, uint32_t x, uint32_t y, int lane, QueryScratch &qs,
                                                unsigned long long &bytes)
{
    if (x >= v.n || y >= v.n) return (x == y) ? 0 : I16_INF;
    const uint32_t rx = v.rank ? v.rank[x] : x;
    const uint32_t ry = v.rank ? v.rank[y] : y;
    uint64_t oa = v.off[rx], ob = v.off[ry];
    uint32_t la = (uint32_t)(v.off[rx + 1] - oa), lb = (uint32_t)(v.off[ry + 1] - ob);
    if (la > lb) {
        const uint64_t o = oa;
        const uint32_t l = la;
        oa = ob, la = lb;
        ob = o, lb = l;
    }
    __syncwarp();
    stage_window(qs.win, v.hub + ob, lb, lane);
    const uint32_t av = (uint32_t)lane < la ? __ldg(v.hub + oa + lane) : 0xfffffffeu;
    uint32_t d = (uint32_t)I16_INF;
    d = intersect_min<int16_t>(qs.win, av, v.hub + oa, v.dist16 + oa, la, v.hub + ob, v.dist16 + ob, lb, d, lane);
    d = __reduce_min_sync(FULL, d);
    bytes += (v.rank ? 8 : 0) + 32 + 6ull * (la + lb);
    return (int16_t)(d >= (uint32_t)(I16_INF - 2) ? I16_INF : d);
}

}  // namespace
}  // namespace pado
