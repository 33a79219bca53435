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
// minimum (see query_unw_pair).  The two hub-sorted label lists are
// intersected in registers when the longer one has at most 32 entries (lane i
// searches its a-hub among the b-hubs by shuffles), else 32 entries of the shorter
// list at a time in a window of the longer one in shared memory.  The result is a
// warp min-reduction.  Everything is integer arithmetic with the reference's
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

// A pair's ranks, label list lengths and offsets, the shorter list first (the BP
// part does not care which vertex is which).  rx = NO_PAIR: an id is out of range and
// ry is the answer.
constexpr uint32_t NO_PAIR = 0xffffffffu;
struct __align__(16) PairHead {
    uint32_t rx, ry, la, lb;
    uint64_t oa, ob;
};

__device__ __forceinline__ PairHead pair_head(const IndexView &v, uint32_t x, uint32_t y, uint32_t inf)
{
    PairHead h{NO_PAIR, x == y ? 0u : inf, 0, 0, 0, 0};
    if (x >= v.n || y >= v.n) return h;
    h.rx = v.rank ? v.rank[x] : x;
    h.ry = v.rank ? v.rank[y] : y;
    h.oa = v.off[h.rx];
    h.ob = v.off[h.ry];
    h.la = (uint32_t)(v.off[h.rx + 1] - h.oa);
    h.lb = (uint32_t)(v.off[h.ry + 1] - h.ob);
    if (h.la > h.lb) {
        const uint32_t r = h.rx, l = h.la;
        const uint64_t o = h.oa;
        h.rx = h.ry, h.la = h.lb, h.oa = h.ob;
        h.ry = r, h.lb = l, h.ob = o;
    }
    return h;
}

// Starts the reads of a pair's first hubs: lane i's of the shorter list (av), and the
// longer list's, in a register (bv) when it has at most 32, else into the window.
// A pair with an empty list has no common hub and reads nothing.
__device__ __forceinline__ void load_hubs(const IndexView &v, const PairHead &h, int lane, uint32_t *win, uint32_t &av,
                                          uint32_t &bv)
{
    av = 0xfffffffeu;
    bv = 0xffffffffu;
    if (h.la == 0) return;
    if (h.lb > 32)
        stage_window(win, v.hub + h.ob, h.lb, lane);
    else if ((uint32_t)lane < h.lb)
        bv = __ldg(v.hub + h.ob + lane);
    if ((uint32_t)lane < h.la) av = __ldg(v.hub + h.oa + lane);
}

// Minimum of da(h) + db(h) over hubs h common to the two sorted lists, and d, for
// lists of at most 32 entries.
template <typename D>
__device__ __forceinline__ uint32_t intersect_short(uint32_t av, uint32_t bv, const D *__restrict__ da,
                                                    const D *__restrict__ db, uint32_t d, int lane)
{
    uint32_t lo = 0;
#pragma unroll
    for (uint32_t step = 16; step > 0; step >>= 1)
        if (__shfl_sync(FULL, bv, lo + step - 1) < av) lo += step;
    if (__shfl_sync(FULL, bv, lo) == av) d = min(d, (uint32_t)(int32_t)da[lane] + (uint32_t)(int32_t)db[lo]);
    return d;
}

// The same for any two lists, la <= lb and not empty: the window holds (or
// awaits) b's first entries.  32 hubs of a at a time are searched in the window
// (7 steps in shared memory); whichever side ends at the lower hub moves on.
// AHEAD, for batches that the chain of loads bounds: a's next hubs are read before the
// search and the distances of a match are added a turn later, so that a turn
// waits for one round trip instead of two (1,000 pairs, us: weighted complete
// graph of 1,000 vertices, every hub shared, 24.7 -> 18.7; weighted random graph of
// 6,000, 264 labels a vertex, 12.6 -> 10.5; 20,000 pairs of it 29.3 -> 26.0).  Where
// the instructions bound it the plain form is as fast and needs fewer registers
// (2M weighted pairs, s16: 338 us; 354 with both ahead).
template <bool AHEAD, typename D>
__device__ __forceinline__ uint32_t intersect_min(uint32_t *win, uint32_t av, const uint32_t *__restrict__ ha,
                                                  const D *__restrict__ da, uint32_t la,
                                                  const uint32_t *__restrict__ hb, const D *__restrict__ db,
                                                  uint32_t lb, uint32_t d, int lane)
{
    window_ready();
    uint32_t ia = 0, ib = 0, xa = d, xb = 0;
    for (;;) {
        uint32_t an = 0;
        if (AHEAD) an = ia + 32 + lane < la ? __ldg(ha + ia + 32 + lane) : 0xfffffffeu;
        uint32_t lo = 0;
#pragma unroll
        for (uint32_t step = QWIN / 2; step > 0; step >>= 1)
            if (win[lo + step - 1] < av) lo += step;
        if (AHEAD) d = min(d, xa + xb);
        if (ia + lane < la && win[lo] == av) {
            xa = (uint32_t)(int32_t)da[ia + lane];
            xb = (uint32_t)(int32_t)db[ib + lo];
            if (!AHEAD) d = min(d, xa + xb);
        }
        const uint32_t amax = __shfl_sync(FULL, av, (int)(min(la - ia, 32u) - 1));
        if (lb - ib > QWIN && amax > win[QWIN - 1]) {
            ib += QWIN;
            __syncwarp();
            stage_window(win, hb + ib, lb - ib, lane);
            window_ready();
        } else {
            ia += 32;
            if (ia >= la) return AHEAD ? min(d, xa + xb) : d;
            av = AHEAD ? an : ia + lane < la ? __ldg(ha + ia + lane) : 0xfffffffeu;
        }
    }
}

// Distance of a pair on an unweighted index (every lane returns it).  `bytes`
// accumulates the algorithmic bytes read (lane 0 only).
template <bool AHEAD>
__device__ __forceinline__ uint8_t query_unw_pair(const IndexView &v, const PairHead &h, int lane, QueryScratch &qs,
                                                  unsigned long long &bytes)
{
    if (h.rx == NO_PAIR) return (uint8_t)h.ry;
    __syncwarp();  // the previous pair's list and window are done with
    uint32_t av, bv;
    load_hubs(v, h, lane, qs.win, av, bv);
    // BP part: lane i takes roots i and i + 32.  A root takes part when
    // 2 <= td <= 257 (the unsigned td - 2 <= 255; absent roots read as 0) and
    // gives td, td - 1 or td - 2.  With m the least td - 2, a root of td - 2 >= m + 2
    // gives at least m + 2 and cannot lower the minimum that the least root gives, so the
    // sets are read only where td - 2 <= m + 1 -- for no root at all when either
    // vertex reaches none.
    const uint64_t kx = (uint64_t)h.rx * v.K, ky = (uint64_t)h.ry * v.K;
    const uint8_t *pdx = v.bpd + kx, *pdy = v.bpd + ky;
    const uint32_t i0 = lane, i1 = lane + 32;
    const uint32_t e0 = (i0 < v.K ? (uint32_t)pdx[i0] + (uint32_t)pdy[i0] : 0u) - 2u;
    const uint32_t e1 = (i1 < v.K ? (uint32_t)pdx[i1] + (uint32_t)pdy[i1] : 0u) - 2u;
    const uint32_t lim = min(__reduce_min_sync(FULL, min(e0, e1)) + 1u, (uint32_t)U8_INF);
    // the roots to read, packed to the front (td - 2 << 6 | root): one per lane
    // and round, which needs half the registers of a lane's two roots at once
    const bool n0 = e0 <= lim, n1 = e1 <= lim;
    const uint32_t m0 = __ballot_sync(FULL, n0), m1 = __ballot_sync(FULL, n1);
    const uint32_t below = (1u << lane) - 1u, c0 = __popc(m0), cnt = c0 + __popc(m1);
    if (n0) qs.root[__popc(m0 & below)] = (uint16_t)(e0 << 6 | i0);
    if (n1) qs.root[c0 + __popc(m1 & below)] = (uint16_t)(e1 << 6 | i1);
    bytes += (v.rank ? 8 : 0) + 32 + 2ull * v.K + 5ull * (h.la + h.lb) + 32ull * cnt;
    __syncwarp();
    uint32_t d = U8_INF;
#pragma unroll 1
    for (uint32_t c = lane; c < cnt; c += 32) {
        const uint32_t i = qs.root[c] & 63u, td = (qs.root[c] >> 6) + 2u;
        const ulonglong2 sx = reinterpret_cast<const ulonglong2 *>(v.bps)[kx + i];
        const ulonglong2 sy = reinterpret_cast<const ulonglong2 *>(v.bps)[ky + i];
        d = min(d, td - ((sx.x & sy.x) ? 2u : (((sx.x & sy.y) | (sx.y & sy.x)) ? 1u : 0u)));
    }
    if (h.la)
        d = h.lb <= 32 ? intersect_short<uint8_t>(av, bv, v.dist8 + h.oa, v.dist8 + h.ob, d, lane)
                       : intersect_min<AHEAD, uint8_t>(qs.win, av, v.hub + h.oa, v.dist8 + h.oa, h.la,
                                                       v.hub + h.ob, v.dist8 + h.ob, h.lb, d, lane);
    d = __reduce_min_sync(FULL, d);
    return (uint8_t)(d >= (uint32_t)(U8_INF - 2) ? U8_INF : d);
}

// Same on a weighted index (int16 distances, I16_INF = unreachable).
template <bool AHEAD>
__device__ __forceinline__ int16_t query_w_pair(const IndexView &v, const PairHead &h, int lane, QueryScratch &qs,
                                                unsigned long long &bytes)
{
    if (h.rx == NO_PAIR) return (int16_t)h.ry;
    bytes += (v.rank ? 8 : 0) + 32 + 6ull * (h.la + h.lb);
    if (h.la == 0) return I16_INF;
    __syncwarp();
    uint32_t av, bv, d = (uint32_t)I16_INF;
    load_hubs(v, h, lane, qs.win, av, bv);
    d = h.lb <= 32 ? intersect_short<int16_t>(av, bv, v.dist16 + h.oa, v.dist16 + h.ob, d, lane)
                   : intersect_min<AHEAD, int16_t>(qs.win, av, v.hub + h.oa, v.dist16 + h.oa, h.la,
                                                   v.hub + h.ob, v.dist16 + h.ob, h.lb, d, lane);
    d = __reduce_min_sync(FULL, d);
    return (int16_t)(d >= (uint32_t)(I16_INF - 2) ? I16_INF : d);
}

}  // namespace
}  // namespace pado
