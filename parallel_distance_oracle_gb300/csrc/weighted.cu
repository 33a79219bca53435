// weighted.cu -- batched pruned relaxation labeling for weighted graphs.
//
// Restates WeightedVertexCentricPLL (reference
// includes/pado_weighted_unv_unp.h:281-1526; OpenMP variant
// includes/pado_weighted_unv_para.h:305-1706).  Per batch of B consecutive
// ranks [s, e) (every vertex is a root; there are no BP labels):
//   initialize (:281-330): roots_labels_buffer[c][h] = d for each committed
//     label (h, d) of root c, buffer[c][c] = 0; each root holds the temporary
//     label (c, 0) and is active.
//   rounds until nothing is active:
//     send (:409-474): an active head h relaxes every root c it accepted in the
//       previous round to each neighbour t > c (lists are descending; t <= s
//       ends the scan): m = (int16)(d_h(c) + w(h, t)) is kept when
//       m < dists_table[t][c] and m < this round's best for (t, c);
//       dists_table[t][c] becomes the round minimum.
//     check (:476-870, :1300-1345): candidate (t, c, m) is pruned when
//       (1) some committed label (h, d) of t has buffer[c][h] finite and
//           d + buffer[c][h] <= m, or
//       (2) some temporary label r < c of t gives d_t(r) + T[c][r] <= m, where
//           T is the temporary table of the vertex whose id is c's batch-local
//           index (:585) -- a no-op after batch 0, since those vertices hold no
//           temporary labels then.
//       Pruned with a smaller covering value q lowers dists_table[t][c] to q.
//       Otherwise t's temporary label for c becomes m and t is active.
//   filter (:1052-1184): drop temporary (v, c) when a temporary r < c of v has
//     d_v(r) <= d_v(c), d_c(r) <= d_v(c) and d_v(r) + d_c(r) <= d_v(c).
//   update_index (:913-950): append the survivors (hub = c's rank, int16 d).
// Device schedule: the reference runs these phases in queue order on one
// thread; here each round is level-synchronous -- all candidates of a round
// are checked against the temporary labels as they stood when the round
// started, and the filter reads the pre-filter values.  The CPU restatement of
// exactly this schedule (the oracle's snapshot mode) produced byte-identical
// label sets to the reference on every graph it was compared on.
//
// Device mapping: as in the unweighted labeler -- the tails of the active
// heads are stamped and listed, and a pull runs a warp per tail that owns the
// tail's rows of dists_table / temporary labels for the round: it min-reduces
// the incoming relaxations per root in shared memory, walks checks (1) and (2)
// per candidate (list entries across the lanes, a ballot for the first
// covering entry), and commits.  The previous round's accepted (root,
// distance) pairs of each vertex are read from a parity-double-buffered log,
// so heads can be read while their owners accept new roots.  dists_table
// entries carry a batch stamp and never need resetting.
//
// Schedule: one persistent cooperative launch (w_loop_kernel) runs every
// batch with a bounded grid barrier between phases instead of a kernel launch
// and a host round trip each: start (the previous batch's roots' temporary
// rows cleared; root tables; the roots mark the first round's tails), one
// phase per round (the pull; a tail that accepts marks the next round's tails
// itself; batch 0 takes a snapshot phase first; a round with heavy tails takes
// a second phase for their checks and commits), end (later batches: filter
// and commit each vertex in one phase; batch 0: filter, then the long lists'
// remaining chunks over the grid, then commit).  It returns to the host only
// to grow the round logs or the label pool (the failed tails or vertices are
// re-run exactly afterwards) or on an error.  PADO_LEVEL_LOOP=host selects the
// host-driven loop of separate kernels (mark, pull, filter, commit) instead.

#include <algorithm>
#include <climits>
#include <cstring>
#include <type_traits>

#include "grid_barrier.cuh"
#include "pado_internal.cuh"

namespace pado {
namespace {

constexpr unsigned FULL = 0xffffffffu;
// Warps of a pull block.  The loop takes blocks of eight where that leaves as many warps
// resident as blocks of four do (shared memory decides: B up to 700 or so, and B = 2048):
// half the blocks make the barriers cheaper (wrmat18, B = 512: a build 57.7 -> 55.2 ms).
// At B = 1000 sixteen warps per SM fit instead of twenty: 68.3 ms against 61.8.
constexpr int WPULL_WARPS = 4, WLOOP_WARPS = 8;
constexpr int32_t RMIN_EMPTY = INT_MAX;
// Tails of at least this degree are worked on by the whole grid: their heads
// in items of WITEM adjacency entries, then a block each (see WTails).  Where more
// than WHEAVY_MAX vertices reach it the degree is doubled until no more do: with
// thousands of tails as long as each other a warp each fills the grid, and the
// second phase only costs.  n random vertices of average degree 800, ms of the
// build with all of them split / none: n = 4,096 19.2 / 19.9 (B = 512) and
// 27.2 / 23.1 (B = 128), 8,192 72.3 / 77.6 and 113 / 92, 12,000 172 / 163 and
// 291 / 200; R-MAT s18/ef64 (12,616 vertices of 512 and more) 219 / 245, and 197 with
// those of 1,024 split.
constexpr uint32_t WHEAVY_DEG = 512, WHEAVY_MAX = 8192, WITEM = 64;
constexpr uint32_t WHEAVY_CLASSES = 23;  // degrees from WHEAVY_DEG << k to twice that, below 2^32
constexpr uint32_t WHEAVY_BIT = 0x80000000u;  // of tail_stamp (rounds stay far below 2^31)
constexpr int32_t HMIN_EMPTY = 0x7f7f7f7f;  // above every distance; a byte fill writes it

struct WDev {
    uint32_t n, B;
    const uint32_t *off;
    const uint32_t *adj;
    const uint8_t *w;
    uint32_t *pool_hub;
    int16_t *pool_dist;
    unsigned long long pool_cap;
    unsigned long long *pool_top;
    uint64_t *lab_off;
    uint32_t *lab_len;
    uint32_t *lab_cap;
    int16_t *buf;        // [B][n]  roots' committed labels
    int16_t *vd;         // [n][B]  temporary label distances
    uint16_t *vq;        // [n][B]  temporary label roots, first-acceptance order
    uint32_t *vq_len;    // n
    uint32_t *dt;        // [n][B]  (batch+1) << 16 | uint16 distance
    uint32_t *log[2];    // accepted (c << 16 | uint16 d) of each round, by parity
    unsigned long long log_cap;
    unsigned long long *log_top;  // [2]
    uint64_t *last_pos[2];
    uint32_t *last_cnt[2];
    uint32_t *last_min[2];
    uint32_t *act_stamp[2];  // by round parity: round id at which the vertex accepted roots
    uint32_t *tail_stamp;  // round for which the vertex was last marked; top bit: heavy
    int16_t *snap;       // [B][B] rows of vertices < B at round start (batch 0)
    uint64_t *rbase;     // [B] pool position of root c's labels when its buf row was filled
    uint32_t *rlen;      // [B] their count (the row's reset reads these, not the live list,
                         // which a commit in the same phase may extend or move)
    uint32_t *status;
    unsigned long long *work;
};

// The tails of one round, in one of three slots by round mod 3: light ones, a
// warp each, and, in the persistent loop, heavy ones with the items of their
// adjacency.  A heavy tail's relaxations are min-reduced per item in shared
// memory and then into its row of hmin; once all items are done a block
// checks and commits it.  A warp alone would bound the round: in the first batch
// of weighted R-MAT s18 a vertex of several thousand neighbours receives
// hundreds of roots from each, and one round took 18.3 ms for 148,000 tails (5.8
// now; the batch's eleven rounds 35.7 and 15.4).  Build loop by the limit: 57.5 ms
// from degree 256 on, 55.7 from 512 or 1,024; items of 32 entries 55.9.
struct WTails {
    uint32_t *light, *light_cnt;
    uint32_t *heavy = nullptr, *heavy_cnt = nullptr;
    uint2 *items = nullptr;  // (index in `heavy`, item number)
    uint32_t *items_cnt = nullptr;
};

__device__ __forceinline__ int32_t dt_get(const WDev &d, uint32_t t, uint32_t c, uint32_t stamp)
{
    const uint32_t x = d.dt[(uint64_t)t * d.B + c];
    return (x >> 16) == stamp ? (int32_t)(int16_t)(x & 0xffffu) : (int32_t)I16_INF;
}

__device__ __forceinline__ void dt_put(const WDev &d, uint32_t t, uint32_t c, uint32_t stamp, int32_t v)
{
    d.dt[(uint64_t)t * d.B + c] = (stamp << 16) | (uint32_t)(uint16_t)(int16_t)v;
}

__device__ __forceinline__ uint32_t warp_min_u32(uint32_t v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(FULL, v, o));
    return v;
}

__device__ __forceinline__ bool warp_reserve_w(const WDev &d, uint32_t v, uint32_t need, uint64_t &base, int lane)
{
    const uint32_t len = d.lab_len[v], cap = d.lab_cap[v];
    base = d.lab_off[v];
    if (need <= cap) return true;
    uint32_t ncap = max(max(2u * cap, need), 8u);
    ncap = (ncap + 7u) & ~7u;
    unsigned long long pos = 0;
    if (lane == 0) pos = atomicAdd(d.pool_top, (unsigned long long)ncap);
    pos = __shfl_sync(FULL, pos, 0);
    if (pos + ncap > d.pool_cap) return false;
    for (uint32_t j = lane; j < len; j += 32) {
        d.pool_hub[pos + j] = d.pool_hub[base + j];
        d.pool_dist[pos + j] = d.pool_dist[base + j];
    }
    __syncwarp();
    if (lane == 0) {
        d.lab_off[v] = pos;
        d.lab_cap[v] = ncap;
    }
    base = pos;
    return true;
}

// Vertices per class of degree, added to classes[WHEAVY_CLASSES].
__global__ void __launch_bounds__(256) w_heavy_count_kernel(const uint32_t *off, uint32_t n, uint32_t *classes)
{
    __shared__ uint32_t h[WHEAVY_CLASSES];
    if (threadIdx.x < WHEAVY_CLASSES) h[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const uint32_t k = (off[v + 1] - off[v]) / WHEAVY_DEG;
        if (k) atomicAdd(&h[31 - __clz(k)], 1u);
    }
    __syncthreads();
    if (threadIdx.x < WHEAVY_CLASSES && h[threadIdx.x]) atomicAdd(&classes[threadIdx.x], h[threadIdx.x]);
}

__global__ void __launch_bounds__(256) w_heavy_flag_kernel(const uint32_t *off, uint32_t n, const uint32_t *classes,
                                                           uint32_t *tail_stamp)
{
    uint64_t least = WHEAVY_DEG;
    uint32_t cnt = 0;
    for (uint32_t k = 0; k < WHEAVY_CLASSES; ++k) cnt += classes[k];
    for (uint32_t k = 0; cnt > WHEAVY_MAX; ++k, least *= 2) cnt -= classes[k];
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        tail_stamp[v] = off[v + 1] - off[v] >= least ? WHEAVY_BIT : 0u;
}

// A head h of round lid - 1 whose smallest accepted root is mn: its
// neighbours t > mn become tails of round lid (stamp lid), once each.  The
// adjacency is in descending order, so the walk stops at the first t <= mn.
// Called by whole warps; warp w of nw starts at chunk w.
__device__ __forceinline__ void w_mark_head(const WDev &d, uint32_t h, uint32_t mn, uint32_t lid, const WTails &out,
                                            uint32_t w = 0, uint32_t nw = 1)
{
    const int lane = threadIdx.x & 31;
    const uint32_t e_end = d.off[h + 1];
    for (uint32_t e0 = d.off[h] + 32 * w; e0 < e_end; e0 += 32 * nw) {
        const uint32_t e = e0 + lane;
        const bool in = e < e_end;
        const uint32_t t = in ? d.adj[e] : 0u;
        const bool ok = in && t > mn;
        const uint32_t ts = ok ? d.tail_stamp[t] : lid, mark = lid | (ts & WHEAVY_BIT);
        if (ok && ts != mark && atomicExch(&d.tail_stamp[t], mark) != mark) {
            if (!(ts & WHEAVY_BIT) || !out.heavy) {
                out.light[agg_append(out.light_cnt)] = t;
            } else {
                const uint32_t slot = atomicAdd(out.heavy_cnt, 1u);
                const uint32_t k = (d.off[t + 1] - d.off[t] + WITEM - 1) / WITEM;
                const uint32_t at = atomicAdd(out.items_cnt, k);
                out.heavy[slot] = t;
                for (uint32_t j = 0; j < k; ++j) out.items[at + j] = make_uint2(slot, j);
            }
        }
        if (__ballot_sync(FULL, in && !ok)) break;
    }
}

// The temporary rows of the B vertices from s on (a batch's roots), back to
// INF (the rows are contiguous).
__device__ void w_rows_clear_phase(const WDev &d, uint32_t s)
{
    const uint32_t rows = min(d.B, d.n - s);
    const uint64_t tot = (uint64_t)rows * d.B;
    int16_t *p = d.vd + (uint64_t)s * d.B;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < tot; i += (uint64_t)gridDim.x * blockDim.x)
        p[i] = I16_INF;
}

// initialize_tables (pado_weighted_unv_unp.h:281-330).
// front: the batch roots as the heads of the first round (host-driven loop);
// with `tails` instead, the roots mark the first round's tails themselves.
__device__ void w_root_init_phase(const WDev &d, uint32_t s, uint32_t nroots, uint32_t lid0, uint32_t *front,
                                  uint32_t *front_cnt, uint32_t *news, uint32_t *news_cnt,
                                  const WTails *tails = nullptr)
{
    const int lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const int p = lid0 & 1;
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < nroots; c += nw) {
        const uint32_t r = s + c;
        int16_t *row = d.buf + (uint64_t)c * d.n;
        const uint64_t base = d.lab_off[r];
        const uint32_t len = d.lab_len[r];
        for (uint32_t j = lane; j < len; j += 32) row[d.pool_hub[base + j]] = d.pool_dist[base + j];
        __syncwarp();
        if (lane == 0) {
            d.rbase[c] = base;
            d.rlen[c] = len;
            row[r] = 0;
            d.vq[(uint64_t)r * d.B] = (uint16_t)c;
            d.vq_len[r] = 1;
            d.vd[(uint64_t)r * d.B + c] = 0;
            const unsigned long long pos = atomicAdd(&d.log_top[p], 1ull);
            d.log[p][pos] = (uint32_t)c << 16;
            d.last_pos[p][r] = pos;
            d.last_cnt[p][r] = 1;
            d.last_min[p][r] = r;
            d.act_stamp[p][r] = lid0;
            if (front) front[atomicAdd(front_cnt, 1u)] = r;
            news[atomicAdd(news_cnt, 1u)] = r;
        }
        if (tails) w_mark_head(d, r, r, lid0 + 1, *tails);
    }
}

__global__ void __launch_bounds__(256) w_root_init_kernel(WDev d, uint32_t s, uint32_t nroots, uint32_t lid0,
                                                          uint32_t *front, uint32_t *front_cnt, uint32_t *news,
                                                          uint32_t *news_cnt)
{
    w_root_init_phase(d, s, nroots, lid0, front, front_cnt, news, news_cnt);
}

__device__ void w_mark_phase(const WDev &d, const uint32_t *front, uint32_t cnt, uint32_t lid_cur, uint32_t *tails,
                             uint32_t *tails_cnt)
{
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const int pp = (lid_cur - 1) & 1;
    for (uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < cnt; q += nw) {
        const uint32_t h = front[q];
        w_mark_head(d, h, d.last_min[pp][h], lid_cur, WTails{tails, tails_cnt});
    }
}

__global__ void __launch_bounds__(256) w_mark_kernel(WDev d, const uint32_t *front, const uint32_t *front_cnt,
                                                     uint32_t lid_cur, uint32_t *tails, uint32_t *tails_cnt)
{
    w_mark_phase(d, front, *front_cnt, lid_cur, tails, tails_cnt);
}

__device__ void w_snap_phase(const WDev &d, uint32_t rows)
{
    const uint64_t tot = (uint64_t)rows * d.B;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < tot; i += (uint64_t)gridDim.x * blockDim.x)
        d.snap[i] = d.vd[i];
}

__global__ void w_snap_kernel(WDev d, uint32_t rows) { w_snap_phase(d, rows); }

// One chunk of an in-order covering walk (checks (1) and (2) of the pull):
// lane l holds list entry l of the chunk (`in`: the entry exists) with row
// index `key`, order key `kcmp` and distance `el`.  Each pending lane j (bit j
// of `pend`) has candidate root c_j, round minimum m_j and dists row
// base + c_j * stride; the first entry with kcmp < s + c_j whose row value is
// not INF and whose 16-bit sum with el is <= m_j covers it: lane j's r takes
// that sum and bit j leaves the returned mask.  Four candidates are gathered
// per step so that four loads are in flight.
__device__ __forceinline__ uint32_t cover_chunk(uint32_t pend, bool in, uint32_t key, uint32_t kcmp, int32_t el,
                                                const int16_t *base, uint64_t stride, uint32_t c, int32_t m,
                                                uint32_t s, int32_t &r)
{
    const int lane = threadIdx.x & 31;
    uint32_t todo = pend;
    while (todo) {
        int jj[4];
        int32_t mm[4], sk[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            jj[u] = todo ? __ffs(todo) - 1 : -1;
            todo &= todo - 1;  // (0 stays 0)
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t cu = __shfl_sync(FULL, c, jj[u] & 31);
            mm[u] = __shfl_sync(FULL, m, jj[u] & 31);
            sk[u] = (jj[u] >= 0 && in && kcmp < s + cu) ? (int32_t)base[(uint64_t)cu * stride + key] : (int32_t)I16_INF;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int32_t val = (int16_t)(el + sk[u]);
            const uint32_t cov = __ballot_sync(FULL, sk[u] != I16_INF && val <= mm[u]);
            if (cov) {
                const int32_t v = __shfl_sync(FULL, val, __ffs(cov) - 1);
                if (lane == jj[u]) r = v;
                pend &= ~(1u << jj[u]);
            }
        }
    }
    return pend;
}

// Round minimum of the relaxations arriving at t over the adjacency entries
// [e_begin, e_end), per root, in rmin (RMIN_EMPTY before); returns the number
// of roots touched, listed in `touched`.  Short logs of active heads are
// flattened into one item list over the lanes (inclusive counts sa), so one
// round of loads covers 32 entries whichever heads they belong to; logs of 32
// roots and more on average are walked head by head, without the search for
// each item's head and with the touched roots listed at the end (a fifth of the
// instructions per item; nearly all items of the first batch).
template <bool FIRST>
__device__ __forceinline__ uint32_t w_gather(const WDev &d, uint32_t t, uint32_t e_begin, uint32_t e_end, uint32_t s,
                                             uint32_t lid_cur, int32_t *rmin, uint16_t *touched,
                                             unsigned long long &bytes)
{
    const int lane = threadIdx.x & 31;
    const uint32_t below = (1u << lane) - 1u;
    const int pp = (lid_cur - 1) & 1;
    const uint32_t lid_prev = lid_cur - 1;
    uint32_t ntouch = 0;
    bool dense = false;
    for (uint32_t e0 = e_begin; e0 < e_end; e0 += 32) {
        const uint32_t e = e0 + lane;
        const bool in = e < e_end;
        const uint32_t h = in ? d.adj[e] : 0u;
        const bool ge = in && h >= s;
        // stamp, log position and size of every head: independent loads
        const uint32_t st = ge ? d.act_stamp[pp][h] : 0u;
        const uint64_t hp = ge ? d.last_pos[pp][h] : 0ull;
        const uint32_t hc = ge ? d.last_cnt[pp][h] : 0u;
        const bool act = ge && st == lid_prev;
        const int32_t wt = act ? (int32_t)d.w[e] : 0;
        const uint32_t ca = act ? hc : 0u;
        const uint64_t pa = act ? hp : 0ull;
        uint32_t sa = ca;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, sa, o);
            if (lane >= o) sa += y;
        }
        const uint32_t tot = __shfl_sync(FULL, sa, 31);
        uint32_t heads = __ballot_sync(FULL, act);
        if (d.work)
            bytes += __popc(__ballot_sync(FULL, in)) * 4ull + __popc(__ballot_sync(FULL, ge)) * 4ull +
                     __popc(__ballot_sync(FULL, act)) * 13ull + 4ull * tot;
        if (FIRST && tot >= 32u * __popc(heads) && tot) {
            dense = true;
            for (; heads; heads &= heads - 1) {
                const int k = __ffs(heads) - 1;
                const uint32_t *log = d.log[pp] + __shfl_sync(FULL, pa, k);
                const uint32_t cnt = __shfl_sync(FULL, ca, k);
                const int32_t ww = __shfl_sync(FULL, wt, k);
#pragma unroll 4
                for (uint32_t i = lane; i < cnt; i += 32) {
                    const uint32_t x = log[i], cr = x >> 16;
                    if (s + cr < t) atomicMin(&rmin[cr], (int32_t)(int16_t)((int32_t)(int16_t)(x & 0xffffu) + ww));
                }
            }
            __syncwarp();
            if (__ballot_sync(FULL, in && !ge)) break;
            continue;
        }
        for (uint32_t i0 = 0; i0 < tot; i0 += 32) {
            const uint32_t i = i0 + lane;
            uint32_t L = 0;  // head lane: the lanes whose inclusive count is <= i
#pragma unroll
            for (uint32_t step = 16; step > 0; step >>= 1)
                if (__shfl_sync(FULL, sa, L + step - 1) <= i) L += step;
            const uint64_t qp = __shfl_sync(FULL, pa, L);
            const uint32_t x0 = __shfl_sync(FULL, sa - ca, L);
            const int32_t ww = __shfl_sync(FULL, wt, L);
            bool fresh = false;
            uint32_t cr = 0;
            if (i < tot) {
                const uint32_t x = d.log[pp][qp + (i - x0)];
                cr = x >> 16;
                if (s + cr < t) {
                    const int32_t m = (int32_t)(int16_t)((int32_t)(int16_t)(x & 0xffffu) + ww);
                    fresh = atomicMin(&rmin[cr], m) == RMIN_EMPTY;
                }
            }
            // first touches of this round appended in lane order
            const uint32_t fm = __ballot_sync(FULL, fresh);
            if (fresh) touched[ntouch + __popc(fm & below)] = (uint16_t)cr;
            ntouch += __popc(fm);
        }
        if (__ballot_sync(FULL, in && !ge)) break;
    }
    __syncwarp();
    if (FIRST && dense) {
        ntouch = 0;
        for (uint32_t c0 = 0; c0 < d.B; c0 += 32) {
            const uint32_t c = c0 + lane;
            const bool have = c < d.B && rmin[c] != RMIN_EMPTY;
            const uint32_t m = __ballot_sync(FULL, have);
            if (have) touched[ntouch + __popc(m & below)] = (uint16_t)c;
            ntouch += __popc(m);
        }
        __syncwarp();
    }
    return ntouch;
}

// The checks of one group of touched roots of t, one per lane (root c when
// `have`, its round minimum in rmin): returns INT_MAX where the minimum is not
// below dists_table, INT_MIN where it is accepted, else the value that covers it.
template <bool FIRST>
__device__ __forceinline__ int32_t w_check_group(const WDev &d, uint32_t t, bool have, uint32_t c, const int32_t *rmin,
                                                 uint32_t s, uint32_t b, uint64_t cbase, uint32_t clen, uint32_t vql)
{
    const int lane = threadIdx.x & 31;
    const uint32_t B = d.B;
    // checks (1) and (2) walk a list in order and stop at its first
    // covering entry, as the reference's loops do.  The lanes hold 32
    // consecutive entries of the list; the candidates still looking
    // (bits of `pend`, one per lane of this group) are taken 4 at a
    // time, each gathering its own row at the 32 entries' keys, and a
    // ballot gives the first covering entry of each.  A candidate
    // leaves the walk at the chunk that covers it.
    int32_t m = 0, r = INT_MAX;
    if (have) {
        m = rmin[c];
        if (m < dt_get(d, t, c, b + 1)) r = INT_MIN;  // accepted unless pruned below
    }
    uint32_t pend = __ballot_sync(FULL, r == INT_MIN);
    // check (1): t's committed labels (hub, distance) against the
    // candidate roots' dists_table rows (buf[c][hub])
    for (uint32_t j0 = 0; j0 < clen && pend; j0 += 32) {
        const bool in = j0 + lane < clen;
        const uint32_t hl = in ? d.pool_hub[cbase + j0 + lane] : 0xffffffffu;
        const int32_t dl = in ? (int32_t)d.pool_dist[cbase + j0 + lane] : 0;
        pend = cover_chunk(pend, in, hl, hl, dl, d.buf, d.n, c, m, s, r);
    }
    // check (2) (batch 0 only): t's temporary labels in acceptance
    // order (root, distance) against the snapshot rows of the
    // candidates' temporary tables, roots before the candidate only
    if (FIRST) {
        const uint16_t *tqp = d.vq + (uint64_t)t * B;
        const int16_t *trow = d.vd + (uint64_t)t * B;
        for (uint32_t k0 = 0; k0 < vql && pend; k0 += 32) {
            const bool in = k0 + lane < vql;
            const uint32_t rl = in ? (uint32_t)tqp[k0 + lane] : 0u;
            const int32_t tl = in ? (int32_t)trow[rl] : 0;
            pend = cover_chunk(pend, in, rl, s + rl, tl, d.snap, B, c, m, s, r);
        }
    }
    return r;
}

// The pull of one round (send_messages, pado_weighted_unv_unp.h:409-870, as
// a pull).  Per-warp dynamic shared memory: rmin[B] int32, res[B] int32,
// touched[B] u16.
// tq: the round's work counter for dynamic tail claiming (null: static
// grid-stride assignment).  FIRST: batch 0, whose rounds are few, large and
// need check (2) and the walk of long logs; the other batches' many small rounds
// run a shorter instance.  front_next (may be null) collects the next round's
// heads; next (may be null) collects the next round's tails directly.
template <bool FIRST>
__device__ void w_pull_phase(const WDev &d, const uint32_t *tails, uint32_t cnt, uint32_t s, uint32_t b,
                             uint32_t lid_cur, uint32_t *front_next, uint32_t *front_next_cnt, uint32_t *news,
                             uint32_t *news_cnt, uint32_t *retry, uint32_t *retry_cnt, unsigned char *wsm,
                             uint32_t *tq = nullptr, const WTails *next = nullptr)
{
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    const uint32_t B = d.B;
    int32_t *rmin = reinterpret_cast<int32_t *>(wsm) + (size_t)w * B;
    const uint32_t bw = blockDim.x >> 5;
    int32_t *res = reinterpret_cast<int32_t *>(wsm) + (size_t)bw * B + (size_t)w * B;
    uint16_t *touched = reinterpret_cast<uint16_t *>(reinterpret_cast<int32_t *>(wsm) + (size_t)2 * bw * B) +
                        (size_t)w * B;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const int cp = lid_cur & 1;
    const uint32_t stamp = b + 1;
    for (uint32_t c = lane; c < B; c += 32) rmin[c] = RMIN_EMPTY;
    __syncwarp();
    unsigned long long bytes = 0;
    auto pull_tail = [&](const uint32_t t) {
        bytes += 8;
        // (a) round minimum of the relaxations arriving at t, per root
        const uint32_t ntouch = w_gather<FIRST>(d, t, d.off[t], d.off[t + 1], s, lid_cur, rmin, touched, bytes);
        if (ntouch == 0) return;
        // (b) candidates: round minimum below dists_table; checks (1) and (2)
        const uint64_t cbase = d.lab_off[t];
        const uint32_t clen = d.lab_len[t];
        const uint32_t vql = d.vq_len[t];
        uint32_t nacc = 0, nnew = 0, mnacc = 0xffffffffu;
        for (uint32_t i0 = 0; i0 < ntouch; i0 += 32) {
            const uint32_t i = i0 + lane;
            bool acc = false, isnew = false;
            const uint32_t c = i < ntouch ? touched[i] : 0u;
            const int32_t r = w_check_group<FIRST>(d, t, i < ntouch, c, rmin, s, b, cbase, clen, vql);
            if (i < ntouch) {
                if (r == INT_MIN) {
                    acc = true;
                    isnew = d.vd[(uint64_t)t * B + c] == I16_INF;
                    mnacc = min(mnacc, s + c);
                }
                res[i] = r;
            }
            nacc += __popc(__ballot_sync(FULL, acc));
            nnew += __popc(__ballot_sync(FULL, isnew));
        }
        mnacc = warp_min_u32(mnacc);
        // dists_table reads, committed-label scans (6 B each), accepted entries
        bytes += 4ull * ntouch + 12 + 6ull * clen * ntouch + 8ull * nacc;
        // (c) reserve the log slots for the accepted roots, then commit
        unsigned long long lpos = 0;
        if (nacc) {
            if (lane == 0) lpos = atomicAdd(&d.log_top[cp], (unsigned long long)nacc);
            lpos = __shfl_sync(FULL, lpos, 0);
            if (lpos + nacc > d.log_cap) {
                if (lane == 0) {
                    atomicOr(d.status, ST_POOL_RETRY);
                    retry[atomicAdd(retry_cnt, 1u)] = t;
                }
                for (uint32_t i = lane; i < ntouch; i += 32) rmin[touched[i]] = RMIN_EMPTY;
                __syncwarp();
                return;
            }
        }
        uint32_t accb = 0, newb = 0;
        for (uint32_t i0 = 0; i0 < ntouch; i0 += 32) {
            const uint32_t i = i0 + lane;
            bool acc = false, isnew = false;
            uint32_t c = 0;
            int32_t m = 0;
            if (i < ntouch) {
                c = touched[i];
                m = rmin[c];
                const int32_t r = res[i];
                if (r != INT_MAX) {
                    dt_put(d, t, c, stamp, m);
                    if (r == INT_MIN) {
                        acc = true;
                        isnew = d.vd[(uint64_t)t * B + c] == I16_INF;
                    } else if (r < m) {
                        dt_put(d, t, c, stamp, r);
                    }
                }
            }
            const uint32_t am = __ballot_sync(FULL, acc), nm = __ballot_sync(FULL, isnew);
            const uint32_t below = (1u << lane) - 1u;
            if (acc) {
                d.log[cp][lpos + accb + __popc(am & below)] = (c << 16) | (uint32_t)(uint16_t)(int16_t)m;
                d.vd[(uint64_t)t * B + c] = (int16_t)m;
            }
            if (isnew) d.vq[(uint64_t)t * B + vql + newb + __popc(nm & below)] = (uint16_t)c;
            accb += __popc(am);
            newb += __popc(nm);
        }
        for (uint32_t i = lane; i < ntouch; i += 32) rmin[touched[i]] = RMIN_EMPTY;
        __syncwarp();
        bytes += 4ull * ntouch;  // dists_table writes
        if (lane == 0) {
            if (nnew) {
                d.vq_len[t] = vql + nnew;
                if (vql == 0) news[atomicAdd(news_cnt, 1u)] = t;
            }
            if (nacc) {
                d.last_pos[cp][t] = lpos;
                d.last_cnt[cp][t] = nacc;
                d.last_min[cp][t] = mnacc;
                d.act_stamp[cp][t] = lid_cur;
                if (front_next) front_next[atomicAdd(front_next_cnt, 1u)] = t;
            }
        }
        __syncwarp();
        // t is a head of the next round: with `next` it marks that round's
        // tails itself (no separate mark phase)
        if (nacc && next) w_mark_head(d, t, mnacc, lid_cur + 1, *next);
    };
    if (tq) {
        for_claimed<0>(cnt, tq, [&](uint32_t q) { pull_tail(tails[q]); });
    } else {
        for (uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < cnt; q += nw) pull_tail(tails[q]);
    }
    if (d.work && lane == 0 && bytes) atomicAdd(&d.work[W_WPULL], bytes);
}

// The items of a round's heavy tails, a warp each: WITEM adjacency entries
// min-reduced in shared memory, then into the tail's row of hmin.
template <bool FIRST>
__device__ __noinline__ void w_heavy_items_phase(const WDev &d, const WTails &tl, uint32_t nitems, uint32_t s, uint32_t lid_cur,
                                    int32_t *hmin, uint32_t *claim, unsigned char *wsm)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t B = d.B;
    int32_t *rmin = reinterpret_cast<int32_t *>(wsm) + (size_t)w * B;
    uint16_t *touched = reinterpret_cast<uint16_t *>(reinterpret_cast<int32_t *>(wsm) + (size_t)2 * (blockDim.x >> 5) * B) +
                        (size_t)w * B;
    for (uint32_t c = lane; c < B; c += 32) rmin[c] = RMIN_EMPTY;
    __syncwarp();
    unsigned long long bytes = 0;
    for_claimed<0>(nitems, claim, [&](uint32_t q) {
        const uint2 it = tl.items[q];
        const uint32_t t = tl.heavy[it.x], e0 = d.off[t] + it.y * WITEM;
        const uint32_t ntouch = w_gather<FIRST>(d, t, e0, min(e0 + WITEM, d.off[t + 1]), s, lid_cur, rmin, touched, bytes);
        for (uint32_t i = lane; i < ntouch; i += 32) {
            const uint32_t c = touched[i];
            atomicMin(&hmin[(uint64_t)it.x * B + c], rmin[c]);
            rmin[c] = RMIN_EMPTY;
        }
        __syncwarp();
    });
    if (d.work && lane == 0 && bytes) atomicAdd(&d.work[W_WPULL], bytes);
}

// The checks and commit of a round's heavy tails, a block each, once their
// items are done: what pull_tail does from (b) on, the groups of 32 touched
// roots spread over the block's warps.  Leaves the rows of hmin empty.
template <bool FIRST>
__device__ __noinline__ void w_heavy_finish_phase(const WDev &d, const uint32_t *heavy, uint32_t nheavy, uint32_t s, uint32_t b,
                                     uint32_t lid_cur, uint32_t *news, uint32_t *news_cnt, uint32_t *retry,
                                     uint32_t *retry_cnt, unsigned char *wsm, int32_t *hmin, const WTails &next)
{
    __shared__ uint32_t sum[5];  // touched, accepted, new, least accepted root, log room
    __shared__ unsigned long long slpos;
    __shared__ uint32_t gacc[MAX_BATCH / 32], gnew[MAX_BATCH / 32];  // per group: accepted and new lanes
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, cp = lid_cur & 1;
    const uint32_t B = d.B, below = (1u << lane) - 1u;
    int32_t *rmin = reinterpret_cast<int32_t *>(wsm);
    const uint32_t bw = blockDim.x >> 5;
    int32_t *res = rmin + (size_t)bw * B;
    uint16_t *touched = reinterpret_cast<uint16_t *>(rmin + (size_t)2 * bw * B);
    for (uint32_t q = blockIdx.x; q < nheavy; q += gridDim.x) {
        const uint32_t t = heavy[q];
        int32_t *row = hmin + (uint64_t)q * B;
        __syncthreads();  // the previous tail's shared state is done with
        for (uint32_t c = threadIdx.x; c < B; c += blockDim.x) {
            const int32_t x = __ldcg(row + c);
            rmin[c] = x == HMIN_EMPTY ? RMIN_EMPTY : x;
            if (x != HMIN_EMPTY) row[c] = HMIN_EMPTY;
        }
        if (threadIdx.x < 5) sum[threadIdx.x] = threadIdx.x == 3 ? 0xffffffffu : threadIdx.x == 4 ? 1u : 0u;
        __syncthreads();
        if (w == 0) {
            uint32_t k = 0;
            for (uint32_t c0 = 0; c0 < B; c0 += 32) {
                const uint32_t c = c0 + lane;
                const bool have = c < B && rmin[c] != RMIN_EMPTY;
                const uint32_t m = __ballot_sync(FULL, have);
                if (have) touched[k + __popc(m & below)] = (uint16_t)c;
                k += __popc(m);
            }
            if (lane == 0) sum[0] = k;
        }
        __syncthreads();
        const uint32_t ntouch = sum[0], ng = (ntouch + 31) / 32;
        const uint64_t cbase = d.lab_off[t];
        const uint32_t clen = d.lab_len[t], vql = d.vq_len[t];
        for (uint32_t g = w; g < ng; g += bw) {
            const uint32_t i = g * 32 + lane;
            const uint32_t c = i < ntouch ? touched[i] : 0u;
            const int32_t r = w_check_group<FIRST>(d, t, i < ntouch, c, rmin, s, b, cbase, clen, vql);
            if (i < ntouch) res[i] = r;
            const bool acc = i < ntouch && r == INT_MIN;
            const bool isnew = acc && d.vd[(uint64_t)t * B + c] == I16_INF;
            const uint32_t am = __ballot_sync(FULL, acc), nm = __ballot_sync(FULL, isnew);
            const uint32_t mn = warp_min_u32(acc ? s + c : 0xffffffffu);
            if (lane == 0) {
                gacc[g] = am;
                gnew[g] = nm;
                atomicAdd(&sum[1], (uint32_t)__popc(am));
                atomicAdd(&sum[2], (uint32_t)__popc(nm));
                atomicMin(&sum[3], mn);
            }
        }
        __syncthreads();
        const uint32_t nacc = sum[1], nnew = sum[2], mnacc = sum[3];
        if (threadIdx.x == 0) {
            if (d.work) atomicAdd(&d.work[W_WPULL], 8ull * ntouch + 12 + 6ull * clen * ntouch + 8ull * nacc);
            if (nacc) {
                slpos = atomicAdd(&d.log_top[cp], (unsigned long long)nacc);
                if (slpos + nacc > d.log_cap) {  // re-run as a light tail after the log grows
                    sum[4] = 0;
                    atomicOr(d.status, ST_POOL_RETRY);
                    retry[atomicAdd(retry_cnt, 1u)] = t;
                }
            }
        }
        __syncthreads();
        if (!sum[4]) continue;  // uniform; nothing committed
        const unsigned long long lpos = slpos;
        for (uint32_t g = w; g < ng; g += bw) {
            // accepted and new roots of the groups before g
            uint32_t accb = 0, newb = 0;
            for (uint32_t j = lane; j < g; j += 32) {
                accb += __popc(gacc[j]);
                newb += __popc(gnew[j]);
            }
            accb = __reduce_add_sync(FULL, accb);
            newb = __reduce_add_sync(FULL, newb);
            const uint32_t i = g * 32 + lane;
            if (i < ntouch) {
                const uint32_t c = touched[i];
                const int32_t m = rmin[c], r = res[i];
                if (r != INT_MAX) dt_put(d, t, c, b + 1, r != INT_MIN && r < m ? r : m);
                if (gacc[g] >> lane & 1u) {
                    d.log[cp][lpos + accb + __popc(gacc[g] & below)] = (c << 16) | (uint32_t)(uint16_t)(int16_t)m;
                    d.vd[(uint64_t)t * B + c] = (int16_t)m;
                }
                if (gnew[g] >> lane & 1u) d.vq[(uint64_t)t * B + vql + newb + __popc(gnew[g] & below)] = (uint16_t)c;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            if (nnew) {
                d.vq_len[t] = vql + nnew;
                if (vql == 0) news[atomicAdd(news_cnt, 1u)] = t;
            }
            if (nacc) {
                d.last_pos[cp][t] = lpos;
                d.last_cnt[cp][t] = nacc;
                d.last_min[cp][t] = mnacc;
                d.act_stamp[cp][t] = lid_cur;
            }
        }
        if (nacc) w_mark_head(d, t, mnacc, lid_cur + 1, next, w, bw);
    }
}

__global__ void __launch_bounds__(WPULL_WARPS * 32, 8) w_pull_kernel(WDev d, const uint32_t *tails, const uint32_t *tails_cnt,
                                                                  uint32_t s, uint32_t b, uint32_t lid_cur,
                                                                  uint32_t *front_next, uint32_t *front_next_cnt,
                                                                  uint32_t *news, uint32_t *news_cnt, uint32_t *retry,
                                                                  uint32_t *retry_cnt)
{
    extern __shared__ __align__(16) unsigned char wsm[];
    if (b == 0)
        w_pull_phase<true>(d, tails, *tails_cnt, s, b, lid_cur, front_next, front_next_cnt, news, news_cnt, retry,
                           retry_cnt, wsm);
    else
        w_pull_phase<false>(d, tails, *tails_cnt, s, b, lid_cur, front_next, front_next_cnt, news, news_cnt, retry,
                            retry_cnt, wsm);
}

// filter_out_labels (pado_weighted_unv_unp.h:1052-1184) on pre-filter values
// for the temporary labels i0 .. i0 + 31 of v: label c is dropped, by setting
// bit 15 of its vq slot, when some root r < c of v's list has
// d(v, r) <= d(v, c), d(c, r) <= d(v, c) and d(v, r) + d(c, r) <= d(v, c),
// d(c, r) read from root c's temporary row.  v's list is walked 32 entries at
// a time across the lanes; the labels still looking (bits of `pend`) are taken
// four at a time, each gathering its own row at the 32 entries' roots, and
// leave at the chunk that drops them (most leave in the first chunks: a lane per
// label, all walking the whole list, took 9.1 ms for the first batch of
// weighted R-MAT s18).  Bit 15 is masked off wherever a slot is read, so chunks
// of one v may run in different warps at once.
__device__ __forceinline__ void w_filter_chunk(const WDev &d, uint32_t v, uint32_t L, uint32_t i0, uint32_t s)
{
    const int lane = threadIdx.x & 31;
    const uint32_t B = d.B;
    uint16_t *vq = d.vq + (uint64_t)v * B;
    const int16_t *row = d.vd + (uint64_t)v * B;
    const int16_t *rows = d.vd + (uint64_t)s * B;  // the roots' temporary rows
    const uint32_t i = i0 + lane;
    const bool valid = i < L;
    uint32_t c = 0;
    int32_t dvc = 0;
    if (valid) {
        c = vq[i] & 0x7fffu;
        dvc = row[c];
    }
    uint32_t pend = __ballot_sync(FULL, valid);
    const uint32_t all = pend;
    for (uint32_t k0 = 0; k0 < L && pend; k0 += 32) {
        const bool in = k0 + lane < L;
        const uint32_t rl = in ? (uint32_t)(vq[k0 + lane] & 0x7fffu) : 0u;
        const int32_t dl = in ? (int32_t)row[rl] : 0;
        uint32_t todo = pend;
        while (todo) {
            int jj[4];
            int32_t mm[4], gg[4];
            bool ok[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                jj[u] = todo ? __ffs(todo) - 1 : -1;
                todo &= todo - 1;  // (0 stays 0)
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t cu = __shfl_sync(FULL, c, jj[u] & 31);
                mm[u] = __shfl_sync(FULL, dvc, jj[u] & 31);
                ok[u] = jj[u] >= 0 && in && rl < cu && dl <= mm[u];
                gg[u] = ok[u] ? (int32_t)rows[(uint64_t)cu * B + rl] : 0;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (__ballot_sync(FULL, ok[u] && gg[u] <= mm[u] && dl + gg[u] <= mm[u])) pend &= ~(1u << jj[u]);
        }
    }
    __syncwarp();
    if ((all & ~pend) >> lane & 1u) vq[i] |= 0x8000u;
    __syncwarp();
}

// update_index (pado_weighted_unv_unp.h:913-950) for one vertex v: append the
// unfiltered temporary labels in ascending root order, then clear v's
// temporary row unless `keep_row` (a batch root's row, which other vertices'
// filters still read; it is cleared when the next batch starts).
__device__ __forceinline__ void w_commit_one(const WDev &d, uint32_t v, uint32_t s, uint32_t *retry,
                                             uint32_t *retry_cnt, bool keep_row)
{
    const int lane = threadIdx.x & 31;
    const uint32_t B = d.B;
    const uint32_t L = d.vq_len[v];
    uint16_t *vq = d.vq + (uint64_t)v * B;
    int16_t *row = d.vd + (uint64_t)v * B;
    uint32_t keep = 0;
    for (uint32_t i = lane; i < L; i += 32) keep += (vq[i] & 0x8000u) ? 0u : 1u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) keep += __shfl_xor_sync(FULL, keep, o);
    const uint32_t len = d.lab_len[v];
    uint64_t base;
    if (keep && !warp_reserve_w(d, v, len + keep, base, lane)) {
        if (lane == 0) {
            atomicOr(d.status, ST_POOL_RETRY);
            retry[atomicAdd(retry_cnt, 1u)] = v;
        }
        return;
    }
    if (keep && L <= 32) {
        // one round: each root ranked by counting the smaller ones
        const bool mine = (uint32_t)lane < L && !(vq[lane] & 0x8000u);
        const uint32_t key = mine ? vq[lane] : 0xffffffffu;
        uint32_t rank = 0;
        for (uint32_t k = 0; k < L; ++k) rank += (__shfl_sync(FULL, key, k) < key) ? 1u : 0u;
        if (mine) {
            d.pool_hub[base + len + rank] = s + key;
            d.pool_dist[base + len + rank] = row[key];
        }
    } else if (keep) {
        // a bitmap of the batch's roots (B bits), read off in order
        __shared__ uint32_t bitmaps[8][MAX_BATCH / 32];
        uint32_t *bm = bitmaps[threadIdx.x >> 5];
        for (uint32_t x = lane; x < (B + 31) / 32; x += 32) bm[x] = 0;
        __syncwarp();
        for (uint32_t i = lane; i < L; i += 32)
            if (!(vq[i] & 0x8000u)) atomicOr(&bm[vq[i] >> 5], 1u << (vq[i] & 31));
        __syncwarp();
        uint64_t at = base + len;
        for (uint32_t x = 0; x < (B + 31) / 32; ++x) {
            const uint32_t m = bm[x];
            if (m >> lane & 1u) {
                const uint64_t o = at + __popc(m & ((1u << lane) - 1u));
                d.pool_hub[o] = s + x * 32 + lane;
                d.pool_dist[o] = row[x * 32 + lane];
            }
            at += __popc(m);
        }
    }
    __syncwarp();
    if (!keep_row)
        for (uint32_t i = lane; i < L; i += 32) row[vq[i] & 0x7fffu] = I16_INF;
    __syncwarp();
    if (lane == 0) {
        d.lab_len[v] = len + keep;
        d.vq_len[v] = 0;
    }
}

// Filter of a batch's new-label vertices, a warp per vertex.  With `heavy`,
// a warp filters only the first 32 labels of its vertex and lists the
// vertices with more, whose other chunks w_filter_heavy_phase spreads over the
// grid; with `commit`, each warp commits its vertex right after filtering it
// (roots' rows kept, see w_commit_one).
__device__ void w_filter_phase(const WDev &d, const uint32_t *news, uint32_t nnews, uint32_t s,
                               uint32_t *heavy = nullptr, uint32_t *heavy_cnt = nullptr, bool commit = false,
                               uint32_t nroots = 0, uint32_t *retry = nullptr, uint32_t *retry_cnt = nullptr)
{
    const int lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < nnews; q += nw) {
        const uint32_t v = news[q];
        const uint32_t L = d.vq_len[v];
        if (heavy) {
            w_filter_chunk(d, v, L, 0, s);
            if (L > 32 && lane == 0) heavy[atomicAdd(heavy_cnt, 1u)] = v;
        } else {
            for (uint32_t i0 = 0; i0 < L; i0 += 32) w_filter_chunk(d, v, L, i0, s);
        }
        if (commit) w_commit_one(d, v, s, retry, retry_cnt, v >= s && v - s < nroots);
    }
}

// The chunks after the first of the listed vertices, one (vertex, chunk) item
// per warp: item j is chunk 1 + j / nheavy of vertex heavy[j % nheavy].
__device__ void w_filter_heavy_phase(const WDev &d, const uint32_t *heavy, uint32_t nheavy, uint32_t s)
{
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const uint64_t items = (uint64_t)nheavy * ((d.B + 31) / 32 - 1);
    for (uint64_t j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < items; j += nw) {
        const uint32_t v = heavy[j % nheavy];
        const uint32_t i0 = 32u * (uint32_t)(1 + j / nheavy);
        const uint32_t L = d.vq_len[v];
        if (i0 < L) w_filter_chunk(d, v, L, i0, s);
    }
}

__global__ void __launch_bounds__(256) w_filter_kernel(WDev d, const uint32_t *news, uint32_t nnews, uint32_t s)
{
    w_filter_phase(d, news, nnews, s);
}

// reset_tables for the roots' buffer rows (pado_weighted_unv_unp.h:872-891):
// the entries the root init set, from the label list as it was then (a list
// slot keeps its first entries when the list grows or moves).
__device__ void w_buf_reset_phase(const WDev &d, uint32_t s, uint32_t nroots)
{
    const int lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < nroots; c += nw) {
        const uint32_t r = s + c;
        int16_t *row = d.buf + (uint64_t)c * d.n;
        const uint64_t base = d.rbase[c];
        const uint32_t len = d.rlen[c];
        for (uint32_t j = lane; j < len; j += 32) row[d.pool_hub[base + j]] = I16_INF;
        if (lane == 0) row[r] = I16_INF;
    }
}

__global__ void __launch_bounds__(256) w_buf_reset_kernel(WDev d, uint32_t s, uint32_t nroots)
{
    w_buf_reset_phase(d, s, nroots);
}

// update_index (pado_weighted_unv_unp.h:913-950) for a list of vertices.
__device__ void w_commit_phase(const WDev &d, const uint32_t *news, uint32_t nnews, uint32_t s, uint32_t *retry,
                               uint32_t *retry_cnt, uint32_t nroots = 0)
{
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < nnews; q += nw) {
        const uint32_t v = news[q];
        w_commit_one(d, v, s, retry, retry_cnt, v >= s && v - s < nroots);
    }
}

__global__ void __launch_bounds__(256) w_commit_kernel(WDev d, const uint32_t *news, uint32_t nnews, uint32_t s,
                                                       uint32_t *retry, uint32_t *retry_cnt)
{
    w_commit_phase(d, news, nnews, s, retry, retry_cnt);
}

// The int16 tables start at INF (0x7fff, which no byte fill can write): 16
// bytes per thread and step, bound by the stores.  2 x 268 MB (n = 262,144,
// B = 512) take 0.09 ms; copies of a host array of INFs, one stream
// synchronisation per 2 MB, took 5.6 ms of every build.
__global__ void __launch_bounds__(256) w_fill_inf_kernel(int16_t *p, uint64_t cnt)
{
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x, tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint32_t inf2 = (uint32_t)I16_INF << 16 | (uint32_t)I16_INF;
    uint4 *p8 = reinterpret_cast<uint4 *>(p);  // the tables are whole allocations, so aligned
    for (uint64_t i = tid; i < cnt / 8; i += nth) p8[i] = make_uint4(inf2, inf2, inf2, inf2);
    for (uint64_t i = cnt / 8 * 8 + tid; i < cnt; i += nth) p[i] = I16_INF;
}

__global__ void __launch_bounds__(256) w_compact_kernel(WDev d, const uint64_t *fin_off, uint32_t *fin_hub,
                                                        int16_t *fin_dist)
{
    const int lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < d.n; v += nw) {
        const uint64_t base = d.lab_off[v], fo = fin_off[v];
        const uint32_t len = d.lab_len[v];
        for (uint32_t j = lane; j < len; j += 32) {
            fin_hub[fo + j] = d.pool_hub[base + j];
            fin_dist[fo + j] = d.pool_dist[base + j];
        }
    }
}

// ---------------------------------------------------------------------------
// Persistent loop.  Every block keeps the loop state in registers and derives
// the same transitions from the same post-barrier counters; the leader saves
// the state to WLoopCtl only when the launch returns.  Counters are reused by
// parity and cleared one phase ahead of their next use (see each site).
// ---------------------------------------------------------------------------
enum WPhase : uint32_t { WP_START = 0, WP_ROUND = 1, WP_PULL_RETRY = 2, WP_END = 3, WP_COMMIT_RETRY = 4, WP_DONE = 5 };
enum WExit : uint32_t { WX_RUNNING = 0, WX_DONE = 1, WX_NEED_LOG = 2, WX_NEED_POOL = 3, WX_STALL = 4 };

// Round lid reads slot lid % 3 of the tails and appends the next round's to
// slot (lid + 1) % 3 as its heads accept; the leader clears the third slot for
// the round after.
struct WLoopCtl {
    GridBar bar;
    uint32_t phase, b, lid;           // resume point: phase, batch, last stamp
    uint32_t rounds, levels;
    uint32_t news_cnt[2];
    struct Slot {                     // by round mod 3
        uint32_t light_cnt, heavy_cnt, items_cnt;
        uint32_t tq, iq;              // claims of light tails and of heavy tails' items
    } slot[3];
    uint32_t heavy_cnt;               // batch 0's vertices with more than 32 temporary labels
    uint32_t rr_cnt, retry_cnt, status, exit_code;
};

struct WLoopBufs {
    uint32_t *tails[3], *htails[3], *news[2];  // news by batch parity
    uint2 *items[3];
    int32_t *hmin;                 // a row of B minima per heavy tail, HMIN_EMPTY between rounds
    uint32_t *rr, *retry, *heavy;
    uint32_t nbatches;
};

// The heavy phases are functions of their own (the parameters in constant
// memory can be passed by reference): inlined, their registers made the many
// small rounds spill (55.5 ms against 54.1 ms on wrmat18).
__global__ void __launch_bounds__(WLOOP_WARPS * 32, 4) w_loop_kernel(const __grid_constant__ WDev d, WLoopCtl *c, const __grid_constant__ WLoopBufs bf)
{
    extern __shared__ __align__(16) unsigned char wsm[];
    const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
    GridSync sync(&c->bar, &c->status);
    uint32_t phase = vload(&c->phase), b = vload(&c->b), lid = vload(&c->lid);
    uint32_t rounds = vload(&c->rounds), levels = vload(&c->levels);
    auto save = [&](uint32_t ph, uint32_t ex) {
        if (leader) {
            c->phase = ph;
            c->b = b;
            c->lid = lid;
            c->rounds = rounds;
            c->levels = levels;
            c->exit_code = ex;
        }
    };
    auto tails_of = [&](uint32_t x) {
        WLoopCtl::Slot &t = c->slot[x];
        return WTails{bf.tails[x], &t.light_cnt, bf.htails[x], &t.heavy_cnt, bf.items[x], &t.items_cnt};
    };
    for (;;) {
        if (phase == WP_START) {
            if (b >= bf.nbatches) {
                save(WP_DONE, WX_DONE);
                return;
            }
            const uint32_t s = b * d.B, nr = min(d.B, d.n - s);
            const uint32_t lid0 = lid + 1;
            // news[b & 1], log[lid0 & 1] and the first round's tails slot
            // were cleared at the end of the previous batch; the roots mark
            // the first round's tails
            if (b > 0) w_rows_clear_phase(d, s - d.B);  // the previous batch's roots' temporary rows
            const WTails first = tails_of((lid0 + 1) % 3);
            w_root_init_phase(d, s, nr, lid0, nullptr, nullptr, bf.news[b & 1], &c->news_cnt[b & 1], &first);
            if (leader) {
                c->slot[(lid0 + 2) % 3] = {};      // filled by the first round
                d.log_top[(lid0 + 1) & 1] = 0;     // the first round's log
            }
            if (!sync.wait()) return;
            lid = lid0;
            rounds = 0;
            phase = WP_ROUND;
            continue;
        }
        if (phase == WP_ROUND || phase == WP_PULL_RETRY) {
            const uint32_t s = b * d.B, nr = min(d.B, d.n - s);
            const uint32_t lid_cur = lid + 1, tp = lid_cur % 3, tn = (lid_cur + 1) % 3;
            if (phase == WP_ROUND) {
                // Bellman-Ford rounds are bounded by the vertex count
                if (rounds > d.n + 2) {
                    save(WP_DONE, WX_STALL);
                    return;
                }
                if (b == 0) {
                    // check (2) reads the batch's temporary tables as of the round start
                    w_snap_phase(d, nr);
                    if (!sync.wait()) return;
                }
            }
            const WTails cur = tails_of(tp), next = tails_of(tn);
            const uint32_t nheavy = vload(cur.heavy_cnt), nitems = vload(cur.items_cnt), nlight = vload(cur.light_cnt);
            auto round = [&](auto first) {
                constexpr bool FIRST = decltype(first)::value;
                if (nheavy) w_heavy_items_phase<FIRST>(d, cur, nitems, s, lid_cur, bf.hmin, &c->slot[tp].iq, wsm);
                w_pull_phase<FIRST>(d, cur.light, nlight, s, b, lid_cur, nullptr, nullptr, bf.news[b & 1],
                                    &c->news_cnt[b & 1], bf.retry, &c->retry_cnt, wsm, &c->slot[tp].tq, &next);
                if (!nheavy) return true;
                if (!sync.wait()) return false;
                w_heavy_finish_phase<FIRST>(d, cur.heavy, nheavy, s, b, lid_cur, bf.news[b & 1], &c->news_cnt[b & 1],
                                            bf.retry, &c->retry_cnt, wsm, bf.hmin, next);
                return true;
            };
            if (!(b == 0 ? round(std::true_type()) : round(std::false_type()))) return;
            if (leader) {
                c->slot[(lid_cur + 2) % 3] = {};      // read by the previous round's pull
                d.log_top[(lid_cur + 1) & 1] = 0;     // the next round's log, last read by this pull
            }
            if (!sync.wait()) return;
            if (vload(&c->retry_cnt)) {
                save(WP_PULL_RETRY, WX_NEED_LOG);
                return;
            }
            ++levels;
            ++rounds;
            lid = lid_cur;
            phase = vload(next.light_cnt) + vload(next.heavy_cnt) ? WP_ROUND : WP_END;
            continue;
        }
        if (phase == WP_END || phase == WP_COMMIT_RETRY) {
            const uint32_t s = b * d.B, nr = min(d.B, d.n - s), nb = b & 1;
            if (phase == WP_END) {
                const uint32_t nn = vload(&c->news_cnt[nb]);
                if (leader) {
                    d.log_top[(lid + 1) & 1] = 0;  // the next batch's root log (read by the last pull)
                    c->news_cnt[nb ^ 1] = 0;       // the next batch's new-label list
                    c->slot[(lid + 2) % 3] = {};   // the next batch's first tails
                }
                if (b == 0) {
                    // batch 0 has vertices with hundreds of temporary labels:
                    // their chunks after the first are spread over the grid,
                    // and the commit follows once every filter is done
                    w_filter_phase(d, bf.news[nb], nn, s, bf.heavy, &c->heavy_cnt);
                    if (!sync.wait()) return;
                    w_filter_heavy_phase(d, bf.heavy, vload(&c->heavy_cnt), s);
                    w_buf_reset_phase(d, s, nr);
                    if (!sync.wait()) return;
                    w_commit_phase(d, bf.news[nb], nn, s, bf.retry, &c->retry_cnt);
                } else {
                    // filter and commit each vertex in one go; the roots'
                    // rows, read by other vertices' filters, are cleared when
                    // the next batch starts
                    w_filter_phase(d, bf.news[nb], nn, s, nullptr, nullptr, true, nr, bf.retry, &c->retry_cnt);
                    w_buf_reset_phase(d, s, nr);
                }
            } else {
                w_commit_phase(d, bf.rr, vload(&c->rr_cnt), s, bf.retry, &c->retry_cnt);
            }
            if (!sync.wait()) return;
            if (vload(&c->retry_cnt)) {
                save(WP_COMMIT_RETRY, WX_NEED_POOL);
                return;
            }
            ++b;
            phase = WP_START;
            continue;
        }
        save(WP_DONE, WX_STALL);  // unknown phase
        return;
    }
}

}  // namespace

LabelRun w_label(const DevGraph &g, uint32_t B, LabelStore &out, cudaStream_t s)
{
    LabelRun run;
    const uint32_t n = g.n;
    PADO_CHECK(B >= 1 && B <= MAX_BATCH, PADO_E_ARG, "batch size must be in [1, 2048]");
    PADO_CHECK(n < (1u << 31), PADO_E_ARG, "too many vertices");

    uint64_t cap = initial_pool_entries(n);
    uint64_t lcap = initial_log_entries(n, B);
    DBuf<uint32_t> pool_hub(cap);
    DBuf<int16_t> pool_dist(cap);
    DBuf<int16_t> buf((uint64_t)B * n), vd((uint64_t)n * B);
    DBuf<uint16_t> vq((uint64_t)n * B);
    DBuf<uint32_t> log0(lcap), log1(lcap);
    // the per-vertex arrays in two allocations: one that starts as zeros
    // (with dt: stamp 0 never matches a batch, stamps start at 1) and one
    // whose contents do not matter
    Arena zeros, ws;
    DBuf<unsigned long long> pool_top, log_top;
    DBuf<uint64_t> lab_off, last_pos0, last_pos1, rbase;
    DBuf<uint32_t> lab_len, lab_cap, act_stamp0, act_stamp1, tail_stamp, vq_len, dt, status, hclasses;
    DBuf<uint32_t> last_cnt0, last_cnt1, last_min0, last_min1, rlen, front0, front1, tails, tails2, tails3, retry, news,
        news2, rr, heavy, counters;
    DBuf<int16_t> snap;
    DBuf<WLoopCtl> ctl;
    zeros.add(pool_top, 1);
    zeros.add(log_top, 2);
    zeros.add(lab_off, n);
    for (DBuf<uint32_t> *x : {&lab_len, &lab_cap, &act_stamp0, &act_stamp1, &tail_stamp, &vq_len}) zeros.add(*x, n);
    zeros.add(dt, (uint64_t)n * B);
    zeros.add(status, 1);
    zeros.add(hclasses, WHEAVY_CLASSES);
    zeros.add(ctl, 1);
    ws.add(last_pos0, n);
    ws.add(last_pos1, n);
    for (DBuf<uint32_t> *x : {&last_cnt0, &last_cnt1, &last_min0, &last_min1, &front0, &front1, &tails, &tails2, &tails3,
                              &retry, &news, &news2, &rr, &heavy})
        ws.add(*x, n);
    ws.add(rbase, B);
    ws.add(rlen, B);
    ws.add(counters, 8);
    ws.add(snap, (uint64_t)B * B);
    // at most m / WHEAVY_DEG vertices are heavy, and WHEAVY_MAX, with m / WITEM whole
    // items and one partial each
    const uint64_t hcan = std::min<uint64_t>(n, g.m / WHEAVY_DEG);
    const uint64_t hmax = std::min<uint64_t>(hcan, WHEAVY_MAX) + 1, imax = g.m / WITEM + hmax;
    DBuf<int32_t> hmin;
    DBuf<uint32_t> ht[3];
    DBuf<uint2> hi[3];
    ws.add(hmin, hmax * B);
    for (int x = 0; x < 3; ++x) {
        ws.add(ht[x], hmax);
        ws.add(hi[x], imax);
    }
    zeros.commit();
    ws.commit();
    zeros.mem.fill_bytes(0, s);
    hmin.fill_bytes(0x7f, s);
    if (hcan > WHEAVY_MAX)  // else too few vertices for another degree
        PADO_LAUNCH("w_heavy_count_kernel", s,
                    w_heavy_count_kernel<<<grid_for(n, 256), 256, 0, s>>>(g.off.p, n, hclasses.p));
    if (n)
        PADO_LAUNCH("w_heavy_flag_kernel", s,
                    w_heavy_flag_kernel<<<grid_for(n, 256), 256, 0, s>>>(g.off.p, n, hclasses.p, tail_stamp.p));
    for (DBuf<int16_t> *t : {&buf, &vd})
        if (t->n)
            PADO_LAUNCH("w_fill_inf_kernel", s,
                        w_fill_inf_kernel<<<grid_for((t->n + 7) / 8, 256, 152u * 8u), 256, 0, s>>>(t->p, t->n));

    WDev d{};
    d.n = n;
    d.B = B;
    d.off = g.off.p;
    d.adj = g.adj.p;
    d.w = g.w.p;
    d.pool_hub = pool_hub.p;
    d.pool_dist = pool_dist.p;
    d.pool_cap = cap;
    d.pool_top = pool_top.p;
    d.lab_off = lab_off.p;
    d.lab_len = lab_len.p;
    d.lab_cap = lab_cap.p;
    d.buf = buf.p;
    d.vd = vd.p;
    d.vq = vq.p;
    d.vq_len = vq_len.p;
    d.dt = dt.p;
    d.log[0] = log0.p;
    d.log[1] = log1.p;
    d.log_cap = lcap;
    d.log_top = log_top.p;
    d.last_pos[0] = last_pos0.p;
    d.last_pos[1] = last_pos1.p;
    d.last_cnt[0] = last_cnt0.p;
    d.last_cnt[1] = last_cnt1.p;
    d.last_min[0] = last_min0.p;
    d.last_min[1] = last_min1.p;
    d.act_stamp[0] = act_stamp0.p;
    d.act_stamp[1] = act_stamp1.p;
    d.tail_stamp = tail_stamp.p;
    d.rbase = rbase.p;
    d.rlen = rlen.p;
    d.snap = snap.p;
    d.status = status.p;
    d.work = work_counters();

    const size_t pull_smem = (size_t)WPULL_WARPS * B * (4 + 4 + 2);
    PADO_CUDA(cudaFuncSetAttribute(w_pull_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pull_smem));

    struct Ctr { uint32_t front_next, tails, retry, news; unsigned long long top; unsigned long long ltop[2]; };
    Ctr ctr{}, *hc = &ctr;
    uint32_t *c_front[2] = {counters.p + 0, counters.p + 1};
    uint32_t *c_tails = counters.p + 2, *c_retry = counters.p + 3, *c_news = counters.p + 4;
    uint32_t *fronts[2] = {front0.p, front1.p};
    auto read_ctrs = [&](uint32_t *c_fn) {
        PADO_CUDA(cudaMemcpyAsync(&hc->front_next, c_fn, 4, cudaMemcpyDeviceToHost, s));
        PADO_CUDA(cudaMemcpyAsync(&hc->tails, c_tails, 4, cudaMemcpyDeviceToHost, s));
        PADO_CUDA(cudaMemcpyAsync(&hc->retry, c_retry, 4, cudaMemcpyDeviceToHost, s));
        PADO_CUDA(cudaMemcpyAsync(&hc->news, c_news, 4, cudaMemcpyDeviceToHost, s));
        PADO_CUDA(cudaMemcpyAsync(&hc->top, pool_top.p, 8, cudaMemcpyDeviceToHost, s));
        PADO_CUDA(cudaMemcpyAsync(&hc->ltop[0], log_top.p, 16, cudaMemcpyDeviceToHost, s));
        PADO_CUDA(cudaStreamSynchronize(s));
    };
    auto grow_pool = [&](unsigned long long need) {
        uint64_t ncap = std::max<uint64_t>(cap * 2, need + need / 2 + (1u << 20));
        DBuf<uint32_t> nh(ncap);
        DBuf<int16_t> nd(ncap);
        PADO_CUDA(cudaMemcpyAsync(nh.p, pool_hub.p, cap * 4, cudaMemcpyDeviceToDevice, s));
        PADO_CUDA(cudaMemcpyAsync(nd.p, pool_dist.p, cap * 2, cudaMemcpyDeviceToDevice, s));
        PADO_CUDA(cudaStreamSynchronize(s));
        pool_hub = std::move(nh);
        pool_dist = std::move(nd);
        cap = ncap;
        d.pool_hub = pool_hub.p;
        d.pool_dist = pool_dist.p;
        d.pool_cap = cap;
    };
    // Grow both round logs (the one being written and the one being read).
    auto grow_logs = [&](unsigned long long need) {
        uint64_t ncap = std::max<uint64_t>(lcap * 4, 2 * need);  // a growth costs a relaunch: grow far
        DBuf<uint32_t> n0(ncap), n1(ncap);
        PADO_CUDA(cudaMemcpyAsync(n0.p, log0.p, lcap * 4, cudaMemcpyDeviceToDevice, s));
        PADO_CUDA(cudaMemcpyAsync(n1.p, log1.p, lcap * 4, cudaMemcpyDeviceToDevice, s));
        PADO_CUDA(cudaStreamSynchronize(s));
        log0 = std::move(n0);
        log1 = std::move(n1);
        lcap = ncap;
        d.log[0] = log0.p;
        d.log[1] = log1.p;
        d.log_cap = lcap;
    };

    cudaEvent_t e0, e1;
    PADO_CUDA(cudaEventCreate(&e0));
    PADO_CUDA(cudaEventCreate(&e1));
    PADO_CUDA(cudaEventRecord(e0, s));
    uint32_t lid = 0;
    const uint32_t nbatches = (uint32_t)(((uint64_t)n + B - 1) / B);
    const char *loop_env = std::getenv("PADO_LEVEL_LOOP");
    const bool host_loop = loop_env && !strcmp(loop_env, "host");
    try {
        PADO_CHECK(nbatches < 65535u, PADO_E_ARG, "more than 65534 batches");
        if (!host_loop && n) {
            WLoopBufs bf{{tails.p, tails2.p, tails3.p}, {ht[0].p, ht[1].p, ht[2].p}, {news.p, news2.p},
                         {hi[0].p, hi[1].p, hi[2].p}, hmin.p, rr.p, retry.p, heavy.p, nbatches};
            const void *kfn = (const void *)w_loop_kernel;
            const size_t loop_smem = pull_smem * WLOOP_WARPS / WPULL_WARPS;
            PADO_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)loop_smem));
            int dev = 0, sms = 0, per_sm = 0, wide = 0;
            PADO_CUDA(cudaGetDevice(&dev));
            PADO_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
            PADO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, WPULL_WARPS * 32, pull_smem));
            PADO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&wide, kfn, WLOOP_WARPS * 32, loop_smem));
            PADO_CHECK(per_sm >= 1 || wide >= 1, PADO_E_CUDA, "weighted labeling loop kernel cannot be resident");
            const bool big = wide * WLOOP_WARPS >= per_sm * WPULL_WARPS;
            const int threads = 32 * (big ? WLOOP_WARPS : WPULL_WARPS);
            const unsigned grid = (unsigned)(sms * (big ? wide : per_sm));
            WLoopCtl h{};
            WLoopCtl *cptr = ctl.p;
            for (int launch = 0;; ++launch) {
                PADO_CHECK(launch < 512, PADO_E_NOMEM, "round log or label pool could not be grown enough");
                void *args[] = {&d, &cptr, &bf};
                PADO_LAUNCH("w_loop_kernel", s,
                            PADO_CUDA(cudaLaunchCooperativeKernel(kfn, grid, threads, args,
                                                                  big ? loop_smem : pull_smem, s)));
                PADO_CUDA(cudaMemcpyAsync(&h, ctl.p, sizeof(WLoopCtl), cudaMemcpyDeviceToHost, s));
                PADO_CUDA(cudaStreamSynchronize(s));
                if (h.status & ST_BARRIER_TIMEOUT)
                    throw Error(PADO_E_TIMEOUT, "weighted labeling loop: a grid barrier timed out");
                if (std::getenv("PADO_TRACE"))
                    fprintf(stderr, "weighted loop launch %d: exit %u at batch %u (retry %u)\n", launch, h.exit_code,
                            h.b, h.retry_cnt);
                if (h.exit_code == WX_DONE) break;
                if (h.exit_code == WX_STALL) throw Error(PADO_E_STATE, "relaxation did not converge");
                if (h.exit_code == WX_NEED_LOG) {
                    unsigned long long lt[2];
                    PADO_CUDA(cudaMemcpy(lt, log_top.p, 16, cudaMemcpyDeviceToHost));
                    grow_logs(lt[(h.lid + 1) & 1]);
                    // the failed tails become the whole tail list of the round;
                    // the next round's tails marked so far stay
                    const uint32_t tp = (h.lid + 1) % 3;
                    PADO_CUDA(cudaMemcpyAsync(bf.tails[tp], retry.p, h.retry_cnt * 4ull, cudaMemcpyDeviceToDevice, s));
                    h.slot[tp] = {};  // the re-run pull claims from zero
                    h.slot[tp].light_cnt = h.retry_cnt;
                } else {
                    PADO_CHECK(h.exit_code == WX_NEED_POOL, PADO_E_STATE, "weighted labeling loop stopped unexpectedly");
                    unsigned long long top = 0;
                    PADO_CUDA(cudaMemcpy(&top, pool_top.p, 8, cudaMemcpyDeviceToHost));
                    grow_pool(top);
                    PADO_CUDA(cudaMemcpyAsync(rr.p, retry.p, h.retry_cnt * 4ull, cudaMemcpyDeviceToDevice, s));
                    h.rr_cnt = h.retry_cnt;
                }
                h.bar = GridBar{};  // a launch starts its barriers from zero
                h.retry_cnt = 0;
                h.status = 0;
                h.exit_code = WX_RUNNING;
                PADO_CUDA(cudaMemsetAsync(status.p, 0, 4, s));
                PADO_CUDA(cudaMemcpyAsync(ctl.p, &h, sizeof(WLoopCtl), cudaMemcpyHostToDevice, s));
            }
            run.levels = h.levels;
            run.batches = nbatches;
        }
        for (uint32_t bs = 0, b = 0; host_loop && bs < n; bs += B, ++b) {
            PADO_CHECK(b + 1 < 65536u, PADO_E_ARG, "more than 65534 batches");
            const uint32_t nr = (uint32_t)std::min<uint64_t>(B, (uint64_t)n - bs);
            ++run.batches;
            const uint32_t lid0 = ++lid;
            int cur = lid0 & 1;
            PADO_CUDA(cudaMemsetAsync(counters.p, 0, 8 * sizeof(uint32_t), s));
            PADO_CUDA(cudaMemsetAsync(&log_top.p[lid0 & 1], 0, 8, s));
            PADO_LAUNCH("w_root_init_kernel", s,
                        w_root_init_kernel<<<grid_for((uint64_t)nr * 32, 256), 256, 0, s>>>(d, bs, nr, lid0, fronts[cur], c_front[cur],
                                                                                news.p, c_news));
            uint32_t fsize = nr;
            for (uint64_t round = 0; fsize > 0; ++round) {
                // Bellman-Ford rounds are bounded by the vertex count
                PADO_CHECK(round <= (uint64_t)n + 2, PADO_E_STATE, "relaxation did not converge");
                const uint32_t lid_cur = ++lid;
                const int nxt = cur ^ 1;
                PADO_CUDA(cudaMemsetAsync(c_tails, 0, 4, s));
                PADO_CUDA(cudaMemsetAsync(c_front[nxt], 0, 4, s));
                PADO_CUDA(cudaMemsetAsync(&log_top.p[lid_cur & 1], 0, 8, s));
                if (b == 0) {
                    PADO_LAUNCH("w_snap_kernel", s,
                                w_snap_kernel<<<grid_for((uint64_t)nr * B, 256), 256, 0, s>>>(d, nr));
                }
                PADO_LAUNCH("w_mark_kernel", s,
                            w_mark_kernel<<<grid_for((uint64_t)fsize * 32, 256), 256, 0, s>>>(d, fronts[cur], c_front[cur], lid_cur,
                                                                                 tails.p, c_tails));
                PADO_LAUNCH("w_pull_kernel", s,
                            w_pull_kernel<<<grid_for((uint64_t)n * 32, WPULL_WARPS * 32, 152u * 8u), WPULL_WARPS * 32, pull_smem, s>>>(
                    d, tails.p, c_tails, bs, b, lid_cur, fronts[nxt], c_front[nxt], news.p, c_news, retry.p, c_retry));
                read_ctrs(c_front[nxt]);
                ++run.levels;
                for (int attempt = 0; hc->retry; ++attempt) {
                    PADO_CHECK(attempt < 64, PADO_E_NOMEM, "round log could not be grown enough");
                    grow_logs(hc->ltop[lid_cur & 1]);
                    PADO_CUDA(cudaMemcpyAsync(tails.p, retry.p, hc->retry * 4, cudaMemcpyDeviceToDevice, s));
                    PADO_CUDA(cudaMemcpyAsync(c_tails, c_retry, 4, cudaMemcpyDeviceToDevice, s));
                    PADO_CUDA(cudaMemsetAsync(c_retry, 0, 4, s));
                    PADO_CUDA(cudaMemsetAsync(status.p, 0, 4, s));
                    PADO_LAUNCH("w_pull_kernel(retry)", s,
                                w_pull_kernel<<<grid_for((uint64_t)hc->retry * 32, WPULL_WARPS * 32, 152u * 8u), WPULL_WARPS * 32,
                                    pull_smem, s>>>(d, tails.p, c_tails, bs, b, lid_cur, fronts[nxt], c_front[nxt],
                                                    news.p, c_news, retry.p, c_retry));
                    read_ctrs(c_front[nxt]);
                }
                fsize = hc->front_next;
                cur = nxt;
            }
            read_ctrs(c_front[cur]);
            const uint32_t nn = hc->news;
            PADO_LAUNCH("w_filter_kernel", s,
                        w_filter_kernel<<<grid_for((uint64_t)nn * 32, 256), 256, 0, s>>>(d, news.p, nn, bs));
            PADO_LAUNCH("w_buf_reset_kernel", s,
                        w_buf_reset_kernel<<<grid_for((uint64_t)nr * 32, 256), 256, 0, s>>>(d, bs, nr));
            const uint32_t *clist = news.p;
            uint32_t cn = nn;
            for (int attempt = 0;; ++attempt) {
                PADO_CHECK(attempt < 64, PADO_E_NOMEM, "label pool could not be grown enough");
                PADO_LAUNCH("w_commit_kernel", s,
                            w_commit_kernel<<<grid_for((uint64_t)cn * 32, 256), 256, 0, s>>>(d, clist, cn, bs, retry.p, c_retry));
                read_ctrs(c_front[cur]);
                if (!hc->retry) break;
                grow_pool(hc->top);
                PADO_CUDA(cudaMemcpyAsync(tails.p, retry.p, hc->retry * 4, cudaMemcpyDeviceToDevice, s));
                PADO_CUDA(cudaMemsetAsync(c_retry, 0, 4, s));
                PADO_CUDA(cudaMemsetAsync(status.p, 0, 4, s));
                clist = tails.p;
                cn = hc->retry;
            }
        }
        std::vector<uint32_t> lens(n);
        lab_len.download(lens.data(), n, s);
        PADO_CUDA(cudaStreamSynchronize(s));
        std::vector<uint64_t> fo(n + 1, 0);
        for (uint32_t v = 0; v < n; ++v) fo[v + 1] = fo[v] + lens[v];
        out.total = fo[n];
        out.off.alloc(n + 1);
        out.off.upload(fo.data(), n + 1, s);
        out.hub.alloc(std::max<uint64_t>(out.total, 1));
        out.dist16.alloc(std::max<uint64_t>(out.total, 1));
        if (n) {
            PADO_LAUNCH("w_compact_kernel", s,
                        w_compact_kernel<<<grid_for((uint64_t)n * 32, 256), 256, 0, s>>>(d, out.off.p, out.hub.p, out.dist16.p));
        }
        PADO_CUDA(cudaEventRecord(e1, s));
        PADO_CUDA(cudaEventSynchronize(e1));
        PADO_CUDA(cudaEventElapsedTime(&run.ms, e0, e1));
    } catch (...) {
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        throw;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return run;
}

}  // namespace pado
