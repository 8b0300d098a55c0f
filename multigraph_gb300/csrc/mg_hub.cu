// mg_hub.cu -- shared-memory segmented pull for PageRank sweeps.
//
// The reference turns the random gathers of its dense PageRank phases into
// partition-local work: edges are regrouped into 16-bit tile streams by
// source partition (gen_structure.cu:1534-1947, sp1/sp2/mapper) and each
// partition's values are summed in shared memory (processi.cu:682-894,
// _phase1/_phase2).  Re-derived for GB300: the source ids are cut into
// segments of H = SEG_H vertices (the most a CTA's 227 KB of shared memory
// holds as FP32 contributions, 224 KB), and each pull row's in-edges are
// grouped by segment once per layout:
//   pairs, pieces   : a (row, segment) pair is the row's in-edges from the
//                     segment; it is cut into pieces of at most PIECE_MAX
//                     edges (the row's order kept);
//   warp groups     : per segment, pieces of equal length lambda are bucketed
//                     (rows ascending) and packed GROUP at a time, padded;
//                     a group stores its ids as 16-bit local ids (id - s*H)
//                     step-major, [lambda][GROUP], so each step is one
//                     coalesced 256-byte warp load (four pieces per lane);
//   P, pair_off     : the pieces' sums in row-major order (row v's pieces at
//                     P[pair_off[v] .. pair_off[v+1]), segments ascending),
//                     summed by the row's finish; pslot gives each packed
//                     piece its place in P;
//   sorted windows  : where the row finish copies 32 rows' piece sums to
//                     shared memory anyway (at most HUB_WIN pieces, no warp
//                     row, no tail), the window's P is ordered by (segment,
//                     length, row) instead and porder gives each place its
//                     piece's place in row order.  A group's pieces are
//                     neighbours in that order, so the sweep's stores of
//                     their sums share sectors: one sector a piece's sum was
//                     what short groups cost (R-MAT 21: 0.96 sectors stored
//                     a piece -> 0.34; a group 155 cycles of its SM where a
//                     step takes 19).
//   tail            : in-edges from ids beyond the last segment (graphs
//                     with more than SEG_MAX segments' worth of vertices),
//                     int32 ids gathered through L2 by the degree-binned
//                     sweep.
// One sweep: k_hub_sweep gives each CTA a contiguous range of groups (the
// least largest load under the groups' cost weights and the segments to be
// staged; the weights are a model of steps, groups and stored sectors at
// first, re-weighted by mg_autotune from measured per-CTA times), stages the
// contributions c[s*H, (s+1)*H) of every segment its range enters, and
// its warps claim chunks of consecutive groups from a shared-memory counter
// and stream them: a lane adds its four pieces' edges in order from shared
// memory and stores the four totals to P.  Pieces never cross a group, so
// there are no carries between lanes, warps or CTAs; every sum is formed in
// a fixed order, whichever warp runs it, so sweeps are reproducible.
//
// Per sweep the streams move 2 B per edge (plus padding, ~2.4 % on R-MAT),
// a 4-byte slot and a 4-byte store per piece (about one piece per ten
// edges), instead of 4 B of ids and a 32-byte L2 sector per gather.  The
// row finish (k_pr_seg in mg_pr.cu) reads each row's piece sums.

#include "mg_device.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <functional>
#include <thread>
#include <type_traits>

namespace {

constexpr int32_t SEG_H = 57344;    // vertices per segment: 224 KB of FP32 contributions
constexpr int32_t SEG_MAX = 64;     // segments at most; ids beyond stay in the L2 tail
constexpr int32_t PIECE_MAX = 64;   // edges per piece at most
constexpr int32_t GROUP = 128;      // pieces per warp group: four per lane
constexpr int HUB_THREADS = 1024;   // one CTA per SM (shared memory bound)
constexpr int HUB_UNROLL = 4;       // steps (256-byte warp loads) in flight per warp
constexpr int STAGE_BATCH = 4;      // 16-byte loads in flight per thread while staging a segment
// what a CTA takes for its groups, in cycles of its SM (for the initial split
// of the groups among the CTAs)
// (least squares over the CTAs of R-MAT 20 to 22: within 3-9 % of the measured cycles)
constexpr double STEP_COST = 18.7;     // a step: 128 gathers from shared memory
constexpr double GROUP_COST = 25.0;    // a group's slots, claim and switch
constexpr double SECTOR_COST = 1.05;   // a 32-byte sector of P that a group's stores touch
constexpr double STAGE_COST = 9000.0;  // a segment staged
constexpr double CHUNK_COST = 600.0;   // a chunk, the unit that warps claim
// the row finish sums rows with more than FIN_WARP pieces a warp each, the
// rest a thread each (8-lane groups for rows of 5-64 pieces walked their
// rows one after another and were slower)
constexpr int32_t FIN_WARP = 32;

struct HubArgs {
    const uint2 *hdat;        // groups' ids, four 16-bit ids per lane per step
    const int32_t *goff;      // [ngroups+1] each group's first step
    const int4 *pslot;        // [ngroups*GROUP/4] the four P slots of each lane's pieces
    const int32_t *cpart;     // [grid+1] each CTA's parts
    const int32_t *pseg;      // [nparts] each part's segment
    const int32_t *pch;       // [nparts+1] each part's chunks
    const int32_t *cb;        // [nchunks+1] chunk k = groups [cb[k], cb[k+1])
    const float *c[2];        // contributions (ping-pong, ctl selects)
    const int32_t *cur;       // current iterate index (loop control block)
    const int32_t *more;      // loop continue flag
    const int32_t *off;       // non-zero: sweeps run elsewhere (queue sweeps)
    float *P;                 // piece sums, row-major
    long long *ctime;         // [grid] each CTA's clock cycles (read back to re-split the work)
    int32_t n, H, nseg;
};

// One warp streams groups [ga, gb) (contiguous in hdat): the next
// HUB_UNROLL steps are loaded while the current ones are summed, across
// group ends, so the loads run back to back instead of one latency chain per
// group.  Every edge gets one compensated add, in edge order, so a piece's
// sum does not depend on where a warp's range starts (the work split is
// re-cut from measurements; a faster pairwise add of four steps at a time,
// applied where a batch of loads fell inside one group, made the rounding
// follow the split).  The groups' first steps come from goff 32 at a time
// (one load, then shuffles); each group's slots are loaded when it starts.
__device__ __forceinline__ void stream_groups(const HubArgs &a, const float *s_c, int32_t ga, int32_t gb, int lane)
{
    constexpr unsigned FULL = 0xffffffffu;
    const uint2 *D = a.hdat + lane;
    int32_t cbase = ga;
    int32_t cg = __ldg(&a.goff[min(cbase + lane, gb)]);
    int32_t t = __shfl_sync(FULL, cg, 0);
    const int32_t tend = __ldg(&a.goff[gb]);
    int32_t g = ga;
    int32_t gend = __shfl_sync(FULL, cg, 1);
    // slots and ids are streamed once per sweep: evict-first loads keep L2
    // for the piece sums the row finish reads next
    int4 sl = __ldcs(&a.pslot[(int64_t)g * 32 + lane]);
    // compensated sums (Kahan): a piece of up to PIECE_MAX edges is exact to
    // about one rounding, so a hub row's total does not drift by a few 1e-6
    // from sweep to sweep as its inputs settle
    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f, r0 = 0.0f, r1 = 0.0f, r2 = 0.0f, r3 = 0.0f;
    uint2 wc[HUB_UNROLL], wn[HUB_UNROLL];
#pragma unroll
    for (int j = 0; j < HUB_UNROLL; j++) wc[j] = t + j < tend ? __ldcs(D + (int64_t)(t + j) * 32) : make_uint2(0u, 0u);
    while (t < tend) {
#pragma unroll
        for (int j = 0; j < HUB_UNROLL; j++) {
            const int32_t q = t + HUB_UNROLL + j;
            wn[j] = q < tend ? __ldcs(D + (int64_t)q * 32) : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int j = 0; j < HUB_UNROLL; j++) {
            if (t < tend) {
                mgd::kahan_add(s0, r0, s_c[wc[j].x & 0xffffu]);
                mgd::kahan_add(s1, r1, s_c[wc[j].x >> 16]);
                mgd::kahan_add(s2, r2, s_c[wc[j].y & 0xffffu]);
                mgd::kahan_add(s3, r3, s_c[wc[j].y >> 16]);
                t++;
                if (t == gend) {   // group g is complete (warp-uniform)
                    a.P[sl.x] = s0 - r0;
                    a.P[sl.y] = s1 - r1;
                    a.P[sl.z] = s2 - r2;
                    a.P[sl.w] = s3 - r3;
                    s0 = s1 = s2 = s3 = r0 = r1 = r2 = r3 = 0.0f;
                    g++;
                    if (g < gb) {
                        if (g + 1 - cbase >= 32) {
                            cbase = g + 1;
                            cg = __ldg(&a.goff[min(cbase + lane, gb)]);
                        }
                        gend = __shfl_sync(FULL, cg, g + 1 - cbase);
                        sl = __ldcs(&a.pslot[(int64_t)g * 32 + lane]);
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < HUB_UNROLL; j++) wc[j] = wn[j];
    }
}

// One sweep over every piece: each CTA walks its parts (one segment each),
// stages the segment's contributions in shared memory, and its warps claim
// the part's chunks from a shared-memory counter; the CTA's clock cycles go
// to ctime for the next re-split.
__global__ void __launch_bounds__(HUB_THREADS, 1) k_hub_sweep(HubArgs a)
{
    extern __shared__ __align__(16) float s_c[];   // [H + 4]
    if (__ldg(a.more) == 0 || __ldg(a.off) != 0) return;
    const float *c = __ldg(a.cur) ? a.c[1] : a.c[0];
    if (threadIdx.x < 4) s_c[a.H + threadIdx.x] = 0.0f;   // the padding id's slot
    __shared__ int32_t s_next;   // the part's next unclaimed chunk
    const long long t_start = clock64();
    const int32_t lane = threadIdx.x & 31;
    const int32_t p0 = __ldg(&a.cpart[blockIdx.x]), p1 = __ldg(&a.cpart[blockIdx.x + 1]);
    for (int32_t pi = p0; pi < p1; pi++) {
        const int32_t s = __ldg(&a.pseg[pi]);
        // stage c[s*H, s*H + len) (16-byte units; the arrays carry 16 bytes
        // of slack past the last vertex)
        const int32_t base = s * a.H;
        const int32_t n4 = (min(a.H, a.n - base) + 3) >> 2;
        __syncthreads();   // every warp is done with the previous segment
        const int32_t k1 = __ldg(&a.pch[pi + 1]);
        if (threadIdx.x == 0) s_next = __ldg(&a.pch[pi]);
        const float4 *src = reinterpret_cast<const float4 *>(c + base);
        float4 *dst = reinterpret_cast<float4 *>(s_c);
        // all of a thread's loads in flight at once, in batches of STAGE_BATCH
        for (int32_t i0 = threadIdx.x; i0 < n4; i0 += STAGE_BATCH * HUB_THREADS) {
            float4 v[STAGE_BATCH];
#pragma unroll
            for (int k = 0; k < STAGE_BATCH; k++) {
                const int32_t i = i0 + k * HUB_THREADS;
                if (i < n4) v[k] = __ldcg(&src[i]);
            }
#pragma unroll
            for (int k = 0; k < STAGE_BATCH; k++) {
                const int32_t i = i0 + k * HUB_THREADS;
                if (i < n4) dst[i] = v[k];
            }
        }
        __syncthreads();
        // the warps claim the part's chunks in order until none is left
        while (true) {
            int32_t k = 0;
            if (lane == 0) k = atomicAdd(&s_next, 1);
            k = __shfl_sync(0xffffffffu, k, 0);
            if (k >= k1) break;
            stream_groups(a, s_c, __ldg(&a.cb[k]), __ldg(&a.cb[k + 1]), lane);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) a.ctime[blockIdx.x] = clock64() - t_start;
}

// A bucket's q-th piece's place in its group: consecutive pieces (ascending
// rows) go to consecutive lanes, so that a lane's j-th total is stored beside
// its neighbours' j-th.
__host__ __device__ inline int32_t group_place(int64_t q) { return (int32_t)((q % 32) * 4 + (q % GROUP) / 32); }

// ---------------------------------------------------------------------------
// The layout built on the device.  T = chunks of contiguous windows of 32
// rows, even in rows + edges, a warp each: pass 1 counts every (row, segment)
// and adds up the chunk's buckets, a scan over the chunks gives every chunk
// its places in every bucket (rows ascending, whichever warp runs when), pass
// 2 counts again and writes.  A window's rows are counted flat, 32 edges of
// any of its rows at a time.  Rows of more than HB_ROW edges would keep one
// warp busy for milliseconds: they are cut into subs of HB_ROW edges, a warp
// each.  Built on the host, from the columns copied back, the layout took
// most of the 434 ms of R-MAT 22's first PageRank call (here 17).
// ---------------------------------------------------------------------------
// (R-MAT 22's first call with 2048, 4096, 8192 and 16384 chunks: 27, 20, 17 and 16 ms -- the more of
// them, the closer in time the warps that fill one group)
constexpr int32_t HB_CHUNKS = 8192;
constexpr int32_t HB_ROW = 2048;
constexpr int HB_WARPS = 2;   // a block: shared memory of 20-30 KB a warp decides how many an SM holds

// A long row [begin, end) in subs: their number; sub s's first edge and length.
// (No sum passes end, which may be the last int32.)
__host__ __device__ inline int32_t hb_subs(int32_t begin, int32_t end) { return (end - begin - 1) / HB_ROW + 1; }
__host__ __device__ inline int32_t hb_sub_begin(int32_t begin, int32_t s) { return begin + s * HB_ROW; }
__host__ __device__ inline int32_t hb_sub_len(int32_t begin, int32_t end, int32_t s)
{
    const int32_t left = end - hb_sub_begin(begin, s);
    return left < HB_ROW ? left : HB_ROW;
}

struct HubBuild {
    const int32_t *prow, *pcol;
    int32_t n, nseg, cover, chunks;
    int32_t nb;          // buckets: nseg * (PIECE_MAX + 1)
    int32_t ncol;        // columns of a row's counts: the segments, then the tail
    int32_t stride;      // ncol made odd (rows in shared memory, a lane each)
    uint32_t *table;     // [chunks][nb + 3] bucket counts, then pieces, tail edges, warp rows; scanned in place
    uint32_t *total;     // [nb + 3]
    const uint32_t *place;   // [nb] each bucket's first place
    int32_t *hid;        // [n] a long row's number + 1, or 0
    int32_t *nlong;      // [2] long rows; their subs
    int2 *lrow;          // long rows: (row, first sub)
    int32_t *sub;        // subs: the long row's number
    uint32_t *subcnt;    // [subs][ncol] counts, then the sub's first index in the row's segment
    uint32_t *lcnt;      // [long rows][ncol] counts
    uint32_t *lplace;    // [long rows][2][ncol] first places: full pieces (the tail's edges), the rest
    const int32_t *goff;
    int32_t *pair_off, *toff, *tcol, *fin, *pslot;
    uint16_t *hdat, *porder;
    int32_t ntail;
};

__device__ __forceinline__ int32_t hb_segment(const HubBuild &b, int32_t c) { return c < b.cover ? c / SEG_H : b.nseg; }

__global__ void __launch_bounds__(256) k_hb_long(HubBuild b)
{
    for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < b.n; v += gridDim.x * blockDim.x) {
        const int32_t d = b.prow[v + 1] - b.prow[v];
        int32_t id = 0;
        if (d > HB_ROW) {
            const int32_t ns = hb_subs(b.prow[v], b.prow[v + 1]);
            id = atomicAdd(&b.nlong[0], 1) + 1;
            const int32_t first = atomicAdd(&b.nlong[1], ns);
            b.lrow[id - 1] = make_int2(v, first);
            for (int32_t s = 0; s < ns; s++) b.sub[first + s] = id - 1;
        }
        b.hid[v] = id;
    }
}

__global__ void __launch_bounds__(HB_WARPS * 32) k_hb_sub_count(HubBuild b)
{
    __shared__ uint32_t s_cnt[HB_WARPS][SEG_MAX + 1];
    uint32_t *cnt = s_cnt[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int32_t nsub = b.nlong[1];
    for (int32_t s = blockIdx.x * HB_WARPS + (threadIdx.x >> 5); s < nsub; s += gridDim.x * HB_WARPS) {
        for (int k = lane; k < b.ncol; k += 32) cnt[k] = 0;
        __syncwarp();
        const int2 r = b.lrow[b.sub[s]];
        const int32_t begin = b.prow[r.x], len = hb_sub_len(begin, b.prow[r.x + 1], s - r.y);
        const int32_t *col = b.pcol + hb_sub_begin(begin, s - r.y);
#pragma unroll 4
        for (int32_t i = lane; i < len; i += 32) atomicAdd(&cnt[hb_segment(b, __ldg(&col[i]))], 1u);
        __syncwarp();
        for (int k = lane; k < b.ncol; k += 32) b.subcnt[(size_t)s * b.ncol + k] = cnt[k];
        __syncwarp();
    }
}

__global__ void __launch_bounds__(128) k_hb_long_scan(HubBuild b)
{
    const int k = threadIdx.x;
    const int32_t nl = b.nlong[0];
    if (k >= b.ncol) return;
    for (int32_t i = blockIdx.x; i < nl; i += gridDim.x) {
        const int2 r = b.lrow[i];
        const int32_t ns = hb_subs(b.prow[r.x], b.prow[r.x + 1]);
        uint32_t run = 0;
        for (int32_t s = 0; s < ns; s++) {
            uint32_t *c = &b.subcnt[(size_t)(r.y + s) * b.ncol + k];
            const uint32_t x = *c;
            *c = run;
            run += x;
        }
        b.lcnt[(size_t)i * b.ncol + k] = run;
    }
}

// first row of chunk t: rows + edges in even shares, whole windows
__device__ __forceinline__ int32_t hb_chunk_row(const HubBuild &b, int32_t t)
{
    if (t >= b.chunks) return b.n;
    const long long goal = ((long long)b.prow[b.n] + b.n) * t / b.chunks;
    int32_t lo = 0, hi = b.n;
    while (lo < hi) {
        const int32_t mid = lo + (hi - lo) / 2;
        if ((long long)b.prow[mid] + mid < goal) lo = mid + 1;
        else hi = mid;
    }
    return min((lo + 31) & ~31, b.n);
}

// the window's rows, a lane each, and their edges but the long rows' in one
// list: lane l's at [off, off + deg) of it
struct HubWindow {
    int32_t v, start, id, off, total;
};

__device__ __forceinline__ HubWindow hb_window(const HubBuild &b, int32_t vb, int lane)
{
    HubWindow w;
    w.v = vb + lane;
    const bool act = w.v < b.n;
    w.start = act ? b.prow[w.v] : 0;
    w.id = act ? b.hid[w.v] : 0;
    const int32_t deg = act && w.id == 0 ? b.prow[w.v + 1] - w.start : 0;
    const int incl = mgd::warp_scan_incl(deg);
    w.off = incl - deg;
    w.total = __shfl_sync(0xffffffffu, incl, 31);
    return w;
}

// fn(row's lane, column id, whether there is one), in edge order, 32 at a time
template <class Fn>
__device__ __forceinline__ void hb_edges(const HubBuild &b, const HubWindow &w, int lane, Fn fn)
{
    constexpr int AHEAD = 4;
    for (int32_t i = 0; i < w.total; i += 32 * AHEAD) {
        int32_t r[AHEAD], c[AHEAD];
#pragma unroll
        for (int j = 0; j < AHEAD; j++) {
            const int32_t k = i + 32 * j + lane;
            r[j] = mgd::owner_lane(w.off, min(k, w.total - 1));
            const int32_t p = __shfl_sync(0xffffffffu, w.start, r[j]) + k - __shfl_sync(0xffffffffu, w.off, r[j]);
            c[j] = k < w.total ? __ldg(&b.pcol[p]) : -1;
        }
#pragma unroll
        for (int j = 0; j < AHEAD; j++)
            if (i + 32 * j < w.total) fn(r[j], c[j]);
    }
}

__device__ __forceinline__ void hb_count(const HubBuild &b, const HubWindow &w, int lane, uint32_t *cnt)
{
    for (int k = lane; k < 32 * b.stride; k += 32) cnt[k] = 0;
    __syncwarp();
    hb_edges(b, w, lane, [&](int32_t r, int32_t c) {
        if (c >= 0) atomicAdd(&cnt[r * b.stride + hb_segment(b, c)], 1u);
    });
    unsigned longs = __ballot_sync(0xffffffffu, w.id > 0);
    while (longs) {
        const int r = __ffs(longs) - 1;
        longs &= longs - 1;
        const int32_t id = __shfl_sync(0xffffffffu, w.id, r) - 1;
        for (int k = lane; k < b.ncol; k += 32) cnt[r * b.stride + k] = b.lcnt[(size_t)id * b.ncol + k];
    }
    __syncwarp();
}

__device__ __forceinline__ int32_t hb_pieces(const HubBuild &b, const uint32_t *row)
{
    int32_t np = 0;
    for (int sg = 0; sg < b.nseg; sg++) np += (int32_t)((row[sg] + PIECE_MAX - 1) / PIECE_MAX);
    return np;
}

__global__ void __launch_bounds__(HB_WARPS * 32) k_hb_count(HubBuild b)
{
    extern __shared__ uint32_t s_hb[];
    const int lane = threadIdx.x & 31;
    uint32_t *cnt = s_hb + (size_t)(threadIdx.x >> 5) * (32 * b.stride + b.nb), *hist = cnt + 32 * b.stride;
    const int32_t t = blockIdx.x * HB_WARPS + (threadIdx.x >> 5);
    if (t >= b.chunks) return;
    for (int k = lane; k < b.nb; k += 32) hist[k] = 0;
    const int32_t v0 = hb_chunk_row(b, t), v1 = hb_chunk_row(b, t + 1);
    uint32_t pieces = 0, tail = 0, fin = 0;
    for (int32_t vb = v0; vb < v1; vb += 32) {
        const HubWindow w = hb_window(b, vb, lane);
        hb_count(b, w, lane, cnt);
        const uint32_t *row = cnt + lane * b.stride;
        uint32_t np = 0;
        for (int sg = 0; sg < b.nseg; sg++) {
            const uint32_t full = row[sg] / PIECE_MAX, rem = row[sg] % PIECE_MAX;
            if (full) atomicAdd(&hist[sg * (PIECE_MAX + 1) + PIECE_MAX], full);
            if (rem) atomicAdd(&hist[sg * (PIECE_MAX + 1) + rem], 1u);
            np += full + (rem > 0);
        }
        pieces += np;
        tail += row[b.nseg];
        fin += np > (uint32_t)FIN_WARP;
        __syncwarp();
    }
    uint32_t *out = b.table + (size_t)t * (b.nb + 3);
    for (int k = lane; k < b.nb; k += 32) out[k] = hist[k];
    pieces = __reduce_add_sync(0xffffffffu, pieces);
    tail = __reduce_add_sync(0xffffffffu, tail);
    fin = __reduce_add_sync(0xffffffffu, fin);
    if (lane == 0) {
        out[b.nb] = pieces;
        out[b.nb + 1] = tail;
        out[b.nb + 2] = fin;
    }
}

// exclusive scan of every column of the table: 32 columns a block, the rows
// in 32 slices
__global__ void __launch_bounds__(1024) k_hb_scan(HubBuild b)
{
    __shared__ uint32_t s_sum[32][33];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int32_t w = b.nb + 3, k = blockIdx.x * 32 + x;
    const int32_t per = (b.chunks + 31) / 32, t0 = min(y * per, b.chunks), t1 = min(t0 + per, b.chunks);
    uint32_t sum = 0;
    if (k < w)
#pragma unroll 8
        for (int32_t t = t0; t < t1; t++) sum += b.table[(size_t)t * w + k];
    s_sum[y][x] = sum;
    __syncthreads();
    if (k >= w) return;
    uint32_t run = 0;
    for (int j = 0; j < y; j++) run += s_sum[j][x];
    for (int32_t t = t0; t < t1; t++) {
        uint32_t *c = &b.table[(size_t)t * w + k];
        const uint32_t v = *c;
        *c = run;
        run += v;
    }
    if (y == 31) b.total[k] = run;
}

__global__ void __launch_bounds__(256) k_hb_fill(uint32_t *p, uint32_t x, long long count)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x)
        p[i] = x;
}

__device__ __forceinline__ void hb_slot(const HubBuild &b, uint32_t q, int32_t slot)
{
    b.pslot[(size_t)(q / GROUP) * GROUP + group_place(q)] = slot;
}

// the e-th of a row's edges from segment sg, whose pieces start at qf (full) and qr
__device__ __forceinline__ void hb_put(const HubBuild &b, uint32_t e, uint32_t count, uint32_t qf, uint32_t qr, int32_t sg,
                                       int32_t c)
{
    const uint32_t i = e / PIECE_MAX, k = e % PIECE_MAX;
    const uint32_t q = i < count / PIECE_MAX ? qf + i : qr;
    const size_t grp = q / GROUP;
    b.hdat[((size_t)__ldg(&b.goff[grp]) + k) * GROUP + group_place(q)] = (uint16_t)(c - sg * SEG_H);
}

__global__ void __launch_bounds__(HB_WARPS * 32) k_hb_place(HubBuild b)
{
    extern __shared__ uint32_t s_hb[];
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int mat = 32 * b.stride;
    uint32_t *cnt = s_hb + (size_t)(threadIdx.x >> 5) * (3 * mat + 2 * mgi::HUB_WIN), *qf = cnt + mat, *qr = qf + mat;
    uint32_t *key = qr + mat, *at = key + mgi::HUB_WIN;
    const int32_t t = blockIdx.x * HB_WARPS + (threadIdx.x >> 5);
    if (t >= b.chunks) return;
    uint32_t *next = b.table + (size_t)t * (b.nb + 3);   // this warp's own
    for (int k = lane; k < b.nb; k += 32) next[k] += b.place[k];
    int32_t base = (int32_t)next[b.nb], tbase = (int32_t)next[b.nb + 1], fbase = (int32_t)next[b.nb + 2];
    __syncwarp();
    const int32_t v0 = hb_chunk_row(b, t), v1 = hb_chunk_row(b, t + 1);
    for (int32_t vb = v0; vb < v1; vb += 32) {
        const HubWindow w = hb_window(b, vb, lane);
        const bool act = w.v < b.n;
        hb_count(b, w, lane, cnt);
        uint32_t *row = cnt + lane * b.stride;
        const int32_t np = hb_pieces(b, row), nt = (int32_t)row[b.nseg];
        const int32_t pincl = mgd::warp_scan_incl(np), tincl = mgd::warp_scan_incl(nt);
        const int32_t len = __shfl_sync(FULL, pincl, 31);
        const int32_t tlen = __shfl_sync(FULL, tincl, 31);
        int32_t piece = pincl - np;   // the row's next piece, in row order
        if (act) {
            b.pair_off[w.v] = base + piece;
            b.toff[w.v] = tbase + tincl - nt;
        }
        const unsigned fins = __ballot_sync(FULL, np > FIN_WARP);
        if (np > FIN_WARP) b.fin[fbase + __popc(fins & ((1u << lane) - 1u))] = w.v;
        const bool sorted = b.ntail == 0 && len <= mgi::HUB_WIN && fins == 0;
        if (sorted) {
            int32_t i = piece;
            for (int sg = 0; sg < b.nseg; sg++)
                for (int32_t left = (int32_t)row[sg]; left > 0; left -= PIECE_MAX, i++)
                    key[i] = (uint32_t)sg << 16 | (uint32_t)(PIECE_MAX - min(left, PIECE_MAX)) << 9 | (uint32_t)i;
            int size = 32;
            while (size < len) size *= 2;   // at most HUB_WIN
            for (int k = len + lane; k < size; k += 32) key[k] = FULL;
            __syncwarp();
            for (int up = 2; up <= size; up *= 2)
                for (int d = up / 2; d > 0; d /= 2) {
                    for (int k = lane; k < size / 2; k += 32) {
                        const int x = 2 * d * (k / d) + k % d, y = x + d;
                        const uint32_t kx = key[x], ky = key[y];
                        if ((kx > ky) == ((x & up) == 0)) {
                            key[x] = ky;
                            key[y] = kx;
                        }
                    }
                    __syncwarp();
                }
            for (int k = lane; k < len; k += 32) {
                const uint32_t o = key[k] & 511u;
                at[o] = (uint32_t)k;
                b.porder[base + k] = (uint16_t)o;
            }
            __syncwarp();
        } else if (b.ntail == 0) {
            for (int32_t k = lane; k < len; k += 32) b.porder[base + k] = (uint16_t)k;
        }
        // every piece's place in its bucket, rows ascending; the buckets' next
        // places are read BATCH segments at a time
        constexpr int BATCH = 4;
        for (int sb = 0; sb < b.nseg; sb += BATCH) {
            uint32_t nfull[BATCH], nrem[BATCH];
#pragma unroll
            for (int j = 0; j < BATCH; j++) {
                if (sb + j >= b.nseg) break;
                const uint32_t *nk = next + (sb + j) * (PIECE_MAX + 1);
                nfull[j] = nk[PIECE_MAX];
                nrem[j] = nk[row[sb + j] % PIECE_MAX];
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < BATCH; j++) {
                const int sg = sb + j;
                if (sg >= b.nseg) break;
                const uint32_t count = row[sg], full = count / PIECE_MAX, rem = count % PIECE_MAX;
                uint32_t *nk = next + sg * (PIECE_MAX + 1);
                if (__any_sync(FULL, full > 0)) {
                    const uint32_t incl = (uint32_t)mgd::warp_scan_incl((int)full);
                    const uint32_t q = nfull[j] + incl - full;
                    qf[lane * b.stride + sg] = q;
                    for (uint32_t i = 0; i < full; i++, piece++)
                        hb_slot(b, q + i, base + (sorted ? (int32_t)at[piece] : piece));
                    if (lane == 31) nk[PIECE_MAX] = nfull[j] + incl;
                }
                const unsigned same = __match_any_sync(FULL, rem);
                if (rem) {
                    const uint32_t q = nrem[j] + __popc(same & ((1u << lane) - 1u));
                    qr[lane * b.stride + sg] = q;
                    hb_slot(b, q, base + (sorted ? (int32_t)at[piece] : piece));
                    piece++;
                    if (lane == 31 - __clz(same)) nk[rem] = nrem[j] + __popc(same);
                }
                // a row that is not long has at most HB_ROW edges: its count in
                // the upper half, the edges written so far in the lower
                if (w.id == 0) row[sg] = count << 16;
            }
        }
        qf[lane * b.stride + b.nseg] = (uint32_t)(tbase + tincl - nt);
        if (w.id == 0) row[b.nseg] = (uint32_t)nt << 16;
        __syncwarp();
        hb_edges(b, w, lane, [&](int32_t r, int32_t c) {
            const int32_t sg = c < 0 ? 0 : hb_segment(b, c);
            const unsigned same = __match_any_sync(FULL, c < 0 ? -1 : r << 8 | sg);
            const int at0 = r * b.stride + sg;
            const uint32_t rc = cnt[at0];
            const uint32_t e = (rc & 0xffffu) + __popc(same & ((1u << lane) - 1u));
            __syncwarp();
            if (c >= 0) {
                if (lane == 31 - __clz(same)) cnt[at0] = rc + __popc(same);
                if (sg == b.nseg) b.tcol[qf[at0] + e] = c;
                else hb_put(b, e, rc >> 16, qf[at0], qr[at0], sg, c);
            }
            __syncwarp();
        });
        unsigned longs = __ballot_sync(FULL, w.id > 0);
        while (longs) {
            const int r = __ffs(longs) - 1;
            longs &= longs - 1;
            const int32_t id = __shfl_sync(FULL, w.id, r) - 1;
            uint32_t *lp = b.lplace + (size_t)id * 2 * b.ncol;
            for (int k = lane; k < b.ncol; k += 32) {
                lp[k] = qf[r * b.stride + k];
                lp[b.ncol + k] = qr[r * b.stride + k];
            }
        }
        __syncwarp();
        base += len;
        tbase += tlen;
        fbase += __popc(fins);
    }
    if (t == b.chunks - 1 && lane == 0) {
        b.pair_off[b.n] = base;
        b.toff[b.n] = tbase;
    }
}

// the long rows' edges, a sub a warp
__global__ void __launch_bounds__(HB_WARPS * 32) k_hb_sub_place(HubBuild b)
{
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ uint32_t s_e[HB_WARPS][SEG_MAX + 1];
    uint32_t *pos = s_e[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int32_t nsub = b.nlong[1];
    for (int32_t s = blockIdx.x * HB_WARPS + (threadIdx.x >> 5); s < nsub; s += gridDim.x * HB_WARPS) {
        const int32_t id = b.sub[s];
        const int2 r = b.lrow[id];
        const uint32_t *count = b.lcnt + (size_t)id * b.ncol, *lp = b.lplace + (size_t)id * 2 * b.ncol;
        for (int k = lane; k < b.ncol; k += 32) pos[k] = b.subcnt[(size_t)s * b.ncol + k];
        __syncwarp();
        const int32_t begin = b.prow[r.x], len = hb_sub_len(begin, b.prow[r.x + 1], s - r.y);
        const int32_t *col = b.pcol + hb_sub_begin(begin, s - r.y);
        for (int32_t i = lane; i - lane < len; i += 32) {
            const int32_t c = i < len ? __ldg(&col[i]) : -1;
            const int32_t sg = c < 0 ? 0 : hb_segment(b, c);
            const unsigned same = __match_any_sync(FULL, c < 0 ? -1 : sg);
            const uint32_t first = pos[sg], e = first + __popc(same & ((1u << lane) - 1u));
            __syncwarp();
            if (c >= 0) {
                if (lane == 31 - __clz(same)) pos[sg] = first + __popc(same);
                if (sg == b.nseg) b.tcol[lp[sg] + e] = c;
                else hb_put(b, e, __ldg(&count[sg]), lp[sg], lp[b.ncol + sg], sg, c);
            }
            __syncwarp();
        }
        __syncwarp();
    }
}

// the sectors of P that each group's stores touch
__global__ void __launch_bounds__(256) k_hb_sectors(const int4 *pslot, int32_t ngroups, uint16_t *out)
{
    const int lane = threadIdx.x & 31;
    for (int32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < ngroups; q += (gridDim.x * blockDim.x) >> 5) {
        const int4 s = pslot[(size_t)q * 32 + lane];
        int sectors = 0;
        for (const int32_t x : {s.x, s.y, s.z, s.w}) {
            const int32_t before = __shfl_up_sync(0xffffffffu, x / 8, 1);
            sectors += __popc(__ballot_sync(0xffffffffu, lane == 0 || before != x / 8));
        }
        if (lane == 0) out[q] = (uint16_t)sectors;
    }
}

}  // namespace

namespace mgi {

static std::atomic<uint64_t> g_hub_builds{0};

static double group_cost(int32_t steps, int32_t sectors) { return STEP_COST * steps + GROUP_COST + SECTOR_COST * sectors; }

void hub_free(mg_graph *g)
{
    HubSplit &h = g->hub;
    DevBuf *bufs[] = {&h.hdat, &h.goff, &h.pslot, &h.cpart, &h.pseg, &h.pch, &h.cb, &h.ctime, &h.pair_off, &h.porder,
                      &h.P, &h.toff, &h.tcol, &h.fin};
    for (DevBuf *b : bufs) dev_free(*b);
    h = HubSplit();
}

// Split the groups among the CTAs by the groups' cost weights h.w:
// contiguous ranges of the least largest load, cut at segment boundaries into
// parts and each part into chunks of up to CHUNK_COST that the CTA's warps
// claim one at a time.  The captured loops that launch the sweep take the new
// split (the build number changes).  Even shares of the weight, a staging
// charged to each segment's first group, left CTAs that stage a segment for
// its last few groups: a sweep of R-MAT 20 took 57-68 us by the accident of
// where the cuts fell, 57 now (even shares with a group taken as 16 steps and
// row-major piece sums: 63.5); R-MAT 20 of degree 6 45-55 -> 46 (48), R-MAT 19
// 42-55 -> 43 (46), R-MAT 22 161-170 -> 160 (191).  With chunks bounded by a
// warp's share as well (below), k_hub_sweep alone: R-MAT 18 22 -> 17 us, 19 26 ->
// 23, 20 37.5 -> 35, of degree 6 28 -> 23, 21 61 -> 54.5, 22 as it was (107).
static mg_status hub_split(mg_graph *g)
{
    HubSplit &h = g->hub;
    cudaStream_t s = g->stream;
    const int G = h.grid;
    const int32_t ngroups = (int32_t)h.hglam.size();
    const std::vector<int32_t> &segg = h.hsegg;
    std::vector<double> gcum((size_t)ngroups + 1, 0.0);
    for (int32_t q = 0; q < ngroups; q++) gcum[q + 1] = gcum[q] + h.w[q];
    // CHUNK_COST in units of the weights as they are now
    double wn = 0.0;
    for (int32_t q = 0; q < ngroups; q++) wn += h.w[q];
    const double chunk_w = CHUNK_COST * (h.w0 > 0.0 ? wn / h.w0 : 1.0);
    // the least load T under which G CTAs, filled one after another, take all
    // groups; a CTA pays for every segment that it stages, and leaves a
    // segment that it has no room to stage to the next
    const double stage = STAGE_COST * (h.w0 > 0.0 ? wn / h.w0 : 1.0);
    std::vector<int32_t> cta_lo((size_t)G + 1, ngroups);
    auto fill = [&](double T) {
        int32_t at = 0;
        for (int b = 0; b < G; b++) {
            cta_lo[b] = at;
            double room = T;
            for (bool first = true; at < ngroups; first = false) {
                const int32_t sg = (int32_t)(std::upper_bound(segg.begin(), segg.end(), at) - segg.begin()) - 1;
                room -= stage;
                int32_t e = (int32_t)(std::upper_bound(gcum.begin() + at, gcum.begin() + segg[sg + 1] + 1, gcum[at] + room) -
                                      gcum.begin()) - 1;
                e = std::max(e, first ? at + 1 : at);
                if (e <= at) break;
                room -= gcum[e] - gcum[at];
                at = e;
                if (at < segg[sg + 1]) break;
            }
        }
        return at == ngroups;
    };
    double lo_t = 0.0, hi_t = gcum[ngroups] + stage * (double)segg.size();
    for (int it = 0; it < 40; it++) {
        const double T = 0.5 * (lo_t + hi_t);
        (fill(T) ? hi_t : lo_t) = T;
    }
    fill(hi_t);
    cta_lo[G] = ngroups;
    std::vector<int32_t> cpart((size_t)G + 1, 0), pseg, pch, cb;
    for (int b = 0; b < G; b++) {
        cpart[b] = (int32_t)pseg.size();
        int32_t lo = cta_lo[b];
        const int32_t hi = cta_lo[b + 1];
        while (lo < hi) {
            const int32_t sg = (int32_t)(std::upper_bound(segg.begin(), segg.end(), lo) - segg.begin()) - 1;
            const int32_t e = std::min(hi, segg[sg + 1]);
            pseg.push_back(sg);
            pch.push_back((int32_t)cb.size());
            // A chunk takes groups while they stay within CHUNK_COST and
            // within a warp's even share of the part: a warp with two groups
            // of a part that has fewer groups than the CTA warps doubles the
            // part's time (cuts of equal weight, groups of 64 steps: a band of
            // 200 K rows 36 us a sweep, 26 so; directed R-MAT 18 21, 19)
            const double most = std::min(chunk_w, (gcum[e] - gcum[lo]) / (HUB_THREADS / 32));
            for (int32_t q = lo; q < e; q++)
                if (q == lo || gcum[q + 1] - gcum[cb.back()] > most) cb.push_back(q);
            lo = e;
        }
    }
    cpart[G] = (int32_t)pseg.size();
    pch.push_back((int32_t)cb.size());
    cb.push_back(ngroups);
    auto up = [&](DevBuf &b, const void *src, size_t bytes) -> mg_status {
        MG_TRY(dev_alloc(b, std::max<size_t>(bytes, 16) + 16));
        if (bytes) MG_CUDA(cudaMemcpyAsync(b.p, src, bytes, cudaMemcpyHostToDevice, s));
        return MG_OK;
    };
    MG_TRY(up(h.cpart, cpart.data(), cpart.size() * 4));
    MG_TRY(up(h.pseg, pseg.data(), pseg.size() * 4));
    MG_TRY(up(h.pch, pch.data(), pch.size() * 4));
    MG_TRY(up(h.cb, cb.data(), cb.size() * 4));
    MG_CUDA(cudaStreamSynchronize(s));   // the host vectors go out of scope
    h.gen = ++g_hub_builds;
    return MG_OK;
}

// The layout from a pull CSR on the host (prow [n+1], pcol [m], engine ids),
// what the device's builder is checked against: row-parallel passes over the edges (count, then write)
// on nt threads, each a contiguous row range whose pieces take consecutive
// places in every (segment, length) bucket, so buckets come out rows
// ascending and the layout does not depend on nt.  o.use stays false when a
// quarter of the edges or fewer fall in the segments.
struct HubHost {
    bool use = false;
    int32_t H = 0, nseg = 0, nfw = 0;
    int64_t covered = 0, npieces = 0;
    std::vector<uint16_t> hdat;
    std::vector<uint16_t> porder;
    std::vector<int32_t> goff, pslot, glam, segg, pair_off, toff, tcol, fin;
};

static mg_status build_hub(const std::vector<int32_t> &prow, const std::vector<int32_t> &pcol, int32_t n, int64_t m,
                           int nt, HubHost &o)
{
    const int32_t H = SEG_H;
    const int32_t nseg = std::min<int32_t>(SEG_MAX, (n + H - 1) / H);
    const int64_t cover = std::min<int64_t>(n, (int64_t)nseg * H);
    constexpr int32_t L = PIECE_MAX;
    o = HubHost();
    o.H = H;
    o.nseg = nseg;
    nt = std::max(1, std::min(nt, 32));
    // row ranges of equal edge counts
    std::vector<int32_t> rlo((size_t)nt + 1, n);
    rlo[0] = 0;
    for (int t = 1; t < nt; t++) {
        const int64_t goal = m * t / nt;
        rlo[t] = (int32_t)(std::lower_bound(prow.begin(), prow.end(), (int32_t)goal) - prow.begin());
        rlo[t] = std::min(std::max((rlo[t] + 31) & ~31, rlo[t - 1]), n);   // whole windows
    }
    auto run = [&](const std::function<void(int)> &fn) {
        std::vector<std::thread> th;
        for (int t = 1; t < nt; t++) th.emplace_back(fn, t);
        fn(0);
        for (auto &x : th) x.join();
    };
    // bucket (segment sg, piece length lam) of thread t: bc[(t * nseg + sg) * (L + 1) + lam]
    const size_t NB = (size_t)nseg * (L + 1);
    std::vector<int64_t> bc((size_t)nt * NB, 0), tcov((size_t)nt, 0);
    std::vector<int32_t> npc((size_t)n, 0), ntl((size_t)n, 0);
    // pass 1: per row its pieces and tail edges; per thread its bucket counts
    run([&](int t) {
        int64_t *b = &bc[(size_t)t * NB];
        int32_t cnt[SEG_MAX];
        int64_t cov = 0;
        for (int32_t v = rlo[t]; v < rlo[t + 1]; v++) {
            std::memset(cnt, 0, sizeof(int32_t) * nseg);
            int32_t tl = 0;
            for (int32_t p = prow[v]; p < prow[v + 1]; p++) {
                const int32_t c = pcol[p];
                if (c < cover) cnt[c / H]++;
                else tl++;
            }
            int32_t pieces = 0;
            for (int sg = 0; sg < nseg; sg++) {
                if (!cnt[sg]) continue;
                cov += cnt[sg];
                const int32_t full = cnt[sg] / L, rem = cnt[sg] % L;
                b[(size_t)sg * (L + 1) + L] += full;
                if (rem) b[(size_t)sg * (L + 1) + rem]++;
                pieces += full + (rem ? 1 : 0);
            }
            npc[v] = pieces;
            ntl[v] = tl;
        }
        tcov[t] = cov;
    });
    int64_t covered = 0;
    for (int64_t x : tcov) covered += x;
    o.covered = covered;
    // the segmented pull pays when a quarter of the edges or more are covered
    if (covered * 4 < m) return MG_OK;
    // buckets in order: segments ascending, lengths descending; each padded
    // to whole groups.  tb: thread t's first place in its bucket.
    std::vector<int64_t> tb((size_t)nt * NB, 0);
    std::vector<int32_t> segg((size_t)nseg + 1, 0);
    std::vector<int32_t> glam;      // steps of every group
    int64_t place = 0;              // padded place of the next bucket's first piece
    for (int sg = 0; sg < nseg; sg++) {
        segg[sg] = (int32_t)glam.size();
        for (int32_t lam = L; lam >= 1; lam--) {
            const size_t k = (size_t)sg * (L + 1) + lam;
            int64_t size = 0;
            for (int t = 0; t < nt; t++) {
                tb[(size_t)t * NB + k] = place + size;
                size += bc[(size_t)t * NB + k];
            }
            const int64_t groups = (size + GROUP - 1) / GROUP;
            for (int64_t q = 0; q < groups; q++) glam.push_back(lam);
            place += groups * GROUP;
        }
    }
    const int32_t ngroups = (int32_t)glam.size();
    segg[nseg] = ngroups;
    std::vector<int64_t> goff64((size_t)ngroups + 1, 0);
    for (int32_t q = 0; q < ngroups; q++) goff64[q + 1] = goff64[q] + glam[q];
    std::vector<int32_t> pair_off((size_t)n + 1, 0), toff((size_t)n + 1, 0);
    for (int32_t v = 0; v < n; v++) {
        pair_off[v + 1] = pair_off[v] + npc[v];
        toff[v + 1] = toff[v] + ntl[v];
    }
    const int64_t npieces = pair_off[n];
    if (npieces >= INT32_MAX || goff64[ngroups] >= INT32_MAX)
        return fail(MG_ERR_RANGE, "segmented PageRank layout too large");
    std::vector<int32_t> goff(goff64.begin(), goff64.end());
    std::vector<uint16_t> hdat((size_t)goff64[ngroups] * GROUP, (uint16_t)H);
    std::vector<int32_t> pslot((size_t)ngroups * GROUP, (int32_t)npieces);
    std::vector<int32_t> tcol((size_t)toff[n]);
    std::vector<uint16_t> porder(toff[n] == 0 ? (size_t)npieces : 0);
    // pass 2: every row's pieces into their buckets, every edge into its
    // piece's step and lane, a window of 32 rows at a time
    run([&](int t) {
        std::vector<int64_t> next(tb.begin() + (size_t)t * NB, tb.begin() + (size_t)(t + 1) * NB);
        int32_t cnts[32][SEG_MAX], full[SEG_MAX], e[SEG_MAX];
        int64_t qfull[SEG_MAX], qrem[SEG_MAX];
        std::vector<uint32_t> key;       // the window's pieces: (segment, length descending, place in row order)
        std::vector<int32_t> at;         // their places in P from the window's first
        int32_t base = 0;
        for (int32_t v = rlo[t]; v < rlo[t + 1]; v++) {
            if (v % 32 == 0) {
                const int32_t vend = std::min(v + 32, n);
                base = pair_off[v];
                key.clear();
                at.clear();
                bool sorted = toff[n] == 0 && pair_off[vend] - base <= HUB_WIN;
                for (int32_t u = v; u < vend; u++) {
                    int32_t *cnt = cnts[u - v];
                    std::memset(cnt, 0, sizeof(int32_t) * nseg);
                    int32_t tp = toff[u];
                    for (int32_t p = prow[u]; p < prow[u + 1]; p++) {
                        const int32_t c = pcol[p];
                        if (c < cover) cnt[c / H]++;
                        else tcol[tp++] = c;
                    }
                    sorted = sorted && npc[u] <= FIN_WARP;
                    if (!sorted) continue;
                    for (int sg = 0; sg < nseg; sg++)
                        for (int32_t left = cnt[sg]; left > 0; left -= L)
                            key.push_back((uint32_t)sg << 16 | (uint32_t)(L - std::min(left, L)) << 9 |
                                          (uint32_t)key.size());
                }
                at.resize((size_t)(pair_off[vend] - base));
                if (sorted) std::sort(key.begin(), key.end());
                for (size_t i = 0; i < at.size(); i++) {
                    const int32_t k = sorted ? (int32_t)(key[i] & 511u) : (int32_t)i;
                    at[k] = (int32_t)i;
                    if (!porder.empty()) porder[(size_t)base + i] = (uint16_t)k;
                }
            }
            const int32_t *cnt = cnts[v % 32];
            int32_t piece = pair_off[v] - base;   // the row's pieces: segments ascending, pieces in order
            for (int sg = 0; sg < nseg; sg++) {
                e[sg] = 0;
                if (!cnt[sg]) continue;
                full[sg] = cnt[sg] / L;
                const int32_t rem = cnt[sg] % L;
                int64_t &nf = next[(size_t)sg * (L + 1) + L];
                qfull[sg] = nf;
                for (int32_t i = 0; i < full[sg]; i++, nf++)
                    pslot[(size_t)(nf / GROUP * GROUP + group_place(nf))] = base + at[piece++];
                if (rem) {
                    int64_t &nr = next[(size_t)sg * (L + 1) + rem];
                    qrem[sg] = nr;
                    pslot[(size_t)(nr / GROUP * GROUP + group_place(nr))] = base + at[piece++];
                    nr++;
                }
            }
            for (int32_t p = prow[v]; p < prow[v + 1]; p++) {
                const int32_t c = pcol[p];
                if (c >= cover) continue;
                const int sg = c / H;
                const int32_t i = e[sg] / L, k = e[sg] % L;
                e[sg]++;
                const int64_t q = i < full[sg] ? qfull[sg] + i : qrem[sg];
                const int64_t grp = q / GROUP;
                hdat[(size_t)(goff64[grp] * GROUP + (int64_t)k * GROUP + group_place(q))] = (uint16_t)(c - sg * H);
            }
        }
    });
    o.hdat.swap(hdat);
    o.goff.swap(goff);
    o.pslot.swap(pslot);
    o.porder.swap(porder);
    o.glam.swap(glam);
    o.segg.swap(segg);
    o.pair_off.swap(pair_off);
    o.toff.swap(toff);
    o.tcol.swap(tcol);
    o.npieces = npieces;
    o.use = true;
    // rows of more than FIN_WARP pieces, which k_pr_seg sums a warp each
    // (graphs without a tail finish every row there)
    for (int32_t v = 0; v < n; v++)
        if (npc[v] > FIN_WARP) o.fin.push_back(v);
    o.nfw = (int32_t)o.fin.size();
    return MG_OK;
}

namespace {
// device buffers for the time of a build
struct BuildBufs {
    DevBuf table, total, place, hid, nlong, lrow, sub, subcnt, lcnt, lplace, sectors;
    ~BuildBufs()
    {
        for (DevBuf *b : {&table, &total, &place, &hid, &nlong, &lrow, &sub, &subcnt, &lcnt, &lplace, &sectors}) dev_free(*b);
    }
};
}  // namespace

// Build the segmented layout from the pull CSR on the device and split the
// sweep's work among the CTAs (first PageRank call with the layout built on
// the host -> here: R-MAT 22 434 -> 17 ms, R-MAT 20 69 -> 5, R-MAT 19 29 -> 3).
mg_status hub_prepare(mg_graph *g)
{
    HubSplit &h = g->hub;
    if (h.valid) return MG_OK;
    h.gen = ++g_hub_builds;
    h.use = false;
    cudaStream_t s = g->stream;
    const int32_t n = g->nv;
    const int64_t m = g->ne;
    if (n < 4 || m == 0) {
        h.valid = true;
        return MG_OK;
    }
    constexpr int32_t L = PIECE_MAX;
    HubBuild b;
    std::memset(&b, 0, sizeof(b));
    b.prow = g->trow;
    b.pcol = g->tcol;
    b.n = n;
    b.nseg = std::min<int32_t>(SEG_MAX, (n + SEG_H - 1) / SEG_H);
    b.cover = (int32_t)std::min<int64_t>(n, (int64_t)b.nseg * SEG_H);
    b.chunks = std::min(HB_CHUNKS, (n + 31) / 32);
    b.nb = b.nseg * (L + 1);
    b.ncol = b.nseg + 1;
    b.stride = b.ncol | 1;
    const size_t nlong = (size_t)(m / HB_ROW) + 1, nsub = 2 * nlong, tw = (size_t)b.nb + 3;
    BuildBufs t;
    auto make = [&](DevBuf &buf, size_t bytes, auto *&ptr) -> mg_status {
        MG_TRY(dev_alloc(buf, std::max<size_t>(bytes, 16) + 16));
        ptr = buf.as<std::remove_reference_t<decltype(*ptr)>>();
        return MG_OK;
    };
    MG_TRY(make(t.table, (size_t)b.chunks * tw * 4, b.table));
    MG_TRY(make(t.total, tw * 4, b.total));
    MG_TRY(make(t.place, (size_t)b.nb * 4, b.place));
    MG_TRY(make(t.hid, (size_t)n * 4, b.hid));
    MG_TRY(make(t.nlong, 8, b.nlong));
    MG_TRY(make(t.lrow, nlong * 8, b.lrow));
    MG_TRY(make(t.sub, nsub * 4, b.sub));
    MG_TRY(make(t.subcnt, nsub * b.ncol * 4, b.subcnt));
    MG_TRY(make(t.lcnt, nlong * b.ncol * 4, b.lcnt));
    MG_TRY(make(t.lplace, nlong * 2 * b.ncol * 4, b.lplace));
    const int grid = launch_grid(g, 256, 4), wgrid = (b.chunks + HB_WARPS - 1) / HB_WARPS;
    const size_t sm_count = (size_t)HB_WARPS * (32 * b.stride + b.nb) * 4,
                 sm_place = (size_t)HB_WARPS * (3 * 32 * b.stride + 2 * HUB_WIN) * 4;
    MG_CUDA(cudaFuncSetAttribute(k_hb_count, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_count));
    MG_CUDA(cudaFuncSetAttribute(k_hb_place, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_place));
    MG_CUDA(cudaMemsetAsync(b.nlong, 0, 8, s));
    k_hb_long<<<grid, 256, 0, s>>>(b);
    k_hb_sub_count<<<grid, HB_WARPS * 32, 0, s>>>(b);
    k_hb_long_scan<<<grid, 128, 0, s>>>(b);
    k_hb_count<<<wgrid, HB_WARPS * 32, sm_count, s>>>(b);
    k_hb_scan<<<(int)((tw + 31) / 32), 1024, 0, s>>>(b);
    MG_CUDA(cudaGetLastError());
    std::vector<uint32_t> total(tw), place((size_t)b.nb, 0);
    MG_CUDA(cudaMemcpyAsync(total.data(), b.total, tw * 4, cudaMemcpyDeviceToHost, s));
    MG_CUDA(cudaStreamSynchronize(s));
    const int64_t npieces = total[b.nb], ntail = total[b.nb + 1];
    h.covered = m - ntail;
    // the segmented pull pays when a quarter of the edges or more are covered
    if (h.covered * 4 < m) {
        h.valid = true;
        return MG_OK;
    }
    // buckets in order: segments ascending, lengths descending; each padded
    // to whole groups
    h.hglam.clear();
    h.hsegg.assign((size_t)b.nseg + 1, 0);
    std::vector<int32_t> goff(1, 0);
    int64_t steps = 0;
    for (int32_t sg = 0; sg < b.nseg; sg++) {
        h.hsegg[sg] = (int32_t)h.hglam.size();
        for (int32_t lam = L; lam >= 1; lam--) {
            const size_t k = (size_t)sg * (L + 1) + lam;
            place[k] = (uint32_t)(h.hglam.size() * GROUP);
            for (uint32_t q = 0; q < (total[k] + GROUP - 1) / GROUP; q++) {
                h.hglam.push_back(lam);
                steps += lam;
                goff.push_back((int32_t)steps);
            }
        }
    }
    const int32_t ngroups = (int32_t)h.hglam.size();
    h.hsegg[b.nseg] = ngroups;
    if (npieces >= INT32_MAX || steps >= INT32_MAX) return fail(MG_ERR_RANGE, "segmented PageRank layout too large");
    b.ntail = (int32_t)ntail;
    h.nfw = (int32_t)total[b.nb + 2];
    const size_t words = (size_t)steps * GROUP / 2, slots = (size_t)ngroups * GROUP;
    MG_TRY(make(h.hdat, words * 4, b.hdat));
    MG_TRY(make(h.goff, goff.size() * 4, b.goff));
    MG_TRY(make(h.pslot, slots * 4, b.pslot));
    MG_TRY(make(h.pair_off, ((size_t)n + 1) * 4, b.pair_off));
    MG_TRY(make(h.porder, ntail == 0 ? (size_t)npieces * 2 : 0, b.porder));
    MG_TRY(make(h.toff, ((size_t)n + 1) * 4, b.toff));
    MG_TRY(make(h.tcol, (size_t)ntail * 4, b.tcol));
    MG_TRY(make(h.fin, (size_t)h.nfw * 4, b.fin));
    MG_TRY(dev_alloc(h.P, (size_t)(npieces + 1) * 4));
    uint16_t *sectors = nullptr;
    MG_TRY(make(t.sectors, (size_t)ngroups * 2, sectors));
    MG_CUDA(cudaMemcpyAsync(t.place.p, place.data(), place.size() * 4, cudaMemcpyHostToDevice, s));
    MG_CUDA(cudaMemcpyAsync(h.goff.p, goff.data(), goff.size() * 4, cudaMemcpyHostToDevice, s));
    k_hb_fill<<<grid, 256, 0, s>>>(h.hdat.as<uint32_t>(), (uint32_t)SEG_H << 16 | (uint32_t)SEG_H, (long long)words);
    k_hb_fill<<<grid, 256, 0, s>>>(h.pslot.as<uint32_t>(), (uint32_t)npieces, (long long)slots);
    k_hb_place<<<wgrid, HB_WARPS * 32, sm_place, s>>>(b);
    k_hb_sub_place<<<grid, HB_WARPS * 32, 0, s>>>(b);
    k_hb_sectors<<<grid, 256, 0, s>>>(h.pslot.as<int4>(), ngroups, sectors);
    MG_CUDA(cudaGetLastError());
    std::vector<uint16_t> sec((size_t)ngroups);
    MG_CUDA(cudaMemcpyAsync(sec.data(), sectors, sec.size() * 2, cudaMemcpyDeviceToHost, s));
    MG_CUDA(cudaStreamSynchronize(s));
    h.w.resize((size_t)ngroups);
    for (int32_t q = 0; q < ngroups; q++) h.w[q] = group_cost(h.hglam[q], sec[q]);
    h.w0 = 0.0;
    for (double x : h.w) h.w0 += x;
    h.grid = g->num_sms;
    MG_TRY(dev_alloc(h.ctime, (size_t)h.grid * 8));
    MG_TRY(hub_split(g));
    h.H = SEG_H;
    h.nseg = b.nseg;
    h.ngroups = ngroups;
    h.npieces = npieces;
    h.ntail = ntail;
    h.fin_warp = FIN_WARP;
    h.use = true;
    h.valid = true;
    return MG_OK;
}

bool hub_covers_all(const mg_graph *g) { return (int64_t)g->nv <= (int64_t)SEG_MAX * SEG_H; }

// Re-split the sweep's work from the last sweep's per-CTA clock counts:
// every group's weight is scaled by its CTA's measured time over the
// CTA's share of the weight (normalised to the mean), so groups whose real
// cost the initial model misjudges move to other CTAs.
mg_status hub_rebalance(mg_graph *g)
{
    HubSplit &h = g->hub;
    if (!h.use) return MG_OK;
    const int G = h.grid;
    std::vector<long long> t((size_t)G);
    std::vector<int32_t> cpart((size_t)G + 1), pch, cb;
    MG_CUDA(cudaMemcpyAsync(t.data(), h.ctime.p, (size_t)G * 8, cudaMemcpyDeviceToHost, g->stream));
    MG_CUDA(cudaMemcpyAsync(cpart.data(), h.cpart.p, cpart.size() * 4, cudaMemcpyDeviceToHost, g->stream));
    MG_CUDA(cudaStreamSynchronize(g->stream));
    // each CTA's first and last group: from its parts' chunks
    const size_t nparts = (size_t)cpart[G];
    pch.resize(nparts + 1);
    MG_CUDA(cudaMemcpy(pch.data(), h.pch.p, pch.size() * 4, cudaMemcpyDeviceToHost));
    cb.resize((size_t)pch[nparts] + 1);
    MG_CUDA(cudaMemcpy(cb.data(), h.cb.p, cb.size() * 4, cudaMemcpyDeviceToHost));
    std::vector<double> ratio((size_t)G, 0.0);
    double tt = 0.0, tw = 0.0;
    for (int b = 0; b < G; b++) {
        if (cpart[b] == cpart[b + 1]) continue;
        const int32_t lo = cb[(size_t)pch[(size_t)cpart[b]]], hi = cb[(size_t)pch[(size_t)cpart[b + 1]]];
        double wb = 0.0;
        for (int32_t q = lo; q < hi; q++) wb += h.w[q];
        if (wb <= 0.0 || t[b] <= 0) continue;
        ratio[b] = (double)t[b] / wb;
        tt += (double)t[b];
        tw += wb;
    }
    if (tt <= 0.0 || tw <= 0.0) return MG_OK;
    const double mean = tt / tw;
    for (int b = 0; b < G; b++) {
        if (ratio[b] <= 0.0) continue;
        const int32_t lo = cb[(size_t)pch[(size_t)cpart[b]]], hi = cb[(size_t)pch[(size_t)cpart[b + 1]]];
        for (int32_t q = lo; q < hi; q++) h.w[q] *= ratio[b] / mean;
    }
    return hub_split(g);
}

// Read (get) or replace (set) the groups' cost weights; false when the
// segmented layout is not in use or set has the wrong length.
bool hub_weights(mg_graph *g, std::vector<double> *get, const std::vector<double> *set)
{
    HubSplit &h = g->hub;
    if (!h.use) return false;
    if (get) *get = h.w;
    if (set) {
        if (set->size() != h.w.size()) return false;
        h.w = *set;
        if (hub_split(g) != MG_OK) return false;
    }
    return true;
}

size_t hub_smem_bytes(const mg_graph *g) { return (size_t)(g->hub.H + 4) * 4; }

mg_status hub_launch(mg_graph *g, const float *c0, const float *c1, const int32_t *cur, const int32_t *more,
                     const int32_t *off, cudaStream_t st, int slot_sweep)
{
    HubSplit &h = g->hub;
    HubArgs a;
    std::memset(&a, 0, sizeof(a));
    a.hdat = h.hdat.as<uint2>();
    a.goff = h.goff.as<int32_t>();
    a.pslot = h.pslot.as<int4>();
    a.cpart = h.cpart.as<int32_t>();
    a.pseg = h.pseg.as<int32_t>();
    a.pch = h.pch.as<int32_t>();
    a.cb = h.cb.as<int32_t>();
    a.c[0] = c0;
    a.c[1] = c1;
    a.cur = cur;
    a.more = more;
    a.off = off;
    a.P = h.P.as<float>();
    a.ctime = h.ctime.as<long long>();
    a.n = g->nv;
    a.H = h.H;
    a.nseg = h.nseg;
    const size_t smem = hub_smem_bytes(g);
    MG_CUDA(cudaFuncSetAttribute(k_hub_sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    Profiler &P = g->prof;
    P.begin(slot_sweep);
    k_hub_sweep<<<h.grid, HUB_THREADS, smem, st>>>(a);
    P.end();
    MG_CUDA(cudaGetLastError());
    return MG_OK;
}

// The sweep has no waits of its own (plain loads stage the segments), so
// there is nothing to report after a run.
mg_status hub_check(mg_graph *) { return MG_OK; }

}  // namespace mgi

// ---------------------------------------------------------------------------
// The layout that the device built for g, against the host's, byte for byte.
// ---------------------------------------------------------------------------
extern "C" mg_status mg_selftest_segmented_build(mg_graph *g, int64_t *pieces_out)
{
    using namespace mgi;
    clear_error();
    if (!g || !pieces_out) return fail(MG_ERR_INVALID, "null argument");
    MG_CUDA(cudaSetDevice(g->device));
    *pieces_out = 0;
    MG_TRY(hub_prepare(g));
    HubSplit &h = g->hub;
    const int32_t n = g->nv;
    const int64_t m = g->ne;
    if (n < 4 || m == 0) return h.use ? fail(MG_ERR_INTERNAL, "segmented layout of nothing") : MG_OK;
    std::vector<int32_t> prow((size_t)n + 1), pcol((size_t)m);
    MG_CUDA(cudaMemcpy(prow.data(), g->trow, prow.size() * 4, cudaMemcpyDeviceToHost));
    MG_CUDA(cudaMemcpy(pcol.data(), g->tcol, pcol.size() * 4, cudaMemcpyDeviceToHost));
    HubHost o;
    MG_TRY(build_hub(prow, pcol, n, m, host_threads(0), o));
    if (o.use != h.use || o.covered != h.covered) return fail(MG_ERR_INTERNAL, "segmented build: covered edges");
    if (!o.use) return MG_OK;
    if (o.nseg != h.nseg || o.npieces != h.npieces || o.glam != h.hglam || o.segg != h.hsegg || o.nfw != h.nfw ||
        (int64_t)o.tcol.size() != h.ntail)
        return fail(MG_ERR_INTERNAL, "segmented build: sizes");
    auto same = [&](const DevBuf &d, const auto &v, const char *what) -> mg_status {
        std::vector<char> got(v.size() * sizeof(v[0]));
        if (!got.empty()) MG_CUDA(cudaMemcpy(got.data(), d.p, got.size(), cudaMemcpyDeviceToHost));
        if (!got.empty() && std::memcmp(got.data(), v.data(), got.size()))
            return fail(MG_ERR_INTERNAL, "segmented build: %s", what);
        return MG_OK;
    };
    MG_TRY(same(h.goff, o.goff, "group offsets"));
    MG_TRY(same(h.pair_off, o.pair_off, "piece offsets"));
    MG_TRY(same(h.toff, o.toff, "tail offsets"));
    MG_TRY(same(h.tcol, o.tcol, "tail"));
    MG_TRY(same(h.fin, o.fin, "warp rows"));
    MG_TRY(same(h.porder, o.porder, "window order"));
    MG_TRY(same(h.pslot, o.pslot, "slots"));
    MG_TRY(same(h.hdat, o.hdat, "ids"));
    *pieces_out = o.npieces;
    return MG_OK;
}

// ---------------------------------------------------------------------------
// Host-only check of the segmented layout (no GPU): builds it from a host
// pull CSR on `threads` threads and on one, requires the two to be equal,
// and verifies every invariant the sweep and the row finish rely on, with
// exact integer sums (each edge's id + 1 in place of its contribution).
// ---------------------------------------------------------------------------
extern "C" mg_status mg_selftest_segmented_layout(int32_t nv, int64_t ne, const int32_t *row, const int32_t *col,
                                                  int32_t threads, int64_t *pieces_out)
{
    using namespace mgi;
    clear_error();
    if (!row || (ne > 0 && !col) || !pieces_out || nv < 0 || ne < 0 || ne > INT32_MAX)
        return fail(MG_ERR_INVALID, "bad argument");
    if (row[0] != 0 || row[nv] != ne) return fail(MG_ERR_INVALID, "row offsets must run from 0 to ne");
    for (int32_t v = 0; v < nv; v++)
        if (row[v + 1] < row[v]) return fail(MG_ERR_INVALID, "row offsets decrease at row %d", v);
    for (int64_t p = 0; p < ne; p++)
        if (col[p] < 0 || col[p] >= nv) return fail(MG_ERR_INVALID, "column id out of range at %lld", (long long)p);
    *pieces_out = 0;
    // the device build's subs tile a long row, wherever it lies
    const int32_t ends[][2] = {{0, HB_ROW + 1}, {5, 5 + 2 * HB_ROW}, {INT32_MAX - 5000, INT32_MAX},
                               {INT32_MAX - 2 * HB_ROW - 1, INT32_MAX - 1}, {0, INT32_MAX}};
    for (const auto &r : ends) {
        int64_t at = r[0];
        const int32_t ns = hb_subs(r[0], r[1]);
        for (int32_t s = 0; s < ns; s++) {
            const int32_t len = hb_sub_len(r[0], r[1], s);
            if (hb_sub_begin(r[0], s) != at || len < 1 || len > HB_ROW)
                return fail(MG_ERR_INTERNAL, "segmented build: sub %d of the row at %d", s, r[0]);
            at += len;
        }
        if (at != r[1]) return fail(MG_ERR_INTERNAL, "segmented build: subs of the row at %d", r[0]);
    }
    if (nv < 4 || ne == 0) return MG_OK;
    const std::vector<int32_t> prow(row, row + nv + 1), pcol(col, col + ne);
    HubHost a, b;
    MG_TRY(build_hub(prow, pcol, nv, ne, threads, a));
    MG_TRY(build_hub(prow, pcol, nv, ne, 1, b));
    if (a.use != b.use || a.covered != b.covered || a.npieces != b.npieces || a.hdat != b.hdat || a.goff != b.goff ||
        a.pslot != b.pslot || a.porder != b.porder || a.glam != b.glam || a.segg != b.segg || a.pair_off != b.pair_off || a.toff != b.toff ||
        a.tcol != b.tcol || a.fin != b.fin)
        return fail(MG_ERR_INTERNAL, "segmented layout differs between %d threads and one", threads);
    if (!a.use) return MG_OK;
    const int32_t H = a.H, nseg = a.nseg;
    const int64_t cover = std::min<int64_t>(nv, (int64_t)nseg * H);
    const int64_t np = a.npieces;
    const int32_t ngroups = (int32_t)a.glam.size();
    if ((int32_t)a.goff.size() != ngroups + 1 || (int64_t)a.hdat.size() != (int64_t)a.goff[ngroups] * GROUP ||
        (int64_t)a.pslot.size() != (int64_t)ngroups * GROUP || (int32_t)a.segg.size() != nseg + 1 ||
        a.segg[0] != 0 || a.segg[nseg] != ngroups || (int32_t)a.pair_off.size() != nv + 1 || a.pair_off[0] != 0 ||
        a.pair_off[nv] != np || (int32_t)a.toff.size() != nv + 1)
        return fail(MG_ERR_INTERNAL, "segmented layout: array sizes");
    // every packed piece: its slot (once), segment, length and id sum
    std::vector<int32_t> seen((size_t)np, 0), pseg((size_t)np, -1), plen((size_t)np, 0);
    std::vector<int64_t> psum((size_t)np, 0);
    for (int32_t sg = 0; sg < nseg; sg++) {
        for (int32_t q = a.segg[sg]; q < a.segg[sg + 1]; q++) {
            const int32_t lam = a.goff[q + 1] - a.goff[q];
            if (lam != a.glam[q] || lam < 1 || lam > PIECE_MAX || (q > a.segg[sg] && lam > a.glam[q - 1]))
                return fail(MG_ERR_INTERNAL, "segmented layout: group %d length", q);
            for (int32_t j = 0; j < GROUP; j++) {
                const int32_t slot = a.pslot[(size_t)q * GROUP + j];
                int64_t sum = 0;
                bool pad = true, real = true;
                for (int32_t k = 0; k < lam; k++) {
                    const int32_t id = a.hdat[((size_t)a.goff[q] + k) * GROUP + j];
                    pad = pad && id == H;
                    real = real && id < H && (int64_t)sg * H + id < nv;
                    sum += (int64_t)sg * H + id + 1;
                }
                if (slot == np) {
                    if (!pad) return fail(MG_ERR_INTERNAL, "segmented layout: padding of group %d", q);
                    continue;
                }
                if (slot < 0 || slot > np || !real || seen[slot]++)
                    return fail(MG_ERR_INTERNAL, "segmented layout: piece %d of group %d", j, q);
                pseg[slot] = sg;
                plen[slot] = lam;
                psum[slot] = sum;
            }
        }
    }
    for (int64_t p = 0; p < np; p++)
        if (seen[p] != 1) return fail(MG_ERR_INTERNAL, "segmented layout: slot %lld unused", (long long)p);
    // sorted windows back in row order: porder is a permutation of each, and
    // the identity where the row finish reads P directly
    if (a.porder.size() != (a.tcol.empty() ? (size_t)np : 0))
        return fail(MG_ERR_INTERNAL, "segmented layout: window order size");
    for (int32_t vb = 0; vb < nv && !a.porder.empty(); vb += 32) {
        const int32_t ve = std::min(vb + 32, nv), base = a.pair_off[vb], len = a.pair_off[ve] - base;
        bool sorted = len <= HUB_WIN;
        for (int32_t v = vb; v < ve; v++) sorted = sorted && a.pair_off[v + 1] - a.pair_off[v] <= FIN_WARP;
        if (!sorted) {   // (never read there; the low 16 bits of the place)
            for (int32_t i = 0; i < len; i++)
                if (a.porder[(size_t)base + i] != (uint16_t)i)
                    return fail(MG_ERR_INTERNAL, "segmented layout: order of the window of row %d", vb);
            continue;
        }
        const std::vector<int32_t> s0(pseg.begin() + base, pseg.begin() + base + len),
            l0(plen.begin() + base, plen.begin() + base + len);
        const std::vector<int64_t> x0(psum.begin() + base, psum.begin() + base + len);
        std::vector<int32_t> used((size_t)len, 0);
        for (int32_t i = 0; i < len; i++) {
            const int32_t k = a.porder[(size_t)base + i];
            if (k >= len || used[k]++)
                return fail(MG_ERR_INTERNAL, "segmented layout: order of the window of row %d", vb);
            pseg[base + k] = s0[i];
            plen[base + k] = l0[i];
            psum[base + k] = x0[i];
        }
    }
    // every row: its pieces (segments ascending, full pieces first) hold
    // exactly its covered in-edges; its tail holds the rest in row order
    std::vector<int32_t> fin;
    for (int32_t v = 0; v < nv; v++) {
        int64_t cnt[SEG_MAX] = {0}, sum[SEG_MAX] = {0};
        std::vector<int32_t> tail;
        for (int32_t p = row[v]; p < row[v + 1]; p++) {
            if (col[p] < cover) {
                cnt[col[p] / H]++;
                sum[col[p] / H] += (int64_t)col[p] + 1;
            } else {
                tail.push_back(col[p]);
            }
        }
        int64_t pcnt[SEG_MAX] = {0}, pss[SEG_MAX] = {0};
        for (int32_t p = a.pair_off[v]; p < a.pair_off[v + 1]; p++) {
            const int32_t sg = pseg[p];
            if (p > a.pair_off[v] && sg < pseg[p - 1]) return fail(MG_ERR_INTERNAL, "row %d: segments out of order", v);
            if (p > a.pair_off[v] && sg == pseg[p - 1] && plen[p - 1] != PIECE_MAX)
                return fail(MG_ERR_INTERNAL, "row %d: a short piece before another of its segment", v);
            pcnt[sg] += plen[p];
            pss[sg] += psum[p];
        }
        for (int32_t sg = 0; sg < nseg; sg++)
            if (pcnt[sg] != cnt[sg] || pss[sg] != sum[sg])
                return fail(MG_ERR_INTERNAL, "row %d: segment %d holds other edges", v, sg);
        if (a.toff[v + 1] - a.toff[v] != (int32_t)tail.size() ||
            !std::equal(tail.begin(), tail.end(), a.tcol.begin() + a.toff[v]))
            return fail(MG_ERR_INTERNAL, "row %d: tail", v);
        if (a.pair_off[v + 1] - a.pair_off[v] > FIN_WARP) fin.push_back(v);
    }
    if (fin != a.fin) return fail(MG_ERR_INTERNAL, "segmented layout: warp-row list");
    *pieces_out = np;
    return MG_OK;
}
