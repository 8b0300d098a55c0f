// mg_frontier_engine.cuh -- the hybrid push/pull frontier engine, a
// template over the operator (include/mg_ops.cuh): BFS, SSSP and the BC
// forward sweep are instantiations, and so is any operator a caller defines
// with the same hooks and capability flags (include/mg_plugin.cuh).
//
// Replaces MultiGraph_V_E_V (process.cu:1079-1368) with its kernels
// process_f1 / make_frontier / phase1 / phase11 / phase2 and the sampling
// heuristic; the reference selects the operator by macro (user_function.h).
//
// The loop lives inside a CUDA graph with a device-side WHILE node; one
// pass of its body is four launches with fixed grids:
//   k_sparse_levels  (cooperative, persistent) every consecutive push level:
//            frontier queue -> neighbours (warp load-balanced search over the
//            degrees of 32 queue entries; vertices above PUSH_HEAVY cut into
//            chunks that teams of warps share), claims / relaxes destinations with the
//            operator hooks, appends the next queue with warp-aggregated
//            atomics and sets the next-frontier bitmap; one grid barrier
//            per level, after which every block takes the end-of-level
//            decision itself from the level's counters;
//   k_pull   (when the frontier is dense) every candidate row scans its
//            in-edges against the frontier bitmap (first-parent operators
//            stop at the first parent; the others fold every frontier
//            offer), light rows in degree bins (warp / thread per row),
//            heavy rows in 2048-edge chunks;
//   k_compact (after a pull) next queue from the next-frontier bitmap;
//   k_decide 1 warp: next size, direction switch (frontier edges against
//            unvisited edges, Beamer), iteration cap, loop condition.
// The push phase returns as soon as the switch picks pull; k_pull /
// k_compact / k_decide then run one dense level and the body repeats.
// Frontier bitmaps are triple-buffered: the active kernel clears the buffer
// the next iteration will write.
#pragma once

#include "mg_device.cuh"
#include "mg_ops.cuh"

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <type_traits>

namespace {

constexpr int MODE_PUSH = 0, MODE_PULL = 1;
// Frontier vertices above PUSH_HEAVY out-edges are listed as chunks of
// PUSH_CHUNK edges (at most PUSH_CHUNKS a vertex), which a push level spreads
// over teams of warps; the rest go one or more to a warp.  A 32-edge step is
// a chain of dependent L2 accesses of 2-3 us, so what counts is the longest
// run of steps in one warp: with one warp for any vertex of up to 4096
// edges, the first level of a traversal from a hub took 317 us on R-MAT 20
// (a 3,400-edge source: 100+ steps); with the chunks it is one step.
constexpr int32_t PUSH_HEAVY = 128;
constexpr int32_t PUSH_CHUNK = 512;
constexpr int32_t PUSH_CHUNKS = 1024;
constexpr int THREADS = 256;
// persistent kernels: blocks of 1024 threads, and for the push phase one
// block per SM: 152 arrivals at the grid barrier instead of 304, and 64
// registers a thread instead of 32 with spills in the edge loops (lattice
// BFS 5.8 -> 4.8 us a level at 100 K vertices, 8.5 -> 7.9 at 16.8 M; R-MAT
// pushes 5-15 % faster).  Graphs without heavy vertices whose rows average
// more than DENSE_ROWS edges (random graphs) push few and large levels, where
// twice the warps in flight are worth more: two blocks per SM (push levels of
// a BFS, one block / two: 1 M vertices of degree 64 630 / 456 us, 4 M of degree
// 16 1384 / 1143; of degree 8 and less one block is as fast or faster).
constexpr int PTHREADS = 1024;
constexpr int64_t DENSE_ROWS = 8;
// grid barrier words (2 + GRID_SYNC_GROUPS), the barrier error flag, the BC
// path-count overflow flag, rounded up
constexpr size_t BAR_BYTES = 4 * (2 + mgd::GRID_SYNC_GROUPS + 1 + 7);
constexpr int OVF_WORD = 2 + mgd::GRID_SYNC_GROUPS + 1;
constexpr int FMIN_WORD = OVF_WORD + 1;  // SSSP: least distance on the current frontier (pull levels)

struct FCtl {
    int32_t more;       // continue flag (host loop readback)
    int32_t iter;       // level / round being expanded
    int32_t mode;       // MODE_PUSH / MODE_PULL
    int32_t cur;        // current bitmap buffer 0..2
    int32_t qoff, qsize;  // current queue slice
    int32_t nqoff, nq;    // next queue slice (nq: atomic counter)
    int32_t hcur, nhcur;  // heavy chunk list sizes: current / next (atomic)
    int32_t hpar;         // heavy list parity
    int32_t status;       // 0 ok, 1 iteration cap
    int32_t pull_iters;
    int32_t max_iter;
    int32_t dirmode;      // MG_DIR_*
    int32_t alpha, beta;
    int32_t nlevels;      // BC: levels archived
    int32_t archive;      // 1: queue slices are appended (BFS/BC), 0: ping-pong (SSSP)
    int32_t qedges;         // out-edges of the current frontier
    long long nf_edges;      // out-edges of the next frontier (atomic)
    long long visited_edges; // out-edges of every vertex visited so far
    long long scanned;       // edges scanned (statistics, atomic)
};

struct Args {
    int32_t n;
    int32_t m;
    const int32_t *row, *col, *wt;     // push side
    const int32_t *trow, *tcol, *twt;  // pull side
    const int32_t *wrows, *trows;  // degree bins of the pull rows
    int32_t nwrows, ntrows, nwlong;
    const int32_t *hchunk;
    int32_t nhchunks;
    int32_t heavy_deg;
    int32_t *label;
    mgops::PathCount *sigma;
    int32_t bc_ext;      // BC path counts in extended mode (mgops::PathCount)
    int32_t *bc_ovf;     // set when a plain-mode path count reaches mgops::PC_PLAIN_MAX
    int32_t *fmin;       // SSSP pull levels: least distance on the frontier (k_fmin)
    int32_t wmin;        // least edge weight
    uint32_t *bm;        // 3 * words
    uint32_t *visited;
    int32_t words;
    int32_t *queue;
    int4 *heavy;         // 2 * hcap chunks (parity): vertex, first edge, end
    int32_t hcap;
    int32_t has_heavy;   // some vertex may have more than PUSH_HEAVY out-edges
    int32_t short_pull;  // the graph's in-rows are short (mg_graph)
    int32_t *lvl_off;
    FCtl *ctl;
    unsigned *bar;       // grid barrier words of the persistent kernels
    int *bar_err;        // set when a grid barrier wait times out
    int bar_never;       // failure injection: barriers never complete (MG_FAIL_BARRIER)
    struct LevelCnt *cnt;  // persistent push phase: per-level counters, 4 rotating slots
};

// Counters one push level produces (next queue size, heavy chunks, next
// frontier's out-edges).  The persistent push phase keeps them in 4 slots
// by level mod 4, so every block can read level L's counters after the one
// barrier while level L+1 appends to the next slot; block 0 clears slot
// L+2 during level L (its last readers finished before the barrier that
// began level L).
struct LevelCnt {
    int32_t nq;
    int32_t nhcur;
    long long nfe;
    int32_t fmin;        // least label on the frontier that enters the level (k_frontier_all, min-plus pulls)
    int32_t pad[3];
};

__device__ __forceinline__ uint32_t *bm_buf(const Args &a, int idx) { return a.bm + (size_t)idx * a.words; }

// The loop state as the persistent kernel re-reads it after every grid
// barrier: through L2, never from a stale L1 line.
static_assert(sizeof(FCtl) % 8 == 0, "FCtl is copied as 8-byte words");
__device__ __forceinline__ FCtl load_ctl(const FCtl *p)
{
    FCtl c;
    const int2 *s = reinterpret_cast<const int2 *>(p);
    int2 *d = reinterpret_cast<int2 *>(&c);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(FCtl) / 8); i++) d[i] = __ldcg(s + i);
    return c;
}

// warp-wide: add v (64-bit) from every lane to *dst with one atomic
__device__ __forceinline__ void warp_add64(long long *dst, long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (mgd::lane() == 0 && v) atomicAdd((unsigned long long *)dst, (unsigned long long)v);
}

// Edges per chunk of a heavy vertex: PUSH_CHUNK, or more (a multiple of 32)
// where that would make more than PUSH_CHUNKS chunks.
__device__ __forceinline__ int32_t push_chunk(int32_t deg)
{
    return max(PUSH_CHUNK, (((deg - 1) / PUSH_CHUNKS + 1) + 31) & ~31);
}

// chunks that the heavy list can hold at most: a vertex above PUSH_HEAVY
// edges has at most deg / PUSH_CHUNK + 1 of them
inline int32_t heavy_cap(int64_t m) { return (int32_t)(m / PUSH_CHUNK + m / (PUSH_HEAVY + 1) + 2); }

// The chunks of the lanes' heavy vertices (deg <= PUSH_HEAVY: none) to the
// list `out`: one atomic a warp, the chunks spread over the lanes; all lanes
// of the warp call.
__device__ __forceinline__ void list_heavy(int4 *out, int32_t *count, int32_t v, int32_t begin, int32_t deg)
{
    const int lane = mgd::lane();
    const int32_t ch = push_chunk(deg), nc = deg > PUSH_HEAVY ? (deg - 1) / ch + 1 : 0;
    const int incl = mgd::warp_scan_incl(nc);
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    int32_t base = 0;
    if (lane == 0) base = atomicAdd(count, total);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (int k0 = 0; k0 < total; k0 += 32) {
        const int k = min(k0 + lane, total - 1);
        const int own = mgd::owner_lane(incl - nc, k);
        const int i = k - __shfl_sync(0xffffffffu, incl - nc, own);
        const int32_t u = __shfl_sync(0xffffffffu, v, own), b = __shfl_sync(0xffffffffu, begin, own),
                      d = __shfl_sync(0xffffffffu, deg, own), c = __shfl_sync(0xffffffffu, ch, own);
        if (k0 + lane < total) out[base + k] = make_int4(u, b + i * c, b + min(d, (i + 1) * c), 0);
    }
}

// record a newly reached vertex in the next frontier (push sweeps; all lanes
// call).  A relaxed operator has already set the vertex's bit when it
// improved it.
template <class Op, bool HEAVY>
__device__ __forceinline__ void emit_next(const Args &a, const FCtl &c, int nextbuf, bool found, int32_t v,
                                          long long &dsum, int32_t *nq, int32_t *nhcur)
{
    int slot = mgd::warp_append(nq, found);
    int32_t b = 0, dg = 0;
    if (found) {
        a.queue[c.nqoff + slot] = v;
        if (Op::kLevelSync) mgd::bm_set(bm_buf(a, nextbuf), v);
        b = a.row[v];
        dg = a.row[v + 1] - b;
        dsum += dg;
    }
    if (HEAVY && __any_sync(0xffffffffu, dg > PUSH_HEAVY))
        list_heavy(a.heavy + (size_t)(c.hpar ^ 1) * a.hcap, nhcur, v, b, dg);
}

// ----------------------------------------------------------------------------
// push: one edge (u -> v) with the source's payload
// ----------------------------------------------------------------------------
template <class Op>
__device__ __forceinline__ bool push_edge(const Args &a, int it1, int32_t v, int32_t payload_i,
                                          mgops::PathCount payload_d, int32_t w, uint32_t *next_bm)
{
    if constexpr (Op::kPathCounts) {
        // claim at this level, or collect the path count on it
        bool on_level;
        bool claimed = Op::fused_update_condition(&a.label[v], it1, on_level);
        if (on_level) Op::accumulate(&a.sigma[v], payload_d, a.bc_ext != 0, a.bc_ovf);
        if (claimed) mgd::bm_set(a.visited, v);
        return claimed;
    } else if constexpr (Op::kLevelSync) {
        // the visited bitmap claims the vertex once; its label is the level
        if (mgd::bm_test(a.visited, v)) return false;
        if (!mgd::bm_set(a.visited, v)) return false;
        a.label[v] = Op::get_partial_result(it1 - 1, w);
        return true;
    } else {
        // relaxation: the offer folded in with one atomic; an improved
        // vertex enters the next frontier once (its bit)
        const int32_t nd = Op::get_partial_result(payload_i, w);
        if (!Op::update_condition(a.label[v], nd, it1)) return false;
        if (!Op::fused_update_condition(&a.label[v], nd, it1)) return false;
        return mgd::bm_set(next_bm, v);
    }
}

// One push level.  Queue entries, heavy entries and the frontier's labels /
// path counts were written by other blocks in the previous level, so they
// are loaded through L2 (__ldcg): the persistent kernel runs many levels in
// one launch.
template <class Op, bool HEAVY>
__device__ __forceinline__ void push_level(const Args &a, const FCtl &c, LevelCnt *lc)
{
    const int it1 = c.iter + 1;
    const int nextbuf = (c.cur + 1) % 3, sparebuf = (c.cur + 2) % 3;
    // clear the buffer the next iteration writes
    {
        uint32_t *sp = bm_buf(a, sparebuf);
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.words; i += gridDim.x * blockDim.x) sp[i] = 0;
    }
    const int lane = mgd::lane();
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    long long scanned = 0, dsum = 0;
    // chunks of heavy frontier vertices: a warp each, or a team of warps when
    // there are fewer chunks than warps
    if (HEAVY && c.hcur > 0) {
        const int tw = c.hcur >= nwarps ? 1 : nwarps / c.hcur;
        const int4 *list = a.heavy + (size_t)c.hpar * a.hcap;
        for (int h = gwarp / tw; h < c.hcur; h += nwarps / tw) {
            const int4 it = __ldcg(&list[h]);
            const int32_t u = it.x, e = it.z;
            const int32_t pi = __ldcg(&a.label[u]);
            const mgops::PathCount pd = Op::kPathCounts ? mgops::pc_load_cg(&a.sigma[u]) : mgops::pc_zero();
            if (Op::kPathCounts && !a.bc_ext && pd.m >= mgops::PC_PLAIN_MAX) *a.bc_ovf = 1;
            for (int32_t k0 = it.y + (gwarp % tw) * 32; k0 < e; k0 += tw * 32) {
                const int32_t k = k0 + lane;
                bool found = false;
                int32_t v = 0;
                if (k < e) {
                    v = a.col[k];
                    found = push_edge<Op>(a, it1, v, pi, pd, Op::kWeighted ? a.wt[k] : 0, bm_buf(a, nextbuf));
                }
                emit_next<Op, HEAVY>(a, c, nextbuf, found, v, dsum, &lc->nq, &lc->nhcur);
            }
            if (lane == 0 && gwarp % tw == 0) scanned += e - it.y;
        }
    }
    // light frontier vertices: vpw per warp (32, or fewer when the frontier
    // would leave warps idle), load-balanced over their edges
    int vpw = 32;
    if (c.qsize < nwarps * 32) {
        const int want = max(1, c.qsize / nwarps);
        vpw = 1;
        while (vpw * 2 <= want) vpw *= 2;
    }
    for (int base = gwarp * vpw; base < c.qsize; base += nwarps * vpw) {
        int32_t u = -1, start = 0, deg = 0, pi = 0;
        mgops::PathCount pd = mgops::pc_zero();
        if (lane < vpw && base + lane < c.qsize) {
            u = __ldcg(&a.queue[c.qoff + base + lane]);
            start = a.row[u];
            deg = a.row[u + 1] - start;
            if (HEAVY && deg > PUSH_HEAVY) deg = 0;
            pi = __ldcg(&a.label[u]);
            if (Op::kPathCounts) {
                pd = mgops::pc_load_cg(&a.sigma[u]);
                if (!a.bc_ext && pd.m >= mgops::PC_PLAIN_MAX) *a.bc_ovf = 1;
            }
        }
        int incl = mgd::warp_scan_incl(deg);
        int excl = incl - deg;
        int total = __shfl_sync(0xffffffffu, incl, 31);
        scanned += (lane == 0) ? total : 0;
        for (int k0 = 0; k0 < total; k0 += 32) {
            int k = k0 + lane;
            int kk = k < total ? k : total - 1;
            int own = mgd::owner_lane(excl, kk);
            int32_t e = __shfl_sync(0xffffffffu, start, own) + (kk - __shfl_sync(0xffffffffu, excl, own));
            int32_t opi = __shfl_sync(0xffffffffu, pi, own);
            const mgops::PathCount opd = Op::kPathCounts ? mgops::shfl_val(pd, own) : pd;
            bool found = false;
            int32_t v = 0;
            if (k < total) {
                v = a.col[e];
                found = push_edge<Op>(a, it1, v, opi, opd, Op::kWeighted ? a.wt[e] : 0, bm_buf(a, nextbuf));
            }
            emit_next<Op, HEAVY>(a, c, nextbuf, found, v, dsum, &lc->nq, &lc->nhcur);
        }
    }
    warp_add64(&lc->nfe, dsum);
    if (lane == 0 && scanned) atomicAdd((unsigned long long *)&a.ctl->scanned, (unsigned long long)scanned);
}

// The end-of-level decision on a copy of the loop state, given the level's
// counters; block 0 (write_lvl) also records the level offset.
__device__ __forceinline__ int decide_local(const Args &a, FCtl &c, int32_t nq, int32_t nhcur, long long nfe_in,
                                            bool write_lvl)
{
    int more = c.more;
    if (more) {
        if (c.mode == MODE_PULL) c.pull_iters++;
        c.iter += 1;
        if (c.archive && c.iter + 1 < a.n + 3) {
            if (write_lvl) a.lvl_off[c.iter + 1] = c.nqoff + nq;
            if (nq > 0) c.nlevels = c.iter + 1;
        }
        c.qoff = c.nqoff;
        c.qsize = nq;
        c.nqoff = c.archive ? (c.qoff + nq) : (c.qoff == 0 ? a.n : 0);
        c.nq = 0;
        c.hcur = nhcur;
        c.nhcur = 0;
        c.hpar ^= 1;
        c.cur = (c.cur + 1) % 3;
        const long long nfe = nfe_in;
        c.visited_edges += nfe;
        c.qedges = (int32_t)min(nfe, (long long)INT32_MAX);
        c.nf_edges = 0;
        if (nq == 0) {
            more = 0;
        } else {
            if (c.dirmode == MG_DIR_PUSH) c.mode = MODE_PUSH;
            else if (c.dirmode == MG_DIR_PULL) c.mode = MODE_PULL;
            else if (c.archive) {
                // Beamer: push -> pull when frontier edges exceed unvisited
                // edges / alpha; pull -> push when the frontier is below n / beta
                const long long unvisited = (long long)a.m - c.visited_edges;
                if (c.mode == MODE_PUSH) {
                    if (nfe * (long long)c.alpha > unvisited && nq > 64) c.mode = MODE_PULL;
                } else {
                    if ((long long)nq * c.beta < a.n) c.mode = MODE_PUSH;
                }
            } else {
                // SSSP: pull when the frontier's edges are a large share of m
                c.mode = (nfe * (long long)c.alpha > (long long)a.m) ? MODE_PULL : MODE_PUSH;
            }
            if (c.iter >= c.max_iter) { c.status = 1; more = 0; }
        }
        c.more = more;
    }
    return more;
}

// ----------------------------------------------------------------------------
// push, one block: consecutive levels of a small frontier on a graph without
// heavy vertices (a lattice, a road network: hundreds or thousands of levels
// of a few hundred vertices).  A level of the whole grid is a barrier and a
// chain of L2 round trips (atomics, loads that must see other blocks' writes)
// whatever its size: 4.8 us for BFS and 9 us for BC on a 320 x 311 lattice.
// One block needs neither: the frontier lies in shared memory with its row
// offsets, a level's candidates are told apart in a shared hash table, path
// counts are pulled by the new vertices instead of added atomically, and
// labels and counts are read back through the block's own L1.  us per level,
// grid -> block: BFS 4.8 -> 2.9 and BC 9.1 -> 5.6 at 230 vertices a level;
// at 660 a level one SM's load rate makes it 7.5 and 14.5 against the grid's
// 4.7 and 7.0, so the block takes over below CTA_ENTER and hands back above
// CTA_Q.
// ----------------------------------------------------------------------------
constexpr int CTA_Q = 512;           // frontier entries held in shared memory
constexpr int CTA_ENTER = 384;       // the block takes over at this many vertices
constexpr int CTA_EDGES = 4096;      // and while the frontier has at most this many edges
constexpr int CTA_HASH = 2 * CTA_EDGES;
constexpr int CTA_LEVELS = 20000;    // levels before the grid meets again (a fraction of the barrier's time limit)

struct CtaShared {
    int32_t v[2][CTA_Q], b[2][CTA_Q];     // frontier: vertex, first edge
    int32_t d[2][CTA_Q];                  // out-degree
    int32_t slot[CTA_Q];                  // the new entries' hash slots
    int32_t hash[CTA_HASH];
    int32_t count;
    int32_t nfe;                          // (at most CTA_EDGES vertices of fewer than 128 edges)
};

// The block tells new vertices by their label and writes the level as the
// label: the built-in operators' labels, whose start value is UNSET.  Another
// level-synchronous operator may start its labels at any value (even at the
// source's) and label by its own offer; the grid's levels claim by the visited
// bitmap and run it.
template <class Op>
constexpr bool kBlockLevels = std::is_same<Op, mgops::Bfs>::value || std::is_same<Op, mgops::BcForward>::value;

// Runs levels from the loop state c (shared memory, all threads of block 0
// call) until the frontier outgrows the block, the traversal ends or the
// direction switch picks pull; the queue archive, labels, visited bits and
// level offsets are kept in global memory as the grid's levels keep them, the
// frontier bitmaps (all zero on entry) hold the last frontier on return.
template <class Op>
__device__ __noinline__ void cta_push_levels(const Args &a, FCtl &c, CtaShared &s)
{
    static_assert(kBlockLevels<Op>, "labels are levels, UNSET before");
    const int t = threadIdx.x;
    for (int i = t; i < CTA_HASH; i += PTHREADS) s.hash[i] = -1;
    for (int i = t; i < c.qsize; i += PTHREADS) {
        const int32_t u = __ldcg(&a.queue[c.qoff + i]), b = a.row[u];
        s.v[0][i] = u;
        s.b[0][i] = b;
        s.d[0][i] = a.row[u + 1] - b;
    }
    if (t == 0) {
        s.count = 0;
        s.nfe = 0;
    }
    __syncthreads();
    int p = 0;
    for (int lv = 0; lv < CTA_LEVELS; lv++) {
        const int32_t it1 = c.iter + 1, n0 = c.qsize, out = c.nqoff;
        // threads per vertex: 8, or fewer when the frontier fills the block
        const int tpv = n0 <= 128 ? 8 : n0 <= 256 ? 4 : n0 <= 512 ? 2 : 1;
        int32_t nfe = 0;
        for (int i0 = (t & ~31) / tpv; i0 < n0; i0 += PTHREADS / tpv) {
            const int i = i0 + (t & 31) / tpv;
            const int32_t b = i < n0 ? s.b[p][i] : 0, d = i < n0 ? s.d[p][i] : 0;
            const int32_t steps = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)((d + tpv - 1) / tpv));
            // two edges a step, their loads together
            for (int32_t k0 = 0; k0 < steps; k0 += 2) {
                int32_t w[2], h[2], wb[2], wd[2];
                bool fresh[2];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const int32_t k = (k0 + j) * tpv + t % tpv;
                    w[j] = k < d ? __ldg(&a.col[b + k]) : -1;
                }
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    fresh[j] = w[j] >= 0 && a.label[w[j]] == mgops::UNSET;
                    wb[j] = fresh[j] ? __ldg(&a.row[w[j]]) : 0;
                    wd[j] = fresh[j] ? __ldg(&a.row[w[j] + 1]) - wb[j] : 0;
                }
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    if (fresh[j]) {
                        h[j] = (int)(((uint32_t)w[j] * 2654435761u) >> 19) & (CTA_HASH - 1);
                        int32_t old;
                        while ((old = atomicCAS(&s.hash[h[j]], -1, w[j])) != -1 && old != w[j])
                            h[j] = (h[j] + 1) & (CTA_HASH - 1);
                        fresh[j] = old == -1;   // else another edge of this level has it
                    }
                    __syncwarp();
                    const unsigned m = __ballot_sync(0xffffffffu, fresh[j]);
                    if (m == 0) continue;
                    int at = 0;
                    if (mgd::lane() == 0) at = atomicAdd(&s.count, __popc(m));
                    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << mgd::lane()) - 1u));
                    if (!fresh[j]) continue;
                    a.queue[out + at] = w[j];
                    atomicOr(&a.visited[w[j] >> 5], 1u << (w[j] & 31));
                    nfe += wd[j];
                    if (at < CTA_Q) {
                        s.v[p ^ 1][at] = w[j];
                        s.b[p ^ 1][at] = wb[j];
                        s.d[p ^ 1][at] = wd[j];
                        s.slot[at] = h[j];
                    }                         // (else too many for the block: this is its last level)
                }
            }
        }
        __syncwarp();
        nfe = (int32_t)__reduce_add_sync(0xffffffffu, (unsigned)nfe);
        if (mgd::lane() == 0 && nfe) atomicAdd(&s.nfe, nfe);
        __syncthreads();
        const int32_t nq = s.count;
        // path counts and labels of the new vertices: sums over the
        // neighbours at this level.  (Labels are set after the candidates of
        // the level are known, so the test above sees no label of its own.)
        for (int i = t; i < nq; i += PTHREADS) {
            const bool held = i < CTA_Q;
            const int32_t w = held ? s.v[p ^ 1][i] : a.queue[out + i];
            if constexpr (Op::kPathCounts) {
                const bool own = held && a.trow == a.row;
                const int32_t b = own ? s.b[p ^ 1][i] : __ldg(&a.trow[w]);
                const int32_t d = own ? s.d[p ^ 1][i] : __ldg(&a.trow[w + 1]) - b;
                mgops::PathCount sum = mgops::pc_zero();
                for (int32_t k = b; k < b + d; k += 4) {
                    int32_t u[4], lu[4];
                    mgops::PathCount x[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) u[j] = k + j < b + d ? __ldg(&a.tcol[k + j]) : w;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        lu[j] = a.label[u[j]];
                        x[j] = a.sigma[u[j]];
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (u[j] != w && lu[j] == it1 - 1) sum = mgops::pc_add(sum, x[j], a.bc_ext != 0);
                }
                a.sigma[w] = sum;
                if (!a.bc_ext && sum.m >= mgops::PC_PLAIN_MAX) *a.bc_ovf = 1;
            }
            if (held) s.hash[s.slot[i]] = -1;
        }
        // every warp has read s.count (thread 0 sets it back below) and, with
        // path counts, every label test of the sums above is done
        __syncthreads();
        for (int i = t; i < nq; i += PTHREADS) a.label[i < CTA_Q ? s.v[p ^ 1][i] : a.queue[out + i]] = it1;
        if (t == 0) {
            FCtl n = c;
            atomicAdd((unsigned long long *)&a.ctl->scanned, (unsigned long long)n.qedges);
            decide_local(a, n, nq, 0, (long long)s.nfe, true);
            c = n;
            s.count = 0;
            s.nfe = 0;
        }
        p ^= 1;
        __syncthreads();
        if (c.more == 0 || c.mode != MODE_PUSH || c.qsize > CTA_Q || c.qedges > CTA_EDGES) break;
    }
    uint32_t *bm = bm_buf(a, c.cur);
    if (c.more)
        for (int i = t; i < c.qsize; i += PTHREADS) {
            const int32_t u = a.queue[c.qoff + i];
            atomicOr(&bm[u >> 5], 1u << (u & 31));
        }
    __syncthreads();
}

// ----------------------------------------------------------------------------
// pull: row reductions over in-edges against the frontier bitmap
// ----------------------------------------------------------------------------
// A pull sweep only marks the rows it reaches in the next-frontier bitmap
// (atomicOr on distinct words, no shared counter); k_compact then builds the
// queue, the frontier's edge count and its heavy list from the bitmap.
struct PullEmit {
    const Args &a;
    uint32_t *next_bm;
    __device__ void flush() {}
};

// Relaxed operators: fold the offers of frontier in-neighbours in row order
// (accumulate_nonAtomics), then one fused update + next-frontier bit on the
// row.  With a dense frontier (all_in) every in-neighbour's offer is folded
// without the bitmap test: operators are monotone (mg_ops.cuh), so offers of
// unreached or earlier-relaxed vertices never spoil a label, labels still
// converge to the same fixed point, and one dependent load per edge goes away.
//
// Min-plus operators take every reached in-neighbour's offer at any frontier
// that the direction switch pulls for (it holds a quarter of the edges by
// default): the bitmap test puts a dependent load in front of every label
// (device time of SSSP with the test where the frontier has few vertices ->
// without: R-MAT 22 1.69 -> 1.48 ms, R-MAT 20 0.51 -> 0.48, R-MAT 18 0.32 ->
// 0.30).  Where the caller has every level pulled, most frontiers are small and
// most edges end at the bitmap, which stays in L1: k_pull has a form with the
// test for that (ALL false; SSSP of 1 M vertices of degree 64 so pulled, with
// the test / without, 3.5 / 4.1 ms; a test on the level's size inside the one
// form cost the switched runs 4 %).  An unreached neighbour is told by its
// initial label, to which no weight is added, so that no sum of the two can
// wrap.
//
// Min-plus operators (kMinPlusBound) skip rows whose label is at most (least
// frontier label + least weight): every offer is label[u] + w from a
// frontier vertex u, or from a vertex whose edges an earlier level already
// relaxed, so such a row cannot improve this level.  On R-MAT the hubs
// settle first, so the later pull levels read a fraction of the edges.
template <class Op, bool ALL>
__device__ __forceinline__ bool pull_offer(const Args &a, const uint32_t *fb, bool all_in, int32_t u, int32_t w,
                                           int32_t &offer)
{
    if constexpr (Op::kMinPlusBound) {
        if (!ALL && !all_in && !mgd::bm_test(fb, u)) return false;
        const int32_t label = a.label[u];
        if (label == Op::initialize()) return false;
        offer = Op::get_partial_result(label, w);
    } else {
        if (!all_in && !mgd::bm_test(fb, u)) return false;
        offer = Op::get_partial_result(a.label[u], w);
    }
    return true;
}

// whether a relaxed level with the test folds every in-neighbour's offer
template <class Op>
__device__ __forceinline__ bool pull_all_in(const Args &a, const FCtl &c)
{
    return (long long)c.qsize * 8 > a.n || (Op::kMinPlusBound && (long long)c.qedges * 4 > a.m);
}

template <class Op, bool ALL>
struct PullRelax : PullEmit {
    using T = int32_t;
    static constexpr bool kRowAware = Op::kMinPlusBound;
    static constexpr bool kWeights = Op::kWeighted;
    const uint32_t *fb;
    int it1;
    bool all_in;
    int32_t bound;
    __device__ T identity() const { return Op::initialize(); }
    __device__ bool skip(int32_t v) const { return a.label[v] <= bound; }
    __device__ T edge(int32_t, int32_t, int32_t u, int32_t w) const
    {
        int32_t offer;
        return pull_offer<Op, ALL>(a, fb, all_in, u, w, offer) ? offer : Op::initialize();
    }
    __device__ T combine(T x, T y) const
    {
        Op::accumulate_nonAtomics(x, y, it1);
        return x;
    }
    __device__ void finish(int32_t v, T best)
    {
        if (Op::update_condition(a.label[v], best, it1) && Op::fused_update_condition(&a.label[v], best, it1))
            mgd::bm_set(next_bm, v);
    }
};

// Path-count operators (BC forward): unvisited rows sum the path counts of
// frontier in-neighbours
template <class Op>
struct PullCounts : PullEmit {
    using T = mgops::PathCount;
    static constexpr bool kRowAware = true;  // visited rows are skipped
    static constexpr bool kWeights = false;
    const uint32_t *fb;
    int it1;
    bool all_in;
    int32_t bound;
    __device__ T identity() const { return mgops::pc_zero(); }
    __device__ bool skip(int32_t v) const { return mgd::bm_test(a.visited, v); }
    __device__ T edge(int32_t, int32_t, int32_t u, int32_t) const
    {
        return mgd::bm_test(fb, u) ? a.sigma[u] : mgops::pc_zero();
    }
    __device__ T combine(T x, T y) const
    {
        Op::accumulate_nonAtomics(x, y, a.bc_ext != 0);
        return x;
    }
    __device__ void finish(int32_t v, T s)
    {
        if (s.m > 0.0) {
            a.label[v] = it1;
            a.sigma[v] = s;
            if (!a.bc_ext && s.m >= mgops::PC_PLAIN_MAX) *a.bc_ovf = 1;
            mgd::bm_set(a.visited, v);
            mgd::bm_set(next_bm, v);
        }
    }
};

template <class Op, bool ALL>
using PullOp = std::conditional_t<Op::kPathCounts, PullCounts<Op>, PullRelax<Op, ALL>>;

// min-plus pull levels: rows at or below this label cannot improve
__device__ __forceinline__ int32_t sssp_bound(int32_t fmin, int32_t wmin)
{
    return fmin >= INT32_MAX - wmin ? INT32_MAX : fmin + wmin;
}

// least label over the frontier queue (before a min-plus pull level)
__device__ __forceinline__ void frontier_min(const Args &a, const FCtl &c, int32_t *out)
{
    int32_t mn = INT32_MAX;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.qsize; i += gridDim.x * blockDim.x)
        mn = min(mn, a.label[a.queue[c.qoff + i]]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    if (mgd::lane() == 0 && mn < INT32_MAX) atomicMin(out, mn);
}

__global__ void __launch_bounds__(THREADS) k_fmin(Args a)
{
    const FCtl c = *a.ctl;
    if (c.mode != MODE_PULL || c.more == 0) return;
    frontier_min(a, c, a.fmin);
}

// One pull level by blocks of NT threads; bound: min-plus rows at or below
// this label cannot improve; ALL: min-plus without the bitmap test.
template <class Op, bool ALL, int NT>
__device__ __forceinline__ void pull_level(const Args &a, const FCtl &c, int32_t bound)
{
    const int it1 = c.iter + 1;
    const int nextbuf = (c.cur + 1) % 3, sparebuf = (c.cur + 2) % 3;
    const uint32_t *fb = bm_buf(a, c.cur);
    {
        uint32_t *sp = bm_buf(a, sparebuf);
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.words; i += gridDim.x * blockDim.x) sp[i] = 0;
    }
    const int lane = mgd::lane();
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    long long scanned = 0;

    if constexpr (Op::kFirstParent) {
        // bottom-up: a thread per unvisited light row, first frontier parent wins
        const int32_t stride = gridDim.x * blockDim.x;
        const int32_t nround = (a.n + stride - 1) / stride;
        for (int32_t r = 0; r < nround; r++) {
            int32_t v = r * stride + blockIdx.x * blockDim.x + threadIdx.x;
            bool found = false;
            if (v < a.n && !mgd::bm_test(a.visited, v)) {
                int32_t b = a.trow[v], e = a.trow[v + 1];
                if (e - b <= a.heavy_deg) {
                    for (int32_t p = b; p < e; p++) {
                        scanned++;
                        if (mgd::bm_test(fb, a.tcol[p])) { found = true; break; }
                    }
                    if (found) {
                        a.label[v] = it1;
                        mgd::bm_set(a.visited, v);
                        mgd::bm_set(bm_buf(a, nextbuf), v);
                    }
                }
            }
        }
    } else {
        // degree-binned rows; reached rows marked in the next-frontier bitmap
        PullOp<Op, ALL> op{{a, bm_buf(a, nextbuf)}, fb, it1, false, 0};
        if constexpr (!Op::kLevelSync && !ALL) op.all_in = pull_all_in<Op>(a, c);
        if constexpr (Op::kMinPlusBound) op.bound = bound;
        mgd::bins_reduce(op, a.trow, a.tcol, a.twt, a.wrows, a.nwrows, a.nwlong, a.trows, a.ntrows);
        (void)gwarp;
        (void)nwarps;
    }

    // heavy rows: one CTA per 2048-edge chunk
    __shared__ int32_t s_min[NT / 32];
    __shared__ mgops::PathCount s_sum[NT / 32];
    __shared__ int s_hit, s_skip;
    for (int32_t ch = blockIdx.x; ch < a.nhchunks; ch += gridDim.x) {
        int32_t v = a.hchunk[3 * ch], b = a.hchunk[3 * ch + 1], e = a.hchunk[3 * ch + 2];
        // thread 0 decides for the block (the row may be claimed concurrently
        // by another chunk, so a per-thread test could diverge).  BFS / BC
        // skip only rows reached at an earlier level; the label is read from
        // L2: hub-first ids put the heavy rows' labels in a few lines, and an
        // L1 copy from an earlier chunk can predate this level's claim, which
        // would drop this chunk's share of the row's path count
        if (threadIdx.x == 0) {
            if constexpr (!Op::kLevelSync) {
                s_skip = Op::kMinPlusBound && a.label[v] <= bound;
            } else {
                const int32_t lv = __ldcg(&a.label[v]);
                s_skip = lv != Op::initialize() && lv != it1;
            }
        }
        __syncthreads();
        const bool skip = s_skip;
        __syncthreads();
        if (skip) continue;
        int32_t best = Op::initialize();
        mgops::PathCount ssum = mgops::pc_zero();
        const bool ext = a.bc_ext != 0;
        int hit = 0;
        const bool all_in = !Op::kLevelSync && !ALL && pull_all_in<Op>(a, c);  // as PullRelax
        for (int32_t p = b + threadIdx.x; p < e; p += blockDim.x) {
            int32_t u = __ldcs(&a.tcol[p]);  // streamed once: evict-first
            if constexpr (!Op::kLevelSync) {
                int32_t offer;
                if (pull_offer<Op, ALL>(a, fb, all_in, u, Op::kWeighted ? __ldcs(&a.twt[p]) : 0, offer)) {
                    hit = 1;
                    Op::accumulate_nonAtomics(best, offer, it1);
                }
            } else if (mgd::bm_test(fb, u)) {
                hit = 1;
                if constexpr (Op::kPathCounts) ssum = mgops::pc_add(ssum, a.sigma[u], ext);
            }
        }
        if (threadIdx.x == 0) s_hit = 0;
        __syncthreads();
        if (hit) s_hit = 1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            if constexpr (!Op::kLevelSync) Op::accumulate_nonAtomics(best, __shfl_xor_sync(0xffffffffu, best, o), it1);
            if constexpr (Op::kPathCounts) ssum = mgops::pc_add(ssum, mgops::shfl_xor_val(ssum, o), ext);
        }
        if (lane == 0) { s_min[threadIdx.x >> 5] = best; s_sum[threadIdx.x >> 5] = ssum; }
        __syncthreads();
        if (threadIdx.x == 0) {
            int32_t bm = Op::initialize();
            mgops::PathCount bs = mgops::pc_zero();
            for (int w = 0; w < NT / 32; w++) {
                if constexpr (!Op::kLevelSync) Op::accumulate_nonAtomics(bm, s_min[w], it1);
                if constexpr (Op::kPathCounts) bs = mgops::pc_add(bs, s_sum[w], ext);
            }
            uint32_t *nb = bm_buf(a, nextbuf);
            if (s_hit) {
                if constexpr (Op::kFirstParent) {
                    if (atomicCAS(&a.label[v], Op::initialize(), it1) == Op::initialize()) {
                        mgd::bm_set(a.visited, v);
                        mgd::bm_set(nb, v);
                    }
                } else if constexpr (!Op::kLevelSync) {
                    if (Op::update_condition(a.label[v], bm, it1) && Op::fused_update_condition(&a.label[v], bm, it1))
                        mgd::bm_set(nb, v);
                } else {
                    bool on_level;
                    bool found = Op::fused_update_condition(&a.label[v], it1, on_level);
                    if (on_level) Op::accumulate(&a.sigma[v], bs, ext, a.bc_ovf);
                    if (found) {
                        mgd::bm_set(a.visited, v);
                        mgd::bm_set(nb, v);
                    }
                }
            }
            scanned += e - b;
        }
        __syncthreads();
    }
    warp_add64(&a.ctl->scanned, scanned);
}

template <class Op, bool ALL>
__global__ void __launch_bounds__(THREADS) k_pull(Args a)
{
    const FCtl c = *a.ctl;
    if (c.mode != MODE_PULL || c.more == 0) return;
    pull_level<Op, ALL, THREADS>(a, c, Op::kMinPlusBound ? sssp_bound(*a.fmin, a.wmin) : 0);
}

// ----------------------------------------------------------------------------
// compact: after a pull sweep, the next frontier's bitmap -> queue slice,
// edge count and heavy list.  A block takes every gridDim-th word of the
// bitmap (hub-first ids: the first words hold the heavy vertices, whose
// chunks take the time), its words dealt out to its warps in turn, and
// reserves its queue slots with one atomicAdd; a warp goes through its words
// a lane per vertex, so the row offsets come in coalesced.
// ----------------------------------------------------------------------------
template <int NT>
__device__ __forceinline__ void compact_level(const Args &a, const FCtl &c, int32_t *nq, int32_t *nhcur, long long *nfe)
{
    constexpr int NW = NT / 32;
    __shared__ int s_cnt[NW], s_base;
    const uint32_t *nb = bm_buf(a, (c.cur + 1) % 3);
    const int lane = mgd::lane(), warp = threadIdx.x >> 5;
    int4 *heavy = a.heavy + (size_t)(c.hpar ^ 1) * a.hcap;
    long long dsum = 0;
    for (int64_t w0 = blockIdx.x; w0 < a.words; w0 += (int64_t)gridDim.x * NT) {
        const int64_t wi = w0 + (int64_t)(lane * NW + warp) * gridDim.x;
        const uint32_t bits = wi < a.words ? nb[wi] : 0u;
        const int total = __reduce_add_sync(0xffffffffu, __popc(bits));
        if (lane == 0) s_cnt[warp] = total;
        __syncthreads();
        int base = 0, all = 0;
        for (int k = 0; k < NW; k++) {
            base += k < warp ? s_cnt[k] : 0;
            all += s_cnt[k];
        }
        if (threadIdx.x == 0 && all) s_base = atomicAdd(nq, all);
        __syncthreads();
        base += s_base;
        unsigned full = __ballot_sync(0xffffffffu, bits != 0);
        while (full) {
            const int j = __ffs(full) - 1;
            full &= full - 1;
            const uint32_t word = __shfl_sync(0xffffffffu, bits, j);
            const int32_t v = (int32_t)(w0 + (int64_t)(j * NW + warp) * gridDim.x) * 32 + lane;
            int32_t rb = 0, dg = 0;
            if ((word >> lane) & 1u) {
                a.queue[c.nqoff + base + __popc(word & ((1u << lane) - 1u))] = v;
                rb = a.row[v];
                dg = a.row[v + 1] - rb;
                dsum += dg;
            }
            base += __popc(word);
            if (a.has_heavy && __any_sync(0xffffffffu, dg > PUSH_HEAVY)) list_heavy(heavy, nhcur, v, rb, dg);
        }
        __syncthreads();   // s_cnt / s_base are reused
    }
    warp_add64(nfe, dsum);
}

__global__ void __launch_bounds__(THREADS) k_compact(Args a)
{
    const FCtl c = *a.ctl;
    if (c.mode != MODE_PULL || c.more == 0) return;
    compact_level<THREADS>(a, c, &a.ctl->nq, &a.ctl->nhcur, &a.ctl->nf_edges);
}

// ----------------------------------------------------------------------------
// decide: 1 thread
// ----------------------------------------------------------------------------
__device__ __forceinline__ void store_ctl(FCtl *p, const FCtl &c)
{
    int2 *d = reinterpret_cast<int2 *>(p);
    const int2 *s = reinterpret_cast<const int2 *>(&c);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(FCtl) / 8); i++) d[i] = s[i];
}

// End of a level (one thread, no other thread touching the loop state):
// next queue slice, direction switch, caps.  Works on a register copy (one
// batch of parallel loads, one batch of stores).  Returns the continue flag.
__device__ __forceinline__ int decide_step(const Args &a)
{
    FCtl c = load_ctl(a.ctl);
    if (c.more == 0) return 0;
    const int more = decide_local(a, c, c.nq, c.nhcur, c.nf_edges, true);
    store_ctl(a.ctl, c);
    return more;
}

__global__ void k_decide(Args a, cudaGraphConditionalHandle h, int use_cond)
{
    if (threadIdx.x != 0) return;
    *a.fmin = INT32_MAX;  // the next pull level's k_fmin starts from here
    const int more = decide_step(a);
    if (use_cond) cudaGraphSetConditional(h, more ? 1u : 0u);
}

// Persistent push phase: consecutive push levels in one cooperative launch,
// one grid barrier per level (push level | barrier | every block decides
// from the level's counters on its own copy of the loop state, the same
// inputs giving the same decision everywhere), until the traversal ends or
// the direction switch picks pull; block 0 writes the loop state back.
// High-diameter graphs (lattices, road networks) spend thousands of levels
// here, each a few microseconds instead of a round of kernel launches.  A
// barrier timeout sets status 3 and ends the traversal.
// Every block reads the loop state once per level: one warp loads it
// (one L2 request per block instead of one per warp) and shares it.
__device__ __forceinline__ FCtl block_load_ctl(const FCtl *p)
{
    __shared__ int2 s_c[sizeof(FCtl) / 8];
    if (threadIdx.x < sizeof(FCtl) / 8) s_c[threadIdx.x] = __ldcg(reinterpret_cast<const int2 *>(p) + threadIdx.x);
    __syncthreads();
    FCtl c;
    int2 *d = reinterpret_cast<int2 *>(&c);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(FCtl) / 8); i++) d[i] = s_c[i];
    __syncthreads();
    return c;
}

// the push phase's loop state back to global memory for the other kernels
// (and blocks), all but the last word (the scanned-edges statistic, which
// the push levels add to atomically)
__device__ __forceinline__ void store_ctl_push(FCtl *p, const FCtl &c)
{
    int2 *d = reinterpret_cast<int2 *>(p);
    const int2 *src = reinterpret_cast<const int2 *>(&c);
    for (int i = 0; i < (int)(sizeof(FCtl) / 8) - 1; i++) __stcg(&d[i], src[i]);
}

// Whether the next push levels are block 0's alone.  Path counts are summed
// there over a new vertex's whole in-row by one thread: not on graphs whose
// rows average more than eight edges (a level of 4,096 edges pulls thousands of
// whole rows: BC of 256 K vertices of degree 16 345 us with it, 218 without;
// the push levels of 1 M of degree 64 464 and 73), nor on a directed graph
// with a long in-row, of which its out-degrees say nothing (reaching a vertex
// of two million in-edges: 220 ms by one thread, 0.4 ms in the grid's levels,
// which touch the frontier's out-edges only).
template <class Op, bool HEAVY>
__device__ __forceinline__ bool block_phase_due(const Args &a, const FCtl &c)
{
    return !HEAVY && kBlockLevels<Op> && (!Op::kPathCounts || a.short_pull) && c.qsize <= CTA_ENTER &&
           c.qedges <= CTA_EDGES;
}

// Block 0's levels while the others wait; false when a barrier failed
template <class Op>
__device__ __forceinline__ bool block_phase(const Args &a, FCtl &c)
{
    if constexpr (kBlockLevels<Op>) {
        // the bitmaps start from zero
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * a.words; i += gridDim.x * blockDim.x) a.bm[i] = 0;
        if (!mgd::grid_sync(a.bar, a.bar_err, a.bar_never)) return false;
        if (blockIdx.x == 0) {
            extern __shared__ __align__(16) unsigned char s_dyn[];
            cta_push_levels<Op>(a, c, *reinterpret_cast<CtaShared *>(s_dyn));
            if (threadIdx.x == 0) store_ctl_push(a.ctl, c);
        }
        if (!mgd::grid_sync(a.bar, a.bar_err, a.bar_never)) return false;
        const FCtl c1 = block_load_ctl(a.ctl);
        if (threadIdx.x == 0) c = c1;
        __syncthreads();
    }
    return true;
}

// HEAVY: the graph may have vertices above PUSH_HEAVY out-edges (graphs that
// have none run without the chunk code and its votes).
// PER_SM: blocks of it on an SM; with two, no levels are one block's alone.
template <class Op, bool HEAVY, int PER_SM>
__global__ void __launch_bounds__(PTHREADS, PER_SM) k_sparse_levels(Args a)
{
    __shared__ FCtl s_c;
    __shared__ int4 s_cnt;
    {
        const FCtl c0 = block_load_ctl(a.ctl);
        if (threadIdx.x == 0) s_c = c0;
        __syncthreads();
    }
    bool ran = false;
    for (int32_t lv = 0; lv <= a.n + 2; lv++) {
        if (s_c.more == 0 || s_c.mode != MODE_PUSH) break;
        ran = true;
        LevelCnt *lc = a.cnt + (lv & 3);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            LevelCnt *z = a.cnt + ((lv + 2) & 3);
            z->nq = 0;
            z->nhcur = 0;
            z->nfe = 0;
        }
        if constexpr (PER_SM == 1) {
            if (block_phase_due<Op, HEAVY>(a, s_c)) {
                if (!block_phase<Op>(a, s_c)) break;
                continue;
            }
        }
        push_level<Op, HEAVY>(a, s_c, lc);
        if (!mgd::grid_sync(a.bar, a.bar_err, a.bar_never)) break;
        if (threadIdx.x == 0) {
            s_cnt = __ldcg(reinterpret_cast<const int4 *>(lc));  // nq, nhcur, nfe (lo, hi)
            FCtl c = s_c;
            const long long nfe = (long long)(((unsigned long long)(unsigned)s_cnt.w << 32) | (unsigned)s_cnt.z);
            decide_local(a, c, s_cnt.x, s_cnt.y, nfe, blockIdx.x == 0);
            s_c = c;
        }
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        FCtl c = s_c;
        if (*(volatile int *)a.bar_err) {
            c.status = 3;
            c.more = 0;
        }
        if (ran || c.status) store_ctl_push(a.ctl, c);
    }
}

// ----------------------------------------------------------------------------
// init: source
// ----------------------------------------------------------------------------
// sources: srcs[0..nsrc) when srcs is non-null, else the single `src`
// (several sources = one traversal of a disjoint union of graphs), a thread
// each of one block (one thread walking 30 sources took 33 us)
constexpr int INIT_THREADS = 256;
struct StartArgs {
    int32_t src;
    const int32_t *srcs;
    int32_t nsrc;
    int dirmode, alpha, beta, max_iter;
};

template <class Op>
__device__ __forceinline__ void start_sources(const Args &a, const StartArgs &st)
{
    __shared__ int s_q;
    __shared__ unsigned long long s_ve;
    FCtl *c = a.ctl;
    if (threadIdx.x == 0) {
        s_q = 0;
        s_ve = 0;
        std::memset(c, 0, sizeof(FCtl));
        c->more = 1;
        c->archive = Op::kLevelSync;
        c->max_iter = st.max_iter;
        c->dirmode = st.dirmode;
        c->alpha = st.alpha;
        c->beta = st.beta;
        c->mode = (st.dirmode == MG_DIR_PULL) ? MODE_PULL : MODE_PUSH;
        *a.fmin = INT32_MAX;
    }
    __syncthreads();
    const int32_t count = st.srcs ? st.nsrc : 1;
    for (int32_t i0 = threadIdx.x & ~31; i0 < count; i0 += blockDim.x) {
        const int32_t i = i0 + mgd::lane();
        const int32_t s = i < count ? (st.srcs ? st.srcs[i] : st.src) : -1;
        int32_t b = 0, d = 0;
        if (s >= 0 && mgd::bm_set(a.visited, s)) {  // (a duplicate source is queued once)
            a.label[s] = Op::source_value();
            if (Op::kPathCounts) a.sigma[s] = mgops::pc_one();
            mgd::bm_set(a.bm, s);  // buffer 0 is the current frontier
            a.queue[atomicAdd(&s_q, 1)] = s;
            b = a.row[s];
            d = a.row[s + 1] - b;
            atomicAdd(&s_ve, (unsigned long long)d);
        }
        if (a.has_heavy && __any_sync(0xffffffffu, d > PUSH_HEAVY)) list_heavy(a.heavy, &c->hcur, s, b, d);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int32_t q = s_q;
        c->qsize = q;
        c->nqoff = Op::kLevelSync ? q : a.n;
        c->visited_edges = (long long)s_ve;
        c->qedges = (int32_t)min(s_ve, (unsigned long long)INT32_MAX);
        if (Op::kLevelSync) { a.lvl_off[0] = 0; a.lvl_off[1] = q; c->nlevels = 1; }
    }
}

template <class Op>
__global__ void __launch_bounds__(INIT_THREADS) k_init(Args a, StartArgs st)
{
    start_sources<Op>(a, st);
}

// The whole traversal of a small graph in one cooperative launch: start
// values, push and pull levels, the result in caller order.  The loop of the
// large form (k_sparse_levels, k_fmin, k_pull, k_compact, k_decide inside a
// WHILE node) costs 15 to 20 us per switch between push and pull however
// small the levels; here a pull level is two phases and two grid barriers.
// BFS R-MAT 12: 97 -> 65 us on the device.
template <class Op, bool HEAVY>
__global__ void __launch_bounds__(PTHREADS, 1) k_frontier_all(Args a, StartArgs st, const int32_t *old2new,
                                                              int32_t *out)
{
    __shared__ FCtl s_c;
    __shared__ int32_t s_fmin;
    const int gtid = blockIdx.x * PTHREADS + threadIdx.x, nthreads = gridDim.x * PTHREADS;
    for (int32_t v = gtid; v < a.n; v += nthreads) {
        a.label[v] = Op::initialize();
        if (Op::kPathCounts) a.sigma[v] = mgops::pc_zero();
    }
    for (int32_t i = gtid; i < 3 * a.words; i += nthreads) a.bm[i] = 0;
    for (int32_t i = gtid; i < a.words; i += nthreads) a.visited[i] = 0;
    if (gtid < 4) {
        a.cnt[gtid].nq = a.cnt[gtid].nhcur = 0;
        a.cnt[gtid].nfe = 0;
        a.cnt[gtid].fmin = INT32_MAX;
    }
    bool ok = mgd::grid_sync(a.bar, a.bar_err, a.bar_never);
    if (ok && blockIdx.x == 0) start_sources<Op>(a, st);
    ok = ok && mgd::grid_sync(a.bar, a.bar_err, a.bar_never);
    if (ok) {
        const FCtl c0 = block_load_ctl(a.ctl);
        if (threadIdx.x == 0) s_c = c0;
    }
    __syncthreads();
    for (int32_t lv = 0; ok && s_c.more; lv++) {
        LevelCnt *lc = a.cnt + (lv & 3);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            LevelCnt *z = a.cnt + ((lv + 2) & 3);
            z->nq = 0;
            z->nhcur = 0;
            z->nfe = 0;
            z->fmin = INT32_MAX;
        }
        if (s_c.mode == MODE_PUSH) {
            if (block_phase_due<Op, HEAVY>(a, s_c)) {
                ok = block_phase<Op>(a, s_c);
                continue;
            }
            push_level<Op, HEAVY>(a, s_c, lc);
        } else {
            int32_t bound = 0;
            if constexpr (Op::kMinPlusBound) {
                frontier_min(a, s_c, &lc->fmin);
                if (!(ok = mgd::grid_sync(a.bar, a.bar_err, a.bar_never))) break;
                if (threadIdx.x == 0) s_fmin = __ldcg(&lc->fmin);
                __syncthreads();
                bound = sssp_bound(s_fmin, a.wmin);
            }
            pull_level<Op, Op::kMinPlusBound, PTHREADS>(a, s_c, bound);
            if (!(ok = mgd::grid_sync(a.bar, a.bar_err, a.bar_never))) break;
            compact_level<PTHREADS>(a, s_c, &lc->nq, &lc->nhcur, &lc->nfe);
        }
        if (!(ok = mgd::grid_sync(a.bar, a.bar_err, a.bar_never))) break;
        if (threadIdx.x == 0) {
            const int4 cnt = __ldcg(reinterpret_cast<const int4 *>(lc));  // nq, nhcur, nfe (lo, hi)
            FCtl c = s_c;
            const long long nfe = (long long)(((unsigned long long)(unsigned)cnt.w << 32) | (unsigned)cnt.z);
            decide_local(a, c, cnt.x, cnt.y, nfe, blockIdx.x == 0);
            s_c = c;
        }
        __syncthreads();
    }
    if (ok && out)
        for (int32_t v = gtid; v < a.n; v += nthreads) out[v] = __ldcg(&a.label[__ldg(&old2new[v])]);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        FCtl c = s_c;
        if (!ok || *(volatile int *)a.bar_err) {
            c.status = 3;
            c.more = 0;
        }
        store_ctl_push(a.ctl, c);
    }
}

// ----------------------------------------------------------------------------

// every vertex's label = the operator's initial value
template <class Op>
__global__ void k_label_init(int32_t *label, int32_t n)
{
    for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        label[v] = Op::initialize();
}

// per-instantiation tag: its address keys the workspace's captured loop and
// the persistent kernel's resident grid for this operator
template <class Op>
struct OpTag {
    static const char id;
};
template <class Op>
const char OpTag<Op>::id = 0;

}  // namespace

// ----------------------------------------------------------------------------
// workspace (shared by every operator run on a graph; freed with the graph)
// ----------------------------------------------------------------------------
struct FrontierWS {
    mgi::DevBuf label, sigma, sigma_d, bm, visited, queue, heavy, lvl_off, ctl;
    mgi::DevBuf q, delta, bc, bctl, bitem, barrive, bpart, srcbuf;
    mgi::DevBuf bar;        // grid barrier words + error flag of the persistent kernels
    mgi::DevBuf cnt;        // LevelCnt[4] of the persistent push phase
    std::map<const void *, int> coop_grid;      // resident blocks of k_sparse_levels<Op>, by operator tag
    int coop_back = 0;                          // resident blocks of k_bc_back_levels
    std::map<const void *, mgi::LoopGraph> lg;  // captured loop per operator tag
};

namespace {

using namespace mgi;

// no vertex of 128 edges, rows of more than DENSE_ROWS edges on average
inline bool dense_rows(const mg_graph *g) { return !g->relabeled && (int64_t)g->ne > DENSE_ROWS * g->nv; }

template <class Op>
mg_status ensure_ws(mg_graph *g)
{
    if (!g->fws) g->fws = new FrontierWS();
    FrontierWS *w = g->fws;
    const size_t n = (size_t)std::max(g->nv, 1);
    const size_t words = (n + 31) / 32;
    MG_TRY(dev_alloc(w->label, n * 4));
    MG_TRY(dev_alloc(w->bm, 3 * words * 4));
    MG_TRY(dev_alloc(w->visited, words * 4));
    MG_TRY(dev_alloc(w->queue, 2 * n * 4));
    MG_TRY(dev_alloc(w->heavy, 2 * (size_t)heavy_cap(g->ne) * sizeof(int4)));
    MG_TRY(dev_alloc(w->ctl, sizeof(FCtl)));
    MG_TRY(dev_alloc(w->lvl_off, (n + 3) * 4));
    MG_TRY(dev_alloc(w->bar, BAR_BYTES));
    MG_TRY(dev_alloc(w->cnt, 4 * sizeof(LevelCnt)));
    if (Op::kPathCounts) MG_TRY(dev_alloc(w->sigma, n * sizeof(mgops::PathCount)));
    int &cg = w->coop_grid[&OpTag<Op>::id];
    if (cg == 0) {
        int per_sm = 0;
        if (g->relabeled)
            MG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sparse_levels<Op, true, 1>, PTHREADS, 0));
        else if (dense_rows(g))
            MG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sparse_levels<Op, false, 2>, PTHREADS, 0));
        else {
            MG_CUDA(cudaFuncSetAttribute(k_sparse_levels<Op, false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(CtaShared)));
            MG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sparse_levels<Op, false, 1>, PTHREADS,
                                                                  sizeof(CtaShared)));
        }
        if (per_sm < 1) return fail(MG_ERR_CUDA, "persistent push kernel does not fit on an SM");
        cg = (dense_rows(g) ? std::min(per_sm, 2) : 1) * g->num_sms;
    }
    return MG_OK;
}

// cooperative launch (all blocks resident) of the persistent push phase
template <class Op>
mg_status launch_sparse_levels(const mg_graph *g, const Args &a, int grid, cudaStream_t st)
{
    const bool dense = dense_rows(g);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(PTHREADS);
    cfg.dynamicSmemBytes = a.has_heavy || dense ? 0 : sizeof(CtaShared);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (a.has_heavy) MG_CUDA(cudaLaunchKernelEx(&cfg, k_sparse_levels<Op, true, 1>, a));
    else if (dense) MG_CUDA(cudaLaunchKernelEx(&cfg, k_sparse_levels<Op, false, 2>, a));
    else MG_CUDA(cudaLaunchKernelEx(&cfg, k_sparse_levels<Op, false, 1>, a));
    return MG_OK;
}

// Graphs of up to this many edges run a traversal in one launch
// (k_frontier_all); past them the pull kernels' twice as many resident warps
// are worth the launches.  us, one launch / separate: BFS R-MAT 16 (1.8 M
// edges) 77 / 111, R-MAT 18 (7.6 M) 163 / 144; SSSP 190 / 223 and 372 / 296.
// Without heavy vertices the levels are more even and the line for
// level-synchronous operators lies higher.  BFS of random graphs: 1 M vertices
// of degree 16 (16.8 M edges) 157 / 230, 4 M of degree 8 (33 M) 483 / 446, 1 M
// of degree 64 (67 M; only pushed, 653 / 503), 4 M of degree 16 (67 M) 483 /
// 423; lattices, ms: 1500 x 1400 (8.6 M) 9.1 / 10.2, 3000 x 3000 (36 M) 28.2 /
// 28.4.
constexpr int64_t ONE_LAUNCH_EDGES_SYNC = 4 << 20, ONE_LAUNCH_EDGES_FLAT = 16 << 20, ONE_LAUNCH_EDGES_RELAX = 3 << 20;
template <class Op>
bool one_launch_pays(const mg_graph *g)
{
    if (Op::kLevelSync) return g->ne <= (g->relabeled ? ONE_LAUNCH_EDGES_SYNC : ONE_LAUNCH_EDGES_FLAT);
    return g->ne <= ONE_LAUNCH_EDGES_RELAX;
}

template <class Op>
mg_status launch_frontier_all(const Args &a, const StartArgs &st, int grid, const int32_t *old2new, int32_t *out,
                              cudaStream_t s)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(PTHREADS);
    cfg.dynamicSmemBytes = a.has_heavy ? 0 : sizeof(CtaShared);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (a.has_heavy) {
        MG_CUDA(cudaLaunchKernelEx(&cfg, k_frontier_all<Op, true>, a, st, old2new, out));
    } else {
        MG_CUDA(cudaFuncSetAttribute(k_frontier_all<Op, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(CtaShared)));
        MG_CUDA(cudaLaunchKernelEx(&cfg, k_frontier_all<Op, false>, a, st, old2new, out));
    }
    return MG_OK;
}

inline Args make_args(mg_graph *g)
{
    FrontierWS *w = g->fws;
    Args a;
    std::memset(&a, 0, sizeof(a));
    a.n = g->nv;
    a.m = g->ne;
    a.row = g->row.as<int32_t>(); a.col = g->col.as<int32_t>(); a.wt = g->wt.as<int32_t>();
    a.trow = g->trow; a.tcol = g->tcol; a.twt = g->twt;
    a.wrows = g->wrows.as<int32_t>(); a.nwrows = g->nwrows; a.nwlong = g->nwlong;
    a.trows = g->trows.as<int32_t>(); a.ntrows = g->ntrows;
    a.hchunk = g->hchunk.as<int32_t>(); a.nhchunks = g->nhchunks;
    a.heavy_deg = g->heavy_deg;
    a.label = w->label.as<int32_t>();
    a.sigma = w->sigma.as<mgops::PathCount>();
    a.bc_ext = g->bc_ext ? 1 : 0;
    a.bc_ovf = reinterpret_cast<int32_t *>(w->bar.as<unsigned>() + OVF_WORD);
    a.fmin = reinterpret_cast<int32_t *>(w->bar.as<unsigned>() + FMIN_WORD);
    a.wmin = std::max(g->min_weight, 0);
    a.bm = w->bm.as<uint32_t>();
    a.visited = w->visited.as<uint32_t>();
    a.words = (std::max(g->nv, 1) + 31) / 32;
    a.queue = w->queue.as<int32_t>();
    a.heavy = w->heavy.as<int4>();
    a.hcap = heavy_cap(g->ne);
    a.has_heavy = g->relabeled;  // (graphs with a degree of 128 or more are relabeled)
    a.short_pull = g->short_pull;
    a.lvl_off = w->lvl_off.as<int32_t>();
    a.ctl = w->ctl.as<FCtl>();
    a.bar = w->bar.as<unsigned>();
    a.cnt = w->cnt.as<LevelCnt>();
    a.bar_err = reinterpret_cast<int *>(w->bar.as<unsigned>() + 2 + mgd::GRID_SYNC_GROUPS);
    a.bar_never = mgi::fail_barrier();
    return a;
}

// every by-value argument of the captured kernels: the whole Args (pointers,
// sizes, the min-plus skip bound's least weight, the injection flag, the
// path-count mode), the operator and the launch grids
inline LoopKey key_of(const Args &a, const void *op_tag, int grid, int coop_grid)
{
    return LoopKey().add(op_tag).add(a).add(grid).add(coop_grid);
}

// result slot `which` in caller ids (mapped on the device before the run ends)
inline mg_status publish(mg_graph *g, int which, const void *src, size_t elem)
{
    const void *p = nullptr;
    MG_TRY(to_caller(g, which, src, elem, 1, &p));
    g->res[which] = p;
    return MG_OK;
}

template <class Op>
mg_status frontier_run_impl(mg_graph *g, int32_t src, const int32_t *srcs_host, int32_t nsrc, const mg_opts &opt,
                            mg_run_info *info, int which);

// what the loop state says after a run; an overflow of plain path counts
// starts the run over with extended ones
template <class Op>
mg_status frontier_outcome(mg_graph *g, const Args &a, int32_t src, const int32_t *srcs_host, int32_t nsrc,
                           const mg_opts &opt, int max_iter, mg_run_info *info, int which)
{
    cudaStream_t s = g->stream;
    // (page-locked: the loop state, then the overflow word)
    static_assert(sizeof(FCtl) <= 256, "pinned_flag holds 512 bytes");
    int32_t *hovf = g->pinned_flag + 64;
    *hovf = 0;
    MG_CUDA(cudaMemcpyAsync(g->pinned_flag, a.ctl, sizeof(FCtl), cudaMemcpyDeviceToHost, s));
    if (Op::kPathCounts) MG_CUDA(cudaMemcpyAsync(hovf, a.bc_ovf, 4, cudaMemcpyDeviceToHost, s));
    MG_TRY(run_status_wait(g));
    FCtl hc;
    std::memcpy(&hc, g->pinned_flag, sizeof(hc));
    const int32_t ovf = *hovf;
    if (ovf && !g->bc_ext) {
        // a path count passed FP64's comfortable range: this graph's BC runs
        // use extended path counts from now on, starting with this one
        g->bc_ext = true;
        return frontier_run_impl<Op>(g, src, srcs_host, nsrc, opt, info, which);
    }
    if (info) {
        info->iterations = hc.iter;
        info->pull_iterations = hc.pull_iters;
        info->edges_scanned = hc.scanned;
    }
    if (hc.status == 3) return fail(MG_ERR_CUDA, "grid barrier of a persistent traversal kernel timed out");
    if (hc.status != 0) return fail(MG_ERR_ITER_LIMIT, "iteration cap %d reached", max_iter);
    return MG_OK;
}

// Forward traversal with operator Op from src (or from the nsrc sources in
// srcs_host when it is non-null); the labels in the workspace and, for
// which >= 0, in caller order in the graph's result slot `which`.
template <class Op>
mg_status frontier_run_impl(mg_graph *g, int32_t src, const int32_t *srcs_host, int32_t nsrc, const mg_opts &opt,
                            mg_run_info *info, int which)
{
    static_assert(!Op::kLevelSync || Op::kFirstParent || Op::kPathCounts,
                  "a level-synchronous operator is first-parent (BFS) or carries path counts (BC)");
    if (!srcs_host && (src < 0 || src >= g->nv)) return fail(MG_ERR_RANGE, "source %d out of range [0,%d)", src, g->nv);
    if (Op::kMinPlusBound && g->min_weight < 0)
        return fail(MG_ERR_INVALID, "%s needs non-negative edge weights (min weight %d)", Op::kTag, g->min_weight);
    MG_TRY(ensure_ws<Op>(g));
    const int32_t *srcs_dev = nullptr;
    if (srcs_host) {
        if (nsrc <= 0 || nsrc > g->nv) return fail(MG_ERR_INVALID, "invalid source count %d", nsrc);
        MG_TRY(dev_alloc(g->fws->srcbuf, (size_t)nsrc * 4));
        MG_CUDA(cudaMemcpyAsync(g->fws->srcbuf.p, srcs_host, (size_t)nsrc * 4, cudaMemcpyHostToDevice, g->stream));
        srcs_dev = g->fws->srcbuf.as<int32_t>();
    }
    FrontierWS *w = g->fws;
    Args a = make_args(g);
    cudaStream_t s = g->stream;
    const size_t n = (size_t)g->nv;
    const int grid = launch_grid(g, THREADS, 8);
    int max_iter = opt.max_iter > 0 ? opt.max_iter : (Op::kLevelSync ? g->nv + 2 : 4 * g->nv + 16);
    int alpha = opt.alpha > 0 ? opt.alpha : (Op::kLevelSync ? 15 : 4), beta = opt.beta > 0 ? opt.beta : 18;
    StartArgs st;
    std::memset(&st, 0, sizeof(st));
    st.src = src;
    st.srcs = srcs_dev;
    st.nsrc = nsrc;
    st.dirmode = opt.direction;
    st.alpha = alpha;
    st.beta = beta;
    st.max_iter = max_iter;
    if (opt.exec == MG_EXEC_GRAPH && !opt.profile && one_launch_pays<Op>(g)) {
        int32_t *out = nullptr;
        if (which >= 0 && g->relabeled) {
            MG_TRY(dev_alloc(g->res_out[which], std::max<size_t>(n, 1) * 4));
            out = g->res_out[which].as<int32_t>();
        }
        MG_CUDA(cudaMemsetAsync(w->bar.p, 0, BAR_BYTES, s));
        MG_TRY(launch_frontier_all<Op>(a, st, g->num_sms, g->old2new.as<int32_t>(), out, s));
        if (which >= 0) g->res[which] = out ? (const void *)out : w->label.p;
        return frontier_outcome<Op>(g, a, src, srcs_host, nsrc, opt, max_iter, info, which);
    }
    if (n) k_label_init<Op><<<grid, THREADS, 0, s>>>(a.label, (int32_t)n);
    MG_CUDA(cudaMemsetAsync(a.bm, 0, 3 * (size_t)a.words * 4, s));
    MG_CUDA(cudaMemsetAsync(a.visited, 0, (size_t)a.words * 4, s));
    MG_CUDA(cudaMemsetAsync(w->bar.p, 0, BAR_BYTES, s));
    if (Op::kPathCounts) MG_CUDA(cudaMemsetAsync(a.sigma, 0, n * sizeof(mgops::PathCount), s));
    k_init<Op><<<1, INIT_THREADS, 0, s>>>(a, st);
    MG_CUDA(cudaGetLastError());
    const void *tag = &OpTag<Op>::id;
    const int coop = w->coop_grid[tag];
    Profiler &P = g->prof;
    const std::string t(Op::kTag);
    const int sp = P.slot((t + "_push").c_str());
    const int sl = P.slot((t + "_pull").c_str());
    const int sc = P.slot("frontier_compact");
    const int sf = Op::kMinPlusBound ? P.slot((t + "_fmin").c_str()) : -1;
    const int sd = P.slot("frontier_decide");
    const bool every_offer = Op::kMinPlusBound && opt.direction != MG_DIR_PULL;   // k_pull's form
    BodyFn body = [&](cudaStream_t st, cudaGraphConditionalHandle h, int use_cond) -> mg_status {
        MG_CUDA(cudaMemsetAsync(a.cnt, 0, 4 * sizeof(LevelCnt), st));
        P.begin(sp);
        MG_TRY(launch_sparse_levels<Op>(g, a, coop, st));
        P.end();
        if (Op::kMinPlusBound) {
            P.begin(sf);
            k_fmin<<<grid, THREADS, 0, st>>>(a);
            P.end();
        }
        P.begin(sl);
        if (every_offer) k_pull<Op, Op::kMinPlusBound><<<grid, THREADS, 0, st>>>(a);
        else k_pull<Op, false><<<grid, THREADS, 0, st>>>(a);
        P.end();
        P.begin(sc);
        k_compact<<<grid, THREADS, 0, st>>>(a);
        P.end();
        P.begin(sd);
        k_decide<<<1, 32, 0, st>>>(a, h, use_cond);
        P.end();
        MG_CUDA(cudaGetLastError());
        return MG_OK;
    };
    MG_TRY(run_loop(opt.profile ? MG_EXEC_HOST : opt.exec, opt.profile != 0, s, w->lg[tag],
                    key_of(a, tag, grid, coop).add(every_offer), body, &a.ctl->more, g->pinned_flag, max_iter + 2));
    if (which >= 0) MG_TRY(publish(g, which, a.label, 4));
    return frontier_outcome<Op>(g, a, src, srcs_host, nsrc, opt, max_iter, info, which);
}

// One whole run of a label operator through the C ABI's conventions:
// source in caller ids, labels out in caller order (nv int32, when
// label_out is non-NULL), status and run info as mg_bfs / mg_sssp.
template <class Op>
mg_status frontier_operator_run(mg_graph *g, int32_t source, const mg_opts *o, int32_t *label_out,
                                mg_run_info *info)
{
    mg_opts opt;
    MG_TRY(begin_run(g, o, opt, info));
    if (source < 0 || source >= g->nv) return fail(MG_ERR_RANGE, "source %d out of range [0,%d)", source, g->nv);
    const size_t bytes = (size_t)g->nv * 4;
    HostPages pages(g, {{label_out, nullptr, bytes}});
    MG_TRY(frontier_run_impl<Op>(g, to_engine(g, source), nullptr, 0, opt, info, MG_RES_LEVEL));
    pages.wait();
    return end_run(g, opt, info, {{label_out, g->res[MG_RES_LEVEL], bytes}});
}

}  // namespace
