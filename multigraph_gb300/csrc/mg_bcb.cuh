// mg_bcb.cuh -- batched multi-source Brandes BC: 32 sources per traversal,
// one lane of a warp per source.  Structures, helpers and the phase bodies
// of the per-level kernels in mg_bcb.cu.
//
// The reference runs one BC source per program invocation (main.cu:52-86:
// MultiGraph_V_E_V forward, then MultiGraph_V_E_V_pull backward over the
// archived levels, process2.cu:263-325).  Here a group of up to 32 sources
// is traversed together, level-synchronously:
//
//   vis[v]   bit s set once v has been reached from source s
//   fm[v]    bit s set when v is on source s's current frontier
//   path counts  of v from source s, in one of three forms; a count that does
//                not fit sets a flag and the run repeats in the next form:
//                  M_INT   uint32 below INT_LIMIT = 2^29, so that eight add
//                          up in 32 bits, summed in 64 (exact); graphs above
//                          TP_AVG_DEG start here
//                  M_PLAIN FP64 below mgops::PC_PLAIN_MAX = 2^90
//                          (low-degree graphs start here)
//                  M_EXT   mgops::PathCount, FP64 mantissa with a 2^512 scale
//                M_INT keeps two arrays [n][32], one per level parity
//                (cnt[level & 1]); the others one PathCount array sig
//   q[v*32+s]    (1 + delta_s[v]) / count   (backward; FP32, FP64 in M_EXT;
//                M_INT: qp[level & 1])
//   archive  (vertex, mask) entries, grouped by level: entry (v, M) at
//            level d means v is at distance d from exactly the sources in M
//
// Forward level d -> d+1 (three launches, four with heavy rows, looped by a
// CUDA-graph WHILE node):
//   k_bb_mark     sparse levels only: frontier entries scan their out-edges
//                 and collect the distinct candidate destinations (a vertex
//                 not yet reached by some source of the entry's mask)
//   k_bb_pull     each candidate row (sparse) or every row that some source
//                 has not reached (dense) scans its in-edges; a warp loads 32
//                 column ids and their frontier masks at once, keeps the
//                 lanes that hit (ballot), and lane s adds sig[u*32+s] for
//                 each hit of source s.  Rows above heavy_deg go in 2048-edge
//                 chunks whose partials land in hpart.
//   k_bb_heavy    (graphs with heavy rows) folds the chunk partials of heavy
//                 rows in chunk order
//   k_bb_compact  archives the new frontier (one atomic per warp), sums its
//                 out-degrees for the direction switch, clears the old
//                 frontier's masks; the last block to finish decides the
//                 next level (sparse/dense: Beamer, frontier out-edges x
//                 alpha against m) and the loop condition
// Backward level L (two launches, three with heavy rows): level l's masks
// sit in a dense array fm[l % 3]; every level-L entry sums q over
// successors whose level-(L+1) mask shares the source, and lane s finishes
//   delta_s[u] = sig_s[u] * sum,  q_s[u] = (1 + delta_s[u]) / sig_s[u]
// with the per-vertex score bc[u] += sum of delta_s[u] over the entry's
// sources (u excluded as its own source); k_bbb_next then clears level
// L+1's masks, scatters level L-1's into the third buffer and steps L.
//
// Dense levels in M_INT (frontier out-edges above m / GATHER_FWD, resp.
// level out-edges above m / GATHER_BACK) need no masks at all.  An unreached
// row's reached in-neighbours are all on the frontier (a neighbour one level
// up would have reached it before), so the row's new counts are the plain
// sums of its in-neighbours' counts -- zero where unreached -- once the
// counts being written this level sit in another array: the parity arrays.
// The backward sums are the same over q (levels below L+1 still hold zero).
// k_bb_gather / k_bbb_gather then read a neighbour's 32 values as one line,
// eight lanes a row with a 16-byte load each, eight edges in flight (the
// layout of personalised PageRank's sweep), where the masked path tests,
// shuffles and loads one neighbour after another.  R-MAT 20, us per dense
// level: forward 1,340 -> 330, backward 1,280 -> 330.  FP64 is out of both
// paths: GB300's FP64 pipe was 60 % busy in the forward sums and 48 % in the
// backward finish (its score sums are pairs of FP32 now).
//
// On low-degree graphs (average degree <= 8) both pull kernels first give
// each row / entry with at most 8 edges and at most 4 sources at this level
// to one thread, which forms the same per-source sums in the same edge
// order (a lattice level is mostly such rows, with one source each, so a
// warp per row left 31 lanes idle); the rest go to the warp path above.
//
// Every sum runs in a fixed order (the warp's edge order, then chunk order),
// so results do not depend on scheduling; path counts are integers in FP64
// and exact up to 2^53.  The column stream and the frontier-mask gathers are
// shared by the 32 sources of a group, which is where the batch gains over
// one traversal per source.

#pragma once

#include "mg_device.cuh"
#include "mg_ops.cuh"

#include <algorithm>
#include <type_traits>
#include <cstring>
#include <vector>

namespace mgbc {

constexpr int W = 32;                 // sources per group (one per lane)
constexpr int THREADS = 256;
constexpr int32_t MARK_HEAVY = 2048;  // frontier entries above this out-degree are marked by the whole grid
// rows with at most TDEG edges whose level touches at most TBITS sources are
// handled by one thread (low-degree graphs: a lattice row has four or five
// edges and usually one source per level); the rest by a warp, lane per source
constexpr int TDEG = 8;
constexpr int TBITS = 4;
constexpr int TP_AVG_DEG = 8;  // graphs up to this average degree use the thread path
enum { M_INT = 0, M_PLAIN = 1, M_EXT = 2 };  // path-count forms
constexpr unsigned long long INT_LIMIT = 1ull << 29;
// levels summed without masks: forward when the frontier's out-edges exceed
// m / GATHER_FWD (most edges of a row then hit), backward when the level's
// entries hold more than m / GATHER_BACK edges
constexpr unsigned long long GATHER_FWD = 4, GATHER_BACK = 8;
constexpr int GTHREADS = 512;  // mask-free kernels: two blocks per SM at 64 registers
constexpr int GPER_SM = 2;

// what one forward level counts (atomics): candidates of a sparse level,
// entries archived for the next level, their heavy entries and out-edges,
// whether a path count did not fit.  A persistent sweep's level has a slot of
// its own for all of it: the next level's phases, which a faster block may
// have begun, write another one, so every block decides from the same words.
struct LvlCnt {
    int32_t ncand;
    int32_t nnew;
    int32_t nfh_build;
    int32_t status;            // 2: archive overflow
    unsigned long long nfe;
    int32_t ovf;               // a path count reached the form's limit (ends the sweep)
    int32_t pad;
};

struct BbCtl {
    int32_t more;
    int32_t d;          // forward level being expanded
    int32_t cur;        // fm buffer holding level d
    int32_t dense;      // this level pulls over every row (2: without masks)
    int32_t nfh;        // heavy frontier entries at level d
    int32_t nlevels;    // levels 0..nlevels-1 archived (set when the forward sweep ends)
    int32_t L;          // backward level
    int32_t status;     // 1: level cap reached, 2: archive overflow, 3: grid barrier timeout
    int32_t dirmode;    // MG_DIR_*
    int32_t alpha;
    int32_t max_levels;
    uint32_t gmask;     // lanes holding a source
    int32_t dense_levels;
    int32_t done;       // blocks finished (last-block-done step of the level's final kernel)
    int32_t ovf;        // a path count reached the form's limit (the sweep has ended for a rerun)
    int32_t pad;
    unsigned long long nfe_cur;  // out-edges of level d
    LvlCnt k;                    // this level's counters (per-level kernels)
};

// the next level from level d's counters; off_d2 = archive offset of level d+2
__device__ __forceinline__ void bb_decide(BbCtl &n, const LvlCnt &k, int32_t off_d1, int32_t &off_d2, int32_t m,
                                          int32_t mode)
{
    off_d2 = off_d1 + k.nnew;
    if (k.status) n.status = k.status;
    if (k.nnew == 0 || n.status || k.ovf) {  // (a path-count overflow ends the sweep for a rerun)
        n.more = 0;
        n.nlevels = n.d + 1;
        if (k.ovf) n.ovf = 1;
    } else if (n.d + 2 >= n.max_levels) {
        n.more = 0;
        n.status = 1;
        n.nlevels = n.d + 2;
    } else {
        n.d += 1;
        n.cur ^= 1;
        n.nfe_cur = k.nfe;
        n.nfh = k.nfh_build;
        if (n.dirmode == MG_DIR_PUSH) n.dense = 0;
        else if (n.dirmode == MG_DIR_PULL) n.dense = 1;
        else n.dense = n.nfe_cur * (unsigned long long)n.alpha > (unsigned long long)m;
        n.dense_levels += n.dense;
        if (n.dense && mode == M_INT && n.nfe_cur * GATHER_FWD > (unsigned long long)m) n.dense = 2;
    }
}

struct BbArgs {
    int32_t n;
    int32_t m;
    const int32_t *row, *col;    // out-edges
    const int32_t *trow, *tcol;  // in-edges
    const int32_t *hchunk;       // (row, begin, end) of the heavy in-rows
    int32_t nhchunks;
    const int32_t *hrows, *hrow_chunk;
    int32_t nhrows;
    int32_t heavy_deg;
    uint32_t *vis;
    uint32_t *fm0, *fm1, *fm2;   // frontier masks: forward fm0/fm1, backward level l in fm[l % 3]
    uint32_t *cbm;               // candidate bitmap (sparse levels)
    int32_t *cand;
    int32_t *arch;
    uint32_t *amask;
    size_t cap;                  // archive capacity (32 n)
    int32_t *off;                // level offsets into the archive
    mgops::PathCount *sig;
    void *q;                     // float (plain counts) or double (extended) per (v, source)
    mgops::PathCount *hpart;     // per chunk x 32 lanes (backward reuses it as double)
    int32_t mode;                // M_INT / M_PLAIN / M_EXT
    uint32_t *cnt[2];            // M_INT: counts by level parity
    float *qp[2];                // M_INT: q by level parity
    unsigned long long *lnfe;    // out-edges of every level's entries
    // rows above GCHUNK edges in GCHUNK-edge chunks (mask-free levels)
    const int32_t *gchunk, *grows, *grow_chunk;
    int32_t ngchunks, ngrows;
    void *gpart;                 // [ngchunks][32] partial sums (uint64 / float)
    uint32_t *hmask;
    float2 *bc;                  // scores (all groups): sum as an unevaluated pair high + low
    int32_t *fheavy;
    const int32_t *src;          // the group's sources (engine ids), W entries
    BbCtl *ctl;
    // persistent sweeps (low-degree graphs): grid barrier words (zero before
    // each sweep), the barrier's error word, four rotating level counters
    unsigned *bar;
    int *bar_err;
    LvlCnt *pcnt;
};

__device__ __forceinline__ uint32_t *fm_of(const BbArgs &a, int i) { return i ? a.fm1 : a.fm0; }
__device__ __forceinline__ uint32_t *fmb_of(const BbArgs &a, int32_t l)
{
    const int32_t r = l % 3;
    return r == 0 ? a.fm0 : (r == 1 ? a.fm1 : a.fm2);
}

// the control block as other blocks left it (L2, not a stale L1 line)
__device__ __forceinline__ BbCtl load_ctl_l2(const BbCtl *cp)
{
    BbCtl c;
    const int *src = reinterpret_cast<const int *>(cp);
    int *dst = reinterpret_cast<int *>(&c);
#pragma unroll
    for (int k = 0; k < (int)(sizeof(BbCtl) / 4); k++) dst[k] = __ldcg(src + k);
    return c;
}

// true in one thread of the last block of the grid to get here (every
// block's earlier writes and atomics are visible to it)
__device__ __forceinline__ bool last_block_done(int32_t *done)
{
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(done, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (s_last && threadIdx.x == 0) {
        __threadfence();
        return true;
    }
    return false;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long x)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// (hi, lo) += x, exact up to the rounding of lo (TwoSum)
__device__ __forceinline__ void pair_add(float &hi, float &lo, float x)
{
    const float s = hi + x, bp = s - hi;
    lo += (hi - (s - bp)) + (x - bp);
    hi = s;
}

// the score of u += (hi, lo)
__device__ __forceinline__ void score_add(const BbArgs &a, int32_t u, float hi, float lo)
{
    float2 b = a.bc[u];
    pair_add(b.x, b.y, hi);
    b.y += lo;
    a.bc[u] = b;
}

// a path count of each form: its sum while a row is pulled
template <int M>
struct SumOf {
    using T = mgops::PathCount;
};
template <>
struct SumOf<M_INT> {
    using T = unsigned long long;
};

// ---------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------
// items per warp: `cap`, or fewer (a power of two) when `count` items would
// leave warps idle
__device__ __forceinline__ int entries_per_warp(int32_t count, int nwarps, int cap)
{
    if (count >= nwarps * cap) return cap;
    const int want = max(1, count / nwarps);
    int v = 1;
    while (v * 2 <= want && v * 2 <= cap) v *= 2;
    return v;
}

__device__ __forceinline__ void mark_edge_block(const BbArgs &a, int32_t p, int32_t e, uint32_t f, int32_t *ncand)
{
    bool pred = false;
    int32_t v = 0;
    if (p < e) {
        v = __ldg(&a.col[p]);
        pred = (f & ~a.vis[v]) != 0 && mgd::bm_set(a.cbm, v);
    }
    int slot = mgd::warp_append(ncand, pred);
    if (pred) a.cand[slot] = v;
}

// sparse level d (archive entries [b0, b1)): collect the candidate rows
// (FLAT: no heavy entries)
template <bool FLAT = false>
__device__ __forceinline__ void bb_mark_phase(const BbArgs &a, const BbCtl &c, int32_t b0, int32_t b1, int32_t *ncand)
{
    const int lane = mgd::lane();
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    // up to 32 entries per warp (fewer when the level would leave warps
    // idle), their out-edges spread over the lanes by a load-balanced search
    const int vpw = entries_per_warp(b1 - b0, nwarps, 32);
    for (int32_t base = b0 + gwarp * vpw; base < b1; base += nwarps * vpw) {
        int32_t start = 0, deg = 0;
        uint32_t f = 0;
        if (lane < vpw && base + lane < b1) {
            const int32_t u = a.arch[base + lane];
            f = a.amask[base + lane];
            start = __ldg(&a.row[u]);
            deg = __ldg(&a.row[u + 1]) - start;
            if (!FLAT && deg > MARK_HEAVY) deg = 0;  // the grid-wide loop below
        }
        const int incl = mgd::warp_scan_incl(deg);
        const int excl = incl - deg;
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        for (int k0 = 0; k0 < total; k0 += 32) {
            const int k = k0 + lane;
            const int kk = k < total ? k : total - 1;
            const int own = mgd::owner_lane(excl, kk);
            const int32_t p = __shfl_sync(0xffffffffu, start, own) + (kk - __shfl_sync(0xffffffffu, excl, own));
            const uint32_t fo = __shfl_sync(0xffffffffu, f, own);
            mark_edge_block(a, k < total ? p : 0, k < total ? p + 1 : 0, fo, ncand);
        }
    }
    if (FLAT) return;
    // heavy frontier entries: every warp of the grid takes 32-edge slices
    const uint32_t *fcur = fm_of(a, c.cur);
    for (int32_t h = 0; h < c.nfh; h++) {
        const int32_t u = a.fheavy[h];
        const uint32_t f = fcur[u];
        const int32_t b = __ldg(&a.row[u]), e = __ldg(&a.row[u + 1]);
        for (int32_t base = b + gwarp * 32; base < e; base += nwarps * 32) mark_edge_block(a, base + lane, e, f, ncand);
    }
}

// One row's in-edges [b, e) against the frontier masks: lane s returns the
// sum of the counts over in-neighbours on source s's frontier (level d);
// *hit gets the union of the masks that hit (restricted to `want`).
template <int M>
__device__ __forceinline__ typename SumOf<M>::T pull_span(const BbArgs &a, const uint32_t *fcur, int32_t d, int32_t b,
                                                          int32_t e, uint32_t want, uint32_t &hit)
{
    const int lane = mgd::lane();
    mgops::PathCount acc = mgops::pc_zero();  // extended counts
    double accp = 0.0;                        // plain counts
    unsigned long long acci = 0;              // integer counts
    const uint32_t *cnt = a.cnt[d & 1];
    uint32_t newm = 0;
    for (int32_t base = b; base < e; base += 32) {
        const int32_t p = base + lane;
        int32_t u = 0;
        uint32_t f = 0;
        if (p < e) {
            u = __ldcs(&a.tcol[p]);
            f = fcur[u] & want;
        }
        unsigned hits = __ballot_sync(0xffffffffu, f != 0);
        if constexpr (M == M_INT) {
            // four hits' loads in flight
            while (hits) {
                uint32_t x[4] = {0, 0, 0, 0};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (hits) {
                        const int j = __ffs(hits) - 1;
                        hits &= hits - 1;
                        const int32_t uj = __shfl_sync(0xffffffffu, u, j);
                        const uint32_t fj = __shfl_sync(0xffffffffu, f, j);
                        newm |= fj;
                        if ((fj >> lane) & 1u) x[k] = cnt[(size_t)uj * W + lane];
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; k++) acci += x[k];
            }
        } else {
            while (hits) {
                const int j = __ffs(hits) - 1;
                hits &= hits - 1;
                const int32_t uj = __shfl_sync(0xffffffffu, u, j);
                const uint32_t fj = __shfl_sync(0xffffffffu, f, j);
                newm |= fj;
                if ((fj >> lane) & 1u) {
                    if (M == M_EXT) acc = mgops::pc_add(acc, a.sig[(size_t)uj * W + lane], true);
                    else accp += a.sig[(size_t)uj * W + lane].m;
                }
            }
        }
    }
    hit = newm;
    if constexpr (M == M_INT) {
        return acci;
    } else {
        if (M == M_PLAIN) acc.m = accp;
        return acc;
    }
}

// row v reached at level d + 1 from the sources in newm
template <int M>
__device__ __forceinline__ void settle_row(const BbArgs &a, uint32_t *fnext, int32_t d, int32_t v, uint32_t newm,
                                           typename SumOf<M>::T acc, LvlCnt *k)
{
    const int lane = mgd::lane();
    if ((newm >> lane) & 1u) {
        if constexpr (M == M_INT) {
            a.cnt[(d + 1) & 1][(size_t)v * W + lane] = (uint32_t)acc;
            if (acc >= INT_LIMIT) k->ovf = 1;
        } else {
            a.sig[(size_t)v * W + lane] = acc;
            if (M == M_PLAIN && acc.m >= mgops::PC_PLAIN_MAX) k->ovf = 1;
        }
    }
    if (lane == 0) {
        a.vis[v] |= newm;
        fnext[v] = newm;
    }
}

// One thread, one row v with at most TDEG in-edges: per source s in the
// sources that reach v at this level (at most TBITS of them, else false is
// returned and the row goes to the warp path), the sum of sig over the
// in-neighbours on s's frontier, in edge order as pull_span forms it.  The
// row's columns, their masks and a source's counts are loaded together.
// *reached gets those sources.
__device__ __forceinline__ bool pull_row_thread(const BbArgs &a, const uint32_t *fcur, uint32_t *fnext, int32_t v,
                                                uint32_t want, uint32_t *reached, LvlCnt *k)
{
    const int32_t b = __ldg(&a.trow[v]), e = __ldg(&a.trow[v + 1]);
    if (e - b > TDEG) return false;
    int32_t u[TDEG];
    uint32_t f[TDEG], newm = 0;
#pragma unroll
    for (int j = 0; j < TDEG; j++) u[j] = b + j < e ? __ldg(&a.tcol[b + j]) : -1;
#pragma unroll
    for (int j = 0; j < TDEG; j++) f[j] = u[j] >= 0 ? fcur[u[j]] : 0u;
#pragma unroll
    for (int j = 0; j < TDEG; j++) newm |= f[j];
    newm &= want;
    if (__popc(newm) > TBITS) return false;
    *reached = newm;
    if (newm == 0) return true;
    uint32_t mm = newm;
    while (mm) {
        const int s = __ffs(mm) - 1;
        mm &= mm - 1;
        mgops::PathCount acc = mgops::pc_zero();
#pragma unroll
        for (int h = 0; h < TDEG; h += 4) {
            mgops::PathCount x[4];
#pragma unroll
            for (int j = 0; j < 4; j++)
                x[j] = ((f[h + j] >> s) & 1u) ? a.sig[(size_t)u[h + j] * W + s] : mgops::pc_zero();
#pragma unroll
            for (int j = 0; j < 4; j++)
                if ((f[h + j] >> s) & 1u) acc = mgops::pc_add(acc, x[j], a.mode == M_EXT);
        }
        a.sig[(size_t)v * W + s] = acc;
        if (a.mode != M_EXT && acc.m >= mgops::PC_PLAIN_MAX) k->ovf = 1;
    }
    a.vis[v] |= newm;
    fnext[v] = newm;
    return true;
}

// level d -> d+1 over nrows rows (every row when dense, else the candidates)
template <bool TP, int M>
__device__ __forceinline__ void bb_pull_phase(const BbArgs &a, const BbCtl &c, int32_t nrows, LvlCnt *k)
{
    const int lane = mgd::lane();
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t *fcur = fm_of(a, c.cur);
    uint32_t *fnext = fm_of(a, c.cur ^ 1);
    if constexpr (TP) {
        // up to 32 rows per warp, one per lane; rows the thread path
        // declines are then pulled by the whole warp, one at a time
        const int vpw = entries_per_warp(nrows, nwarps, 32);
        for (int32_t base = gwarp * vpw; base < nrows; base += nwarps * vpw) {
            const int32_t i = base + lane;
            int32_t v = 0;
            uint32_t want = 0;
            bool deferred = false;
            if (lane < vpw && i < nrows) {
                v = c.dense ? i : a.cand[i];
                want = ~a.vis[v] & c.gmask;
                uint32_t reached;
                if (want) deferred = !pull_row_thread(a, fcur, fnext, v, want, &reached, k);
            }
            unsigned dm = __ballot_sync(0xffffffffu, deferred);
            while (dm) {
                const int j = __ffs(dm) - 1;
                dm &= dm - 1;
                const int32_t vj = __shfl_sync(0xffffffffu, v, j);
                const uint32_t wj = __shfl_sync(0xffffffffu, want, j);
                const int32_t b = __ldg(&a.trow[vj]), e = __ldg(&a.trow[vj + 1]);
                if (e - b > a.heavy_deg) continue;  // chunk path below
                uint32_t newm;
                const auto acc = pull_span<M>(a, fcur, c.d, b, e, wj, newm);
                if (newm) settle_row<M>(a, fnext, c.d, vj, newm, acc, k);
            }
        }
    } else {
        for (int32_t i = gwarp; i < nrows; i += nwarps) {  // a warp per row
            const int32_t v = c.dense ? i : a.cand[i];
            const uint32_t want = ~a.vis[v] & c.gmask;
            if (want == 0) continue;
            const int32_t b = __ldg(&a.trow[v]), e = __ldg(&a.trow[v + 1]);
            if (e - b > a.heavy_deg) continue;  // chunk path below
            uint32_t newm;
            const auto acc = pull_span<M>(a, fcur, c.d, b, e, want, newm);
            if (newm) settle_row<M>(a, fnext, c.d, v, newm, acc, k);
        }
    }
    for (int32_t ch = gwarp; ch < a.nhchunks; ch += nwarps) {
        const int32_t v = __ldg(&a.hchunk[3 * ch]), b = __ldg(&a.hchunk[3 * ch + 1]), e = __ldg(&a.hchunk[3 * ch + 2]);
        uint32_t want = ~a.vis[v] & c.gmask;
        if (!c.dense && !mgd::bm_test(a.cbm, v)) want = 0;
        uint32_t newm = 0;
        typename SumOf<M>::T acc{};
        if (want) acc = pull_span<M>(a, fcur, c.d, b, e, want, newm);
        if (newm) reinterpret_cast<typename SumOf<M>::T *>(a.hpart)[(size_t)ch * W + lane] = acc;
        if (lane == 0) a.hmask[ch] = newm;
    }
}

template <int M>
__device__ __forceinline__ void bb_heavy_phase(const BbArgs &a, const BbCtl &c, LvlCnt *k)
{
    const int lane = mgd::lane();
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    uint32_t *fnext = fm_of(a, c.cur ^ 1);
    for (int32_t i = gwarp; i < a.nhrows; i += nwarps) {
        const int32_t v = __ldg(&a.hrows[i]), k0 = __ldg(&a.hrow_chunk[i]), k1 = __ldg(&a.hrow_chunk[i + 1]);
        uint32_t newm = 0;
        typename SumOf<M>::T acc{};
        const auto *part = reinterpret_cast<const typename SumOf<M>::T *>(a.hpart);
        for (int32_t ch = k0; ch < k1; ch++) {
            const uint32_t hm = a.hmask[ch];
            newm |= hm;
            if (!((hm >> lane) & 1u)) continue;
            if constexpr (M == M_INT) acc += part[(size_t)ch * W + lane];
            else acc = mgops::pc_add(acc, part[(size_t)ch * W + lane], M == M_EXT);
        }
        if (newm) settle_row<M>(a, fnext, c.d, v, newm, acc, k);
    }
}

// Archives level d+1 (entries from off_d1 on), clears level d's masks
// (entries [off_d, off_d1)), counts into *k
__device__ __forceinline__ void bb_compact_phase(const BbArgs &a, const BbCtl &c, int32_t off_d, int32_t off_d1,
                                                 int32_t nrows, LvlCnt *k)
{
    const int lane = mgd::lane();
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const int gwarp = gtid >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    uint32_t *fcur = fm_of(a, c.cur);
    const uint32_t *fnext = fm_of(a, c.cur ^ 1);
    // the old frontier's masks (every reader of level d has finished)
    for (int32_t i = off_d + gtid; i < off_d1; i += gridDim.x * blockDim.x) fcur[a.arch[i]] = 0;
    const int32_t base_out = off_d1;
    for (int32_t base = gwarp * 32; base < nrows; base += nwarps * 32) {
        const int32_t i = base + lane;
        int32_t v = -1;
        uint32_t msk = 0;
        if (i < nrows) {
            v = c.dense ? i : a.cand[i];
            if (!c.dense) atomicAnd(&a.cbm[v >> 5], ~(1u << (v & 31)));
            msk = fnext[v];
        }
        const bool pred = msk != 0;
        int32_t deg = 0;
        if (pred) deg = __ldg(&a.row[v + 1]) - __ldg(&a.row[v]);
        const int slot = mgd::warp_append(&k->nnew, pred);
        if (pred) {
            const size_t at = (size_t)base_out + (size_t)slot;
            if (at < a.cap) {
                a.arch[at] = v;
                a.amask[at] = msk;
            } else {
                k->status = 2;
            }
            if (deg > MARK_HEAVY) a.fheavy[atomicAdd(&k->nfh_build, 1)] = v;
        }
        const unsigned long long s = warp_sum_u64((unsigned long long)deg);
        if (lane == 0 && s) atomicAdd(&k->nfe, s);
    }
}

// ---------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------
// Backward start at the deepest level L: the masks of levels L and L-1
// into their buffers (all three are zero after the forward sweep).
__device__ __forceinline__ void bbb_start_phase(const BbArgs &a, int32_t L)
{
    const int32_t stride = gridDim.x * blockDim.x;
    for (int32_t l = L - 1; l <= L; l++) {
        uint32_t *buf = fmb_of(a, l);
        for (int32_t i = a.off[l] + blockIdx.x * blockDim.x + threadIdx.x; i < a.off[l + 1]; i += stride)
            buf[a.arch[i]] = a.amask[i];
    }
}

template <int M>
using QT = typename std::conditional<M == M_EXT, double, float>::type;

// q of level L's vertices
template <int M>
__device__ __forceinline__ QT<M> *q_of(const BbArgs &a, int32_t L)
{
    if constexpr (M == M_INT) return a.qp[L & 1];
    else return reinterpret_cast<QT<M> *>(a.q);
}

// successor v's term for lane s of an entry whose count has scale ku
template <int M>
__device__ __forceinline__ QT<M> back_term(const BbArgs &a, int32_t L, int32_t v, int s, int32_t ku)
{
    QT<M> t = q_of<M>(a, L + 1)[(size_t)v * W + s];
    if (M == M_EXT) {
        const int32_t dk = ku - a.sig[(size_t)v * W + s].k;
        if (dk != 0) t *= (QT<M>)mgops::pc_scale(dk);   // (one level in hundreds)
    }
    return t;
}

// successors' q summed for the sources in `want`: out-edges [b, e); ku is
// this lane's scale of the entry's path count
template <int M>
__device__ __forceinline__ QT<M> back_span(const BbArgs &a, const uint32_t *nxt, int32_t L, const int32_t *col,
                                           int32_t b, int32_t e, uint32_t want, int32_t ku)
{
    const int lane = mgd::lane();
    QT<M> acc = 0;
    for (int32_t base = b; base < e; base += 32) {
        const int32_t p = base + lane;
        int32_t v = 0;
        uint32_t f = 0;
        if (p < e) {
            v = __ldcs(&col[p]);
            f = nxt[v] & want;
        }
        unsigned hits = __ballot_sync(0xffffffffu, f != 0);
        while (hits) {
            const int j = __ffs(hits) - 1;
            hits &= hits - 1;
            const int32_t vj = __shfl_sync(0xffffffffu, v, j);
            const uint32_t fj = __shfl_sync(0xffffffffu, f, j);
            if ((fj >> lane) & 1u) acc += back_term<M>(a, L, vj, lane, ku);
        }
    }
    return acc;
}

// lane's scale of u's path count (0 in plain mode)
template <int M>
__device__ __forceinline__ int32_t lane_scale(const BbArgs &a, int32_t u, uint32_t msk)
{
    const int lane = mgd::lane();
    return (M == M_EXT && ((msk >> lane) & 1u)) ? a.sig[(size_t)u * W + lane].k : 0;
}

// delta = count * sum and q = (1 + delta) / count of one (vertex, source);
// as if formed in FP64 and rounded once.  Integer counts below 2^24 (nearly
// all) stay in FP32: the product of two FP32 numbers rounds once, and the
// quotient is corrected by its remainder (1 + delta as an exact pair).
template <int M>
__device__ __forceinline__ float back_delta(typename SumOf<M>::T count, QT<M> s, QT<M> &q)
{
    if constexpr (M == M_INT) {
        if (count < (1ull << 24)) {
            const float sg = (float)(uint32_t)count;
            const float dv = sg * s;
            float hi = 1.0f, lo = 0.0f;
            pair_add(hi, lo, dv);
            const float q0 = __fdiv_rn(hi, sg);
            q = q0 + __fdividef(fmaf(-q0, sg, hi) + lo, sg);
            return dv;
        }
        const double sg = (double)count;
        const float dv = (float)(sg * (double)s);
        q = (float)((1.0 + (double)dv) / sg);
        return dv;
    } else {
        const float dv = (float)(count.m * (double)s);
        q = (QT<M>)((1.0 + (double)dv) / count.m);
        return dv;
    }
}

// the (vertex, source) count at level L
template <int M>
__device__ __forceinline__ typename SumOf<M>::T count_at(const BbArgs &a, int32_t L, int32_t u, int s)
{
    if constexpr (M == M_INT) return a.cnt[L & 1][(size_t)u * W + s];
    else return a.sig[(size_t)u * W + s];
}

template <int M>
__device__ __forceinline__ void back_finish(const BbArgs &a, int32_t L, int32_t u, uint32_t msk, QT<M> s)
{
    const int lane = mgd::lane();
    float hi = 0.0f, lo = 0.0f;
    if ((msk >> lane) & 1u) {
        const float dv = back_delta<M>(count_at<M>(a, L, u, lane), s, q_of<M>(a, L)[(size_t)u * W + lane]);
        if (__ldg(&a.src[lane]) != u) hi = dv;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float h = __shfl_xor_sync(0xffffffffu, hi, o), l = __shfl_xor_sync(0xffffffffu, lo, o);
        pair_add(hi, lo, h);
        lo += l;
    }
    if (lane == 0) score_add(a, u, hi, lo);
}

// One thread, one level-L entry (u, msk) with at most TDEG out-edges and
// at most TBITS sources: back_span and back_finish for each source of the
// entry in turn (the same sums in the same edge order; the entry's score
// contributions are added in source order).
template <int M>
__device__ __forceinline__ bool back_entry_thread(const BbArgs &a, const uint32_t *nxt, int32_t L, int32_t u,
                                                  uint32_t msk, int32_t b, int32_t e)
{
    if (__popc(msk) > TBITS) return false;
    if (e - b > TDEG) return false;
    int32_t v[TDEG];
    uint32_t f[TDEG];
#pragma unroll
    for (int j = 0; j < TDEG; j++) v[j] = b + j < e ? __ldg(&a.col[b + j]) : -1;
#pragma unroll
    for (int j = 0; j < TDEG; j++) f[j] = v[j] >= 0 ? nxt[v[j]] : 0u;
    float hi = 0.0f, lo = 0.0f;
    uint32_t mm = msk;
    while (mm) {
        const int s = __ffs(mm) - 1;
        mm &= mm - 1;
        const mgops::PathCount su = a.sig[(size_t)u * W + s];
        QT<M> t[TDEG], acc = 0;
#pragma unroll
        for (int j = 0; j < TDEG; j++) t[j] = ((f[j] >> s) & 1u) ? back_term<M>(a, L, v[j], s, su.k) : (QT<M>)0;
#pragma unroll
        for (int j = 0; j < TDEG; j++)
            if ((f[j] >> s) & 1u) acc += t[j];
        const float dv = back_delta<M>(su, acc, q_of<M>(a, L)[(size_t)u * W + s]);
        if (__ldg(&a.src[s]) != u) pair_add(hi, lo, dv);
    }
    score_add(a, u, hi, lo);
    return true;
}

// backward level L: every level-L entry from its level-(L+1) successors
template <bool TP, int M>
__device__ __forceinline__ void bbb_pull_phase(const BbArgs &a, int32_t L)
{
    const int lane = mgd::lane();
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t *cur = fmb_of(a, L);
    const uint32_t *nxt = fmb_of(a, L + 1);
    if constexpr (TP) {
        const int32_t lo = a.off[L], hi = a.off[L + 1];
        // up to 32 entries per warp, one per lane; entries the thread path
        // declines are then handled by the whole warp (lane per source)
        const int vpw = entries_per_warp(hi - lo, nwarps, 32);
        for (int32_t base = lo + gwarp * vpw; base < hi; base += nwarps * vpw) {
            const int32_t i = base + lane;
            int32_t u = 0;
            uint32_t msk = 0;
            bool deferred = false;
            if (lane < vpw && i < hi) {
                u = a.arch[i];
                msk = a.amask[i];
                deferred = !back_entry_thread<M>(a, nxt, L, u, msk, __ldg(&a.row[u]), __ldg(&a.row[u + 1]));
            }
            unsigned dm = __ballot_sync(0xffffffffu, deferred);
            while (dm) {
                const int j = __ffs(dm) - 1;
                dm &= dm - 1;
                const int32_t uj = __shfl_sync(0xffffffffu, u, j);
                const uint32_t mj = __shfl_sync(0xffffffffu, msk, j);
                const int32_t b = __ldg(&a.row[uj]), e = __ldg(&a.row[uj + 1]);
                if (e - b > a.heavy_deg) continue;  // chunk path below
                const QT<M> sj = back_span<M>(a, nxt, L, a.col, b, e, mj, lane_scale<M>(a, uj, mj));
                back_finish<M>(a, L, uj, mj, sj);
            }
        }
    } else {
        for (int32_t i = a.off[L] + gwarp; i < a.off[L + 1]; i += nwarps) {  // a warp per entry
            const int32_t u = a.arch[i];
            const uint32_t msk = a.amask[i];
            const int32_t b = __ldg(&a.row[u]), e = __ldg(&a.row[u + 1]);
            if (e - b > a.heavy_deg) continue;  // chunk path below
            const QT<M> s = back_span<M>(a, nxt, L, a.col, b, e, msk, lane_scale<M>(a, u, msk));
            back_finish<M>(a, L, u, msk, s);
        }
    }
    // heavy rows: the in-row chunks double as out-row chunks (symmetric graphs)
    QT<M> *hp = reinterpret_cast<QT<M> *>(a.hpart);
    for (int32_t ch = gwarp; ch < a.nhchunks; ch += nwarps) {
        const int32_t u = __ldg(&a.hchunk[3 * ch]);
        const uint32_t msk = cur[u];
        if (msk == 0) continue;
        hp[(size_t)ch * W + lane] = back_span<M>(a, nxt, L, a.tcol, __ldg(&a.hchunk[3 * ch + 1]), __ldg(&a.hchunk[3 * ch + 2]), msk,
                                                   lane_scale<M>(a, u, msk));
    }
}

// heavy rows: chunk partials folded in chunk order (graphs with heavy rows)
template <int M>
__device__ __forceinline__ void bbb_heavy_phase(const BbArgs &a, int32_t L)
{
    const int lane = mgd::lane();
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t *cur = fmb_of(a, L);
    const QT<M> *hp = reinterpret_cast<const QT<M> *>(a.hpart);
    for (int32_t i = gwarp; i < a.nhrows; i += nwarps) {
        const int32_t u = __ldg(&a.hrows[i]);
        const uint32_t msk = cur[u];
        if (msk == 0) continue;
        QT<M> s = 0;
        for (int32_t k = __ldg(&a.hrow_chunk[i]); k < __ldg(&a.hrow_chunk[i + 1]); k++) s += hp[(size_t)k * W + lane];
        back_finish<M>(a, L, u, msk, s);
    }
}

// End of backward level L: level L+1's masks are no longer read (cleared),
// level L-1's go into their buffer ((L-1) % 3, cleared at the end of level
// L+1)
__device__ __forceinline__ void bbb_next_phase(const BbArgs &a, int32_t L)
{
    const int32_t stride = gridDim.x * blockDim.x;
    const int32_t gtid = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t *nxt = fmb_of(a, L + 1);
    for (int32_t i = a.off[L + 1] + gtid; i < a.off[L + 2]; i += stride) nxt[a.arch[i]] = 0;
    if (L >= 2) {
        uint32_t *prv = fmb_of(a, L - 1);
        for (int32_t i = a.off[L - 1] + gtid; i < a.off[L]; i += stride) prv[a.arch[i]] = a.amask[i];
    }
}


// ---------------------------------------------------------------------------
// flat sweeps: graphs without heavy rows (no vertex of 128 edges), whole
// sweeps in one persistent launch.  Masks of level l lie in fm[l % 3] forward
// too.
// ---------------------------------------------------------------------------
// An entry a thread, 32 a warp, consecutive warps of entries on different
// SMs: GB300's FP64 pipe takes a warp instruction in the same time whether
// one lane is active or all (extended counts are FP64), and an entry spread
// to a warp of its own kept it busy for 16 us a level (7,700 entries).
__device__ __forceinline__ int flat_warp() { return (int)((threadIdx.x >> 5) * gridDim.x + blockIdx.x); }

// Level d -> d+1 over nrows rows, the reached rows archived as they settle
// (level d+1's entries from off_d1 on), their candidate bits and level d-1's
// masks cleared on the way: nobody reads either in this phase.
template <int M>
__device__ __forceinline__ void bb_flat_phase(const BbArgs &a, const BbCtl &c, int32_t nrows, int32_t off_p,
                                              int32_t off_d, int32_t off_d1, LvlCnt *k)
{
    const int lane = mgd::lane();
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gwarp = flat_warp();
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t *fcur = fmb_of(a, c.d);
    uint32_t *fnext = fmb_of(a, c.d + 1), *fold = fmb_of(a, c.d + 2);
    for (int32_t i = off_p + gtid; i < off_d; i += gridDim.x * blockDim.x) fold[__ldcg(&a.arch[i])] = 0;
    unsigned long long nfe = 0;
    for (int32_t base = gwarp * 32; base < nrows; base += nwarps * 32) {
        const int32_t i = base + lane;
        int32_t v = 0;
        uint32_t want = 0, reached = 0;
        bool deferred = false;
        if (i < nrows) {
            v = c.dense ? i : __ldcg(&a.cand[i]);
            if (!c.dense) atomicAnd(&a.cbm[v >> 5], ~(1u << (v & 31)));
            want = ~a.vis[v] & c.gmask;
            if (want) deferred = !pull_row_thread(a, fcur, fnext, v, want, &reached, k);
            if (deferred) reached = 0;
        }
        unsigned dm = __ballot_sync(0xffffffffu, deferred);
        while (dm) {
            const int j = __ffs(dm) - 1;
            dm &= dm - 1;
            const int32_t vj = __shfl_sync(0xffffffffu, v, j);
            const uint32_t wj = __shfl_sync(0xffffffffu, want, j);
            uint32_t newm;
            const auto acc = pull_span<M>(a, fcur, c.d, __ldg(&a.trow[vj]), __ldg(&a.trow[vj + 1]), wj, newm);
            if (newm) settle_row<M>(a, fnext, c.d, vj, newm, acc, k);
            if (lane == j) reached = newm;
        }
        const unsigned m = __ballot_sync(0xffffffffu, reached != 0);
        if (m == 0) continue;
        int at = 0;
        if (lane == 0) at = atomicAdd(&k->nnew, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
        if (reached) {
            const size_t o = (size_t)off_d1 + (size_t)at;
            if (o < a.cap) {
                a.arch[o] = v;
                a.amask[o] = reached;
            } else {
                k->status = 2;
            }
            nfe += (unsigned long long)(__ldg(&a.row[v + 1]) - __ldg(&a.row[v]));
        }
    }
    nfe = warp_sum_u64(nfe);
    if (lane == 0 && nfe) atomicAdd(&k->nfe, nfe);
}

// A thread's first entry of a backward level, loaded ahead of the barrier
// that opens the level
struct FlatEntry {
    int32_t u, b, e;
    uint32_t msk;
};

__device__ __forceinline__ FlatEntry flat_load(const BbArgs &a, int32_t L)
{
    FlatEntry x{0, 0, 0, 0u};
    if (L < 1) return x;
    const int32_t lo = a.off[L], hi = a.off[L + 1];
    const int32_t i = lo + flat_warp() * 32 + mgd::lane();
    if (i < hi) {
        x.u = a.arch[i];
        x.msk = a.amask[i];
        x.b = __ldg(&a.row[x.u]);
        x.e = __ldg(&a.row[x.u + 1]);
    }
    return x;
}

// Backward level L; the entries' own masks go into fm[L % 3] for level L-1,
// level L+2's are cleared (levels up to Ltop)
template <int M>
__device__ __forceinline__ void bbb_flat_phase(const BbArgs &a, int32_t L, int32_t Ltop, FlatEntry x)
{
    const int lane = mgd::lane();
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gwarp = flat_warp();
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    uint32_t *cur = fmb_of(a, L);
    const uint32_t *nxt = fmb_of(a, L + 1);
    const int32_t lo = a.off[L], hi = a.off[L + 1];
    for (int32_t base = lo + gwarp * 32; base < hi; base += nwarps * 32) {
        if (base != lo + gwarp * 32) {
            x = FlatEntry{0, 0, 0, 0u};
            if (base + lane < hi) {
                x.u = a.arch[base + lane];
                x.msk = a.amask[base + lane];
                x.b = __ldg(&a.row[x.u]);
                x.e = __ldg(&a.row[x.u + 1]);
            }
        }
        const bool deferred = x.msk != 0 && !back_entry_thread<M>(a, nxt, L, x.u, x.msk, x.b, x.e);
        if (x.msk) cur[x.u] = x.msk;
        unsigned dm = __ballot_sync(0xffffffffu, deferred);
        while (dm) {
            const int j = __ffs(dm) - 1;
            dm &= dm - 1;
            const int32_t uj = __shfl_sync(0xffffffffu, x.u, j), bj = __shfl_sync(0xffffffffu, x.b, j),
                          ej = __shfl_sync(0xffffffffu, x.e, j);
            const uint32_t mj = __shfl_sync(0xffffffffu, x.msk, j);
            const QT<M> sj = back_span<M>(a, nxt, L, a.col, bj, ej, mj, lane_scale<M>(a, uj, mj));
            back_finish<M>(a, L, uj, mj, sj);
        }
    }
    if (L + 2 <= Ltop) {
        uint32_t *old = fmb_of(a, L + 2);
        for (int32_t i = a.off[L + 2] + gtid; i < a.off[L + 3]; i += gridDim.x * blockDim.x) old[a.arch[i]] = 0;
    }
}

// ---------------------------------------------------------------------------
// mask-free levels (M_INT): eight lanes a row, four sources (16 bytes) a lane
// ---------------------------------------------------------------------------
constexpr int GL = 8;              // lanes a row
constexpr int32_t GCHUNK = 256;    // rows above this many edges go in chunks

// Sum over the columns [b, e) of the rows val[col][..] (this lane's four
// sources) through add(t[8]).  All lanes of the warp call (a group without
// work passes b == e) and run over the longest of their ranges; the next
// eight ids are loaded ahead of the current gathers.
template <class V, class Add>
__device__ __forceinline__ void gather_rows(const V *__restrict__ val, const int32_t *__restrict__ col, int32_t b,
                                            int32_t e, Add add)
{
    const int gl = threadIdx.x & (GL - 1);
    const int32_t rounds = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)((e - b + GL - 1) / GL));
    int32_t id = b + gl < e ? __ldcs(&col[b + gl]) : -1;
    for (int32_t r = 0; r < rounds; r++) {
        V t[GL];
#pragma unroll
        for (int j = 0; j < GL; j++) {
            const int32_t u = __shfl_sync(0xffffffffu, id, j, GL);
            t[j] = u >= 0 ? val[(size_t)u * GL + gl] : V{};
        }
        b += GL;
        id = b + gl < e ? __ldcs(&col[b + gl]) : -1;
        add(t);
    }
}

struct Sum4 {
    unsigned long long x = 0, y = 0, z = 0, w = 0;
    __device__ __forceinline__ void add(const uint4 (&t)[GL])
    {
        x += ((t[0].x + t[1].x) + (t[2].x + t[3].x)) + ((t[4].x + t[5].x) + (t[6].x + t[7].x));
        y += ((t[0].y + t[1].y) + (t[2].y + t[3].y)) + ((t[4].y + t[5].y) + (t[6].y + t[7].y));
        z += ((t[0].z + t[1].z) + (t[2].z + t[3].z)) + ((t[4].z + t[5].z) + (t[6].z + t[7].z));
        w += ((t[0].w + t[1].w) + (t[2].w + t[3].w)) + ((t[4].w + t[5].w) + (t[6].w + t[7].w));
    }
};

// row v's new counts (this lane's four sums): stored for the sources that
// had not reached v, the row's masks updated (all eight lanes of the row's
// group call)
__device__ __forceinline__ void gather_settle(const BbArgs &a, uint32_t *fnext, int32_t d, int32_t v, uint32_t want,
                                              const Sum4 &s, unsigned gmask, LvlCnt *cnt)
{
    const int gl = threadIdx.x & (GL - 1);
    const unsigned long long x[4] = {s.x, s.y, s.z, s.w};
    uint32_t m = 0;
    uint32_t *out = a.cnt[(d + 1) & 1] + (size_t)v * W + gl * 4;
    bool over = false;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t bit = 1u << (gl * 4 + k);
        if (x[k] != 0 && (want & bit)) {
            m |= bit;
            out[k] = (uint32_t)x[k];
            over |= x[k] >= INT_LIMIT;
        }
    }
    if (over) cnt->ovf = 1;
    const uint32_t newm = __reduce_or_sync(gmask, m);
    if (gl == 0 && newm) {
        a.vis[v] |= newm;
        fnext[v] = newm;
    }
}

__device__ __forceinline__ unsigned group_mask() { return 0xffu << (mgd::lane() & ~(GL - 1)); }

__device__ __forceinline__ void bb_gather_phase(const BbArgs &a, const BbCtl &c, LvlCnt *k)
{
    constexpr int RPW = 32 / GL;
    const int gl = threadIdx.x & (GL - 1), grp = mgd::lane() / GL;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint4 *val = reinterpret_cast<const uint4 *>(a.cnt[c.d & 1]);
    uint32_t *fnext = fm_of(a, c.cur ^ 1);
    const unsigned gm = group_mask();
    ulonglong2 *part = reinterpret_cast<ulonglong2 *>(a.gpart);
    for (int32_t c0 = gwarp * RPW; c0 < a.ngchunks; c0 += nwarps * RPW) {
        const int32_t ch = c0 + grp;
        int32_t b = 0, e = 0;
        if (ch < a.ngchunks && (~a.vis[__ldg(&a.gchunk[3 * ch])] & c.gmask)) {
            b = __ldg(&a.gchunk[3 * ch + 1]);
            e = __ldg(&a.gchunk[3 * ch + 2]);
        }
        Sum4 s;
        gather_rows(val, a.tcol, b, e, [&](const uint4 (&t)[GL]) { s.add(t); });
        if (e > b) {
            part[(size_t)ch * 16 + gl * 2] = make_ulonglong2(s.x, s.y);
            part[(size_t)ch * 16 + gl * 2 + 1] = make_ulonglong2(s.z, s.w);
        }
    }
    // the next row's mask and offsets are loaded ahead of this row's gathers
    int32_t v = gwarp * RPW + grp;
    uint32_t want = v < a.n ? ~a.vis[v] & c.gmask : 0u;
    int32_t b = v < a.n ? __ldg(&a.trow[v]) : 0, e = v < a.n ? __ldg(&a.trow[v + 1]) : 0;
    for (int32_t v0 = gwarp * RPW; v0 < a.n; v0 += nwarps * RPW) {
        const int32_t vn = v + nwarps * RPW;
        const uint32_t wn = vn < a.n ? ~a.vis[vn] & c.gmask : 0u;
        const int32_t bn = vn < a.n ? __ldg(&a.trow[vn]) : 0, en = vn < a.n ? __ldg(&a.trow[vn + 1]) : 0;
        const bool row = want != 0 && e - b <= GCHUNK;
        Sum4 s;
        gather_rows(val, a.tcol, b, row ? e : b, [&](const uint4 (&t)[GL]) { s.add(t); });
        if (row) gather_settle(a, fnext, c.d, v, want, s, gm, k);
        v = vn;
        want = wn;
        b = bn;
        e = en;
    }
}

// rows above GCHUNK edges: their chunks' sums
__device__ __forceinline__ void bb_gather_heavy_phase(const BbArgs &a, const BbCtl &c, LvlCnt *cnt)
{
    constexpr int RPW = 32 / GL;
    const int gl = threadIdx.x & (GL - 1), grp = mgd::lane() / GL;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    uint32_t *fnext = fm_of(a, c.cur ^ 1);
    const ulonglong2 *part = reinterpret_cast<const ulonglong2 *>(a.gpart);
    for (int32_t i = gwarp; i < a.ngrows; i += nwarps) {
        const int32_t v = __ldg(&a.grows[i]);
        const uint32_t want = ~a.vis[v] & c.gmask;
        if (want == 0) continue;   // warp-uniform
        Sum4 s;
        for (int32_t k = __ldg(&a.grow_chunk[i]) + grp, k1 = __ldg(&a.grow_chunk[i + 1]); k < k1; k += RPW) {
            const ulonglong2 p = __ldcs(&part[(size_t)k * 16 + gl * 2]), r = __ldcs(&part[(size_t)k * 16 + gl * 2 + 1]);
            s.x += p.x;
            s.y += p.y;
            s.z += r.x;
            s.w += r.y;
        }
#pragma unroll
        for (int o = GL; o < 32; o <<= 1) {
            s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
            s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
            s.z += __shfl_xor_sync(0xffffffffu, s.z, o);
            s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
        }
        if (grp == 0) gather_settle(a, fnext, c.d, v, want, s, 0xffu, cnt);
    }
}

__device__ __forceinline__ bool back_gathers(const BbArgs &a, int32_t L)
{
    return a.mode == M_INT && __ldcg(&a.lnfe[L]) * GATHER_BACK > (unsigned long long)a.m;
}

__device__ __forceinline__ void f4_sum8(float4 &acc, const float4 (&t)[GL])
{
    acc.x += ((t[0].x + t[1].x) + (t[2].x + t[3].x)) + ((t[4].x + t[5].x) + (t[6].x + t[7].x));
    acc.y += ((t[0].y + t[1].y) + (t[2].y + t[3].y)) + ((t[4].y + t[5].y) + (t[6].y + t[7].y));
    acc.z += ((t[0].z + t[1].z) + (t[2].z + t[3].z)) + ((t[4].z + t[5].z) + (t[6].z + t[7].z));
    acc.w += ((t[0].w + t[1].w) + (t[2].w + t[3].w)) + ((t[4].w + t[5].w) + (t[6].w + t[7].w));
}

// entry (u, msk) of level L from its successors' sums: q of this lane's
// sources and the row's score (the eight lanes of the group call)
__device__ __forceinline__ void gather_finish(const BbArgs &a, int32_t L, int32_t u, uint32_t msk, float4 sum,
                                              const int4 &src, unsigned gm)
{
    const int gl = threadIdx.x & (GL - 1);
    const uint4 c4 = *reinterpret_cast<const uint4 *>(a.cnt[L & 1] + (size_t)u * W + gl * 4);
    const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
    const float s[4] = {sum.x, sum.y, sum.z, sum.w};
    const int32_t sr[4] = {src.x, src.y, src.z, src.w};
    float *out = a.qp[L & 1] + (size_t)u * W + gl * 4;
    float hi = 0.0f, lo = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; k++)
        if ((msk >> (gl * 4 + k)) & 1u) {
            const float dv = back_delta<M_INT>(c[k], s[k], out[k]);
            if (sr[k] != u) pair_add(hi, lo, dv);
        }
#pragma unroll
    for (int o = GL / 2; o > 0; o >>= 1) {
        const float h = __shfl_xor_sync(gm, hi, o), l = __shfl_xor_sync(gm, lo, o);
        pair_add(hi, lo, h);
        lo += l;
    }
    if (gl == 0) score_add(a, u, hi, lo);
}

__device__ __forceinline__ int4 lane_sources(const BbArgs &a)
{
    return *reinterpret_cast<const int4 *>(a.src + (threadIdx.x & (GL - 1)) * 4);
}

__device__ __forceinline__ void bbb_gather_phase(const BbArgs &a, int32_t L)
{
    constexpr int RPW = 32 / GL;
    const int gl = threadIdx.x & (GL - 1), grp = mgd::lane() / GL;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const float4 *val = reinterpret_cast<const float4 *>(a.qp[(L + 1) & 1]);
    const uint32_t *cur = fmb_of(a, L);
    const unsigned gm = group_mask();
    float4 *part = reinterpret_cast<float4 *>(a.gpart);
    for (int32_t c0 = gwarp * RPW; c0 < a.ngchunks; c0 += nwarps * RPW) {
        const int32_t ch = c0 + grp;
        int32_t b = 0, e = 0;
        if (ch < a.ngchunks && cur[__ldg(&a.gchunk[3 * ch])]) {
            b = __ldg(&a.gchunk[3 * ch + 1]);
            e = __ldg(&a.gchunk[3 * ch + 2]);
        }
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        gather_rows(val, a.tcol, b, e, [&](const float4 (&t)[GL]) { f4_sum8(s, t); });
        if (e > b) part[(size_t)ch * GL + gl] = s;
    }
    const int4 src = lane_sources(a);
    const int32_t lo = a.off[L], hi = a.off[L + 1];
    int32_t i = lo + gwarp * RPW + grp;
    int32_t u = i < hi ? a.arch[i] : 0;
    uint32_t msk = i < hi ? a.amask[i] : 0u;
    int32_t b = __ldg(&a.trow[u]), e = __ldg(&a.trow[u + 1]);
    for (int32_t i0 = lo + gwarp * RPW; i0 < hi; i0 += nwarps * RPW) {
        const int32_t in = i + nwarps * RPW;
        const int32_t un = in < hi ? a.arch[in] : 0;
        const uint32_t mn = in < hi ? a.amask[in] : 0u;
        const bool row = msk != 0 && e - b <= GCHUNK;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        gather_rows(val, a.tcol, b, row ? e : b, [&](const float4 (&t)[GL]) { f4_sum8(s, t); });
        const int32_t bn = __ldg(&a.trow[un]), en = __ldg(&a.trow[un + 1]);
        if (row) gather_finish(a, L, u, msk, s, src, gm);
        i = in;
        u = un;
        msk = mn;
        b = bn;
        e = en;
    }
}

__device__ __forceinline__ void bbb_gather_heavy_phase(const BbArgs &a, int32_t L)
{
    constexpr int RPW = 32 / GL;
    const int gl = threadIdx.x & (GL - 1), grp = mgd::lane() / GL;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t *cur = fmb_of(a, L);
    const float4 *part = reinterpret_cast<const float4 *>(a.gpart);
    const int4 src = lane_sources(a);
    for (int32_t r = gwarp; r < a.ngrows; r += nwarps) {
        const int32_t u = __ldg(&a.grows[r]);
        const uint32_t msk = cur[u];
        if (msk == 0) continue;   // warp-uniform
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int32_t k = __ldg(&a.grow_chunk[r]) + grp, k1 = __ldg(&a.grow_chunk[r + 1]); k < k1; k += RPW) {
            const float4 p = __ldcs(&part[(size_t)k * GL + gl]);
            s.x += p.x;
            s.y += p.y;
            s.z += p.z;
            s.w += p.w;
        }
#pragma unroll
        for (int o = GL; o < 32; o <<= 1) {
            s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
            s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
            s.z += __shfl_xor_sync(0xffffffffu, s.z, o);
            s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
        }
        if (grp == 0) gather_finish(a, L, u, msk, s, src, 0xffu);
    }
}

}  // namespace mgbc

