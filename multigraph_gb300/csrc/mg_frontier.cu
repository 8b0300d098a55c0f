// mg_frontier.cu -- the built-in frontier operators (BFS, SSSP, the BC
// forward sweep) on the engine of mg_frontier_engine.cuh; the BC backward
// sweep; multi-source BC for directed graphs; their C ABI.
//
// MultiGraph_V_E_V_pull (process2.cu:263-325) becomes k_bc_back_levels.

#include "mg_frontier_engine.cuh"

namespace {

// BC backward: delta[v] = sigma[v] * sum_{w succ, level[w] = L} q[w],
// q[w] = (1 + delta[w]) / sigma[w]  (bc_phase1/2 of process2.cu:135-261 and
// process_fbc :5-132 in one pull form over the archived level lists).
// With path counts sigma = m * 2^(512 k), q is kept as (1 + delta) / m
// (FP64) and a successor's term is scaled by 2^(512 (k_v - k_w)).
// ----------------------------------------------------------------------------
struct BCtl {
    int32_t L0;       // deepest level; levels L0 .. 1 finalise their predecessors
    int32_t src;      // source of this sweep (excluded from the BC sum)
    int32_t hcnt[2];  // chunks of long entries listed at a level, by level parity
};

// q and the successor sums: FP32 with plain counts (below 2^100, so
// (1 + delta) / sigma stays a normal FP32 number); FP64 with extended counts,
// whose mantissas reach 2^512.
template <bool EXT>
using QT = typename std::conditional<EXT, double, float>::type;

template <bool EXT>
__global__ void k_bc_q_init(int32_t n, const mgops::PathCount *sigma, const int32_t *label, QT<EXT> *q, float *delta)
{
    for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        delta[v] = 0.0f;
        const double m = sigma[v].m;
        q[v] = (label[v] != mgops::UNSET && m > 0.0) ? (QT<EXT>)(1.0 / m) : (QT<EXT>)0;
    }
}

// delta and q of one vertex from its successors' sum
template <bool EXT>
__device__ __forceinline__ void bc_finish_vertex(int32_t v, QT<EXT> s, mgops::PathCount su, float *delta, QT<EXT> *q,
                                                 float *bc, int32_t src)
{
    float dv;
    if (!EXT && __double2hiint(su.m) < (1023 + 24) << 20) {
        // a count below 2^24 is exact in FP32: one rounding in the product,
        // and the quotient of the exact pair 1 + delta corrected by its
        // remainder -- as formed in FP64 and rounded, off GB300's FP64 pipe
        const float m = (float)su.m;
        dv = m * (float)s;
        const float hi = 1.0f + dv, bp = hi - 1.0f, lo = (1.0f - (hi - bp)) + (dv - bp);
        const float q0 = __fdiv_rn(hi, m);
        q[v] = (QT<EXT>)(q0 + __fdividef(fmaf(-q0, m, hi) + lo, m));
    } else {
        dv = (float)(su.m * (double)s);
        q[v] = (QT<EXT>)((1.0 + (double)dv) / su.m);
    }
    delta[v] = dv;
    if (bc && v != src) bc[v] += dv;
}

// Backward sweep of graphs with heavy vertices: few, large levels.  q is kept
// in two arrays by level parity, zero where not yet formed: a level-l entry's
// neighbours in array (l + 1) & 1 are its successors (level l + 1) and
// vertices of level l - 1, whose q is still zero, so one gather an edge does
// (the label test took a second, dependent one).  Entries of up to BACK_CHUNK
// edges take eight lanes, four entries a warp, four gathers a lane in flight;
// the others a warp per BACK_CHUNK-edge chunk, the last chunk of an entry
// adding the partial sums up in order.  One warp for any entry of up to 4,096
// edges took a level of R-MAT 20 up to 3 ms.  Backward sweep: R-MAT 16 154 ->
// 49 us, R-MAT 20 1,200 to 4,000 -> 215, R-MAT 22 2,300 -> 800.
constexpr int32_t BACK_CHUNK = 256;

struct BackArgs {
    int32_t *lvl_off;
    void *q[2];
    int4 *item;           // chunks of the level's long entries: vertex, begin, end, the entry's first chunk
    int32_t *arrive;      // [items] chunks finished, at the entry's first chunk (zero between levels)
    void *part;           // [items] partial sums
    int32_t *nitems;      // [2] by level parity
};

template <bool EXT>
__global__ void __launch_bounds__(PTHREADS, 1) k_bc_back_heavy(Args a, BCtl *bc_ctl, BackArgs k, float *delta,
                                                               float *bcacc)
{
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ int4 s_b;
    if (threadIdx.x == 0) s_b = __ldcg(reinterpret_cast<const int4 *>(bc_ctl));
    __syncthreads();
    const int32_t L0 = s_b.x, src = s_b.y;
    const int lane = mgd::lane(), gl = lane & 7, grp = lane >> 3;
    const int32_t gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    QT<EXT> *part = reinterpret_cast<QT<EXT> *>(k.part);
    for (int32_t l = L0; l >= 0; l--) {
        QT<EXT> *qo = reinterpret_cast<QT<EXT> *>(k.q[l & 1]);
        const QT<EXT> *qi = reinterpret_cast<const QT<EXT> *>(k.q[(l + 1) & 1]);
        const int32_t lo = a.lvl_off[l], hi = a.lvl_off[l + 1];
        if (l == L0) {   // no successors
            for (int32_t i = lo + gwarp * 32 + lane; i < hi; i += nwarps * 32) {
                const int32_t u = a.queue[i];
                bc_finish_vertex<EXT>(u, (QT<EXT>)0, a.sigma[u], delta, qo, bcacc, src);
            }
            if (!mgd::grid_sync(a.bar, a.bar_err, a.bar_never)) return;
            continue;
        }
        // One gathered term: the successor's q, scaled to the entry's count.
        // A successor's count is at least the entry's, so only scales down:
        // a neighbour of a smaller scale is one level up, its q still zero,
        // and must not be multiplied by an infinite 2^(512 dk).
        auto term = [&](int32_t w, int32_t ku) {
            QT<EXT> t = qi[w];
            if (EXT) {
                const int32_t dk = ku - a.sigma[w].k;
                if (dk < 0) t *= (QT<EXT>)mgops::pc_scale(dk);
            }
            return t;
        };
        if (blockIdx.x == 0 && threadIdx.x == 0) k.nitems[(l + 1) & 1] = 0;
        int32_t *nitems = &k.nitems[l & 1];
        for (int32_t i0 = lo + gwarp * 4; i0 < hi; i0 += nwarps * 4) {
            const int32_t i = i0 + grp;
            int32_t u = 0, b = 0, e = 0;
            if (i < hi) {
                u = a.queue[i];
                b = __ldg(&a.row[u]);
                e = __ldg(&a.row[u + 1]);
            }
            // long entries to the chunk list (their groups' first lanes)
            const int32_t nc = e - b > BACK_CHUNK && gl == 0 ? (e - b - 1) / BACK_CHUNK + 1 : 0;
            if (__any_sync(FULL, nc > 0)) {
                int32_t base = 0;
                if (nc > 0) base = atomicAdd(nitems, nc);
                unsigned lm = __ballot_sync(FULL, nc > 0);
                while (lm) {
                    const int j = __ffs(lm) - 1;
                    lm &= lm - 1;
                    const int32_t uj = __shfl_sync(FULL, u, j), bj = __shfl_sync(FULL, b, j), ej = __shfl_sync(FULL, e, j),
                                  nj = __shfl_sync(FULL, nc, j), pj = __shfl_sync(FULL, base, j);
                    for (int32_t c = lane; c < nj; c += 32)
                        k.item[pj + c] = make_int4(uj, bj + c * BACK_CHUNK, bj + min(ej - bj, (c + 1) * BACK_CHUNK), pj);
                }
            }
            const bool row = i < hi && e - b <= BACK_CHUNK;
            const mgops::PathCount su = row ? a.sigma[u] : mgops::pc_zero();
            const int32_t len = row ? e - b : 0;
            const int32_t rounds = (int32_t)__reduce_max_sync(FULL, (unsigned)((len + 31) >> 5));
            QT<EXT> acc = 0;
            for (int32_t r = 0; r < rounds; r++) {
                QT<EXT> t[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int32_t p = r * 32 + j * 8 + gl;
                    t[j] = p < len ? term(__ldcs(&a.col[b + p]), su.k) : (QT<EXT>)0;
                }
                acc += (t[0] + t[1]) + (t[2] + t[3]);
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
            if (row && gl == 0) bc_finish_vertex<EXT>(u, acc, su, delta, qo, bcacc, src);
        }
        if (!mgd::grid_sync(a.bar, a.bar_err, a.bar_never)) return;
        const int32_t ni = __ldcg(nitems);
        if (ni == 0) continue;   // (the same for every block: nobody adds to it in this phase)
        for (int32_t c = gwarp; c < ni; c += nwarps) {
            const int4 it = __ldcg(&k.item[c]);
            const mgops::PathCount su = a.sigma[it.x];
            QT<EXT> t[BACK_CHUNK / 32];
#pragma unroll
            for (int j = 0; j < BACK_CHUNK / 32; j++) {
                const int32_t p = lane + 32 * j;
                t[j] = p < it.z - it.y ? term(__ldcs(&a.col[it.y + p]), su.k) : (QT<EXT>)0;
            }
            QT<EXT> acc = ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
            const int32_t n = (__ldg(&a.row[it.x + 1]) - __ldg(&a.row[it.x]) - 1) / BACK_CHUNK + 1;
            int last = 0;
            if (lane == 0) {
                __stcg(&part[c], acc);
                __threadfence();
                last = atomicAdd(&k.arrive[it.w], 1) == n - 1;
            }
            if (!__shfl_sync(FULL, last, 0)) continue;
            __threadfence();
            acc = 0;
            for (int32_t x = it.w + lane; x < it.w + n; x += 32) acc += __ldcg(&part[x]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
            if (lane == 0) {
                k.arrive[it.w] = 0;
                bc_finish_vertex<EXT>(it.x, acc, su, delta, qo, bcacc, src);
            }
        }
        if (!mgd::grid_sync(a.bar, a.bar_err, a.bar_never)) return;
    }
}

// One level-(L-1) entry u (fewer than 128 edges [b, e)) by one thread, in
// edge order; q read through L1 (the barrier before the level makes the
// other blocks' values visible)
template <bool EXT>
__device__ __forceinline__ void bc_back_entry(const Args &a, int32_t L, int32_t u, int32_t b, int32_t e, int32_t src,
                                              QT<EXT> *q, float *delta, float *bcacc)
{
    const mgops::PathCount su = a.sigma[u];
    QT<EXT> acc = 0;
    for (int32_t k = b; k < e; k += 4) {
        int32_t w[4], lw[4], dk[4];
        QT<EXT> x[4];
#pragma unroll
        for (int j = 0; j < 4; j++) w[j] = k + j < e ? __ldg(&a.col[k + j]) : u;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            lw[j] = a.label[w[j]];
            x[j] = q[w[j]];
            dk[j] = EXT ? su.k - a.sigma[w[j]].k : 0;
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (w[j] != u && lw[j] == L) {
                if (EXT && dk[j] != 0) x[j] *= (QT<EXT>)mgops::pc_scale(dk[j]);   // (one level in hundreds)
                acc += x[j];
            }
    }
    bc_finish_vertex<EXT>(u, acc, su, delta, q, bcacc, src);
}

// the same level over the whole grid: an entry a thread, 32 a warp (a warp
// FP64 instruction costs the same for one lane as for all), the warps of
// entries dealt out over the SMs.  3000 x 3000 lattice: 8.5 us a level with
// an entry a warp -> 5.5.
template <bool EXT>
__device__ __forceinline__ void bc_back_level_flat(const Args &a, int32_t L, int32_t src, QT<EXT> *q, float *delta,
                                                   float *bcacc)
{
    const int32_t b0 = a.lvl_off[L - 1], b1 = a.lvl_off[L];
    const int32_t gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int32_t i = b0 + gw * 32 + mgd::lane(); i < b1; i += nwarps * 32) {
        const int32_t u = a.queue[i];
        bc_back_entry<EXT>(a, L, u, __ldg(&a.row[u]), __ldg(&a.row[u + 1]), src, q, delta, bcacc);
    }
}

// Consecutive levels L .. of at most CTA_BACK entries by one block on a graph
// without heavy vertices: a thread per entry, the next level's entries and
// row offsets loaded ahead, a block barrier per level instead of a grid
// barrier and L2 round trips (320 x 311 lattice, 230 entries a level: 11.7 ->
// 3.0 us per level, the grid's flat form 4.4; at 1,100 a level 14 against
// 5.2, so the bound lies between).  All threads of block 0 call; stops above
// L1.
constexpr int CTA_BACK = 768;
template <bool EXT>
__device__ __noinline__ void cta_back_levels(const Args &a, int32_t L, int32_t L1, int32_t src, QT<EXT> *q,
                                             float *delta, float *bcacc)
{
    const int t = threadIdx.x;
    // levels with entries of at most one per thread are preloaded
    int32_t b0 = a.lvl_off[L - 1], b1 = a.lvl_off[L];
    int32_t v = -1, rb = 0, re = 0;
    auto load = [&](int32_t lo, int32_t hi) {
        v = -1;
        rb = re = 0;
        if (lo + t < hi) {
            v = a.queue[lo + t];
            rb = __ldg(&a.row[v]);
            re = __ldg(&a.row[v + 1]);
        }
    };
    load(b0, b1);
    for (; L > L1; L--) {
        const int32_t cv = v, cb = rb, ce = re;
        const int32_t n0 = L - 1 > L1 ? a.lvl_off[L - 2] : 0, n1 = L - 1 > L1 ? b0 : 0;
        load(n0, n1);
        if (cv >= 0) bc_back_entry<EXT>(a, L, cv, cb, ce, src, q, delta, bcacc);
        for (int32_t i = b0 + PTHREADS + t; i < b1; i += PTHREADS) {
            const int32_t u = a.queue[i];
            bc_back_entry<EXT>(a, L, u, __ldg(&a.row[u]), __ldg(&a.row[u + 1]), src, q, delta, bcacc);
        }
        b0 = n0;
        b1 = n1;
        __syncthreads();
    }
}

// Backward sweep of graphs without heavy vertices: every level in one
// cooperative launch, runs of small levels by block 0.  A barrier timeout
// sets the error flag; the host reads it and fails the run.
template <bool EXT>
__global__ void __launch_bounds__(PTHREADS, 1) k_bc_back_levels(Args a, BCtl *bc_ctl, QT<EXT> *q, float *delta,
                                                                float *bcacc)
{
    __shared__ int4 s_b;
    if (threadIdx.x == 0) s_b = __ldcg(reinterpret_cast<const int4 *>(bc_ctl));
    __syncthreads();
    const int32_t L0 = s_b.x, src = s_b.y;
    for (int32_t L = L0; L >= 1; L--) {
        // a run of small levels is block 0's alone; the offsets are the same
        // for every block
        int32_t L1 = L;
        while (L1 >= 1 && L - L1 < CTA_LEVELS && a.lvl_off[L1] - a.lvl_off[L1 - 1] <= CTA_BACK) L1--;
        if (L - L1 >= 4) {
            if (blockIdx.x == 0) cta_back_levels<EXT>(a, L, L1, src, q, delta, bcacc);
            L = L1 + 1;
        } else {
            bc_back_level_flat<EXT>(a, L, src, q, delta, bcacc);
        }
        if (!mgd::grid_sync(a.bar, a.bar_err, a.bar_never)) return;
    }
}

__global__ void k_pc_to_double(int32_t n, const mgops::PathCount *sigma, double *out)
{
    for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        out[v] = mgops::pc_to_double(sigma[v]);
}

__global__ void k_bc_back_init(const FCtl *fc, BCtl *bc_ctl, int32_t src)
{
    if (threadIdx.x != 0) return;
    bc_ctl->src = src;
    bc_ctl->L0 = fc->nlevels - 1;
    bc_ctl->hcnt[0] = 0;
    bc_ctl->hcnt[1] = 0;
}

}  // namespace

namespace mgi {

void free_frontier_ws(mg_graph *g)
{
    if (!g->fws) return;
    FrontierWS *w = g->fws;
    DevBuf *bufs[] = {&w->label, &w->sigma, &w->sigma_d, &w->bm, &w->visited, &w->queue, &w->heavy,
                      &w->lvl_off, &w->ctl, &w->q, &w->delta, &w->bc, &w->bctl, &w->bitem, &w->barrive, &w->bpart, &w->srcbuf, &w->bar,
                      &w->cnt};
    for (DevBuf *b : bufs) dev_free(*b);
    for (auto &kv : w->lg) kv.second.destroy();
    delete w;
    g->fws = nullptr;
}

// BFS from several sources at once (one traversal of a disjoint union of
// graphs: the multi-graph batch)
mg_status frontier_bfs_multi(mg_graph *g, const int32_t *srcs_host, int32_t nsrc, const mg_opts &opt,
                             mg_run_info *info)
{
    return frontier_run_impl<mgops::Bfs>(g, 0, srcs_host, nsrc, opt, info, MG_RES_LEVEL);
}


mg_status bc_backward(mg_graph *g, int32_t src, const mg_opts &opt, float *bcacc)
{
    FrontierWS *w = g->fws;
    const size_t n = (size_t)std::max(g->nv, 1);
    Args a = make_args(g);
    // chunks of the long entries: at most this many a level
    const size_t items = (size_t)g->ne / BACK_CHUNK + (size_t)g->ne / (BACK_CHUNK + 1) + 2;
    MG_TRY(dev_alloc(w->q, n * 8 * (a.has_heavy ? 2 : 1)));
    MG_TRY(dev_alloc(w->delta, n * 4));
    MG_TRY(dev_alloc(w->bctl, sizeof(BCtl)));
    cudaStream_t s = g->stream;
    void *q = w->q.p;
    float *delta = w->delta.as<float>();
    BCtl *bc = w->bctl.as<BCtl>();
    const int grid = launch_grid(g, THREADS, 8);
    if (!w->coop_back) {
        int occ[4] = {0, 0, 0, 0};
        MG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ[0], k_bc_back_levels<false>, PTHREADS, 0));
        MG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ[1], k_bc_back_levels<true>, PTHREADS, 0));
        MG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ[2], k_bc_back_heavy<false>, PTHREADS, 0));
        MG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ[3], k_bc_back_heavy<true>, PTHREADS, 0));
        if (std::min(std::min(occ[0], occ[1]), std::min(occ[2], occ[3])) < 1)
            return fail(MG_ERR_CUDA, "persistent backward kernel does not fit on an SM");
        w->coop_back = g->num_sms;
    }
    k_bc_back_init<<<1, 32, 0, s>>>(a.ctl, bc, src);
    MG_CUDA(cudaMemsetAsync(w->bar.p, 0, BAR_BYTES, s));
    BackArgs k;
    std::memset(&k, 0, sizeof(k));
    if (a.has_heavy) {
        MG_TRY(dev_alloc(w->bitem, items * sizeof(int4)));
        MG_TRY(dev_alloc(w->barrive, items * 4));
        MG_TRY(dev_alloc(w->bpart, items * 8));
        const size_t qb = n * (a.bc_ext ? 8 : 4);
        k.q[0] = q;
        k.q[1] = (char *)q + qb;
        k.item = w->bitem.as<int4>();
        k.arrive = w->barrive.as<int32_t>();
        k.part = w->bpart.p;
        k.nitems = bc->hcnt;
        MG_CUDA(cudaMemsetAsync(q, 0, 2 * qb, s));
        MG_CUDA(cudaMemsetAsync(delta, 0, n * 4, s));
        MG_CUDA(cudaMemsetAsync(k.arrive, 0, items * 4, s));
    } else if (a.bc_ext) {
        k_bc_q_init<true><<<grid, THREADS, 0, s>>>(g->nv, a.sigma, a.label, (double *)q, delta);
    } else {
        k_bc_q_init<false><<<grid, THREADS, 0, s>>>(g->nv, a.sigma, a.label, (float *)q, delta);
    }
    MG_CUDA(cudaGetLastError());
    // every level in one cooperative launch
    Profiler &P = g->prof;
    const int sb = P.slot("bc_back");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)w->coop_back);
    cfg.blockDim = dim3(PTHREADS);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    P.begin(sb);
    if (a.has_heavy && a.bc_ext) MG_CUDA(cudaLaunchKernelEx(&cfg, k_bc_back_heavy<true>, a, bc, k, delta, bcacc));
    else if (a.has_heavy) MG_CUDA(cudaLaunchKernelEx(&cfg, k_bc_back_heavy<false>, a, bc, k, delta, bcacc));
    else if (a.bc_ext) MG_CUDA(cudaLaunchKernelEx(&cfg, k_bc_back_levels<true>, a, bc, (double *)q, delta, bcacc));
    else MG_CUDA(cudaLaunchKernelEx(&cfg, k_bc_back_levels<false>, a, bc, (float *)q, delta, bcacc));
    P.end();
    MG_CUDA(cudaMemcpyAsync(g->pinned_flag, a.bar_err, 4, cudaMemcpyDeviceToHost, s));
    MG_TRY(run_status_wait(g));
    if (*g->pinned_flag) return fail(MG_ERR_CUDA, "grid barrier of the persistent backward kernel timed out");
    (void)opt;
    return MG_OK;
}

}  // namespace mgi

using namespace mgi;

extern "C" {

static mg_status check_source(const mg_graph *g, int32_t s)
{
    if (s < 0 || s >= g->nv) return fail(MG_ERR_RANGE, "source %d out of range [0,%d)", s, g->nv);
    return MG_OK;
}

mg_status mg_bfs(mg_graph *g, int32_t source, const mg_opts *o, int32_t *level_out, mg_run_info *info)
{
    mg_opts opt;
    MG_TRY(begin_run(g, o, opt, info));
    MG_TRY(check_source(g, source));
    const size_t bytes = (size_t)g->nv * 4;
    HostPages pages(g, {{level_out, nullptr, bytes}});
    MG_TRY(frontier_run_impl<mgops::Bfs>(g, to_engine(g, source), nullptr, 0, opt, info, MG_RES_LEVEL));
    pages.wait();
    return end_run(g, opt, info, {{level_out, g->res[MG_RES_LEVEL], bytes}});
}

mg_status mg_sssp(mg_graph *g, int32_t source, const mg_opts *o, int32_t *dist_out, mg_run_info *info)
{
    mg_opts opt;
    MG_TRY(begin_run(g, o, opt, info));
    MG_TRY(check_source(g, source));
    const size_t bytes = (size_t)g->nv * 4;
    HostPages pages(g, {{dist_out, nullptr, bytes}});
    MG_TRY(frontier_run_impl<mgops::Sssp>(g, to_engine(g, source), nullptr, 0, opt, info, MG_RES_DIST));
    pages.wait();
    return end_run(g, opt, info, {{dist_out, g->res[MG_RES_DIST], bytes}});
}

mg_status mg_bc(mg_graph *g, int32_t source, const mg_opts *o, int32_t *level_out, double *sigma_out,
                float *delta_out, mg_run_info *info)
{
    mg_opts opt;
    MG_TRY(begin_run(g, o, opt, info));
    MG_TRY(check_source(g, source));
    const int32_t s = to_engine(g, source);
    const size_t n4 = (size_t)g->nv * 4;
    HostPages pages(g, {{level_out, nullptr, n4}, {sigma_out, nullptr, 2 * n4}, {delta_out, nullptr, n4}});
    MG_TRY(frontier_run_impl<mgops::BcForward>(g, s, nullptr, 0, opt, info, MG_RES_LEVEL));
    MG_TRY(bc_backward(g, s, opt, nullptr));
    FrontierWS *w = g->fws;
    // path counts as FP64 values (infinity where a count exceeds the FP64 range)
    MG_TRY(dev_alloc(w->sigma_d, (size_t)std::max(g->nv, 1) * 8));
    k_pc_to_double<<<launch_grid(g, THREADS, 8), THREADS, 0, g->stream>>>(g->nv, w->sigma.as<mgops::PathCount>(),
                                                                           w->sigma_d.as<double>());
    MG_CUDA(cudaGetLastError());
    MG_TRY(publish(g, MG_RES_SIGMA, w->sigma_d.p, 8));
    MG_TRY(publish(g, MG_RES_DELTA, w->delta.p, 4));
    pages.wait();
    return end_run(g, opt, info, {{level_out, g->res[MG_RES_LEVEL], n4},
                                  {sigma_out, g->res[MG_RES_SIGMA], 2 * n4},
                                  {delta_out, g->res[MG_RES_DELTA], n4}});
}

mg_status mg_bc_multi(mg_graph *g, const int32_t *sources, int32_t nsrc, const mg_opts *o, float *bc_out,
                      mg_run_info *info)
{
    mg_opts opt;
    MG_TRY(begin_run(g, o, opt, info));
    if (nsrc < 0 || (nsrc > 0 && !sources)) return fail(MG_ERR_INVALID, "invalid sources");
    for (int32_t i = 0; i < nsrc; i++)
        if (sources[i] < 0 || sources[i] >= g->nv) return fail(MG_ERR_RANGE, "source %d out of range", sources[i]);
    const size_t bytes = (size_t)g->nv * 4;
    HostPages pages(g, {{bc_out, nullptr, bytes}});
    if (g->symmetric) {
        // 32 sources per traversal (mg_bcb.cu)
        std::vector<int32_t> eng((size_t)nsrc);
        for (int32_t i = 0; i < nsrc; i++) eng[(size_t)i] = to_engine(g, sources[i]);
        const float *bcd = nullptr;
        MG_TRY(bc_batched(g, eng.data(), nsrc, opt, info, &bcd));
        MG_TRY(publish(g, MG_RES_BC, bcd, 4));
        mg_run_info keep;
        if (info) keep = *info;
        pages.wait();
        MG_TRY(end_run(g, opt, info, {{bc_out, g->res[MG_RES_BC], bytes}}));
        if (info) { info->iterations = keep.iterations; info->pull_iterations = keep.pull_iterations; }
        return MG_OK;
    }
    // directed graphs: one forward/backward traversal per source
    MG_TRY(ensure_ws<mgops::BcForward>(g));
    FrontierWS *w = g->fws;
    MG_TRY(dev_alloc(w->bc, (size_t)std::max(g->nv, 1) * 4));
    MG_CUDA(cudaMemsetAsync(w->bc.p, 0, (size_t)g->nv * 4, g->stream));
    int32_t iters = 0;
    for (int32_t i = 0; i < nsrc; i++) {
        mg_run_info sub;
        const int32_t s = to_engine(g, sources[i]);
        MG_TRY(frontier_run_impl<mgops::BcForward>(g, s, nullptr, 0, opt, &sub, -1));
        MG_TRY(bc_backward(g, s, opt, w->bc.as<float>()));
        iters += sub.iterations;
    }
    MG_TRY(publish(g, MG_RES_BC, w->bc.p, 4));
    pages.wait();
    MG_TRY(end_run(g, opt, info, {{bc_out, g->res[MG_RES_BC], bytes}}));
    if (info) info->iterations = iters;
    return MG_OK;
}

}  // extern "C"
