// mg_pr.cu -- PageRank engines: the reference's PR_T / PR_D recurrences,
// normalised topology- and data-driven PageRank, batched personalised
// PageRank, weighted PageRank and its adjoint (edge-weight gradient).
//
// Replaces MultiGraph_V_E_V_NOTIDEM (processi.cu:682-894) with _phase1 /
// _phase11 / _phase2.  The reference scatters pr/deg with FP32 atomicAdd into
// an intermediate buffer and gathers it in shared memory (order-dependent
// sums, ~12.5 B/edge).  Here every sweep is a pull over in-edges, in one of
// two layouts (mg_opts.pr_layout; MG_PR_LAYOUT_AUTO picks):
//   segmented (the default where the segments hold every id): k_hub_sweep
//               (mg_hub.cu) sums every in-edge from a source segment staged
//               in shared memory into per-(row, segment) piece sums, then
//   k_pr_seg    sums each row's pieces in order, applies the update and
//               (last block) closes the sweep;
//   gather (contribution gathers through L2):
//   k_pr_light  degree bins (mg_bins.cuh): a warp per row of tbin+1..heavy
//               in-edges (lanes read one 128 B line of column ids per step,
//               a fixed shuffle tree sums them), a thread per row of <= tbin
//               in-edges; then rows above heavy in-edges in chunks, one CTA
//               each, partial sums written per chunk (tbin / heavy / chunk
//               default to 32 / 512 / 2048, mg_autotune re-picks them);
//   k_pr_apply  heavy rows summed chunk by chunk in order (thread per row),
//               then the last block to finish sums every block's residual
//               partials in slot order: convergence test, loop condition
//               (without heavy rows k_pr_light closes the sweep itself).
// Sums are therefore deterministic (fixed order) run to run.
// Algorithmic bytes per sweep: 4m (column ids) + 4(n+1) (offsets) + 12n
// (old value read, new value and contribution written); in the gather
// layout the contribution gathers (4n bytes) are served by L2.

#include "mg_device.cuh"
#include "mg_ops.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace {

constexpr int THREADS = 256;


struct PCtl {
    int32_t more;
    int32_t iter;
    int32_t cur;
    int32_t status;
    int32_t max_iter;
    int32_t any;          // a vertex changed beyond tolerance / is active
    int32_t done;         // blocks of k_pr_apply that have finished this sweep
    int32_t pad2;
    double resid;         // L1 change of the last sweep
    double dangling;      // sum of x over zero out-degree vertices (current iterate)
    double lam_mean;      // adjoint: mean of lambda (dangling rows)
    float damping, tol;
    int32_t n;
    float base;           // (1-d)/n + d*dangling/n of the current sweep (set once per sweep)
    float tol_row;        // tol / n: per-vertex activity threshold of the data-driven form
    float lam_meanf;      // lam_mean as float
    // data-driven form, frontier sweeps: once the active vertices' in-edges
    // fall below m / SPARSE_ALPHA the sweeps run over a queue of them and
    // update x[cur] / c[cur] in place (frozen vertices keep their values)
    int32_t sparse;       // 1: queue sweeps
    int32_t need_compact; // the queue is to be built from the active flags
    int32_t qc;           // current queue (0 / 1)
    int32_t dense_iters;  // sweeps that ran over every row
    int32_t qn[2];        // queue sizes (qn[qc ^ 1]: appends of this sweep)
    double dang_frozen;   // dangling mass of frozen vertices
    long long act_edges;  // in-edges of the vertices still active
};

// per-sweep constants derived once (FP64 math stays out of the per-row path)
__device__ __forceinline__ void pctl_derive(PCtl *c)
{
    c->base = (float)((1.0 - (double)c->damping) / c->n + (double)c->damping * c->dangling / c->n);
    c->tol_row = c->tol / (float)c->n;
    c->lam_meanf = (float)c->lam_mean;
}

struct PArgs {
    int32_t n;
    const int32_t *prow;     // rows scanned (in-edges for PR, out-edges for the adjoint)
    const int32_t *pcol;
    const float *pw;         // per-entry weights of the scanned rows (weighted / adjoint), or null
    const int32_t *outrow;   // push-side offsets (out-degrees)
    float *S;                // weighted: out-weight sums
    const int32_t *wrows, *trows;  // degree bins
    int32_t nwrows, ntrows, nwlong;
    const int32_t *hchunk;
    int32_t nhchunks;
    const int32_t *hrows;
    const int32_t *hrow_chunk;
    int32_t nhrows;
    int32_t heavy_deg;
    // segmented pull (unweighted forms on graphs where it covers enough
    // edges): prow / pcol hold the tail part, P the sweep's per-(row,
    // segment) sums, row v's at P[pair_off[v] .. pair_off[v+1]); heavy
    // chunks keep their full-row numbering (prow_full, chunk)
    const float *P;
    const int32_t *pair_off;
    const uint16_t *porder;  // sorted windows (mg_hub.cu): each place's piece in row order
    const int32_t *prow_full;
    int32_t chunk;
    int32_t seg_only;        // every in-edge sits in a segment: rows finish in k_pr_seg
    const int32_t *fin;      // k_pr_seg's warp rows (more than fin_warp pieces)
    int32_t nfw, fin_warp;
    float *x[2];             // iterate (ping-pong)
    float *c[2];             // gathered quantity: contribution x/deg (PR) or lambda (adjoint)
    const float *gvec;       // adjoint: g
    int32_t *active;         // data-driven masks
    float *hpart;            // heavy chunk partial sums
    double *bpart;           // per-block partials: [NPART*slots] (resid, dangling, any, active edges, frozen dangling)
    int32_t nblocks;
    int32_t qblocks;          // grid of the queue sweeps (k_prd_gather / k_prd_apply)
    PCtl *ctl;
    // data-driven frontier sweeps: the full pull rows (the hub split keeps
    // only the tail in prow / pcol), two queues, the queue sweep's new values
    const int32_t *frow, *fcol;
    int32_t *queue[2];
    float *qval;
    int64_t m;
};

constexpr int NPART = 5;       // partials per block slot
constexpr int SPARSE_ALPHA = 16;  // queue sweeps once active in-edges < m / SPARSE_ALPHA

// ---------------------------------------------------------------------------
// PageRank operators: the engine (k_pr_light / k_pr_apply / k_prd_*, k_pr_all)
// is a template over one of these.  Hooks:
//   apply(a, c, v, s, any, dang)  row v's update from its gathered sum s:
//                                 writes the next iterate and contribution,
//                                 returns |change|, sets any when the row
//                                 counts as changed / active, dang = the new
//                                 value when the row is dangling
//   init(a, v, x0)                start value and contribution of row v
//   more(any, R, tol)             continue after a sweep with any / L1 change R
// Flags: kDataDriven (inactive rows frozen and skipped; queue sweeps),
// kWeights (gathers scaled by the staged per-edge weight; the others take
// the shared-memory hub split), kAdjoint (the iterate lives in c; its mean
// replaces the dangling mass); kSlot: the workspace's captured-loop slot.
// ---------------------------------------------------------------------------
// PR_T: the reference recurrence (processi.cu:631-638 / validate.cu:59-70)
struct PrTopologyRef {
    static constexpr bool kDataDriven = false, kWeights = false, kAdjoint = false;
    static constexpr int kSlot = 0;
    __device__ static __forceinline__ float apply(const PArgs &a, const PCtl &c, int32_t v, float s, int &any, float &)
    {
        const int cur = c.cur, nxt = cur ^ 1;
        const float xo = a.x[cur][v];
        const int32_t od = a.outrow[v + 1] - a.outrow[v];
        const float f1 = mgops::PrRef::apply(s);
        float xn = xo;
        if (fabsf(f1 - xo) > mgops::PrRef::TOL) { xn = f1; any = 1; }
        a.x[nxt][v] = xn;
        a.c[nxt][v] = mgops::PrRef::get_partial_result(xn, od);
        return fabsf(xn - xo);
    }
    __device__ static __forceinline__ int more(int any, double, float) { return any; }
};

// PR_D: the reference recurrence with the sticky per-vertex mask
// (processi.cu:640-655 / validate.cu:71-84): values always move, the mask
// only decides termination
struct PrDataRef {
    static constexpr bool kDataDriven = false, kWeights = false, kAdjoint = false;
    static constexpr int kSlot = 1;
    __device__ static __forceinline__ float apply(const PArgs &a, const PCtl &c, int32_t v, float s, int &any, float &)
    {
        const int cur = c.cur, nxt = cur ^ 1;
        const float xo = a.x[cur][v];
        const int32_t od = a.outrow[v + 1] - a.outrow[v];
        const float f1 = mgops::PrRef::apply(s);
        if (a.active[v] == 1 && fabsf(f1 - xo) > mgops::PrRef::TOL * xo) any = 1;
        else a.active[v] = 0;
        a.x[nxt][v] = f1;
        a.c[nxt][v] = mgops::PrRef::get_partial_result(f1, od);
        return fabsf(f1 - xo);
    }
    __device__ static __forceinline__ int more(int any, double, float) { return any; }
};

// normalised topology-driven: (1-d)/n + d (sum + dangling/n) for every row
struct PrTopology {
    static constexpr bool kDataDriven = false, kWeights = false, kAdjoint = false;
    static constexpr int kSlot = 2;
    __device__ static __forceinline__ float apply(const PArgs &a, const PCtl &c, int32_t v, float s, int &,
                                                  float &dang)
    {
        return put(a, c, v, c.base + c.damping * s, dang);
    }
    // from the row's sum as a pair high + low: rounded once
    __device__ static __forceinline__ float apply_pair(const PArgs &a, const PCtl &c, int32_t v, float2 s, float &dang)
    {
        return put(a, c, v, fmaf(c.damping, s.x, fmaf(c.damping, s.y, c.base)), dang);
    }
    __device__ static __forceinline__ float put(const PArgs &a, const PCtl &c, int32_t v, float xn, float &dang)
    {
        const int cur = c.cur, nxt = cur ^ 1;
        const float xo = a.x[cur][v];
        const int32_t od = a.outrow[v + 1] - a.outrow[v];
        a.x[nxt][v] = xn;
        a.c[nxt][v] = od > 0 ? xn / (float)od : 0.0f;
        if (od == 0) dang = xn;
        return fabsf(xn - xo);
    }
    __device__ static __forceinline__ int more(int, double R, float tol) { return R > (double)tol; }
};

// normalised data-driven: a row freezes (for good) once its change is at
// most tol / n; frozen rows keep their value and are skipped
struct PrData {
    static constexpr bool kDataDriven = true, kWeights = false, kAdjoint = false;
    static constexpr int kSlot = 3;
    __device__ static __forceinline__ float apply(const PArgs &a, const PCtl &c, int32_t v, float s, int &any,
                                                  float &dang)
    {
        const int cur = c.cur, nxt = cur ^ 1;
        const float xo = a.x[cur][v];
        const int32_t od = a.outrow[v + 1] - a.outrow[v];
        float xn = xo;   // frozen
        if (a.active[v] != 0) {
            xn = c.base + c.damping * s;
            if (fabsf(xn - xo) <= c.tol_row) a.active[v] = 0;
            else any = 1;
        }
        a.x[nxt][v] = xn;
        a.c[nxt][v] = od > 0 ? xn / (float)od : 0.0f;
        if (od == 0) dang = xn;
        return fabsf(xn - xo);
    }
    __device__ static __forceinline__ int more(int any, double R, float tol) { return any && R > (double)tol; }
};

// weighted: P_uv = w_uv / S_u
struct PrWeighted {
    static constexpr bool kDataDriven = false, kWeights = true, kAdjoint = false;
    static constexpr int kSlot = 4;
    __device__ static __forceinline__ float apply(const PArgs &a, const PCtl &c, int32_t v, float s, int &,
                                                  float &dang)
    {
        const int cur = c.cur, nxt = cur ^ 1;
        const float xo = a.x[cur][v];
        const float xn = c.base + c.damping * s;
        a.x[nxt][v] = xn;
        const float Su = a.S[v];
        a.c[nxt][v] = Su > 0.0f ? xn / Su : 0.0f;
        if (!(Su > 0.0f)) dang = xn;
        return fabsf(xn - xo);
    }
    __device__ static __forceinline__ int more(int, double R, float tol) { return R > (double)tol; }
};

// adjoint: lambda_new = g + d * (t + [S_u == 0] * mean(lambda))
struct PrAdjoint {
    static constexpr bool kDataDriven = false, kWeights = true, kAdjoint = true;
    static constexpr int kSlot = 5;
    __device__ static __forceinline__ float apply(const PArgs &a, const PCtl &c, int32_t v, float s, int &,
                                                  float &dang)
    {
        const int cur = c.cur, nxt = cur ^ 1;
        const float Su = a.S[v];
        const float t = Su > 0.0f ? s / Su : c.lam_meanf;
        const float xn = a.gvec[v] + c.damping * t;
        const float xo = a.c[cur][v];
        a.c[nxt][v] = xn;
        dang = xn;  // sum of lambda for the mean
        return fabsf(xn - xo);
    }
    __device__ static __forceinline__ int more(int, double R, float tol) { return R > (double)tol; }
};

// start values: x = x0, contributions (lambda = g for the adjoint), masks
template <class Op>
__device__ __forceinline__ void pr_init_row(const PArgs &a, int32_t v, float x0)
{
    if constexpr (Op::kAdjoint) {
        a.c[0][v] = a.gvec[v];
        return;
    }
    a.x[0][v] = x0;
    if constexpr (Op::kWeights) {
        const float Su = a.S[v];
        a.c[0][v] = Su > 0.0f ? x0 / Su : 0.0f;
    } else {
        const int32_t od = a.outrow[v + 1] - a.outrow[v];
        a.c[0][v] = od > 0 ? x0 / (float)od : 0.0f;
    }
    if (a.active) a.active[v] = 1;
}

// gathered value for edge e from source u
template <class Op>
__device__ __forceinline__ float pr_gather(const PArgs &a, int cur, int32_t e, int32_t u)
{
    float cv = a.c[cur][u];
    if (Op::kWeights) cv *= a.pw[e];
    return cv;
}

template <class Op>
__device__ __forceinline__ bool pr_row_skipped(const PArgs &a, int32_t v)
{
    return Op::kDataDriven && a.active[v] == 0;
}

// Per-block partials to bpart[slot]: the L1 change and the dangling mass
// summed in FP32 within each warp (FP64 arithmetic is slow on this part; a
// warp adds 32 per-thread FP32 sums), then in FP64 across warps; the
// data-driven form's active in-edge count and frozen dangling mass stay FP64
// throughout.
template <bool kDD>
__device__ __forceinline__ void block_partials(const PArgs &a, int slot, float r, float dg, int any,
                                               double act = 0.0, double dfz = 0.0)
{
    __shared__ double sp[NPART - 1][THREADS / 32];
    __shared__ int sa[THREADS / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        r += __shfl_xor_sync(0xffffffffu, r, o);
        dg += __shfl_xor_sync(0xffffffffu, dg, o);
        any |= __shfl_xor_sync(0xffffffffu, any, o);
        if (kDD) {
            act += __shfl_xor_sync(0xffffffffu, act, o);
            dfz += __shfl_xor_sync(0xffffffffu, dfz, o);
        }
    }
    if ((threadIdx.x & 31) == 0) {
        sp[0][threadIdx.x >> 5] = (double)r;
        sp[1][threadIdx.x >> 5] = (double)dg;
        sp[2][threadIdx.x >> 5] = kDD ? act : 0.0;
        sp[3][threadIdx.x >> 5] = kDD ? dfz : 0.0;
        sa[threadIdx.x >> 5] = any;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double T[NPART - 1] = {0, 0, 0, 0};
        int A = 0;
        for (int w = 0; w < THREADS / 32; w++) {
#pragma unroll
            for (int k = 0; k < NPART - 1; k++) T[k] += sp[k][w];
            A |= sa[w];
        }
        double *o = a.bpart + (size_t)NPART * slot;
        o[0] = T[0];
        o[1] = T[1];
        o[2] = (double)A;
        o[3] = T[2];
        o[4] = T[3];
    }
}

// the row's segment partial sums (segments ascending; 0 without the split)
__device__ __forceinline__ float seg_sum(const PArgs &a, int32_t v)
{
    float s = 0.0f;
    if (a.P)
        for (int32_t p = __ldg(&a.pair_off[v]), e = __ldg(&a.pair_off[v + 1]); p < e; p++) s += __ldcg(&a.P[p]);
    return s;
}

// row reduction for one PageRank sweep (bins_reduce interface)
template <class Op>
struct PrRowOp {
    using T = float;
    static constexpr bool kRowAware = Op::kDataDriven;  // inactive rows are skipped
    static constexpr bool kWeights = Op::kWeights;      // staged float weight bits
    const PArgs &a;
    const PCtl &c;
    float resid = 0.0f, dangs = 0.0f;  // per-thread partials (blocks sum in FP64)
    float dfz = 0.0f;                  // data-driven: dangling mass of frozen rows
    double act = 0.0;                  // data-driven: in-edges of rows still active
    int any = 0;
    __device__ float identity() const { return 0.0f; }
    __device__ bool skip(int32_t v) const { return pr_row_skipped<Op>(a, v); }
    __device__ float edge(int32_t, int32_t, int32_t u, int32_t w) const
    {
        float cv = a.c[c.cur][u];
        if (kWeights) cv *= __int_as_float(w);
        return cv;
    }
    __device__ float combine(float x, float y) const { return x + y; }
    __device__ void flush() {}
    __device__ void finish(int32_t v, float s) { finish_row(v, s + seg_sum(a, v)); }
    // the row's whole in-edge sum s
    __device__ void finish_row(int32_t v, float s)
    {
        float dg = 0.0f;
        resid += Op::apply(a, c, v, s, any, dg);
        dangs += dg;
        if (Op::kDataDriven) {
            if (a.active[v]) act += (double)(a.frow[v + 1] - a.frow[v]);
            else dfz += dg;
        }
    }
    // the same, s = high + low (one-launch form)
    __device__ void finish_pair(int32_t v, float2 s)
    {
        float dg = 0.0f;
        resid += Op::apply_pair(a, c, v, s, dg);
        dangs += dg;
    }
};

// Sum of the partials of slots [s0, s1): lane-strided in slot order, then a
// fixed shuffle tree and warp order (thread 0 gets T[0..3] and A).
__device__ __forceinline__ void reduce_slots(const double *bpart, int s0, int s1, double T[NPART - 1], int &A)
{
    __shared__ double sp[NPART - 1][THREADS / 32];
    __shared__ int sa[THREADS / 32];
    double v[NPART - 1] = {0, 0, 0, 0};
    int any = 0;
    int b = s0 + (int)threadIdx.x;
    // four slots' loads in flight, then added in slot order (the same sums
    // as one slot at a time)
    for (; b + 3 * (int)blockDim.x < s1; b += 4 * blockDim.x) {
        double r[4][NPART];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const double *o = bpart + (size_t)NPART * (b + j * blockDim.x);
#pragma unroll
            for (int k = 0; k < NPART; k++) r[j][k] = __ldcg(&o[k]);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            v[0] += r[j][0];
            v[1] += r[j][1];
            any |= r[j][2] != 0.0;
            v[2] += r[j][3];
            v[3] += r[j][4];
        }
    }
    for (; b < s1; b += blockDim.x) {
        const double *o = bpart + (size_t)NPART * b;
        v[0] += __ldcg(&o[0]);
        v[1] += __ldcg(&o[1]);
        any |= __ldcg(&o[2]) != 0.0;
        v[2] += __ldcg(&o[3]);
        v[3] += __ldcg(&o[4]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < NPART - 1; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        any |= __shfl_xor_sync(0xffffffffu, any, o);
    }
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int k = 0; k < NPART - 1; k++) sp[k][threadIdx.x >> 5] = v[k];
        sa[threadIdx.x >> 5] = any;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 0; k < NPART - 1; k++) T[k] = 0.0;
        A = 0;
        for (int w = 0; w < THREADS / 32; w++) {
            for (int k = 0; k < NPART - 1; k++) T[k] += sp[k][w];
            A |= sa[w];
        }
    }
}

// last block to arrive (per-launch counter ctl->done) returns true
__device__ __forceinline__ bool last_block(PCtl *cp)
{
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(&cp->done, 1) == (int)gridDim.x - 1);
    __syncthreads();
    return s_last != 0;
}

// End of a sweep over every row: the last block to arrive sums the blocks'
// partials of slots [0, nslots) in slot order and updates the loop state
// (iterate index, residual, dangling mass, continue flag and the graph's
// loop condition; the data-driven form's switch to queue sweeps).
template <class Op>
__device__ __forceinline__ void close_sweep(const PArgs &a, const PCtl &c, int nslots, cudaGraphConditionalHandle h,
                                            int use_cond)
{
    PCtl *cp = a.ctl;
    if (!last_block(cp)) return;
    double T[NPART - 1];
    int A;
    reduce_slots(a.bpart, 0, nslots, T, A);
    if (threadIdx.x == 0) {
        const double R = T[0], D = T[1];
        int more = 1;
        cp->done = 0;
        cp->iter = c.iter + 1;
        cp->cur = c.cur ^ 1;
        cp->resid = R;
        cp->any = A;
        if (Op::kAdjoint) cp->lam_mean = D / c.n;
        else cp->dangling = D;
        pctl_derive(cp);
        more = Op::more(A, R, c.tol) ? 1 : 0;
        if (more && cp->iter >= c.max_iter) { cp->status = 1; more = 0; }
        cp->more = more;
        if (Op::kDataDriven) {
            cp->dense_iters = c.dense_iters + 1;
            cp->act_edges = (long long)T[2];
            cp->dang_frozen = T[3];
            if (more && T[2] * SPARSE_ALPHA < (double)a.m) {
                cp->sparse = 1;
                cp->need_compact = 1;
                cp->qc = 0;
                cp->qn[0] = cp->qn[1] = 0;
            }
        }
        if (use_cond) cudaGraphSetConditional(h, more ? 1u : 0u);
    }
}

template <class Op>
__global__ void __launch_bounds__(THREADS) k_pr_light(PArgs a)
{
    // lets k_pr_apply (launched with programmatic dependent launch) be
    // scheduled while this sweep runs; it waits for the sweep's completion
    mgd::pdl_enter();
    const PCtl c = *a.ctl;
    if (c.more == 0 || c.sparse) return;
    PrRowOp<Op> op{a, c};
    const int32_t *pwt = reinterpret_cast<const int32_t *>(a.pw);
    mgd::bins_reduce(op, a.prow, a.pcol, pwt, a.wrows, a.nwrows, a.nwlong, a.trows, a.ntrows);
    // heavy-row chunks, one per CTA, in batches of 8 * THREADS edges: each
    // thread issues its 8 column loads, then its 8 gathers (one batch for
    // the default 2048-edge chunks)
    __shared__ float s_part[THREADS / 32];
    for (int32_t ch = blockIdx.x; ch < a.nhchunks; ch += gridDim.x) {
        int32_t v = a.hchunk[3 * ch], b = a.hchunk[3 * ch + 1], e = a.hchunk[3 * ch + 2];
        if (a.P) {
            // the same piece of the row's tail part: piece k of the full
            // row covers tail positions [k * chunk, (k + 1) * chunk)
            const int32_t k = (b - a.prow_full[v]) / a.chunk;
            const int32_t tb = a.prow[v], te = a.prow[v + 1];
            b = min(te, tb + k * a.chunk);
            e = min(te, b + a.chunk);
        }
        float acc = 0.0f;
        if (!pr_row_skipped<Op>(a, v)) {
            for (int32_t b0 = b; b0 < e; b0 += 8 * THREADS) {
                int32_t u[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    int32_t p = b0 + threadIdx.x + j * THREADS;
                    u[j] = p < e ? __ldcs(&a.pcol[p]) : -1;  // streamed once: evict-first
                }
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (u[j] >= 0) acc += pr_gather<Op>(a, c.cur, b0 + threadIdx.x + j * THREADS, u[j]);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            float s = 0.0f;
            for (int w = 0; w < THREADS / 32; w++) s += s_part[w];
            a.hpart[ch] = s;
        }
        __syncthreads();
    }
    block_partials<Op::kDataDriven>(a, blockIdx.x, op.resid, op.dangs, op.any, op.act, op.dfz);
}

// The whole sweep of a graph without heavy rows (and no segmented part): the
// last block to finish closes it, so there is no k_pr_apply with nothing to
// do (1000 x 1000 lattice, weighted: 31 -> 24 us a sweep).  With heavy rows,
// letting the last of a row's chunks finish it costs more than the apply
// kernel: a fence and an atomic a chunk took the weighted R-MAT 19 sweep from
// 71 to 86 us.  With longer rows (above eight edges on average) the weighted
// forms lose more to the 32 registers that eight blocks an SM leave than the
// launch costs: us a sweep with the apply kernel / closed here, forward, random
// graphs of 256 K vertices of degree 16 41 / 47, 1 M of degree 16 116 / 123;
// adjoint, 200 K rows of 120 edges in a band (24 M) 62 / 71, 1 M of degree 16
// (16.8 M) 142 / 131.  (With six blocks an SM the forward stays at 126, the
// band's adjoint at 77.)
template <class Op>
bool light_closes(const mg_graph *g)
{
    constexpr int64_t ADJOINT_EDGES = 16 << 20;
    return !Op::kWeights || (int64_t)g->ne <= (int64_t)8 * g->nv || (Op::kAdjoint && g->ne <= ADJOINT_EDGES);
}

template <class Op>
__global__ void __launch_bounds__(THREADS, 8) k_pr_light_close(PArgs a, cudaGraphConditionalHandle h, int use_cond)
{
    const PCtl c = *a.ctl;
    if (c.more == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0 && use_cond) cudaGraphSetConditional(h, 0u);
        return;
    }
    if (c.sparse) return;
    PrRowOp<Op> op{a, c};
    mgd::bins_reduce(op, a.prow, a.pcol, reinterpret_cast<const int32_t *>(a.pw), a.wrows, a.nwrows, a.nwlong, a.trows,
                     a.ntrows);
    block_partials<Op::kDataDriven>(a, blockIdx.x, op.resid, op.dangs, op.any, op.act, op.dfz);
    close_sweep<Op>(a, c, gridDim.x, h, use_cond);
}

// Row finish when every in-edge sits in a segment (no tail, no heavy-row
// chunks): each row sums its pieces' partials (P[pair_off[v] ..], segments
// ascending) and applies the update.  Rows are binned by piece count at
// layout time: long rows a warp each (lane-strided, then a fixed xor tree;
// listed), the rest a thread each in row order (compensated FP32; a warp's
// 32 rows read their piece sums as one coalesced window staged in shared
// memory) -- fixed orders, so sweeps stay reproducible.
template <class Op>
__global__ void __launch_bounds__(THREADS, 8) k_pr_seg(PArgs a, cudaGraphConditionalHandle h, int use_cond)
{
    const PCtl c = *a.ctl;
    if (c.more == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0 && use_cond) cudaGraphSetConditional(h, 0u);
        return;
    }
    if (c.sparse) return;   // queue sweeps (k_prd_*) drive the loop
    PrRowOp<Op> op{a, c};
    const int lane = mgd::lane();
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int32_t *fw = a.fin;
    for (int32_t i = gwarp; i < a.nfw; i += nwarps) {
        const int32_t v = __ldg(&fw[i]);
        // compensated sums, lane-strided then a compensated xor tree: a
        // long row's total stays steady between sweeps
        float s = 0.0f, r = 0.0f;
        if (!op.skip(v)) {
            // four loads in flight per lane (the longest rows hold about a
            // thousand pieces), added in order
            int32_t p = __ldg(&a.pair_off[v]) + lane;
            const int32_t e = __ldg(&a.pair_off[v + 1]);
            for (; p + 96 < e; p += 128) {
                const float f0 = __ldcg(&a.P[p]), f1 = __ldcg(&a.P[p + 32]), f2 = __ldcg(&a.P[p + 64]),
                            f3 = __ldcg(&a.P[p + 96]);
                mgd::kahan_add(s, r, f0);
                mgd::kahan_add(s, r, f1);
                mgd::kahan_add(s, r, f2);
                mgd::kahan_add(s, r, f3);
            }
            for (; p < e; p += 32) mgd::kahan_add(s, r, __ldcg(&a.P[p]));
        }
        const float tot = mgd::warp_sum_comp(s, r);
        if (lane == 0) op.finish_row(v, tot);
    }
    // every other row a thread each, rows in order (the warp rows skipped):
    // a warp takes 32 consecutive rows, copies their piece sums (one
    // contiguous window of P) into shared memory with coalesced loads, and
    // each lane sums its row from there; windows longer than HUB_WIN (rows
    // near the hubs) are read from P directly.  A window without a warp row is
    // sorted by segment in P (mg_hub.cu) and put back in row order on the way
    // in.  Same adds in the same order every way.
    __shared__ float s_win[THREADS / 32][mgi::HUB_WIN];
    float *win = s_win[threadIdx.x >> 5];
    for (int32_t vb = gwarp * 32; vb < a.n; vb += nwarps * 32) {
        const int32_t v = vb + lane;
        const bool act = v < a.n;
        const int32_t p0 = act ? __ldg(&a.pair_off[v]) : 0;
        const int32_t p1 = act ? __ldg(&a.pair_off[v + 1]) : 0;
        const int32_t last = min(a.n - vb, 32) - 1;
        const int32_t base = __shfl_sync(0xffffffffu, p0, 0), wend = __shfl_sync(0xffffffffu, p1, last);
        const int32_t len = wend - base;
        const bool in_win = len <= mgi::HUB_WIN;
        const bool sorted = in_win && !__any_sync(0xffffffffu, p1 - p0 > a.fin_warp);
        if (sorted) {
            int32_t i = lane;
            for (; i + 96 < len; i += 128) {
                const int k0 = __ldcs(&a.porder[base + i]), k1 = __ldcs(&a.porder[base + i + 32]),
                          k2 = __ldcs(&a.porder[base + i + 64]), k3 = __ldcs(&a.porder[base + i + 96]);
                const float f0 = __ldcg(&a.P[base + i]), f1 = __ldcg(&a.P[base + i + 32]),
                            f2 = __ldcg(&a.P[base + i + 64]), f3 = __ldcg(&a.P[base + i + 96]);
                win[k0] = f0;
                win[k1] = f1;
                win[k2] = f2;
                win[k3] = f3;
            }
            for (; i < len; i += 32) win[__ldcs(&a.porder[base + i])] = __ldcg(&a.P[base + i]);
        } else if (in_win) {
            int32_t i = lane;
            for (; i + 96 < len; i += 128) {
                const float f0 = __ldcg(&a.P[base + i]), f1 = __ldcg(&a.P[base + i + 32]),
                            f2 = __ldcg(&a.P[base + i + 64]), f3 = __ldcg(&a.P[base + i + 96]);
                win[i] = f0;
                win[i + 32] = f1;
                win[i + 64] = f2;
                win[i + 96] = f3;
            }
            for (; i < len; i += 32) win[i] = __ldcg(&a.P[base + i]);
        }
        __syncwarp();
        if (act && p1 - p0 <= a.fin_warp) {
            float s = 0.0f, r = 0.0f;
            if (!op.skip(v)) {
                if (in_win) {
                    for (int32_t p = p0 - base; p < p1 - base; p++) mgd::kahan_add(s, r, win[p]);
                } else {
                    int32_t p = p0;
                    for (; p + 4 <= p1; p += 4) {
                        const float f0 = __ldcg(&a.P[p]), f1 = __ldcg(&a.P[p + 1]), f2 = __ldcg(&a.P[p + 2]),
                                    f3 = __ldcg(&a.P[p + 3]);
                        mgd::kahan_add(s, r, f0);
                        mgd::kahan_add(s, r, f1);
                        mgd::kahan_add(s, r, f2);
                        mgd::kahan_add(s, r, f3);
                    }
                    for (; p < p1; p++) mgd::kahan_add(s, r, __ldcg(&a.P[p]));
                }
            }
            op.finish_row(v, s - r);
        }
        __syncwarp();   // the window is reused by the next 32 rows
    }
    block_partials<Op::kDataDriven>(a, blockIdx.x, op.resid, op.dangs, op.any, op.act, op.dfz);
    close_sweep<Op>(a, c, gridDim.x, h, use_cond);
}

// Heavy rows (warp per row, chunk partials summed lane-strided then by a
// fixed shuffle tree), then the last block to arrive reduces every block's
// partials in slot order and updates the loop state -- no block waits.
// The data-driven form switches to queue sweeps here once the active
// vertices' in-edges fall below m / SPARSE_ALPHA.
template <class Op>
__global__ void __launch_bounds__(THREADS) k_pr_apply(PArgs a, cudaGraphConditionalHandle h, int use_cond)
{
    mgd::pdl_enter();
    PCtl *cp = a.ctl;
    const PCtl c = *cp;
    if (c.more == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0 && use_cond) cudaGraphSetConditional(h, 0u);
        return;
    }
    if (c.sparse) return;   // queue sweeps (k_prd_*) drive the loop
    double resid = 0.0, dangs = 0.0, act = 0.0, dfz = 0.0;
    int any = 0;
    // a thread per heavy row: its chunk partials summed in chunk order, four
    // loads in flight (a row has a few chunks; every row's chain of loads
    // runs side by side instead of one warp walking two rows in turn)
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.nhrows; i += gridDim.x * blockDim.x) {
        const int32_t v = a.hrows[i];
        const int32_t k1 = a.hrow_chunk[i + 1];
        int32_t k = a.hrow_chunk[i];
        float s = 0.0f;
        for (; k + 4 <= k1; k += 4) {
            const float p0 = a.hpart[k], p1 = a.hpart[k + 1], p2 = a.hpart[k + 2], p3 = a.hpart[k + 3];
            s += p0;
            s += p1;
            s += p2;
            s += p3;
        }
        for (; k < k1; k++) s += a.hpart[k];
        float dg = 0.0f;
        s += seg_sum(a, v);
        resid += Op::apply(a, c, v, s, any, dg);
        dangs += dg;
        if (Op::kDataDriven) {
            if (a.active[v]) act += (double)(a.frow[v + 1] - a.frow[v]);
            else dfz += dg;
        }
    }
    block_partials<Op::kDataDriven>(a, a.nblocks + blockIdx.x, (float)resid, (float)dangs, any, act, dfz);
    close_sweep<Op>(a, c, a.nblocks + gridDim.x, h, use_cond);
}

// ---------------------------------------------------------------------------
// Small graphs: the whole run -- start values, every sweep, the result in
// caller order -- in one cooperative launch, a grid barrier per sweep.
// A sweep of the other layouts costs two launches, 152 stagings of up to
// 224 KB and a reduction over 1,216 blocks: 33 us on R-MAT 16 (1.8 M edges)
// whatever the size.  Here rows of up to ALL_CHUNK in-edges take eight lanes
// each (four rows a warp), the short rows at the end of the hub-first order
// (fewer than ALL_SHORT in-edges; every row of a low-degree graph) a thread,
// longer ones a warp per ALL_CHUNK-edge chunk, the last chunk to finish
// adding up the row (chunk order, so the sum does not depend on who is last).
// Contributions are gathered through L1 (the barrier's fence makes the other
// blocks' values visible there): the hubs' few sectors read by every edge
// straight from L2 took the R-MAT 16 sweep from 18 to 48 us.  Sums are
// compensated and kept as exact pairs, so an update rounds once.  After the
// barrier every block adds up the 152 blocks' partial sums itself and comes to
// the same decision.  Only for the normalised form: the data-driven form freezes and
// PR_T holds a row by comparing its change with a threshold, where one last
// bit can decide, and the weighted forms' order of additions shows in the
// gradient (k_row_sums).  R-MAT 16: 30 -> 18 us per sweep, 320 x 311 lattice 18 -> 7 us.
// Error against 64 bits (relative rms, geometric mean over R-MAT 9 to 16):
// 4.0e-8 the segmented layout, 6.1e-8 the gather layout, less than either here
// (R-MAT 16 2.9e-8 and 3.7e-8 segmented).
// ---------------------------------------------------------------------------
constexpr int ALL_THREADS = 1024;
constexpr int32_t ALL_CHUNK = 256;
constexpr int32_t ALL_SHORT = 16;
// Up to this many edges; past them the other layouts' sweeps, whose blocks
// are resident twice as densely, are the faster ones.  us per sweep, here /
// segmented / gather: R-MAT 17 (3.7 M edges) 24 / 32 / 36, of edge factor 24
// (5.4 M) 31 / 33 / 39, R-MAT 19 of edge factor 6 (6.0 M) 33 / 34 / 39, R-MAT
// 18 (7.6 M) 40 / 35 / 42, R-MAT 19 (15.5 M) 84 / 41 / 57.  Graphs of short
// rows only: 1400 x 1400 lattice (8.0 M) 19 / 43 / 29, 1700 x 1700 (11.8 M)
// 39 / 53 / 47.
constexpr int64_t ALL_MAX_EDGES = 6 << 20, ALL_MAX_EDGES_SHORT = 12 << 20;

struct PrAllArgs {
    const int32_t *chunk, *chunk_at, *row_chunk;         // rows above ALL_CHUNK edges (mgi::ppr_chunks)
    int32_t nchunks;
    int32_t split;          // rows [0, split) take eight lanes, the others a thread each
    int32_t *arrive;        // [rows] chunks finished (zero before the launch and between sweeps)
    float2 *part;           // [chunks] partial sums, high + low
    double *bsum;           // [2][grid][3] blocks' sums by sweep parity
    unsigned *bar;          // grid barrier word (zero before the launch), error word
    int *bar_err;
    int bar_never;
    const int32_t *old2new; // null: engine ids are the caller's
    float *out;             // result in caller order (null: left in x[cur])
    float x0;
};

template <class Op>
__global__ void __launch_bounds__(ALL_THREADS, 1) k_pr_all(PArgs a, PrAllArgs z)
{
    static_assert(!Op::kDataDriven && !Op::kWeights && !Op::kAdjoint, "the normalised form");
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NW = ALL_THREADS / 32;
    __shared__ PCtl s_c;
    __shared__ double s_r[NW], s_d[NW];
    __shared__ int s_a[NW];
    const int lane = mgd::lane(), warp = threadIdx.x >> 5, gl = lane & 7, grp = lane >> 3;
    const int gwarp = blockIdx.x * NW + warp, nwarps = gridDim.x * NW;
    if (threadIdx.x == 0) s_c = *a.ctl;
    for (int32_t v = blockIdx.x * ALL_THREADS + threadIdx.x; v < a.n; v += gridDim.x * ALL_THREADS)
        pr_init_row<Op>(a, v, z.x0);
    bool ok = mgd::grid_sync(z.bar, z.bar_err, z.bar_never);
    const double base0 = (1.0 - (double)s_c.damping) / a.n, basek = (double)s_c.damping / a.n;
    while (ok && s_c.more) {
        PrRowOp<Op> op{a, s_c};
        const float *cc = a.c[s_c.cur];
        for (int32_t ch = gwarp; ch < z.nchunks; ch += nwarps) {
            const int32_t v = __ldg(&z.chunk[3 * ch]), b = __ldg(&z.chunk[3 * ch + 1]), e = __ldg(&z.chunk[3 * ch + 2]);
            float s = 0.0f, r = 0.0f, t[ALL_CHUNK / 32];
#pragma unroll
            for (int j = 0; j < ALL_CHUNK / 32; j++) {
                const int32_t p = b + lane + 32 * j;
                t[j] = p < e ? cc[__ldg(&a.pcol[p])] : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < ALL_CHUNK / 32; j++) mgd::kahan_add(s, r, t[j]);
            float2 sum = mgd::warp_pair_comp(s, r);
            const int32_t at = __ldg(&z.chunk_at[ch]), k0 = __ldg(&z.row_chunk[at]), k1 = __ldg(&z.row_chunk[at + 1]);
            int last = 0;
            if (lane == 0) {
                __stcg(&z.part[ch], sum);
                __threadfence();
                last = atomicAdd(&z.arrive[at], 1) == k1 - k0 - 1;
                if (last) z.arrive[at] = 0;   // (the next sweep adds to it behind the barrier)
            }
            if (__shfl_sync(FULL, last, 0)) {
                __threadfence();
                s = r = 0.0f;
                for (int32_t k = k0 + lane; k < k1; k += 32) {
                    const float2 p = __ldcg(&z.part[k]);
                    mgd::kahan_add(s, r, p.x);
                    mgd::kahan_add(s, r, p.y);
                }
                sum = mgd::warp_pair_comp(s, r);
                if (lane == 0) op.finish_pair(v, sum);
            }
        }
        // the next rows' offsets are loaded ahead of the current rows' sums
        int32_t v = gwarp * 4 + grp;
        int32_t b = v < z.split ? __ldg(&a.prow[v]) : 0, e = v < z.split ? __ldg(&a.prow[v + 1]) : 0;
        for (int32_t v0 = gwarp * 4; v0 < z.split; v0 += nwarps * 4) {
            const int32_t vn = v + nwarps * 4;
            const int32_t bn = vn < z.split ? __ldg(&a.prow[vn]) : 0, en = vn < z.split ? __ldg(&a.prow[vn + 1]) : 0;
            const bool row = v < z.split && e - b <= ALL_CHUNK;
            const int32_t len = row ? e - b : 0;
            const int32_t rounds = (int32_t)__reduce_max_sync(FULL, (unsigned)((len + 31) >> 5));
            float s = 0.0f, r = 0.0f;
            for (int32_t k = 0; k < rounds; k++) {
                float t[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int32_t i = k * 32 + j * 8 + gl;
                    t[j] = i < len ? cc[__ldg(&a.pcol[b + i])] : 0.0f;
                }
#pragma unroll
                for (int j = 0; j < 4; j++) mgd::kahan_add(s, r, t[j]);
            }
            const float2 sum = mgd::warp_pair_comp<8>(s, r);
            if (row && gl == 0) op.finish_pair(v, sum);
            v = vn;
            b = bn;
            e = en;
        }
        for (int32_t w = z.split + gwarp * 32 + lane; w < a.n; w += nwarps * 32) {
            const int32_t wb = __ldg(&a.prow[w]), we = __ldg(&a.prow[w + 1]);
            if (we - wb > ALL_CHUNK) continue;   // (a directed graph's long in-rows: chunks above)
            const int32_t len = we - wb;
            float s = 0.0f, r = 0.0f;
            for (int32_t k = 0; k < len; k += 4) {
                float t[4];
#pragma unroll
                for (int j = 0; j < 4; j++) t[j] = k + j < len ? cc[__ldg(&a.pcol[wb + k + j])] : 0.0f;
#pragma unroll
                for (int j = 0; j < 4; j++) mgd::kahan_add(s, r, t[j]);
            }
            op.finish_pair(w, make_float2(s, -r));
        }
        // the block's sums, FP32 within a warp as in block_partials, FP64 across
        float r = op.resid, dg = op.dangs;
        int any = op.any;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            r += __shfl_xor_sync(FULL, r, o);
            dg += __shfl_xor_sync(FULL, dg, o);
        }
        any = __any_sync(FULL, any);
        if (lane == 0) {
            s_r[warp] = (double)r;
            s_d[warp] = (double)dg;
            s_a[warp] = any;
        }
        __syncthreads();
        double *bs = z.bsum + (size_t)(s_c.iter & 1) * gridDim.x * 3;
        if (warp == 0) {
            double R = s_r[lane], D = s_d[lane];
            any = __any_sync(FULL, s_a[lane]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                R += __shfl_xor_sync(FULL, R, o);
                D += __shfl_xor_sync(FULL, D, o);
            }
            if (lane == 0) {
                __stcg(&bs[blockIdx.x * 3], R);
                __stcg(&bs[blockIdx.x * 3 + 1], D);
                __stcg(&bs[blockIdx.x * 3 + 2], (double)any);
            }
        }
        ok = mgd::grid_sync(z.bar, z.bar_err, z.bar_never);
        if (!ok) break;
        if (warp == 0) {
            double R = 0.0, D = 0.0;
            any = 0;
            for (int i = lane; i < (int)gridDim.x; i += 32) {
                R += __ldcg(&bs[i * 3]);
                D += __ldcg(&bs[i * 3 + 1]);
                any |= __ldcg(&bs[i * 3 + 2]) != 0.0;
            }
            any = __any_sync(FULL, any);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                R += __shfl_xor_sync(FULL, R, o);
                D += __shfl_xor_sync(FULL, D, o);
            }
            if (lane == 0) {
                s_c.iter += 1;
                s_c.cur ^= 1;
                s_c.resid = R;
                s_c.any = any;
                s_c.dangling = D;
                s_c.base = (float)(base0 + basek * D);
                int more = Op::more(any, R, s_c.tol) ? 1 : 0;
                if (more && s_c.iter >= s_c.max_iter) {
                    s_c.status = 1;
                    more = 0;
                }
                s_c.more = more;
            }
        }
        __syncthreads();
    }
    if (z.out && ok) {
        const float *x = a.x[s_c.cur];
        for (int32_t i = blockIdx.x * ALL_THREADS + threadIdx.x; i < a.n; i += gridDim.x * ALL_THREADS)
            z.out[i] = __ldcg(&x[z.old2new ? __ldg(&z.old2new[i]) : i]);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (!ok) {
            s_c.status = 3;
            s_c.more = 0;
        }
        *a.ctl = s_c;
    }
}

// ---------------------------------------------------------------------------
// data-driven frontier sweeps (processi.cu:182-407: _process_f1 works from
// the active vertices, process_f3 applies and requeues those still above
// the per-vertex tolerance).  Pull form over the queue of active vertices;
// the sweep's new values go to qval first and are applied in place by the
// next kernel, so every gather of a sweep reads the previous iterate.
// ---------------------------------------------------------------------------
// queue = every still-active vertex (once, at the switch)
__global__ void __launch_bounds__(THREADS) k_prd_compact(PArgs a)
{
    const PCtl c = *a.ctl;
    if (!c.more || !c.sparse || !c.need_compact) return;
    const int lane = mgd::lane();
    for (int32_t b0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; b0 < a.n; b0 += gridDim.x * blockDim.x) {
        const int32_t v = b0 + lane;
        const bool p = v < a.n && a.active[v] != 0;
        const unsigned m = __ballot_sync(0xffffffffu, p);
        int base = 0;
        if (lane == 0 && m) base = atomicAdd(&a.ctl->qn[0], __popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (p) a.queue[0][base + __popc(m & ((1u << lane) - 1u))] = v;
    }
}

// one queue sweep: an 8-lane group per queued vertex (four per warp), its
// full in-edge row summed lane-strided then by a fixed shuffle tree
__global__ void __launch_bounds__(THREADS) k_prd_gather(PArgs a)
{
    const PCtl c = *a.ctl;
    if (!c.more || !c.sparse) return;
    const int lane = mgd::lane(), grp = lane >> 3, gl = lane & 7;
    const int32_t gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const int32_t nq = c.qn[c.qc];
    const int32_t *q = a.queue[c.qc];
    int32_t *nextq = a.queue[c.qc ^ 1];
    const float *cc = a.c[c.cur];
    const float *xc = a.x[c.cur];
    const float d = c.damping;
    double resid = 0.0, dangs = 0.0, act = 0.0, dfz = 0.0;
    int any = 0;
    for (int32_t base = gwarp * 4; base < nq; base += nwarps * 4) {
        const int32_t i = base + grp;
        int32_t v = -1, b = 0, e = 0;
        if (i < nq) {
            v = q[i];
            b = a.frow[v];
            e = a.frow[v + 1];
        }
        float sum = 0.0f;
        for (int32_t p = b + gl; p < e; p += 8) sum += cc[__ldg(&a.fcol[p])];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        bool keep = false;
        if (v >= 0 && gl == 0) {
            const float xo = xc[v];
            const float xn = c.base + d * sum;
            const float diff = fabsf(xn - xo);
            const int32_t od = a.outrow[v + 1] - a.outrow[v];
            a.qval[i] = xn;
            resid += diff;
            if (od == 0) dangs += xn;
            if (diff > c.tol_row) {
                keep = true;
                any = 1;
                act += (double)(e - b);
            } else {
                a.active[v] = 0;   // frozen from now on, at xn
                if (od == 0) dfz += xn;
            }
        }
        // the group leaders that stay active requeue with one atomic per warp
        const unsigned km = __ballot_sync(0xffffffffu, keep);
        int qb = 0;
        if (lane == 0 && km) qb = atomicAdd(&a.ctl->qn[c.qc ^ 1], __popc(km));
        qb = __shfl_sync(0xffffffffu, qb, 0);
        if (keep) nextq[qb + __popc(km & ((1u << lane) - 1u))] = v;
    }
    block_partials<true>(a, blockIdx.x, (float)resid, (float)dangs, any, act, dfz);
}

// apply the queue sweep's values in place, then the last block updates the
// loop state (the iterate stays in x[cur] / c[cur])
__global__ void __launch_bounds__(THREADS) k_prd_apply(PArgs a, cudaGraphConditionalHandle h, int use_cond)
{
    PCtl *cp = a.ctl;
    const PCtl c = *cp;
    if (!c.more || !c.sparse) return;   // the dense apply set the loop condition
    const int32_t nq = c.qn[c.qc];
    const int32_t *q = a.queue[c.qc];
    float *xc = a.x[c.cur];
    float *cc = a.c[c.cur];
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nq; i += gridDim.x * blockDim.x) {
        const int32_t v = q[i];
        const float xn = a.qval[i];
        const int32_t od = a.outrow[v + 1] - a.outrow[v];
        xc[v] = xn;
        cc[v] = od > 0 ? xn / (float)od : 0.0f;
    }
    if (!last_block(cp)) return;
    double T[NPART - 1];
    int A;
    reduce_slots(a.bpart, 0, gridDim.x, T, A);
    if (threadIdx.x == 0) {
        cp->done = 0;
        cp->iter = c.iter + 1;
        cp->resid = T[0];
        cp->any = A;
        cp->dangling = c.dang_frozen + T[1];
        cp->dang_frozen = c.dang_frozen + T[3];
        cp->act_edges = (long long)T[2];
        cp->need_compact = 0;
        cp->qn[c.qc] = 0;
        cp->qc = c.qc ^ 1;
        pctl_derive(cp);
        int more = (A && T[0] > (double)c.tol) ? 1 : 0;
        if (more && cp->iter >= c.max_iter) { cp->status = 1; more = 0; }
        cp->more = more;
        if (use_cond) cudaGraphSetConditional(h, more ? 1u : 0u);
    }
}

// init: x = x0, contributions, masks
template <class Op>
__global__ void k_pr_init(PArgs a, float x0)
{
    for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.n; v += gridDim.x * blockDim.x)
        pr_init_row<Op>(a, v, x0);
}

__global__ void k_pr_ctl_init(PCtl *c, int32_t n, int32_t max_iter, float damping, float tol, double dangling0,
                              double lam_mean0)
{
    if (threadIdx.x != 0) return;
    std::memset(c, 0, sizeof(PCtl));
    c->more = 1;
    c->max_iter = max_iter;
    c->damping = damping;
    c->tol = tol;
    c->n = n;
    c->dangling = dangling0;
    c->lam_mean = lam_mean0;
    pctl_derive(c);
}

// Loop control for the adjoint: start mean of lambda = mean of g (for
// dangling rows); the stopping threshold relative to |g|_1 (lambda scales
// with g, and an absolute L1 threshold would sit below FP32 resolution for
// large n).  part: (sum g, sum |g|) of each block of k_gvec_sums, added in
// slot order.  (The host used to add g up while the GPU waited.)
__global__ void __launch_bounds__(THREADS) k_gvec_sums(int32_t n, const float *g, double2 *part)
{
    __shared__ double2 sp[THREADS / 32];
    double a = 0.0, b = 0.0;
    for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const double x = (double)g[v];
        a += x;
        b += fabs(x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (mgd::lane() == 0) sp[threadIdx.x >> 5] = make_double2(a, b);
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < THREADS / 32; w++) {
            a += sp[w].x;
            b += sp[w].y;
        }
        part[blockIdx.x] = make_double2(a, b);
    }
}

__global__ void k_adjoint_ctl_init(PCtl *c, int32_t n, int32_t max_iter, float damping, float tol, const double2 *part,
                                   int nparts)
{
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < nparts; i += 32) {
        const double2 p = part[i];
        a += p.x;
        b += p.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (threadIdx.x != 0) return;
    std::memset(c, 0, sizeof(PCtl));
    c->more = 1;
    c->max_iter = max_iter;
    c->damping = damping;
    c->tol = (float)(tol * fmax(b, 1e-30));
    c->n = n;
    c->lam_mean = n > 0 ? a / n : 0.0;
    pctl_derive(c);
}

// Row totals of the weighted forms.  The order of their additions is part of
// the result: an edge of a vertex with one or two light edges has a gradient
// near zero that is a difference of nearly equal numbers times 1 / w, so the
// last bit of S or of a row total shows there.  Rows of the thread bin take a
// thread (S) or eight lanes / a warp (totals), the others a warp each, longest
// bin first, loads well ahead of the additions.
//
// S[u] = w[b] + w[b + 1] + .. one after another.  Heavy rows: a block loads
// the next 2,048 weights into shared memory while its first warp adds the
// last ones from there, four a load, about four cycles an addition (one
// thread loading and adding took 1.3 ms for a hub row of R-MAT 19, and a warp
// shuffling them one by one 0.25).
__global__ void __launch_bounds__(THREADS) k_row_sums(PArgs a, const float *__restrict__ w, float *S)
{
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int BATCH = 8 * THREADS;
    __shared__ __align__(16) float s_w[2][BATCH];
    const int lane = mgd::lane();
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int32_t i = blockIdx.x; i < a.nhrows; i += gridDim.x) {
        const int32_t u = a.hrows[i], b = a.outrow[u], e = a.outrow[u + 1];
        float s = 0.0f, x[8];
        auto load = [&](int64_t p0) {
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int64_t p = p0 + threadIdx.x + j * THREADS;
                x[j] = p < e ? __ldcs(&w[p]) : 0.0f;   // (adding +0 changes nothing)
            }
        };
        load(b);
        int buf = 0;
        for (int64_t p0 = b; p0 < e; p0 += BATCH, buf ^= 1) {
#pragma unroll
            for (int j = 0; j < 8; j++) s_w[buf][threadIdx.x + j * THREADS] = x[j];
            __syncthreads();
            load(p0 + BATCH);
            if (threadIdx.x < 32) {
                const float4 *q = reinterpret_cast<const float4 *>(s_w[buf]);
                const int n4 = (int)(min((int64_t)BATCH, e - p0) + 3) >> 2;
                for (int k = 0; k < n4; k += 8) {   // (BATCH is a multiple of 32; past the row lie zeros)
                    float4 f[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) f[j] = q[k + j];
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        s += f[j].x;
                        s += f[j].y;
                        s += f[j].z;
                        s += f[j].w;
                    }
                }
            }
        }
        if (threadIdx.x == 0) S[u] = s;
        __syncthreads();   // the buffers are reused
    }
    for (int32_t i = gwarp; i < a.nwrows; i += nwarps) {
        const int32_t u = a.wrows[i], b = a.outrow[u], e = a.outrow[u + 1];
        float s = 0.0f;
        float x = b + lane < e ? __ldcs(&w[b + lane]) : 0.0f;
        for (int32_t p = b; p < e; p += 32) {
            const int64_t q = (int64_t)p + 32 + lane;
            const float y = q < e ? __ldcs(&w[q]) : 0.0f;
#pragma unroll
            for (int k0 = 0; k0 < 32; k0 += 8) {
                float f[8];
#pragma unroll
                for (int k = 0; k < 8; k++) f[k] = __shfl_sync(FULL, x, k0 + k);
#pragma unroll
                for (int k = 0; k < 8; k++) s += f[k];
            }
            x = y;
        }
        if (lane == 0) S[u] = s;
    }
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.ntrows; i += gridDim.x * blockDim.x) {
        const int32_t u = a.trows[i], b = a.outrow[u], e = a.outrow[u + 1];
        float s = 0.0f;
        for (int32_t p = b; p < e; p += 8) {
            float x[8];
#pragma unroll
            for (int k = 0; k < 8; k++) x[k] = p + k < e ? __ldg(&w[p + k]) : 0.0f;
#pragma unroll
            for (int k = 0; k < 8; k++) s += x[k];
        }
        S[u] = s;
    }
}

// The adjoint's row value t_u = sum_e w[e] lam[v] / S[u] and the factor
// d x_u / S_u of its edges, ct[u] = (factor, t_u): lane k of a warp adds edges
// k, k + 32, .. in order, then an xor tree (of eight lanes for rows of up to
// eight edges: the others' terms are zero).  Heavy rows: a block loads, its
// first warp adds.
__global__ void __launch_bounds__(THREADS) k_back_rows(PArgs a, const float *__restrict__ w, const float *__restrict__ S,
                                                       const float *__restrict__ x, const float *__restrict__ lam,
                                                       float damping, float2 *ct)
{
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = mgd::lane(), gl = lane & 7, grp = lane >> 3;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    auto finish = [&](int32_t u, float t) {
        const float Su = S[u];
        ct[u] = make_float2(Su > 0.0f ? damping * x[u] / Su : 0.0f, Su > 0.0f ? t / Su : 0.0f);
    };
    auto warp_row = [&](int32_t u) {
        const int32_t b = a.outrow[u], e = a.outrow[u + 1];
        float t = 0.0f;
        int32_t p = b + lane;
        for (; p + 224 < e; p += 256) {
            float f[8], g[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                f[j] = __ldcs(&w[p + 32 * j]);
                g[j] = __ldg(&lam[__ldcs(&a.pcol[p + 32 * j])]);
            }
#pragma unroll
            for (int j = 0; j < 8; j++) t = fmaf(f[j], g[j], t);
        }
        for (; p < e; p += 32) t = fmaf(__ldcs(&w[p]), __ldg(&lam[__ldcs(&a.pcol[p])]), t);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(FULL, t, o);
        if (lane == 0) finish(u, t);
    };
    constexpr int BATCH = 8 * THREADS;
    __shared__ float2 s_term[BATCH];
    for (int32_t i = blockIdx.x; i < a.nhrows; i += gridDim.x) {
        const int32_t u = a.hrows[i], b = a.outrow[u], e = a.outrow[u + 1];
        float t = 0.0f;
        for (int64_t p0 = b; p0 < e; p0 += BATCH) {
            float2 x[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int64_t p = p0 + threadIdx.x + j * THREADS;
                x[j] = make_float2(0.0f, 0.0f);
                if (p < e) x[j] = make_float2(__ldcs(&w[p]), __ldg(&lam[__ldcs(&a.pcol[p])]));
            }
            __syncthreads();   // the last batch has been added up
#pragma unroll
            for (int j = 0; j < 8; j++) s_term[threadIdx.x + j * THREADS] = x[j];
            __syncthreads();
            if (threadIdx.x < 32) {
                const int n = (int)min((int64_t)BATCH, e - p0);
#pragma unroll 8
                for (int k = lane; k < n; k += 32) t = fmaf(s_term[k].x, s_term[k].y, t);
            }
        }
        if (threadIdx.x < 32) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(FULL, t, o);
            if (lane == 0) finish(u, t);
        }
    }
    for (int32_t i = gwarp; i < a.nwrows; i += nwarps) warp_row(a.wrows[i]);
    for (int32_t i0 = gwarp * 4; i0 < a.ntrows; i0 += nwarps * 4) {
        const int32_t i = i0 + grp;
        const int32_t u = i < a.ntrows ? a.trows[i] : -1;
        const int32_t b = u >= 0 ? a.outrow[u] : 0, e = u >= 0 ? a.outrow[u + 1] : 0;
        if (__any_sync(FULL, e - b > 8)) {
            for (int k = 0; k < 4; k++) {
                const int32_t uk = __shfl_sync(FULL, u, 8 * k);
                if (uk >= 0) warp_row(uk);
            }
            continue;
        }
        float t = b + gl < e ? fmaf(__ldg(&w[b + gl]), __ldg(&lam[__ldg(&a.pcol[b + gl])]), 0.0f) : 0.0f;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(FULL, t, o);
        if (u >= 0 && gl == 0) finish(u, t);
    }
}

// ---------------------------------------------------------------------------
// Personalised PageRank, up to 32 seeds per pass.  X / C are [n][4 LPR]: a
// vertex's values for the pass's seeds lie side by side, four seeds (a
// float4) a lane, LPR lanes a vertex (1, 2, 4 or 8: the fewest that hold the
// pass's seeds), 32 / LPR rows a warp at a time.  With the hub-first order
// the rows of a warp have similar lengths; they run in step over the longest
// one.  Rows with more than PPR_HEAVY in-edges are split into PPR_HEAVY-edge
// chunks (partial sums per chunk) that k_ppr_close combines in order.
//
// What bounds the sweep is bytes in flight towards L2 (4 GB of gathers on
// R-MAT 20, L2 and L1 both under half of their rates): eight 16-byte gathers
// a lane in 64 registers keep 128 KB in flight per SM, where one 4-byte
// gather of eight edges a lane in 32 registers kept 55 KB.
// R-MAT 20, 32 seeds: 527 -> 358 us per sweep (11.5 TB/s of gathers).
//
// Sums run in a fixed order that does not depend on LPR: pairwise over eight
// consecutive edges, the eights compensated in order; a heavy row's chunks in
// eight streams.  So a hub's total does not drift between sweeps, and a seed's
// ranks do not depend on how many seeds share its pass.  The update takes a
// total as a pair high + low and rounds once.
// ---------------------------------------------------------------------------
constexpr int32_t PPR_HEAVY = 256;
constexpr int PPR_THREADS = 512;       // two blocks per SM at 64 registers
constexpr int PPR_PER_SM = 2;
constexpr int PPR_CLOSE_THREADS = 512;
constexpr int PPR_CLOSE_PER_SM = 2;

struct PPCtl {
    int32_t more, iter, cur, status, max_iter, nseed;
    int32_t done;            // blocks of k_ppr_close that have finished this sweep
    int32_t pad;
    double resid[32];
};

struct PPArgs {
    int32_t n;
    const int32_t *prow, *pcol, *outrow;
    int32_t *seeds;          // [32] the pass's seeds (-1: none)
    const int32_t *hchunk;   // (row, begin, end)
    int32_t nhchunks;
    const int32_t *hrows, *hrow_chunk;
    int32_t nhrows;
    float4 *X[2], *C[2];
    float4 *hpart;           // [nhchunks][LPR]
    double2 *bpart;          // [sweep + close blocks][32] (residual, dangling mass)
    double *dang;            // [32] dangling mass of the current iterate
    PPCtl *ctl;
    float damping;
};

// start of a pass (X[0] and C[0] are zero): one block of 32 threads
__global__ void k_ppr_init(PPArgs a, const int32_t *seeds, int32_t nseed, int32_t width, int32_t max_iter)
{
    const int s = threadIdx.x;
    const int32_t v = s < nseed ? seeds[s] : -1;
    a.seeds[s] = v;
    double dg = 0.0;
    if (v >= 0) {
        const int32_t od = a.outrow[v + 1] - a.outrow[v];
        reinterpret_cast<float *>(a.X[0])[(size_t)v * width + s] = 1.0f;
        reinterpret_cast<float *>(a.C[0])[(size_t)v * width + s] = od > 0 ? 1.0f / (float)od : 0.0f;
        dg = od == 0 ? 1.0 : 0.0;
    }
    a.dang[s] = dg;
    if (s == 0) {
        std::memset(a.ctl, 0, sizeof(PPCtl));
        a.ctl->more = 1;
        a.ctl->max_iter = max_iter;
        a.ctl->nseed = nseed;
    }
}

__device__ __forceinline__ float4 f4_add(float4 a, float4 b)
{
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

// four compensated adds (mgd::kahan_add)
__device__ __forceinline__ void f4_kahan(float4 &t, float4 &r, float4 x)
{
    mgd::kahan_add(t.x, r.x, x.x);
    mgd::kahan_add(t.y, r.y, x.y);
    mgd::kahan_add(t.z, r.z, x.z);
    mgd::kahan_add(t.w, r.w, x.w);
}

// Per-lane state of the sweep: the lane's seeds, and compensated sums of the
// residual and the dangling mass.
struct PprLane {
    int32_t seed[4];
    float r[4], rc[4], d[4], dc[4];
};

template <int LPR>
__device__ __forceinline__ PprLane ppr_lane(const PPArgs &a)
{
    PprLane l;
    const int gl = threadIdx.x & (LPR - 1);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        l.seed[k] = a.seeds[gl * 4 + k];
        l.r[k] = l.rc[k] = l.d[k] = l.dc[k] = 0.0f;
    }
    return l;
}

// a gathered sum, high + low
struct PprSum {
    float4 hi, lo;
};

__device__ __forceinline__ float4 f4_neg(float4 a) { return make_float4(-a.x, -a.y, -a.z, -a.w); }

__device__ __forceinline__ float4 f4_xor(float4 a, int o)
{
    return make_float4(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o),
                       __shfl_xor_sync(0xffffffffu, a.z, o), __shfl_xor_sync(0xffffffffu, a.w, o));
}

// a += b, the same value in either operand order (TwoSum)
__device__ __forceinline__ void ppr_pair_add(PprSum &a, const PprSum &b)
{
    auto add = [](float &h, float &l, float x, float y) {
        const float u = h + x, bp = u - h;
        l = (l + y) + ((h - (u - bp)) + (x - bp));
        h = u;
    };
    add(a.hi.x, a.lo.x, b.hi.x, b.lo.x);
    add(a.hi.y, a.lo.y, b.hi.y, b.lo.y);
    add(a.hi.z, a.lo.z, b.hi.z, b.lo.z);
    add(a.hi.w, a.lo.w, b.hi.w, b.lo.w);
}

// row v's update from its gathered sum s (this lane's four seeds)
template <int LPR, bool DANG>
__device__ __forceinline__ void ppr_apply(const PPArgs &a, int cur, int32_t v, const PprSum &sum, PprLane &l)
{
    const int gl = threadIdx.x & (LPR - 1);
    const size_t at = (size_t)v * LPR + gl;
    const int32_t od = __ldg(&a.outrow[v + 1]) - __ldg(&a.outrow[v]);
    // the iterate is streamed; L2 is kept for the contributions
    const float4 xo4 = __ldcs(&a.X[cur][at]);
    const float s[4] = {sum.hi.x, sum.hi.y, sum.hi.z, sum.hi.w}, low[4] = {sum.lo.x, sum.lo.y, sum.lo.z, sum.lo.w};
    const float xo[4] = {xo4.x, xo4.y, xo4.z, xo4.w};
    float xn[4], cn[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        float base = 0.0f;
        if (v == l.seed[k]) base = (1.0f - a.damping) + a.damping * (float)a.dang[gl * 4 + k];
        xn[k] = fmaf(a.damping, s[k], fmaf(a.damping, low[k], base));
        cn[k] = od > 0 ? xn[k] / (float)od : 0.0f;
        mgd::kahan_add(l.r[k], l.rc[k], fabsf(xn[k] - xo[k]));
        if (DANG && od == 0) mgd::kahan_add(l.d[k], l.dc[k], xn[k]);
    }
    __stcs(&a.X[cur ^ 1][at], make_float4(xn[0], xn[1], xn[2], xn[3]));
    a.C[cur ^ 1][at] = make_float4(cn[0], cn[1], cn[2], cn[3]);
}

// Sum of C over the columns [b, e) for this lane's seeds.  All lanes of the
// warp call (a group without a row passes b == e) and run over the longest
// of their ranges; the next eight ids are loaded ahead of the current
// gathers.
template <int LPR>
__device__ __forceinline__ PprSum ppr_gather(const float4 *__restrict__ C, const int32_t *__restrict__ pcol, int32_t b,
                                             int32_t e)
{
    constexpr int IPL = 8 / LPR;   // ids a lane loads of eight
    const int gl = threadIdx.x & (LPR - 1);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f), low = acc;
    const int32_t rounds = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)((e - b + 7) >> 3));
    int32_t id[IPL];
#pragma unroll
    for (int k = 0; k < IPL; k++) {
        const int32_t p = b + gl + k * LPR;
        id[k] = p < e ? __ldcs(&pcol[p]) : -1;
    }
    for (int32_t r = 0; r < rounds; r++) {
        float4 t[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int32_t u = __shfl_sync(0xffffffffu, id[j / LPR], j % LPR, LPR);
            t[j] = u >= 0 ? C[(size_t)u * LPR + gl] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        b += 8;
#pragma unroll
        for (int k = 0; k < IPL; k++) {
            const int32_t p = b + gl + k * LPR;
            id[k] = p < e ? __ldcs(&pcol[p]) : -1;
        }
        f4_kahan(acc, low, f4_add(f4_add(f4_add(t[0], t[1]), f4_add(t[2], t[3])),
                                  f4_add(f4_add(t[4], t[5]), f4_add(t[6], t[7]))));
    }
    return PprSum{acc, f4_neg(low)};
}

// the block's residual and dangling sums of every seed to bpart[slot]
template <int LPR, int NT>
__device__ __forceinline__ void ppr_block_partials(const PPArgs &a, int slot, const PprLane &l)
{
    __shared__ double sr[NT / 32][4 * LPR], sd[NT / 32][4 * LPR];
    const int lane = mgd::lane(), warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        double r = (double)l.r[k] - (double)l.rc[k], d = (double)l.d[k] - (double)l.dc[k];
#pragma unroll
        for (int o = 16; o >= LPR; o >>= 1) {
            r += __shfl_xor_sync(0xffffffffu, r, o);
            d += __shfl_xor_sync(0xffffffffu, d, o);
        }
        if (lane < LPR) {
            sr[warp][lane * 4 + k] = r;
            sd[warp][lane * 4 + k] = d;
        }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        double R = 0.0, D = 0.0;
        if (threadIdx.x < 4 * LPR)
            for (int w = 0; w < NT / 32; w++) {
                R += sr[w][threadIdx.x];
                D += sd[w][threadIdx.x];
            }
        a.bpart[(size_t)slot * 32 + threadIdx.x] = make_double2(R, D);
    }
}

template <int LPR, bool DANG>
__global__ void __launch_bounds__(PPR_THREADS, PPR_PER_SM) k_ppr_sweep(PPArgs a)
{
    if (a.ctl->more == 0) return;
    constexpr int RPW = 32 / LPR;   // rows a warp
    const int cur = a.ctl->cur;
    const float4 *C = a.C[cur];
    const int gl = threadIdx.x & (LPR - 1), grp = mgd::lane() / LPR;
    const int gwarp = (blockIdx.x * PPR_THREADS + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * PPR_THREADS) >> 5;
    PprLane l = ppr_lane<LPR>(a);
    // chunks of heavy rows first: the longest
    for (int32_t c0 = gwarp * RPW; c0 < a.nhchunks; c0 += nwarps * RPW) {
        const int32_t ch = c0 + grp;
        const bool ok = ch < a.nhchunks;
        const int32_t b = ok ? __ldg(&a.hchunk[3 * ch + 1]) : 0, e = ok ? __ldg(&a.hchunk[3 * ch + 2]) : 0;
        const PprSum s = ppr_gather<LPR>(C, a.pcol, b, e);
        if (ok) a.hpart[(size_t)ch * LPR + gl] = f4_add(s.hi, s.lo);
    }
    // the next rows' offsets are loaded ahead of the current rows' gathers
    int32_t v = gwarp * RPW + grp;
    int32_t b = v < a.n ? __ldg(&a.prow[v]) : 0, e = v < a.n ? __ldg(&a.prow[v + 1]) : 0;
    for (int32_t v0 = gwarp * RPW; v0 < a.n; v0 += nwarps * RPW) {
        const int32_t vn = v + nwarps * RPW;
        const int32_t bn = vn < a.n ? __ldg(&a.prow[vn]) : 0, en = vn < a.n ? __ldg(&a.prow[vn + 1]) : 0;
        const bool row = v < a.n && e - b <= PPR_HEAVY;
        const PprSum s = ppr_gather<LPR>(C, a.pcol, b, row ? e : b);
        if (row) ppr_apply<LPR, DANG>(a, cur, v, s, l);
        v = vn;
        b = bn;
        e = en;
    }
    ppr_block_partials<LPR, PPR_THREADS>(a, blockIdx.x, l);
}

// Closes a sweep: the heavy rows (a warp each: eight streams of every eighth
// chunk whatever LPR, a lane group one or two, combined by a fixed tree), then the last block to
// arrive adds up every block's residual and dangling sums (a warp per share
// of the slots, fixed order) and updates the loop state.  (One warp adding
// 2,432 slots one after another took 300 us of an 830 us sweep.)
template <int LPR, bool DANG>
__global__ void __launch_bounds__(PPR_CLOSE_THREADS, PPR_CLOSE_PER_SM) k_ppr_close(PPArgs a, int sweep_blocks, float tol,
                                                                 cudaGraphConditionalHandle h, int use_cond)
{
    PPCtl *ctl = a.ctl;
    if (ctl->more == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0 && use_cond) cudaGraphSetConditional(h, 0u);
        return;
    }
    constexpr int RPW = 32 / LPR, NW = PPR_CLOSE_THREADS / 32;
    constexpr int STREAMS = 8, PER = RPW < STREAMS ? STREAMS / RPW : 1;   // streams of chunks; a lane group's
    const int cur = ctl->cur;
    const int gl = threadIdx.x & (LPR - 1), grp = mgd::lane() / LPR, warp = threadIdx.x >> 5;
    const int gwarp = blockIdx.x * NW + warp;
    PprLane l = ppr_lane<LPR>(a);
    for (int32_t i = gwarp; i < a.nhrows; i += gridDim.x * NW) {
        const int32_t v = __ldg(&a.hrows[i]), k0 = __ldg(&a.hrow_chunk[i]), k1 = __ldg(&a.hrow_chunk[i + 1]);
        float4 s[PER], low[PER];
#pragma unroll
        for (int p = 0; p < PER; p++) s[p] = low[p] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int32_t k = k0 + grp; k < k1 && grp < STREAMS; k += 4 * STREAMS) {
            float4 t[PER][4];
#pragma unroll
            for (int p = 0; p < PER; p++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int32_t at = k + p * RPW + j * STREAMS;
                    t[p][j] = at < k1 ? __ldcs(&a.hpart[(size_t)at * LPR + gl]) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
            for (int p = 0; p < PER; p++)
                f4_kahan(s[p], low[p], f4_add(f4_add(t[p][0], t[p][1]), f4_add(t[p][2], t[p][3])));
        }
        // the streams' totals, i and i + 4, then i and i + 2, then i and i + 1
        PprSum x{s[0], f4_neg(low[0])};
        if (PER == 2) ppr_pair_add(x, PprSum{s[PER - 1], f4_neg(low[PER - 1])});
#pragma unroll
        for (int o = (PER == 2 ? 2 : 4) * LPR; o >= LPR; o >>= 1) ppr_pair_add(x, PprSum{f4_xor(x.hi, o), f4_xor(x.lo, o)});
        if (grp == 0) ppr_apply<LPR, DANG>(a, cur, v, x, l);
    }
    ppr_block_partials<LPR, PPR_CLOSE_THREADS>(a, sweep_blocks + blockIdx.x, l);
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&ctl->done, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __shared__ double tr[NW][32], td[NW][32];
    const int lane = mgd::lane(), nslots = sweep_blocks + gridDim.x;
    double R = 0.0, D = 0.0;
    int b = warp;
    for (; b + 3 * NW < nslots; b += 4 * NW) {
        double2 t[4];
#pragma unroll
        for (int j = 0; j < 4; j++) t[j] = __ldcg(&a.bpart[(size_t)(b + j * NW) * 32 + lane]);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            R += t[j].x;
            D += t[j].y;
        }
    }
    for (; b < nslots; b += NW) {
        const double2 t = __ldcg(&a.bpart[(size_t)b * 32 + lane]);
        R += t.x;
        D += t.y;
    }
    tr[warp][lane] = R;
    td[warp][lane] = D;
    __syncthreads();
    if (warp != 0) return;
    for (int w = 1; w < NW; w++) {
        R += tr[w][lane];
        D += td[w][lane];
    }
    ctl->resid[lane] = R;
    a.dang[lane] = D;
    int more = __any_sync(0xffffffffu, lane < ctl->nseed && R > (double)tol);
    if (lane == 0) {
        ctl->iter += 1;
        ctl->cur = cur ^ 1;
        ctl->done = 0;
        if (more && ctl->iter >= ctl->max_iter) {
            ctl->status = 1;
            more = 0;
        }
        ctl->more = more;
        if (use_cond) cudaGraphSetConditional(h, more ? 1u : 0u);
    }
}

// The pass's result rows out[s0 + s][v] in caller order: 32 caller vertices
// at a time through a shared-memory tile, so both the 16 LPR byte rows of X
// and the result rows move in whole lines.  old2new null: the ids are equal.
__global__ void __launch_bounds__(THREADS) k_ppr_store(int32_t n, const float *X, int32_t width, const int32_t *old2new,
                                                       int32_t nseed, float *out)
{
    __shared__ float tile[THREADS / 32][32][33];
    float (*t)[33] = tile[threadIdx.x >> 5];
    const int lane = mgd::lane();
    const int32_t gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int64_t v0 = (int64_t)gwarp * 32; v0 < n; v0 += (int64_t)nwarps * 32) {
        const int cnt = (int)min((int64_t)32, n - v0);
        int32_t src = 0;
        if (lane < cnt) src = old2new ? __ldg(&old2new[v0 + lane]) : (int32_t)(v0 + lane);
        for (int k = 0; k < cnt; k++) {
            const int32_t u = __shfl_sync(0xffffffffu, src, k);
            if (lane < width) t[k][lane] = __ldcs(&X[(size_t)u * width + lane]);
        }
        __syncwarp();
        if (lane < cnt)
            for (int s = 0; s < nseed; s++) __stcs(&out[(size_t)s * n + v0 + lane], t[lane][s]);
        __syncwarp();
    }
}

}  // namespace

struct PrWS {
    mgi::DevBuf x0, x1, c0, c1, active, hpart, bpart, ctl, S, wT, gvec, lam_keep, xkeep;
    mgi::DevBuf gvec_caller, grad_caller;  // caller-order vectors
    mgi::DevBuf tpos;          // int32 [ne]: caller position of the reverse of each engine position's edge
    mgi::DevBuf ct, gsum;      // adjoint: row factors and totals; partial sums of g
    uint64_t tpos_version = 0; // col_version that tpos was built from (0: none)
    mgi::DevBuf q0, q1, qval;  // data-driven queue sweeps
    mgi::DevBuf arrive, apart, bsum, bar;  // k_pr_all
    uint64_t wT_version = 0;  // fw_version that S and wT were derived from (0: none)
    mgi::LoopGraph lg[6];
};

struct PprWS {
    mgi::DevBuf X0, X1, C0, C1, seeds, gseeds, ctl, bpart, dang, hpart, out;
    mgi::LoopGraph lg[8];   // by lanes per row and dangling vertices
};

struct WprWS {};

namespace mgi {

void free_pr_ws(mg_graph *g)
{
    if (!g->pws) return;
    PrWS *w = g->pws;
    DevBuf *bufs[] = {&w->x0, &w->x1, &w->c0, &w->c1, &w->active, &w->hpart, &w->bpart, &w->ctl, &w->S,
                      &w->wT, &w->gvec, &w->lam_keep, &w->xkeep, &w->gvec_caller, &w->grad_caller, &w->tpos,
                      &w->ct, &w->gsum, &w->q0, &w->q1, &w->qval, &w->arrive,
                      &w->apart, &w->bsum, &w->bar};
    for (DevBuf *b : bufs) dev_free(*b);
    for (auto &l : w->lg) l.destroy();
    delete w;
    g->pws = nullptr;
}

void free_ppr_ws(mg_graph *g)
{
    if (!g->ppws) return;
    PprWS *w = g->ppws;
    DevBuf *bufs[] = {&w->X0, &w->X1, &w->C0, &w->C1, &w->seeds, &w->gseeds, &w->ctl, &w->bpart, &w->dang,
                      &w->hpart, &w->out};
    for (DevBuf *b : bufs) dev_free(*b);
    for (auto &l : w->lg) l.destroy();
    delete w;
    g->ppws = nullptr;
}

void free_wpr_ws(mg_graph *g) { (void)g; }


// what the loop control block says after a run: info, the iterate's index,
// the status as an error
static mg_status pr_outcome(mg_graph *g, const PCtl &hc, bool dd, int32_t max_iter, mg_run_info *info, int *final_cur)
{
    if (info) {
        info->iterations = hc.iter;
        info->pull_iterations = dd ? hc.dense_iters : hc.iter;   // sweeps over every row
        info->residual = hc.resid;
        info->edges_scanned = (int64_t)hc.iter * g->ne;
    }
    *final_cur = hc.cur;
    if (hc.status == 3) return fail(MG_ERR_CUDA, "grid barrier of the persistent PageRank kernel timed out");
    if (hc.status != 0)
        return fail(MG_ERR_ITER_LIMIT, "PageRank did not converge in %d sweeps (residual %g)", max_iter, hc.resid);
    return MG_OK;
}

// Runs sweeps of variant V until convergence; the result is x[ctl.cur]
// (c[ctl.cur] for the adjoint).
// apply CTAs per SM: more blocks shorten nothing (one heavy row per warp is
// already in flight) but lengthen the last-block-done reduction and its
// counter (R-MAT 22: 27 us per apply at 8, 20 us at 4)
constexpr int APPLY_PER_SM = 4;

template <class Op>
static mg_status pr_loop(mg_graph *g, PArgs &a, const mg_opts &opt, const char *name, mg_run_info *info,
                         int *final_cur)
{
    cudaStream_t s = g->stream;
    const int grid = a.nblocks;
    Profiler &P = g->prof;
    const int sl = P.slot(name);
    std::string hn = std::string(name) + "_apply";
    const int sh = P.slot(hn.c_str());
    const int apply_grid = std::max(1, std::min(std::min(grid, (a.nhrows + THREADS - 1) / THREADS),
                                                g->num_sms * APPLY_PER_SM));
    const int shs = a.P ? P.slot("pr_hub") : -1;
    const int sqc = Op::kDataDriven ? P.slot("prd_compact") : -1, sqg = Op::kDataDriven ? P.slot("prd_gather") : -1,
              sqa = Op::kDataDriven ? P.slot("prd_apply") : -1;
    BodyFn body = [&](cudaStream_t st, cudaGraphConditionalHandle h, int use_cond) -> mg_status {
        if (a.P) MG_TRY(hub_launch(g, a.c[0], a.c[1], &a.ctl->cur, &a.ctl->more, &a.ctl->sparse, st, shs));
        P.begin(sl);
        if (a.seg_only) {
            // every row finishes in k_pr_seg, which also closes the sweep
            k_pr_seg<Op><<<grid, THREADS, 0, st>>>(a, h, use_cond);
            P.end();
        } else if (!a.P && a.nhchunks == 0 && light_closes<Op>(g)) {
            k_pr_light_close<Op><<<grid, THREADS, 0, st>>>(a, h, use_cond);
            P.end();
        } else {
            k_pr_light<Op><<<grid, THREADS, 0, st>>>(a);
            P.end();
            P.begin(sh);
            MG_TRY(launch_pdl(k_pr_apply<Op>, apply_grid, THREADS, st, a, h, use_cond));
            P.end();
        }
        if (Op::kDataDriven) {
            // queue sweeps once the switch has happened (no-ops before)
            P.begin(sqc);
            k_prd_compact<<<grid, THREADS, 0, st>>>(a);
            P.end();
            P.begin(sqg);
            k_prd_gather<<<a.qblocks, THREADS, 0, st>>>(a);
            P.end();
            P.begin(sqa);
            k_prd_apply<<<a.qblocks, THREADS, 0, st>>>(a, h, use_cond);
            P.end();
        }
        MG_CUDA(cudaGetLastError());
        return MG_OK;
    };
    int max_iter = opt.max_iter > 0 ? opt.max_iter : 10000;
    // the key holds every by-value argument of the captured kernels
    // (and the hub split's build, whose sizes the hub kernels take by value)
    const LoopKey key = LoopKey().add(Op::kSlot).add(a).add(grid).add(apply_grid).add(a.P ? g->hub.gen : 0ull);
    MG_TRY(run_loop(opt.profile ? MG_EXEC_HOST : opt.exec, opt.profile != 0, s, g->pws->lg[Op::kSlot], key, body,
                    &a.ctl->more, g->pinned_flag, max_iter + 2));
    static_assert(sizeof(PCtl) <= 512, "pinned_flag holds 512 bytes");
    MG_CUDA(cudaMemcpyAsync(g->pinned_flag, a.ctl, sizeof(PCtl), cudaMemcpyDeviceToHost, s));
    MG_TRY(run_status_wait(g));
    PCtl hc;
    std::memcpy(&hc, g->pinned_flag, sizeof(hc));
    if (a.P) MG_TRY(hub_check(g));
    return pr_outcome(g, hc, Op::kDataDriven, max_iter, info, final_cur);
}

// Whether a run takes the one-launch form.  A host-driven or profiled loop, a
// layout the caller names and one that mg_autotune measured faster on this
// graph keep their kernels.
static bool pr_small(const mg_graph *g, const mg_opts &opt, bool named_layout)
{
    return opt.exec == MG_EXEC_GRAPH && !opt.profile && !named_layout && !g->pr_no_one_launch && pr_one_launch_size(g);
}

// the one-launch form, after the control block's start values; out: result
// in caller order, or null
template <class Op>
static mg_status pr_all(mg_graph *g, const PArgs &a, const mg_opts &opt, float x0, float *out, mg_run_info *info,
                        int *final_cur)
{
    PrWS *w = g->pws;
    cudaStream_t s = g->stream;
    MG_TRY(ppr_chunks(g));
    PrAllArgs z;
    std::memset(&z, 0, sizeof(z));
    const int grid = g->num_sms;
    const size_t nrows = (size_t)std::max(g->ppr_nhrows, 1);
    MG_TRY(dev_alloc(w->arrive, nrows * 4));
    MG_TRY(dev_alloc(w->apart, (size_t)std::max(g->ppr_nhchunks, 1) * sizeof(float2)));
    MG_TRY(dev_alloc(w->bsum, (size_t)grid * 2 * 3 * 8));
    MG_TRY(dev_alloc(w->bar, 64));
    z.chunk = g->ppr_hchunk.as<int32_t>(); z.chunk_at = g->ppr_hchunk_at.as<int32_t>();
    z.row_chunk = g->ppr_hrow_chunk.as<int32_t>();
    z.nchunks = g->ppr_nhchunks;
    z.split = g->short_rows;
    z.arrive = w->arrive.as<int32_t>();
    z.part = w->apart.as<float2>();
    z.bsum = w->bsum.as<double>();
    z.bar = w->bar.as<unsigned>();
    z.bar_err = reinterpret_cast<int *>(z.bar + 8);
    z.bar_never = fail_barrier();
    z.old2new = g->relabeled ? g->old2new.as<int32_t>() : nullptr;
    z.out = out;
    z.x0 = x0;
    MG_CUDA(cudaMemsetAsync(z.arrive, 0, nrows * 4, s));
    MG_CUDA(cudaMemsetAsync(z.bar, 0, 64, s));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(ALL_THREADS);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    MG_CUDA(cudaLaunchKernelEx(&cfg, k_pr_all<Op>, a, z));
    static_assert(sizeof(PCtl) <= 512, "pinned_flag holds 512 bytes");
    MG_CUDA(cudaMemcpyAsync(g->pinned_flag, a.ctl, sizeof(PCtl), cudaMemcpyDeviceToHost, s));
    MG_TRY(run_status_wait(g));
    PCtl hc;
    std::memcpy(&hc, g->pinned_flag, sizeof(hc));
    return pr_outcome(g, hc, Op::kDataDriven, opt.max_iter > 0 ? opt.max_iter : 10000, info, final_cur);
}

static mg_status pr_setup(mg_graph *g, PArgs &a, bool weighted_or_adj, int32_t layout = MG_PR_LAYOUT_GATHER)
{
    if (!g->pws) g->pws = new PrWS();
    PrWS *w = g->pws;
    const size_t n = (size_t)std::max(g->nv, 1);
    const int grid = launch_grid(g, THREADS, 8);
    MG_TRY(dev_alloc(w->x0, n * 4));
    MG_TRY(dev_alloc(w->x1, n * 4));
    // 16 bytes of slack: the segmented sweep stages contributions in
    // 16-byte units, up to 12 bytes past the last vertex
    MG_TRY(dev_alloc(w->c0, n * 4 + 16));
    MG_TRY(dev_alloc(w->c1, n * 4 + 16));
    MG_TRY(dev_alloc(w->active, n * 4));
    MG_TRY(dev_alloc(w->hpart, (size_t)std::max(g->nhchunks, 1) * 4));
    MG_TRY(dev_alloc(w->bpart, (size_t)grid * 2 * NPART * 8));  // sweep blocks + apply blocks
    MG_TRY(dev_alloc(w->q0, n * 4));
    MG_TRY(dev_alloc(w->q1, n * 4));
    MG_TRY(dev_alloc(w->qval, n * 4));
    MG_TRY(dev_alloc(w->ctl, sizeof(PCtl)));
    std::memset(&a, 0, sizeof(a));
    a.n = g->nv;
    a.prow = g->trow;
    a.pcol = g->tcol;
    a.outrow = g->row.as<int32_t>();
    a.wrows = g->wrows.as<int32_t>(); a.nwrows = g->nwrows; a.nwlong = g->nwlong;
    a.trows = g->trows.as<int32_t>(); a.ntrows = g->ntrows;
    a.hchunk = g->hchunk.as<int32_t>(); a.nhchunks = g->nhchunks;
    a.hrows = g->hrows.as<int32_t>(); a.hrow_chunk = g->hrow_chunk.as<int32_t>(); a.nhrows = g->nhrows;
    a.heavy_deg = g->heavy_deg;
    a.x[0] = w->x0.as<float>(); a.x[1] = w->x1.as<float>();
    a.c[0] = w->c0.as<float>(); a.c[1] = w->c1.as<float>();
    a.active = w->active.as<int32_t>();
    a.hpart = w->hpart.as<float>();
    a.bpart = w->bpart.as<double>();
    a.nblocks = grid;
    // queue sweeps run while the active in-edges are below m / SPARSE_ALPHA:
    // two blocks per SM keep their block partials and the last block's
    // reduction small
    a.qblocks = std::min(grid, 2 * g->num_sms);
    a.ctl = w->ctl.as<PCtl>();
    a.frow = g->trow;
    a.fcol = g->tcol;
    a.queue[0] = w->q0.as<int32_t>();
    a.queue[1] = w->q1.as<int32_t>();
    a.qval = w->qval.as<float>();
    a.m = g->ne;
    // AUTO: segmented when the segments hold every source id (a graph with
    // ids past them gathers the rest through L2 and sums each row's parts
    // one by one, slower than the binned gather sweep), unless mg_autotune
    // measured otherwise
    if (layout == MG_PR_LAYOUT_AUTO)
        layout = (!g->pr_prefer_gather && hub_covers_all(g)) ? MG_PR_LAYOUT_SEGMENTED : MG_PR_LAYOUT_GATHER;
    if (!weighted_or_adj && layout == MG_PR_LAYOUT_SEGMENTED) {
        MG_TRY(hub_prepare(g));
        if (g->hub.use) {
            a.prow = g->hub.toff.as<int32_t>();
            a.pcol = g->hub.tcol.as<int32_t>();
            a.P = g->hub.P.as<float>();
            a.pair_off = g->hub.pair_off.as<int32_t>();
            a.porder = g->hub.porder.as<uint16_t>();
            if (g->hub.ntail == 0) {
                // rows finish in k_pr_seg, which closes the sweep
                a.seg_only = 1;
                a.fin = g->hub.fin.as<int32_t>();
                a.nfw = g->hub.nfw;
                a.fin_warp = g->hub.fin_warp;
                a.nhchunks = 0;
                a.nhrows = 0;
            }
            a.prow_full = g->trow;
            a.chunk = g->hchunk_size;
        }
    }
    if (weighted_or_adj) {
        if (!g->has_fw) return fail(MG_ERR_UNSUPPORTED, "float edge weights not set (mg_graph_set_float_weights)");
        if (!g->symmetric) return fail(MG_ERR_UNSUPPORTED, "weighted PageRank needs a structurally symmetric graph");
        MG_TRY(dev_alloc(w->S, n * 4));
        a.S = w->S.as<float>();
    }
    return MG_OK;
}

// Reverse positions of a symmetric CSR: rev[pos of (v,u) in row v] = pos of
// (u,v) in row u.  One thread per edge: the owner row u of position p by
// binary search over the row offsets, then u among row v's (ascending)
// columns.  Once per set of columns; a new set of weights then costs one
// gather (the searches took 535 us per set on R-MAT 19, the gather 45).
__global__ void k_reverse_positions(int32_t n, int32_t m, const int32_t *row, const int32_t *col, int32_t *rev)
{
    for (int32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < m; p += gridDim.x * blockDim.x) {
        int32_t lo = 0, hi = n - 1;  // last u with row[u] <= p
        while (lo < hi) {
            const int32_t mid = (lo + hi + 1) >> 1;
            if (__ldg(&row[mid]) <= p) lo = mid; else hi = mid - 1;
        }
        const int32_t u = lo, v = __ldg(&col[p]);
        int32_t a = __ldg(&row[v]), b = __ldg(&row[v + 1]) - 1, q = -1;
        while (a <= b) {
            const int32_t mid = (a + b) >> 1;
            const int32_t cm = __ldg(&col[mid]);
            if (cm == u) { q = mid; break; }
            if (cm < u) a = mid + 1; else b = mid - 1;
        }
        if (q >= 0) rev[q] = p;
    }
}

// dst[p] = src[at[p]] (0 where at[p] is -1), four positions a thread in flight
__global__ void __launch_bounds__(THREADS) k_gather_weights(int32_t m, const int32_t *__restrict__ at,
                                                            const float *__restrict__ src, float *__restrict__ dst)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < m; p += 4 * stride) {
        int32_t q[4];
#pragma unroll
        for (int j = 0; j < 4; j++) q[j] = p + j * stride < m ? __ldcs(&at[p + j * stride]) : -1;
        float x[4];
#pragma unroll
        for (int j = 0; j < 4; j++) x[j] = q[j] >= 0 ? __ldg(&src[q[j]]) : 0.0f;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (p + j * stride < m) __stcs(&dst[p + j * stride], x[j]);
    }
}

}  // namespace mgi

using namespace mgi;

extern "C" {

mg_status mg_pagerank(mg_graph *g, int32_t variant, const mg_opts *o, float *rank_out, mg_run_info *info)
{
    mg_opts opt;
    MG_TRY(begin_run(g, o, opt, info));
    if (variant < 0 || variant > 3) return fail(MG_ERR_INVALID, "unknown PageRank variant %d", variant);
    if (opt.pr_layout != MG_PR_LAYOUT_GATHER && opt.pr_layout != MG_PR_LAYOUT_SEGMENTED &&
        opt.pr_layout != MG_PR_LAYOUT_AUTO)
        return fail(MG_ERR_INVALID, "unknown PageRank layout %d", opt.pr_layout);
    const size_t bytes = (size_t)g->nv * 4;
    HostPages pages(g, {{rank_out, nullptr, bytes}});
    PArgs a;
    const bool small = variant == MG_PR_TOPOLOGY && pr_small(g, opt, opt.pr_layout != MG_PR_LAYOUT_AUTO);
    MG_TRY(pr_setup(g, a, false, small ? MG_PR_LAYOUT_GATHER : opt.pr_layout));
    cudaStream_t s = g->stream;
    const int grid = a.nblocks;
    const bool ref = variant == MG_PR_TOPOLOGY_REF || variant == MG_PR_DATA_REF;
    float d = opt.damping > 0 ? opt.damping : 0.85f;
    float tol = opt.tol > 0 ? opt.tol : 1e-6f;
    int max_iter = opt.max_iter > 0 ? opt.max_iter : 10000;
    // dangling mass of the start vector: (#zero out-degree) / n
    double dang0 = (!ref && g->nv > 0) ? (double)g->n_dangling / g->nv : 0.0;
    float x0 = ref ? 0.0f : (g->nv > 0 ? 1.0f / g->nv : 0.0f);
    k_pr_ctl_init<<<1, 32, 0, s>>>(a.ctl, g->nv, max_iter, d, tol, dang0, 0.0);
    int cur = 0;
    if (small) {
        // one launch, the result in caller order included
        float *out = nullptr;
        if (g->relabeled) {
            MG_TRY(dev_alloc(g->res_out[MG_RES_RANK], (size_t)g->nv * 4));
            out = g->res_out[MG_RES_RANK].as<float>();
        }
        MG_TRY(pr_all<PrTopology>(g, a, opt, x0, out, info, &cur));
        g->res[MG_RES_RANK] = out ? (const void *)out : a.x[cur];
        pages.wait();
        return end_run(g, opt, info, {{rank_out, g->res[MG_RES_RANK], bytes}});
    }
    switch (variant) {
    case MG_PR_TOPOLOGY_REF:
        k_pr_init<PrTopologyRef><<<grid, THREADS, 0, s>>>(a, x0);
        MG_TRY(pr_loop<PrTopologyRef>(g, a, opt, "pr_pull", info, &cur));
        break;
    case MG_PR_DATA_REF:
        k_pr_init<PrDataRef><<<grid, THREADS, 0, s>>>(a, x0);
        MG_TRY(pr_loop<PrDataRef>(g, a, opt, "pr_pull", info, &cur));
        break;
    case MG_PR_TOPOLOGY:
        k_pr_init<PrTopology><<<grid, THREADS, 0, s>>>(a, x0);
        MG_TRY(pr_loop<PrTopology>(g, a, opt, "pr_pull", info, &cur));
        break;
    default:
        k_pr_init<PrData><<<grid, THREADS, 0, s>>>(a, x0);
        MG_TRY(pr_loop<PrData>(g, a, opt, "pr_pull", info, &cur));
        break;
    }
    MG_TRY(to_caller(g, MG_RES_RANK, a.x[cur], 4, 1, &g->res[MG_RES_RANK]));
    pages.wait();
    return end_run(g, opt, info, {{rank_out, g->res[MG_RES_RANK], bytes}});
}

mg_status mg_wpagerank(mg_graph *g, const mg_opts *o, float *x_out, mg_run_info *info)
{
    mg_opts opt;
    MG_TRY(begin_run(g, o, opt, info));
    const size_t bytes = (size_t)g->nv * 4;
    HostPages pages(g, {{x_out, nullptr, bytes}});
    PArgs a;
    MG_TRY(pr_setup(g, a, true));
    PrWS *w = g->pws;
    cudaStream_t s = g->stream;
    const int grid = a.nblocks;
    const size_t n = (size_t)std::max(g->nv, 1), m = (size_t)std::max(g->ne, 1);
    MG_TRY(dev_alloc(w->wT, m * 4 + 16));  // 16 bytes of tail padding, as the column arrays
    MG_TRY(dev_alloc(w->xkeep, n * 4));
    if (w->wT_version != g->fw_version) {
        // out-weight sums and transposed weights, once per set of weights
        k_row_sums<<<grid, THREADS, 0, s>>>(a, g->fw.as<float>(), a.S);
        const int egrid = launch_grid(g, THREADS, 16);
        if (w->tpos_version != g->col_version) {
            // the reverse positions are found in the caller's CSR (ascending
            // columns) and carried to engine order like the column ids
            MG_TRY(dev_alloc(w->tpos, m * 4));
            DevBuf rev;
            int32_t *at = w->tpos.as<int32_t>();
            if (g->relabeled) {
                MG_TRY(dev_alloc(rev, m * 4));
                at = rev.as<int32_t>();
            }
            const int32_t *crow = g->relabeled ? g->o_row.as<int32_t>() : g->row.as<int32_t>();
            const int32_t *ccol = g->relabeled ? g->o_col.as<int32_t>() : g->col.as<int32_t>();
            cudaError_t e = cudaMemsetAsync(at, 0xff, (size_t)g->ne * 4, s);
            k_reverse_positions<<<egrid, THREADS, 0, s>>>(g->nv, g->ne, crow, ccol, at);
            if (e == cudaSuccess) e = cudaGetLastError();
            mg_status st = MG_OK;
            if (g->relabeled && e == cudaSuccess) {
                st = edges_to_engine(g, at, w->tpos.p);
                e = cudaStreamSynchronize(s);
            }
            dev_free(rev);
            MG_TRY(st);
            MG_CUDA(e);
            w->tpos_version = g->col_version;
        }
        k_gather_weights<<<egrid, THREADS, 0, s>>>(g->ne, w->tpos.as<int32_t>(),
                                                   g->relabeled ? g->o_fw.as<float>() : g->fw.as<float>(),
                                                   w->wT.as<float>());
        MG_CUDA(cudaGetLastError());
        w->wT_version = g->fw_version;
    }
    a.pw = w->wT.as<float>();
    float d = opt.damping > 0 ? opt.damping : 0.85f;
    float tol = opt.tol > 0 ? opt.tol : 1e-6f;
    int max_iter = opt.max_iter > 0 ? opt.max_iter : 10000;
    // rows without out-edges are dangling (their mass is spread uniformly)
    float x0 = g->nv > 0 ? 1.0f / g->nv : 0.0f;
    k_pr_ctl_init<<<1, 32, 0, s>>>(a.ctl, g->nv, max_iter, d, tol, g->nv ? (double)g->n_dangling / g->nv : 0.0, 0.0);
    int cur = 0;
    k_pr_init<PrWeighted><<<grid, THREADS, 0, s>>>(a, x0);
    MG_TRY(pr_loop<PrWeighted>(g, a, opt, "wpr_pull", info, &cur));
    MG_CUDA(cudaMemcpyAsync(w->xkeep.p, a.x[cur], (size_t)g->nv * 4, cudaMemcpyDeviceToDevice, s));
    MG_TRY(to_caller(g, MG_RES_RANK, w->xkeep.p, 4, 1, &g->res[MG_RES_RANK]));
    pages.wait();
    return end_run(g, opt, info, {{x_out, g->res[MG_RES_RANK], bytes}});
}

mg_status mg_wpagerank_backward(mg_graph *g, const float *g_host, const mg_opts *o, float *grad_w_out,
                                float *lambda_out, mg_run_info *info)
{
    mg_opts opt;
    MG_TRY(begin_run(g, o, opt, info));
    if (!g_host && g->nv > 0) return fail(MG_ERR_INVALID, "null loss weights");
    if (!g->pws || !g->pws->xkeep.p || !g->pws->wT.p) return fail(MG_ERR_INVALID, "run mg_wpagerank first");
    HostPages pages(g, {{grad_w_out, nullptr, (size_t)g->ne * 4}, {lambda_out, nullptr, (size_t)g->nv * 4}});
    PArgs a;
    MG_TRY(pr_setup(g, a, true));
    PrWS *w = g->pws;
    cudaStream_t s = g->stream;
    const int grid = a.nblocks;
    const size_t n = (size_t)std::max(g->nv, 1), m = (size_t)std::max(g->ne, 1);
    MG_TRY(dev_alloc(w->gvec, n * 4));
    MG_TRY(dev_alloc(w->ct, n * sizeof(float2)));
    MG_TRY(dev_alloc(w->gsum, (size_t)g->num_sms * sizeof(double2)));
    MG_TRY(dev_alloc(w->lam_keep, n * 4));
    MG_TRY(dev_alloc(w->gvec_caller, n * 4));
    MG_TRY(dev_alloc(w->grad_caller, m * 4));
    if (g->nv) MG_CUDA(cudaMemcpyAsync(w->gvec_caller.p, g_host, (size_t)g->nv * 4, cudaMemcpyHostToDevice, s));
    MG_TRY(vertices_to_engine(g, w->gvec_caller.p, w->gvec.p));
    // lambda = g + d * P lambda : rows of P are the CSR rows (out-edges) with weights w
    a.prow = g->row.as<int32_t>();
    a.pcol = g->col.as<int32_t>();
    a.pw = g->fw.as<float>();
    a.gvec = w->gvec.as<float>();
    k_row_sums<<<grid, THREADS, 0, s>>>(a, g->fw.as<float>(), a.S);
    float d = opt.damping > 0 ? opt.damping : 0.85f;
    float tol = opt.tol > 0 ? opt.tol : 1e-6f;
    int max_iter = opt.max_iter > 0 ? opt.max_iter : 10000;
    double2 *gsum = w->gsum.as<double2>();
    k_gvec_sums<<<g->num_sms, THREADS, 0, s>>>(g->nv, w->gvec_caller.as<float>(), gsum);
    k_adjoint_ctl_init<<<1, 32, 0, s>>>(a.ctl, g->nv, max_iter, d, tol, gsum, g->num_sms);
    int cur = 0;
    k_pr_init<PrAdjoint><<<grid, THREADS, 0, s>>>(a, 0.0f);
    MG_TRY(pr_loop<PrAdjoint>(g, a, opt, "wpr_adjoint", info, &cur));
    float *lam = a.c[cur];
    MG_CUDA(cudaMemcpyAsync(w->lam_keep.p, lam, (size_t)g->nv * 4, cudaMemcpyDeviceToDevice, s));
    int sg = g->prof.slot("wpr_grad");
    g->prof.begin(sg);
    k_back_rows<<<grid, THREADS, 0, s>>>(a, g->fw.as<float>(), a.S, w->xkeep.as<float>(), w->lam_keep.as<float>(), d,
                                         w->ct.as<float2>());
    MG_TRY(edge_grad_to_caller(g, w->ct.as<float2>(), w->lam_keep.as<float>(), w->grad_caller.as<float>()));
    g->prof.end();
    const void *lam_out = nullptr;
    MG_TRY(to_caller(g, MG_RES_DELTA, w->lam_keep.p, 4, 1, &lam_out));
    pages.wait();
    return end_run(g, opt, info, {{lambda_out, lam_out, (size_t)g->nv * 4},
                                  {grad_w_out, w->grad_caller.p, (size_t)g->ne * 4}});
}

}  // extern "C"

bool mgi::pr_one_launch_size(const mg_graph *g)
{
    const bool short_rows = !g->relabeled && (int64_t)g->ne <= (int64_t)8 * g->nv;  // (as ppr_chunks)
    return g->nv > 0 && g->ne <= (short_rows ? ALL_MAX_EDGES_SHORT : ALL_MAX_EDGES);
}

// heavy-row chunk table (built once per layout from the pull offsets)
mg_status mgi::ppr_chunks(mg_graph *g)
{
    if (g->ppr_nhchunks >= 0) return MG_OK;
    const std::vector<int32_t> &pr = g->h_prow;
    std::vector<int32_t> hc, hr, hrc{0};
    for (int32_t v = 0; v < g->nv; v++) {
        if (pr[v + 1] - pr[v] <= PPR_HEAVY) continue;
        hr.push_back(v);
        for (int32_t b = pr[v]; b < pr[v + 1]; b += PPR_HEAVY) {
            hc.push_back(v); hc.push_back(b); hc.push_back(std::min(pr[v + 1], b + PPR_HEAVY));
        }
        hrc.push_back((int32_t)(hc.size() / 3));
    }
    cudaStream_t s = g->stream;
    MG_TRY(dev_alloc(g->ppr_hchunk, std::max<size_t>(hc.size(), 3) * 4));
    MG_TRY(dev_alloc(g->ppr_hrows, std::max<size_t>(hr.size(), 1) * 4));
    MG_TRY(dev_alloc(g->ppr_hrow_chunk, hrc.size() * 4));
    std::vector<int32_t> at;
    for (size_t i = 0; i < hr.size(); i++) at.insert(at.end(), (size_t)(hrc[i + 1] - hrc[i]), (int32_t)i);
    MG_TRY(dev_alloc(g->ppr_hchunk_at, std::max<size_t>(at.size(), 1) * 4));
    if (!at.empty()) MG_CUDA(cudaMemcpyAsync(g->ppr_hchunk_at.p, at.data(), at.size() * 4, cudaMemcpyHostToDevice, s));
    if (!hc.empty()) MG_CUDA(cudaMemcpyAsync(g->ppr_hchunk.p, hc.data(), hc.size() * 4, cudaMemcpyHostToDevice, s));
    if (!hr.empty()) MG_CUDA(cudaMemcpyAsync(g->ppr_hrows.p, hr.data(), hr.size() * 4, cudaMemcpyHostToDevice, s));
    MG_CUDA(cudaMemcpyAsync(g->ppr_hrow_chunk.p, hrc.data(), hrc.size() * 4, cudaMemcpyHostToDevice, s));
    MG_CUDA(cudaStreamSynchronize(s));
    // first of the short rows at the end (hub-first order: degrees fall by
    // powers of two); a low-degree graph is all short rows
    int32_t split = g->nv;
    while (g->symmetric && split > 0 && pr[split] - pr[split - 1] < ALL_SHORT) split--;
    if (!g->relabeled) split = (int64_t)g->ne <= (int64_t)8 * g->nv ? 0 : g->nv;
    g->short_rows = split;
    g->ppr_nhchunks = (int32_t)(hc.size() / 3);
    g->ppr_nhrows = (int32_t)hr.size();
    return MG_OK;
}

// one pass of up to 4 LPR seeds: sweeps until every seed's L1 change is at
// most tol
template <int LPR, bool DANG>
static mg_status ppr_pass(mg_graph *g, const PPArgs &a, const int32_t *seeds_dev, int32_t nseed, const mg_opts &opt,
                          float tol, int32_t max_iter, PPCtl &hc)
{
    PprWS *w = g->ppws;
    cudaStream_t s = g->stream;
    const size_t bytes = (size_t)std::max(g->nv, 1) * LPR * 16;
    const int grid = launch_grid(g, PPR_THREADS, PPR_PER_SM), close_grid = launch_grid(g, PPR_CLOSE_THREADS, PPR_CLOSE_PER_SM);
    MG_CUDA(cudaMemsetAsync(a.X[0], 0, bytes, s));
    MG_CUDA(cudaMemsetAsync(a.C[0], 0, bytes, s));
    k_ppr_init<<<1, 32, 0, s>>>(a, seeds_dev, nseed, 4 * LPR, max_iter);
    MG_CUDA(cudaGetLastError());
    Profiler &P = g->prof;
    const int sl = P.slot("ppr_pull"), sc = P.slot("ppr_close");
    BodyFn body = [&](cudaStream_t st, cudaGraphConditionalHandle h, int use_cond) -> mg_status {
        P.begin(sl);
        k_ppr_sweep<LPR, DANG><<<grid, PPR_THREADS, 0, st>>>(a);
        P.end();
        P.begin(sc);
        k_ppr_close<LPR, DANG><<<close_grid, PPR_CLOSE_THREADS, 0, st>>>(a, grid, tol, h, use_cond);
        P.end();
        MG_CUDA(cudaGetLastError());
        return MG_OK;
    };
    // the captured kernels take the whole PPArgs (pointers, counts, the
    // heavy-row table, damping), the tolerance and the grids by value; the
    // pass's seeds lie in a buffer, so every pass of a call replays one loop
    const LoopKey key = LoopKey().add(a).add(tol).add(grid).add(close_grid);
    const int slot = (LPR == 1 ? 0 : LPR == 2 ? 1 : LPR == 4 ? 2 : 3) * 2 + (DANG ? 1 : 0);
    MG_TRY(run_loop(opt.profile ? MG_EXEC_HOST : opt.exec, opt.profile != 0, s, w->lg[slot], key, body, &a.ctl->more,
                    g->pinned_flag, max_iter + 2));
    static_assert(sizeof(PPCtl) <= 512, "pinned_flag holds 512 bytes");
    MG_CUDA(cudaMemcpyAsync(g->pinned_flag, a.ctl, sizeof(PPCtl), cudaMemcpyDeviceToHost, s));
    MG_TRY(run_status_wait(g));
    std::memcpy(&hc, g->pinned_flag, sizeof(hc));
    return MG_OK;
}

template <int LPR>
static mg_status ppr_pass(mg_graph *g, const PPArgs &a, const int32_t *seeds_dev, int32_t nseed, const mg_opts &opt,
                          float tol, int32_t max_iter, PPCtl &hc)
{
    return g->n_dangling > 0 ? ppr_pass<LPR, true>(g, a, seeds_dev, nseed, opt, tol, max_iter, hc)
                             : ppr_pass<LPR, false>(g, a, seeds_dev, nseed, opt, tol, max_iter, hc);
}

extern "C" {

mg_status mg_ppr_batch(mg_graph *g, const int32_t *seeds, int32_t nseeds, const mg_opts *o, float *out,
                       mg_run_info *info)
{
    mg_opts opt;
    MG_TRY(begin_run(g, o, opt, info));
    if (nseeds < 0 || (nseeds > 0 && !seeds)) return fail(MG_ERR_INVALID, "invalid seeds");
    for (int32_t i = 0; i < nseeds; i++)
        if (seeds[i] < 0 || seeds[i] >= g->nv) return fail(MG_ERR_RANGE, "seed %d out of range", seeds[i]);
    HostPages pages(g, {{out, nullptr, (size_t)nseeds * g->nv * 4}});
    if (!g->ppws) g->ppws = new PprWS();
    PprWS *w = g->ppws;
    const size_t n = (size_t)std::max(g->nv, 1);
    cudaStream_t s = g->stream;
    MG_TRY(ppr_chunks(g));
    // lanes per row: as many as the widest pass of this call needs
    const int32_t widest = std::min(nseeds, 32);
    const size_t width = widest > 16 ? 32 : widest > 8 ? 16 : widest > 4 ? 8 : 4;
    MG_TRY(dev_alloc(w->X0, n * width * 4));
    MG_TRY(dev_alloc(w->X1, n * width * 4));
    MG_TRY(dev_alloc(w->C0, n * width * 4));
    MG_TRY(dev_alloc(w->C1, n * width * 4));
    MG_TRY(dev_alloc(w->seeds, (size_t)std::max(nseeds, 1) * 4));
    MG_TRY(dev_alloc(w->gseeds, 32 * 4));
    MG_TRY(dev_alloc(w->ctl, sizeof(PPCtl)));
    MG_TRY(dev_alloc(w->bpart, (size_t)g->num_sms * (PPR_PER_SM + PPR_CLOSE_PER_SM) * 32 * sizeof(double2)));
    MG_TRY(dev_alloc(w->dang, 32 * 8));
    MG_TRY(dev_alloc(w->hpart, (size_t)std::max(g->ppr_nhchunks, 1) * width * 4));
    MG_TRY(dev_alloc(w->out, (size_t)std::max(nseeds, 1) * n * 4));
    std::vector<int32_t> eseeds(seeds, seeds + nseeds);
    for (int32_t &v : eseeds) v = to_engine(g, v);
    if (nseeds) MG_CUDA(cudaMemcpyAsync(w->seeds.p, eseeds.data(), (size_t)nseeds * 4, cudaMemcpyHostToDevice, s));
    float tol = opt.tol > 0 ? opt.tol : 1e-6f;
    int max_iter = opt.max_iter > 0 ? opt.max_iter : 10000;
    PPArgs a;
    std::memset(&a, 0, sizeof(a));
    a.n = g->nv;
    a.prow = g->trow; a.pcol = g->tcol; a.outrow = g->row.as<int32_t>();
    a.seeds = w->gseeds.as<int32_t>();
    a.hchunk = g->ppr_hchunk.as<int32_t>(); a.nhchunks = g->ppr_nhchunks;
    a.hrows = g->ppr_hrows.as<int32_t>(); a.hrow_chunk = g->ppr_hrow_chunk.as<int32_t>(); a.nhrows = g->ppr_nhrows;
    a.X[0] = w->X0.as<float4>(); a.X[1] = w->X1.as<float4>();
    a.C[0] = w->C0.as<float4>(); a.C[1] = w->C1.as<float4>();
    a.hpart = w->hpart.as<float4>();
    a.bpart = w->bpart.as<double2>();
    a.dang = w->dang.as<double>();
    a.ctl = w->ctl.as<PPCtl>();
    a.damping = opt.damping > 0 ? opt.damping : 0.85f;
    int32_t total_iters = 0;
    double max_resid = 0.0;
    for (int32_t s0 = 0; s0 < nseeds; s0 += 32) {
        const int32_t cnt = std::min(32, nseeds - s0);
        const int32_t *sd = w->seeds.as<int32_t>() + s0;
        PPCtl hc;
        int32_t pass_width;
        if (cnt > 16) { pass_width = 32; MG_TRY(ppr_pass<8>(g, a, sd, cnt, opt, tol, max_iter, hc)); }
        else if (cnt > 8) { pass_width = 16; MG_TRY(ppr_pass<4>(g, a, sd, cnt, opt, tol, max_iter, hc)); }
        else if (cnt > 4) { pass_width = 8; MG_TRY(ppr_pass<2>(g, a, sd, cnt, opt, tol, max_iter, hc)); }
        else { pass_width = 4; MG_TRY(ppr_pass<1>(g, a, sd, cnt, opt, tol, max_iter, hc)); }
        if (hc.status) return fail(MG_ERR_ITER_LIMIT, "PPR did not converge in %d sweeps", max_iter);
        total_iters += hc.iter;
        for (int i = 0; i < cnt; i++) max_resid = std::max(max_resid, hc.resid[i]);
        k_ppr_store<<<launch_grid(g, THREADS, 6), THREADS, 0, s>>>(
            g->nv, (const float *)a.X[hc.cur], pass_width, g->relabeled ? g->old2new.as<int32_t>() : nullptr, cnt,
            w->out.as<float>() + (size_t)s0 * g->nv);
        MG_CUDA(cudaGetLastError());
    }
    pages.wait();
    MG_TRY(end_run(g, opt, info, {{out, w->out.p, (size_t)nseeds * g->nv * 4}}));
    if (info) { info->iterations = total_iters; info->residual = max_resid; }
    return MG_OK;
}
}  // extern "C"
