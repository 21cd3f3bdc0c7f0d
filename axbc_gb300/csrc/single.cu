// Plain form: one pivot.  axbc_run_pivot runs the whole pass in one cooperative
// launch (k_pivot below).  The level-by-level form, one launch sequence per BFS
// level with the host reading the frontier size after each -- the structure of
// bc_func_mono (src/axbc2d.c:1514-1659) -- serves the reference-named entry
// points and runs under the profiling hooks:
//   forward level: push from the frontier queue (warp per frontier vertex,
//     lanes over its neighbours, atomicCAS claims, atomicAdd path counts) or
//     pull into every unvisited vertex (warp per vertex, integer warp sum);
//   backward level: warp per vertex of the depth, the canonical dependency
//     sum (lane = adjacency position, tree per 32, chunks then spans in order);
//   update: one thread per vertex.
// Vertices with more than AXBC_SPAN neighbours are split into span items.
#include <algorithm>

#include "barrier.cuh"
#include "common.cuh"

__global__ void k_reset1(int32_t *__restrict__ lvl, uint32_t *__restrict__ sigma,
                         float *__restrict__ delta, const uint32_t *__restrict__ reach, uint64_t n)
{
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
         v += (uint64_t)gridDim.x * blockDim.x) {
        lvl[v] = -1;
        sigma[v] = 0;
        delta[v] = __uint2float_rn(reach[v]);
    }
}

// warp-aggregated append of the lanes' newly discovered vertices
__device__ __forceinline__ void append_new(bool isnew, uint32_t r, uint32_t deg_r, uint32_t rdeg_r,
                                           uint32_t *queue, PivotCounters *pc)
{
    const unsigned lane = lane_id();
    unsigned m = __ballot_sync(FULL_MASK, isnew);
    if (!m) return;
    const int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if ((int)lane == leader) base = atomicAdd(&pc->qtail, (uint32_t)__popc(m));
    base = __shfl_sync(FULL_MASK, base, leader);
    if (isnew) queue[base + __popc(m & ((1u << lane) - 1u))] = r;
    uint32_t d = __reduce_add_sync(FULL_MASK, isnew ? deg_r : 0u);
    uint32_t rd = __reduce_add_sync(FULL_MASK, isnew ? rdeg_r : 0u);
    if ((int)lane == leader) {
        atomicAdd(&pc->newdeg, (unsigned long long)d);
        atomicAdd(&pc->visited_rdeg, (unsigned long long)rd);
    }
}

// Forward level L, push: tasks [0,nf) are the frontier vertices of depth L-1
// (light ones), then the span items of heavy vertices at depth L-1
// (scan_col_mono2, src/cuda_kernels.cu:588-658: a neighbour r is new if its
// level is unset; sigma[r] += sigma[c] when r's level is L).
__global__ void k_fwd_push1(Adj a, const uint32_t *__restrict__ rcol, uint32_t qs, uint32_t nf,
                            int32_t *lvl, uint32_t *sigma, uint32_t *queue, PivotCounters *pc, int L)
{
    const unsigned lane = lane_id();
    const uint64_t ntask = nf + a.n_heavy_items;
    const uint64_t nw = (uint64_t)gridDim.x * blockDim.x / 32;
    for (uint64_t t = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32; t < ntask; t += nw) {
        uint32_t c, b0, b1;
        if (t < nf) {
            c = queue[qs + t];
            b0 = a.col[c];
            b1 = a.col[c + 1];
            if (b1 - b0 > AXBC_SPAN) continue;
        } else {
            const uint64_t h = t - nf;
            c = a.hitem_v[h];
            if (lvl[c] != L - 1) continue;
            b0 = a.col[c] + a.hitem_k[h] * AXBC_SPAN;
            b1 = min(a.col[c + 1], b0 + AXBC_SPAN);
        }
        const uint32_t sc = sigma[c];
        for (uint32_t base = b0; base < b1; base += 32) {
            const uint32_t e = base + lane;
            bool isnew = false;
            uint32_t r = 0, dr = 0, rdr = 0;
            if (e < b1) {
                r = a.row[e];
                int l = lvl[r];
                if (l == -1) {
                    int old = atomicCAS(&lvl[r], -1, L);
                    isnew = (old == -1);
                    l = isnew ? L : old;
                }
                if (l == L) atomicAdd(&sigma[r], sc);
                if (isnew) {
                    dr = a.col[r + 1] - a.col[r];
                    rdr = rcol[r + 1] - rcol[r];
                }
            }
            append_new(isnew, r, dr, rdr, queue, pc);
        }
    }
}

// Forward level L, pull: every unvisited vertex sums sigma over all of its
// in-neighbours at level L-1 (no early exit: every parent counts).  Tasks:
// blocks of 32 vertex ids, then the span items of heavy vertices.
__global__ void k_fwd_pull1(Adj rv, const uint32_t *__restrict__ fcol, int32_t *lvl,
                            uint32_t *sigma, uint32_t *queue, PivotCounters *pc, int L)
{
    const unsigned lane = lane_id();
    const uint64_t n = rv.n;
    const uint64_t nblk = (n + 31) / 32;
    const uint64_t ntask = nblk + rv.n_heavy_items;
    const uint64_t nw = (uint64_t)gridDim.x * blockDim.x / 32;
    for (uint64_t t = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32; t < ntask; t += nw) {
        if (t < nblk) {
            const uint64_t u_l = t * 32 + lane;
            bool cand = false;
            if (u_l < n && lvl[u_l] == -1) {
                uint32_t d = rv.col[u_l + 1] - rv.col[u_l];
                cand = d > 0 && d <= AXBC_SPAN;
            }
            unsigned act = __ballot_sync(FULL_MASK, cand);
            bool mine_new = false;
            uint32_t mine_sigma = 0;
            while (act) {
                const int j = __ffs(act) - 1;
                act &= act - 1;
                const uint32_t u = (uint32_t)(t * 32 + j);
                const uint32_t b0 = rv.col[u], b1 = rv.col[u + 1];
                uint32_t acc = 0;
                bool found = false;
                for (uint32_t e = b0 + lane; e < b1; e += 32) {
                    const uint32_t v = rv.row[e];
                    if (lvl[v] == L - 1) {
                        acc += sigma[v];
                        found = true;
                    }
                }
                acc = __reduce_add_sync(FULL_MASK, acc);
                const bool any = __any_sync(FULL_MASK, found);
                if ((int)lane == j) {
                    mine_new = any;
                    mine_sigma = acc;
                }
            }
            if (mine_new) {
                lvl[u_l] = L;
                sigma[u_l] = mine_sigma;
            }
            uint32_t dr = 0, rdr = 0;
            if (mine_new) {
                dr = fcol[u_l + 1] - fcol[u_l];
                rdr = rv.col[u_l + 1] - rv.col[u_l];
            }
            append_new(mine_new, (uint32_t)u_l, dr, rdr, queue, pc);
        } else {
            const uint64_t h = t - nblk;
            const uint32_t u = rv.hitem_v[h];
            const int lu = lvl[u];
            if (lu != -1 && lu != L) continue;
            const uint32_t b0 = rv.col[u] + rv.hitem_k[h] * AXBC_SPAN;
            const uint32_t b1 = min(rv.col[u + 1], b0 + AXBC_SPAN);
            uint32_t acc = 0;
            bool found = false;
            for (uint32_t e = b0 + lane; e < b1; e += 32) {
                const uint32_t v = rv.row[e];
                if (lvl[v] == L - 1) {
                    acc += sigma[v];
                    found = true;
                }
            }
            acc = __reduce_add_sync(FULL_MASK, acc);
            const bool any = __any_sync(FULL_MASK, found);
            bool isnew = false;
            if (any && lane == 0) {
                atomicAdd(&sigma[u], acc);
                isnew = atomicCAS(&lvl[u], -1, L) == -1;
            }
            uint32_t dr = 0, rdr = 0;
            if (isnew) {
                dr = fcol[u + 1] - fcol[u];
                rdr = rv.col[u + 1] - rv.col[u];
            }
            append_new(isnew, u, dr, rdr, queue, pc);
        }
    }
}

// Backward depth d (scan_frt_mono, src/cuda_kernels.cu:719-772): tasks
// [0,nseg) are the light vertices of the depth, then heavy span items whose
// partial sums go to partial[item].
__global__ void k_bwd1(Adj a, const uint32_t *__restrict__ queue, uint32_t ls, uint32_t nseg,
                       const int32_t *__restrict__ lvl, const uint32_t *__restrict__ sigma,
                       float *delta, const uint32_t *__restrict__ reach, float *partial, int d)
{
    const unsigned lane = lane_id();
    const uint64_t ntask = nseg + a.n_heavy_items;
    const uint64_t nw = (uint64_t)gridDim.x * blockDim.x / 32;
    for (uint64_t t = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32; t < ntask; t += nw) {
        uint32_t c, b0, b1;
        const bool light = t < nseg;
        if (light) {
            c = queue[ls + t];
            b0 = a.col[c];
            b1 = a.col[c + 1];
            if (b1 - b0 > AXBC_SPAN) continue;
        } else {
            const uint64_t h = t - nseg;
            c = a.hitem_v[h];
            if (lvl[c] != d) continue;
            b0 = a.col[c] + a.hitem_k[h] * AXBC_SPAN;
            b1 = min(a.col[c + 1], b0 + AXBC_SPAN);
        }
        const float sc = __uint2float_rn(sigma[c]);
        float P = 0.0f;
        for (uint32_t base = b0; base < b1; base += 32) {
            const uint32_t e = base + lane;
            float tl = 0.0f;
            bool succ = false;
            if (e < b1) {
                const uint32_t r = a.row[e];
                if (lvl[r] == d + 1) {
                    succ = true;
                    tl = dep_term(delta[r], sigma[r], sc);
                }
            }
            if (!__any_sync(FULL_MASK, succ)) continue;
            P = __fadd_rn(P, warp_tree_sum(tl));
        }
        if (lane == 0) {
            if (light) delta[c] = __fadd_rn(__uint2float_rn(reach[c]), P);
            else partial[t - nseg] = P;
        }
    }
}

// heavy vertices of depth d: reach + span partials, in span order
__global__ void k_bwd_combine1(Adj a, const int32_t *__restrict__ lvl, float *delta,
                               const uint32_t *__restrict__ reach, const float *__restrict__ partial,
                               int d)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n_heavy;
         i += gridDim.x * blockDim.x) {
        const uint32_t v = a.heavy_v[i];
        if (lvl[v] != d) continue;
        float acc = __uint2float_rn(reach[v]);
        for (uint32_t k = a.heavy_first[i]; k < a.heavy_first[i + 1]; k++)
            acc = __fadd_rn(acc, partial[k]);
        delta[v] = acc;
    }
}

// pre_update_bc_cuda (src/cuda_kernels.cu:339-373): sum of reach over lvl > 0
__global__ void k_reach_sum1(const int32_t *__restrict__ lvl, const uint32_t *__restrict__ reach,
                             uint64_t n, PivotCounters *pc)
{
    unsigned long long s = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
         v += (uint64_t)gridDim.x * blockDim.x)
        if (lvl[v] > 0) s += reach[v];
    s = __reduce_add_sync(FULL_MASK, (unsigned)s);
    if (lane_id() == 0 && s) atomicAdd(&pc->reach_sum, s);
}

// update_bc (src/cuda_kernels.cu:269-286), applied to every vertex.  The
// root term uses nvt = nvt_base (+ all, when add_all: all = reach_v0, plus
// the reach sum when add_sum), all in uint32 as in bc_func_mono.
__global__ void k_update1(float *bc, const float *__restrict__ delta, uint64_t n, uint32_t v0,
                          double p, const uint32_t *__restrict__ reach_v0_ptr,
                          unsigned long long nvt_base, const PivotCounters *__restrict__ pc,
                          int add_all, int add_sum)
{
    const uint32_t reach_v0 = *reach_v0_ptr;
    uint32_t all = 0;
    if (add_all) all = (add_sum ? (uint32_t)pc->reach_sum : 0u) + reach_v0;
    const unsigned long long nvt = nvt_base + all;
    const InvSplit iv = inv_split(p);
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
         v += (uint64_t)gridDim.x * blockDim.x) {
        if (v == v0) {
            if (reach_v0 > 0) bc[v] = __fadd_rn(bc[v], bc_root_term(reach_v0, nvt));
            continue;
        }
        const float dv = delta[v];
        if (dv == 0.0f && p > 0.0) continue;  // x + float(0/p) == x
        bc[v] = __fadd_rn(bc[v], bc_term_fast(dv, reach_v0, p, iv));
    }
}

__global__ void k_set_root1(uint32_t v0, int level, uint32_t sig, int32_t *lvl, uint32_t *sigma,
                            uint32_t *queue, PivotCounters *pc, const uint32_t *col,
                            const uint32_t *rcol)
{
    lvl[v0] = level;
    sigma[v0] = sig;
    queue[0] = v0;
    pc->qtail = 1;
    pc->newdeg = col[v0 + 1] - col[v0];
    pc->reach_sum = 0;
    pc->visited_rdeg = rcol[v0 + 1] - rcol[v0];
}

int axbc_ensure_single(axbc_ctx *c)
{
    if (c->single_ready) return AXBC_OK;
    const uint64_t n = c->g->n;
    ALLOC_MISSING(c->lvl, n * 4, &c->bytes);
    ALLOC_MISSING(c->sigma, n * 4, &c->bytes);
    ALLOC_MISSING(c->delta, n * 4, &c->bytes);
    ALLOC_MISSING(c->queue, (n + 1) * 4, &c->bytes);
    ALLOC_MISSING(c->partial, (c->g->fwd.n_heavy_items + 1) * 4, &c->bytes);
    ALLOC_MISSING(c->pc, sizeof(PivotCounters), &c->bytes);
    if (!c->pc_host) CU(cudaMallocHost((void **)&c->pc_host, sizeof(PivotCounters)));
    CU(cudaMemset(c->pc, 0, sizeof(PivotCounters)));
    c->single_ready = true;
    return AXBC_OK;
}

// setcuda (src/cuda_kernels.cu:1532-1554): levels unset, sigma 0, delta = reach
int axbc_single_reset(axbc_ctx *c)
{
    TRY(axbc_ensure_single(c));
    ProfScope ps(c, KP_PLAIN_OTHER, (double)c->g->n * 16.0);
    k_reset1<<<axbc_grid_for(c, 256, 8), 256, 0, c->stream>>>(c->lvl, c->sigma, c->delta,
                                                             c->g->reach, c->g->n);
    CU_LAUNCH("k_reset1");
    return AXBC_OK;
}

// set_mlp_cuda (:862-876) for the root: level, sigma, queue[0]; counters
int axbc_single_set_root(axbc_ctx *c, uint32_t v0, int level, uint32_t sig)
{
    cudaStream_t s = c->stream;
    {
        ProfScope ps(c, KP_PLAIN_OTHER, 0);
        k_set_root1<<<1, 1, 0, s>>>(v0, level, sig, c->lvl, c->sigma, c->queue, c->pc,
                                    c->g->fwd.col, c->g->rev.col);
    }
    CU_LAUNCH("k_set_root1");
    CU(cudaMemcpyAsync(c->pc_host, c->pc, sizeof(PivotCounters), cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    c->s_front_deg = c->pc_host->newdeg;
    c->s_prev_newdeg = c->pc_host->newdeg;
    c->s_visited_rdeg = c->pc_host->visited_rdeg;
    c->level_te.assign(1, (double)c->pc_host->newdeg);
    return AXBC_OK;
}

// One forward level (scan_col_csc_cuda_mono, src/cuda_kernels.cu:1088-1177):
// the frontier is queue[qs, qs+nf); new vertices are appended after it.
int axbc_single_forward_level(axbc_ctx *c, uint32_t qs, uint32_t nf, int level, uint64_t *nfrt)
{
    axbc_graph *g = c->g;
    cudaStream_t s = c->stream;
    const int grid = axbc_grid_for(c, 256, 8);
    const uint32_t tail = qs + nf;
    CU(cudaMemcpyAsync(&c->pc->qtail, &tail, 4, cudaMemcpyHostToDevice, s));
    const uint64_t unvisited = g->m - c->s_visited_rdeg;
    const bool push = (double)c->s_front_deg * c->push_factor_single < (double)unvisited;
    {
        ProfScope ps(c, KP_PLAIN_FWD, (double)c->s_front_deg * 8.0);
        if (push) k_fwd_push1<<<grid, 256, 0, s>>>(g->fwd, g->rev.col, qs, nf, c->lvl, c->sigma,
                                                  c->queue, c->pc, level);
        else k_fwd_pull1<<<grid, 256, 0, s>>>(g->rev, g->fwd.col, c->lvl, c->sigma, c->queue,
                                             c->pc, level);
    }
    CU_LAUNCH("forward level");
    CU(cudaMemcpyAsync(c->pc_host, c->pc, sizeof(PivotCounters), cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    *nfrt = c->pc_host->qtail - tail;
    c->s_front_deg = c->pc_host->newdeg - c->s_prev_newdeg;
    c->s_prev_newdeg = c->pc_host->newdeg;
    c->s_visited_rdeg = c->pc_host->visited_rdeg;
    c->level_te.push_back((double)c->s_front_deg);
    return AXBC_OK;
}

// One backward depth (scan_frt_csc_cuda_mono, src/cuda_kernels.cu:1013-1080)
// over the vertices queue[ls, ls+nseg) at depth d.
int axbc_single_backward_level(axbc_ctx *c, uint32_t ls, uint32_t nseg, int d)
{
    axbc_graph *g = c->g;
    cudaStream_t s = c->stream;
    const double te = d >= 0 && d < (int)c->level_te.size() ? c->level_te[d] : 0.0;
    {
        ProfScope ps(c, KP_PLAIN_BWD, te * 12.0);
        k_bwd1<<<axbc_grid_for(c, 256, 8), 256, 0, s>>>(g->fwd, c->queue, ls, nseg, c->lvl,
                                                       c->sigma, c->delta, g->reach, c->partial, d);
    }
    if (g->fwd.n_heavy) {
        ProfScope ps(c, KP_PLAIN_BWD, 0);
        k_bwd_combine1<<<(g->fwd.n_heavy + 255) / 256, 256, 0, s>>>(g->fwd, c->lvl, c->delta,
                                                                   g->reach, c->partial, d);
    }
    CU_LAUNCH("backward level");
    return AXBC_OK;
}

// sum of reach over vertices with level > 0 into pc->reach_sum
int axbc_single_reach_sum(axbc_ctx *c)
{
    CU(cudaMemsetAsync(&c->pc->reach_sum, 0, 8, c->stream));
    ProfScope ps(c, KP_PLAIN_OTHER, (double)c->g->n * 8.0);
    k_reach_sum1<<<axbc_grid_for(c, 256, 8), 256, 0, c->stream>>>(c->lvl, c->g->reach, c->g->n, c->pc);
    CU_LAUNCH("reach sum");
    return AXBC_OK;
}

int axbc_single_update(axbc_ctx *c, uint32_t v0, double p, const uint32_t *reach_v0_dev,
                       uint64_t nvt_base, int add_all, int add_sum)
{
    {
        ProfScope ps(c, KP_PLAIN_OTHER, (double)c->g->n * 12.0);
        k_update1<<<axbc_grid_for(c, 256, 8), 256, 0, c->stream>>>(
            c->bc, c->delta, c->g->n, v0, p, reach_v0_dev, nvt_base, c->pc, add_all, add_sum);
    }
    CU_LAUNCH("update");
    c->delta_last_valid = false;  // the last pivot's delta is c->delta
    return AXBC_OK;
}

// ------------------------------------------- a pivot in one launch
#define PIVOT_TPB 256
#define PIVOT_BPS 4
#define PIVOT_NW (PIVOT_TPB / 32)
// Reset, forward levels, backward depths and the update with a grid barrier
// between them: one per level and depth.  The level-by-level form spent 200 us
// on a graph of a thousand vertices, most of it between a dozen launches and
// six waits of the host, and 500 us on a scale-18 pivot, where a span of 1024
// positions sat on one warp.  Here big vertices are split as in the batched
// passes (Adj::part forward, Adj::tile backward), small ones share a warp, and
// lanes are adjacency positions; work goes round the warps in fixed strides.
struct PivotCtl {
    GridSync gs;
    uint32_t qtail, pad;
    unsigned long long newdeg, rdeg, rsum;  // of every vertex reached
    unsigned long long prev_newdeg;
    int32_t alive, push, levels, pad2;
};

struct PivotRun {
    int32_t *lvl;
    uint32_t *sigma;
    float *delta, *q;
    uint32_t *queue, *lev;
    float *partial;
    uint32_t *arrive;
    const uint32_t *reach;
    float *bc;
    PivotCtl *ctl;
    uint64_t n, m;
    uint32_t v0;
    int H;
    double p, push_factor;
    // a pass of one pivot: the root comes from bi, its totals and the level
    // tables go there, and the update is left to k_one_update
    BatchInfo *bi;
    unsigned long long *level_te, *level_cnt;
    int32_t *level_mode;
};

// what a thread has discovered in a level
struct Found {
    unsigned long long deg = 0, rdeg = 0, rsum = 0;
    __device__ __forceinline__ void flush(PivotCtl *ctl)
    {
        if (!__any_sync(FULL_MASK, deg | rdeg | rsum)) return;
        for (int o = 16; o; o >>= 1) {
            deg += __shfl_xor_sync(FULL_MASK, deg, o);
            rdeg += __shfl_xor_sync(FULL_MASK, rdeg, o);
            rsum += __shfl_xor_sync(FULL_MASK, rsum, o);
        }
        if (lane_id() == 0) {
            atomicAdd(&ctl->newdeg, deg);
            atomicAdd(&ctl->rdeg, rdeg);
            if (rsum) atomicAdd(&ctl->rsum, rsum);
        }
    }
};

// the lanes' new vertices go to the queue
__device__ __forceinline__ void pivot_found(const Adj &a, const Adj &rv, const PivotRun &R, bool isnew, uint32_t r,
                                            Found &fnd)
{
    const unsigned m = __ballot_sync(FULL_MASK, isnew), lane = lane_id();
    if (!m) return;
    const int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if ((int)lane == leader) base = atomicAdd(&R.ctl->qtail, (uint32_t)__popc(m));
    base = __shfl_sync(FULL_MASK, base, leader);
    if (!isnew) return;
    R.queue[base + __popc(m & ((1u << lane) - 1u))] = r;
    fnd.deg += a.col[r + 1] - a.col[r];
    fnd.rdeg += rv.col[r + 1] - rv.col[r];
    if (R.H) fnd.rsum += R.reach[r];
}

// one edge per lane from a vertex at depth L-1 with sc paths (in: a real edge)
__device__ __forceinline__ void pivot_push(const Adj &a, const Adj &rv, const PivotRun &R, bool in, uint32_t e,
                                           uint32_t sc, int L, Found &fnd)
{
    bool isnew = false;
    uint32_t r = 0;
    if (in) {
        r = a.row[e];
        int l = R.lvl[r];
        if (l == -1) {
            const int old = atomicCAS(&R.lvl[r], -1, L);
            isnew = old == -1;
            l = isnew ? L : old;
        }
        if (l == L) atomicAdd(&R.sigma[r], sc);
    }
    pivot_found(a, rv, R, isnew, r, fnd);
}

__device__ __forceinline__ uint32_t stride_unit(uint64_t items, uint64_t nw)
{
    return (uint32_t)max((uint64_t)1, min((uint64_t)32, items / nw));
}

__device__ __forceinline__ void pivot_push_level(const Adj &a, const Adj &rv, const PivotRun &R, uint32_t qs,
                                                 uint32_t nf, int L)
{
    const unsigned lane = lane_id();
    const uint64_t nw = (uint64_t)gridDim.x * blockDim.x / 32;
    const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32;
    Found fnd;
    const uint32_t gp = stride_unit(a.n_part, nw), ent = stride_unit(nf, nw);
    const uint64_t up = (a.n_part + gp - 1) / gp;
    for (uint64_t t = w; t < up; t += nw) {
        const uint64_t i = lane * up + t;  // a hub's parts fall into different units
        uint32_t b_l = 0, n_l = 0, s_l = 0;
        bool on = false;
        if (lane < gp && i < a.n_part) {
            const uint2 pt = a.part[i];
            on = R.lvl[pt.x] == L - 1;
            if (on) {
                b_l = a.col[pt.x] + pt.y * a.part_len;
                n_l = min(a.col[pt.x + 1] - b_l, a.part_len);
                s_l = R.sigma[pt.x];
            }
        }
        for (unsigned act = __ballot_sync(FULL_MASK, on); act; act &= act - 1) {
            const int j = __ffs(act) - 1;
            const uint32_t b0 = __shfl_sync(FULL_MASK, b_l, j), len = __shfl_sync(FULL_MASK, n_l, j);
            const uint32_t sc = __shfl_sync(FULL_MASK, s_l, j);
            for (uint32_t o = lane; o - lane < len; o += 32) pivot_push(a, rv, R, o < len, b0 + o, sc, L, fnd);
        }
    }
    // the frontier's other vertices: up to 32 adjacency lists walked as one
    const uint64_t uq = (nf + ent - 1) / ent;
    for (uint64_t t = w; t < uq; t += nw) {
        const uint64_t i = t * ent + lane;
        uint32_t b = 0, d = 0, sc = 0;
        if (lane < ent && i < nf) {
            const uint32_t v = R.queue[qs + i];
            b = a.col[v];
            d = a.col[v + 1] - b;
            if (d > a.big) d = 0;
            else sc = R.sigma[v];
        }
        uint32_t inc = d;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(FULL_MASK, inc, o);
            if ((int)lane >= o) inc += x;
        }
        const uint32_t total = __shfl_sync(FULL_MASK, inc, 31), shift = b - (inc - d);
        for (uint32_t base = 0; base < total; base += 32) {
            const uint32_t e = base + lane;
            uint32_t k = 0;
#pragma unroll
            for (int step = 16; step; step >>= 1)
                if (__shfl_sync(FULL_MASK, inc, k + step - 1) <= e) k += step;
            const uint32_t pos = __shfl_sync(FULL_MASK, shift, k) + e, sk = __shfl_sync(FULL_MASK, sc, k);
            pivot_push(a, rv, R, e < total, pos, sk, L, fnd);
        }
    }
    fnd.flush(R.ctl);
}

// path counts of the parents among positions e, e + step, ... (four of them,
// below end) of a list, their entries, levels and counts loaded together: one
// entry at a time a lane spent three dependent loads on each (a pivot of the
// 1024^2 mesh 5.8 ms, four together 4.3; scale 20 0.93 and 0.80 ms)
__device__ __forceinline__ void pivot_parents(const PivotRun &R, const uint32_t *__restrict__ row, uint32_t e,
                                              uint32_t step, uint32_t end, int L, uint32_t &acc, bool &found)
{
    uint32_t v[4], x[4];
    bool on[4];
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = e + step * i < end ? row[e + step * i] : 0xffffffffu;
#pragma unroll
    for (int i = 0; i < 4; i++) on[i] = v[i] != 0xffffffffu && R.lvl[v[i]] == L - 1;
#pragma unroll
    for (int i = 0; i < 4; i++) x[i] = on[i] ? R.sigma[v[i]] : 0u;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        acc += x[i];
        found |= on[i];
    }
}

// Pull: a part of a big unvisited vertex per warp, the others by eight lanes
// each (no early exit: every parent counts).
__device__ __forceinline__ void pivot_pull_level(const Adj &a, const Adj &rv, const PivotRun &R, int L)
{
    const unsigned lane = lane_id();
    const uint64_t nw = (uint64_t)gridDim.x * blockDim.x / 32;
    const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32;
    Found fnd;
    const uint64_t np = rv.n_part, nl = rv.n_linked - rv.n_big;
    const uint32_t gp = stride_unit(np, nw), gl = max(4u, stride_unit(nl, 4 * nw));
    const uint64_t up = (np + gp - 1) / gp, ul = (nl + gl - 1) / gl;
    for (uint64_t t = w; t < up; t += nw) {
        const uint64_t i = lane * up + t;
        uint32_t u_l = 0, b_l = 0, n_l = 0, acc_l = 0;
        bool on = false;
        if (lane < gp && i < np) {
            const uint2 pt = rv.part[i];
            u_l = pt.x;
            const int l = R.lvl[u_l];
            on = l == -1 || l == L;  // another part may have claimed it already
            b_l = rv.col[u_l] + pt.y * rv.part_len;
            n_l = min(rv.col[u_l + 1] - b_l, rv.part_len);
        }
        bool hit = false;
        for (unsigned act = __ballot_sync(FULL_MASK, on); act; act &= act - 1) {
            const int j = __ffs(act) - 1;
            const uint32_t b0 = __shfl_sync(FULL_MASK, b_l, j), len = __shfl_sync(FULL_MASK, n_l, j);
            uint32_t acc = 0;
            bool found = false;
            for (uint32_t o = 0; o < len; o += 128) pivot_parents(R, rv.row + b0, o + lane, 32, len, L, acc, found);
            if (!__any_sync(FULL_MASK, found)) continue;
            acc = __reduce_add_sync(FULL_MASK, acc);
            if ((int)lane == j) {
                acc_l = acc;
                hit = true;
            }
        }
        bool isnew = false;
        if (hit) {
            atomicAdd(&R.sigma[u_l], acc_l);
            isnew = atomicCAS(&R.lvl[u_l], -1, L) == -1;
        }
        pivot_found(a, rv, R, isnew, u_l, fnd);
    }
    // The order is by degree: the warps that got one part fewer above get the
    // unit of larger lists here, and four units a warp even out the rest (a
    // pivot at scale 18: 330 us, 303 so).
    const int sl = lane & 7, g = lane >> 3;
    for (uint64_t t = nw - 1 - w; t < ul; t += nw) {
        const uint64_t i = t * gl + lane;
        uint32_t u_l = 0, b_l = 0, d_l = 0, acc_l = 0;
        bool cand = false;
        if (lane < gl && i < nl) {
            u_l = rv.order[rv.n_big + i];
            cand = R.lvl[u_l] == -1;
            b_l = rv.col[u_l];
            d_l = rv.col[u_l + 1] - b_l;
        }
        bool hit = false;
        for (unsigned act = __ballot_sync(FULL_MASK, cand); act;) {
            int j4[4], j = -1;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                j4[k] = act ? __ffs(act) - 1 : -1;
                if (k == g) j = j4[k];
                act &= act - 1;
            }
            const uint32_t b = __shfl_sync(FULL_MASK, b_l, j & 31), dj = __shfl_sync(FULL_MASK, d_l, j & 31);
            const uint32_t d = j < 0 ? 0u : dj;
            uint32_t acc = 0;
            bool found = false;
            for (uint32_t o = sl; o < d; o += 32) pivot_parents(R, rv.row + b, o, 8, d, L, acc, found);
            const unsigned any = __ballot_sync(FULL_MASK, found);
            if (!any) continue;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) acc += __shfl_xor_sync(FULL_MASK, acc, o);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t x = __shfl_sync(FULL_MASK, acc, 8 * k);
                if ((int)lane == j4[k] && (any >> (8 * k) & 0xffu)) {
                    acc_l = x;
                    hit = true;
                }
            }
        }
        if (hit) {
            R.lvl[u_l] = L;
            R.sigma[u_l] = acc_l;
        }
        pivot_found(a, rv, R, hit, u_l, fnd);
    }
    fnd.flush(R.ctl);
}

// delta of v at its depth, and what its parents multiply by their path counts
__device__ __forceinline__ void pivot_dep(const PivotRun &R, uint32_t v, float delta)
{
    R.delta[v] = delta;
    R.q[v] = __fdiv_rn(__fadd_rn(delta, 1.0f), __uint2float_rn(R.sigma[v]));
}

// the terms of NC chunks, their loads together, and the chunks' tree sums
template <int NC>
__device__ __forceinline__ void pivot_chunks(const PivotRun &R, const uint32_t r[NC], const bool in[NC], int d,
                                             const float sc[NC], float sum[NC])
{
    int l[NC];
    float x[NC];
#pragma unroll
    for (int i = 0; i < NC; i++) l[i] = in[i] ? R.lvl[r[i]] : -1;
#pragma unroll
    for (int i = 0; i < NC; i++) x[i] = l[i] == d + 1 ? R.q[r[i]] : 0.0f;
#pragma unroll
    for (int i = 0; i < NC; i++) sum[i] = warp_tree_sum(l[i] == d + 1 ? __fmul_rn(x[i], sc[i]) : 0.0f);
}

// Backward depth d over the vertices queue[ls, ls + cnt): the canonical sum.
__device__ __forceinline__ void pivot_bwd_depth(const Adj &a, const PivotRun &R, uint32_t ls, uint32_t cnt, int d,
                                                float (*csum)[BWD_TILE_CHUNKS])
{
    constexpr int NC = BWD_TILE_CHUNKS / PIVOT_NW;  // chunks per warp of a tile
    constexpr int NL = 4;                           // and of a list read at once
    const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
    // tiles of the big vertices, each by a block: chunk sums in shared memory
    int buf = 0;
    for (uint64_t base = blockIdx.x; base < a.n_tile; base += 32ull * gridDim.x) {
        const uint64_t t_l = base + (uint64_t)lane * gridDim.x;
        uint2 tl_l = make_uint2(0, 0);
        bool any = false;
        if (t_l < a.n_tile) {
            tl_l = a.tile[t_l];
            const uint32_t c = tl_l.y & BWD_SPAN_TILE ? 1u : tl_l.y;
            for (uint32_t j = 0; j < c; j++) any |= R.lvl[a.order[tl_l.x + j]] == d;
        }
        for (unsigned act = __ballot_sync(FULL_MASK, any); act; act &= act - 1, buf ^= 1) {
            const int ja = __ffs(act) - 1;
            const uint64_t t = base + (uint64_t)ja * gridDim.x;
            const uint2 tl = make_uint2(__shfl_sync(FULL_MASK, tl_l.x, ja), __shfl_sync(FULL_MASK, tl_l.y, ja));
            const bool span = (tl.y & BWD_SPAN_TILE) != 0;
            const uint32_t k = span ? tl.y & ~BWD_SPAN_TILE : 0u, c = span ? 1u : tl.y;
            uint32_t v_l = 0, b_l = 0, e_l = 0, c_l = 0;
            float s_l = 0.0f;
            if (lane < c) {
                v_l = a.order[tl.x + lane];
                if (R.lvl[v_l] == d) {
                    b_l = a.col[v_l] + k * AXBC_SPAN;
                    e_l = min(a.col[v_l + 1], b_l + AXBC_SPAN);
                    c_l = (e_l - b_l + AXBC_CHUNK - 1) / AXBC_CHUNK;
                    s_l = __uint2float_rn(R.sigma[v_l]);
                }
            }
            uint32_t inc = c_l;
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) {
                const uint32_t x = __shfl_up_sync(FULL_MASK, inc, o);
                if ((int)lane >= o) inc += x;
            }
            const uint32_t S = __shfl_sync(FULL_MASK, inc, 15);
            uint32_t r[NC];
            bool in[NC];
            float sc[NC], sum[NC];
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const uint32_t s = wid + PIVOT_NW * i;
                const int j = __popc(__ballot_sync(FULL_MASK, lane < 16 && inc <= s)) & 31;
                const uint32_t e = __shfl_sync(FULL_MASK, b_l + AXBC_CHUNK * (s - (inc - c_l)), j) + lane;
                const uint32_t end = __shfl_sync(FULL_MASK, e_l, j);
                sc[i] = __shfl_sync(FULL_MASK, s_l, j);
                in[i] = s < S && e < end;
                r[i] = in[i] ? a.row[e] : 0u;
            }
            pivot_chunks<NC>(R, r, in, d, sc, sum);
#pragma unroll
            for (int i = 0; i < NC; i++)
                if (lane == 0 && wid + PIVOT_NW * i < S) csum[buf][wid + PIVOT_NW * i] = sum[i];
            __syncthreads();
            // one lane per vertex adds its chunks
            if (wid == 0 && c_l) {
                float P = 0.0f;
                for (uint32_t s = inc - c_l; s < inc; s++) P = __fadd_rn(P, csum[buf][s]);
                if (!span) {
                    pivot_dep(R, v_l, __fadd_rn(__uint2float_rn(R.reach[v_l]), P));
                } else {
                    R.partial[t] = P;
                    __threadfence();
                    const uint32_t spans = (a.col[v_l + 1] - a.col[v_l] + AXBC_SPAN - 1) / AXBC_SPAN;
                    if (atomicAdd(&R.arrive[tl.x], 1u) == spans - 1) {
                        // the last span to arrive adds them in span order
                        R.arrive[tl.x] = 0;
                        __threadfence();
                        const float *part = R.partial + (t - k);
                        float acc = __uint2float_rn(R.reach[v_l]);
                        for (uint32_t i = 0; i < spans; i += 8) {
                            float x[8];
#pragma unroll
                            for (int q = 0; q < 8; q++) x[q] = i + q < spans ? __ldcg(part + i + q) : 0.0f;
#pragma unroll
                            for (int q = 0; q < 8; q++)
                                if (i + q < spans) acc = __fadd_rn(acc, x[q]);
                        }
                        pivot_dep(R, v_l, acc);
                    }
                }
            }
        }
    }
    // the others by warps: chunks of 32 four at once, of at most 8 neighbours
    // four vertices to a chunk
    const uint64_t nw = (uint64_t)gridDim.x * blockDim.x / 32;
    const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32;
    const uint32_t ent = stride_unit(cnt, nw);
    const int l8 = lane & 7, g = lane >> 3;
    for (uint64_t t = w; t < (cnt + ent - 1) / ent; t += nw) {
        const uint64_t i = t * ent + lane;
        uint32_t v_l = 0, b_l = 0, d_l = 0xffffffffu, r_l = 0;
        float s_l = 0.0f, P_l = 0.0f;
        if (lane < ent && i < cnt) {
            v_l = R.queue[ls + i];
            b_l = a.col[v_l];
            d_l = a.col[v_l + 1] - b_l;
            s_l = __uint2float_rn(R.sigma[v_l]);
            r_l = R.reach[v_l];
        }
        // NL chunks at once, of whichever vertices
        const uint32_t c_l = d_l > 8 && d_l <= a.big ? (d_l + 31) / 32 : 0u;
        uint32_t inc = c_l;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(FULL_MASK, inc, o);
            if ((int)lane >= o) inc += x;
        }
        const uint32_t S = __shfl_sync(FULL_MASK, inc, 31);
        for (uint32_t s0 = 0; s0 < S; s0 += NL) {
            uint32_t r[NL];
            bool in[NL];
            float sc[NL], sum[NL];
            int j[NL];
#pragma unroll
            for (int q = 0; q < NL; q++) {
                const uint32_t s = s0 + q;
                j[q] = __popc(__ballot_sync(FULL_MASK, inc <= s));
                const uint32_t o = __shfl_sync(FULL_MASK, AXBC_CHUNK * (s - (inc - c_l)), j[q] & 31) + lane;
                const uint32_t d = __shfl_sync(FULL_MASK, d_l, j[q] & 31);
                const uint32_t b = __shfl_sync(FULL_MASK, b_l, j[q] & 31);
                sc[q] = __shfl_sync(FULL_MASK, s_l, j[q] & 31);
                in[q] = s < S && o < d;
                r[q] = in[q] ? a.row[b + o] : 0u;
            }
            pivot_chunks<NL>(R, r, in, d, sc, sum);
#pragma unroll
            for (int q = 0; q < NL; q++)
                if ((int)lane == j[q]) P_l = __fadd_rn(P_l, sum[q]);
        }
        for (unsigned act = __ballot_sync(FULL_MASK, d_l <= 8); act;) {
            int j4[4], j = -1;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                j4[q] = act ? __ffs(act) - 1 : -1;
                if (q == g) j = j4[q];
                act &= act - 1;
            }
            const uint32_t b0 = __shfl_sync(FULL_MASK, b_l, j & 31), dj = __shfl_sync(FULL_MASK, d_l, j & 31);
            const float sj = __shfl_sync(FULL_MASK, s_l, j & 31);
            float tl = 0.0f;
            if (j >= 0 && (uint32_t)l8 < dj) {
                const uint32_t r = a.row[b0 + l8];
                if (R.lvl[r] == d + 1) tl = __fmul_rn(R.q[r], sj);
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) tl = __fadd_rn(tl, __shfl_xor_sync(FULL_MASK, tl, o));
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float x = __shfl_sync(FULL_MASK, tl, 8 * q);
                if ((int)lane == j4[q]) P_l = x;
            }
        }
        if (d_l <= a.big) pivot_dep(R, v_l, __fadd_rn(__uint2float_rn(r_l), P_l));
    }
}

// close forward level L (one warp): its end in the queue, the next direction
struct PivotLead {
    const PivotRun &R;
    int L;
    __device__ void operator()() const
    {
        if (lane_id()) return;
        PivotCtl *c = R.ctl;
        const uint32_t tail = __ldcg(&c->qtail);
        const unsigned long long nd = __ldcg(&c->newdeg), unvis = R.m - __ldcg(&c->rdeg);
        const uint32_t from = vload_u(&R.lev[L]);
        const bool alive = tail != from;
        R.lev[L + 1] = tail;
        if (R.bi) {
            R.level_te[L] = nd - __ldcg(&c->prev_newdeg);
            R.level_cnt[L] = tail - from;
            R.level_mode[L] = vload_i(&c->push);
        }
        c->push = (double)(nd - __ldcg(&c->prev_newdeg)) * R.push_factor < (double)unvis;
        c->prev_newdeg = nd;
        // a pass whose last level would have no room in the level tables ends
        // here: refused, as in the other forms
        const bool deep = R.bi && alive && L == AXBC_MAX_LEVELS - 3;
        c->alive = alive && !deep;
        if (!alive || deep) c->levels = deep ? L + 1 : L;
    }
};

__global__ void __launch_bounds__(PIVOT_TPB, PIVOT_BPS) k_pivot(Adj a, Adj rv, PivotRun R, long long budget)
{
    __shared__ float s_csum[2][BWD_TILE_CHUNKS];
    PivotCtl *ctl = R.ctl;
    unsigned epoch = 0;
    const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint64_t nt = (uint64_t)gridDim.x * blockDim.x;
    const uint32_t v0 = R.bi ? R.bi->root[0] : R.v0;
    for (uint64_t v = tid; v < R.n; v += nt) {
        const bool root = v == v0;
        R.lvl[v] = root ? 0 : -1;
        R.sigma[v] = root ? 1u : 0u;
        R.delta[v] = __uint2float_rn(R.reach[v]);
    }
    if (tid == 0) {
        const uint32_t deg = a.col[v0 + 1] - a.col[v0], rdeg = rv.col[v0 + 1] - rv.col[v0];
        R.queue[0] = v0;
        R.lev[0] = 0;
        R.lev[1] = 1;
        ctl->qtail = 1;
        ctl->newdeg = ctl->prev_newdeg = deg;
        ctl->rdeg = rdeg;
        ctl->rsum = 0;
        ctl->alive = 1;
        ctl->push = (double)deg * R.push_factor < (double)(R.m - rdeg);
        if (R.bi) {
            BatchInfo *bi = R.bi;
            bi->nsrc = 1;
            bi->srcmask = bi->applymask = 1;
            bi->H = R.H;
            bi->root_reach[0] = R.reach[v0];
            bi->pool_short = 0;
            R.level_te[0] = deg;
            R.level_cnt[0] = 1;
        }
    }
    if (R.bi && blockIdx.x == 0)
        for (int i = threadIdx.x; i < AXBC_WMAX; i += blockDim.x) R.bi->lane_bc[i] = R.bc;
    if (!grid_barrier(&ctl->gs, budget, 1, epoch, NoLead{})) return;
    int L = 1;
    for (;; L++) {
        const uint32_t qs = vload_u(&R.lev[L - 1]), nf = vload_u(&R.lev[L]) - qs;
        if (vload_i(&ctl->push)) pivot_push_level(a, rv, R, qs, nf, L);
        else pivot_pull_level(a, rv, R, L);
        const PivotLead lead{R, L};
        if (!grid_barrier(&ctl->gs, budget, 2, epoch, lead)) return;
        if (!vload_i(&ctl->alive)) break;
    }
    if (R.bi && vload_i(&ctl->levels) != L) return;  // too deep
    // backward: the deepest vertices have delta = reach; then depths L-2 .. 1,
    // and 0 when the BFS ended at level 2
    if (L >= 2) {
        const uint32_t b0 = vload_u(&R.lev[L - 1]), b1 = vload_u(&R.lev[L]);
        for (uint64_t i = b0 + tid; i < b1; i += nt) pivot_dep(R, R.queue[i], R.delta[R.queue[i]]);
        for (int d = L - 2; d >= (L == 2 ? 0 : 1); d--) {
            if (!grid_barrier(&ctl->gs, budget, 3, epoch, NoLead{})) return;
            const uint32_t ls = vload_u(&R.lev[d]);
            pivot_bwd_depth(a, R, ls, vload_u(&R.lev[d + 1]) - ls, d, s_csum);
        }
        if (!grid_barrier(&ctl->gs, budget, 4, epoch, NoLead{})) return;
    }
    if (R.bi) {
        if (tid == 0) {
            BatchInfo *bi = R.bi;
            bi->nvis[0] = vload_u(&ctl->qtail);
            bi->rsum[0] = __ldcg(&ctl->rsum);
            bi->te[0] = __ldcg(&ctl->newdeg);
            bi->Ls[0] = L;
            bi->depth0mask = L == 2;
            bi->cur = bi->lend = L;
            bi->alive = 0;
            bi->dmax = L - 1;
        }
        return;
    }
    // update_bc (src/cuda_kernels.cu:269-286) of every vertex
    const uint32_t reach_v0 = R.reach[v0];
    const uint32_t all = (R.H ? (uint32_t)__ldcg(&ctl->rsum) : 0u) + reach_v0;
    const unsigned long long nvt = vload_u(&ctl->qtail) + (unsigned long long)all;
    const InvSplit iv = inv_split(R.p);
    for (uint64_t v = tid; v < R.n; v += nt) {
        if (v == v0) {
            if (reach_v0 > 0) R.bc[v] = __fadd_rn(R.bc[v], bc_root_term(reach_v0, nvt));
            continue;
        }
        const float dv = R.delta[v];
        if (dv == 0.0f && R.p > 0.0) continue;  // x + float(0/p) == x
        R.bc[v] = __fadd_rn(R.bc[v], bc_term_fast(dv, reach_v0, R.p, iv));
    }
}

// update_bc of a one-pivot pass into its lane's bc vector, when the replay of
// Bader's test applies it, and its dependencies as the last ones
__global__ void k_one_update(const float *__restrict__ delta, uint64_t n, const BatchInfo *__restrict__ bi,
                             float *__restrict__ delta_out)
{
    if (!(bi->applymask & 1ull)) return;
    float *bc = bi->lane_bc[0];
    const uint32_t root = bi->root[0], rr = bi->root_reach[0];
    const uint32_t all = (bi->H == 1 ? (uint32_t)bi->rsum[0] : 0u) + rr;
    const unsigned long long nvt = bi->nvis[0] + all;
    const double p = bi->p[0];
    const InvSplit iv = inv_split(p);
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
         v += (uint64_t)gridDim.x * blockDim.x) {
        const float dv = delta[v];
        if (delta_out) delta_out[v] = dv;
        if (v == root) {
            if (rr > 0) bc[v] = __fadd_rn(bc[v], bc_root_term(rr, nvt));
            continue;
        }
        if (dv == 0.0f && p > 0.0) continue;  // x + float(0/p) == x
        bc[v] = __fadd_rn(bc[v], bc_term_fast(dv, rr, p, iv));
    }
}

void axbc_pivot_free(PivotBuf &b)
{
    if (b.owns) {
        axbc_dfree(b.lvl);
        axbc_dfree(b.sigma);
        axbc_dfree(b.queue);
        axbc_dfree(b.delta);
        axbc_dfree(b.partial);
    }
    axbc_dfree(b.q);
    axbc_dfree(b.lev);
    axbc_dfree(b.arrive);
    axbc_dfree(b.ctl);
    if (b.ctl_host) cudaFreeHost(b.ctl_host);
    b = PivotBuf();
}

static int pivot_fit(axbc_ctx *c)
{
    if (!c->pivot_fit)
        CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c->pivot_fit, k_pivot, PIVOT_TPB, 0));
    return AXBC_OK;
}

// owns: with path counts, levels, dependencies and queue of its own; else those
// of the level-by-level form, which are there
static int ensure_pivot(axbc_ctx *c, PivotBuf &b, bool owns)
{
    if (b.ready) return AXBC_OK;
    const uint64_t n = c->g->n;
    b.owns = owns;
    if (owns) {
        ALLOC_MISSING(b.lvl, n * 4, &c->bytes);
        ALLOC_MISSING(b.sigma, n * 4, &c->bytes);
        ALLOC_MISSING(b.queue, (n + 1) * 4, &c->bytes);
        ALLOC_MISSING(b.delta, n * 4, &c->bytes);
        ALLOC_MISSING(b.partial, (c->g->fwd.n_heavy_items + 1) * 4, &c->bytes);
    } else {
        b.lvl = c->lvl;
        b.sigma = c->sigma;
        b.queue = c->queue;
        b.delta = c->delta;
        b.partial = c->partial;
    }
    ALLOC_MISSING(b.q, n * 4, &c->bytes);
    ALLOC_MISSING(b.lev, (n + 2) * 4, &c->bytes);
    ALLOC_MISSING(b.arrive, (c->g->fwd.n_heavy + 1) * 4, &c->bytes);
    ALLOC_MISSING(b.ctl, sizeof(PivotCtl), &c->bytes);
    if (!b.ctl_host) CU(cudaMallocHost((void **)&b.ctl_host, sizeof(PivotCtl)));
    CU(cudaMemsetAsync(b.arrive, 0, (c->g->fwd.n_heavy + 1) * 4, c->stream));
    b.ready = true;
    return AXBC_OK;
}

// The same, but *room = false (and no further tries) when only the one launch's
// buffers find no room: the caller has a form that does without them.
static int pivot_room(axbc_ctx *c, PivotBuf &b, bool owns, bool *room)
{
    const int rc = !b.ready && c->pivot_short ? AXBC_ERR_NOMEM : ensure_pivot(c, b, owns);
    *room = rc == AXBC_OK;
    if (rc == AXBC_ERR_NOMEM) c->pivot_short = true;
    return rc == AXBC_ERR_NOMEM ? AXBC_OK : rc;
}

// One launch of k_pivot; its control block on the way to b.ctl_host.  *done =
// false: the device refuses it.
static int pivot_launch(axbc_ctx *c, PivotBuf &b, PivotRun &R, bool *done)
{
    axbc_graph *g = c->g;
    cudaStream_t s = c->stream;
    R.lvl = b.lvl;
    R.sigma = b.sigma;
    R.delta = b.delta;
    R.q = b.q;
    R.queue = b.queue;
    R.lev = b.lev;
    R.partial = b.partial;
    R.arrive = b.arrive;
    R.reach = g->reach;
    R.bc = c->bc;
    R.ctl = b.ctl;
    R.n = g->n;
    R.m = g->m;
    R.push_factor = c->push_factor_single;
    long long budget = AXBC_BAR_BUDGET;
    // Blocks per SM: two where the levels are short or narrow and a barrier
    // waits for every block, else four; or as many as have work.  Measured, us a
    // pivot with 1, 2, 4: scale 14 121, 115, 126, scale 18 548, 382, 318, scale 22
    // 7158, 3973, 2685, 256^2 grid 2472, 2695, 3327, 1024^2 grid 4336, 4271, 5290.
    const int want = g->m < (1ull << 19) || g->max_deg <= 64 ? 2 : PIVOT_BPS;
    const uint64_t work = std::max<uint64_t>(std::max<uint64_t>(g->fwd.n_part, g->rev.n_part) +
                                                 std::max(g->fwd.n_linked, g->rev.n_linked),
                                             g->n / 32);
    const int grid = (int)std::max<uint64_t>(
        1, std::min<uint64_t>((uint64_t)axbc_grid_for(c, PIVOT_TPB, std::min(want, c->pivot_fit)),
                              (work + PIVOT_NW - 1) / PIVOT_NW));
    CU(cudaMemsetAsync(b.ctl, 0, sizeof(GridSync), s));
    void *args[] = {(void *)&g->fwd, (void *)&g->rev, (void *)&R, (void *)&budget};
    TRY(axbc_coop_launch(c, (const void *)k_pivot, grid, PIVOT_TPB, args, done));
    if (!*done) return AXBC_OK;
    CU_LAUNCH("k_pivot");
    CU(cudaMemcpyAsync(b.ctl_host, b.ctl, sizeof(PivotCtl), cudaMemcpyDeviceToHost, s));
    return AXBC_OK;
}

// *site: the barrier whose wait ran out, or 0
static int pivot_wait(axbc_ctx *c, PivotBuf &b, int *site)
{
    CU(cudaStreamSynchronize(c->stream));
    return axbc_wait_ran_out(c, b.ctl_host->gs.err, b.arrive, c->g->fwd.n_heavy + 1, site);
}

bool axbc_one_fits(axbc_ctx *c, int *rc)
{
    *rc = pivot_fit(c);
    return *rc == AXBC_OK && c->coop && c->pivot_fit > 0;
}

// *done = false: no room for its buffers, no cooperative launch, or a barrier
// wait that ran out; the root in c->bi is as it was
int axbc_one_traverse(axbc_ctx *c, int H, int *levels, bool *done)
{
    TRY(pivot_room(c, c->one, true, done));
    if (!*done) return AXBC_OK;
    PivotRun R;
    R.v0 = 0;
    R.p = 1.0;
    R.H = H;
    R.bi = c->bi;
    R.level_te = c->d_level_te;
    R.level_cnt = c->d_level_cnt;
    R.level_mode = c->d_level_mode;
    TRY(pivot_launch(c, c->one, R, done));
    if (!*done) return AXBC_OK;
    int site = 0;
    TRY(pivot_wait(c, c->one, &site));
    *done = site == 0;
    *levels = c->one.ctl_host->levels;
    return AXBC_OK;
}

int axbc_one_apply(axbc_ctx *c, float *delta_out)
{
    ProfScope ps(c, KP_UPDATE, (double)c->g->n * 20.0);
    k_one_update<<<(int)std::min<uint64_t>(axbc_grid_for(c, 256, 8), (c->g->n + 255) / 256), 256, 0, c->stream>>>(
        c->one.delta, c->g->n, c->bi, delta_out);
    CU_LAUNCH("k_one_update");
    return AXBC_OK;
}

// *done = false: bc is as it was, the level-by-level form has to run
static int run_pivot_once(axbc_ctx *c, uint32_t v0, double p, int H, axbc_pivot_stats *st, bool *done)
{
    *done = false;
    if (axbc_pass_fails(AXBC_FAIL_WAIT)) return AXBC_OK;
    PivotRun R;
    R.v0 = v0;
    R.p = p;
    R.H = H;
    R.bi = nullptr;
    R.level_te = R.level_cnt = nullptr;
    R.level_mode = nullptr;
    TRY(pivot_launch(c, c->piv, R, done));
    if (!*done) return AXBC_OK;
    c->delta_last_valid = false;  // the last pivot's delta is c->delta
    CU(cudaMemcpyAsync(&c->pc_host->pad, c->g->reach + v0, 4, cudaMemcpyDeviceToHost, c->stream));
    int site = 0;
    TRY(pivot_wait(c, c->piv, &site));
    // a block waited in vain at the last barrier: others may have gone on to bc
    if (site == 4) {
        axbc_set_error("pivot in one launch: the wait before the bc update ran out of its budget");
        return AXBC_ERR_TIMEOUT;
    }
    *done = site == 0;
    if (!*done) return AXBC_OK;
    const PivotCtl &h = *c->piv.ctl_host;
    if (st) {
        st->nvisited = h.qtail;
        st->all = (H == 1 ? (uint32_t)h.rsum : 0u) + c->pc_host->pad;
        st->te = 2 * h.newdeg;
        st->levels = h.levels;
        st->pad = 0;
    }
    return AXBC_OK;
}

extern "C" int axbc_run_pivot(axbc_ctx *c, uint32_t v0, double p, int H, axbc_pivot_stats *st)
{
    CHECK_ARG(c, "axbc_run_pivot: null context");
    axbc_graph *g = c->g;
    CHECK_ARG(v0 < g->n, "axbc_run_pivot: v0 >= n");
    CHECK_ARG(H == 0 || H == 1, "axbc_run_pivot: H must be 0 or 1");
    // one launch, unless every kernel is to be timed or the caller wants none
    TRY(pivot_fit(c));
    if (!c->prof_on && c->persist_mode >= 0 && c->coop && c->pivot_fit > 0) {
        bool done = false;
        TRY(axbc_ensure_single(c));
        TRY(pivot_room(c, c->piv, false, &done));
        if (done) TRY(run_pivot_once(c, v0, p, H, st, &done));
        if (done) return AXBC_OK;
    }
    TRY(axbc_single_reset(c));
    TRY(axbc_single_set_root(c, v0, 0, 1));

    c->levstart.assign(2, 0);
    c->levstart[1] = 1;
    uint64_t nvisited = 1;
    int level = 0;
    for (;;) {
        level++;
        const uint32_t qs = (uint32_t)c->levstart[level - 1];
        const uint32_t nf = (uint32_t)(c->levstart[level] - c->levstart[level - 1]);
        uint64_t nfrt = 0;
        TRY(axbc_single_forward_level(c, qs, nf, level, &nfrt));
        c->levstart.push_back(c->levstart[level] + nfrt);
        if (!nfrt) break;
        nvisited += nfrt;
    }
    // backward: depth level-2 down to 1; depth 0 only when level == 2
    int depth = level - 2;
    if (depth >= 0) {
        do {
            TRY(axbc_single_backward_level(c, (uint32_t)c->levstart[depth],
                                           (uint32_t)(c->levstart[depth + 1] - c->levstart[depth]),
                                           depth));
            depth--;
        } while (depth > 0);
    }
    if (H == 1) TRY(axbc_single_reach_sum(c));
    else CU(cudaMemsetAsync(&c->pc->reach_sum, 0, 8, c->stream));
    TRY(axbc_single_update(c, v0, p, g->reach + v0, nvisited, 1, H == 1));
    if (st) {
        cudaStream_t s = c->stream;
        CU(cudaMemcpyAsync(c->pc_host, c->pc, sizeof(PivotCounters), cudaMemcpyDeviceToHost, s));
        uint32_t reach_v0 = 0;
        CU(cudaMemcpyAsync(&reach_v0, g->reach + v0, 4, cudaMemcpyDeviceToHost, s));
        CU(cudaStreamSynchronize(s));
        st->nvisited = nvisited;
        st->all = (H == 1 ? (uint32_t)c->pc_host->reach_sum : 0u) + reach_v0;
        st->te = 2 * c->pc_host->newdeg;
        st->levels = level;
        st->pad = 0;
    }
    return AXBC_OK;
}
