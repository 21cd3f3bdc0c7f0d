// Passes over meshes and road-like graphs: a cluster of blocks per pivot.
//
// On a graph of a few neighbours per vertex and hundreds of levels a level of
// one pivot is a few hundred vertices.  The batched rows then carry one pivot of
// 32 or 64 (a vertex lies at another depth from every pivot), and each level
// costs launches or a grid barrier: 25 us a level and depth of a 512^2 grid with
// 32 pivots, of which the work is a tenth.  Here every pivot runs by itself on one
// thread-block cluster -- one block, or up to eight where a level is too wide for
// 1024 threads, sixteen for one or two pivots -- whose hardware barrier costs a
// fraction of a microsecond, with one thread per vertex of the level, and the
// clusters of a pass run side by side.  The bound is the chain of dependent
// loads of a level (queue, offsets, entries, level, claim), two to three
// microseconds.  Measured, ms a pass, rows : this: 128^2 grid 5.2 : 1.2 (32 pivots),
// 6.7 : 1.2 (64); 512^2 16.5 : 3.2 and 24.8 : 3.7; 1024^2 65 : 15 (64); 2048^2 216 : 80
// (64).  Sums run in the canonical order, so the bits are the batched pass's.
//
// A pivot's vectors are whole (pivot-major): path counts, dependencies and
// quotients in the buffers of the batched rows, levels and queues beside them.  A
// level wider than the limit ends the kernel, and the pass runs in the batched
// form instead, as it does without room for the levels and queues.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <vector>

#include "common.cuh"

namespace cg = cooperative_groups;

#define MESH_TPB 1024

struct MeshArgs {
    Adj a;
    const uint32_t *reach;
    BatchInfo *bi;
    float *bc;
    int32_t *lvl;
    uint32_t *sigma, *queue;
    float *delta, *q;
    uint32_t *lev;   // per pivot lev_cap starts of its levels in its queue
    int *stop;       // 1: a level exceeded `limit`, 2: too many levels
    uint64_t n, lev_cap;
    uint32_t limit;
    int most;  // levels it may take
    int nsrc, H, trial;
};

__device__ __forceinline__ int ld_lvl(const int32_t *p) { return __ldcg(p); }

// levels unset, path counts 0 (the grid: nsrc vectors of n)
__global__ void k_mesh_reset(MeshArgs A)
{
    const uint64_t words = (uint64_t)A.nsrc * A.n;
    const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, nt = (uint64_t)gridDim.x * blockDim.x;
    uint4 *l = reinterpret_cast<uint4 *>(A.lvl), *s = reinterpret_cast<uint4 *>(A.sigma);
    for (uint64_t i = tid; i < words / 4; i += nt) {
        l[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
        s[i] = make_uint4(0, 0, 0, 0);
    }
    if (tid < words % 4) {
        A.lvl[words / 4 * 4 + tid] = -1;
        A.sigma[words / 4 * 4 + tid] = 0;
    }
    if (tid == 0) {
        BatchInfo *bi = A.bi;
        bi->nsrc = A.nsrc;
        bi->srcmask = bi->applymask = A.nsrc >= 64 ? ~0ull : (1ull << A.nsrc) - 1ull;
        bi->H = A.H;
        bi->depth0mask = 0;
        bi->pool_short = 0;
        bi->alive = 0;
        bi->cur = bi->lend = 0;
        *A.stop = 0;
    }
    if (tid < AXBC_WMAX) {
        A.bi->lane_bc[tid] = A.bc;
        A.bi->Ls[tid] = 0;
        A.bi->root_reach[tid] = 0;
        A.bi->nvis[tid] = A.bi->rsum[tid] = A.bi->te[tid] = 0;
    }
}

// Terms of adjacency positions [b, b + 8) cut at e, as the canonical 8-position
// subtree.
__device__ __forceinline__ float mesh_tree8(const Adj &a, uint32_t b, uint32_t e, const int32_t *lvl, const float *q,
                                            int d, float sc)
{
    uint32_t r[8];
    int l[8];
    float t[8];
#pragma unroll
    for (int i = 0; i < 8; i++) r[i] = b + i < e ? a.row[b + i] : 0u;
    // levels and quotients load together: a hop less than waiting for the level
#pragma unroll
    for (int i = 0; i < 8; i++) {
        l[i] = b + i < e ? ld_lvl(lvl + r[i]) : -1;
        t[i] = b + i < e ? __ldcg(q + r[i]) : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) t[i] = l[i] == d + 1 ? __fmul_rn(t[i], sc) : 0.0f;
    return __fadd_rn(__fadd_rn(__fadd_rn(t[0], t[1]), __fadd_rn(t[2], t[3])),
                     __fadd_rn(__fadd_rn(t[4], t[5]), __fadd_rn(t[6], t[7])));
}

__global__ void __launch_bounds__(MESH_TPB, 1) k_mesh(MeshArgs A)
{
    cg::cluster_group cl = cg::this_cluster();
    // new vertices of a level, in the first block's memory: level L counts in
    // s_new[L % 3], read after the level's barrier; level L clears the counter
    // of level L + 1, last read before the barrier that ended level L - 1
    __shared__ uint32_t s_new[3];
    __shared__ unsigned long long s_te, s_rs;
    const unsigned lane = lane_id();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int s = blockIdx.x / C;  // the cluster's pivot
    const uint32_t T = C * MESH_TPB, tid = rank * MESH_TPB + threadIdx.x;
    int32_t *lvl = A.lvl + s * A.n;
    uint32_t *sigma = A.sigma + s * A.n, *queue = A.queue + s * A.n;
    float *delta = A.delta + s * A.n, *q = A.q + s * A.n;
    uint32_t *lev = A.lev + s * A.lev_cap;
    uint32_t *cnt = cl.map_shared_rank(s_new, 0);
    const uint32_t root = A.bi->root[s];
    if (threadIdx.x == 0) {
        s_new[0] = s_new[1] = s_new[2] = 0;
        s_te = s_rs = 0;
    }
    unsigned long long te = 0, rs = 0;
    if (tid == 0) {
        lvl[root] = 0;
        sigma[root] = 1;
        delta[root] = __uint2float_rn(A.reach[root]);
        queue[0] = root;
        te = A.a.col[root + 1] - A.a.col[root];
        A.bi->root_reach[s] = A.reach[root];
    }
    cl.sync();

    // forward: thread i takes vertex i of the level, its edges one after
    // another four at a time
    uint32_t qs = 0, qe = 1;
    int L = 1;
    int stop = 0;
    if (tid == 0) lev[0] = 0, lev[1] = 1;
    for (;; L++) {
        if (tid == 0) cnt[(L + 1) % 3] = 0;
        for (uint32_t i0 = qs; i0 < qe; i0 += T) {
            const uint32_t i = i0 + tid;
            uint32_t b = 0, e = 0, sc = 0;
            if (i < qe) {
                const uint32_t v = __ldcg(queue + i);
                b = A.a.col[v];
                e = A.a.col[v + 1];
                sc = __ldcg(sigma + v);
            }
            while (__any_sync(FULL_MASK, b < e)) {
                uint32_t r[4];
                bool nw[4];
#pragma unroll
                for (int k = 0; k < 4; k++) r[k] = b + k < e ? A.a.row[b + k] : 0xffffffffu;
                int l[4], old[4];
#pragma unroll
                for (int k = 0; k < 4; k++) l[k] = r[k] != 0xffffffffu ? ld_lvl(lvl + r[k]) : 0;
                // all claims under way before the first is looked at
#pragma unroll
                for (int k = 0; k < 4; k++) old[k] = l[k] == -1 ? atomicCAS(lvl + r[k], -1, L) : 0;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    nw[k] = l[k] == -1 && old[k] == -1;
                    if (nw[k] || l[k] == L || (l[k] == -1 && old[k] == L)) atomicAdd(sigma + r[k], sc);
                }
                // the warp's new vertices: one addition, then their places
                unsigned m[4];
                int total = 0;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    m[k] = __ballot_sync(FULL_MASK, nw[k]);
                    total += __popc(m[k]);
                }
                if (total) {
                    uint32_t base = 0;
                    if (lane == 0) base = atomicAdd(cnt + L % 3, (uint32_t)total);
                    base = qe + __shfl_sync(FULL_MASK, base, 0);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const uint32_t at = base + __popc(m[k] & ((1u << lane) - 1u));
                        if (nw[k] && at < A.n) queue[at] = r[k];
                        base += __popc(m[k]);
                    }
                }
                b += 4;
            }
        }
        cl.sync();
        const uint32_t found = *(volatile uint32_t *)(cnt + L % 3);
        qs = qe;
        qe += found;
        if (found == 0) break;
        stop = found > A.limit || qe > A.n ? 1 : L >= A.most ? 2 : 0;
        if (stop) break;
        if (tid == 0) lev[L + 1] = qe;
    }
    // L: the first empty level
    if (stop && tid == 0) atomicMax(A.stop, stop);
    if (stop || A.trial) {
        cl.sync();  // no block leaves while another may use its counters
        return;
    }

    // backward: the deepest vertices have delta = reach; then depths L-2 .. 1,
    // and 0 when the BFS ended at level 2
    cl.sync();
    uint32_t i1 = qe, i0 = __ldcg(lev + L - 1);
    for (int d = L - 1; d >= (L == 2 ? 0 : 1); d--) {
        const uint32_t below = d > 0 ? __ldcg(lev + d - 1) : 0u;  // for the next depth
        for (uint32_t i = i0 + tid; i < i1; i += T) {
            const uint32_t v = __ldcg(queue + i);
            const uint32_t b0 = A.a.col[v], b1 = A.a.col[v + 1], sg = __ldcg(sigma + v);
            const float sc = __uint2float_rn(sg);
            float P = 0.0f;
            if (d < L - 1)
                for (uint32_t b = b0; b < b1; b += AXBC_CHUNK) {
                    const uint32_t e = min(b1, b + AXBC_CHUNK);
                    float g = mesh_tree8(A.a, b, e, lvl, q, d, sc);
                    if (b + 8 < e) {
                        g = __fadd_rn(g, mesh_tree8(A.a, b + 8, e, lvl, q, d, sc));
                        if (b + 16 < e) {
                            float h = mesh_tree8(A.a, b + 16, e, lvl, q, d, sc);
                            if (b + 24 < e) h = __fadd_rn(h, mesh_tree8(A.a, b + 24, e, lvl, q, d, sc));
                            g = __fadd_rn(g, h);
                        }
                    }
                    P = __fadd_rn(P, g);
                }
            const uint32_t rv = A.reach[v];
            const float dl = __fadd_rn(__uint2float_rn(rv), P);
            delta[v] = dl;
            q[v] = __fdiv_rn(__fadd_rn(dl, 1.0f), sc);
            if (d > 0) {  // every vertex but the root passes here once
                te += b1 - b0;
                rs += rv;
            }
        }
        cl.sync();
        i1 = i0;
        i0 = below;
    }
    for (int o = 16; o; o >>= 1) {
        te += __shfl_xor_sync(FULL_MASK, te, o);
        rs += __shfl_xor_sync(FULL_MASK, rs, o);
    }
    if (lane == 0 && (te | rs)) {
        atomicAdd(&s_te, te);
        atomicAdd(&s_rs, rs);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(&A.bi->te[s], s_te);
        atomicAdd(&A.bi->rsum[s], s_rs);
        if (rank == 0) {
            A.bi->nvis[s] = qe;
            A.bi->Ls[s] = L;
            if (L == 2) atomicOr(&A.bi->depth0mask, 1ull << s);
            atomicMax(&A.bi->lend, L);
        }
    }
}

// bc update for the applied pivots in lane order, as k_update_m, one thread per
// vertex over the pivots' vectors; delta_out (when given): the last applied
// pivot's dependencies
__global__ void __launch_bounds__(256) k_mesh_update(const int32_t *__restrict__ lvl, const float *__restrict__ delta,
                                                     const uint32_t *__restrict__ reach, uint64_t n,
                                                     const BatchInfo *__restrict__ bi, float *__restrict__ delta_out)
{
    __shared__ uint32_t s_root[AXBC_WMAX], s_rr[AXBC_WMAX];
    __shared__ unsigned long long s_nvt[AXBC_WMAX];
    __shared__ double s_p[AXBC_WMAX];
    __shared__ InvSplit s_iv[AXBC_WMAX];
    __shared__ float *s_bc[AXBC_WMAX];
    const unsigned long long am = bi->applymask & bi->srcmask;
    if (am == 0) return;
    for (int s = threadIdx.x; s < AXBC_WMAX; s += blockDim.x)
        if ((am >> s) & 1ull) {
            s_root[s] = bi->root[s];
            s_rr[s] = bi->root_reach[s];
            s_nvt[s] = bi->nvis[s] + ((bi->H == 1 ? (uint32_t)bi->rsum[s] : 0u) + bi->root_reach[s]);
            s_p[s] = bi->p[s];
            s_iv[s] = inv_split(bi->p[s]);
            s_bc[s] = bi->lane_bc[s];
        }
    __syncthreads();
    const int last = 63 - __clzll(am);
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
         v += (uint64_t)gridDim.x * blockDim.x) {
        const float rf = __uint2float_rn(reach[v]);
        float *tgt = nullptr;
        float b = 0.0f, dv = 0.0f;
        for (int s0 = 0; s0 <= last; s0 += 8) {
            // eight pivots' loads together
            float x[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int s = s0 + k;
                x[k] = rf;
                if (s <= last && (am >> s & 1ull) && lvl[s * n + v] >= 0) x[k] = delta[s * n + v];
            }
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int s = s0 + k;
                if (s > last || !(am >> s & 1ull)) continue;
                dv = x[k];
                if (s_bc[s] != tgt) {
                    if (tgt) tgt[v] = b;
                    tgt = s_bc[s];
                    b = tgt[v];
                }
                if ((uint32_t)v == s_root[s]) {
                    if (s_rr[s] > 0) b = __fadd_rn(b, bc_root_term(s_rr[s], s_nvt[s]));
                    continue;
                }
                if (dv == 0.0f && s_p[s] > 0.0) continue;  // x + float(0/p) == x
                b = __fadd_rn(b, bc_term_fast(dv, s_rr[s], s_p[s], s_iv[s]));
            }
        }
        tgt[v] = b;
        if (delta_out) delta_out[v] = dv;
    }
}

// the dependencies of the last applied pivot of lanes [lo, hi)
__global__ void k_mesh_extract(float *out, const int32_t *__restrict__ lvl, const float *__restrict__ delta,
                               const uint32_t *__restrict__ reach, uint64_t n, const BatchInfo *__restrict__ bi, int lo,
                               int hi)
{
    unsigned long long am = bi->applymask & bi->srcmask & (hi >= 64 ? ~0ull : (1ull << hi) - 1ull);
    am &= ~((1ull << lo) - 1ull);
    if (am == 0) return;
    const uint64_t at = (uint64_t)(63 - __clzll(am)) * n;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
         v += (uint64_t)gridDim.x * blockDim.x)
        out[v] = lvl[at + v] >= 0 ? delta[at + v] : __uint2float_rn(reach[v]);
}

// per level, over all pivots: vertices and their degree sum
__global__ void k_mesh_levels(const uint32_t *__restrict__ col, const int32_t *__restrict__ lvl, uint64_t n, int nsrc,
                              unsigned long long *cnt, unsigned long long *te)
{
    const uint64_t words = (uint64_t)nsrc * n;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < words;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const int l = lvl[i];
        if (l < 0) continue;
        const uint64_t v = i % n;
        atomicAdd(&cnt[l], 1ull);
        atomicAdd(&te[l], (unsigned long long)(col[v + 1] - col[v]));
    }
}

// ------------------------------------------------------------------ host

// Graphs without a vertex of more than 64 neighbours (the batched passes keep
// their numbering), until a pass meets a level too wide for it or finds no room
// for its vectors.
bool axbc_mesh_fits(const axbc_ctx *c)
{
    return c->g->max_deg <= AXBC_RENUMBER_MIN_DEG && !c->g->renumbered && c->g->mesh_form.load() >= 0 && !c->mesh_off &&
           !c->mesh_short;
}

// starts of levels kept per pivot: a level has a vertex at least
static uint64_t mesh_lev_cap(const axbc_graph *g) { return std::min<uint64_t>(AXBC_MAX_LEVELS, g->n + 2); }
static uint64_t mesh_bytes(const axbc_graph *g) { return g->n * 8 + mesh_lev_cap(g) * 4; }

// the vectors go (no pass has its results in them any more)
static void mesh_free(axbc_ctx *c)
{
    axbc_dfree(c->mesh_lvl);
    axbc_dfree(c->mesh_queue);
    axbc_dfree(c->mesh_lev);
    c->mesh_lvl = nullptr;
    c->mesh_queue = c->mesh_lev = nullptr;
    c->bytes -= c->mesh_cap * mesh_bytes(c->g);
    c->mesh_cap = 0;
}

// AXBC_ERR_NOMEM: the batched form's buffers are there, the vectors are not
static int mesh_room(axbc_ctx *c, int nsrc)
{
    if (nsrc <= c->mesh_cap) return AXBC_OK;
    const int cap = nsrc <= 1 ? 1 : nsrc <= 8 ? 8 : AXBC_WMAX;
    DBuf l, q, v;
    TRY(l.alloc((uint64_t)cap * c->g->n * 4));
    TRY(q.alloc((uint64_t)cap * c->g->n * 4));
    TRY(v.alloc(cap * mesh_lev_cap(c->g) * 4));
    CU(cudaStreamSynchronize(c->stream));
    mesh_free(c);
    c->mesh_lvl = l.as<int32_t>();
    c->mesh_queue = q.as<uint32_t>();
    c->mesh_lev = v.as<uint32_t>();
    l.p = q.p = v.p = nullptr;
    c->bytes += cap * mesh_bytes(c->g);
    c->mesh_cap = cap;
    return AXBC_OK;
}

struct MeshLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    MeshLaunch(const axbc_ctx *c, int blocks, int C)
    {
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(MESH_TPB);
        cfg.stream = c->stream;
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = C;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
};

// clusters held, plus one (0: not asked), by device and size: asked for once in a
// process, since every context would wait for the same answer
static std::atomic<int> g_cluster_fit[16][5];

// *C blocks per pivot, or as many fewer as the device holds a cluster of (a part
// of it may be out of reach: SMs taken away from this process); 0: not even one
static int mesh_cluster(axbc_ctx *c, int *C)
{
    for (; *C; *C /= 2) {
        int &fit = c->mesh_fit[31 - __builtin_clz(*C)];
        if (fit < 0) {
            if (axbc_pass_fails(AXBC_FAIL_CLUSTER)) {
                fit = 0;
                continue;
            }
            std::atomic<int> &asked = g_cluster_fit[c->g->device & 15][31 - __builtin_clz(*C)];
            fit = asked.load() - 1;
            if (fit < 0) {
                if (*C > 8) CU(cudaFuncSetAttribute(k_mesh, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
                MeshLaunch ml(c, *C, *C);
                if (cudaOccupancyMaxActiveClusters(&fit, k_mesh, &ml.cfg) != cudaSuccess) {
                    (void)cudaGetLastError();
                    fit = 0;
                }
                asked.store(fit + 1);
            }
        }
        if (fit > 0) break;
    }
    return AXBC_OK;
}

// A test's choice of the blocks per pivot of a context's mesh passes.
extern "C" int axbc_ctx_mesh_blocks(axbc_ctx *c, int blocks, int *used)
{
    CHECK_ARG(c, "axbc_ctx_mesh_blocks: null context");
    CHECK_ARG(blocks >= 0 && blocks <= 16 && (blocks & (blocks - 1)) == 0,
              "axbc_ctx_mesh_blocks: blocks must be 0, 1, 2, 4, 8 or 16");
    c->mesh_force = blocks;
    if (used) *used = c->mesh_used;
    return AXBC_OK;
}

// Reset and traversal of A's pivots, and the wait for it.  *stop: 0, or 1 a level
// was too wide, 2 there are more than A.most levels, 3 the device holds no block
// of it.
static int mesh_pass(axbc_ctx *c, const MeshArgs &A, int *stop)
{
    axbc_graph *g = c->g;
    cudaStream_t s = c->stream;
    const int nsrc = A.nsrc;
    const uint64_t words = ((uint64_t)nsrc * g->n + 3) / 4;
    // Blocks per pivot: as many as give the vertices of a level four times the
    // average width a thread each, and leave every pivot its own SMs; sixteen
    // only for one or two pivots, since few such clusters fit the chip at once.
    // The width is guessed from the last pass's depth, or the square root of the
    // graph.  Measured, ms a pass with 1, 2, 4, 8, 16 blocks: 512^2 grid, 32 pivots
    // 4.7, 3.6, 3.2; 1024^2, 1 pivot 14.6, 8.5, 5.5, 4.2, 3.4, and 8 pivots 15.2, 9.1,
    // 6.1, 4.9, 7.2; 2048^2, 1 pivot 56, 30, 17, 10, 6.9, 8 pivots 57, 31, 18, 12, 15.
    const uint64_t depth = c->last_batch_levels > 0 ? c->last_batch_levels : (uint64_t)__builtin_sqrt((double)g->n);
    const uint64_t width = g->n / std::max<uint64_t>(1, depth);
    int C = 1;
    const int sms = c->num_sms > 0 ? c->num_sms : 152, most = nsrc <= 2 ? 16 : 8;
    while (C < most && (uint64_t)C * MESH_TPB < 4 * width && 2 * C * nsrc <= sms) C *= 2;
    if (A.trial) C = 16;  // its levels may be wide
    if (c->mesh_force) C = c->mesh_force;
    TRY(mesh_cluster(c, &C));
    *stop = C ? 0 : 3;
    if (!C) return AXBC_OK;
    c->mesh_blocks = C;
    {
        ProfScope ps(c, KP_PERSIST, 0);
        k_mesh_reset<<<(int)std::max<uint64_t>(1, std::min<uint64_t>(axbc_grid_for(c, 256, 8), (words + 255) / 256)),
                       256, 0, s>>>(A);
    }
    CU_LAUNCH("k_mesh_reset");
    {
        ProfScope ps(c, KP_PERSIST, 0);
        MeshLaunch ml(c, nsrc * C, C);
        CU(cudaLaunchKernelEx(&ml.cfg, k_mesh, A));
    }
    CU_LAUNCH("k_mesh");
    const size_t off = offsetof(BatchInfo, depth0mask), len = offsetof(BatchInfo, push_factor) - off;
    CU(cudaMemcpyAsync((char *)c->bi_host + off, (char *)c->bi + off, len, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    *stop = c->bi_host->gs.need;
    return AXBC_OK;
}

// On a graph of low degree that is no mesh (a random one) a pass of many pivots
// would find that out only after it has allocated and cleared its vectors and
// taken every pivot to the wide level.  The first pass on such a graph takes its
// first pivot alone that far, MESH_TRIAL_LEVELS at most (a tenfold growth a
// level reaches the limit in six, a twofold in seventeen); smaller graphs lose
// less by the attempt than by the trial.
#define MESH_TRIAL_N (1ull << 16)
#define MESH_TRIAL_LEVELS 20

// A pass of nsrc pivots (roots in c->bi).  *done = false: a level was too wide
// or the vectors found no room (512 bytes a vertex beside the rows' 768, which
// the batched form does without); nothing is left behind but the roots.
int axbc_mesh_traverse(axbc_ctx *c, int nsrc, int H, int *levels, bool *done)
{
    axbc_graph *g = c->g;
    cudaStream_t s = c->stream;
    *done = false;
    c->mesh_used = 0;
    TRY(axbc_ensure_batch(c));
    MeshArgs A;
    A.a = g->fwd;
    A.reach = g->reach;
    A.bi = c->bi;
    A.bc = c->bc;
    A.sigma = c->msigma;
    A.delta = c->mdelta;
    A.q = c->mq;
    A.stop = &c->bi->gs.need;
    A.n = g->n;
    A.H = H;
    // a level of a sixteenth of the graph is no narrow one
    A.limit = (uint32_t)std::max<uint64_t>(2048, g->n / 16);
    int stop = 0;
    if (nsrc > 1 && g->n >= MESH_TRIAL_N && g->mesh_form.load() == 0) {
        // in the rows of a pass, which its forward levels do not use yet
        A.lvl = reinterpret_cast<int32_t *>(c->mdelta);
        A.queue = reinterpret_cast<uint32_t *>(c->mq);
        A.lev = c->msigma + g->n;
        A.lev_cap = MESH_TRIAL_LEVELS + 2;
        A.most = MESH_TRIAL_LEVELS;
        A.nsrc = A.trial = 1;
        TRY(mesh_pass(c, A, &stop));
    }
    if (stop != 1) {
        const int room = mesh_room(c, nsrc);
        if (room == AXBC_ERR_NOMEM) {
            CU(cudaStreamSynchronize(s));
            mesh_free(c);  // smaller ones of an earlier pass
            c->mesh_short = true;
            return AXBC_OK;
        }
        TRY(room);
        A.lvl = c->mesh_lvl;
        A.queue = c->mesh_queue;
        A.lev = c->mesh_lev;
        A.lev_cap = mesh_lev_cap(g);
        A.most = AXBC_MAX_LEVELS - 3;
        A.nsrc = nsrc;
        A.trial = 0;
        TRY(mesh_pass(c, A, &stop));
    }
    if (stop == 1) {
        g->mesh_form.store(-1);  // for good: nothing reads the vectors again
        mesh_free(c);
        return AXBC_OK;
    }
    if (stop == 3) {
        c->mesh_off = true;
        mesh_free(c);
        return AXBC_OK;
    }
    if (stop == 2) {
        axbc_set_error("traversal deeper than %d levels", AXBC_MAX_LEVELS - 2);
        return AXBC_ERR_RANGE;
    }
    int unknown = 0;
    g->mesh_form.compare_exchange_strong(unknown, 1);
    c->mesh_used = c->mesh_blocks;
    *levels = c->bi_host->lend;
    *done = true;
    return AXBC_OK;
}

int axbc_mesh_apply(axbc_ctx *c, float *const *delta_out, const int *lane_lo, const int *lane_hi, int nseg)
{
    axbc_graph *g = c->g;
    cudaStream_t s = c->stream;
    const int grid = (int)std::min<uint64_t>(axbc_grid_for(c, 256, 8), (g->n + 255) / 256);
    const bool whole = nseg == 1 && (!lane_lo || lane_lo[0] == 0) && (!lane_hi || lane_hi[0] >= c->last_batch_nsrc);
    {
        ProfScope ps(c, KP_UPDATE, (double)g->n * c->last_batch_nsrc * 20.0);
        k_mesh_update<<<grid, 256, 0, s>>>(c->mesh_lvl, c->mdelta, g->reach, g->n, c->bi,
                                           whole ? (delta_out ? delta_out[0] : c->delta_last) : nullptr);
    }
    for (int i = 0; i < nseg && !whole; i++) {
        ProfScope ps(c, KP_UPDATE, 0);
        k_mesh_extract<<<grid, 256, 0, s>>>(delta_out ? delta_out[i] : c->delta_last, c->mesh_lvl, c->mdelta, g->reach,
                                            g->n, c->bi, lane_lo ? lane_lo[i] : 0, lane_hi ? lane_hi[i] : AXBC_WMAX);
    }
    CU_LAUNCH("mesh update");
    return AXBC_OK;
}

// one pivot's path counts, depths and dependencies
int axbc_mesh_source(axbc_ctx *c, int src, uint32_t *sigma_host, int32_t *lvl_host, float *delta_host)
{
    const uint64_t n = c->g->n, at = (uint64_t)src * n;
    cudaStream_t s = c->stream;
    std::vector<int32_t> lvl(delta_host ? n : 0);
    std::vector<uint32_t> reach(delta_host ? n : 0);
    if (sigma_host) CU(cudaMemcpyAsync(sigma_host, c->msigma + at, n * 4, cudaMemcpyDeviceToHost, s));
    if (lvl_host) CU(cudaMemcpyAsync(lvl_host, c->mesh_lvl + at, n * 4, cudaMemcpyDeviceToHost, s));
    if (delta_host) {
        CU(cudaMemcpyAsync(delta_host, c->mdelta + at, n * 4, cudaMemcpyDeviceToHost, s));
        CU(cudaMemcpyAsync(lvl.data(), c->mesh_lvl + at, n * 4, cudaMemcpyDeviceToHost, s));
        CU(cudaMemcpyAsync(reach.data(), c->g->reach, n * 4, cudaMemcpyDeviceToHost, s));
    }
    CU(cudaStreamSynchronize(s));
    for (uint64_t v = 0; delta_host && v < n; v++)
        if (lvl[v] < 0) delta_host[v] = (float)reach[v];
    return AXBC_OK;
}

// the level tables of axbc_ctx_level_stats, made on request
int axbc_mesh_level_tables(axbc_ctx *c, int L)
{
    CU(cudaMemsetAsync(c->d_level_cnt, 0, L * 8, c->stream));
    CU(cudaMemsetAsync(c->d_level_te, 0, L * 8, c->stream));
    k_mesh_levels<<<1024, 256, 0, c->stream>>>(c->g->fwd.col, c->mesh_lvl, c->g->n, c->last_batch_nsrc, c->d_level_cnt,
                                               c->d_level_te);
    CU_LAUNCH("k_mesh_levels");
    return AXBC_OK;
}
