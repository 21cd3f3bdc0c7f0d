// Local clustering coefficients (lcc_func, src/axbc2d.c:1847-1935).
//
// counter(i) = sum over neighbours w of |adj(w) \ {i} and adj(i)|.  On a
// symmetric graph without self-loops and repeated entries that is twice the
// number of triangles at i, and every triangle need be found only once: order
// the vertices by descending degree (the batched passes' view), let N(u) be
// u's neighbours of higher rank, and for every u and every v in N(u) look up
// which w in N(v) are in N(u) too.  |N(u)| is at most sqrt(m), so N(u) fits a
// hash table in shared memory.  Scale 16 (1.8 M entries): 56 ms by binary
// searches over whole adjacency lists.  Other graphs take those.
#include <cub/cub.cuh>

#include <algorithm>

#include "common.cuh"

// |adj(w) ∩ adj(i)| without i, by binary search of the shorter list's entries
// in the longer one (adjacency lists are sorted and duplicate-free)
__device__ __forceinline__ uint32_t isect_count(const uint32_t *a, uint32_t da, const uint32_t *b,
                                                uint32_t db, uint32_t skip)
{
    if (da > db) {
        const uint32_t *t = a;
        a = b;
        b = t;
        uint32_t td = da;
        da = db;
        db = td;
    }
    uint32_t c = 0;
    for (uint32_t k = 0; k < da; k++) {
        uint32_t x = a[k];
        if (x == skip) continue;
        uint32_t lo = 0, hi = db;
        while (lo < hi) {
            uint32_t mid = (lo + hi) >> 1;
            if (b[mid] < x) lo = mid + 1;
            else hi = mid;
        }
        c += (lo < db && b[lo] == x);
    }
    return c;
}

// lcc_func (src/axbc2d.c:1847-1935): counter(i) = sum over neighbours w of
// |adj(w) \ {i} ∩ adj(i)|, uint32.  Lanes take neighbours; vertices with more
// than SPAN neighbours are split over their span items.
__global__ void k_lcc_count(Adj a, uint32_t *__restrict__ counter)
{
    const unsigned lane = lane_id();
    const uint64_t ntask = a.n + a.n_heavy_items;
    const uint64_t nw = (uint64_t)gridDim.x * blockDim.x / 32;
    for (uint64_t t = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32; t < ntask; t += nw) {
        uint32_t i, b0, b1;
        if (t < a.n) {
            i = (uint32_t)t;
            uint32_t d = a.col[i + 1] - a.col[i];
            if (d < 2 || d > AXBC_SPAN) continue;
            b0 = a.col[i];
            b1 = a.col[i + 1];
        } else {
            i = a.hitem_v[t - a.n];
            uint32_t k = a.hitem_k[t - a.n];
            b0 = a.col[i] + k * AXBC_SPAN;
            b1 = min(a.col[i + 1], b0 + AXBC_SPAN);
        }
        const uint32_t *ai = a.row + a.col[i];
        const uint32_t di = a.col[i + 1] - a.col[i];
        uint32_t c = 0;
        for (uint32_t e = b0 + lane; e < b1; e += 32) {
            uint32_t w = a.row[e];
            c += isect_count(a.row + a.col[w], a.col[w + 1] - a.col[w], ai, di, i);
        }
        c = __reduce_add_sync(FULL_MASK, c);
        if (lane == 0 && c) atomicAdd(&counter[i], c);
    }
}

// counter is indexed as the adjacency col is; out by vertex id
__global__ void k_lcc_final(const uint32_t *__restrict__ col, const uint32_t *__restrict__ counter,
                            const uint32_t *__restrict__ vertex, float *__restrict__ out, uint64_t n)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t d = col[i + 1] - col[i];
        out[vertex ? vertex[i] : i] = (d < 2) ? 0.0f
                         : __fdiv_rn(__uint2float_rn(counter[i]), __uint2float_rn(d * (d - 1u)));
    }
}


// ------------------------------------------------- triangles once each

// Items of an adjacency: the parts of its big vertices, then its other linked
// vertices; item t of a warp is (vertex, [b0, b1)).
__device__ __forceinline__ bool lcc_item(const Adj &a, uint64_t t, uint32_t &v, uint32_t &b0, uint32_t &b1)
{
    if (t < a.n_part) {
        const uint2 p = a.part[t];
        v = p.x;
        b0 = a.col[v] + p.y * a.part_len;
        b1 = min(a.col[v + 1], b0 + a.part_len);
        return true;
    }
    v = a.order[a.n_big + (t - a.n_part)];
    b0 = a.col[v];
    b1 = a.col[v + 1];
    return false;
}
__host__ __device__ __forceinline__ uint64_t lcc_items(const Adj &a) { return a.n_part + (a.n_linked - a.n_big); }

// *bad = 1 when some list is not strictly ascending or holds its own vertex
__global__ void k_lcc_simple(Adj a, uint32_t *bad)
{
    const unsigned lane = lane_id();
    const uint64_t nw = (uint64_t)gridDim.x * blockDim.x / 32;
    bool b = false;
    for (uint64_t t = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32; t < lcc_items(a); t += nw) {
        uint32_t v, b0, b1;
        lcc_item(a, t, v, b0, b1);
        const uint32_t first = a.col[v];
        for (uint32_t e = b0 + lane; e < b1; e += 32) b |= a.row[e] == v || (e > first && a.row[e] <= a.row[e - 1]);
    }
    if (b) *bad = 1;
}

// |N(u)| of every vertex, and (FILL) N(u) itself, in any order, from cur[u] on
template <bool FILL>
__global__ void k_lcc_up(Adj a, uint32_t *__restrict__ cur, uint32_t *__restrict__ up)
{
    const unsigned lane = lane_id();
    const uint64_t nw = (uint64_t)gridDim.x * blockDim.x / 32;
    for (uint64_t t = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32; t < lcc_items(a); t += nw) {
        uint32_t v, b0, b1;
        const bool part = lcc_item(a, t, v, b0, b1);
        uint32_t cnt = 0, at = 0;
        if (FILL && !part) at = cur[v];
        for (uint32_t base = b0; base < b1; base += 32) {
            const uint32_t e = base + lane, w = e < b1 ? a.row[e] : 0xffffffffu;
            const unsigned m = __ballot_sync(FULL_MASK, w < v);
            if (FILL) {
                if (part) {
                    if (lane == 0) at = atomicAdd(&cur[v], (uint32_t)__popc(m));
                    at = __shfl_sync(FULL_MASK, at, 0);
                }
                if (w < v) up[at + __popc(m & ((1u << lane) - 1u))] = w;
                at += __popc(m);
            } else {
                cnt += __popc(m);
            }
        }
        if (!FILL && lane == 0) {
            if (part) atomicAdd(&cur[v], cnt);
            else cur[v] = cnt;
        }
    }
}

#define LCC_EMPTY 0xffffffffu
#define LCC_WARP_UP 64      // |N(u)| up to which a warp takes u
#define LCC_BLOCK_UP 2048   // members of N(u) in a block's table at a time
#define LCC_TPB 256

__device__ __forceinline__ uint32_t lcc_slot(uint32_t w, uint32_t mask) { return (w * 2654435761u >> 12) & mask; }

// Look the members of N(v) up in the table for the lane's v (of [0, nv) v's,
// one per lane): the lists are walked as one concatenation, lane e finding its
// list by a binary search over the length prefix.  Returns the lane's hits.
__device__ __forceinline__ uint32_t lcc_probe(const uint32_t *__restrict__ off, const uint32_t *__restrict__ up,
                                              uint32_t v, bool have, const uint32_t *keys, uint32_t *hits,
                                              uint32_t mask, uint32_t *counter)
{
    const unsigned lane = lane_id();
    uint32_t b = 0, d = 0, mine = 0;
    if (have) {
        b = off[v];
        d = off[v + 1] - b;
    }
    uint32_t inc = d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL_MASK, inc, o);
        if ((int)lane >= o) inc += t;
    }
    const uint32_t total = __shfl_sync(FULL_MASK, inc, 31), shift = b - (inc - d);
    for (uint32_t base = 0; base < total; base += 32) {
        const uint32_t e = base + lane;
        uint32_t k = 0;
#pragma unroll
        for (int step = 16; step; step >>= 1)
            if (__shfl_sync(FULL_MASK, inc, k + step - 1) <= e) k += step;
        const uint32_t pos = __shfl_sync(FULL_MASK, shift, k) + e;
        bool hit = false;
        if (e < total) {
            const uint32_t w = up[pos];
            for (uint32_t s = lcc_slot(w, mask);; s = (s + 1) & mask) {
                const uint32_t key = keys[s];
                if (key == LCC_EMPTY) break;
                if (key == w) {
                    atomicAdd(&hits[s], 1u);
                    hit = true;
                    break;
                }
            }
        }
        // the triangles of each v found in this window, added by the lane that
        // owns v
        const unsigned m = __ballot_sync(FULL_MASK, hit);
        const uint32_t lo = inc - d > base ? inc - d - base : 0u, hi = inc > base ? min(32u, inc - base) : 0u;
        if (lo < hi) mine += __popc(m & (0xffffffffu >> (32 - (hi - lo)) << lo));
    }
    if (mine) atomicAdd(&counter[v], 2 * mine);
    return mine;
}

__device__ __forceinline__ void lcc_insert(uint32_t *keys, uint32_t w, uint32_t mask)
{
    for (uint32_t s = lcc_slot(w, mask);; s = (s + 1) & mask)
        if (atomicCAS(&keys[s], LCC_EMPTY, w) == LCC_EMPTY) return;
}

// u with 2 to LCC_WARP_UP higher neighbours: one warp, a table of twice that;
// those with more go into big
__global__ void __launch_bounds__(LCC_TPB) k_lcc_warp(const uint32_t *__restrict__ off,
                                                      const uint32_t *__restrict__ up, uint64_t n,
                                                      uint32_t *__restrict__ counter, uint32_t *__restrict__ big,
                                                      uint32_t *__restrict__ nbig)
{
    constexpr uint32_t T = 2 * LCC_WARP_UP;
    __shared__ uint32_t s_keys[LCC_TPB / 32][T], s_hits[LCC_TPB / 32][T];
    const unsigned lane = lane_id();
    uint32_t *keys = s_keys[threadIdx.x >> 5], *hits = s_hits[threadIdx.x >> 5];
    const uint64_t nw = (uint64_t)gridDim.x * blockDim.x / 32;
    for (uint64_t u = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32; u < n; u += nw) {
        const uint32_t b = off[u], d = off[u + 1] - b;
        if (d > LCC_WARP_UP && lane == 0) big[atomicAdd(nbig, 1u)] = (uint32_t)u;
        if (d < 2 || d > LCC_WARP_UP) continue;
        for (uint32_t i = lane; i < T; i += 32) keys[i] = LCC_EMPTY, hits[i] = 0;
        __syncwarp();
        for (uint32_t i = lane; i < d; i += 32) lcc_insert(keys, up[b + i], T - 1);
        __syncwarp();
        uint32_t mine = 0;
        for (uint32_t i = 0; i < d; i += 32)
            mine += lcc_probe(off, up, i + lane < d ? up[b + i + lane] : 0u, i + lane < d, keys, hits, T - 1, counter);
        mine = __reduce_add_sync(FULL_MASK, mine);
        if (lane == 0 && mine) atomicAdd(&counter[u], 2 * mine);
        __syncwarp();
        for (uint32_t i = lane; i < T; i += 32)
            if (hits[i]) atomicAdd(&counter[keys[i]], 2 * hits[i]);
        __syncwarp();
    }
}

// u with more: one block, LCC_BLOCK_UP members of N(u) in the table at a time;
// next hands the listed vertices out
__global__ void __launch_bounds__(LCC_TPB) k_lcc_block(const uint32_t *__restrict__ off,
                                                       const uint32_t *__restrict__ up,
                                                       uint32_t *__restrict__ counter,
                                                       const uint32_t *__restrict__ big,
                                                       const uint32_t *__restrict__ nbig, uint32_t *__restrict__ next)
{
    __shared__ uint32_t keys[2 * LCC_BLOCK_UP], hits[2 * LCC_BLOCK_UP];
    __shared__ uint32_t s_i, s_cnt;
    const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_i = atomicAdd(next, 1u), s_cnt = 0;
        __syncthreads();
        if (s_i >= *nbig) return;
        const uint32_t u = big[s_i];
        const uint32_t b = off[u], d = off[u + 1] - b;
        uint32_t mine = 0;
        for (uint32_t p = 0; p < d; p += LCC_BLOCK_UP) {
            const uint32_t c = min((uint32_t)LCC_BLOCK_UP, d - p);
            uint32_t T = 2 * LCC_WARP_UP;
            while (T < 2 * c) T *= 2;
            for (uint32_t i = threadIdx.x; i < T; i += LCC_TPB) keys[i] = LCC_EMPTY, hits[i] = 0;
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < c; i += LCC_TPB) lcc_insert(keys, up[b + p + i], T - 1);
            __syncthreads();
            for (uint32_t i = 32 * wid; i < d; i += LCC_TPB)
                mine += lcc_probe(off, up, i + lane < d ? up[b + i + lane] : 0u, i + lane < d, keys, hits, T - 1,
                                  counter);
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < T; i += LCC_TPB)
                if (hits[i]) atomicAdd(&counter[keys[i]], 2 * hits[i]);
            __syncthreads();
        }
        mine = __reduce_add_sync(FULL_MASK, mine);
        if (lane == 0 && mine) atomicAdd(&s_cnt, mine);
        __syncthreads();
        if (threadIdx.x == 0 && s_cnt) atomicAdd(&counter[u], 2 * s_cnt);
    }
}

// counter by the triangles of the degree-ordered view
static int lcc_triangles(axbc_graph *g, uint32_t *counter, cudaStream_t s)
{
    const uint64_t n = g->n;
    DBuf cnt, off, up, tmp, next;
    TRY(cnt.alloc((n + 1) * 4));
    TRY(off.alloc((n + 1) * 4));
    TRY(next.alloc(8));
    CU(cudaMemsetAsync(cnt.p, 0, (n + 1) * 4, s));
    CU(cudaMemsetAsync(next.p, 0, 8, s));
    k_lcc_up<false><<<2048, 256, 0, s>>>(g->bfwd, cnt.as<uint32_t>(), nullptr);
    size_t tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt.as<uint32_t>(), off.as<uint32_t>(), (int64_t)n + 1, s);
    TRY(tmp.alloc(tb));
    cub::DeviceScan::ExclusiveSum(tmp.p, tb, cnt.as<uint32_t>(), off.as<uint32_t>(), (int64_t)n + 1, s);
    TRY(up.alloc((g->m / 2 + 1) * 4));  // each edge is in one list
    CU(cudaMemcpyAsync(cnt.p, off.p, (n + 1) * 4, cudaMemcpyDeviceToDevice, s));
    k_lcc_up<true><<<2048, 256, 0, s>>>(g->bfwd, cnt.as<uint32_t>(), up.as<uint32_t>());
    // cnt has done its work: the list of the long ones
    uint32_t *nbig = next.as<uint32_t>(), *ctr = nbig + 1;
    int sms = 0;
    CU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device));
    k_lcc_warp<<<sms * 8, LCC_TPB, 0, s>>>(off.as<uint32_t>(), up.as<uint32_t>(), n, counter, cnt.as<uint32_t>(), nbig);
    k_lcc_block<<<sms * 6, LCC_TPB, 0, s>>>(off.as<uint32_t>(), up.as<uint32_t>(), counter, cnt.as<uint32_t>(), nbig,
                                            ctr);
    CU_LAUNCH("lcc triangles");
    CU(cudaStreamSynchronize(s));  // the scratch lists are freed
    return AXBC_OK;
}

int axbc_build_lcc(axbc_graph *g, cudaStream_t s)
{
    if (g->have_lcc) return AXBC_OK;
    const uint64_t n = g->n;
    DBuf cnt, bad;
    TRY(cnt.alloc(n * 4));
    ALLOC_MISSING(g->lcc, n * 4, &g->bytes);
    ALLOC_MISSING(g->lcc_local, n * 8, &g->bytes);
    ALLOC_MISSING(g->lcc_csum, ((n + AXBC_SAMPLE_BLOCK - 1) / AXBC_SAMPLE_BLOCK) * 8, &g->bytes);
    CU(cudaMemsetAsync(cnt.p, 0, n * 4, s));
    // triangles where ranks exist and the lists are those of a simple graph;
    // meshes (no degree above AXBC_RENUMBER_MIN_DEG) have short lists anyway
    bool tri = g->symmetric && g->renumbered;
    if (tri) {
        uint32_t hbad = 0;
        TRY(bad.alloc(4));
        CU(cudaMemsetAsync(bad.p, 0, 4, s));
        k_lcc_simple<<<2048, 256, 0, s>>>(g->fwd, bad.as<uint32_t>());
        CU_LAUNCH("k_lcc_simple");
        CU(cudaMemcpyAsync(&hbad, bad.p, 4, cudaMemcpyDeviceToHost, s));
        CU(cudaStreamSynchronize(s));
        tri = hbad == 0;
    }
    if (tri) TRY(lcc_triangles(g, cnt.as<uint32_t>(), s));
    else k_lcc_count<<<4096, 256, 0, s>>>(g->fwd, cnt.as<uint32_t>());
    k_lcc_final<<<1024, 256, 0, s>>>(tri ? g->bfwd.col : g->fwd.col, cnt.as<uint32_t>(), tri ? g->from_view : nullptr,
                                     g->lcc, n);
    CU_LAUNCH("lcc");
    TRY(axbc_hprefix_launch(g->lcc, n, g->lcc_local, g->lcc_csum, s));
    const uint64_t nb = (n + AXBC_SAMPLE_BLOCK - 1) / AXBC_SAMPLE_BLOCK;
    CU(cudaMemcpyAsync(&g->S_lcc, g->lcc_csum + nb - 1, 8, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    g->have_lcc = true;
    return AXBC_OK;
}
