// Batched form: up to 64 pivots in one multi-source pass.  Lane s of a warp
// owns pivot s (and s + 32 in a pass of more than 32); every vertex carries one
// 32- or 64-bit mask per BFS level (bit s: the vertex is at that depth from
// pivot s), a `seen` mask, and per-pivot path counts / dependencies laid out
// [vertex][32 or 64] so a warp touches one 128-byte line per 32 pivots.
// Results equal those of the plain form bit for bit: path counts are integers,
// and each lane accumulates its dependency sum in the canonical order
// (32-position chunks summed as a tree in registers, chunks then spans left to
// right).
#include <algorithm>
#include <cstddef>
#include <vector>

#include "barrier.cuh"
#include "common.cuh"

#define BATCH_TPB 256

// K: 32-bit mask words per vertex.  K = 1: a pass of up to 32 pivots, lane s
// of a warp owns pivot s.  K = 2: up to 64 pivots, lane l owns pivots l and
// l + 32 (its two "halves"), masks are 64-bit, per-pivot rows hold 64 values
// and one adjacency entry and one mask load serve all 64 pivots.
template <int K> struct MaskOf;
template <> struct MaskOf<1> {
    typedef uint32_t T;
};
template <> struct MaskOf<2> {
    typedef unsigned long long T;
};

template <int K> __device__ __forceinline__ uint64_t row_base(uint64_t v) { return v * (uint64_t)(AXBC_W * K); }

// bit of this lane's pivot of half h (a 32-bit mask has only half 0)
__device__ __forceinline__ bool pbit(uint32_t m, int) { return (m >> lane_id()) & 1u; }
__device__ __forceinline__ bool pbit(unsigned long long m, int h)
{
    return (uint32_t)(m >> (32 * h)) >> lane_id() & 1u;
}
template <class M> __device__ __forceinline__ M lane_mask(int s) { return (M)1 << s; }

__device__ __forceinline__ uint32_t warp_or(uint32_t m) { return __reduce_or_sync(FULL_MASK, m); }
__device__ __forceinline__ unsigned long long warp_or(unsigned long long m)
{
    const uint32_t lo = __reduce_or_sync(FULL_MASK, (uint32_t)m);
    const uint32_t hi = __reduce_or_sync(FULL_MASK, (uint32_t)(m >> 32));
    return (unsigned long long)lo | ((unsigned long long)hi << 32);
}

// Resident blocks per SM the kernels are compiled for, their register budgets.
// The persistent loop: 80 registers at both widths (64 and 48: 2-20% slower).
// The forward step: 32 registers at one mask word, where pushed and pulled levels
// in one kernel spill (156 bytes stored, 176 loaded), and 64 at two, without spills.
// (The pull by itself, three scale-23 passes at 5, 6, 7, 8 blocks: 14.0, 15.0, 13.6,
// 13.6 ms.)  The backward, which runs 32 pivots at a time at either width: 32
// registers by warps, where throughput follows the resident warps (52 bytes stored,
// 88 loaded; three scale-23 passes 23.6 ms, 30.2 at 6 blocks), 48 in tiles (96, 112).
#define PERSIST_BLOCKS 3
#ifndef AXBC_FWD_MIN_BLOCKS
#define AXBC_FWD_MIN_BLOCKS 7
#endif
#ifndef AXBC_BWD_MIN_BLOCKS
#define AXBC_BWD_MIN_BLOCKS 8
#endif
#ifndef AXBC_BWD_TILE_BLOCKS
#define AXBC_BWD_TILE_BLOCKS 5
#endif
#ifndef AXBC_BWD_WIDE_MIN
#define AXBC_BWD_WIDE_MIN (1u << 22)
#endif
#ifndef AXBC_FWD_MIN_BLOCKS2
#define AXBC_FWD_MIN_BLOCKS2 4
#endif
#define FWD_BLOCKS(K) ((K) == 1 ? AXBC_FWD_MIN_BLOCKS : AXBC_FWD_MIN_BLOCKS2)

// Per-level vertex lists: the vertices whose level-L mask is nonzero, appended
// by the forward kernels that set the mask.  A level whose list would exceed
// its capacity keeps counting but stops storing (count > cap: no list), and
// its consumers fall back to the degree-ordered task scan.
struct LevelLists {
    uint32_t *pool;
    uint32_t *start;  // per level: offset into pool
    uint32_t *count;  // per level: vertices appended
    uint32_t *cap;    // per level: capacity
    uint32_t *heavy;  // per level: listed vertices with more than Adj::big neighbours
};


// What a pass starts from.
struct PassStart {
    BatchInfo *bi;
    uint32_t **tab;
    uint32_t *seen, *msigma, *ctrs;
    LevelLists ll;
    unsigned long long *level_te, *level_cnt;
    const uint32_t *col, *rcol, *reach, *to_view;
    float *bc;
    uint64_t n;
    unsigned long long m, push_min;
    double push_factor;
    uint32_t pool_cap, list_max, big;
    int nsrc, H;
    int prev_k, prev_last;  // mask words of the previous pass, last level it may have touched
};

// zero `bytes` (a multiple of 4) from the 16-byte aligned p, all threads of the grid
__device__ __forceinline__ void grid_zero(void *p, uint64_t bytes, uint64_t tid, uint64_t nt)
{
    uint4 *q = reinterpret_cast<uint4 *>(p);
    for (uint64_t i = tid; i < bytes / 16; i += nt) q[i] = make_uint4(0, 0, 0, 0);
    uint32_t *t = reinterpret_cast<uint32_t *>(q + bytes / 16);
    if (tid < bytes % 16 / 4) t[tid] = 0;
}

// Level masks 2..last of the previous pass, width PK: a level whose list was
// stored has nonzero entries only at its listed vertices; an overflowed level
// is cleared whole.
template <int PK>
__device__ __forceinline__ void clean_levels(const PassStart &P, uint64_t tid, uint64_t nt)
{
    typedef typename MaskOf<PK>::T M;
    for (int L = 2; L <= P.prev_last; L++) {
        M *f = reinterpret_cast<M *>(P.tab[L]);
        const uint32_t cnt = P.ll.count[L];
        if (cnt <= P.ll.cap[L]) {
            const uint32_t *lst = P.ll.pool + P.ll.start[L];
            for (uint64_t i = tid; i < cnt; i += nt) f[lst[i]] = 0;
        } else {
            for (uint64_t i = tid; i < P.n; i += nt) f[i] = 0;
        }
    }
}

// Roots: depth 0, sigma 1 (set_mlp_cuda, src/cuda_kernels.cu:862-876); one
// warp, lane l setting up pivots l + 32 h.
template <int K>
__device__ __forceinline__ void pass_roots(const PassStart &P)
{
    typedef typename MaskOf<K>::T M;
    BatchInfo *bi = P.bi;
    const LevelLists &ll = P.ll;
    M *fmask0 = reinterpret_cast<M *>(P.tab[0]), *seen = reinterpret_cast<M *>(P.seen);
    uint32_t *msigma = P.msigma;
    const uint32_t *to_view = P.to_view, *col = P.col, *rcol = P.rcol;
    const int nsrc = P.nsrc, H = P.H;
    const uint32_t pool_cap = P.pool_cap, list_max = P.list_max;
    const int l = threadIdx.x;
    // the roots arrive as vertex ids; the pass runs in the graph's view
    if (to_view) {
#pragma unroll
        for (int h = 0; h < K; h++)
            if (l + 32 * h < nsrc) bi->root[l + 32 * h] = to_view[bi->root[l + 32 * h]];
        __syncwarp();
    }
    if (l == 0) {
        bi->nsrc = nsrc;
        bi->srcmask = nsrc >= 64 ? ~0ull : ((1ull << nsrc) - 1ull);
        bi->applymask = bi->srcmask;
        bi->depth0mask = 0;
        bi->H = H;
        bi->cur = 0;
        bi->alive = 1;
        bi->lend = 0;
        bi->dmax = -1;
        bi->push_factor = P.push_factor;
        bi->lvl_te = 0;
        bi->any_new = 0;
        bi->pool_short = 0;
        bi->gs.count = bi->gs.gen = 0;
        bi->gs.err = bi->gs.need = 0;
    }
    unsigned long long fd = 0, rd = 0;
    uint32_t nroots = 0, heavy_roots = 0;
    const uint32_t rt0 = l < nsrc ? bi->root[l] : 0xffffffffu;
#pragma unroll
    for (int h = 0; h < K; h++) {
        const int s = l + 32 * h;
        bi->Ls[s] = 0;
        bi->lvl_new[s] = 0;
        bi->lane_bc[s] = P.bc;
        bi->root_reach[s] = 0;
        if (s < nsrc) {
            const uint32_t v = bi->root[s];
            bi->root_reach[s] = P.reach[v];
            atomicOr(&fmask0[v], lane_mask<M>(s));
            atomicOr(&seen[v], lane_mask<M>(s));
            msigma[row_base<K>(v) + s] = 1;
            bi->nvis[s] = 1;
            bi->rsum[s] = 0;
            bi->te[s] = col[v + 1] - col[v];
            fd += col[v + 1] - col[v];
            rd += rcol[v + 1] - rcol[v];
        } else {
            bi->nvis[s] = 0;
            bi->rsum[s] = 0;
            bi->te[s] = 0;
        }
        // the level-0 list: each root once (lanes of different runs may share one)
        const uint32_t rt = s < nsrc ? bi->root[s] : 0xffffffffu;
        const uint32_t same = __match_any_sync(FULL_MASK, rt);
        bool first = s < nsrc && (__ffs(same) - 1) == l;
        if (h == 1) {
            bool dup = false;
            for (int j = 0; j < 32; j++) dup |= __shfl_sync(FULL_MASK, rt0, j) == rt;
            first = first && !dup;
        }
        const uint32_t firsts = __ballot_sync(FULL_MASK, first);
        if (first) ll.pool[nroots + __popc(firsts & ((1u << l) - 1u))] = rt;
        nroots += __popc(firsts);
        heavy_roots += __popc(__ballot_sync(FULL_MASK, first && col[rt + 1] - col[rt] > P.big));
    }
    for (int o = 16; o; o >>= 1) {
        fd += __shfl_xor_sync(FULL_MASK, fd, o);
        rd += __shfl_xor_sync(FULL_MASK, rd, o);
    }
    if (l == 0) {
        ll.heavy[0] = heavy_roots;
        // a vertex counts as unvisited until every pivot has seen it: with one
        // pivot its root is fully seen at once
        const unsigned long long unvis = nsrc == 1 ? P.m - rd : P.m;
        bi->front_deg = 0;
        bi->unvis_deg = unvis;
        bi->unvis_dec = 0;
        bi->push_min = P.push_min;
        bi->push_next = (double)fd * P.push_factor < (double)unvis || fd < P.push_min;
        P.level_te[0] = fd;
        P.level_cnt[0] = nsrc;
        ll.start[0] = 0;
        ll.count[0] = nroots;
        ll.cap[0] = nroots;
        ll.start[1] = nroots;
        ll.cap[1] = min(list_max, pool_cap - nroots);
    }
}

// The last block of a launch to get here (all its threads call); its later
// loads past L1 see what every block wrote before calling.  The count wraps to
// zero by itself.
__device__ __forceinline__ bool last_block(uint32_t *ticket)
{
    __shared__ int s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    return s_last != 0;
}

// Everything a pass finds zero, and its roots, in one launch (it took ten: the
// memsets of five arrays and three tables, the clearing of the level masks and
// the roots, about 30 us of a 400-us pass at scale 14).  The last block clears
// the per-level tables, which the others read, and sets the roots.
template <int K>
__global__ void __launch_bounds__(256) k_pass_start(PassStart P)
{
    const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint64_t nt = (uint64_t)gridDim.x * blockDim.x;
    grid_zero(P.seen, P.n * 4 * K, tid, nt);
    grid_zero(P.tab[0], P.n * 4 * K, tid, nt);
    grid_zero(P.tab[1], P.n * 4 * K, tid, nt);
    grid_zero(P.msigma, P.n * AXBC_W * K * 4, tid, nt);
    if (P.prev_k == 2) clean_levels<2>(P, tid, nt);
    else clean_levels<1>(P, tid, nt);
    if (!last_block(&P.bi->ticket[0])) return;
    const int used = min(P.prev_last + 4, AXBC_MAX_LEVELS);
    for (int i = threadIdx.x; i < 2 * used; i += blockDim.x)
        P.ctrs[i] = P.ctrs[2 * AXBC_MAX_LEVELS + i] = 0;
    for (int i = threadIdx.x; i < used; i += blockDim.x) P.ll.count[i] = P.ll.heavy[i] = 0;
    __syncthreads();
    if (threadIdx.x < 32) pass_roots<K>(P);
}

// ---------------------------------------------------------- task scheduling
// Work units are handed out by an atomic counter.
__device__ __forceinline__ uint32_t grab_unit(uint32_t *ctr)
{
    uint32_t t = 0;
    if (lane_id() == 0) t = atomicAdd(ctr, 1u);
    return __shfl_sync(FULL_MASK, t, 0);
}

__device__ __forceinline__ uint32_t warp_global()
{
    return (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
}

__device__ __forceinline__ void list_append(const LevelLists &ll, int L, bool isnew, uint32_t v)
{
    const unsigned lane = lane_id();
    const unsigned m = __ballot_sync(FULL_MASK, isnew);
    if (!m) return;
    const int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if ((int)lane == leader) base = atomicAdd(&ll.count[L], (uint32_t)__popc(m));
    base = __shfl_sync(FULL_MASK, base, leader);
    const uint32_t idx = base + __popc(m & ((1u << lane) - 1u));
    if (isnew && idx < ll.cap[L]) ll.pool[ll.start[L] + idx] = v;
}

// A warp's newly reached vertices on their way to the level's list, 32 to an
// add of its count: with an add every chunk of 32 edges, the warps of a pushed
// level queued for that one word (three scale-23 passes' pushes 1.11 ms, 0.90
// so; the scale-14 run 2.14 and 1.99 ms).
struct ListBuf {
    uint32_t *v;  // 64 entries in shared memory
    uint32_t n = 0;
    __device__ __forceinline__ void flush(const LevelLists &ll, int L, uint32_t cnt)
    {
        const unsigned lane = lane_id();
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&ll.count[L], cnt);
        const uint32_t idx = __shfl_sync(FULL_MASK, base, 0) + lane;
        if (lane < cnt && idx < ll.cap[L]) ll.pool[ll.start[L] + idx] = v[lane];
        __syncwarp();
    }
    __device__ __forceinline__ void add(const LevelLists &ll, int L, bool isnew, uint32_t u)
    {
        const unsigned m = __ballot_sync(FULL_MASK, isnew), lane = lane_id();
        if (!m) return;
        if (isnew) v[n + __popc(m & ((1u << lane) - 1u))] = u;
        n += __popc(m);
        __syncwarp();
        if (n < 32) return;
        flush(ll, L, 32);
        n -= 32;
        const uint32_t x = v[32 + lane];
        __syncwarp();
        v[lane] = x;
        __syncwarp();
    }
    __device__ __forceinline__ void close(const LevelLists &ll, int L)
    {
        if (n) flush(ll, L, n);
        n = 0;
    }
};

// Items per work unit: at least `least`, and as many as
// leave every resident warp about four units (at most 32, one per lane).
__device__ __forceinline__ uint32_t unit_of(uint64_t items, uint32_t least)
{
    const uint64_t nwarps = gridDim.x * (blockDim.x / 32);
    return (uint32_t)max((uint64_t)least, min((uint64_t)32, items / (4 * nwarps)));
}
// A warp's first unit is its own number; further ones come from the counter,
// which nobody touches when there are no more units than warps.
__device__ __forceinline__ uint64_t next_unit(uint32_t *ctr, uint64_t nu)
{
    const uint64_t nwarps = gridDim.x * (blockDim.x / 32);
    return nu <= nwarps ? nu : nwarps + grab_unit(ctr);
}

// the stored list of level L, or nullptr when the level overflowed its capacity
__device__ __forceinline__ const uint32_t *level_list(const LevelLists &ll, int L, uint32_t &cnt)
{
    cnt = ll.count[L];
    if (cnt > ll.cap[L]) return nullptr;
    return ll.pool + ll.start[L];
}

// Path counts are added either an edge at a time, lane = pivot (one line per
// edge), or a pivot of every edge at a time, lane = edge.  The second takes as
// many steps as the fullest edge has pivots: the frontiers that are pushed are
// small and most of their vertices belong to one pivot or two, and 32 steps of
// one lane each were 40 us of a pushed level.  act: lanes with any.
template <class M> __device__ __forceinline__ bool bits_apart(M nm, unsigned act)
{
    const unsigned most = __reduce_max_sync(FULL_MASK, (unsigned)__popcll((unsigned long long)nm));
    return 4 * most <= (unsigned)__popc(act);
}

// Forward level L, push from the vertices of depth L-1: for each neighbour u
// and each pivot s with v at depth L-1 and u unseen, sigma_s[u] += sigma_s[v]
// and bit s joins u's level-L mask.  Atomics are fire-and-forget reductions.
template <int K, class WC>
__device__ __forceinline__ void push_span(const Adj &a, uint32_t v, typename MaskOf<K>::T f, uint32_t b0,
                                          uint32_t b1, const typename MaskOf<K>::T *__restrict__ seen,
                                          typename MaskOf<K>::T *fcur, uint32_t *msigma,
                                          const LevelLists &ll, int L, ListBuf &lb, WC &wc)
{
    typedef typename MaskOf<K>::T M;
    const unsigned lane = lane_id();
    uint32_t sig[K];
#pragma unroll
    for (int h = 0; h < K; h++) {
        sig[h] = pbit(f, h) ? msigma[row_base<K>(v) + 32 * h + lane] : 0u;
        if (pbit(f, h)) wc.add(WC_BYTES, 4);
    }
    for (uint32_t base = b0; base < b1; base += 32) {
        const uint32_t e = base + lane;
        uint32_t u = 0;
        M nm = 0;
        if (e < b1) {
            u = a.row[e];
            nm = f & ~seen[u];
            wc.add(WC_ENTRIES, 1);
            wc.add(WC_BYTES, 4 + 4 * K);  // adjacency entry, seen mask
        }
        const M old = nm ? atomicOr(&fcur[u], nm) : (M)1;
        if (nm) wc.add(WC_BYTES, old == 0 ? 4 + 4 * K : 4 * K);  // level mask, list entry
        lb.add(ll, L, old == 0, u);
        unsigned act = __ballot_sync(FULL_MASK, nm != 0);
        if (bits_apart(nm, act)) {
            while (__any_sync(FULL_MASK, nm != 0)) {
                const int b = nm ? __ffsll((long long)nm) - 1 : 0;
                uint32_t x = __shfl_sync(FULL_MASK, sig[0], b & 31);
                if (K == 2) {
                    const uint32_t hi = __shfl_sync(FULL_MASK, sig[K - 1], b & 31);
                    if (b >= 32) x = hi;
                }
                if (nm) {
                    atomicAdd(&msigma[row_base<K>(u) + b], x);
                    wc.add(WC_PAIRS, 1);
                    wc.add(WC_BYTES, 4);
                }
                nm &= nm - 1;
            }
            continue;
        }
        while (act) {
            const int j = __ffs(act) - 1;
            act &= act - 1;
            const uint32_t uj = __shfl_sync(FULL_MASK, u, j);
            const M mj = __shfl_sync(FULL_MASK, nm, j);
#pragma unroll
            for (int h = 0; h < K; h++)
                if (pbit(mj, h)) {
                    atomicAdd(&msigma[row_base<K>(uj) + 32 * h + lane], sig[h]);
                    wc.add(WC_PAIRS, 1);
                    wc.add(WC_BYTES, 4);
                }
        }
    }
}

// Push from up to 32 light frontier vertices at once, one per lane (f_l = 0:
// none), edge-parallel: the warp walks the concatenation of their adjacency
// lists 32 positions at a time, so a chunk of low-degree vertices costs one
// pass instead of one pass per vertex.  Lane e finds its vertex by a binary
// search over the inclusive degree prefix held across the lanes.
template <int K, class WC>
__device__ __forceinline__ void push_light32(const Adj &a, uint32_t v_l, typename MaskOf<K>::T f_l,
                                             const typename MaskOf<K>::T *__restrict__ seen,
                                             typename MaskOf<K>::T *fcur, uint32_t *msigma,
                                             const LevelLists &ll, int L, ListBuf &lb, WC &wc)
{
    typedef typename MaskOf<K>::T M;
    const unsigned lane = lane_id();
    uint32_t b = 0, d = 0;
    if (f_l) {
        b = a.col[v_l];
        d = a.col[v_l + 1] - b;
        wc.add(WC_BYTES, 8);  // adjacency bounds
    }
    uint32_t inc = d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL_MASK, inc, o);
        if ((int)lane >= o) inc += t;
    }
    const uint32_t total = __shfl_sync(FULL_MASK, inc, 31);
    const uint32_t shift = b - (inc - d);  // position of concatenated index e: shift_k + e
    for (uint32_t base = 0; base < total; base += 32) {
        const uint32_t e = base + lane;
        uint32_t k = 0;  // lanes whose inclusive prefix is <= e
#pragma unroll
        for (int step = 16; step; step >>= 1)
            if (__shfl_sync(FULL_MASK, inc, k + step - 1) <= e) k += step;
        const uint32_t pk = __shfl_sync(FULL_MASK, shift, k) + e;
        const M fk = __shfl_sync(FULL_MASK, f_l, k);
        uint32_t u = 0;
        M nm = 0;
        if (e < total) {
            u = a.row[pk];
            nm = fk & ~seen[u];
            wc.add(WC_ENTRIES, 1);
            wc.add(WC_BYTES, 4 + 4 * K);  // adjacency entry, seen mask
        }
        const M old = nm ? atomicOr(&fcur[u], nm) : (M)1;
        if (nm) wc.add(WC_BYTES, old == 0 ? 4 + 4 * K : 4 * K);  // level mask, list entry
        lb.add(ll, L, old == 0, u);
        unsigned act = __ballot_sync(FULL_MASK, nm != 0);
        const uint32_t vk = __shfl_sync(FULL_MASK, v_l, k);
        if (bits_apart(nm, act)) {
            for (; nm; nm &= nm - 1) {
                const int b = __ffsll((long long)nm) - 1;
                atomicAdd(&msigma[row_base<K>(u) + b], msigma[row_base<K>(vk) + b]);
                wc.add(WC_GATHERS, 1);
                wc.add(WC_PAIRS, 1);
                wc.add(WC_BYTES, 8);  // parent's path count, child's sum
            }
            __syncwarp();
            continue;
        }
        while (act) {
            // up to 4 edges: gather the parents' sigma rows, then add
            uint32_t uu[4], sg[4][K];
            M mm[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int j = act ? __ffs(act) - 1 : 0;
                const bool ok = act != 0;
                act &= act - 1;
                uu[q] = __shfl_sync(FULL_MASK, u, j);
                const M mj = __shfl_sync(FULL_MASK, nm, j);
                mm[q] = ok ? mj : (M)0;
                const uint32_t vj = __shfl_sync(FULL_MASK, vk, j);
#pragma unroll
                for (int h = 0; h < K; h++)
                    sg[q][h] = pbit(mm[q], h) ? msigma[row_base<K>(vj) + 32 * h + lane] : 0u;
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int h = 0; h < K; h++)
                    if (pbit(mm[q], h)) {
                        atomicAdd(&msigma[row_base<K>(uu[q]) + 32 * h + lane], sg[q][h]);
                        wc.add(WC_GATHERS, 1);
                        wc.add(WC_PAIRS, 1);
                        wc.add(WC_BYTES, 8);  // parent's path count, child's sum
                    }
        }
    }
}

template <int K, class WC>
__device__ __forceinline__ void fwd_push_body(const Adj &a, const typename MaskOf<K>::T *__restrict__ fprev,
                                              typename MaskOf<K>::T *fcur,
                                              const typename MaskOf<K>::T *__restrict__ seen,
                                              uint32_t *msigma, uint32_t *ctr, const LevelLists &ll,
                                              int L, uint32_t *stage, WC &wc)
{
    typedef typename MaskOf<K>::T M;
    const unsigned lane = lane_id();
    ListBuf lb{stage};
    uint32_t lcnt = 0;
    const uint32_t *lst = level_list(ll, L - 1, lcnt);  // the frontier, when stored
    // parts of big vertices only when one is in the frontier
    const uint64_t np = lst && ll.heavy[L - 1] == 0 ? 0 : a.n_part;
    const uint64_t nl = lst ? lcnt : a.n_linked - a.n_big;
    const uint32_t gp = unit_of(np, 1), ent = unit_of(nl, 1);
    const uint64_t up = (np + gp - 1) / gp, nu = up + (nl + ent - 1) / ent;
    for (uint64_t t = warp_global(); t < nu; t = next_unit(ctr, nu)) {
        if (t < up) {
            // a unit of parts: one lane looks each part's frontier mask up
            const uint64_t i = lane * up + t;  // a hub's parts fall into different units
            uint2 pt = make_uint2(0, 0);
            M f_l = 0;
            if (lane < gp && i < np) {
                pt = a.part[i];
                f_l = fprev[pt.x];
                wc.add(WC_BYTES, 4 * K);
            }
            for (unsigned act = __ballot_sync(FULL_MASK, f_l != 0); act; act &= act - 1) {
                const int j = __ffs(act) - 1;
                const uint32_t v = __shfl_sync(FULL_MASK, pt.x, j);
                const uint32_t b0 = a.col[v] + __shfl_sync(FULL_MASK, pt.y, j) * a.part_len;
                push_span<K>(a, v, __shfl_sync(FULL_MASK, f_l, j), b0, min(a.col[v + 1], b0 + a.part_len), seen, fcur,
                             msigma, ll, L, lb, wc);
            }
            continue;
        }
        const uint64_t i = (t - up) * ent + lane;
        uint32_t v_l = 0;
        M f_l = 0;
        if (lane < ent && i < nl) {
            v_l = lst ? lst[i] : a.order[a.n_big + i];
            if (a.col[v_l + 1] - a.col[v_l] <= a.big) f_l = fprev[v_l];
            wc.add(WC_BYTES, lst ? 4 + 4 * K : 4 * K);  // list entry, level mask
        }
        // a vertex that fills half a chunk or more by itself: its path counts
        // load once; the others share chunks
        const uint32_t b_l = f_l ? a.col[v_l] : 0u, e_l = f_l ? a.col[v_l + 1] : 0u;
        for (unsigned act = __ballot_sync(FULL_MASK, e_l - b_l >= 16); act; act &= act - 1) {
            const int j = __ffs(act) - 1;
            push_span<K>(a, __shfl_sync(FULL_MASK, v_l, j), __shfl_sync(FULL_MASK, f_l, j),
                         __shfl_sync(FULL_MASK, b_l, j), __shfl_sync(FULL_MASK, e_l, j), seen, fcur, msigma, ll, L, lb, wc);
        }
        if (e_l - b_l >= 16) f_l = 0;
        if (__any_sync(FULL_MASK, f_l != 0)) push_light32<K>(a, v_l, f_l, seen, fcur, msigma, ll, L, lb, wc);
    }
    lb.close(ll, L);
}

// Forward level L, pull: every vertex u that some pivots (`ns`) have not seen
// sums sigma_s over its in-neighbours at depth L-1 from pivot s (u32 sums: any
// order gives the same bits).  Bound by instruction issue, not by memory, so
// the gathers are laid out for few instructions: a lane owns four neighbouring
// pivots (one 16-byte load per parent row), 8 K lanes -- a subgroup -- cover a
// row, and the warp's 4 / K subgroups gather that many parents at once.  One
// row per instruction took 18.8 ms of three scale-23 passes, this 13.6 ms;
// 573 M against 411 M warp instructions on a scale-20 level of 64 pivots.  The
// positions with a parent are staged in shared memory as (parent, mask) pairs,
// one array per 32-pivot half, compacted.
template <int K> struct PullShape {
    static constexpr int SUB = 8 * K;       // lanes that cover one row
    static constexpr int NSUB = 32 / SUB;   // rows gathered at once
    // staged pairs of one warp: slot i of half h at 37 h + i + i / 8, so that
    // the subgroups' simultaneous reads fall into different banks
    static constexpr int STAGE = K == 1 ? 36 : 74;
};
__device__ __forceinline__ int stage_at(int i) { return i + (i >> 3); }

template <int K>
__device__ __forceinline__ void stage_pair(uint2 *st, int slot, uint32_t v, typename MaskOf<K>::T m)
{
    st[stage_at(slot)] = make_uint2(v, (uint32_t)m);
    if (K == 2) st[37 + stage_at(slot)] = make_uint2(v, (uint32_t)((unsigned long long)m >> 32));
}

// Add the rows staged in slots first, first + stride, ... (cnt of them, the
// slots after them hold empty masks) into the lane's four sums; fo collects
// the lane's found pivots.  st_h: the stage of the lane's half.
template <int K>
__device__ __forceinline__ void pull_rows(const uint2 *st_h, int first, int stride, int cnt,
                                          const uint32_t *__restrict__ msig_l, unsigned sh, uint32_t acc[4],
                                          uint32_t &fo)
{
#pragma unroll 1
    for (int i = 0; i < cnt; i += 2) {
        const int s0 = first + i * stride, s1 = s0 + stride;
        const uint2 e0 = st_h[stage_at(s0)], e1 = st_h[stage_at(s1)];
        const uint32_t n0 = (e0.y >> sh) & 15u, n1 = (e1.y >> sh) & 15u;
        uint4 x0 = make_uint4(0, 0, 0, 0), x1 = x0;
        if (n0) x0 = *reinterpret_cast<const uint4 *>(msig_l + row_base<K>(e0.x));
        if (n1) x1 = *reinterpret_cast<const uint4 *>(msig_l + row_base<K>(e1.x));
        if (n0 & 1u) acc[0] += x0.x;
        if (n0 & 2u) acc[1] += x0.y;
        if (n0 & 4u) acc[2] += x0.z;
        if (n0 & 8u) acc[3] += x0.w;
        if (n1 & 1u) acc[0] += x1.x;
        if (n1 & 2u) acc[1] += x1.y;
        if (n1 & 4u) acc[2] += x1.z;
        if (n1 & 8u) acc[3] += x1.w;
        fo |= n0 | n1;
    }
}

// One part [b0, b1) of a big vertex's in-adjacency: all subgroups share it,
// slot i of a chunk's staged pairs going to subgroup i mod NSUB.  Adjacency
// entries load two chunks ahead and level masks one ahead.
template <int K, class WC>
__device__ __forceinline__ void pull_part(const Adj &rv, uint32_t u, typename MaskOf<K>::T ns, uint32_t b0,
                                          uint32_t b1, const typename MaskOf<K>::T *__restrict__ fprev,
                                          typename MaskOf<K>::T *fcur, uint32_t *msigma, uint2 *st,
                                          const LevelLists &ll, int L, WC &wc)
{
    typedef typename MaskOf<K>::T M;
    typedef PullShape<K> S;
    const unsigned lane = lane_id();
    const int sl = lane & (S::SUB - 1), g = lane / S::SUB;
    const unsigned sh = 4 * (sl & 7);
    const uint2 *st_h = st + (K == 2 && sl >= 8 ? 37 : 0);
    uint32_t acc[4] = {0, 0, 0, 0}, fo = 0;
    uint32_t e = b0 + lane;
    uint32_t v = e < b1 ? rv.row[e] : 0u, vn = e + 32 < b1 ? rv.row[e + 32] : 0u;
    M fm = e < b1 ? fprev[v] & ns : (M)0;
    for (; e - lane < b1; e += 32) {
        if (e < b1) {
            wc.add(WC_ENTRIES, 1);
            wc.add(WC_GATHERS, __popcll((unsigned long long)fm));
            wc.add(WC_BYTES, 4 + 4 * K + 4 * __popcll((unsigned long long)fm));  // entry, mask, parents' counts
        }
        const unsigned act = __ballot_sync(FULL_MASK, fm != 0);
        const int nh = __popc(act);
        if (nh) {
            if (fm) stage_pair<K>(st, __popc(act & ((1u << lane) - 1u)), v, fm);
            if ((int)lane >= nh) stage_pair<K>(st, lane, 0u, (M)0);
        }
        v = vn;
        vn = e + 64 < b1 ? rv.row[e + 64] : 0u;
        fm = e + 32 < b1 ? fprev[v] & ns : (M)0;
        if (!nh) continue;
        __syncwarp();
        pull_rows<K>(st_h, g, S::NSUB, (nh + S::NSUB - 1) / S::NSUB, msigma + 4 * sl, sh, acc, fo);
        __syncwarp();
    }
#pragma unroll
    for (int o = S::SUB; o < 32; o <<= 1) {
#pragma unroll
        for (int q = 0; q < 4; q++) acc[q] += __shfl_xor_sync(FULL_MASK, acc[q], o);
        fo |= __shfl_xor_sync(FULL_MASK, fo, o);
    }
    // the other parts of u add into the same row; subgroup g adds pivots g,
    // g + NSUB, ... of each lane's four
    uint32_t *r = msigma + row_base<K>(u) + 4 * sl;
#pragma unroll
    for (int q = 0; q < 4; q++)
        if ((q & (S::NSUB - 1)) == g && ((fo >> q) & 1u)) {
            atomicAdd(r + q, acc[q]);
            wc.add(WC_PAIRS, 1);
            wc.add(WC_BYTES, 4);
        }
    M nm = (M)__reduce_or_sync(FULL_MASK, sl < 8 ? fo << sh : 0u);
    if (K == 2) nm |= (M)((unsigned long long)__reduce_or_sync(FULL_MASK, sl < 8 ? 0u : fo << sh) << 32);
    bool first = false;
    if (lane == 0 && nm) {
        first = atomicOr(&fcur[u], nm) == 0;
        wc.add(WC_BYTES, first ? 4 + 4 * K : 4 * K);  // level mask, list entry
    }
    list_append(ll, L, first, u);
}

// Up to 32 vertices of at most rv.big in-neighbours, one per lane (pivots
// ns_l; 0: none).  Each subgroup takes one of them at a time: its lanes read
// 8 K positions per step and then gather the rows of those with a parent.
template <int K, class WC>
__device__ __forceinline__ void pull_small(const Adj &rv, uint32_t u_l, typename MaskOf<K>::T ns_l,
                                           const typename MaskOf<K>::T *__restrict__ fprev,
                                           typename MaskOf<K>::T *fcur, uint32_t *msigma, uint2 *st,
                                           const LevelLists &ll, int L, WC &wc)
{
    typedef typename MaskOf<K>::T M;
    typedef PullShape<K> S;
    const unsigned lane = lane_id();
    const int sl = lane & (S::SUB - 1), g = lane / S::SUB;
    const unsigned sh = 4 * (sl & 7);
    const uint2 *st_h = st + (K == 2 && sl >= 8 ? 37 : 0);
    uint32_t b_l = 0, d_l = 0;
    if (ns_l) {
        b_l = rv.col[u_l];
        d_l = rv.col[u_l + 1] - b_l;
        wc.add(WC_BYTES, 8);  // adjacency bounds
    }
    for (unsigned act = __ballot_sync(FULL_MASK, d_l != 0); act;) {
        // the next NSUB vertices, one per subgroup
        int j = -1;
#pragma unroll
        for (int q = 0; q < S::NSUB; q++) {
            if (q == g && act) j = __ffs(act) - 1;
            act &= act - 1;
        }
        const uint32_t u = __shfl_sync(FULL_MASK, u_l, j & 31), b = __shfl_sync(FULL_MASK, b_l, j & 31);
        const M ns = __shfl_sync(FULL_MASK, ns_l, j & 31);
        const uint32_t dj = __shfl_sync(FULL_MASK, d_l, j & 31);
        const uint32_t d = j < 0 ? 0u : dj;
        const uint32_t dmax = __reduce_max_sync(FULL_MASK, d);
        uint32_t acc[4] = {0, 0, 0, 0}, fo = 0;
        uint32_t vn = (uint32_t)sl < d ? rv.row[b + sl] : 0u;
        for (uint32_t s = 0; s < dmax; s += S::SUB) {
            const uint32_t e = s + sl, v = vn;
            vn = e + S::SUB < d ? rv.row[b + e + S::SUB] : 0u;
            M fm = 0;
            if (e < d) {
                fm = fprev[v] & ns;
                wc.add(WC_ENTRIES, 1);
                wc.add(WC_GATHERS, __popcll((unsigned long long)fm));
                wc.add(WC_BYTES, 4 + 4 * K + 4 * __popcll((unsigned long long)fm));  // entry, mask, parents' counts
            }
            const unsigned hit = __ballot_sync(FULL_MASK, fm != 0);
            if (!hit) continue;
            const unsigned mine = (hit >> (S::SUB * g)) & ((1u << S::SUB) - 1u);
            const int nh = __popc(mine);
            if (fm) stage_pair<K>(st, S::SUB * g + __popc(mine & ((1u << sl) - 1u)), v, fm);
            if (sl >= nh) stage_pair<K>(st, S::SUB * g + sl, 0u, (M)0);
            const int most = (int)__reduce_max_sync(FULL_MASK, (unsigned)nh);
            __syncwarp();
            pull_rows<K>(st_h, S::SUB * g, 1, most, msigma + 4 * sl, sh, acc, fo);
            __syncwarp();
        }
        // this vertex has no other part: plain stores
        if (!__any_sync(FULL_MASK, fo != 0)) continue;
        uint32_t *r = msigma + row_base<K>(u) + 4 * sl;
        if (fo & 1u) r[0] = acc[0];
        if (fo & 2u) r[1] = acc[1];
        if (fo & 4u) r[2] = acc[2];
        if (fo & 8u) r[3] = acc[3];
        uint32_t w = fo << sh;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) w |= __shfl_xor_sync(FULL_MASK, w, o);
        M nm = (M)w;
        if (K == 2) nm |= (M)((unsigned long long)__shfl_xor_sync(FULL_MASK, w, 8) << 32);  // read at sl == 0
        const bool isnew = sl == 0 && nm != 0;
        if (isnew) {
            fcur[u] = nm;
            wc.add(WC_PAIRS, __popcll((unsigned long long)nm));
            wc.add(WC_BYTES, 4 + 4 * K + 4 * __popcll((unsigned long long)nm));  // mask, list, counts
        }
        list_append(ll, L, isnew, u);
    }
}

template <int K, class WC>
__device__ __forceinline__ void fwd_pull_body(const Adj &rv, typename MaskOf<K>::T srcmask,
                                              const typename MaskOf<K>::T *__restrict__ fprev,
                                              typename MaskOf<K>::T *fcur,
                                              const typename MaskOf<K>::T *__restrict__ seen, uint32_t *msigma,
                                              uint32_t *ctr, uint2 *st, const LevelLists &ll, int L, WC &wc)
{
    typedef typename MaskOf<K>::T M;
    const unsigned lane = lane_id();
    const uint64_t np = rv.n_part, nl = rv.n_linked - rv.n_big;
    const uint32_t gp = unit_of(np, 1), gl = unit_of(nl, PullShape<K>::NSUB);
    const uint64_t up = (np + gp - 1) / gp, nu = up + (nl + gl - 1) / gl;
    for (uint64_t t = warp_global(); t < nu; t = next_unit(ctr, nu)) {
        uint2 pt = make_uint2(0, 0);
        M ns_l = 0;
        if (t < up) {
            // a unit of parts: one lane looks each part's unseen pivots up
            const uint64_t i = lane * up + t;  // a hub's parts fall into different units
            if (lane < gp && i < np) {
                pt = rv.part[i];
                ns_l = srcmask & ~seen[pt.x];
                wc.add(WC_BYTES, 4 * K);  // seen mask
            }
            for (unsigned act = __ballot_sync(FULL_MASK, ns_l != 0); act; act &= act - 1) {
                const int j = __ffs(act) - 1;
                const uint32_t u = __shfl_sync(FULL_MASK, pt.x, j);
                const uint32_t b0 = rv.col[u] + __shfl_sync(FULL_MASK, pt.y, j) * rv.part_len;
                pull_part<K>(rv, u, __shfl_sync(FULL_MASK, ns_l, j), b0, min(rv.col[u + 1], b0 + rv.part_len), fprev,
                             fcur, msigma, st, ll, L, wc);
            }
            continue;
        }
        const uint64_t i = (t - up) * gl + lane;
        uint32_t u_l = 0;
        if (lane < gl && i < nl) {
            u_l = rv.order[rv.n_big + i];
            ns_l = srcmask & ~seen[u_l];
            wc.add(WC_BYTES, 4 * K);  // seen mask
        }
        pull_small<K>(rv, u_l, ns_l, fprev, fcur, msigma, st, ll, L, wc);
    }
}

// One forward level, device-driven: the level is bi->cur + 1 and the direction
// bi->push_next (set when the previous level was closed); nothing once a level
// discovered nothing.  CNT: the counting build (work counts into
// wc[KP_FWD_PUSH / KP_FWD_PULL]).
template <int K, bool CNT>
__global__ void __launch_bounds__(BATCH_TPB, FWD_BLOCKS(K)) k_fwd_step(Adj a, Adj rv, const BatchInfo *__restrict__ bi,
                                                             uint32_t *const *__restrict__ tab,
                                                             const uint32_t *__restrict__ seen,
                                                             uint32_t *msigma, uint32_t *ctrs,
                                                             LevelLists ll, unsigned long long *wc)
{
    typedef typename MaskOf<K>::T M;
    __shared__ uint2 s_st[BATCH_TPB / 32][PullShape<K>::STAGE];
    if (!bi->alive) return;
    const int L = bi->cur + 1, push = bi->push_next;
    WorkCount<CNT> cnt;
    const M *fprev = reinterpret_cast<const M *>(tab[L - 1]);
    M *fcur = reinterpret_cast<M *>(tab[L]);
    if (push)
        fwd_push_body<K>(a, fprev, fcur, reinterpret_cast<const M *>(seen), msigma, ctrs + 2 * L, ll, L,
                         reinterpret_cast<uint32_t *>(s_st[threadIdx.x >> 5]), cnt);
    else
        fwd_pull_body<K>(rv, (M)bi->srcmask, fprev, fcur, reinterpret_cast<const M *>(seen), msigma, ctrs + 2 * L,
                         s_st[threadIdx.x >> 5], ll, L, cnt);
    cnt.flush(wc + (push ? KP_FWD_PUSH : KP_FWD_PULL) * WC_NFIELDS);
}

// After level L = bi->cur + 1: fold the level mask into `seen` and count, per
// pivot, the vertices reached, their degree sum and their reach sum; subtract
// from the unvisited-edge total the in-degrees of vertices now seen by every
// pivot.  Visits only level L's list when stored.
template <class M>
__device__ __forceinline__ void stats_vertex(uint64_t u, M srcmask, const M *__restrict__ fcur, M *seen,
                                             const uint32_t *__restrict__ col,
                                             const uint32_t *__restrict__ rcol,
                                             const uint32_t *__restrict__ reach, M &nm,
                                             uint32_t &d, uint32_t &r, unsigned long long &fdeg,
                                             unsigned long long &udec, bool &any)
{
    nm = fcur[u];
    if (!nm) return;
    any = true;
    const M sn = seen[u];
    const M sn2 = sn | nm;
    seen[u] = sn2;
    d = col[u + 1] - col[u];
    r = reach[u];
    fdeg += d;
    if ((sn & srcmask) != srcmask && (sn2 & srcmask) == srcmask) udec += rcol[u + 1] - rcol[u];
}

// a block's totals: per pivot vertices, degrees and reach, then the level's
// degree sum, frontier degrees, unvisited decrease, big vertices, and whether any
template <int K> struct StatsShared {
    unsigned long long x[3 * 32 * K + 5];
};
template <int K>
__device__ __forceinline__ void stats_body(uint64_t n, BatchInfo *bi, int L, typename MaskOf<K>::T srcmask,
                                           const typename MaskOf<K>::T *__restrict__ fcur,
                                           typename MaskOf<K>::T *seen, const uint32_t *__restrict__ col,
                                           const uint32_t *__restrict__ rcol,
                                           const uint32_t *__restrict__ reach, uint32_t big, StatsShared<K> &sh,
                                           const LevelLists &ll)
{
    typedef typename MaskOf<K>::T M;
    const unsigned lane = lane_id();
    const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
    uint32_t lcnt = 0;
    const uint32_t *lst = level_list(ll, L, lcnt);
    const uint64_t items = lst ? lcnt : n;
    const uint64_t nblk = (items + 31) / 32;
    const uint64_t nw = nthreads / 32;
    unsigned long long cnt[K], te[K], rs[K];
#pragma unroll
    for (int h = 0; h < K; h++) cnt[h] = te[h] = rs[h] = 0;
    unsigned long long fdeg = 0, udec = 0, tsum = 0;
    uint32_t hv = 0;  // big vertices of the level (their parts or span items are scanned)
    bool any = false;
    for (uint64_t t = tid / 32; t < nblk; t += nw) {
        const uint64_t i = t * 32 + lane;
        M nm = 0;
        uint32_t d = 0, r = 0;
        if (i < items) {
            const uint64_t u = lst ? lst[i] : i;
            stats_vertex<M>(u, srcmask, fcur, seen, col, rcol, reach, nm, d, r, fdeg, udec, any);
            if (nm && d > big) hv++;
            tsum += (unsigned long long)d * __popcll((unsigned long long)nm);
        }
        unsigned act = __ballot_sync(FULL_MASK, nm != 0);
        while (act) {
            const int j = __ffs(act) - 1;
            act &= act - 1;
            const M mj = __shfl_sync(FULL_MASK, nm, j);
            const uint32_t dj = __shfl_sync(FULL_MASK, d, j);
            const uint32_t rj = __shfl_sync(FULL_MASK, r, j);
#pragma unroll
            for (int h = 0; h < K; h++)
                if (pbit(mj, h)) {
                    cnt[h]++;
                    te[h] += dj;
                    rs[h] += rj;
                }
        }
    }
    // the block's totals in shared memory first: ten thousand warps adding to
    // the same few lines took most of this kernel's time
    {
        uint32_t hsum = hv;
        for (int o = 16; o; o >>= 1) {
            tsum += __shfl_xor_sync(FULL_MASK, tsum, o);
            fdeg += __shfl_xor_sync(FULL_MASK, fdeg, o);
            udec += __shfl_xor_sync(FULL_MASK, udec, o);
            hsum += __shfl_xor_sync(FULL_MASK, hsum, o);
        }
        any = __any_sync(FULL_MASK, any);
        for (uint32_t i = threadIdx.x; i < 3 * 32 * K + 5; i += blockDim.x) sh.x[i] = 0;
        __syncthreads();
        if (any) {
            if (lane == 0) {
                atomicAdd(&sh.x[96 * K], tsum);
                atomicAdd(&sh.x[96 * K + 1], fdeg);
                atomicAdd(&sh.x[96 * K + 2], udec);
                atomicAdd(&sh.x[96 * K + 3], (unsigned long long)hsum);
                sh.x[96 * K + 4] = 1;
            }
#pragma unroll
            for (int h = 0; h < K; h++)
                if (cnt[h]) {
                    const int s = lane + 32 * h;
                    atomicAdd(&sh.x[s], cnt[h]);
                    atomicAdd(&sh.x[32 * K + s], te[h]);
                    atomicAdd(&sh.x[64 * K + s], rs[h]);
                }
        }
        __syncthreads();
    }
    if (!sh.x[96 * K + 4]) return;
    for (int s = threadIdx.x; s < 32 * K; s += blockDim.x)
        if (sh.x[s]) {
            atomicAdd(&bi->lvl_new[s], sh.x[s]);
            atomicAdd(&bi->nvis[s], sh.x[s]);
            atomicAdd(&bi->te[s], sh.x[32 * K + s]);
            atomicAdd(&bi->rsum[s], sh.x[64 * K + s]);
        }
    if (threadIdx.x == blockDim.x - 1) {
        if (sh.x[96 * K]) atomicAdd(&bi->lvl_te, sh.x[96 * K]);
        if (sh.x[96 * K + 1]) atomicAdd(&bi->front_deg, sh.x[96 * K + 1]);
        if (sh.x[96 * K + 2]) atomicAdd(&bi->unvis_dec, sh.x[96 * K + 2]);
        if (sh.x[96 * K + 3]) atomicAdd(&ll.heavy[L], (uint32_t)sh.x[96 * K + 3]);
        atomicOr(&bi->any_new, 1u);
    }
}

// Close forward level L = bi->cur + 1 (one warp, lane l for pivots l + 32 h):
// per-pivot termination, the per-level totals, the direction of the next
// level, and -- once nothing was discovered -- the deepest depth and the
// depth-0 pivots of the backward pass.
template <int K>
__device__ __forceinline__ void level_advance_warp(BatchInfo *bi, unsigned long long *level_te,
                                                   unsigned long long *level_cnt, int32_t *level_mode,
                                                   const LevelLists &ll, uint32_t pool_cap,
                                                   uint32_t list_max)
{
    const unsigned l = lane_id();
    const int L = __ldcg(&bi->cur) + 1;
    const uint32_t nsrc = bi->nsrc;
    // every total loads before the first is used
    const unsigned long long front = __ldcg(&bi->front_deg), unvis = __ldcg(&bi->unvis_deg) - __ldcg(&bi->unvis_dec);
    const unsigned long long lvl_te = __ldcg(&bi->lvl_te);
    const uint32_t listed = __ldcg(&ll.count[L]), cap = __ldcg(&ll.cap[L]), start = __ldcg(&ll.start[L]);
    const uint32_t any_new = __ldcg(&bi->any_new);
    unsigned long long cnt = 0, d0 = 0;
#pragma unroll
    for (int h = 0; h < K; h++) {
        const uint32_t s = l + 32 * h;
        const unsigned long long nw = s < nsrc ? __ldcg(&bi->lvl_new[s]) : 0ull;
        if (s < nsrc && bi->Ls[s] == 0 && nw == 0) bi->Ls[s] = L;
        cnt += nw;
        const bool two = s < nsrc && bi->Ls[s] == 2;
        d0 |= (unsigned long long)__ballot_sync(FULL_MASK, two) << (32 * h);
    }
    for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(FULL_MASK, cnt, o);
    __syncwarp();
    if (l == 0) {
        level_te[L] = lvl_te;
        level_cnt[L] = cnt;
        level_mode[L] = bi->push_next;
        bi->unvis_deg = unvis;
        bi->unvis_dec = 0;
        // push from a frontier whose degree sum is small against the graph:
        // a pull would scan every vertex some pivot has not seen
        const bool push = (double)front * bi->push_factor < (double)unvis || front < bi->push_min;
        // where level L+1's list goes and how long it may grow
        const uint32_t used = start + (listed <= cap ? listed : 0u);
        ll.start[L + 1] = used;
        ll.cap[L + 1] = min(list_max, pool_cap - min(pool_cap, used));
        if (pool_cap - min(pool_cap, used) < list_max) bi->pool_short = 1;
        if (!any_new) {
            bi->alive = 0;
            bi->lend = L;
            bi->dmax = L - 1;
            bi->depth0mask = d0;
        }
        bi->push_next = push;
        bi->cur = L;
        bi->lvl_te = 0;
        bi->front_deg = 0;
        bi->any_new = 0;
    }
#pragma unroll
    for (int h = 0; h < K; h++) bi->lvl_new[l + 32 * h] = 0;
}

// The level's statistics; the last block to finish closes the level.
template <int K>
__global__ void __launch_bounds__(BATCH_TPB) k_stats_step(uint64_t n, BatchInfo *bi, uint32_t *const *__restrict__ tab,
                                                          uint32_t *seen, const uint32_t *__restrict__ col,
                                                          const uint32_t *__restrict__ rcol,
                                                          const uint32_t *__restrict__ reach, LevelLists ll,
                                                          unsigned long long *level_te,
                                                          unsigned long long *level_cnt, int32_t *level_mode,
                                                          uint32_t pool_cap, uint32_t list_max, uint32_t big)
{
    typedef typename MaskOf<K>::T M;
    __shared__ StatsShared<K> sh;
    if (!__ldcg(&bi->alive)) return;
    const int L = __ldcg(&bi->cur) + 1;
    stats_body<K>(n, bi, L, (M)__ldcg(&bi->srcmask), reinterpret_cast<const M *>(tab[L]), reinterpret_cast<M *>(seen),
                  col, rcol, reach, big, sh, ll);
    if (last_block(&bi->ticket[1]) && threadIdx.x < 32)
        level_advance_warp<K>(bi, level_te, level_cnt, level_mode, ll, pool_cap, list_max);
}

// The backward pass runs one 32-pivot half of a pass at a time (hh = 0, or 0
// and 1 for a 64-pivot pass): lane l owns pivot l + 32 hh.  The functions
// below see the half through offset pointers: level masks as 32-bit words at
// stride K (word hh of each vertex's mask, little-endian), rows and span
// partials shifted by 32 hh columns.  A half has the register footprint of a
// 32-pivot pass, which keeps 8 blocks per SM resident for this latency-bound
// kernel.
template <int K> __device__ __forceinline__ uint32_t half_of(typename MaskOf<K>::T m, int hh)
{
    return (uint32_t)((unsigned long long)m >> (32 * hh));
}

// Layout of the dependency sums: a lane owns four neighbouring pivots (one
// 16-byte load per successor row) and eight lanes cover the half's 32; the
// warp's four groups of eight lanes work on the four 8-position subtrees of a
// chunk's canonical tree (or on four tiny vertices) at once, so that 16 rows
// are in flight per load round at one quarter of the load, address and
// test instructions of one row per instruction.  Folding the four subtrees
// leaves the lane with the sum of one pivot, own_pivot().
__device__ __forceinline__ int own_slot() { return 2 * ((lane_id() >> 3) & 1) + (lane_id() >> 4); }
__device__ __forceinline__ int own_pivot() { return 4 * (lane_id() & 7) + own_slot(); }
__device__ __forceinline__ float own_of(const float s[4])
{
    const unsigned lane = lane_id();
    const float a = lane & 16 ? s[1] : s[0], b = lane & 16 ? s[3] : s[2];
    return lane & 8 ? b : a;
}

// Terms of four staged successors as a tree (pairs differing in the lowest
// position bit first).  q[u][s] = (delta_s[u] + 1) / sigma_s[u] was stored when
// u's dependency was final, so a term is q * sigma_s[v], bit for bit the
// reference's ((delta + 1) / sigma[r]) * sigma[c].  mq_l points at the lane's
// columns of row 0.
template <int K>
__device__ __forceinline__ void quad_sum(const uint2 *st, const float *__restrict__ mq_l, unsigned sh,
                                         const float sv[4], float out[4])
{
    float4 x[4];
    uint32_t nb[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint2 e = st[j];
        nb[j] = (e.y >> sh) & 15u;
        x[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (nb[j]) x[j] = *reinterpret_cast<const float4 *>(mq_l + row_base<K>(e.x));
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        float t[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float xq = q == 0 ? x[j].x : q == 1 ? x[j].y : q == 2 ? x[j].z : x[j].w;
            t[j] = (nb[j] >> q) & 1u ? __fmul_rn(xq, sv[q]) : 0.0f;
        }
        out[q] = __fadd_rn(__fadd_rn(t[0], t[1]), __fadd_rn(t[2], t[3]));
    }
}

// The 8-position subtree sums of the lane's group for its four pivots, of the
// chunk whose lanes hold successors u with pivots gm (pm: lanes with any).  A
// quad of positions without successors in any group sums to +0 and is skipped.
template <int K>
__device__ __forceinline__ void group_sums(uint2 *st, uint32_t u, uint32_t gm, unsigned pm,
                                           const float *__restrict__ mq_l, const float sv[4], float s[4])
{
    const unsigned lane = lane_id(), g9 = 9 * (lane >> 3), sh = 4 * (lane & 7);
    st[g9 + (lane & 7)] = make_uint2(u, gm);
    __syncwarp();
    unsigned pj = pm | pm >> 16;
    pj |= pj >> 8;
    float b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    s[0] = s[1] = s[2] = s[3] = 0.0f;
    if (pj & 0x0fu) quad_sum<K>(st + g9, mq_l, sh, sv, s);
    if (pj & 0xf0u) quad_sum<K>(st + g9 + 4, mq_l, sh, sv, b);
#pragma unroll
    for (int q = 0; q < 4; q++) s[q] = __fadd_rn(s[q], b[q]);
    __syncwarp();
}

// The top two levels of the chunk's tree: groups g and g ^ 1, then the two
// halves, each lane keeping fewer pivots of more positions.
__device__ __forceinline__ float fold_groups(const float s[4])
{
    const unsigned lane = lane_id();
    const bool h1 = (lane & 8) != 0, h2 = (lane & 16) != 0;
    const float r0 = __fadd_rn(h1 ? s[2] : s[0], __shfl_xor_sync(FULL_MASK, h1 ? s[0] : s[2], 8));
    const float r1 = __fadd_rn(h1 ? s[3] : s[1], __shfl_xor_sync(FULL_MASK, h1 ? s[1] : s[3], 8));
    return __fadd_rn(h2 ? r1 : r0, __shfl_xor_sync(FULL_MASK, h2 ? r0 : r1, 16));
}

// path counts of v for the lane's four pivots (of those in f)
template <int K>
__device__ __forceinline__ void load_sv(const uint32_t *__restrict__ msigma, uint32_t v, uint32_t f, float sv[4])
{
    const unsigned l = lane_id() & 7;
    uint4 x = make_uint4(0, 0, 0, 0);
    if ((f >> (4 * l)) & 15u) x = *reinterpret_cast<const uint4 *>(msigma + row_base<K>(v) + 4 * l);
    sv[0] = __uint2float_rn(x.x);
    sv[1] = __uint2float_rn(x.y);
    sv[2] = __uint2float_rn(x.z);
    sv[3] = __uint2float_rn(x.w);
}

// delta and q of vertex v for one pivot; sv: its path count
template <int K>
__device__ __forceinline__ void write_dep(float *mdelta, float *mq, uint32_t v, int pivot, float delta, float sv)
{
    mdelta[row_base<K>(v) + pivot] = delta;
    mq[row_base<K>(v) + pivot] = __fdiv_rn(__fadd_rn(delta, 1.0f), sv);
}

// work counts of one lane's adjacency entry
template <class WC> __device__ __forceinline__ void count_entry(WC &wc, bool valid, uint32_t gm)
{
    if (!valid) return;
    wc.add(WC_ENTRIES, 1);
    wc.add(WC_GATHERS, __popc(gm));
    wc.add(WC_BYTES, 8 + 4 * __popc(gm));  // adjacency entry, level mask word, successors' q
}

// Backward depth d for the half's pivots: arrays of one pass half.
struct BwdHalf {
    uint32_t dmask;   // the half's pivots that are processed at this depth
    int no_succ;      // the deepest depth: nothing lies below, delta = reach
    const uint32_t *fd, *fnext;
    const uint32_t *msigma;
    float *mdelta, *mq, *mpartial;
    uint32_t *harrive;
    const uint32_t *reach;
};

// Positions [b0, b1) of a vertex by one warp: chunk sums left to right, own
// pivot per lane.  Adjacency entries load two chunks ahead and level masks one.
template <int K, class WC>
__device__ __forceinline__ float bwd_span(const Adj &a, const BwdHalf &B, uint32_t f, const float sv[4], uint32_t b0,
                                          uint32_t b1, uint2 *st, WC &wc)
{
    const unsigned lane = lane_id();
    float P = 0.0f;
    if (!B.no_succ) {
        const float *mq_l = B.mq + 4 * (lane & 7);
        uint32_t e = b0 + lane;
        uint32_t u = e < b1 ? a.row[e] : 0u, un = e + 32 < b1 ? a.row[e + 32] : 0u;
        uint32_t gm = e < b1 ? B.fnext[(uint64_t)u * K] & f : 0u;
        for (; e - lane < b1; e += 32) {
            count_entry(wc, e < b1, gm);
            const uint32_t uc = u, gc = gm;
            u = un;
            un = e + 64 < b1 ? a.row[e + 64] : 0u;
            gm = e + 32 < b1 ? B.fnext[(uint64_t)u * K] & f : 0u;
            const unsigned pm = __ballot_sync(FULL_MASK, gc != 0);
            if (!pm) continue;
            float s[4];
            group_sums<K>(st, uc, gc, pm, mq_l, sv, s);
            P = __fadd_rn(P, fold_groups(s));
        }
    }
    return P;
}

// Vertices of at most a.big neighbours, one per lane (pivots f_l; 0: none):
// those of at most 8 four at a time, one group of lanes each, the others one
// by one.
template <int K, class WC>
__device__ __forceinline__ void bwd_small(const Adj &a, const BwdHalf &B, uint32_t v_l, uint32_t f_l, uint2 *st,
                                          WC &wc)
{
    const unsigned lane = lane_id();
    const int l = lane & 7, g = lane >> 3;
    if (!__ballot_sync(FULL_MASK, f_l != 0)) return;
    uint32_t b_l = 0, d_l = 0;
    if (f_l) {
        b_l = a.col[v_l];
        d_l = a.col[v_l + 1] - b_l;
        if (d_l > a.big) f_l = 0;  // in a tile
    }
    if (f_l) {
        // adjacency bounds and reach; per pivot its path count read, its
        // dependency and q written
        wc.add(WC_BYTES, (B.no_succ ? 4 : 12) + 12 * __popc(f_l));
        wc.add(WC_PAIRS, __popc(f_l));
    }
    for (unsigned act = __ballot_sync(FULL_MASK, f_l != 0 && d_l > 8); act; act &= act - 1) {
        const int j = __ffs(act) - 1;
        const uint32_t v = __shfl_sync(FULL_MASK, v_l, j), f = __shfl_sync(FULL_MASK, f_l, j);
        const uint32_t b0 = __shfl_sync(FULL_MASK, b_l, j);
        float sv[4];
        load_sv<K>(B.msigma, v, f, sv);
        const float P = bwd_span<K>(a, B, f, sv, b0, b0 + __shfl_sync(FULL_MASK, d_l, j), st, wc);
        if ((f >> own_pivot()) & 1u)
            write_dep<K>(B.mdelta, B.mq, v, own_pivot(), __fadd_rn(__uint2float_rn(B.reach[v]), P), own_of(sv));
    }
    for (unsigned act = __ballot_sync(FULL_MASK, f_l != 0 && d_l <= 8); act;) {
        int j = -1;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (q == g && act) j = __ffs(act) - 1;
            act &= act - 1;
        }
        const uint32_t v = __shfl_sync(FULL_MASK, v_l, j & 31), fj = __shfl_sync(FULL_MASK, f_l, j & 31);
        const uint32_t b0 = __shfl_sync(FULL_MASK, b_l, j & 31), dj = __shfl_sync(FULL_MASK, d_l, j & 31);
        const uint32_t f = j < 0 ? 0u : fj, d = j < 0 || B.no_succ ? 0u : dj;
        const uint32_t u = (uint32_t)l < d ? a.row[b0 + l] : 0u;
        float sv[4], s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        load_sv<K>(B.msigma, v, f, sv);
        const uint32_t gm = (uint32_t)l < d ? B.fnext[(uint64_t)u * K] & f : 0u;
        count_entry(wc, (uint32_t)l < d, gm);
        const unsigned pm = __ballot_sync(FULL_MASK, gm != 0);
        if (pm) group_sums<K>(st, u, gm, pm, B.mq + 4 * l, sv, s);
        if (f) {
            const float rf = __uint2float_rn(B.reach[v]);
#pragma unroll
            for (int q = 0; q < 4; q++)
                if ((f >> (4 * l + q)) & 1u) write_dep<K>(B.mdelta, B.mq, v, 4 * l + q, __fadd_rn(rf, s[q]), sv[q]);
        }
    }
}

// The span sums of a heavy vertex added in span order: delta and q of the
// lane's pivot `own`.  Out of line: once per heavy vertex, and inlined it would
// cost the traversal loops registers.
template <int K>
__device__ __noinline__ void bwd_combine(const float *part, uint32_t spans, const uint32_t *reach,
                                         const uint32_t *msigma, float *mdelta, float *mq, uint32_t v, bool mine,
                                         int own)
{
    float acc = __uint2float_rn(reach[v]);
    for (uint32_t i = 0; i < spans; i += 8) {
        float x[8];
#pragma unroll
        for (int q = 0; q < 8; q++) x[q] = i + q < spans ? __ldcg(part + (uint64_t)(i + q) * (AXBC_W * K)) : 0.0f;
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (i + q < spans) acc = __fadd_rn(acc, x[q]);
    }
    if (mine) write_dep<K>(mdelta, mq, v, own, acc, __uint2float_rn(msigma[row_base<K>(v) + own]));
}

// The span sum P of a heavy vertex is written (own: the lane's pivot); the warp
// that writes the vertex's last one adds them up.
template <int K>
__device__ __forceinline__ void bwd_span_done(const Adj &a, const BwdHalf &B, uint32_t v, uint32_t f, uint32_t hx,
                                              uint64_t row, uint32_t k, int own, float P)
{
    const unsigned lane = lane_id();
    B.mpartial[row * (AXBC_W * K) + lane] = P;
    __threadfence();
    __syncwarp();
    const uint32_t spans = (a.col[v + 1] - a.col[v] + AXBC_SPAN - 1) / AXBC_SPAN;
    uint32_t last = 0;
    if (lane == 0) {
        last = atomicAdd(&B.harrive[hx], 1u) == spans - 1;
        if (last) B.harrive[hx] = 0;
    }
    if (!__shfl_sync(FULL_MASK, last, 0)) return;
    __threadfence();
    bwd_combine<K>(B.mpartial + (row - k) * (AXBC_W * K) + lane, spans, B.reach, B.msigma, B.mdelta, B.mq, v,
                   (f >> own) & 1u, own);
}

// A tile of big vertices by one block: its chunks go round the warps (up to
// four each, their adjacency entries and then their masks loaded together),
// the chunk sums meet in shared memory and are added left to right.  A span of
// 1024 positions on one warp took 42 us, longer than a whole depth of a
// scale-14 graph should.
template <int K, class WC>
__device__ __forceinline__ void bwd_tile(const Adj &a, const BwdHalf &B, uint64_t t, uint2 tl, uint2 *st,
                                         float (*csum)[32], WC &wc)
{
    constexpr int NW = BATCH_TPB / 32;
    const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
    const bool span = (tl.y & BWD_SPAN_TILE) != 0;
    const uint32_t k = span ? tl.y & ~BWD_SPAN_TILE : 0u, cnt = span ? 1u : tl.y;
    uint32_t v_l = 0, f_l = 0, b_l = 0, e_l = 0, c_l = 0;
    if (lane < cnt) {
        v_l = a.order[tl.x + lane];
        f_l = B.fd[(uint64_t)v_l * K] & B.dmask;
    }
    if (f_l) {
        b_l = a.col[v_l] + k * AXBC_SPAN;
        e_l = min(a.col[v_l + 1], b_l + AXBC_SPAN);
        if (!B.no_succ) c_l = (e_l - b_l + AXBC_CHUNK - 1) / AXBC_CHUNK;
        if (wid == 0) {
            wc.add(WC_BYTES, span ? 4 + 8 * __popc(f_l) : (B.no_succ ? 4 : 12) + 12 * __popc(f_l));
            if (!span) wc.add(WC_PAIRS, __popc(f_l));
        }
    }
    uint32_t inc = c_l;  // chunks up to and including this vertex's
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        const uint32_t x = __shfl_up_sync(FULL_MASK, inc, o);
        if ((int)lane >= o) inc += x;
    }
    const uint32_t S = __shfl_sync(FULL_MASK, inc, 15);  // at most 16 vertices of two chunks
    const float *mq_l = B.mq + 4 * (lane & 7);
    uint32_t u[BWD_TILE_CHUNKS / NW], gm[BWD_TILE_CHUNKS / NW];
#pragma unroll
    for (int i = 0; i < BWD_TILE_CHUNKS / NW; i++) {
        const uint32_t s = wid + NW * i;
        u[i] = 0xffffffffu;
        if (s < S) {
            const int j = __popc(__ballot_sync(FULL_MASK, lane < 16 && inc <= s));
            const uint32_t e = __shfl_sync(FULL_MASK, b_l + AXBC_CHUNK * (s - (inc - c_l)), j) + lane;
            if (e < __shfl_sync(FULL_MASK, e_l, j)) u[i] = a.row[e];
        }
    }
#pragma unroll
    for (int i = 0; i < BWD_TILE_CHUNKS / NW; i++) {
        const uint32_t s = wid + NW * i;
        gm[i] = 0;
        if (s < S) {
            const int j = __popc(__ballot_sync(FULL_MASK, lane < 16 && inc <= s));
            const uint32_t f = __shfl_sync(FULL_MASK, f_l, j);
            if (u[i] != 0xffffffffu) gm[i] = B.fnext[(uint64_t)u[i] * K] & f;
            count_entry(wc, u[i] != 0xffffffffu, gm[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < BWD_TILE_CHUNKS / NW; i++) {
        const uint32_t s = wid + NW * i;
        if (s >= S) break;
        const unsigned pm = __ballot_sync(FULL_MASK, gm[i] != 0);
        float r = 0.0f;
        if (pm) {
            const int j = __popc(__ballot_sync(FULL_MASK, lane < 16 && inc <= s));
            float sv[4], q[4];
            load_sv<K>(B.msigma, __shfl_sync(FULL_MASK, v_l, j), __shfl_sync(FULL_MASK, f_l, j), sv);
            group_sums<K>(st, u[i], gm[i], pm, mq_l, sv, q);
            r = fold_groups(q);
        }
        csum[s][lane] = r;
    }
    __syncthreads();
    for (uint32_t j = wid; j < cnt; j += NW) {
        const uint32_t f = __shfl_sync(FULL_MASK, f_l, j);
        if (!f) continue;
        const uint32_t v = __shfl_sync(FULL_MASK, v_l, j), s1 = __shfl_sync(FULL_MASK, inc, j);
        float P = 0.0f;
        for (uint32_t s = s1 - __shfl_sync(FULL_MASK, c_l, j); s < s1; s++) P = __fadd_rn(P, csum[s][lane]);
        if (span) {
            bwd_span_done<K>(a, B, v, f, tl.x, t, k, own_pivot(), P);
        } else if ((f >> own_pivot()) & 1u) {
            const float sv = __uint2float_rn(B.msigma[row_base<K>(v) + own_pivot()]);
            write_dep<K>(B.mdelta, B.mq, v, own_pivot(), __fadd_rn(__uint2float_rn(B.reach[v]), P), sv);
        }
    }
}

template <int K, class WC>
__device__ __forceinline__ void bwd_body(const Adj &a, const BwdHalf &B, uint32_t *ctr, uint2 *st,
                                         float (*csum)[BWD_TILE_CHUNKS][32], const uint32_t *lst, uint32_t lcnt,
                                         uint32_t lheavy, int symmetric, WC &wc)
{
    const unsigned lane = lane_id();
    // tiles only when a big vertex is at this depth; every warp of a block
    // looks up the same 32 tiles and walks those with a vertex at this depth
    if (!(lst && lheavy == 0)) {
        int buf = 0;
        for (uint64_t base = blockIdx.x; base < a.n_tile; base += 32ull * gridDim.x) {
            const uint64_t t_l = base + (uint64_t)lane * gridDim.x;
            uint2 tl = make_uint2(0, 0);
            uint32_t any = 0;
            if (t_l < a.n_tile) {
                tl = a.tile[t_l];
                const uint32_t cnt = tl.y & BWD_SPAN_TILE ? 1u : tl.y;
                for (uint32_t j = 0; j < cnt; j++) any |= B.fd[(uint64_t)a.order[tl.x + j] * K];
                if (threadIdx.x < 32) wc.add(WC_BYTES, 4 * cnt);  // level mask words
            }
            for (unsigned act = __ballot_sync(FULL_MASK, (any & B.dmask) != 0); act; act &= act - 1, buf ^= 1) {
                const int j = __ffs(act) - 1;
                bwd_tile<K>(a, B, base + (uint64_t)j * gridDim.x,
                            make_uint2(__shfl_sync(FULL_MASK, tl.x, j), __shfl_sync(FULL_MASK, tl.y, j)), st,
                            csum[buf], wc);
            }
        }
    }
    // the others by warps, from the level's list or by a scan; a directed
    // graph's vertices without out-neighbours are at some depth too
    const uint64_t nl = lst ? lcnt : (symmetric ? a.n_linked : a.n) - a.n_big;
    const uint32_t ent = unit_of(nl, 1);
    const uint64_t nu = (nl + ent - 1) / ent;
    for (uint64_t t = warp_global(); t < nu; t = next_unit(ctr, nu)) {
        const uint64_t i = t * ent + lane;
        uint32_t v_l = 0, f_l = 0;
        if (lane < ent && i < nl) {
            v_l = lst ? lst[i] : a.order[a.n_big + i];
            f_l = B.fd[(uint64_t)v_l * K] & B.dmask;
            wc.add(WC_BYTES, lst ? 8 : 4);  // list entry, level mask word
        }
        bwd_small<K>(a, B, v_l, f_l, st, wc);
    }
}

// eight staged words of group g (16-byte shared loads)
__device__ __forceinline__ void load8u(const uint32_t *su, int g, uint32_t u[8])
{
    const uint4 *p = reinterpret_cast<const uint4 *>(su) + 2 * g;
    const uint4 a = p[0], b = p[1];
    u[0] = a.x, u[1] = a.y, u[2] = a.z, u[3] = a.w, u[4] = b.x, u[5] = b.y, u[6] = b.z, u[7] = b.w;
}

// Sum of the 8 staged successor terms of group g as a balanced tree (pairs
// differing in the lowest position bit first).  mq_l points at the lane's
// column of row 0.
template <int K>
__device__ __forceinline__ float tree8(const uint32_t *su, const uint32_t *sg, int g, const float *__restrict__ mq_l,
                                       float sv)
{
    uint32_t u[8], m[8];
    load8u(su, g, u);
    load8u(sg, g, m);
    const unsigned lane = lane_id();
    float t[8];
#pragma unroll
    for (int jj = 0; jj < 8; jj++) {
        const bool hit = (m[jj] >> lane) & 1u;
        const float q = hit ? mq_l[row_base<K>(u[jj])] : 0.0f;
        t[jj] = hit ? __fmul_rn(q, sv) : 0.0f;
    }
    const float a = __fadd_rn(__fadd_rn(t[0], t[1]), __fadd_rn(t[2], t[3]));
    const float b = __fadd_rn(__fadd_rn(t[4], t[5]), __fadd_rn(t[6], t[7]));
    return __fadd_rn(a, b);
}

// the same for a subtree whose successors all lie in one half of it (quad: the
// half's number in the chunk): the other half sums to +0
template <int K>
__device__ __forceinline__ float tree4(const uint32_t *su, const uint32_t *sg, int quad, const float *__restrict__ mq_l, float sv)
{
    const uint4 u4 = reinterpret_cast<const uint4 *>(su)[quad], m4 = reinterpret_cast<const uint4 *>(sg)[quad];
    const uint32_t u[4] = {u4.x, u4.y, u4.z, u4.w}, m[4] = {m4.x, m4.y, m4.z, m4.w};
    const unsigned lane = lane_id();
    float t[4];
#pragma unroll
    for (int jj = 0; jj < 4; jj++) {
        const bool hit = (m[jj] >> lane) & 1u;
        const float q = hit ? mq_l[row_base<K>(u[jj])] : 0.0f;
        t[jj] = hit ? __fmul_rn(q, sv) : 0.0f;
    }
    return __fadd_rn(__fadd_rn(t[0], t[1]), __fadd_rn(t[2], t[3]));
}
template <int K>
__device__ __forceinline__ float subtree(const uint32_t *su, const uint32_t *sg, int g, unsigned pm, const float *__restrict__ mq_l,
                                         float sv)
{
    const unsigned h = (pm >> (8 * g)) & 0xffu;
    if (!h) return 0.0f;
    if (!(h & 0xf0u)) return tree4<K>(su, sg, 2 * g, mq_l, sv);
    if (!(h & 0x0fu)) return tree4<K>(su, sg, 2 * g + 1, mq_l, sv);
    return tree8<K>(su, sg, g, mq_l, sv);
}

// List entries per work unit: 32, or fewer when the list is too short to give
// every resident warp a unit (a short list of high-degree vertices would
// otherwise sit on a few warps).
__device__ __forceinline__ uint32_t list_unit(uint32_t lcnt)
{
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    return max(1u, min(32u, lcnt / nwarps));
}

// Canonical dependency sum of vertex v over adjacency positions [b0,b1) for
// the half's pivots in f.  q[u][s] = (delta_s[u] + 1) / sigma_s[u] was stored
// when u's dependency was final, so a successor term is q * sigma_s[v], bit for
// bit the reference's ((delta + 1) / sigma[r]) * sigma[c].  The 32 positions
// of a chunk form four 8-position subtrees of the canonical tree; a subtree
// without successors sums to +0 and is skipped.  `un` holds the adjacency
// entries of the first chunk (row[b0 + lane]).
template <int K, class WC>
__device__ __forceinline__ float dep_span_from(const Adj &a, uint32_t f, float sv, uint32_t b0, uint32_t b1,
                                               uint32_t un, const uint32_t *__restrict__ fnext,
                                               const float *__restrict__ mq, uint32_t *su, uint32_t *sg, WC &wc)
{
    const unsigned lane = lane_id();
    const float *mq_l = mq + lane;
    float P = 0.0f;
    // the next chunk's adjacency entries load while this chunk is consumed
    for (uint32_t base = b0; base < b1; base += 32) {
        const uint32_t e = base + lane;
        const uint32_t u = un;
        un = e + 32 < b1 ? a.row[e + 32] : 0u;
        const uint32_t gm = e < b1 ? fnext[(uint64_t)u * K] & f : 0u;
        if (e < b1) {
            wc.add(WC_ENTRIES, 1);
            wc.add(WC_GATHERS, __popc(gm));
            wc.add(WC_BYTES, 8 + 4 * __popc(gm));  // adjacency entry, level mask word, successors' q
        }
        const unsigned pm = __ballot_sync(FULL_MASK, gm != 0);
        if (!pm) continue;
        su[lane] = u;
        sg[lane] = gm;
        __syncwarp();
        const float g0 = subtree<K>(su, sg, 0, pm, mq_l, sv), g1 = subtree<K>(su, sg, 1, pm, mq_l, sv);
        const float g2 = subtree<K>(su, sg, 2, pm, mq_l, sv), g3 = subtree<K>(su, sg, 3, pm, mq_l, sv);
        P = __fadd_rn(P, __fadd_rn(__fadd_rn(g0, g1), __fadd_rn(g2, g3)));
        __syncwarp();
    }
    return P;
}

template <int K, class WC>
__device__ __forceinline__ float dep_span(const Adj &a, uint32_t f, float sv, uint32_t b0, uint32_t b1,
                                          const uint32_t *__restrict__ fnext, const float *__restrict__ mq,
                                          uint32_t *su, uint32_t *sg, WC &wc)
{
    const uint32_t e = b0 + lane_id();
    return dep_span_from<K>(a, f, sv, b0, b1, e < b1 ? a.row[e] : 0u, fnext, mq, su, sg, wc);
}

// delta and q of vertex v for the half's pivots in f
template <int K>
__device__ __forceinline__ void write_lane(float *mdelta, float *mq, uint32_t v, uint32_t f, float delta,
                                          uint32_t sig)
{
    const unsigned lane = lane_id();
    if ((f >> lane) & 1u) {
        mdelta[row_base<K>(v) + lane] = delta;
        mq[row_base<K>(v) + lane] = __fdiv_rn(__fadd_rn(delta, 1.0f), __uint2float_rn(sig));
    }
}

// Backward depth d for the half's pivots in dmask.  With no_succ (the deepest
// depth) nothing lies below, so delta = reach.
template <int K, class WC>
__device__ __forceinline__ void wide_vertices(const Adj &a, uint32_t v_l, uint32_t f_l, int no_succ,
                                             const uint32_t *__restrict__ fnext,
                                             const uint32_t *__restrict__ msigma, float *mdelta,
                                             float *mq, const uint32_t *__restrict__ reach,
                                             uint32_t *su, uint32_t *sg, WC &wc)
{
    const unsigned lane = lane_id();
    unsigned act = __ballot_sync(FULL_MASK, f_l != 0);
    if (!act) return;
    // adjacency bounds and reach of each vertex; per pivot its path count
    // read, its dependency and q written
    if (f_l) {
        wc.add(WC_BYTES, (no_succ ? 4 : 12) + 12 * __popc(f_l));
        wc.add(WC_PAIRS, __popc(f_l));
    }
    // the adjacency bounds of all listed vertices load at once; the first
    // chunk of the next vertex's adjacency loads while a vertex is summed
    uint32_t c0_l = 0, c1_l = 0;
    if (f_l && !no_succ) {
        c0_l = a.col[v_l];
        c1_l = a.col[v_l + 1];
    }
    // vertices of at most 8 neighbours four at a time: their adjacency entries
    // and masks load together, each in a subtree of its own (backward of four
    // scale-20 passes of 64 pivots 6.3 -> 5.7 ms, of three at scale 23 21.6 -> 20.7)
    if (!no_succ) {
        const bool tiny = f_l && c1_l - c0_l <= 8;
        unsigned small = __ballot_sync(FULL_MASK, tiny);
        if (__popc(small) > 1) {
            act &= ~small;
            while (small) {
                int j = 32;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (q == (int)(lane >> 3) && small) j = __ffs(small) - 1;
                    small &= small - 1;
                }
                const uint32_t c0 = __shfl_sync(FULL_MASK, c0_l, j & 31), c1 = __shfl_sync(FULL_MASK, c1_l, j & 31);
                const uint32_t v4 = __shfl_sync(FULL_MASK, v_l, j & 31);
                uint32_t f4 = __shfl_sync(FULL_MASK, f_l, j & 31);
                if (j == 32) f4 = 0;
                const uint32_t e = c0 + (lane & 7);
                const bool in = f4 && e < c1;
                const uint32_t u = in ? a.row[e] : 0u;
                const uint32_t gm = in ? fnext[(uint64_t)u * K] & f4 : 0u;
                if (in) {
                    wc.add(WC_ENTRIES, 1);
                    wc.add(WC_GATHERS, __popc(gm));
                    wc.add(WC_BYTES, 8 + 4 * __popc(gm));
                }
                const unsigned pm = __ballot_sync(FULL_MASK, gm != 0);
                if (pm) {
                    su[lane] = u;
                    sg[lane] = gm;
                    __syncwarp();
                }
#pragma unroll 1
                for (int q = 0; q < 4; q++) {
                    const uint32_t f = __shfl_sync(FULL_MASK, f4, 8 * q);
                    if (!f) break;
                    const uint32_t v = __shfl_sync(FULL_MASK, v4, 8 * q);
                    const uint32_t sig = ((f >> lane) & 1u) ? msigma[row_base<K>(v) + lane] : 0u;
                    const float P = subtree<K>(su, sg, q, pm, mq + lane, __uint2float_rn(sig));
                    write_lane<K>(mdelta, mq, v, f, __fadd_rn(__uint2float_rn(reach[v]), P), sig);
                }
                __syncwarp();
            }
            if (!act) return;
        }
    }
    int j = __ffs(act) - 1;
    uint32_t b0 = __shfl_sync(FULL_MASK, c0_l, j), b1 = __shfl_sync(FULL_MASK, c1_l, j);
    uint32_t un = b0 + lane < b1 ? a.row[b0 + lane] : 0u;
    for (;;) {
        act &= act - 1;
        const uint32_t v = __shfl_sync(FULL_MASK, v_l, j);
        const uint32_t f = __shfl_sync(FULL_MASK, f_l, j);
        const uint32_t cb0 = b0, cb1 = b1, cu = un;
        const int jn = act ? __ffs(act) - 1 : -1;
        if (jn >= 0) {
            b0 = __shfl_sync(FULL_MASK, c0_l, jn);
            b1 = __shfl_sync(FULL_MASK, c1_l, jn);
            un = b0 + lane < b1 ? a.row[b0 + lane] : 0u;
        }
        const uint32_t sig = ((f >> lane) & 1u) ? msigma[row_base<K>(v) + lane] : 0u;
        float P = 0.0f;
        if (!no_succ) P = dep_span_from<K>(a, f, __uint2float_rn(sig), cb0, cb1, cu, fnext, mq, su, sg, wc);
        write_lane<K>(mdelta, mq, v, f, __fadd_rn(__uint2float_rn(reach[v]), P), sig);
        if (jn < 0) break;
        j = jn;
    }
}

// The same depth on a graph large enough to keep every warp busy: lane =
// pivot (4-byte loads of a successor's row), a warp takes a span of a heavy vertex
// (its span sums are combined by k_bwd_combine_step) or a group of about one span
// of the others.  At full occupancy (32 registers) this form does more per second
// than the tiles; see bwd_wide() for the line between them.
template <int K, class WC>
__device__ __forceinline__ void bwd_body_wide(const Adj &a, uint32_t dmask, int no_succ,
                                         const uint32_t *__restrict__ fd, const uint32_t *__restrict__ fnext,
                                         const uint32_t *__restrict__ msigma, float *mdelta,
                                         float *mq, float *mpartial,
                                         const uint32_t *__restrict__ reach, uint32_t *ctr,
                                         uint32_t *su, uint32_t *sg, const uint32_t *lst,
                                         uint32_t lcnt, uint32_t lheavy, WC &wc)
{
    const unsigned lane = lane_id();
    // heavy span items only when a heavy vertex is at this depth
    const uint64_t nhi = lst && lheavy == 0 ? 0 : a.n_heavy_items;
    const uint32_t ent = list_unit(lcnt);
    const uint64_t nu = nhi + (lst ? (lcnt + ent - 1) / ent : a.n_ltask);
    if (warp_global() >= nu) return;  // fewer units than warps: no contention
    for (;;) {
        const uint32_t t = grab_unit(ctr);
        if (t >= nu) break;
        if (t < nhi) {
            const uint32_t v = a.hitem_v[t];
            const uint32_t f = fd[(uint64_t)v * K] & dmask;
            if (lane == 0) wc.add(WC_BYTES, 4);  // level mask word
            if (!f) continue;
            float P = 0.0f;
            if (!no_succ) {
                const float sv =
                    __uint2float_rn(((f >> lane) & 1u) ? msigma[row_base<K>(v) + lane] : 0u);
                const uint32_t b0 = a.col[v] + a.hitem_k[t] * AXBC_SPAN;
                P = dep_span<K>(a, f, sv, b0, min(a.col[v + 1], b0 + AXBC_SPAN), fnext, mq, su, sg, wc);
            }
            mpartial[(uint64_t)t * (AXBC_W * K) + lane] = P;
            if ((f >> lane) & 1u) wc.add(WC_BYTES, 8);  // path count read, span partial written
            continue;
        }
        if (lst) {
            const uint32_t i = (uint32_t)(t - nhi) * ent + lane;
            uint32_t v_l = 0, f_l = 0;
            if (lane < ent && i < lcnt) {
                v_l = lst[i];
                if (a.col[v_l + 1] - a.col[v_l] <= AXBC_SPAN) f_l = fd[(uint64_t)v_l * K] & dmask;
                wc.add(WC_BYTES, 8);  // list entry, level mask word
            }
            wide_vertices<K>(a, v_l, f_l, no_succ, fnext, msigma, mdelta, mq, reach, su, sg, wc);
            continue;
        }
        const uint32_t beg = a.ltask[t - nhi], cnt = a.ltask[t - nhi + 1] - beg;
        uint32_t v_l = 0, f_l = 0;
        if (lane < cnt) {
            v_l = a.order[beg + lane];
            f_l = fd[(uint64_t)v_l * K] & dmask;
            wc.add(WC_BYTES, 4);  // level mask word
        }
        wide_vertices<K>(a, v_l, f_l, no_succ, fnext, msigma, mdelta, mq, reach, su, sg, wc);
    }
}

template <int K>
__device__ __forceinline__ void combine_body(const Adj &a, uint32_t dmask, const uint32_t *__restrict__ fd,
                                             const uint32_t *__restrict__ msigma, float *mdelta,
                                             float *mq, const float *__restrict__ mpartial,
                                             const uint32_t *__restrict__ reach)
{
    const unsigned lane = lane_id();
    const uint64_t nw = (uint64_t)gridDim.x * blockDim.x / 32;
    for (uint64_t i = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32; i < a.n_heavy; i += nw) {
        const uint32_t v = a.heavy_v[i];
        const uint32_t f = fd[(uint64_t)v * K] & dmask;
        if (!f) continue;
        float acc = __uint2float_rn(reach[v]);
        for (uint32_t k = a.heavy_first[i]; k < a.heavy_first[i + 1]; k++)
            acc = __fadd_rn(acc, mpartial[(uint64_t)k * (AXBC_W * K) + lane]);
        const uint32_t sig = ((f >> lane) & 1u) ? msigma[row_base<K>(v) + lane] : 0u;
        write_lane<K>(mdelta, mq, v, f, acc, sig);
    }
}

template <int K>
__device__ __forceinline__ BwdHalf bwd_half(const BatchInfo *bi, uint32_t *const *tab, int d, int hh,
                                            const uint32_t *msigma, float *mdelta, float *mq, float *mpartial,
                                            uint32_t *harrive, uint32_t n_heavy, const uint32_t *reach)
{
    typedef typename MaskOf<K>::T M;
    return BwdHalf{half_of<K>((M)(d >= 1 ? bi->srcmask : bi->depth0mask), hh), d == bi->dmax, tab[d] + hh,
                   tab[d + 1] + hh, msigma + 32 * hh, mdelta + 32 * hh, mq + 32 * hh, mpartial + 32 * hh,
                   harrive + (uint64_t)n_heavy * hh, reach};
}

// Backward depth d.  The grid's y index is the half: the blocks of half 1 of a
// 64-pivot pass start as those of half 0 run out of work, each half with its
// own work counter.  CNT: the counting build (work counts into wc[KP_BWD]).
template <int K, bool CNT>
__global__ void __launch_bounds__(BATCH_TPB, AXBC_BWD_TILE_BLOCKS) k_bwd_tile_step(Adj a, const BatchInfo *__restrict__ bi,
                                                        uint32_t *const *__restrict__ tab,
                                                        const uint32_t *__restrict__ msigma,
                                                        float *mdelta, float *mq, float *mpartial, uint32_t *harrive,
                                                        const uint32_t *__restrict__ reach,
                                                        uint32_t *ctrs, LevelLists ll, int d, int symmetric,
                                                        unsigned long long *wc)
{
    __shared__ uint2 s_st[BATCH_TPB / 32][36];
    __shared__ float s_csum[2][BWD_TILE_CHUNKS][32];
    const int hh = K == 1 ? 0 : blockIdx.y;
    const BwdHalf B = bwd_half<K>(bi, tab, d, hh, msigma, mdelta, mq, mpartial, harrive, a.n_heavy, reach);
    if (!B.dmask) return;
    uint32_t lcnt = 0;
    const uint32_t *lst = level_list(ll, d, lcnt);
    WorkCount<CNT> cnt;
    bwd_body<K>(a, B, ctrs + 2 * AXBC_MAX_LEVELS * hh + 2 * d + 1, s_st[threadIdx.x >> 5], s_csum, lst, lcnt,
                ll.heavy[d], symmetric, cnt);
    cnt.flush(wc);
}

template <int K, bool CNT>
__global__ void __launch_bounds__(BATCH_TPB, AXBC_BWD_MIN_BLOCKS) k_bwd_step(Adj a, const BatchInfo *__restrict__ bi,
                                                        uint32_t *const *__restrict__ tab,
                                                        const uint32_t *__restrict__ msigma,
                                                        float *mdelta, float *mq, float *mpartial,
                                                        const uint32_t *__restrict__ reach,
                                                        uint32_t *ctrs, LevelLists ll, int d,
                                                        unsigned long long *wc)
{
    typedef typename MaskOf<K>::T M;
    __shared__ __align__(16) uint32_t s_u[BATCH_TPB];
    __shared__ __align__(16) uint32_t s_g[BATCH_TPB];
    const int hh = K == 1 ? 0 : blockIdx.y;
    const uint32_t dmask = half_of<K>((M)(d >= 1 ? bi->srcmask : bi->depth0mask), hh);
    if (!dmask) return;
    uint32_t *su = s_u + (threadIdx.x & ~31u), *sg = s_g + (threadIdx.x & ~31u);
    uint32_t lcnt = 0;
    const uint32_t *lst = level_list(ll, d, lcnt);
    WorkCount<CNT> cnt;
    bwd_body_wide<K>(a, dmask, d == bi->dmax, tab[d] + hh, tab[d + 1] + hh, msigma + 32 * hh, mdelta + 32 * hh,
                     mq + 32 * hh, mpartial + 32 * hh, reach, ctrs + 2 * AXBC_MAX_LEVELS * hh + 2 * d + 1, su, sg, lst,
                     lcnt, ll.heavy[d], cnt);
    cnt.flush(wc);
}

template <int K>
__global__ void k_bwd_combine_step(Adj a, const BatchInfo *__restrict__ bi, uint32_t *const *__restrict__ tab,
                                   const uint32_t *__restrict__ msigma, float *mdelta, float *mq,
                                   const float *__restrict__ mpartial, const uint32_t *__restrict__ reach,
                                   LevelLists ll, int d)
{
    typedef typename MaskOf<K>::T M;
    uint32_t lcnt;
    if (level_list(ll, d, lcnt) && ll.heavy[d] == 0) return;  // no heavy vertex at this depth
    const int hh = K == 1 ? 0 : blockIdx.y;
    const uint32_t dmask = half_of<K>((M)(d >= 1 ? bi->srcmask : bi->depth0mask), hh);
    if (!dmask) return;
    combine_body<K>(a, dmask, tab[d] + hh, msigma + 32 * hh, mdelta + 32 * hh, mq + 32 * hh, mpartial + 32 * hh,
                    reach);
}

// ------------------------------------------------ persistent level loop
// On small graphs and in narrow passes over deep ones a level's work is a few
// microseconds and the two launches per forward level and one or two per
// backward depth dominate.  k_traverse_persist runs a whole batch -- every
// forward level, then every backward depth -- in one cooperative launch whose
// blocks are all resident, with the step kernels' device bodies separated by a
// grid barrier: two barriers per forward level (expansion | statistics and
// level close) and one per backward depth.

template <int K> struct AdvanceLead {
    BatchInfo *bi;
    unsigned long long *level_te, *level_cnt;
    int32_t *level_mode;
    LevelLists ll;
    uint32_t pool_cap, list_max;
    __device__ void operator()() const
    {
        level_advance_warp<K>(bi, level_te, level_cnt, level_mode, ll, pool_cap, list_max);
    }
};

// The arrays the loop writes are passed without const/__restrict__, so that
// no load of them goes through the read-only cache: they change between
// phases of the one launch.  Levels stop at lmax (the masks allocated): the
// kernel sets gs->need and the host grows the tables and launches again, the
// loop resuming from the level state in bi.
template <int K>
__global__ void __launch_bounds__(BATCH_TPB, PERSIST_BLOCKS) k_traverse_persist(
    Adj a, Adj rv, BatchInfo *bi, uint32_t **tab, uint32_t *seen_, uint32_t *msigma, float *mdelta,
    float *mq, float *mpartial, uint32_t *harrive, const uint32_t *reach, uint32_t *ctrs, LevelLists ll,
    int symmetric, unsigned long long *level_te, unsigned long long *level_cnt, int32_t *level_mode,
    uint32_t pool_cap, uint32_t list_max, uint64_t n, int lmax, GridSync *gs, long long budget)
{
    typedef typename MaskOf<K>::T M;
    __shared__ uint2 s_st[BATCH_TPB / 32][PullShape<K>::STAGE];
    __shared__ float s_csum[2][BWD_TILE_CHUNKS][32];
    __shared__ StatsShared<K> sh;
    uint2 *st = s_st[threadIdx.x >> 5];
    M *seen = reinterpret_cast<M *>(seen_);
    WorkCount<false> none;
    unsigned epoch = 0;
    const AdvanceLead<K> adv{bi, level_te, level_cnt, level_mode, ll, pool_cap, list_max};
    const M srcmask = (M)bi->srcmask;
    // the level counts along in every block: its state, masks and list load at once
    for (int L = vload_i(&bi->cur) + 1;; L++) {
        const int push = vload_i(&bi->push_next);
        if (!vload_i(&bi->alive)) break;
        if (L >= lmax) {
            if (blockIdx.x == 0 && threadIdx.x == 0) gs->need = 1;
            return;
        }
        M *fprev = reinterpret_cast<M *>(tab[L - 1]), *fcur = reinterpret_cast<M *>(tab[L]);
        if (push)
            fwd_push_body<K>(a, fprev, fcur, seen, msigma, ctrs + 2 * L, ll, L, reinterpret_cast<uint32_t *>(st), none);
        else
            fwd_pull_body<K>(rv, srcmask, fprev, fcur, seen, msigma, ctrs + 2 * L, st, ll, L, none);
        if (!grid_barrier(gs, budget, 1, epoch, NoLead{})) return;
        stats_body<K>(n, bi, L, srcmask, fcur, seen, a.col, rv.col, reach, a.big, sh, ll);
        if (!grid_barrier(gs, budget, 2, epoch, adv)) return;
    }
    const uint32_t n_heavy = a.n_heavy;
    for (int d = vload_i(&bi->dmax); d >= 0; d--) {
        if (!(d >= 1 ? bi->srcmask : bi->depth0mask)) break;
        uint32_t lcnt = 0;
        const uint32_t *lst = level_list(ll, d, lcnt);
        const uint32_t lheavy = ll.heavy[d];
        // the halves touch disjoint columns and have their own work counters:
        // one phase takes both
#pragma unroll 1
        for (int hh = 0; hh < K; hh++) {
            const BwdHalf B = bwd_half<K>(bi, tab, d, hh, msigma, mdelta, mq, mpartial, harrive, n_heavy, reach);
            if (B.dmask)
                bwd_body<K>(a, B, ctrs + 2 * AXBC_MAX_LEVELS * hh + 2 * d + 1, st, s_csum, lst, lcnt, lheavy,
                            symmetric, none);
            __syncthreads();  // the chunk sums of the next half
        }
        if (d > 0 && !grid_barrier(gs, budget, 3, epoch, NoLead{})) return;
    }
}

// Self-test of the grid barrier: `rounds` barriers, the leader of each adding
// one to out[0]; block `absent` (if >= 0) never arrives, so the first wait runs
// out of its budget and every block returns.
struct CountLead {
    unsigned *out;
    __device__ void operator()() const
    {
        if (lane_id() == 0) out[0]++;
    }
};
__global__ void __launch_bounds__(BATCH_TPB) k_barrier_selftest(GridSync *gs, int rounds, long long budget,
                                                                int absent, unsigned *out)
{
    if ((int)blockIdx.x == absent) return;
    const CountLead lead{out};
    unsigned epoch = 0;
    for (int r = 0; r < rounds; r++)
        if (!grid_barrier(gs, budget, r + 1, epoch, lead)) return;
}

// bc update for the applied pivots in lane order (update_bc, src/cuda_kernels.cu:
// 269-286), each into its lane's bc vector.  A pivot that did not reach v
// contributes delta = reach[v].  Zero terms are skipped: x + float(0/p) == x for
// p > 0.  One thread per vertex, its 32 K dependencies read from rows a warp
// staged in shared memory.
// 4-byte global -> shared copies that bypass registers (cp.async), so a warp
// keeps up to 32 row loads of one chunk and the next chunk's in flight
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// stage the dependency rows of the chunk's vertices reached by pivots of half
// hh (sv: their masks for that half): lane l copies column 32 hh + l
template <int K>
__device__ __forceinline__ void stage_half(float (*rows)[AXBC_W + 1], const float *__restrict__ mdelta,
                                           uint64_t base, uint32_t sv, int hh)
{
    const unsigned lane = lane_id();
    unsigned need = __ballot_sync(FULL_MASK, sv != 0);
    while (need) {
        const int r = __ffs(need) - 1;
        need &= need - 1;
        cp_async4(&rows[r][lane], mdelta + row_base<K>(base + r) + 32 * hh + lane);
    }
    cp_async_commit();
}

// threads of the update (34 KB of staged rows)
#define UPD_TPB(K) 128
template <int K>
__global__ void __launch_bounds__(UPD_TPB(K)) k_update_m(const float *__restrict__ mdelta,
                                                         const uint32_t *__restrict__ seen_,
                                                         const uint32_t *__restrict__ reach, uint64_t n,
                                                         const BatchInfo *__restrict__ bi,
                                                         float *__restrict__ delta_out,
                                                         const uint32_t *__restrict__ from_view)
{
    typedef typename MaskOf<K>::T M;
    constexpr int NS = AXBC_W * K;  // pivot slots
    constexpr int TPB = UPD_TPB(K);
    const M *seen = reinterpret_cast<const M *>(seen_);
    __shared__ uint32_t s_root[NS], s_reach[NS], s_skip0[NS];
    __shared__ double s_p[NS];
    __shared__ unsigned long long s_nvt[NS];
    __shared__ InvSplit s_iv[NS];
    __shared__ float *s_bc[NS];
    // per lane: float(reach_v0 + 1), the split 1/p, and whether the fast
    // division applies (bit 0) and zero terms may be skipped (bit 1)
    __shared__ float4 s_k[NS];
    __shared__ int s_single;  // every applied lane updates the same vector
    __shared__ int s_allpos;  // every applied lane has p > 0 (zero terms vanish)
    // per warp, two staged units: the dependency rows of 32 vertices for one
    // 32-pivot half, padded to 33 floats so that thread t reading row t,
    // column s hits bank (t + s) mod 32
    __shared__ float s_rows[TPB / 32][2][32][AXBC_W + 1];
    const M amask = (M)(bi->applymask & bi->srcmask);
    for (int s = threadIdx.x; s < NS; s += TPB) {
        s_bc[s] = bi->lane_bc[s];
        if ((amask >> s) & 1u) {
            const uint32_t r = bi->root[s];
            const uint32_t rv = reach[r];
            const uint32_t all = (bi->H == 1 ? (uint32_t)bi->rsum[s] : 0u) + rv;
            s_root[s] = r;
            s_reach[s] = rv;
            s_p[s] = bi->p[s];
            s_skip0[s] = bi->p[s] > 0.0;
            s_nvt[s] = bi->nvis[s] + all;
            s_iv[s] = inv_split(bi->p[s]);
        } else {
            s_root[s] = 0xffffffffu;
            s_reach[s] = 0;
            s_p[s] = 1.0;
            s_skip0[s] = 1;
            s_nvt[s] = 2;
            s_iv[s] = inv_split(1.0);
        }
        const InvSplit iv = s_iv[s];
        s_k[s] = make_float4(__uint2float_rn(s_reach[s] + 1u), iv.hi, iv.lo,
                             __uint_as_float((iv.ok ? 1u : 0u) | (s_skip0[s] ? 2u : 0u)));
        if (s == 0) {
            int single = 1, allpos = 1;
            float *t0 = nullptr;
            for (int l = 0; l < NS; l++)
                if ((amask >> l) & 1u) {
                    if (!t0) t0 = bi->lane_bc[l];
                    else if (bi->lane_bc[l] != t0) single = 0;
                    if (!(bi->p[l] > 0.0)) allpos = 0;
                }
            s_single = single;
            s_allpos = allpos;
        }
    }
    __syncthreads();
    if (amask == 0) return;
    const bool single = s_single != 0;
    // a vertex no pivot reached, with reach 0, gets only zero terms: skipped
    // when they vanish (p > 0; 0/0 is NaN, as in the reference)
    const bool skip_unreached = s_allpos != 0;
    const int slast = 63 - __clzll((unsigned long long)amask);
    // delta_out (when given): the last applied pivot's dependencies, taken
    // from the staged rows (k_extract_delta's rule)
    const uint32_t dl_root = bi->root[slast];
    const bool dl_root_done = (bi->depth0mask >> slast) & 1u;
    const unsigned lane = lane_id();
    const unsigned wid = threadIdx.x >> 5;
    const uint64_t stride = (uint64_t)gridDim.x * (TPB / 32) * 32;
    uint64_t base = (blockIdx.x * (uint64_t)(TPB / 32) + wid) * 32;
    if (base >= n) return;
    M sv = 0;
    uint32_t rv = 0;
    if (base + lane < n) {
        sv = seen[base + lane];
        rv = reach[base + lane];
    }
    // units of (chunk of 32 vertices, 32-pivot half), in order; each vertex
    // sums its slots in slot order across the halves of its chunk
    stage_half<K>(s_rows[wid][0], mdelta, base, (uint32_t)sv, 0);
    int buf = 0;
    for (; base < n; base += stride) {
        const uint64_t next = base + stride;
        M svn = 0;
        uint32_t rvn = 0;
        if (next + lane < n) {
            svn = seen[next + lane];
            rvn = reach[next + lane];
        }
        const uint64_t v = base + lane;
        // v numbers the graph's view; the bc vectors and delta_out are indexed
        // by vertex id
        const uint64_t vo = from_view && v < n ? from_view[v] : v;
        const float rf = __uint2float_rn(rv);
        // unreached by every pivot with delta 0: only a root term could apply,
        // and roots are reached
        const bool work = v < n && (sv != 0 || rv != 0u || !skip_unreached);
        // one target vector, reach 0, every p > 0: a pivot that did not reach
        // v adds +0, so only the reached lanes are visited
        const bool sparse = work && single && rv == 0u && skip_unreached;
        float *tgt = nullptr;
        float b = 0.0f;
        if (work && single) {
            tgt = s_bc[slast];
            b = tgt[vo];
        }
#pragma unroll 1
        for (int hh = 0; hh < K; hh++, buf ^= 1) {
            // the next unit's rows load while this one is summed
            if (hh + 1 < K) {
                stage_half<K>(s_rows[wid][buf ^ 1], mdelta, base, (uint32_t)((unsigned long long)sv >> 32), 1);
                cp_async_wait<1>();
            } else if (next < n) {
                stage_half<K>(s_rows[wid][buf ^ 1], mdelta, next, (uint32_t)svn, 0);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncwarp();
            const float(*rows)[AXBC_W + 1] = s_rows[wid][buf];
            const uint32_t svh = (uint32_t)((unsigned long long)sv >> (32 * hh));
            const uint32_t amh = (uint32_t)((unsigned long long)amask >> (32 * hh));
            const int s0 = 32 * hh;
            if (delta_out && v < n && (slast >> 5) == hh) {
                const bool have = v == dl_root ? dl_root_done : ((svh >> (slast & 31)) & 1u) != 0u;
                delta_out[vo] = have ? rows[lane][slast & 31] : rf;
            }
            if (sparse) {
                for (uint32_t bits = svh & amh; bits; bits &= bits - 1) {
                    const int j = __ffs(bits) - 1, s = s0 + j;
                    if ((uint32_t)v == s_root[s]) {
                        if (s_reach[s] > 0) b = __fadd_rn(b, bc_root_term(s_reach[s], s_nvt[s]));
                        continue;
                    }
                    const float dv = rows[lane][j];
                    if (dv == 0.0f) continue;
                    const float4 k = s_k[s];
                    const uint32_t fl = __float_as_uint(k.w);
                    b = __fadd_rn(b, div_to_float_hl(__fmul_rn(dv, k.x), s_p[s], k.y, k.z, (fl & 1u) != 0u));
                }
            } else if (work && single) {
                // one target vector: every slot in order
#pragma unroll
                for (int j = 0; j < AXBC_W; j++) {
                    if (!((amh >> j) & 1u)) continue;
                    const int s = s0 + j;
                    if ((uint32_t)v == s_root[s]) {
                        if (s_reach[s] > 0) b = __fadd_rn(b, bc_root_term(s_reach[s], s_nvt[s]));
                        continue;
                    }
                    const float dv = ((svh >> j) & 1u) ? rows[lane][j] : rf;
                    const float4 k = s_k[s];
                    const uint32_t fl = __float_as_uint(k.w);
                    if (dv == 0.0f && (fl & 2u)) continue;
                    b = __fadd_rn(b, div_to_float_hl(__fmul_rn(dv, k.x), s_p[s], k.y, k.z, (fl & 1u) != 0u));
                }
            } else if (work) {
                // lanes in order; consecutive lanes of one run add into one
                // register, written back when the target vector changes
                for (int j = 0; j < AXBC_W && s0 + j <= slast; j++) {
                    if (!((amh >> j) & 1u)) continue;
                    const int s = s0 + j;
                    if (s_bc[s] != tgt) {
                        if (tgt) tgt[vo] = b;
                        tgt = s_bc[s];
                        b = tgt[vo];
                    }
                    if ((uint32_t)v == s_root[s]) {
                        if (s_reach[s] > 0) b = __fadd_rn(b, bc_root_term(s_reach[s], s_nvt[s]));
                        continue;
                    }
                    const float dv = ((svh >> j) & 1u) ? rows[lane][j] : rf;
                    if (dv == 0.0f && s_skip0[s]) continue;
                    b = __fadd_rn(b, bc_term_fast(dv, s_reach[s], s_p[s], s_iv[s]));
                }
            }
            __syncwarp();
        }
        if (tgt) tgt[vo] = b;
        sv = svn;
        rv = rvn;
    }
}

// the last applied pivot's dependencies as a plain n-vector
template <int K>
__global__ void k_extract_delta(float *out, const float *__restrict__ mdelta,
                                const uint32_t *__restrict__ seen_,
                                const uint32_t *__restrict__ reach, uint64_t n,
                                const BatchInfo *__restrict__ bi, int lane_lo, int lane_hi,
                                const uint32_t *__restrict__ from_view)
{
    typedef typename MaskOf<K>::T M;
    const M *seen = reinterpret_cast<const M *>(seen_);
    // the highest applied lane of [lane_lo, lane_hi)
    unsigned long long range = lane_hi >= 64 ? ~0ull : ((1ull << lane_hi) - 1ull);
    range &= ~((1ull << lane_lo) - 1ull);
    const unsigned long long am = bi->applymask & bi->srcmask & range;
    if (am == 0) return;
    const int s = 63 - __clzll(am);
    const uint32_t root = bi->root[s];
    const bool root_done = (bi->depth0mask >> s) & 1ull;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
         v += (uint64_t)gridDim.x * blockDim.x) {
        bool have = ((unsigned long long)seen[v] >> s) & 1ull;
        if (v == root) have = root_done;
        out[from_view ? from_view[v] : v] = have ? mdelta[row_base<K>(v) + s] : __uint2float_rn(reach[v]);
    }
}

// one pivot of the last batch: path counts, depths, dependencies
template <int K>
__global__ void k_source_view(int s, int levels, uint32_t *const *fm, const uint32_t *__restrict__ seen_,
                              const uint32_t *__restrict__ msigma, const float *__restrict__ mdelta,
                              const uint32_t *__restrict__ reach, uint64_t n, unsigned long long depth0,
                              uint32_t *sig, int32_t *lvl, float *dl, const uint32_t *__restrict__ from_view)
{
    typedef typename MaskOf<K>::T M;
    const M *seen = reinterpret_cast<const M *>(seen_);
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
         v += (uint64_t)gridDim.x * blockDim.x) {
        int L = -1;
        if (((unsigned long long)seen[v] >> s) & 1ull) {
            for (int l = 0; l < levels; l++)
                if (((unsigned long long)reinterpret_cast<const M *>(fm[l])[v] >> s) & 1ull) {
                    L = l;
                    break;
                }
        }
        // v numbers the graph's view; the outputs are indexed by vertex id
        const uint64_t vo = from_view ? from_view[v] : v;
        lvl[vo] = L;
        sig[vo] = L >= 0 ? msigma[row_base<K>(v) + s] : 0u;
        bool have = L > 0 || (L == 0 && ((depth0 >> s) & 1ull));
        dl[vo] = have ? mdelta[row_base<K>(v) + s] : __uint2float_rn(reach[v]);
    }
}

// ------------------------------------------------------------------ host
static int ensure_level_tables(axbc_ctx *c)
{
    if (c->tables_ready) return AXBC_OK;
    ALLOC_MISSING(c->fmtab, AXBC_MAX_LEVELS * sizeof(uint32_t *), &c->bytes);
    // work counters, list lengths: zero here, then cleared by each pass as far
    // as the one before it went
    if (!c->ctrs) {
        TRY(axbc_dalloc((void **)&c->ctrs, 2 * AXBC_WMAX / 32 * AXBC_MAX_LEVELS * 4, &c->bytes));
        CU(cudaMemsetAsync(c->ctrs, 0, 2 * AXBC_WMAX / 32 * AXBC_MAX_LEVELS * 4, c->stream));
    }
    ALLOC_MISSING(c->d_level_te, AXBC_MAX_LEVELS * 8, &c->bytes);
    ALLOC_MISSING(c->d_level_cnt, AXBC_MAX_LEVELS * 8, &c->bytes);
    ALLOC_MISSING(c->d_level_mode, AXBC_MAX_LEVELS * 4, &c->bytes);
    // level lists: a vertex joins a level's list once per distinct depth at
    // which the batch's pivots reach it (at most 64 n entries); the pool
    // starts at 32 n and grows when a batch runs short; a level may hold up to
    // n/8 vertices before it falls back to the task scan
    if (!c->lpool) {
        const uint32_t cap = (uint32_t)std::min<uint64_t>((uint64_t)AXBC_W * c->g->n + 64, 0xffffffffull);
        TRY(axbc_dalloc((void **)&c->lpool, (uint64_t)cap * 4, &c->bytes));
        c->lpool_cap = cap;
    }
    ALLOC_MISSING(c->lstart, AXBC_MAX_LEVELS * 4, &c->bytes);
    if (!c->lcount) {
        TRY(axbc_dalloc((void **)&c->lcount, AXBC_MAX_LEVELS * 4, &c->bytes));
        CU(cudaMemsetAsync(c->lcount, 0, AXBC_MAX_LEVELS * 4, c->stream));
    }
    ALLOC_MISSING(c->lcap, AXBC_MAX_LEVELS * 4, &c->bytes);
    if (!c->lheavy) {
        TRY(axbc_dalloc((void **)&c->lheavy, AXBC_MAX_LEVELS * 4, &c->bytes));
        CU(cudaMemsetAsync(c->lheavy, 0, AXBC_MAX_LEVELS * 4, c->stream));
    }
    c->tables_ready = true;
    return AXBC_OK;
}

static LevelLists lists_of(const axbc_ctx *c)
{
    return LevelLists{c->lpool, c->lstart, c->lcount, c->lcap, c->lheavy};
}

// Largest stored level list: n/8 vertices, or n/2 when no vertex has more than
// 64 neighbours (a list unit then carries little work whatever it holds, and a
// wide level of a high-diameter graph is still cheaper to walk than to scan).
static uint32_t list_max_of(const axbc_ctx *c)
{
    const uint64_t n = c->g->n;
    return (uint32_t)std::max<uint64_t>(64, c->g->max_deg <= 64 ? n / 2 : n / 8);
}

// Level masks 0..levels-1 exist (two words per vertex, enough for either
// width), and their pointers are in the device table.  Every mask array is
// all zero between batches.
int axbc_batch_levels_alloc(axbc_ctx *c, int levels)
{
    TRY(ensure_level_tables(c));
    if (levels > AXBC_MAX_LEVELS) {
        axbc_set_error("traversal deeper than %d levels", AXBC_MAX_LEVELS - 2);
        return AXBC_ERR_RANGE;
    }
    // masks allocated by an earlier, partly failed call reach the device table
    // here too: fmtab_synced counts the entries copied so far
    int rc = AXBC_OK;
    while ((int)c->fmask.size() < levels) {
        uint32_t *p = nullptr;
        if ((rc = axbc_dalloc((void **)&p, c->g->n * 8, &c->bytes)) != AXBC_OK) break;
        c->fmask.push_back(p);
        CU(cudaMemsetAsync(p, 0, c->g->n * 8, c->stream));
    }
    if (c->fmask.size() > c->fmtab_synced) {
        CU(cudaMemcpy(c->fmtab + c->fmtab_synced, c->fmask.data() + c->fmtab_synced,
                      (c->fmask.size() - c->fmtab_synced) * sizeof(uint32_t *), cudaMemcpyHostToDevice));
        c->fmtab_synced = c->fmask.size();
    }
    return rc;
}

// per-pivot rows of 64 values, masks of two words: a pass of either width
int axbc_ensure_batch(axbc_ctx *c)
{
    if (c->batch_ready) return AXBC_OK;
    const uint64_t n = c->g->n;
    ALLOC_MISSING(c->seen, n * 8, &c->bytes);
    ALLOC_MISSING(c->msigma, n * AXBC_WMAX * 4, &c->bytes);
    ALLOC_MISSING(c->mdelta, n * AXBC_WMAX * 4, &c->bytes);
    ALLOC_MISSING(c->mq, n * AXBC_WMAX * 4, &c->bytes);
    ALLOC_MISSING(c->mpartial, (c->g->bfwd.n_heavy_items + 1) * AXBC_WMAX * 4, &c->bytes);
    if (!c->harrive) {
        TRY(axbc_dalloc((void **)&c->harrive, (uint64_t)(c->g->bfwd.n_heavy + 1) * 2 * 4, &c->bytes));
        CU(cudaMemsetAsync(c->harrive, 0, (uint64_t)(c->g->bfwd.n_heavy + 1) * 2 * 4, c->stream));
    }
    ALLOC_MISSING(c->bi, sizeof(BatchInfo), &c->bytes);
    if (!c->bi_host) CU(cudaMallocHost((void **)&c->bi_host, sizeof(BatchInfo)));
    CU(cudaMemsetAsync(c->bi, 0, sizeof(BatchInfo), c->stream));
    CU(cudaMemsetAsync(c->seen, 0, n * 8, c->stream));
    TRY(axbc_batch_levels_alloc(c, 10));
    c->batch_ready = true;
    return AXBC_OK;
}

// mask words per vertex for a pass of nsrc pivots
static int width_k(int nsrc) { return nsrc > AXBC_W ? 2 : 1; }

// Backward by warps (true) or with the big vertices in block tiles: tiles while
// the pass's adjacency work is too small to keep every warp busy.  Measured
// (us a pass of 32 / 64 pivots, warps against tiles): 0.43 M adjacency entries
// 382 : 123 and 429 : 157, 1.8 M 334 : 196 and 372 : 339, 3.7 M 377 : 246 and
// 451 : 469, 7.6 M 417 : 432 and 694 : 866, 31 M (64 pivots) 1590 : 2590.
static bool bwd_wide(const axbc_graph *g, int K) { return g->m * (uint64_t)K >= AXBC_BWD_WIDE_MIN; }

// dynamic kernels: as many blocks as stay resident (work comes from counters),
// or as many as have work
template <int K> static int occupancy(axbc_ctx *c)
{
    const int i = K - 1;
    if (!c->fwd_blocks_per_sm[i]) {
        int a = 0, b = 0;
        CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_fwd_step<K, false>, BATCH_TPB, 0));
        CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &b, bwd_wide(c->g, K) ? (const void *)k_bwd_step<K, false> : (const void *)k_bwd_tile_step<K, false>,
            BATCH_TPB, 0));
        c->bwd_blocks_per_sm[i] = std::max(1, b);
        c->fwd_blocks_per_sm[i] = std::max(1, a);
    }
    return AXBC_OK;
}
static int grid_of(const axbc_ctx *c, int per_sm, uint64_t blocks)
{
    return (int)std::max<uint64_t>(1, std::min<uint64_t>(axbc_grid_for(c, BATCH_TPB, per_sm), blocks));
}
// warps that could each have a unit of their own
static uint64_t adj_warps(const Adj &a) { return a.n_part + (a.n_linked - a.n_big); }
template <int K> static int fwd_grid(const axbc_ctx *c)
{
    const uint64_t w = std::max(adj_warps(c->g->bfwd), adj_warps(c->g->brev));
    return grid_of(c, c->fwd_blocks_per_sm[K - 1], (w + 7) / 8);
}
template <int K> static int bwd_grid(const axbc_ctx *c)
{
    const Adj &a = c->g->bfwd;
    return grid_of(c, c->bwd_blocks_per_sm[K - 1],
                   std::max<uint64_t>(std::max<uint64_t>(a.n_tile, a.n_heavy_items), (c->g->n - a.n_big + 7) / 8));
}

// the kernels of one forward level, in stream order; one backward depth
template <int K> static void stats_step_kernel(axbc_ctx *c)
{
    axbc_graph *g = c->g;
    k_stats_step<K><<<grid_of(c, 4, (g->n + BATCH_TPB - 1) / BATCH_TPB), BATCH_TPB, 0, c->stream>>>(
        g->n, c->bi, c->fmtab, c->seen, g->bfwd.col, g->brev.col, g->breach, lists_of(c), c->d_level_te,
        c->d_level_cnt, c->d_level_mode, c->lpool_cap, list_max_of(c), g->bfwd.big);
}
template <int K> static void fwd_step_kernel(axbc_ctx *c, unsigned long long *wc)
{
    axbc_graph *g = c->g;
    (wc ? k_fwd_step<K, true> : k_fwd_step<K, false>)<<<fwd_grid<K>(c), BATCH_TPB, 0, c->stream>>>(
        g->bfwd, g->brev, c->bi, c->fmtab, c->seen, c->msigma, c->ctrs, lists_of(c), wc);
}

template <int K> static void bwd_step_kernel(axbc_ctx *c, int d, unsigned long long *wc)
{
    axbc_graph *g = c->g;
    const dim3 grid(bwd_grid<K>(c), K);
    cudaStream_t s = c->stream;
    if (!bwd_wide(g, K)) {
        (wc ? k_bwd_tile_step<K, true> : k_bwd_tile_step<K, false>)<<<grid, BATCH_TPB, 0, s>>>(
            g->bfwd, c->bi, c->fmtab, c->msigma, c->mdelta, c->mq, c->mpartial, c->harrive, g->breach, c->ctrs,
            lists_of(c), d, g->symmetric, wc);
        return;
    }
    (wc ? k_bwd_step<K, true> : k_bwd_step<K, false>)<<<grid, BATCH_TPB, 0, s>>>(
        g->bfwd, c->bi, c->fmtab, c->msigma, c->mdelta, c->mq, c->mpartial, g->breach, c->ctrs, lists_of(c), d, wc);
}

template <int K> static void combine_step_kernel(axbc_ctx *c, int d)
{
    axbc_graph *g = c->g;
    k_bwd_combine_step<K><<<dim3((g->bfwd.n_heavy + 7) / 8, K), 256, 0, c->stream>>>(
        g->bfwd, c->bi, c->fmtab, c->msigma, c->mdelta, c->mq, c->mpartial, g->breach, lists_of(c), d);
}

static void drop_captures(axbc_ctx *c)
{
    for (int i = 0; i < 2; i++) {
        if (c->fwd_step_exec[i]) cudaGraphExecDestroy(c->fwd_step_exec[i]);
        c->fwd_step_exec[i] = nullptr;
    }
}

// Capture one forward step of width K as a CUDA graph; every argument is fixed
// for the context (levels come from device state).
template <int K> static int capture_steps(axbc_ctx *c)
{
    const int i = K - 1;
    if (c->fwd_step_exec[i]) return AXBC_OK;
    cudaGraph_t gr = nullptr;
    CU(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
    fwd_step_kernel<K>(c, nullptr);
    stats_step_kernel<K>(c);
    cudaError_t e = cudaStreamEndCapture(c->stream, &gr);
    if (e != cudaSuccess) return axbc_cuda_fail(e, "capture level step", __FILE__, __LINE__);
    e = cudaGraphInstantiate(&c->fwd_step_exec[i], gr, 0);
    cudaGraphDestroy(gr);
    if (e != cudaSuccess) return axbc_cuda_fail(e, "instantiate level step", __FILE__, __LINE__);
    return AXBC_OK;
}

// Forward levels and backward depths as launches of the step kernels: CUDA
// graph replays of one forward level, in blocks (profiling and counting: each
// kernel launched on its own), then one launch per depth.  *L_out: the first level that discovered
// nothing.
template <int K> static int traverse_stepwise(axbc_ctx *c, int nsrc, int *L_out)
{
    axbc_graph *g = c->g;
    const uint64_t n = g->n;
    cudaStream_t s = c->stream;
    const bool prof = c->prof_on || c->count_on;
    unsigned long long *wc = c->count_on ? c->wcount : nullptr;
    const size_t ctl_off = offsetof(BatchInfo, depth0mask);
    const size_t ctl_len = offsetof(BatchInfo, push_factor) - ctl_off;
    const size_t prof_first = c->prof.size();
    // forward steps launched before the first look at `alive`: one more than
    // the last batch needed, so a batch like it ends after one host round
    // trip; then groups of 8, 16, ... 256
    int launched = 0, B = std::max(4, std::min(4096, c->last_batch_levels + 1)), more = 8;
    if (c->last_batch_levels == 0) B = 8;
    for (;;) {
        TRY(axbc_batch_levels_alloc(c, launched + B + 2));
        for (int i = 0; i < B; i++) {
            if (!prof) {
                CU(cudaGraphLaunch(c->fwd_step_exec[K - 1], s));
            } else {
                const int L = launched + i + 1;
                {
                    // the direction is known once the level has run
                    ProfScope ps(c, KP_FWD_PULL, 0);
                    if (c->prof_on) c->prof.back().tag = L;
                    fwd_step_kernel<K>(c, wc);
                }
                {
                    ProfScope ps(c, KP_LEVEL_STATS, 0);
                    if (c->prof_on) c->prof.back().tag = L;
                    stats_step_kernel<K>(c);
                }
            }
        }
        CU_LAUNCH("forward levels");
        if (!prof) c->launches += 2ull * B;
        launched += B;
        c->prev_lend = std::min(launched, (int)c->fmask.size() - 1);  // masks written so far
        CU(cudaMemcpyAsync((char *)c->bi_host + ctl_off, (char *)c->bi + ctl_off, ctl_len,
                           cudaMemcpyDeviceToHost, s));
        CU(cudaStreamSynchronize(s));
        if (!c->bi_host->alive) break;
        B = more;
        more = std::min(2 * more, 256);
        if (launched + B + 2 > AXBC_MAX_LEVELS) {
            axbc_set_error("traversal deeper than %d levels", AXBC_MAX_LEVELS - 2);
            return AXBC_ERR_RANGE;
        }
    }
    const int L = c->bi_host->lend, Dmax = c->bi_host->dmax;
    *L_out = L;

    // per-level totals for the byte model of the profiling hooks
    std::vector<unsigned long long> lte, lcnt;
    std::vector<int32_t> lmode;
    if (c->prof_on) {
        lte.resize(L + 1);
        lcnt.resize(L + 1);
        lmode.resize(L + 1);
        // one wait for the three per-level arrays
        CU(cudaMemcpyAsync(lte.data(), c->d_level_te, (L + 1) * 8, cudaMemcpyDeviceToHost, s));
        CU(cudaMemcpyAsync(lcnt.data(), c->d_level_cnt, (L + 1) * 8, cudaMemcpyDeviceToHost, s));
        CU(cudaMemcpyAsync(lmode.data(), c->d_level_mode, (L + 1) * 4, cudaMemcpyDeviceToHost, s));
        CU(cudaStreamSynchronize(s));
        const double W = nsrc;
        for (size_t i = prof_first; i < c->prof.size(); i++) {
            ProfRec &r = c->prof[i];
            if (r.tag < 1 || r.tag > L) continue;  // steps past the last level: no work
            if (r.kind == KP_FWD_PULL) {
                if (lmode[r.tag]) r.kind = KP_FWD_PUSH;
                r.bytes = (double)lte[r.tag - 1] * (4.0 / W + 4.0);
            } else if (r.kind == KP_LEVEL_STATS) {
                r.bytes = (double)n * 16.0;
            }
        }
    }

    // backward: depths Dmax .. 0 (depth 0 only for pivots whose BFS ended at level 2)
    const unsigned long long depth0 = c->bi_host->depth0mask;
    if (Dmax >= 0) {
        for (int d = Dmax; d >= (depth0 ? 0 : 1); d--) {
            const bool combine = bwd_wide(g, K) && g->bfwd.n_heavy > 0;
            if (!prof) {
                bwd_step_kernel<K>(c, d, nullptr);
                if (combine) combine_step_kernel<K>(c, d);
                c->launches += combine ? 2 : 1;
                continue;
            }
            const double W = nsrc;
            double bytes = 0.0;
            if (c->prof_on) {
                double te_d = (double)lte[d], cnt_d = (double)lcnt[d];
                if (d == 0) {
                    const double frac = (double)__builtin_popcountll(depth0) / W;
                    te_d *= frac;
                    cnt_d *= frac;
                }
                bytes = d == Dmax ? cnt_d * 4.0 : te_d * (4.0 / W + 8.0);
            }
            {
                ProfScope ps(c, KP_BWD, bytes);
                if (c->prof_on) c->prof.back().tag = d;
                bwd_step_kernel<K>(c, d, wc ? wc + KP_BWD * WC_NFIELDS : nullptr);
            }
            if (combine) {
                ProfScope ps(c, KP_BWD_COMBINE, 0);
                combine_step_kernel<K>(c, d);
            }
        }
        CU_LAUNCH("backward levels");
    }
    return AXBC_OK;
}

// Whether this batch runs as one persistent launch: always or never when the
// context says so; otherwise a batch on a graph of less than 2^21 adjacency
// entries, whose levels are shorter than the launches between them, and a batch
// of at most AXBC_PERSIST_AUTO_WIDTH pivots when the last batch was deep, or --
// for the first batch -- when no vertex has more than 64 neighbours.  (Batches
// that mesh.cu takes, or of one pivot, do not come here.)  Measured, us a pass,
// steps : persistent, 32 and 64 pivots: 0.02 M entries 206 : 161 and 230 : 208; 0.43 M
// 382 : 300 and 404 : 390; 1.4 M 423 : 336 and 564 : 510; 1.8 M 440 : 356 and 645 :
// 565; 3.7 M 605 : 600 and 810 : 977.  Counting runs use the step kernels.
static bool use_persist(axbc_ctx *c, int nsrc)
{
    if (c->count_on || c->persist_mode < 0) return false;
    if (c->persist_mode > 0) return true;
    if (!c->coop) return false;
    if (c->g->m < AXBC_PERSIST_AUTO_M) return true;
    if (nsrc > AXBC_PERSIST_AUTO_WIDTH) return false;
    if (c->last_batch_levels > AXBC_PERSIST_AUTO_LEVELS) return true;
    return c->last_batch_levels == 0 && c->g->max_deg <= 64;
}

// The batch's levels in k_traverse_persist: a cooperative launch of every
// block that fits resident (at most persist_blocks_per_sm per SM).  Level masks
// are allocated up front for the last batch's depth and grown when the loop
// asks for more.  *L_out: the first level that discovered nothing.  *done =
// false: the device refuses the launch or a barrier wait ran out, the pass has
// to start again in another form.
template <int K> static int traverse_persistent(axbc_ctx *c, int *L_out, bool *done)
{
    axbc_graph *g = c->g;
    cudaStream_t s = c->stream;
    int &fit = c->persist_fit[K - 1];
    if (!fit) CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_traverse_persist<K>, BATCH_TPB, 0));
    const int bps = std::min(fit, std::max(1, c->persist_blocks_per_sm));
    *done = false;
    if (bps < 1 && c->persist_mode == 0) return AXBC_OK;
    if (bps < 1) {
        axbc_set_error("persistent level loop: no block of it fits on an SM");
        return AXBC_ERR_CUDA;
    }
    // every resident block, or as many as have work
    int grid = grid_of(c, bps, std::max<uint64_t>((adj_warps(g->bfwd) + 7) / 8, (g->n + 255) / 256));
    const LevelLists ll = lists_of(c);
    const uint32_t lmax_list = list_max_of(c);
    const uint32_t pool_cap = c->lpool_cap;
    const uint64_t n = g->n;
    long long budget = AXBC_BAR_BUDGET;
    int levels = std::max(16, c->last_batch_levels + 8);
    const size_t ctl_off = offsetof(BatchInfo, depth0mask);
    const size_t ctl_len = offsetof(BatchInfo, push_factor) - ctl_off;
    GridSync *gs = &c->bi->gs;
    const GridSync &hs = c->bi_host->gs;
    for (bool first = true;; first = false) {
        levels = std::min(levels, AXBC_MAX_LEVELS - 2);
        TRY(axbc_batch_levels_alloc(c, levels));
        c->prev_lend = levels - 1;  // masks the loop may write, cleared before the next batch
        if (!first) CU(cudaMemsetAsync(gs, 0, sizeof(GridSync), s));
        int lmax = levels;
        void *args[] = {(void *)&g->bfwd, (void *)&g->brev, (void *)&c->bi, (void *)&c->fmtab,
                        (void *)&c->seen, (void *)&c->msigma, (void *)&c->mdelta, (void *)&c->mq,
                        (void *)&c->mpartial, (void *)&c->harrive, (void *)&g->breach, (void *)&c->ctrs,
                        (void *)&ll, (void *)&g->symmetric, (void *)&c->d_level_te, (void *)&c->d_level_cnt, (void *)&c->d_level_mode,
                        (void *)&pool_cap, (void *)&lmax_list, (void *)&n, (void *)&lmax,
                        (void *)&gs, (void *)&budget};
        TRY(axbc_coop_launch(c, (const void *)k_traverse_persist<K>, grid, BATCH_TPB, args, done));
        if (!*done && first && c->persist_mode == 0) return AXBC_OK;
        if (!*done) {
            axbc_set_error("persistent level loop: the device refuses the cooperative launch");
            return AXBC_ERR_CUDA;
        }
        CU_LAUNCH("k_traverse_persist");
        // the level state and the barrier's record in one copy
        CU(cudaMemcpyAsync((char *)c->bi_host + ctl_off, (char *)c->bi + ctl_off, ctl_len, cudaMemcpyDeviceToHost, s));
        CU(cudaStreamSynchronize(s));
        int site = 0;
        TRY(axbc_wait_ran_out(c, hs.err, c->harrive, (uint64_t)(g->bfwd.n_heavy + 1) * 2, &site));
        *done = site == 0;
        if (site && c->persist_mode == 0) return AXBC_OK;
        if (site) {
            axbc_set_error("persistent level loop: a grid barrier wait ran out of its budget (site %d)", site);
            return AXBC_ERR_TIMEOUT;
        }
        if (!hs.need) break;
        if (levels >= AXBC_MAX_LEVELS - 2) {
            axbc_set_error("traversal deeper than %d levels", AXBC_MAX_LEVELS - 2);
            return AXBC_ERR_RANGE;
        }
        levels *= 2;
    }
    *L_out = c->bi_host->lend;
    return AXBC_OK;
}

static int read_back(axbc_ctx *c, int nsrc, int L);

// What a pass finds zero, and its roots (c->bi holds them as vertex ids, or in
// the view's numbering when a start before this one has renumbered them).
template <int K> static int start_pass(axbc_ctx *c, int nsrc, int H, bool in_view)
{
    axbc_graph *g = c->g;
    const uint64_t n = g->n;
    PassStart P;
    P.bi = c->bi;
    P.tab = c->fmtab;
    P.seen = c->seen;
    P.msigma = c->msigma;
    P.ctrs = c->ctrs;
    P.ll = lists_of(c);
    P.level_te = c->d_level_te;
    P.level_cnt = c->d_level_cnt;
    P.col = g->bfwd.col;
    P.rcol = g->brev.col;
    P.reach = g->breach;
    P.to_view = in_view ? nullptr : g->to_view;
    P.bc = c->bc;
    P.n = n;
    P.m = g->m;
    // a factor of 1e30 or more pulls every level
    P.push_min = c->push_factor_batch >= 1e30 ? 0ull : (unsigned long long)(n / 4);
    P.push_factor = c->push_factor_batch;
    P.pool_cap = c->lpool_cap;
    P.list_max = list_max_of(c);
    P.big = g->bfwd.big;
    P.nsrc = nsrc;
    P.H = H;
    P.prev_k = c->last_batch_k;
    P.prev_last = c->prev_lend;
    {
        ProfScope ps(c, KP_LEVEL_STATS, 0);
        k_pass_start<K><<<grid_of(c, 8, (n * K + 31) / 32), 256, 0, c->stream>>>(P);
    }
    CU_LAUNCH("k_pass_start");
    c->last_batch_k = K;
    c->prev_lend = 0;
    return AXBC_OK;
}

// Forward and backward passes of the batch of width K whose roots/p are in
// c->bi.  The host launches forward level steps in blocks (8, then doubling)
// and reads the level state once per block; steps past the last level do
// nothing.
template <int K> static int batch_traverse(axbc_ctx *c, int nsrc, int H)
{
    axbc_graph *g = c->g;
    const uint64_t n = g->n;
    cudaStream_t s = c->stream;
    TRY(occupancy<K>(c));
    // per-launch mode: profiling events around each kernel, or the counting builds
    const bool prof = c->prof_on || c->count_on;
    TRY(ensure_level_tables(c));
    TRY(axbc_batch_levels_alloc(c, 10));
    if (!prof) TRY(capture_steps<K>(c));

    // a larger list pool if the previous batch ran out of list space (its lists,
    // which say where its masks are set, move along)
    TRY(axbc_batch_settle(c));
    const uint64_t pool_limit = (uint64_t)AXBC_WMAX * n + 64;
    if (c->pool_short && c->lpool_cap < pool_limit) {
        // the larger pool is allocated before the old one goes, so a failed
        // allocation leaves the context with a usable (smaller) pool
        const uint32_t ncap = (uint32_t)std::min<uint64_t>(std::min<uint64_t>(4ull * c->lpool_cap, pool_limit),
                                                           0xffffffffull);
        uint32_t *np = nullptr;
        TRY(axbc_dalloc((void **)&np, (uint64_t)ncap * 4, &c->bytes));
        CU(cudaMemcpyAsync(np, c->lpool, (uint64_t)c->lpool_cap * 4, cudaMemcpyDeviceToDevice, s));
        CU(cudaStreamSynchronize(s));
        axbc_dfree(c->lpool);
        c->lpool = np;
        c->lpool_cap = ncap;
        c->pool_short = false;
        drop_captures(c);
        if (!prof) TRY(capture_steps<K>(c));
    }
    TRY(start_pass<K>(c, nsrc, H, false));

    int L = 0;
    bool done = false;
    if (use_persist(c, nsrc)) {
        TRY(traverse_persistent<K>(c, &L, &done));
        if (!done) TRY(start_pass<K>(c, nsrc, H, true));
    }
    if (!done) TRY(traverse_stepwise<K>(c, nsrc, &L));
    TRY(read_back(c, nsrc, L));
    c->prev_lend = L;
    return AXBC_OK;
}

// the per-pivot level counts and the list-pool flag arrive in the background;
// the next batch (or a caller that reports them) waits for them
static int read_back(axbc_ctx *c, int nsrc, int L)
{
    cudaStream_t s = c->stream;
    if (!c->rb_ev) CU(cudaEventCreateWithFlags(&c->rb_ev, cudaEventDisableTiming));
    CU(cudaMemcpyAsync(c->bi_host->Ls, c->bi->Ls, sizeof(c->bi_host->Ls), cudaMemcpyDeviceToHost, s));
    CU(cudaMemcpyAsync(&c->bi_host->pool_short, &c->bi->pool_short, 4, cudaMemcpyDeviceToHost, s));
    CU(cudaEventRecord(c->rb_ev, s));
    c->rb_pending = true;
    c->last_batch_levels = L;
    c->last_batch_nsrc = nsrc;
    return AXBC_OK;
}

// A pass of one pivot runs in the plain form's one launch: rows of 32 pivots
// would carry one (us a pass, persistent rows : this: scale 14 218 : 115, 18 498 :
// 318).  Counting runs and a level loop that the caller
// has chosen keep the batched kernels.
static int traverse_one(axbc_ctx *c, int H, bool *done)
{
    TRY(ensure_level_tables(c));
    TRY(axbc_batch_settle(c));
    int L = 0;
    TRY(axbc_one_traverse(c, H, &L, done));
    if (!*done) return AXBC_OK;
    if (L > AXBC_MAX_LEVELS - 3) {
        axbc_set_error("traversal deeper than %d levels", AXBC_MAX_LEVELS - 2);
        return AXBC_ERR_RANGE;
    }
    c->last_form = axbc_ctx::ONE;
    return read_back(c, 1, L);
}

// A pass on a mesh: a cluster of blocks per pivot (mesh.cu).
static int traverse_mesh(axbc_ctx *c, int nsrc, int H, bool *done)
{
    TRY(ensure_level_tables(c));
    TRY(axbc_batch_settle(c));
    int L = 0;
    TRY(axbc_mesh_traverse(c, nsrc, H, &L, done));
    if (!*done) return AXBC_OK;
    c->last_form = axbc_ctx::MESH;
    return read_back(c, nsrc, L);
}

// A multi-source pass of nsrc <= 64 pivots: 32-bit masks up to 32 pivots,
// 64-bit masks above.
int axbc_batch_traverse(axbc_ctx *c, int nsrc, int H)
{
    if (nsrc < 1 || nsrc > AXBC_WMAX) {
        axbc_set_error("batched pass of %d pivots (1..%d)", nsrc, AXBC_WMAX);
        return AXBC_ERR_INVALID;
    }
    // until this pass is done there is none to show (its depth, last_batch_levels,
    // stays as the guess it is): the pass before may have left its results in
    // another form than the buffers that a failing one leaves behind
    TRY(axbc_batch_settle(c));
    c->last_batch_nsrc = 0;
    if (c->persist_mode == 0 && !c->count_on) {
        if (axbc_mesh_fits(c)) {
            bool done = false;
            TRY(traverse_mesh(c, nsrc, H, &done));
            if (done) return AXBC_OK;
        }
        int rc = AXBC_OK;
        if (nsrc == 1 && axbc_one_fits(c, &rc)) {
            bool done = false;
            TRY(traverse_one(c, H, &done));
            if (done) return AXBC_OK;
        }
        TRY(rc);
    }
    c->last_form = axbc_ctx::ROWS;
    return width_k(nsrc) == 2 ? batch_traverse<2>(c, nsrc, H) : batch_traverse<1>(c, nsrc, H);
}

int axbc_batch_settle(axbc_ctx *c)
{
    if (!c->rb_pending) return AXBC_OK;
    CU(cudaEventSynchronize(c->rb_ev));
    c->rb_pending = false;
    c->pool_short = c->bi_host->pool_short != 0;
    for (int i = 0; i < AXBC_WMAX; i++) c->last_Ls[i] = i < c->last_batch_nsrc ? c->bi_host->Ls[i] : 0;
    return AXBC_OK;
}

// The update of the applied lanes into each lane's bc vector, then the last
// applied dependency vector of each lane segment [lane_lo[i], lane_hi[i]) into
// delta_out[i] (defaults: one segment of all lanes into the context's).
template <int K>
static int apply_lanes(axbc_ctx *c, float *const *delta_out, const int *lane_lo, const int *lane_hi, int nseg)
{
    axbc_graph *g = c->g;
    cudaStream_t s = c->stream;
    // a grid-stride loop: exactly the blocks that stay resident
    if (!c->upd_blocks_per_sm[K - 1]) {
        int b = 0;
        CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_update_m<K>, UPD_TPB(K), 0));
        c->upd_blocks_per_sm[K - 1] = std::max(1, b);
    }
    const int grid = grid_of(c, c->upd_blocks_per_sm[K - 1], (g->n + UPD_TPB(K) - 1) / UPD_TPB(K));
    const bool one_seg = nseg == 1 && (!lane_lo || lane_lo[0] == 0) && (!lane_hi || lane_hi[0] >= AXBC_W * K);
    {
        ProfScope ps(c, KP_UPDATE, (double)g->n * c->last_batch_nsrc * 20.0);
        // one segment over all lanes: the update writes the last delta itself
        k_update_m<K><<<grid, UPD_TPB(K), 0, s>>>(c->mdelta, c->seen, g->breach, g->n, c->bi,
                                                  one_seg ? (delta_out ? delta_out[0] : c->delta_last) : nullptr,
                                                  g->from_view);
    }
    for (int i = 0; i < nseg && !one_seg; i++) {
        ProfScope ps(c, KP_UPDATE, 0);
        k_extract_delta<K><<<grid, 256, 0, s>>>(delta_out ? delta_out[i] : c->delta_last, c->mdelta, c->seen,
                                                g->breach, g->n, c->bi, lane_lo ? lane_lo[i] : 0,
                                                lane_hi ? lane_hi[i] : AXBC_WMAX, g->from_view);
    }
    CU_LAUNCH("update");
    c->delta_last_valid = true;
    return AXBC_OK;
}

int axbc_batch_apply_lanes(axbc_ctx *c, float *const *delta_out, const int *lane_lo,
                           const int *lane_hi, int nseg)
{
    if (c->last_form == axbc_ctx::MESH) {
        TRY(axbc_mesh_apply(c, delta_out, lane_lo, lane_hi, nseg));
        c->delta_last_valid = true;
        return AXBC_OK;
    }
    if (c->last_form == axbc_ctx::ONE) {
        // the segment that holds lane 0
        float *out = nullptr;
        for (int i = 0; i < nseg; i++)
            if ((!lane_lo || lane_lo[i] == 0) && (!lane_hi || lane_hi[i] > 0))
                out = delta_out ? delta_out[i] : c->delta_last;
        TRY(axbc_one_apply(c, out));
        c->delta_last_valid = true;
        return AXBC_OK;
    }
    return c->last_batch_k == 2 ? apply_lanes<2>(c, delta_out, lane_lo, lane_hi, nseg)
                                : apply_lanes<1>(c, delta_out, lane_lo, lane_hi, nseg);
}

// Per forward level of the last batch: vertices newly reached (over all
// pivots), their degree sum, the direction (1 push), and the level's vertex
// list (entries counted, capacity; count > capacity: the level was scanned).
extern "C" int axbc_ctx_level_stats(axbc_ctx *c, uint64_t *count, uint64_t *te, int32_t *push,
                                    uint32_t *list_count, uint32_t *list_cap, int max_levels,
                                    int *levels)
{
    CHECK_ARG(c && levels, "axbc_ctx_level_stats: null argument");
    const int L = std::min(c->last_batch_levels + 1, max_levels);
    *levels = c->last_batch_levels + 1;
    if (!c->d_level_cnt || L <= 0) return AXBC_OK;
    if (c->last_form == axbc_ctx::MESH) TRY(axbc_mesh_level_tables(c, L));
    CU(cudaStreamSynchronize(c->stream));
    if (c->last_form == axbc_ctx::MESH) {
        // every level pushed, every pivot with a list of its own
        std::vector<unsigned long long> n_l(L);
        CU(cudaMemcpy(n_l.data(), c->d_level_cnt, L * 8, cudaMemcpyDeviceToHost));
        for (int i = 0; i < L; i++) {
            if (push) push[i] = 1;
            if (list_count) list_count[i] = (uint32_t)n_l[i];
            if (list_cap) list_cap[i] = std::max(list_max_of(c), (uint32_t)n_l[i]);
        }
        push = nullptr;
        list_count = list_cap = nullptr;
    }
    if (count) CU(cudaMemcpy(count, c->d_level_cnt, L * 8, cudaMemcpyDeviceToHost));
    if (te) CU(cudaMemcpy(te, c->d_level_te, L * 8, cudaMemcpyDeviceToHost));
    if (push) CU(cudaMemcpy(push, c->d_level_mode, L * 4, cudaMemcpyDeviceToHost));
    if (c->last_form == axbc_ctx::ONE) {
        // its queue lists every level
        std::vector<uint32_t> lev(L + 1);
        CU(cudaMemcpy(lev.data(), c->one.lev, (L + 1) * 4, cudaMemcpyDeviceToHost));
        for (int i = 0; i < L; i++) {
            if (list_count) list_count[i] = lev[i + 1] - lev[i];
            if (list_cap) list_cap[i] = std::max(list_max_of(c), lev[i + 1] - lev[i]);
        }
        return AXBC_OK;
    }
    if (list_count) CU(cudaMemcpy(list_count, c->lcount, L * 4, cudaMemcpyDeviceToHost));
    if (list_cap) CU(cudaMemcpy(list_cap, c->lcap, L * 4, cudaMemcpyDeviceToHost));
    return AXBC_OK;
}

int axbc_batch_apply(axbc_ctx *c) { return axbc_batch_apply_lanes(c, nullptr, nullptr, nullptr, 1); }

__global__ void k_set_lane_targets(BatchInfo *bi, LaneTargets t)
{
    if (threadIdx.x < AXBC_WMAX) bi->lane_bc[threadIdx.x] = t.bc[threadIdx.x];
}

// bc_of_lane: AXBC_WMAX vectors, one per lane of the pass
int axbc_batch_set_targets(axbc_ctx *c, float *const *bc_of_lane)
{
    LaneTargets t;
    for (int i = 0; i < AXBC_WMAX; i++) t.bc[i] = bc_of_lane[i];
    k_set_lane_targets<<<1, AXBC_WMAX, 0, c->stream>>>(c->bi, t);
    CU_LAUNCH("k_set_lane_targets");
    return AXBC_OK;
}

extern "C" int axbc_run_batch(axbc_ctx *c, const uint32_t *v0, const double *p, int k, int H,
                              axbc_pivot_stats *stats)
{
    CHECK_ARG(c && v0 && p, "axbc_run_batch: null argument");
    CHECK_ARG(k >= 1 && k <= AXBC_MAX_BATCH, "axbc_run_batch: k must be in [1, 64]");
    CHECK_ARG(H == 0 || H == 1, "axbc_run_batch: H must be 0 or 1");
    for (int i = 0; i < k; i++) CHECK_ARG(v0[i] < c->g->n, "axbc_run_batch: pivot >= n");
    TRY(axbc_ensure_batch(c));
    cudaStream_t s = c->stream;
    for (int i = 0; i < k; i++) {
        c->bi_host->root[i] = v0[i];
        c->bi_host->p[i] = p[i];
    }
    // roots and probabilities lie next to each other
    static_assert(offsetof(BatchInfo, p) == offsetof(BatchInfo, root) + sizeof(BatchInfo::root), "root, p");
    CU(cudaMemcpyAsync(&c->bi->root, c->bi_host->root, sizeof(BatchInfo::root) + sizeof(BatchInfo::p),
                       cudaMemcpyHostToDevice, s));
    TRY(axbc_batch_traverse(c, k, H));
    TRY(axbc_batch_apply(c));
    if (stats) CU(cudaMemcpyAsync(c->bi_host, c->bi, sizeof(BatchInfo), cudaMemcpyDeviceToHost, s));
    if (stats) CU(cudaStreamSynchronize(s));
    TRY(axbc_batch_settle(c));
    if (stats) {
        for (int i = 0; i < k; i++) {
            stats[i].nvisited = c->bi_host->nvis[i];
            stats[i].all = (H == 1 ? (uint32_t)c->bi_host->rsum[i] : 0u) + c->bi_host->root_reach[i];
            stats[i].te = 2 * c->bi_host->te[i];
            stats[i].levels = c->last_Ls[i];
            stats[i].pad = 0;
        }
    }
    return AXBC_OK;
}

extern "C" int axbc_get_batch_source(axbc_ctx *c, int src, uint32_t *sigma_host, int32_t *lvl_host,
                                     float *delta_host)
{
    CHECK_ARG(c && c->seen, "axbc_get_batch_source: no batch has run");
    CHECK_ARG(src >= 0 && src < c->last_batch_nsrc, "axbc_get_batch_source: bad source index");
    const uint64_t n = c->g->n;
    cudaStream_t s = c->stream;
    if (c->last_form == axbc_ctx::MESH) return axbc_mesh_source(c, src, sigma_host, lvl_host, delta_host);
    if (c->last_form == axbc_ctx::ONE) {
        if (sigma_host) CU(cudaMemcpyAsync(sigma_host, c->one.sigma, n * 4, cudaMemcpyDeviceToHost, s));
        if (lvl_host) CU(cudaMemcpyAsync(lvl_host, c->one.lvl, n * 4, cudaMemcpyDeviceToHost, s));
        if (delta_host) CU(cudaMemcpyAsync(delta_host, c->one.delta, n * 4, cudaMemcpyDeviceToHost, s));
        CU(cudaStreamSynchronize(s));
        return AXBC_OK;
    }
    const int levels = c->last_batch_levels + 1;
    uint32_t **d_fm = nullptr;
    uint32_t *sig = nullptr;
    int32_t *lvl = nullptr;
    float *dl = nullptr;
    TRY(axbc_dalloc((void **)&d_fm, levels * sizeof(uint32_t *), nullptr));
    TRY(axbc_dalloc((void **)&sig, n * 4, nullptr));
    TRY(axbc_dalloc((void **)&lvl, n * 4, nullptr));
    TRY(axbc_dalloc((void **)&dl, n * 4, nullptr));
    CU(cudaMemcpyAsync(d_fm, c->fmask.data(), levels * sizeof(uint32_t *), cudaMemcpyHostToDevice, s));
    unsigned long long depth0 = 0;
    CU(cudaMemcpyAsync(&depth0, &c->bi->depth0mask, 8, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    if (c->last_batch_k == 2)
        k_source_view<2><<<axbc_grid_for(c, 256, 4), 256, 0, s>>>(src, levels, d_fm, c->seen, c->msigma, c->mdelta,
                                                                  c->g->breach, n, depth0, sig, lvl, dl,
                                                                  c->g->from_view);
    else
        k_source_view<1><<<axbc_grid_for(c, 256, 4), 256, 0, s>>>(src, levels, d_fm, c->seen, c->msigma, c->mdelta,
                                                                  c->g->breach, n, depth0, sig, lvl, dl,
                                                                  c->g->from_view);
    CU_LAUNCH("k_source_view");
    if (sigma_host) CU(cudaMemcpyAsync(sigma_host, sig, n * 4, cudaMemcpyDeviceToHost, s));
    if (lvl_host) CU(cudaMemcpyAsync(lvl_host, lvl, n * 4, cudaMemcpyDeviceToHost, s));
    if (delta_host) CU(cudaMemcpyAsync(delta_host, dl, n * 4, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    axbc_dfree(d_fm);
    axbc_dfree(sig);
    axbc_dfree(lvl);
    axbc_dfree(dl);
    return AXBC_OK;
}

// ------------------------------------------------------------ self-test
// The update's fast float(double(x)/p) against the double divide on n
// generated (x, p) pairs: random magnitudes, random bit patterns, and x*p
// products chosen to land next to float rounding midpoints.
__device__ __forceinline__ uint64_t st_mix(uint64_t z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__global__ void k_selftest_div(uint64_t n, uint64_t seed, unsigned long long *bad,
                               unsigned long long *slow)
{
    unsigned long long nb = 0, ns = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t h1 = st_mix(seed ^ (i * 3 + 1)), h2 = st_mix(seed ^ (i * 3 + 2));
        float x;
        double p;
        switch (i % 6) {
        case 0:  // pivot probabilities: 1/N-like and products of small integers
            x = (float)((h1 & 0xffffff) + 1) * ldexpf(1.0f, (int)((h1 >> 24) & 31) - 16);
            p = 1.0 / (double)((h2 & 0xffffff) + 1);
            break;
        case 1:  // random float bits (positive, normal), random double p in (0,1]
            x = __uint_as_float(((uint32_t)(h1 & 0x7fffffff) % 0x7f000000u) | 0x00800000u);
            p = (double)((h2 >> 11) + 1) * 0x1.0p-53;
            break;
        case 2: {  // near midpoints: x/p = m + half ulp(m) +- tiny
            const float m = (float)((h1 & 0xffffff) | 0x800000) * ldexpf(1.0f, (int)((h1 >> 24) & 15) - 8);
            p = (double)((h2 >> 11) + 1) * 0x1.0p-53 + 1e-9;
            const double target = ((double)m + (double)m * 0x1.0p-24) * (1.0 + ((int)(h2 & 7) - 3) * 0x1.0p-50);
            x = (float)(target * p);
            break;
        }
        case 3:  // integers times integers
            x = (float)((h1 & 0xfffff) + 1);
            p = (double)((h2 & 0xfff) + 1) / (double)((h2 >> 12 & 0xfffff) + 1);
            break;
        case 4:  // exact powers of two: small integers over p = 2^-k
            x = (float)((h1 & 15) + 1) * ldexpf(1.0f, (int)((h1 >> 4) & 15) - 8);
            p = ldexp(1.0, -(int)(h2 & 31));
            break;
        default: {  // just below a power of two, around the quarter-ulp boundary
            p = (double)((h2 >> 11) + 1) * 0x1.0p-53 + 1e-9;
            const double pw = ldexp(1.0, (int)(h1 & 31) - 8);
            const double target = pw * (1.0 - 0x1.0p-26 * (1.0 + ((int)((h1 >> 5) & 15) - 8) * 0x1.0p-20));
            x = (float)(target * p);
        }
        }
        if (!(x > 0.0f) || !(p > 0.0)) continue;
        const InvSplit iv = inv_split(p);
        const float f = div_to_float(x, p, iv);
        const float e = __double2float_rn(__ddiv_rn((double)x, p));
        if (__float_as_uint(f) != __float_as_uint(e)) nb++;
        // count how often the exact path decided
        const float a = __fmul_rn(x, iv.hi);
        const float ee = __fmaf_rn(x, iv.hi, -a);
        const float b = __fmaf_rn(x, iv.lo, ee);
        const float s = __fadd_rn(a, b);
        if (!iv.ok || __float_as_uint(s) != __float_as_uint(f)) ns++;
    }
    if (nb) atomicAdd(bad, nb);
    if (ns) atomicAdd(slow, ns);
}

extern "C" int axbc_selftest_division(uint64_t n, uint64_t seed, uint64_t *mismatches,
                                      uint64_t *exact_path)
{
    CHECK_ARG(mismatches, "axbc_selftest_division: null argument");
    unsigned long long *d = nullptr;
    TRY(axbc_dalloc((void **)&d, 16, nullptr));
    CU(cudaMemset(d, 0, 16));
    k_selftest_div<<<1024, 256>>>(n, seed, d, d + 1);
    CU_LAUNCH("k_selftest_div");
    unsigned long long h[2];
    CU(cudaMemcpy(h, d, 16, cudaMemcpyDeviceToHost));
    axbc_dfree(d);
    *mismatches = h[0];
    if (exact_path) *exact_path = h[1];
    return AXBC_OK;
}

// ------------------------------------------------ persistent loop controls
extern "C" int axbc_ctx_set_persistent(axbc_ctx *c, int mode, int blocks_per_sm)
{
    CHECK_ARG(c, "axbc_ctx_set_persistent: null context");
    CHECK_ARG(mode >= -1 && mode <= 1, "axbc_ctx_set_persistent: mode must be -1, 0 or 1");
    CHECK_ARG(blocks_per_sm >= 0 && blocks_per_sm <= 8, "axbc_ctx_set_persistent: blocks_per_sm must be in [0, 8]");
    if (mode > 0) {
        int dev = 0, coop = 0;
        CU(cudaGetDevice(&dev));
        CU(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        if (!coop) {
            axbc_set_error("axbc_ctx_set_persistent: the device has no cooperative launch");
            return AXBC_ERR_INVALID;
        }
    }
    c->persist_mode = mode;
    if (blocks_per_sm > 0) c->persist_blocks_per_sm = blocks_per_sm;
    return AXBC_OK;
}

extern "C" int axbc_selftest_grid_barrier(int blocks_per_sm, int rounds, long long budget_cycles,
                                          int absent_block, int *err_site, uint32_t *leads, float *ms)
{
    CHECK_ARG(err_site && leads, "axbc_selftest_grid_barrier: null argument");
    CHECK_ARG(rounds >= 1 && budget_cycles > 0, "axbc_selftest_grid_barrier: bad rounds or budget");
    int dev = 0, sms = 0, fit = 0;
    CU(cudaGetDevice(&dev));
    CU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_barrier_selftest, BATCH_TPB, 0));
    CHECK_ARG(blocks_per_sm >= 1 && blocks_per_sm <= fit, "axbc_selftest_grid_barrier: blocks_per_sm does not fit");
    int grid = sms * blocks_per_sm;
    CHECK_ARG(absent_block < grid, "axbc_selftest_grid_barrier: absent_block beyond the grid");
    DBuf gs, out;
    TRY(gs.alloc(sizeof(GridSync)));
    TRY(out.alloc(4));
    CU(cudaMemset(gs.p, 0, sizeof(GridSync)));
    CU(cudaMemset(out.p, 0, 4));
    cudaEvent_t a, b;
    CU(cudaEventCreate(&a));
    CU(cudaEventCreate(&b));
    GridSync *gsp = gs.as<GridSync>();
    unsigned *outp = out.as<unsigned>();
    void *args[] = {(void *)&gsp, (void *)&rounds, (void *)&budget_cycles, (void *)&absent_block, (void *)&outp};
    CU(cudaEventRecord(a, 0));
    cudaError_t e = cudaLaunchCooperativeKernel((const void *)k_barrier_selftest, grid, BATCH_TPB, args, 0, 0);
    if (e == cudaSuccess) e = cudaEventRecord(b, 0);
    if (e == cudaSuccess) e = cudaEventSynchronize(b);
    float t = 0;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&t, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    if (e != cudaSuccess) return axbc_cuda_fail(e, "k_barrier_selftest", __FILE__, __LINE__);
    GridSync h;
    CU(cudaMemcpy(&h, gs.p, sizeof(h), cudaMemcpyDeviceToHost));
    CU(cudaMemcpy(leads, out.p, 4, cudaMemcpyDeviceToHost));
    *err_site = h.err;
    if (ms) *ms = t;
    return AXBC_OK;
}
