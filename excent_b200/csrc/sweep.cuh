// sweep.cuh -- a chunk-by-chunk pass as gathers (included by engine.cu).
//
// A swept pass pushes most of the graph, where a gather is faster than the
// scatter (pull.cuh): on an R-MAT of 16.8M vertices and 263M entries a swept
// pass takes 1.3 ms for one measure (scatter: 2.5) and 2.0 ms for three (3.4).
// What bounds it is one L1 lookup per entry (284 G/s for the GPU, less where
// lanes share one: 0.93 ms a pass; the long late parts reach 85-100 % of that) and, for the many lists of
// a few entries, chains of dependent loads in each of the phases. (Filling the
// ends of the phases with late segments, and keys loaded a batch ahead, gained
// nothing.) On a symmetric graph the push of vertex u is the same as every
// neighbour adding u's weight P[u] to its own residual, once, at any time
// between u's take and the neighbour's next take that has to see it. So each
// list is split, once per graph, by the order in which a swept pass takes
// vertices: chunk by chunk, a chunk's lists longer than HUB_MIN first, then its
// others. The early part of v's list holds the
// neighbours taken in earlier phases than v; v gathers it and is taken in its
// own phase. The late part holds the others; one last phase gathers it for
// every vertex, after which the residuals are complete, as a push leaves them.
//
// Layout (one copy of the lists, plain ids): for the early and for the late
// parts, those of at most TINY_PART entries, then those of at most PULL_LONG,
// each back to back in vertex order with the vertices that have them listed
// (more than half of an R-MAT graph's vertices have no entry at all), and the
// longer ones, and every early part of a hub vertex, apart with a segment table
// in vertex order. Tiny parts go apart because a phase is a chain of a few
// tiles a warp and a tile's time that of its longest list: with one class three
// measures on 16.8M vertices took 202.6 ms a solve, with two 191.2, PageRank
// 44.8 and 43.2. For the same reason the takes of a warp's two segments run side
// by side and a tile's residuals are loaded before its sums: 186.3 and 41.9 ms.
#pragma once

#include <type_traits>

#include "pull.cuh"

namespace excent {

struct F3 {   // the three measures of a float4 entry
    float x, y, z;
    F3() = default;
    __device__ __forceinline__ explicit F3(int) : x(0.f), y(0.f), z(0.f) {}
    __device__ __forceinline__ F3(float a, float b, float c) : x(a), y(b), z(c) {}
    __device__ __forceinline__ F3& operator+=(const F3& o) { x += o.x; y += o.y; z += o.z; return *this; }
};
__device__ __forceinline__ F3 shfl(const F3& v, int src) { return F3(shfl(v.x, src), shfl(v.y, src), shfl(v.z, src)); }
__device__ __forceinline__ F3 shfl_xor(const F3& v, int o) { return F3(shfl_xor(v.x, o), shfl_xor(v.y, o), shfl_xor(v.z, o)); }
__device__ __forceinline__ F3 warp_sum(F3 v) { return F3(warp_sum(v.x), warp_sum(v.y), warp_sum(v.z)); }

template <int L> struct GSum;
template <> struct GSum<1> { typedef float T; };
template <> struct GSum<4> { typedef F3 T; };
__device__ __forceinline__ float add_sum(float r, float s) { return r + s; }
__device__ __forceinline__ float4 add_sum(float4 r, const F3& s) { return make_float4(r.x + s.x, r.y + s.y, r.z + s.z, r.w); }
__device__ __forceinline__ bool nonzero(const F3& s) { return s.x != 0.f || s.y != 0.f || s.z != 0.f; }
__device__ __forceinline__ void red_sum(float* r, unsigned v, float s) { if (s != 0.f) red_add(r, (int)v, s); }
__device__ __forceinline__ void red_sum(float4* r, unsigned v, const F3& s) {
    if (nonzero(s)) red_add(r, (int)v, make_float4(s.x, s.y, s.z, 0.f));
}

// One segment of a hub vertex's early part (at least one per hub vertex).
struct HubPart {
    unsigned base, row;
    unsigned first;      // number of the vertex's first segment
    unsigned len_nseg;   // entries (10 bits), segments of the vertex
};
__device__ __forceinline__ ListSeg as_seg(const ListSeg& s) { return s; }
__device__ __forceinline__ ListSeg as_seg(const HubPart& s) { return ListSeg{s.base, s.len_nseg & 1023u, s.row}; }

// Vertices in ascending order, their parts back to back, their degrees (early parts only).
struct ListedParts {
    int* v;
    unsigned* off;
    uint16_t* deg;
};

// The split lists of one graph and the phases of its swept passes.
struct SweepLists {
    const int* adj;             // m entries: early parts tiny | short | long, then late parts tiny | short | long
    ListedParts e_tiny;         // vertices with entries and a tiny early part (it may be empty), not hubs
    ListedParts e_short;
    ListedParts l_tiny;         // vertices with a tiny late part of at least one entry
    ListedParts l_short;
    const uint32_t* alone;      // bitmap of the vertices without entries
    const HubPart* e_hub;       // early parts of hub vertices, in vertex order
    const ListSeg* e_mid;       // other early parts longer than PULL_LONG, one segment each, in vertex order
    const ListSeg* l_seg;       // late parts longer than PULL_LONG
    const unsigned* totals;     // [C_KINDS]: entries, segments and vertices of each kind
    const unsigned* hub_at;     // [nc + 1] first hub segment of each chunk
    const unsigned* mid_at;     // [nq + 1] first mid segment of each short phase
    const unsigned* et_at;      // [nq + 1] first of e_tiny of each short phase
    const unsigned* es_at;      // [nq + 1] ... and of e_short
    const int* q_of;            // [nc + 1] first short phase of each chunk
    unsigned* hub_done;         // segments done, at the number of the vertex's first one
    void* P;                    // what each vertex pushed in this pass
};
static constexpr unsigned TINY_PART = 8;   // entries
enum SweepCount { C_E_TINY, C_E_SHORT, C_E_HUB_SEG, C_E_MID_SEG, C_E_LONG, C_L_TINY, C_L_SHORT, C_L_SEG, C_L_LONG,
                  C_ET_V, C_ES_V, C_LT_V, C_LS_V, C_KINDS };

// ------------------------------------------------------------------ building

// The phase of every vertex in a swept pass (hub phase of chunk c: q_of[c] + c;
// short phase q of chunk c: q + c + 1).
__global__ void k_sweep_phase(int n, const ull* idx, const int* cv0, int nc, const int* q_of, int per_phase,
                              uint16_t* phase) {
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const int c = chunk_of(v, cv0, nc);
        const bool hub = idx[v + 1] - idx[v] > HUB_MIN;
        phase[v] = (uint16_t)(hub ? q_of[c] + c : q_of[c] + (int)(v - cv0[c]) / per_phase + c + 1);
    }
}

// A bijective mix of the ordered pair (a, b): variant 1 of David Stafford's finalizers of 64 bits
// ("Better Bit Mixing", 2011).
__device__ __forceinline__ ull mix_pair(int a, int b) {
    ull z = ((ull)(unsigned)a << 32) | (unsigned)b;
    z = (z ^ (z >> 31)) * 0x7FB5D329728EA185ull;
    z = (z ^ (z >> 27)) * 0x81DADEF4BC2DD44Dull;
    return z ^ (z >> 33);
}

struct SweepBuild {
    int n, nc;
    const ull* idx;
    const int* adj;
    const int* hub_id;
    const int* cv0;
    const int* q_of;
    int per_phase;
    const int* hubv;
    const ull* hubv_cnt;
    const uint16_t* phase;
    unsigned* early;
    ull* asym;              // 0: symmetric
    unsigned* counts;       // [C_KINDS][HUB_BLOCKS]
    unsigned* totals;
    ListedParts e_tiny, e_short, l_tiny, l_short;
    uint32_t* alone;
    HubPart* e_hub;
    ListSeg *e_mid, *l_seg;
    unsigned *hub_at, *mid_at, *et_at, *es_at;
    unsigned *e_dst, *l_dst;   // where each vertex's parts go
    unsigned* hub_done;
    int* out;
};

// Contribution of vertex v to each count.
__device__ __forceinline__ void sweep_sizes(const SweepBuild& a, long long v, unsigned (&k)[C_KINDS], unsigned& ec,
                                            unsigned& lc, bool& hub) {
    const unsigned deg = (unsigned)(a.idx[v + 1] - a.idx[v]);
    ec = a.early[v];
    lc = deg - ec;
    hub = deg > HUB_MIN;
    const bool et = !hub && ec <= TINY_PART, es = !hub && !et && ec <= PULL_LONG;
    const bool lt = lc <= TINY_PART, ls = !lt && lc <= PULL_LONG;
    k[C_E_TINY] = et ? ec : 0u;
    k[C_E_SHORT] = es ? ec : 0u;
    k[C_E_HUB_SEG] = hub ? max(1u, (ec + PULL_SEG - 1) / PULL_SEG) : 0u;
    k[C_E_MID_SEG] = !hub && ec > PULL_LONG ? 1u : 0u;
    k[C_E_LONG] = et || es ? 0u : ec;
    k[C_L_TINY] = lt ? lc : 0u;
    k[C_L_SHORT] = ls ? lc : 0u;
    k[C_L_SEG] = lt || ls ? 0u : (lc + PULL_SEG - 1) / PULL_SEG;
    k[C_L_LONG] = lt || ls ? 0u : lc;
    k[C_ET_V] = et && deg ? 1u : 0u;
    k[C_ES_V] = es ? 1u : 0u;
    k[C_LT_V] = lt && lc ? 1u : 0u;
    k[C_LS_V] = ls ? 1u : 0u;
}

// Each block sums a contiguous range of vertices (write 0), then, from the
// scanned sums, writes the offsets and segment tables of its range (write 1).
__global__ void __launch_bounds__(BLOCK) k_sweep_layout(SweepBuild a, int write) {
    __shared__ unsigned s_w[C_KINDS][BLOCK / 32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const long long per = ((long long)a.n + HUB_BLOCKS - 1) / HUB_BLOCKS;
    const long long v0 = blockIdx.x * per, v1 = min(v0 + per, (long long)a.n);
    unsigned at[C_KINDS];
    for (int q = 0; q < C_KINDS; q++) at[q] = write ? a.counts[q * HUB_BLOCKS + blockIdx.x] : 0u;
    // where each kind of part begins in the entries
    const unsigned at_es = write ? a.totals[C_E_TINY] : 0u;
    const unsigned at_el = at_es + (write ? a.totals[C_E_SHORT] : 0u);
    const unsigned at_lt = at_el + (write ? a.totals[C_E_LONG] : 0u);
    const unsigned at_ls = at_lt + (write ? a.totals[C_L_TINY] : 0u);
    const unsigned at_ll = at_ls + (write ? a.totals[C_L_SHORT] : 0u);
    for (long long b0 = v0; b0 < v1; b0 += BLOCK) {
        const long long v = b0 + threadIdx.x;
        unsigned k[C_KINDS], ec = 0, lc = 0, ex[C_KINDS];
        bool hub = false;
        for (int q = 0; q < C_KINDS; q++) k[q] = 0;
        if (v < v1) sweep_sizes(a, v, k, ec, lc, hub);
#pragma unroll
        for (int q = 0; q < C_KINDS; q++) {
            const unsigned in = warp_incl_scan(k[q], lane);
            ex[q] = in - k[q];
            if (lane == 31) s_w[q][wib] = in;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < C_KINDS; q++) {
            unsigned before = 0, all = 0;
            for (int w = 0; w < BLOCK / 32; w++) {
                if (w < wib) before += s_w[q][w];
                all += s_w[q][w];
            }
            ex[q] += at[q] + before;
            at[q] += all;
        }
        if (write && v < v1) {
            unsigned ed = at_el + ex[C_E_LONG], ld = at_ll + ex[C_L_LONG];
            if (k[C_ET_V]) {
                const unsigned j = ex[C_ET_V];
                ed = ex[C_E_TINY];
                a.e_tiny.v[j] = (int)v; a.e_tiny.off[j] = ed; a.e_tiny.deg[j] = (uint16_t)(ec + lc);
            }
            if (k[C_ES_V]) {
                const unsigned j = ex[C_ES_V];
                ed = at_es + ex[C_E_SHORT];
                a.e_short.v[j] = (int)v; a.e_short.off[j] = ed; a.e_short.deg[j] = (uint16_t)(ec + lc);
            }
            if (k[C_LT_V]) {
                ld = at_lt + ex[C_L_TINY];
                a.l_tiny.v[ex[C_LT_V]] = (int)v; a.l_tiny.off[ex[C_LT_V]] = ld;
            }
            if (k[C_LS_V]) {
                ld = at_ls + ex[C_L_SHORT];
                a.l_short.v[ex[C_LS_V]] = (int)v; a.l_short.off[ex[C_LS_V]] = ld;
            }
            if (ec + lc == 0) atomicOr(&a.alone[v >> 5], 1u << (v & 31));
            a.e_dst[v] = ed;
            a.l_dst[v] = ld;
            if (hub) a.hub_done[ex[C_E_HUB_SEG]] = 0;
            for (unsigned i = 0; i < k[C_E_HUB_SEG]; i++)
                a.e_hub[ex[C_E_HUB_SEG] + i] =
                    HubPart{ed + i * PULL_SEG, (unsigned)v, ex[C_E_HUB_SEG],
                            (i * PULL_SEG < ec ? min(PULL_SEG, ec - i * PULL_SEG) : 0u) | k[C_E_HUB_SEG] << 10};
            if (k[C_E_MID_SEG]) a.e_mid[ex[C_E_MID_SEG]] = ListSeg{ed, ec, (unsigned)v};
            for (unsigned i = 0; i < k[C_L_SEG]; i++)
                a.l_seg[ex[C_L_SEG] + i] = ListSeg{ld + i * PULL_SEG, min(PULL_SEG, lc - i * PULL_SEG), (unsigned)v};
            const int c = chunk_of(v, a.cv0, a.nc);
            const int in_chunk = (int)(v - a.cv0[c]);
            if (in_chunk == 0) a.hub_at[c] = ex[C_E_HUB_SEG];
            if (in_chunk % a.per_phase == 0) {
                a.mid_at[a.q_of[c] + in_chunk / a.per_phase] = ex[C_E_MID_SEG];
                a.et_at[a.q_of[c] + in_chunk / a.per_phase] = ex[C_ET_V];
                a.es_at[a.q_of[c] + in_chunk / a.per_phase] = ex[C_ES_V];
            }
            if (v == a.n - 1) {
                a.hub_at[a.nc] = a.totals[C_E_HUB_SEG];
                a.mid_at[a.q_of[a.nc]] = a.totals[C_E_MID_SEG];
                a.et_at[a.q_of[a.nc]] = a.totals[C_ET_V];
                a.es_at[a.q_of[a.nc]] = a.totals[C_ES_V];
                a.e_tiny.off[a.totals[C_ET_V]] = at_es;
                a.e_short.off[a.totals[C_ES_V]] = at_el;
                a.l_tiny.off[a.totals[C_LT_V]] = at_ls;
                a.l_short.off[a.totals[C_LS_V]] = at_ll;
            }
        }
        __syncthreads();
    }
    if (!write && threadIdx.x == 0)
        for (int q = 0; q < C_KINDS; q++) a.counts[q * HUB_BLOCKS + blockIdx.x] = at[q];
}
// One block per kind: its HUB_BLOCKS sums to offsets, and the total.
__global__ void __launch_bounds__(HUB_BLOCKS) k_sweep_scan(unsigned* counts, unsigned* totals) {
    __shared__ unsigned s_w[HUB_BLOCKS / 32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    unsigned* mine = counts + blockIdx.x * HUB_BLOCKS;
    const unsigned c = mine[threadIdx.x];
    unsigned v = warp_incl_scan(c, lane);
    if (lane == 31) s_w[wib] = v;
    __syncthreads();
    for (int w = 0; w < wib; w++) v += s_w[w];
    mine[threadIdx.x] = v - c;
    if (threadIdx.x == HUB_BLOCKS - 1) totals[blockIdx.x] = v;
}
// Entry e of the edge cache as a plain id (none past the end of the list).
__device__ __forceinline__ int plain_entry(const SweepBuild& a, ull e, bool in) {
    int u = in ? ld_edge(a.adj + e) : -1;
    if (in && u < 0) u = a.hub_id[u & HUB_MASK];
    return u;
}

// FILL 0: the length of every early part, and whether the graph is symmetric:
// the pairs (v, u) of all entries are, as a multiset, the pairs (u, v), if the
// sums of a 64-bit mix over both agree (by chance once in 2^64 graphs). FILL 1:
// every list into its two parts. A block takes a hub vertex at a time, then its
// warps tiles of 32 vertices, whose short lists are laid end to end (one warp
// per list took 18 + 15 ms on 16.8M vertices and 263M entries).
template <int FILL>
__global__ void __launch_bounds__(BLOCK) k_sweep_split(SweepBuild a) {
    constexpr int NW = BLOCK / 32, W = 4;
    __shared__ ull s_base[NW][32];
    __shared__ unsigned s_ex[NW][32], s_e[NW][32], s_l[NW][32];
    __shared__ uint16_t s_ph[NW][32];
    __shared__ int s_v[NW][32];
    __shared__ unsigned s_cnt[2];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u, le = lane == 31 ? FULL : (2u << lane) - 1u;
    ull diff = 0;
    const long long nh = (long long)*a.hubv_cnt;
    for (long long h = blockIdx.x; h < nh; h += gridDim.x) {
        const int v = a.hubv[h];
        const ull b = a.idx[v], e = a.idx[v + 1];
        const unsigned pv = a.phase[v];
        if (threadIdx.x == 0) { s_cnt[0] = FILL ? a.e_dst[v] : 0u; s_cnt[1] = FILL ? a.l_dst[v] : 0u; }
        __syncthreads();
        unsigned cnt = 0;
        for (ull i = b + wib * 32 * W; i < e; i += (ull)BLOCK * W) {
            int u[W];
            bool early[W];
#pragma unroll
            for (int k = 0; k < W; k++) u[k] = plain_entry(a, i + 32 * k + lane, i + 32 * k + lane < e);
#pragma unroll
            for (int k = 0; k < W; k++) early[k] = u[k] >= 0 && a.phase[u[k]] < pv;
            if (FILL) {
                unsigned ne = 0, nl = 0;
#pragma unroll
                for (int k = 0; k < W; k++) {
                    const unsigned be = __ballot_sync(FULL, early[k]);
                    ne += __popc(be);
                    nl += __popc(__ballot_sync(FULL, u[k] >= 0) & ~be);
                }
                unsigned ed = 0, ld = 0;
                if (lane == 0) { ed = atomicAdd(&s_cnt[0], ne); ld = atomicAdd(&s_cnt[1], nl); }
                ed = __shfl_sync(FULL, ed, 0);
                ld = __shfl_sync(FULL, ld, 0);
#pragma unroll
                for (int k = 0; k < W; k++) {
                    const unsigned be = __ballot_sync(FULL, early[k]), bl = __ballot_sync(FULL, u[k] >= 0) & ~be;
                    if (early[k]) a.out[ed + __popc(be & lt)] = u[k];
                    else if (u[k] >= 0) a.out[ld + __popc(bl & lt)] = u[k];
                    ed += __popc(be);
                    ld += __popc(bl);
                }
            } else {
#pragma unroll
                for (int k = 0; k < W; k++)
                    if (u[k] >= 0) { cnt += early[k]; diff += mix_pair(v, u[k]) - mix_pair(u[k], v); }
            }
        }
        if (!FILL) {
            cnt = warp_sum(cnt);
            if (lane == 0 && cnt) atomicAdd(&s_cnt[0], cnt);
        }
        __syncthreads();
        if (!FILL && threadIdx.x == 0) a.early[v] = s_cnt[0];
        __syncthreads();
    }
    for (long long tile = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; tile * 32 < a.n;
         tile += ((long long)gridDim.x * blockDim.x) >> 5) {
        const long long v = tile * 32 + lane;
        ull b = 0;
        unsigned ds = 0;
        bool hub = false;
        if (v < a.n) {
            b = a.idx[v];
            const ull deg = a.idx[v + 1] - b;
            hub = deg > HUB_MIN;
            ds = hub ? 0u : (unsigned)deg;
        }
        const unsigned nz = __ballot_sync(FULL, ds != 0);
        unsigned cnt = 0;
        if (nz) {
            const unsigned incl = warp_incl_scan(ds, lane);
            const unsigned tot = __shfl_sync(FULL, incl, 31), ex = incl - ds;
            const int rank = __popc(nz & lt);
            if (ds) {
                s_base[wib][rank] = b; s_ex[wib][rank] = ex; s_ph[wib][rank] = a.phase[v]; s_v[wib][rank] = (int)v;
                if (FILL) { s_e[wib][rank] = a.e_dst[v]; s_l[wib][rank] = a.l_dst[v]; }
            }
            __syncwarp();
            for (unsigned j0 = 0; j0 < tot; j0 += 32 * W) {
                int u[W], own[W];
                unsigned starts[W];
                bool early[W];
#pragma unroll
                for (int k = 0; k < W; k++) {
                    const unsigned wb = j0 + 32 * k, j = wb + lane;
                    starts[k] = __reduce_or_sync(FULL, (ds && ex >= wb && ex - wb < 32) ? 1u << (ex - wb) : 0u);
                    own[k] = __popc(__ballot_sync(FULL, ds && ex <= wb)) - 1 + __popc(starts[k] & le & ~1u);
                    u[k] = plain_entry(a, j < tot ? s_base[wib][own[k]] + (j - s_ex[wib][own[k]]) : 0, j < tot);
                }
#pragma unroll
                for (int k = 0; k < W; k++) early[k] = u[k] >= 0 && a.phase[u[k]] < s_ph[wib][own[k]];
#pragma unroll
                for (int k = 0; k < W; k++) {
                    const unsigned wb = j0 + 32 * k;
                    if (wb >= tot) break;
                    const unsigned be = __ballot_sync(FULL, early[k]), bl = __ballot_sync(FULL, u[k] >= 0) & ~be;
                    // this lane's list within the window, as a mask of window lanes
                    const unsigned lo = ex > wb ? ex - wb : 0u, hi = ex + ds > wb ? ex + ds - wb : 0u;
                    const unsigned mine = lo < 32 && hi > lo ? (hi >= 32 ? FULL : (1u << hi) - 1u) & ~((1u << lo) - 1u) : 0u;
                    if (FILL) {
                        const int first = 31 - __clz((starts[k] & le) | 1u);
                        const unsigned before = lt & ~((1u << first) - 1u);
                        if (early[k]) a.out[s_e[wib][own[k]] + __popc(be & before)] = u[k];
                        else if (u[k] >= 0) a.out[s_l[wib][own[k]] + __popc(bl & before)] = u[k];
                        __syncwarp();
                        if (ds && mine) { s_e[wib][rank] += __popc(be & mine); s_l[wib][rank] += __popc(bl & mine); }
                        __syncwarp();
                    } else {
                        cnt += __popc(be & mine);
                        if (u[k] >= 0) { const int w = s_v[wib][own[k]]; diff += mix_pair(w, u[k]) - mix_pair(u[k], w); }
                    }
                }
            }
            __syncwarp();
        }
        if (!FILL && v < a.n && !hub) a.early[v] = cnt;
    }
    if (!FILL) {
        diff = warp_sum(diff);
        if (lane == 0 && diff) atomicAdd(a.asym, diff);
    }
}

// ------------------------------------------------------------------ running

template <typename V> struct GatherP;
template <> struct GatherP<float> {
    const int* adj;
    const float* P;
    struct Key { int u = -1; };
    __device__ __forceinline__ Key key(ull e) const { Key k; k.u = ld_edge(adj + e); return k; }
    __device__ __forceinline__ float value(const Key& k) const { return k.u >= 0 ? P[k.u] : 0.f; }
};
template <> struct GatherP<F3> {
    const int* adj;
    const float4* P;
    struct Key { int u = -1; };
    __device__ __forceinline__ Key key(ull e) const { Key k; k.u = ld_edge(adj + e); return k; }
    __device__ __forceinline__ F3 value(const Key& k) const {
        if (k.u < 0) return F3(0);
        const float4 p = P[k.u];
        return F3(p.x, p.y, p.z);
    }
};

// Take vertex v whose residual is now rv (nobody adds to it in this phase):
// residual, value and pushed weight, or a weight of 0.
template <int L>
__device__ __forceinline__ void take_here(typename Lane<L>::T* x, typename Lane<L>::T* r, typename Lane<L>::T* P, int v,
                                          typename Lane<L>::T rv, ull deg, bool allowed, bool changed,
                                          const DevMeasures& M, ull& pushed, ull& lanes, ull& taken) {
    typename Lane<L>::T p{};
    if constexpr (L == 1) {
        if (allowed && fabsf(rv) > M.eps[0]) {
            x[v] += rv;
            p = weight(rv, deg, M, 0);
            rv = 0.f;
            changed = true;
        }
    } else {
        float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
        if (allowed) {
            if (fabsf(rv.x) > M.eps[0]) { d.x = rv.x; rv.x = 0.f; }
            if (M.nm > 1 && fabsf(rv.y) > M.eps[1]) { d.y = rv.y; rv.y = 0.f; }
            if (M.nm > 2 && fabsf(rv.z) > M.eps[2]) { d.z = rv.z; rv.z = 0.f; }
        }
        if (nonzero(d)) {
            float4 xv = x[v];
            xv.x += d.x; xv.y += d.y; xv.z += d.z;
            x[v] = xv;
            p = make_float4(weight(d.x, deg, M, 0), weight(d.y, deg, M, 1), weight(d.z, deg, M, 2), 0.f);
            changed = true;
        }
    }
    if (changed) r[v] = rv;
    if (deg) P[v] = p;
    if (nonzero(p) && deg) {
        const unsigned nz = measures_in(p);
        pushed += deg;
        lanes += deg * nz;
        taken += nz;
    }
}

// One swept pass as gathers, per the table k_passes left (HOST: per that of a host-driven push).
static constexpr int GT = 1024, GW = GT / 32, G_PER_SM = 1;   // threads and warps per block, blocks per SM
struct SweepArgs {
    SolveArgs a;
    SweepLists g;
};
template <int L, bool HOST>
__global__ void __launch_bounds__(GT, G_PER_SM) k_sweep_gather(const __grid_constant__ SweepArgs args) {
    const SolveArgs& a = args.a;
    const SweepLists& g = args.g;
    typedef typename Lane<L>::T T;
    typedef typename GSum<L>::T S;
    __shared__ ull s_tot[3][GW];
    __shared__ unsigned s_next;
    Ctrl* ctrl = a.push.ctrl;
    if (!HOST && (ctrl->done || !ctrl->sweep_pass)) return;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nc = a.push.nc;
    unsigned epoch = 0;
    clear_tables(a, GT);
    T* x = reinterpret_cast<T*>(a.push.x);
    T* r = reinterpret_cast<T*>(a.push.r);
    T* P = reinterpret_cast<T*>(g.P);
    const GatherP<S> f{g.adj, P};
    const ull* idx = a.push.idx;
    ull pushed = 0, lanes = 0, taken = 0;
    if (threadIdx.x == 0) s_next = 0;
    __syncthreads();
    auto claim = [&]() -> ull {
        unsigned k = 0;
        if (lane == 0) k = atomicAdd(&s_next, 1u);
        return (ull)__shfl_sync(FULL, k, 0) * gridDim.x + blockIdx.x;
    };
    auto phase_end = [&]() -> bool {
        __syncthreads();
        if (threadIdx.x == 0) s_next = 0;
        return grid_sync(&ctrl->sweep_bar, epoch) || gave_up(a);
    };
    // segments [s0, s1) two at a time, `done(segment, sum)` side by side in lanes 0 and 1 (a take is a
    // chain of some seven accesses); returns the warp's first claim past their pairs
    auto segments = [&](const auto* seg, unsigned s0, unsigned s1, auto&& done) -> ull {
        typedef typename std::decay<decltype(*seg)>::type R;
        const ull npairs = (s1 - s0 + 1) / 2;
        ull i = claim();
        R g0{}, g1{};
        if (i < npairs) g0 = seg[s0 + 2 * i];
        if (s0 + 2 * i + 1 < s1) g1 = seg[s0 + 2 * i + 1];
        while (i < npairs) {
            const ull next = claim();
            R n0{}, n1{};
            if (next < npairs) n0 = seg[s0 + 2 * next];
            if (s0 + 2 * next + 1 < s1) n1 = seg[s0 + 2 * next + 1];
            S a0, a1;
            warp_segment_sums<S>(as_seg(g0), as_seg(g1), f, lane, a0, a1);
            const S b1 = shfl(a1, 0);
            if (lane == 0 || (lane == 1 && s0 + 2 * i + 1 < s1)) done(lane ? g1 : g0, lane ? b1 : a0);
            i = next; g0 = n0; g1 = n1;
        }
        return i;
    };
    // tiles of 32 of the listed vertices [t0, t1), the warp's first claim being `i`, `before` claims taken by
    // segments and other tiles; done(number in the list, vertex, sum); returns the warp's first claim past
    // them. The next tile's records are loaded ahead.
    auto tiles = [&](auto tiny, ull i, ull& before, unsigned t0, unsigned t1, const ListedParts& l, auto&& done) -> ull {
        const ull ntiles = ((ull)(t1 - t0) + 31) / 32;
        int v = -1, nv = -1;
        unsigned b = 0, e = 0, nb = 0, ne = 0;
        auto load = [&](ull t, int& lv, unsigned& lb, unsigned& le) {
            const ull j = t0 + t * 32 + lane;
            lv = -1; lb = 0; le = 0;
            if (t < ntiles && j < t1) { lv = l.v[j]; lb = l.off[j]; le = l.off[j + 1]; }
        };
        ull t = i - before;
        load(t, v, b, e);
        while (t < ntiles) {
            const ull nt = claim() - before;
            load(nt, nv, nb, ne);
            T rv{};
            if (v >= 0) rv = r[v];   // (nobody else adds to it in this phase)
            const S sum = warp_list_sums<S, decltype(tiny)::value>(b, e - b, f, lane);
            if (v >= 0) done((unsigned)(t0 + t * 32 + lane), v, rv, sum);
            t = nt; v = nv; b = nb; e = ne;
        }
        t += before;
        before += ntiles;
        return t;
    };
    constexpr std::true_type TINY{};
    constexpr std::false_type SHORT{};
    for (int c = 0; c < nc; c++) {
        const uint8_t ty = a.push.wt_type[c];
        auto allowed = [&](int v) { return ty == WT_RANGE || (ty == WT_LIST && bit_of(a.snap.bitmap, v)); };
        // hub vertices: the warp that adds a vertex's last segment takes it
        const unsigned h0 = g.hub_at[c], h1 = g.hub_at[c + 1];
        if (h1 > h0) {
            segments(g.e_hub, h0, h1, [&](const HubPart& sg, const S& sum) {
                const int v = (int)sg.row;
                const ull deg = idx[v + 1] - idx[v];
                const unsigned nseg = sg.len_nseg >> 10;
                if (nseg == 1) {
                    take_here<L>(x, r, P, v, add_sum(r[v], sum), deg, allowed(v), nonzero(sum), a.push.M, pushed, lanes,
                                 taken);
                    return;
                }
                red_sum(r, (unsigned)v, sum);
                __threadfence();
                if (atomicAdd(&g.hub_done[sg.first], 1u) + 1 < nseg) return;
                g.hub_done[sg.first] = 0;
                __threadfence();
                take_here<L>(x, r, P, v, __ldcg(r + v), deg, allowed(v), false, a.push.M, pushed, lanes, taken);
            });
            if (!phase_end()) return;
        }
        for (int q = g.q_of[c]; q < g.q_of[c + 1]; q++) {
            const unsigned m0 = g.mid_at[q], m1 = g.mid_at[q + 1];
            ull i = segments(g.e_mid, m0, m1, [&](const ListSeg& sg, const S& sum) {
                const int v = (int)sg.row;
                take_here<L>(x, r, P, v, add_sum(r[v], sum), idx[v + 1] - idx[v], allowed(v), nonzero(sum), a.push.M,
                             pushed, lanes, taken);
            });
            ull before = (m1 - m0 + 1) / 2;
            auto listed = [&](const ListedParts& l) {
                return [&](unsigned j, int v, const T& rv, const S& sum) {
                    take_here<L>(x, r, P, v, add_sum(rv, sum), l.deg[j], allowed(v), nonzero(sum), a.push.M, pushed, lanes,
                                 taken);
                };
            };
            i = tiles(SHORT, i, before, g.es_at[q], g.es_at[q + 1], g.e_short, listed(g.e_short));
            tiles(TINY, i, before, g.et_at[q], g.et_at[q + 1], g.e_tiny, listed(g.e_tiny));
            if (!phase_end()) return;
        }
    }
    // the late parts of every list
    const unsigned nl = g.totals[C_L_SEG];
    ull i = segments(g.l_seg, 0, nl, [&](const ListSeg& sg, const S& sum) { red_sum(r, sg.row, sum); });
    ull before = (nl + 1) / 2;
    auto rest = [&](unsigned, int v, const T& rv, const S& sum) { if (nonzero(sum)) r[v] = add_sum(rv, sum); };
    i = tiles(SHORT, i, before, 0, g.totals[C_LS_V], g.l_short, rest);
    tiles(TINY, i, before, 0, g.totals[C_LT_V], g.l_tiny, rest);
    // a vertex without entries is pending until it is taken, and nobody adds to it
    for (long long w = blockIdx.x * (long long)GT + threadIdx.x; w < a.snap.words; w += (long long)gridDim.x * GT) {
        uint32_t bits = a.snap.bitmap[w] & g.alone[w];
        while (bits) {
            const int v = (int)w * 32 + __ffs(bits) - 1;
            bits &= bits - 1;
            if (HOST && a.push.wt_type[chunk_of(v, a.push.cv0, nc)] == WT_NONE) continue;   // not asked for
            take_here<L>(x, r, P, v, r[v], 0, true, false, a.push.M, pushed, lanes, taken);
        }
    }
    pushed = warp_sum(pushed);
    lanes = warp_sum(lanes);
    taken = warp_sum(taken);
    if (lane == 0) { s_tot[0][wib] = pushed; s_tot[1][wib] = lanes; s_tot[2][wib] = taken; }
    __syncthreads();
    if (wib < 3) {
        const ull s = warp_sum(lane < GW ? s_tot[wib][lane] : 0ull);
        if (lane == 0 && s) atomicAdd(wib == 0 ? &ctrl->pushed : wib == 1 ? &ctrl->lanes : &ctrl->taken, s);
    }
}

}  // namespace excent
