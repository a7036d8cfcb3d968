// passes.cuh -- the passes of a device solve inside one cooperative launch
// (included by engine.cu). k_passes runs snapshot, plan and push of pass
// after pass with a grid barrier between the phases, until nothing is pending
// or a pass is due that goes chunk by chunk; k_sweep runs that one.
//
// Why: a pass of the graph loop was six to eight nodes of its own (62 us a
// pass on 14k entries, 83 us on 956k), of which the work is a few us; a grid
// barrier costs 1.3 us. The order of a pass is the same: its long lists are
// taken, then scattered, then the short lists, and a vertex is taken with
// everything that earlier phases delivered.
//
// Takes of up to `wave` items are separated from their scatter by a barrier.
// They were simultaneous before, too (a wave of resident warps takes all its
// items within a microsecond, long before the first list is scattered), and
// what is taken is then free to be laid out for the scatter: lists of at most
// WAVE_LONG entries compacted, 32 to a tile, longer ones as segments, one warp
// each, so that no warp has much more than its share. More items are claimed
// in batches in table order and scattered as they are taken, as by k_push.
#pragma once

namespace excent {

// Threads per block, one block per SM: 1024 leave 64 registers a thread and spill in the snapshot
// (sample of 2000 vertices: 1.34 ms a solve, 1.23 with 768), 512 are too few for the large passes
// (R-MAT 24 PageRank: 47.7, 48.0 and 49.7 ms with 1024, 768 and 512).
static constexpr int PT = 768;
static constexpr int PW = PT / 32;
static constexpr unsigned WAVE_LONG = 32;     // longer lists of a wave are scattered as segments
static constexpr int PLAN_LOCAL = PT;         // up to this many chunks every block plans for itself

struct SolveArgs {
    SnapArgs snap;
    PushArgs push;
    ull* cnt2;             // second demand table: snapshots alternate between snap.cnt and this one
    int snap_group;        // bitmap words per warp step of the snapshot
    const uint8_t* cmode;
    double list_frac;
    int max_passes;
    int sweep;             // this engine goes chunk by chunk in passes of at least sweep_min entries
    ull sweep_min;
    PassRec* log;
    int log_cap;
    int order;             // where the long lists go: 0 in table order, 1 first, 2 last, 3 first in each launch
    int wave;              // items taken together before they are scattered
    unsigned seg;          // entries per segment
    HubSeg* small;         // taken lists of at most WAVE_LONG entries (wave records)
    int standalone;        // one push of the host-driven loop: its table and counts stay as they are
    int use_cond;          // in a loop with the sweep kernel: its condition, and the barriers cleared in turn
    cudaGraphConditionalHandle again;
};

// Take vertex v, whose residual is rv, in a phase in which nobody adds to
// residuals: the take of device.cuh without its exchanges.
__device__ __forceinline__ float take_alone(float* x, float* r, int v, float rv, ull deg, const DevMeasures& M) {
    if (!(fabsf(rv) > M.eps[0])) return 0.f;
    r[v] = 0.f;
    x[v] += rv;
    return weight(rv, deg, M, 0);
}
__device__ __forceinline__ float4 take_alone(float4* x, float4* r, int v, float4 rv, ull deg, const DevMeasures& M) {
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
    if (fabsf(rv.x) > M.eps[0]) { d.x = rv.x; rv.x = 0.f; }
    if (M.nm > 1 && fabsf(rv.y) > M.eps[1]) { d.y = rv.y; rv.y = 0.f; }
    if (M.nm > 2 && fabsf(rv.z) > M.eps[2]) { d.z = rv.z; rv.z = 0.f; }
    if (!nonzero(d)) return d;
    r[v] = rv;
    float4 xv = x[v];
    xv.x += d.x; xv.y += d.y; xv.z += d.z;
    x[v] = xv;
    return make_float4(weight(d.x, deg, M, 0), weight(d.y, deg, M, 1), weight(d.z, deg, M, 2), 0.f);
}

// Take one hub vertex and queue its segments: called by one lane from the
// snapshot, before the barrier that follows it (nobody adds to residuals
// there). The measures its weight carries. Out of line: it would be unrolled
// with the snapshot's loads and take their registers.
template <int L>
__device__ __noinline__ unsigned take_hub(const SolveArgs& a, WaveCount* w, int v, typename Lane<L>::T rv, unsigned deg) {
    typedef typename Lane<L>::T T;
    const T p = take_alone(reinterpret_cast<T*>(a.push.x), reinterpret_cast<T*>(a.push.r), v, rv, deg, a.push.M);
    if (!nonzero(p)) return 0;
    const unsigned nseg = (deg + a.seg - 1) / a.seg;
    const ull at = atomicAdd(&w->big, nseg);
    if (at + nseg > a.push.hub_cap) { atomicExch(&a.push.ctrl->err, 1); return 0; }
    HubSeg h;
    h.pad = 0;
    if constexpr (L == 1) h.p = make_float4(p, 0.f, 0.f, 0.f); else h.p = p;
    const int* nb = list_at(a.push, a.push.idx[v]);
    for (unsigned k = 0; k < nseg; k++) {
        h.nb = nb + (ull)k * a.seg;
        h.len = min(a.seg, deg - k * a.seg);
        a.push.hubq[at + k] = h;
    }
    return measures_in(p);
}

// Sum of (a, b) of every warp before this one in the block, and of the block.
__device__ __forceinline__ void block_offsets(unsigned a, unsigned b, unsigned (&s)[2][PW], int wib, int lane,
                                              unsigned& oa, unsigned& ob, unsigned& ta, unsigned& tb) {
    if (lane == 0) { s[0][wib] = a; s[1][wib] = b; }
    __syncthreads();
    const unsigned va = lane < PW ? s[0][lane] : 0u, vb = lane < PW ? s[1][lane] : 0u;
    const unsigned ia = warp_incl_scan(va, lane), ib = warp_incl_scan(vb, lane);
    oa = __shfl_sync(FULL, ia - va, wib);
    ob = __shfl_sync(FULL, ib - vb, wib);
    ta = __shfl_sync(FULL, ia, 31);
    tb = __shfl_sync(FULL, ib, 31);
}

// A wait between blocks gave up: the solve ends with an error.
__device__ __noinline__ bool gave_up(const SolveArgs& a) {
    if (threadIdx.x == 0) {
        atomicExch(&a.push.ctrl->err, 4);
        a.push.ctrl->done = 1;
        if (blockIdx.x == 0 && a.use_cond) cudaGraphSetConditional(a.again, 0u);
    }
    return false;
}

// Scratch of one block, and the counters it adds up over the kernel.
template <int L> struct PassShared {
    typedef typename Lane<L>::T T;
    const int* nb[PW][32];
    unsigned ex[PW][32];
    T p[PW][32];
    unsigned cnt[2][PW];
    ull base[2];
    double rs[4][PW];
    ull tot[4][PW];
    unsigned next;
};

template <int L> struct Passes {
    typedef typename Lane<L>::T T;
    const SolveArgs& a;
    PassShared<L>& s;
    T* x;
    T* r;
    T* hacc;
    const unsigned* prefix;    // the pass's work table
    const uint8_t* type;
    int lane, wib;
    unsigned epoch;
    int phase;                 // take phases so far (ring of wave counters)
    ull pushed, hpushed, lanes, taken;

    __device__ __forceinline__ Passes(const SolveArgs& a_, PassShared<L>& s_, T* hacc_, GridBar* bar_)
        : a(a_), s(s_), x(reinterpret_cast<T*>(a_.push.x)), r(reinterpret_cast<T*>(a_.push.r)), hacc(hacc_),
          prefix(a_.push.wt_prefix), type(a_.push.wt_type), lane(threadIdx.x & 31), wib(threadIdx.x >> 5), epoch(0),
          phase(0), pushed(0), hpushed(0), lanes(0), taken(0), bar(bar_) {}

    GridBar* bar;
    __device__ __forceinline__ bool sync() { return grid_sync(bar, epoch) || gave_up(a); }
    __device__ __forceinline__ WaveCount& counts(int ph) const { return a.push.ctrl->wave[ph % 3]; }

    // Table item t: its vertex, in a chunk's list or range.
    __device__ __forceinline__ int item_vertex(long long t, int chunk) const {
        int lo = chunk;
        if (chunk < 0) {
            int hi = a.push.nc - 1;
            lo = 0;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if ((long long)prefix[mid] <= t) lo = mid; else hi = mid - 1;
            }
        }
        const unsigned i = (unsigned)(t - prefix[lo]);
        return type[lo] == WT_LIST ? a.push.list[a.push.cv0[lo] + i] : a.push.cv0[lo] + (int)i;
    }

    __device__ __forceinline__ void count(const T& p, ull deg, ull b) {
        const unsigned nz = measures_in(p);
        pushed += deg;
        lanes += deg * nz;
        taken += nz;
        if (a.push.hcache && b >= a.push.cache_edges) hpushed += deg;
    }

    // Take phase of up to `wave` items: item i of [0, items) is vertex vert(i)
    // (< 0: none). Short lists are appended to a.small, the others to the
    // segment queue, with one reservation of each per block and step. LISTS
    // limits the takes as in k_push.
    template <typename V>
    __device__ __forceinline__ void take_wave(long long items, int which, const V& vert) {
        WaveCount& w = counts(phase);
        if (blockIdx.x == 0 && threadIdx.x == 0) { WaveCount& n = counts(phase + 1); n.small = 0; n.big = 0; n.claim = 0; }
        const long long step = (long long)gridDim.x * PT;
        for (long long i0 = (long long)blockIdx.x * PT; i0 < items; i0 += step) {
            const long long i = i0 + threadIdx.x;
            const int v = i < items ? vert(i) : -1;
            T p{};
            ull b = 0, deg = 0;
            if (v >= 0) {
                b = a.push.idx[v];
                deg = a.push.idx[v + 1] - b;
                if (!(which == LISTS_SHORT && deg > HUB_MIN) && !(which == LISTS_LONG && deg <= HUB_MIN))
                    p = take_alone(x, r, v, r[v], deg, a.push.M);
            }
            const bool act = nonzero(p) && deg > 0;
            if (act) count(p, deg, b);
            const bool sm = act && deg <= WAVE_LONG;
            const unsigned nseg = act && !sm ? (unsigned)((deg + a.seg - 1) / a.seg) : 0u;
            const unsigned sb = __ballot_sync(FULL, sm);
            const unsigned incl = warp_incl_scan(nseg, lane);
            unsigned os, ob, ts, tb;
            block_offsets(__popc(sb), __shfl_sync(FULL, incl, 31), s.cnt, wib, lane, os, ob, ts, tb);
            if (threadIdx.x == 0) {
                s.base[0] = ts ? atomicAdd(&w.small, ts) : 0;
                s.base[1] = tb ? atomicAdd(&w.big, tb) : 0;
            }
            __syncthreads();
            HubSeg h;
            h.pad = 0;
            if constexpr (L == 1) h.p = make_float4(p, 0.f, 0.f, 0.f); else h.p = p;
            if (sm) {
                h.nb = list_at(a.push, b);
                h.len = (unsigned)deg;
                a.small[s.base[0] + os + __popc(sb & ((1u << lane) - 1u))] = h;
            } else if (nseg) {
                const ull at = s.base[1] + ob + (incl - nseg);
                if (at + nseg <= a.push.hub_cap) {
                    const int* nb = list_at(a.push, b);
                    for (unsigned k = 0; k < nseg; k++) {
                        h.nb = nb + (ull)k * a.seg;
                        h.len = (unsigned)min((ull)a.seg, deg - (ull)k * a.seg);
                        a.push.hubq[at + k] = h;
                    }
                } else {
                    atomicExch(&a.push.ctrl->err, 1);
                }
            }
            __syncthreads();   // s.base and s.cnt are used again
        }
        if (threadIdx.x == 0) s.next = 0;
    }

    // One tile of up to 32 short lists, edge-balanced (as in k_push).
    __device__ __forceinline__ void scatter_tile(const int* nb, unsigned ds, const T& p) {
        const unsigned nz = __ballot_sync(FULL, ds != 0);
        if (!nz) return;
        const unsigned incl = warp_incl_scan(ds, lane);
        const unsigned tot = __shfl_sync(FULL, incl, 31);
        const unsigned ex = incl - ds;
        if (ds) {
            const int rank = __popc(nz & ((1u << lane) - 1u));
            s.nb[wib][rank] = nb; s.ex[wib][rank] = ex; s.p[wib][rank] = p;
        }
        __syncwarp();
        const unsigned le = lane == 31 ? FULL : (2u << lane) - 1u;
        for (unsigned j0 = 0; j0 < tot; j0 += 32 * UNROLL) {
            int u[UNROLL];
            int own[UNROLL];
#pragma unroll
            for (int k = 0; k < UNROLL; k++) {
                // owner of entry wb + lane: the last nonempty list starting at or before it
                const unsigned wb = j0 + 32 * k, j = wb + lane;
                const unsigned starts =
                    __reduce_or_sync(FULL, (ds && ex >= wb && ex - wb < 32) ? 1u << (ex - wb) : 0u);
                const int o = __popc(__ballot_sync(FULL, ds && ex <= wb)) - 1 + __popc(starts & le & ~1u);
                own[k] = j < tot ? o : -1;
                u[k] = j < tot ? ld_edge(s.nb[wib][o] + (j - s.ex[wib][o])) : 0;
            }
#pragma unroll
            for (int k = 0; k < UNROLL; k++)
                if (own[k] >= 0) scatter_one(r, u[k], s.p[wib][own[k]], hacc);
        }
        __syncwarp();
    }

    // Scatter what the last take phase queued: segments, one warp each, then
    // tiles of short lists; blocks share them interleaved, a block's warps claim.
    __device__ __forceinline__ void scatter_wave(ull nbig, unsigned nsmall) {
        // 32 lists to a tile, down to 8 while there are warps for them
        const unsigned per_tile = min(32u, max(8u, nsmall / (gridDim.x * PW)));
        const ull ntiles = ((ull)nsmall + per_tile - 1) / per_tile;
        for (;;) {
            unsigned k = 0;
            if (lane == 0) k = atomicAdd(&s.next, 1u);
            const ull i = (ull)__shfl_sync(FULL, k, 0) * gridDim.x + blockIdx.x;
            if (i < nbig) {
                const HubSeg* h = a.push.hubq + i;
                const float4 p4 = h->p;
                T p;
                if constexpr (L == 1) p = p4.x; else p = p4;
                warp_scatter(r, h->nb, h->len, p, lane, hacc);
            } else if (i - nbig < ntiles) {
                const ull j = (i - nbig) * per_tile + lane;
                const int* nb = nullptr;
                unsigned ds = 0;
                T p{};
                if (lane < per_tile && j < nsmall) {
                    const HubSeg h = a.small[j];
                    nb = h.nb;
                    ds = h.len;
                    if constexpr (L == 1) p = h.p.x; else p = h.p;
                }
                scatter_tile(nb, ds, p);
            } else {
                break;
            }
        }
        flush();
    }

    // The hub-target sums of this phase, and the slots back to zero.
    __device__ __forceinline__ void flush() {
        if (!hacc) return;
        __syncthreads();
        for (int i = threadIdx.x; i < a.push.hub_k; i += PT) {
            const T v = hacc[i];
            if (nonzero(v)) { red_add(r, a.push.hub_id[i], v); hacc[i] = T{}; }
        }
    }

    // Take `items` items together, then scatter them. False: a wait gave up.
    template <typename V>
    __device__ __forceinline__ bool push_wave(long long items, int which, const V& vert) {
        take_wave(items, which, vert);
        if (!sync()) return false;
        const ull nbig = min((ull)counts(phase).big, a.push.hub_cap);
        const unsigned nsmall = counts(phase).small;
        phase++;
        if (!nbig && !nsmall) return true;
        scatter_wave(nbig, nsmall);
        return sync();
    }

    // Table items [first, total) of one chunk (-1: all): one wave, or claimed
    // in batches and scattered as they are taken, long lists (LISTS_ALL)
    // queued and scattered last.
    __device__ __forceinline__ bool push_table(long long first, long long total, int chunk, int which) {
        const long long items = total - first;
        if (items <= 0) return true;
        if (items <= a.wave) return push_wave(items, which, [&](long long i) { return item_vertex(first + i, chunk); });
        WaveCount& w = counts(phase);
        if (blockIdx.x == 0 && threadIdx.x == 0) { WaveCount& n = counts(phase + 1); n.small = 0; n.big = 0; n.claim = 0; }
        const long long ntiles = (items + 31) / 32, nwarps = (long long)gridDim.x * PW;
        // as many tiles are in flight as the wave has warps: when it has twice as many as run here, each
        // takes its next tile before it scatters the one before (without that PageRank with host lists, 1M vertices, moved 4.2 times as far
        // from where a launch of all those warps takes it as that moves between runs)
        const unsigned ahead = a.wave >= 64 * nwarps ? 2 : 1;
        const long long per_claim = a.push.claim_tiles > 0
            ? a.push.claim_tiles : max(1ll, min((long long)TILE_BATCH, ntiles / (4 * nwarps * ahead)));
        auto take_tile = [&](long long tile, const int*& nb, unsigned& ds, T& p) {
            const long long t = tile * 32 + lane;
            p = T{};
            nb = nullptr;
            ull b = 0, deg = 0;
            if (tile < ntiles && t < items) {
                const int v = item_vertex(first + t, chunk);
                b = a.push.idx[v];
                deg = a.push.idx[v + 1] - b;
                if (!(which == LISTS_SHORT && deg > HUB_MIN)) p = take(x, r, v, deg, a.push.M);
            }
            const bool act = nonzero(p) && deg > 0;
            if (act) { count(p, deg, b); nb = list_at(a.push, b); }
            const unsigned nseg = act && deg > HUB_MIN ? (unsigned)((deg + a.seg - 1) / a.seg) : 0u;
            const unsigned incl = warp_incl_scan(nseg, lane);
            const unsigned tot = __shfl_sync(FULL, incl, 31);
            if (tot) {
                ull at = 0;
                if (lane == 0) at = atomicAdd(&w.big, tot);
                at = __shfl_sync(FULL, at, 0) + (incl - nseg);
                if (at + nseg <= a.push.hub_cap) {
                    HubSeg h;
                    h.pad = 0;
                    if constexpr (L == 1) h.p = make_float4(p, 0.f, 0.f, 0.f); else h.p = p;
                    for (unsigned k = 0; k < nseg; k++) {
                        h.nb = nb + (ull)k * a.seg;
                        h.len = (unsigned)min((ull)a.seg, deg - (ull)k * a.seg);
                        a.push.hubq[at + k] = h;
                    }
                } else if (nseg) {
                    atomicExch(&a.push.ctrl->err, 1);
                }
            }
            ds = act && !nseg ? (unsigned)deg : 0u;
        };
        long long tile = 0, end = 0;
        T p0{};
        const int* nb0 = nullptr;
        unsigned ds0 = 0;
        for (;;) {
            if (tile == end) {
                unsigned c = 0;
                if (lane == 0) c = atomicAdd(&w.claim, 1u);
                tile = min((long long)__shfl_sync(FULL, c, 0) * per_claim, ntiles);
                end = min(tile + per_claim, ntiles);
            }
            const bool more = tile < ntiles;
            T p1;
            const int* nb1;
            unsigned ds1;
            take_tile(tile, nb1, ds1, p1);
            if (ahead == 2) scatter_tile(nb0, ds0, p0);   // the tile before
            else scatter_tile(nb1, ds1, p1);
            if (!more) break;
            p0 = p1; nb0 = nb1; ds0 = ds1;
            tile++;
        }
        flush();
        if (threadIdx.x == 0) s.next = 0;
        if (!sync()) return false;
        const ull nbig = min((ull)counts(phase).big, a.push.hub_cap);
        phase++;
        if (!nbig) return true;
        scatter_wave(nbig, 0);
        return sync();
    }

    // Scatter what the snapshot took (the phase after its barrier).
    __device__ __forceinline__ bool push_taken_hubs() {
        const ull nbig = min((ull)counts(phase).big, a.push.hub_cap);
        phase++;
        if (!nbig) return true;
        scatter_wave(nbig, 0);
        return sync();
    }

    // The long lists of hub vertices [h0, h1), all taken before any is scattered. A host-driven push
    // (HOST: it may be one) leaves the vertices of other chunks than it was asked for alone: their lists
    // may not be loaded.
    template <bool HOST>
    __device__ __forceinline__ bool push_hubs(long long h0, long long h1, bool listed) {
        if (h1 <= h0) return true;
        return push_wave(h1 - h0, LISTS_LONG, [&](long long i) {
            const int v = a.push.hubv[h0 + i];
            if (HOST && a.standalone && type[chunk_of(v, a.push.cv0, a.push.nc)] == WT_NONE) return -1;
            return listed && !bit_of(a.snap.bitmap, v) ? -1 : v;
        });
    }
    __device__ __forceinline__ long long hub_bound(int v) const {   // hub vertices below v
        long long lo = 0, hi = (long long)*a.push.hubv_cnt;
        while (lo < hi) {
            const long long mid = (lo + hi) >> 1;
            if (a.push.hubv[mid] < v) lo = mid + 1; else hi = mid;
        }
        return lo;
    }

    // The counters of this kernel's takes so far, before the barrier that ends a pass.
    __device__ __forceinline__ void report() {
        pushed = warp_sum(pushed);
        lanes = warp_sum(lanes);
        taken = warp_sum(taken);
        hpushed = warp_sum(hpushed);
        if (lane == 0) { s.tot[0][wib] = pushed; s.tot[1][wib] = lanes; s.tot[2][wib] = taken; s.tot[3][wib] = hpushed; }
        __syncthreads();
        if (wib < 4) {
            const ull t = warp_sum(lane < PW ? s.tot[wib][lane] : 0ull);
            Ctrl* c = a.push.ctrl;
            if (lane == 0 && t) atomicAdd(wib == 0 ? &c->pushed : wib == 1 ? &c->lanes : wib == 2 ? &c->taken : &c->host_pushed, t);
        }
        pushed = lanes = taken = hpushed = 0;
    }
};

// Snapshot of the whole graph by all blocks; sums into acc. on_pending(v, residual, degree) for
// every pending vertex.
template <int L, typename F>
__device__ __forceinline__ void solve_snapshot(const SolveArgs& a, PassShared<L>& s, ull* cnt, SnapAcc* acc, double ev_corr,
                                               int lane, int wib, const F& on_pending) {
    const long long groups = (a.snap.words + a.snap_group - 1) / a.snap_group;
    const long long nwarps = (long long)gridDim.x * PW;
    // a contiguous run of groups per warp; with fewer groups than warps, neighbours on different SMs
    const long long per = (groups + nwarps - 1) / nwarps;
    const long long gw = per > 1 ? (long long)blockIdx.x * PW + wib : (long long)wib * gridDim.x + blockIdx.x;
    SnapSums q;
    snapshot_scan<L>(a.snap, cnt, a.snap_group, gw * per, (gw + 1) * per, ev_corr, q, lane, on_pending);
    q.rs0 = warp_sum(q.rs0); q.rs1 = warp_sum(q.rs1); q.rs2 = warp_sum(q.rs2); q.evd = warp_sum(q.evd);
    if (lane == 0) { s.rs[0][wib] = q.rs0; s.rs[1][wib] = q.rs1; s.rs[2][wib] = q.rs2; s.rs[3][wib] = q.evd; }
    __syncthreads();
    if (wib < 4) {
        const double t = warp_sum(lane < PW ? s.rs[wib][lane] : 0.0);
        if (lane == 0 && t != 0.0) atomicAdd(wib < 3 ? &acc->rsum[wib] : &acc->ev_dot, t);
    }
}

// The work table of a pass into prefix / type (src/excent.cu:639; see k_plan),
// by one block; the items of the whole table in every thread.
__device__ __forceinline__ unsigned solve_table(const SolveArgs& a, const ull* cnt, unsigned* prefix, uint8_t* type,
                                                unsigned (&scan)[PW], unsigned* s_lists, int lane, int wib) {
    const int nc = a.push.nc;
    unsigned carry = 0;
    if (threadIdx.x == 0) { prefix[0] = 0; s_lists[0] = 0; s_lists[1] = 0; }
    __syncthreads();
    for (int base = 0; base < nc; base += PT) {
        const int c = base + (int)threadIdx.x;
        unsigned items = 0;
        uint8_t ty = WT_NONE;
        if (c < nc && a.cmode[c] && cnt[2 * c] > 0) {
            const int v0 = a.push.cv0[c], v1 = c + 1 < nc ? a.push.cv0[c + 1] : a.snap.n;
            if (a.cmode[c] != 2 && (double)cnt[2 * c] < a.list_frac * (v1 - v0)) {
                ty = WT_LIST; items = (unsigned)cnt[2 * c]; atomicAdd(&s_lists[0], 1u);
            } else {
                ty = WT_RANGE; items = (unsigned)(v1 - v0); atomicAdd(&s_lists[1], 1u);
            }
        }
        const unsigned incl = warp_incl_scan(items, lane);
        if (lane == 31) scan[wib] = incl;
        __syncthreads();
        const unsigned w = warp_incl_scan(lane < PW ? scan[lane] : 0u, lane);
        const unsigned before = wib ? __shfl_sync(FULL, w, wib - 1) : 0u;
        const unsigned all = __shfl_sync(FULL, w, 31);
        if (c < nc) { type[c] = ty; prefix[c + 1] = carry + before + incl; }
        carry += all;
        __syncthreads();
    }
    return carry;
}

template <int L>
__global__ void __launch_bounds__(PT, 1) k_passes(const __grid_constant__ SolveArgs a) {
    typedef typename Lane<L>::T T;
    __shared__ PassShared<L> s;
    __shared__ unsigned s_prefix[PLAN_LOCAL + 1];
    __shared__ uint8_t s_type[PLAN_LOCAL];
    __shared__ unsigned s_scan[PW], s_lists[2];
    __shared__ ull s_sum[2];
    Ctrl* ctrl = a.push.ctrl;
    if (ctrl->done) return;
    Passes<L> P(a, s, hacc_init<T>(a.push.hub_k), &a.push.ctrl->bar);
    const int lane = P.lane, wib = P.wib, nc = a.push.nc;
    const bool first_block = blockIdx.x == 0, lead = first_block && threadIdx.x == 0;
    if (lead && a.sweep)   // what the sweep before left (otherwise the solve's reset cleared them)
        for (WaveCount& w : ctrl->wave) { w.small = 0; w.big = 0; w.claim = 0; }
    int pass = ctrl->pass;
    for (int k = 0;; k++, pass++) {
        ull* cnt = k & 1 ? a.cnt2 : a.snap.cnt;
        SnapAcc* acc = &ctrl->acc[k & 1];
        // without chunk-by-chunk passes the high-degree lists of this pass, which go first, can be taken
        // right here (6.5 us less a pass than a phase of their own)
        const bool take_hubs = a.order != 0 && a.order != 2 && !a.sweep && pass < a.max_passes;
        WaveCount* taken_here = &P.counts(P.phase);
        if (lead) {   // the next phase's counters: nobody uses them before the barrier
            WaveCount& w = P.counts(P.phase + 1);
            w.small = 0; w.big = 0; w.claim = 0;
        }
        solve_snapshot<L>(a, s, cnt, acc, a.snap.v1 ? ctrl->ev_corr : 0.0, lane, wib, [&](long long v, const T& rv, ull deg) {
            if (!take_hubs || deg <= HUB_MIN) return;
            const unsigned nz = take_hub<L>(a, taken_here, (int)v, rv, (unsigned)deg);
            if (!nz) return;
            P.pushed += deg;
            P.lanes += deg * nz;
            P.taken += nz;
            if (a.push.hcache && a.push.idx[v] >= a.push.cache_edges) P.hpushed += deg;
        });
        if (threadIdx.x == 0) s.next = 0;
        if (!P.sync()) return;
        // pending vertices and entries of the whole graph, by every block
        if (threadIdx.x < 2) s_sum[threadIdx.x] = 0;
        __syncthreads();
        ull lp = 0, ld = 0;
        for (int c = threadIdx.x; c < nc; c += PT) { lp += cnt[2 * c]; ld += cnt[2 * c + 1]; }
        lp = warp_sum(lp);
        ld = warp_sum(ld);
        if (lane == 0 && lp) { atomicAdd(&s_sum[0], lp); atomicAdd(&s_sum[1], ld); }
        __syncthreads();
        const ull pend = s_sum[0], dem = s_sum[1];
        const bool stop = pass >= a.max_passes || pend == 0;
        const bool sweep = a.sweep && !stop && dem >= a.sweep_min;
        // up to PLAN_LOCAL chunks every block makes the table in shared memory; the first block
        // makes the others' and a sweep's in global memory
        const bool local = nc <= PLAN_LOCAL && !sweep;
        unsigned* prefix = local ? s_prefix : const_cast<unsigned*>(a.push.wt_prefix);
        uint8_t* type = local ? s_type : const_cast<uint8_t*>(a.push.wt_type);
        P.prefix = prefix;
        P.type = type;
        if (!stop && (local || first_block)) solve_table(a, cnt, prefix, type, s_scan, s_lists, lane, wib);
        if (lead) {
            if (!stop && pass < a.log_cap) {
                PassRec& R = a.log[pass];
                R.pending = pend; R.demand = dem; R.hot_pending = 0; R.pushed_before = ctrl->pushed;
                R.lanes_before = ctrl->lanes; R.taken_before = ctrl->taken;
                for (int m = 0; m < MAXM; m++) R.rsum[m] = acc->rsum[m];
                R.n_list = (int)s_lists[0]; R.n_range = (int)s_lists[1];
            }
            for (int m = 0; m < MAXM; m++) ctrl->rsum[m] = acc->rsum[m];
            ctrl->ev_corr = acc->ev_dot;
            ctrl->sweep_pass = sweep ? 1 : 0;
            if (sweep) ctrl->sweeps++;
            if (stop) ctrl->done = 1; else ctrl->pass = pass + 1;
            ctrl->acc[(k & 1) ^ 1] = SnapAcc{};
            if (a.use_cond) {
                cudaGraphSetConditional(a.again, stop ? 0u : 1u);
                ctrl->sweep_bar = GridBar{};   // the sweep's, which is not running
            }
        }
        if (stop && first_block && cnt != a.snap.cnt)   // the lengths of the pending lists, where they are read from
            for (int c = threadIdx.x; c < 2 * nc; c += PT) a.snap.cnt[c] = cnt[c];
        if (stop || sweep) return;   // k_sweep clears the tables of this pass
        if (first_block) {           // the next snapshot's table: nobody uses it before the next barrier
            ull* other = k & 1 ? a.snap.cnt : a.cnt2;
            for (int c = threadIdx.x; c < 2 * nc; c += PT) other[c] = 0;
        }
        if (!local && !P.sync()) return;
        __syncthreads();
        const long long items = prefix[nc];
        if (take_hubs) {
            if (!P.push_taken_hubs()) return;
        } else if (a.order == 1 || a.order == 3) {
            if (!P.template push_hubs<false>(0, (long long)*a.push.hubv_cnt, false)) return;
        }
        if (!P.push_table(0, items, -1, a.order ? LISTS_SHORT : LISTS_ALL)) return;
        if (a.order == 2) { if (!P.template push_hubs<false>(0, (long long)*a.push.hubv_cnt, false)) return; }
        // the counters are read after the next snapshot's barrier
        P.report();
    }
}

// One push of the whole table (host-driven loop).
template <int L>
__global__ void __launch_bounds__(PT, 1) k_table(const __grid_constant__ SolveArgs a) {
    typedef typename Lane<L>::T T;
    __shared__ PassShared<L> s;
    Passes<L> P(a, s, hacc_init<T>(a.push.hub_k), &a.push.ctrl->bar);
    if (blockIdx.x == 0 && threadIdx.x == 0)
        for (WaveCount& w : a.push.ctrl->wave) { w.small = 0; w.big = 0; w.claim = 0; }
    if (!P.sync()) return;
    const long long nh = a.order ? (long long)*a.push.hubv_cnt : 0;
    if ((a.order == 1 || a.order == 3) && !P.template push_hubs<true>(0, nh, false)) return;
    if (!P.push_table(0, P.prefix[a.push.nc], -1, a.order ? LISTS_SHORT : LISTS_ALL)) return;
    if (a.order == 2 && !P.template push_hubs<true>(0, nh, false)) return;
    P.report();
}

// After a swept pass of a device solve: every table and sum of the passes, for the next k_passes.
__device__ __forceinline__ void clear_tables(const SolveArgs& a, int threads) {
    if (a.standalone || blockIdx.x) return;
    if (threadIdx.x == 0) a.push.ctrl->bar = GridBar{};   // that of k_passes, which is not running
    for (int c = threadIdx.x; c < 2 * a.push.nc; c += threads) { a.snap.cnt[c] = 0; a.cnt2[c] = 0; }
    if (threadIdx.x == 0) { a.push.ctrl->acc[0] = SnapAcc{}; a.push.ctrl->acc[1] = SnapAcc{}; }
}

// One pass chunk by chunk, in chunk order, per the table k_passes left.
template <int L>
__global__ void __launch_bounds__(PT, 1) k_sweep(const __grid_constant__ SolveArgs a) {
    typedef typename Lane<L>::T T;
    __shared__ PassShared<L> s;
    Ctrl* ctrl = a.push.ctrl;
    if (!a.standalone && (ctrl->done || !ctrl->sweep_pass)) return;
    Passes<L> P(a, s, hacc_init<T>(a.push.hub_k), &ctrl->sweep_bar);
    const int nc = a.push.nc;
    clear_tables(a, PT);
    if (blockIdx.x == 0 && threadIdx.x == 0)
        for (WaveCount& w : ctrl->wave) { w.small = 0; w.big = 0; w.claim = 0; }
    if (!P.sync()) return;
    const int order = a.order;
    if (order == 1 && !P.template push_hubs<true>(0, (long long)*a.push.hubv_cnt, false)) return;
    for (int c = 0; c < nc; c++) {
        const long long first = P.prefix[c], total = P.prefix[c + 1];
        if (total == first) continue;
        if (order == 3) {
            const int v0 = a.push.cv0[c], v1 = c + 1 < nc ? a.push.cv0[c + 1] : a.snap.n;
            if (!P.template push_hubs<true>(P.hub_bound(v0), P.hub_bound(v1), P.type[c] == WT_LIST)) return;
        }
        if (!P.push_table(first, total, c, order ? LISTS_SHORT : LISTS_ALL)) return;
    }
    if (order == 2 && !P.template push_hubs<true>(0, (long long)*a.push.hubv_cnt, false)) return;
    P.report();
}

}  // namespace excent
