// small.cuh -- the device solve of a graph whose vertices fit the GPU's
// threads (included by engine.cu): every thread keeps one or two vertices'
// values, offsets and degrees in registers for the whole solve.
//
// A pass on such a graph is nothing but the latency of its phases. With a
// vertex per thread a phase is one load of the residual; what a block takes
// stays in its shared memory until the barrier after the takes, and is
// scattered by the block's own warps (neighbouring vertices, and with them the
// long lists, belong to different blocks). The order is that of k_passes: the
// snapshot, in which the high-degree lists are taken; their scatter; the takes
// of the others; their scatter. R-MAT 16 PageRank, 49
// passes: 4.2 ms as graph nodes, 1.46 by k_passes, 0.95 so; 2000 vertices, all three
// measures, 42 passes: 2.6, 1.23 and 0.74 ms. The pass log and the counters of what was taken
// stay out of the chain of phases (by block 0 before its scatter and by every warp: 0.79 ms).
#pragma once

namespace excent {

static constexpr int SMALL_PER_THREAD = 2;   // vertices per thread at most

template <int L> struct SmallRec;            // one taken list
template <> struct __align__(16) SmallRec<1> { const int* nb; unsigned len; float p; };
template <> struct __align__(16) SmallRec<4> { const int* nb; unsigned len, pad; float4 p; };

// A high-degree list to the segment queue (one lane).
template <int L>
__device__ __noinline__ void queue_list(const SolveArgs& a, WaveCount* w, const int* nb, unsigned deg, typename Lane<L>::T p) {
    const unsigned nseg = (deg + a.seg - 1) / a.seg;
    const ull at = atomicAdd(&w->big, nseg);
    if (at + nseg > a.push.hub_cap) { atomicExch(&a.push.ctrl->err, 1); return; }
    HubSeg h;
    h.pad = 0;
    if constexpr (L == 1) h.p = make_float4(p, 0.f, 0.f, 0.f); else h.p = p;
    for (unsigned k = 0; k < nseg; k++) {
        h.nb = nb + (ull)k * a.seg;
        h.len = min(a.seg, deg - k * a.seg);
        a.push.hubq[at + k] = h;
    }
}

// The residuals of rv above eps: out of rv, into x, and as weights of the list.
__device__ __forceinline__ float take_reg(float& x, float& rv, unsigned deg, const DevMeasures& M) {
    if (!(fabsf(rv) > M.eps[0])) return 0.f;
    const float d = rv;
    x += d;
    rv = 0.f;
    return weight(d, deg, M, 0);
}
__device__ __forceinline__ float4 take_reg(float4& x, float4& rv, unsigned deg, const DevMeasures& M) {
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
    if (fabsf(rv.x) > M.eps[0]) { d.x = rv.x; rv.x = 0.f; }
    if (M.nm > 1 && fabsf(rv.y) > M.eps[1]) { d.y = rv.y; rv.y = 0.f; }
    if (M.nm > 2 && fabsf(rv.z) > M.eps[2]) { d.z = rv.z; rv.z = 0.f; }
    x.x += d.x; x.y += d.y; x.z += d.z;
    return make_float4(weight(d.x, deg, M, 0), weight(d.y, deg, M, 1), weight(d.z, deg, M, 2), 0.f);
}

template <int L, int V>
__global__ void __launch_bounds__(PT, 1) k_small(const __grid_constant__ SolveArgs a) {
    typedef typename Lane<L>::T T;
    typedef SmallRec<L> Rec;
    extern __shared__ float4 s_dyn[];
    __shared__ PassShared<L> s;
    __shared__ unsigned s_small, s_big;
    __shared__ ull s_cnt[2][PW];
    __shared__ ull s_took[4][PW];   // entries, entries x measures, measures taken, entries from host memory
    Ctrl* ctrl = a.push.ctrl;
    Passes<L> P(a, s, hacc_init<T>(a.push.hub_k), &ctrl->bar);
    Rec* rec = reinterpret_cast<Rec*>(reinterpret_cast<char*>(s_dyn) + ((size_t)a.push.hub_k * sizeof(T) + 15) / 16 * 16);
    const int lane = P.lane, wib = P.wib, n = a.snap.n;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    // the pass log is written off the critical path, by the last warp of the last block
    const bool scribe = blockIdx.x == gridDim.x - 1 && threadIdx.x == PT - 32;
    T* r = P.r;
    if (lane < 4) s_took[lane][wib] = 0;
    int v[V];
    unsigned deg[V];
    const int* nb[V];
    T x[V];
    float v1[V];
#pragma unroll
    for (int q = 0; q < V; q++) {
        const long long tile = (long long)(q * PW + wib) * gridDim.x + blockIdx.x;
        const long long w = tile * 32 + lane;
        v[q] = w < n ? (int)w : -1;
        deg[q] = 0;
        nb[q] = nullptr;
        x[q] = T{};
        v1[q] = 0.f;
        if (v[q] >= 0) {
            const ull b = a.push.idx[v[q]];
            deg[q] = (unsigned)(a.push.idx[v[q] + 1] - b);
            nb[q] = list_at(a.push, b);
            x[q] = P.x[v[q]];
            if (a.snap.v1) v1[q] = a.snap.v1[v[q]];
        }
    }
    for (int pass = 0;; pass++) {
        SnapAcc* acc = &ctrl->acc[pass % 3];
        WaveCount* wave = &ctrl->wave[pass % 3];
        if (threadIdx.x == 0) { s_small = 0; s_big = 0; s.next = 0; }
        if (lead) {   // the next pass's: nobody uses them before the barrier
            ctrl->wave[(pass + 1) % 3].big = 0;
            ctrl->acc[(pass + 1) % 3] = SnapAcc{};
        }
        // snapshot; the component along v1 as in snapshot_scan
        const double evc_in = a.snap.v1 ? ctrl->ev_corr : 0.0;
        const double evc = fabs(evc_in) > a.snap.ev_skip ? evc_in : 0.0;
        double rs0 = 0, rs1 = 0, rs2 = 0, evd = 0;
        unsigned pend = 0;        // bit q: vertex q is pending
        ull demand = 0;
#pragma unroll
        for (int q = 0; q < V; q++) {
            bool pq = false;
            if (v[q] >= 0) {
                T rv = r[v[q]];
                if (a.snap.v1) {
                    float re;
                    if constexpr (L == 4) re = a.snap.ev == 0 ? rv.x : a.snap.ev == 1 ? rv.y : rv.z; else re = rv;
                    if (evc != 0.0) {
                        re = (float)((double)re - evc * (double)v1[q]);
                        reinterpret_cast<float*>(r + v[q])[L == 1 ? 0 : a.snap.ev] = re;
                        if constexpr (L == 4) { if (a.snap.ev == 0) rv.x = re; else if (a.snap.ev == 1) rv.y = re; else rv.z = re; }
                        else rv = re;
                    }
                    evd += (double)re * (double)v1[q];
                }
                if constexpr (L == 1) rs0 += fabs((double)rv);
                else { rs0 += fabs((double)rv.x); rs1 += fabs((double)rv.y); rs2 += fabs((double)rv.z); }
                pq = pending_of(rv, a.push.M);
                if (pq) {
                    demand += deg[q];
                    if (a.snap.trace) a.snap.trace[v[q]]++;
                    if (deg[q] > HUB_MIN && pass < a.max_passes) {
                        const T p = take_reg(x[q], rv, deg[q], a.push.M);
                        r[v[q]] = rv;
                        if (nonzero(p)) {
                            P.count(p, deg[q], a.push.hcache ? a.push.idx[v[q]] : 0);
                            queue_list<L>(a, wave, nb[q], deg[q], p);
                        }
                    }
                }
            }
            const uint32_t word = __ballot_sync(FULL, pq);
            if (lane == 0 && v[q] >= 0) a.snap.bitmap[v[q] >> 5] = word;
            pend |= pq ? 1u << q : 0u;
        }
        {   // the block's sums
            const ull np = warp_sum((ull)__popc(pend));
            demand = warp_sum(demand);
            rs0 = warp_sum(rs0);
            if (L == 4) { rs1 = warp_sum(rs1); rs2 = warp_sum(rs2); }
            if (a.snap.v1) evd = warp_sum(evd);
            if (lane == 0) {
                s.rs[0][wib] = rs0; s.rs[1][wib] = rs1; s.rs[2][wib] = rs2; s.rs[3][wib] = evd;
                s_cnt[0][wib] = np; s_cnt[1][wib] = demand;
            }
            __syncthreads();
            if (wib < 4) {
                const double t = warp_sum(lane < PW ? s.rs[wib][lane] : 0.0);
                if (lane == 0 && t != 0.0) atomicAdd(wib < 3 ? &acc->rsum[wib] : &acc->ev_dot, t);
            } else if (wib < 6) {
                const ull t = warp_sum(lane < PW ? s_cnt[wib - 4][lane] : 0ull);
                if (lane == 0 && t) atomicAdd(wib == 4 ? &acc->pending : &acc->demand, t);
            } else if (wib < 10) {   // what the pass before took
                const ull t = warp_sum(lane < PW ? s_took[wib - 6][lane] : 0ull);
                if (lane == 0 && t) atomicAdd(wib == 6 ? &ctrl->pushed : wib == 7 ? &ctrl->lanes : wib == 8 ? &ctrl->taken : &ctrl->host_pushed, t);
            }
        }
        if (!P.sync()) return;
        const ull np = acc->pending;
        const bool stop = pass >= a.max_passes || np == 0;
        const bool range = !((double)np < a.list_frac * n);   // (src/excent.cu:639)
        const unsigned nhub = (unsigned)min((ull)wave->big, a.push.hub_cap);
        if (scribe && !stop && pass < a.log_cap) {
            PassRec& R = a.log[pass];
            R.pending = np; R.demand = acc->demand; R.hot_pending = 0; R.pushed_before = ctrl->pushed;
            R.lanes_before = ctrl->lanes; R.taken_before = ctrl->taken;
            for (int m = 0; m < MAXM; m++) R.rsum[m] = acc->rsum[m];
            R.n_list = range ? 0 : 1; R.n_range = range ? 1 : 0;
        }
        if (lead) {
            if (a.snap.v1) ctrl->ev_corr = acc->ev_dot;
            if (stop) {
                for (int m = 0; m < MAXM; m++) ctrl->rsum[m] = acc->rsum[m];
                ctrl->done = 1;
                ctrl->pass = pass;
                a.snap.cnt[1] = acc->demand;
            }
        }
        if (stop) {   // out of passes, perhaps: the pending list as a snapshot leaves it
#pragma unroll
            for (int q = 0; q < V; q++) {
                if (v[q] >= 0) P.x[v[q]] = x[q];
                if (pend >> q & 1u) a.snap.list[atomicAdd(&a.snap.cnt[0], 1ull)] = v[q];
            }
            return;
        }
        if (nhub) {
            P.scatter_wave(nhub, 0);
            if (!P.sync()) return;
        }
        // the other lists: taken into the block's shared memory, short ones from the front, those of
        // more than WAVE_LONG entries from the back
        if (threadIdx.x == 0) s.next = 0;   // (nobody claims before the next barrier)
#pragma unroll
        for (int q = 0; q < V; q++) {
            T p{};
            if (v[q] >= 0 && deg[q] <= HUB_MIN && (range || (pend >> q & 1u))) {
                T rv = r[v[q]];
                if (pending_of(rv, a.push.M)) {
                    p = take_reg(x[q], rv, deg[q], a.push.M);
                    r[v[q]] = rv;
                }
            }
            const bool act = nonzero(p) && deg[q] > 0;
            if (act) P.count(p, deg[q], a.push.hcache ? a.push.idx[v[q]] : 0);
            const bool sm = act && deg[q] <= WAVE_LONG;
            const unsigned ms = __ballot_sync(FULL, sm), mb = __ballot_sync(FULL, act && !sm), lt = (1u << lane) - 1u;
            unsigned as = 0, ab = 0;
            if (lane == 0) {
                if (ms) as = atomicAdd(&s_small, __popc(ms));
                if (mb) ab = atomicAdd(&s_big, __popc(mb));
            }
            as = __shfl_sync(FULL, as, 0);
            ab = __shfl_sync(FULL, ab, 0);
            if (act) {
                Rec& t = rec[sm ? as + __popc(ms & lt) : PT * V - 1 - (ab + __popc(mb & lt))];
                t.nb = nb[q];
                t.len = deg[q];
                t.p = p;
            }
        }
        {   // what this warp took in this pass, high-degree lists included
            const unsigned lo = __reduce_add_sync(FULL, (unsigned)P.pushed & 0xffffu);
            const unsigned hi = __reduce_add_sync(FULL, (unsigned)(P.pushed >> 16));
            const unsigned llo = __reduce_add_sync(FULL, (unsigned)P.lanes & 0xffffu);
            const unsigned lhi = __reduce_add_sync(FULL, (unsigned)(P.lanes >> 16));
            const unsigned tk = __reduce_add_sync(FULL, (unsigned)P.taken);
            const ull h = a.push.hcache ? warp_sum(P.hpushed) : 0;
            if (lane == 0) {
                s_took[0][wib] = lo + ((ull)hi << 16);
                s_took[1][wib] = llo + ((ull)lhi << 16);
                s_took[2][wib] = tk;
                s_took[3][wib] = h;
            }
            P.pushed = P.lanes = P.taken = P.hpushed = 0;
        }
        if (!P.sync()) return;
        const unsigned nsmall = s_small, nbig = s_big;
        const unsigned per_tile = min(32u, max(8u, nsmall / PW)), ntiles = (nsmall + per_tile - 1) / per_tile;
        for (;;) {
            unsigned i = 0;
            if (lane == 0) i = atomicAdd(&s.next, 1u);
            i = __shfl_sync(FULL, i, 0);
            if (i < nbig) {
                const Rec& t = rec[PT * V - 1 - i];
                warp_scatter(r, t.nb, t.len, t.p, lane, P.hacc);
            } else if (i - nbig < ntiles) {
                const unsigned j = (i - nbig) * per_tile + lane;
                const int* tn = nullptr;
                unsigned ds = 0;
                T p{};
                if (lane < per_tile && j < nsmall) { tn = rec[j].nb; ds = rec[j].len; p = rec[j].p; }
                P.scatter_tile(tn, ds, p);
            } else {
                break;
            }
        }
        P.flush();
        if (!P.sync()) return;
    }
}

}  // namespace excent
