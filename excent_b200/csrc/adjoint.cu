// adjoint.cu -- differentiable weighted PageRank / Katz on a directed graph.
//
// Forward (kind EXCENT_PR): x = (1 - d) t + d W^T x, with W the row-normalised
// edge weights wn[e] = w[e] / sum_{e' in row u} w[e'] of edges u -> v, so
// (W^T x)_v = sum_{u -> v} wn[u->v] x_u. Katz (kind EXCENT_KATZ):
// x = beta + alpha W^T x. Both run as a delta-push over out-lists: pushing u
// adds s * wn[e] * d_u to r_v for each edge e = u -> v (s = d or alpha).
//
// Adjoint of a scalar loss L with dL/dx = c: lambda = c + s W lambda, a push
// over the transposed lists with the permuted weights. Gradients:
//   dL/dt = (1 - d) lambda (PageRank),  dL/dbeta = lambda (Katz),
//   dL/dwn[u->v] = s x_u lambda_v,
//   dL/dw[e] = (G_e - sum_{e' in row u} wn[e'] G_e') / rowsum_u, G = dL/dwn.
// No reference counterpart (the reference has no weights and no adjoint).
//
// A solve is one cooperative launch that runs every pass. FP64 pull (Jacobi) solvers of the same fixed
// points give finite differences and the oracle gradient for verification.
#include <cub/cub.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.h"
#include "device.cuh"
#include "gridsync.cuh"
#include "pull.cuh"

namespace excent {

static constexpr int WB = 256;
static constexpr int WP = 1024;             // threads per block of the persistent push, one block per SM
static constexpr int WUNROLL = 4;           // entries per lane in flight

struct WCtrl {
    int pass, max_passes, pad0, pad1;
    ull demand[2];     // entries of the lists of the vertices above eps, by pass parity
    ull above[2];      // vertices above eps
    ull total_e;
    GridBar bar;
};

// A weighted CSR: per-entry weight (row-normalised), long lists also as segments.
struct WLists {
    const ull* idx;
    const int* adj;
    const float* wt;
    const ListSeg* seg;
    ull nseg;
};

struct WArgs {
    int n;
    WLists out;        // the lists a push scatters along
    WLists in;         // the transposed lists: what a vertex gathers from
    ull m;
    ull pull_min;      // a pass after one of at least this demand gathers, the others scatter
    float s;
    float eps;
    float* x;
    float* r;
    float* d;          // what each vertex had taken in this pass (0 at the start)
    WCtrl* ctrl;
};

struct WGather {
    const int* adj;
    const float* wt;
    const float* d;
    struct Key { int u = -1; float w = 0.f; };
    __device__ __forceinline__ Key key(ull e) const {
        Key k;
        k.u = ld_edge(adj + e);
        k.w = __ldcs(wt + e);
        return k;
    }
    __device__ __forceinline__ float value(const Key& k) const {
        const float q = k.u >= 0 ? d[k.u] : 0.f;
        return q != 0.f ? k.w * q : 0.f;   // a vertex that pushed nothing delivers nothing, whatever its weights are
    }
};

// The whole delta-push in one cooperative launch. A pass is two phases with a
// grid barrier after each: residuals are taken into d; then s * d * wt[e] is
// delivered along every list. It gathers over the transposed lists while the
// pass before had at least pull_min entries to deliver, and scatters below
// that; both read the short lists edge-balanced and the long ones as segments.
// A gather reads every list anyway, so its passes take every residual, not
// only those above eps. What such passes leave is nearly the same everywhere,
// where a push leaves anything between 0 and eps, so they go on to eps / 2:
// four more passes, and an error below the push's (to eps itself it was a
// third above it, 1.3e-5 against 9.8e-6 in dL/dt of 1M vertices). x gets what a pass has taken in the next one, so that a pass that
// finds nothing above eps ends the solve with nothing taken.
//
// What bounds it: a gather and 8 bytes per entry in the dense passes, then the
// latency of the phases (75 us for a dense pass of 16.8M entries). On an R-MAT
// of 1M vertices and 16.8M entries, forward and gradient together took 305 ms
// with whole lists on one warp, 58.7 ms scattering them split (38 G entries/s:
// reductions to the same vertices serialise) and take 14.8 ms gathering, to
// eps / 2 (14.5 ms to eps; 181-196 G entries/s).
__global__ void __launch_bounds__(WP, 1) k_wsolve(WArgs a) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const long long gw = (long long)wib * gridDim.x + blockIdx.x;   // neighbouring tiles on different SMs
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    const long long ntiles = ((long long)a.n + 31) / 32;
    __shared__ PullScratch<float> s_tile[WP / 32];   // per warp: the tile's nonempty lists (acc: push weights)
    __shared__ ull s_v[WP / 32], s_e[WP / 32];
    __shared__ unsigned s_next;
    PullScratch<float>& S = s_tile[wib];
    const WGather gather{a.in.adj, a.in.wt, a.d};
    unsigned epoch = 0;
    const int max_passes = a.ctrl->max_passes;
    bool pull = a.pull_min <= a.m;
    for (int pass = 0;; pass++) {
        const int par = pass & 1;
        ull pv = 0, pe = 0;
        for (long long t0 = gw; t0 < ntiles; t0 += 4 * nwarps) {
            float rv[4], dv[4];   // four tiles in flight before they are examined
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const long long v = (t0 + k * nwarps) * 32 + lane;
                rv[k] = v < a.n ? a.r[v] : 0.f;
                dv[k] = v < a.n ? a.d[v] : 0.f;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const long long v = (t0 + k * nwarps) * 32 + lane;
                if (v >= a.n) continue;
                if (dv[k] != 0.f) a.x[v] += dv[k];
                const bool above = fabsf(rv[k]) > a.eps;
                // (a residual that is no number, from a row whose weights sum to 0, is never above eps: it stays)
                const float d = above || (pull && rv[k] == rv[k]) ? rv[k] : 0.f;
                if (d != 0.f) a.r[v] = 0.f;
                if (d != 0.f || dv[k] != 0.f) a.d[v] = d;
                if (above) {
                    pv++;
                    pe += a.out.idx[v + 1] - a.out.idx[v];
                }
            }
        }
        pv = warp_sum(pv);
        pe = warp_sum(pe);
        if (lane == 0) { s_v[wib] = pv; s_e[wib] = pe; }
        __syncthreads();
        if (threadIdx.x == 0) {
            s_next = 0;
            ull tv = 0, te = 0;
            for (int i = 0; i < WP / 32; i++) { tv += s_v[i]; te += s_e[i]; }
            if (tv) atomicAdd(&a.ctrl->above[par], tv);
            if (te) atomicAdd(&a.ctrl->demand[par], te);
        }
        if (!grid_sync(&a.ctrl->bar, epoch)) return;
        const ull above = a.ctrl->above[par], demand = a.ctrl->demand[par];
        if (!above) break;
        if (blockIdx.x == 0 && threadIdx.x == 0) {   // the next pass's counters: nobody uses them before the barrier
            a.ctrl->above[par ^ 1] = 0;
            a.ctrl->demand[par ^ 1] = 0;
            a.ctrl->total_e += pull ? a.m : demand;
            a.ctrl->pass = pass + 1;
        }
        if (pull) {
            gather_phase<float>(a.n, a.in.idx, a.in.seg, a.in.nseg, gather, [&](unsigned v, float sum, bool part) {
                if (sum == 0.f) return;
                if (part) atomicAdd(&a.r[v], a.s * sum);
                else a.r[v] += a.s * sum;
            }, &s_next, S, lane);
        } else if (demand) {
            for (ull i = gw; i < a.out.nseg; i += nwarps) {
                const ListSeg g = a.out.seg[i];
                const float f = a.s * a.d[g.row];
                if (f == 0.f) continue;
                for (unsigned i0 = 0; i0 < g.len; i0 += 32 * WUNROLL) {
                    int u[WUNROLL];
                    float w[WUNROLL];
#pragma unroll
                    for (int q = 0; q < WUNROLL; q++) {
                        const unsigned j = i0 + 32 * q + lane;
                        u[q] = j < g.len ? ld_edge(a.out.adj + g.base + j) : -1;
                        w[q] = j < g.len ? __ldcs(a.out.wt + g.base + j) : 0.f;
                    }
#pragma unroll
                    for (int q = 0; q < WUNROLL; q++)
                        if (u[q] >= 0) red_add(a.r, u[q], f * w[q]);
                }
            }
            for (long long tile = gw; tile < ntiles; tile += nwarps) {
                const long long v = tile * 32 + lane;
                const float f = v < a.n ? a.s * a.d[v] : 0.f;
                if (!__any_sync(FULL, f != 0.f)) continue;
                ull b0 = 0;
                unsigned ds = 0;
                if (f != 0.f) {
                    b0 = a.out.idx[v];
                    const ull dv = a.out.idx[v + 1] - b0;
                    ds = dv > PULL_LONG ? 0u : (unsigned)dv;
                }
                const unsigned nz = __ballot_sync(FULL, ds != 0);
                if (!nz) continue;
                const unsigned incl = warp_incl_scan(ds, lane);
                const unsigned tot = __shfl_sync(FULL, incl, 31);
                const unsigned ex = incl - ds;
                if (ds) {
                    const int rank = __popc(nz & ((1u << lane) - 1u));
                    S.base[rank] = b0; S.ex[rank] = ex; S.acc[rank] = f;
                }
                __syncwarp();
                const unsigned le = lane == 31 ? FULL : (2u << lane) - 1u;
                for (unsigned j0 = 0; j0 < tot; j0 += 32 * WUNROLL) {
                    int u[WUNROLL];
                    float w[WUNROLL];
#pragma unroll
                    for (int q = 0; q < WUNROLL; q++) {
                        // owner of entry wb + lane: the last nonempty list starting at or before it
                        const unsigned wb = j0 + 32 * q, j = wb + lane;
                        const unsigned starts =
                            __reduce_or_sync(FULL, (ds && ex >= wb && ex - wb < 32) ? 1u << (ex - wb) : 0u);
                        const int o = __popc(__ballot_sync(FULL, ds && ex <= wb)) - 1 + __popc(starts & le & ~1u);
                        u[q] = -1;
                        w[q] = 0.f;
                        if (j < tot) {
                            const ull e = S.base[o] + (j - S.ex[o]);
                            u[q] = ld_edge(a.out.adj + e);
                            w[q] = S.acc[o] * __ldcs(a.out.wt + e);
                        }
                    }
#pragma unroll
                    for (int q = 0; q < WUNROLL; q++)
                        if (u[q] >= 0) red_add(a.r, u[q], w[q]);
                }
                __syncwarp();
            }
        }
        pull = demand >= a.pull_min;
        if (!grid_sync(&a.ctrl->bar, epoch)) return;
        if (pass + 1 >= max_passes) {   // out of passes: x gets what this one has taken
            for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < a.n;
                 v += (long long)gridDim.x * blockDim.x)
                a.x[v] += a.d[v];
            break;
        }
    }
}

// x = d = 0, r = c0 * t (t NULL: all ones).
__global__ void k_wseed(int n, const float* t, float c0, float* x, float* r, float* d) {
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        x[v] = 0.f;
        d[v] = 0.f;
        r[v] = c0 * (t ? t[v] : 1.f);
    }
}

// Row sums and normalised weights (FP32 for the push, FP64 for the tools): one
// warp per row of up to PULL_LONG entries. The longer rows start at 0 here; their
// segments are summed by k_wsegsum and scaled by k_wsegnorm, one warp per
// segment (a whole row on one warp took 69k / 32 dependent steps, twice).
__global__ void k_wnorm(int n, const ull* idx, const float* w, float* wn, double* wn64, double* rowsum) {
    const long long u = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (u >= n) return;
    const ull b = idx[u], e1 = idx[u + 1];
    if (e1 - b > PULL_LONG) {
        if (lane == 0) rowsum[u] = 0;
        return;
    }
    double s = 0;
    for (ull e = b + lane; e < e1; e += 32) s += w[e];
    s = warp_sum(s);
    s = __shfl_sync(FULL, s, 0);
    for (ull e = b + lane; e < e1; e += 32) {
        const double q = (double)w[e] / s;
        wn[e] = (float)q;
        wn64[e] = q;
    }
    if (lane == 0) rowsum[u] = s;
}
__global__ void k_wsegsum(ull nseg, const ListSeg* seg, const float* w, double* rowsum) {
    const ull i = (blockIdx.x * (ull)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= nseg) return;
    const ListSeg g = seg[i];
    double s = 0;
    for (unsigned j = lane; j < g.len; j += 32) s += w[g.base + j];
    s = warp_sum(s);
    if (lane == 0) atomicAdd(&rowsum[g.row], s);
}
__global__ void k_wsegnorm(ull nseg, const ListSeg* seg, const float* w, const double* rowsum, float* wn, double* wn64) {
    const ull i = (blockIdx.x * (ull)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= nseg) return;
    const ListSeg g = seg[i];
    const double s = rowsum[g.row];
    for (unsigned j = lane; j < g.len; j += 32) {
        const double q = (double)w[g.base + j] / s;
        wn[g.base + j] = (float)q;
        wn64[g.base + j] = q;
    }
}

__global__ void k_wpermute(ull m, const unsigned* perm, const float* wn, const double* wn64, float* wt, double* wt64) {
    for (ull e = blockIdx.x * (ull)blockDim.x + threadIdx.x; e < m; e += (ull)gridDim.x * blockDim.x) {
        wt[e] = wn[perm[e]];
        wt64[e] = wn64[perm[e]];
    }
}

__global__ void k_winverse(ull m, const unsigned* perm, unsigned* inv) {
    for (ull e = blockIdx.x * (ull)blockDim.x + threadIdx.x; e < m; e += (ull)gridDim.x * blockDim.x)
        inv[perm[e]] = (unsigned)e;
}

// Transposed CSR from keys (dst << scale | src) sorted with the original edge ids.
__global__ void k_wtrans(int n, int shift, ull m, const uint64_t* keys, int* adjT, ull* idxT) {
    const uint64_t mask = (1ull << shift) - 1;
    for (ull e = blockIdx.x * (ull)blockDim.x + threadIdx.x; e <= m; e += (ull)gridDim.x * blockDim.x) {
        const long long s = e < m ? (long long)(keys[e] >> shift) : n;
        const long long p = e > 0 ? (long long)(keys[e - 1] >> shift) : -1;
        if (e < m) adjT[e] = (int)(keys[e] & mask);
        for (long long v = p + 1; v <= s; v++) idxT[v] = e;
    }
}

__global__ void k_wkeys(int n, int shift, const ull* idx, const int* adj, uint64_t* keys, unsigned* vals) {
    const long long u = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (u >= n) return;
    for (ull e = idx[u] + lane; e < idx[u + 1]; e += 32) {
        keys[e] = ((uint64_t)adj[e] << shift) | (uint64_t)u;
        vals[e] = (unsigned)e;
    }
}

// Gradient through the row normalisation: dL/dw[e] = (G_e - sum wn G) / rowsum
// with G_e = s x_u lam_v, one warp per row of up to PULL_LONG entries; the longer
// rows' sums are accumulated by k_wgradsum and finished by k_wgradseg.
__global__ void k_wgrad(int n, const ull* idx, const int* adj, const float* wn, const double* rowsum, const float* x,
                        const float* lam, float s, float* gw, double* rowdot) {
    const long long u = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (u >= n) return;
    const ull b = idx[u], e1 = idx[u + 1];
    if (e1 - b > PULL_LONG) {
        if (lane == 0) rowdot[u] = 0;
        return;
    }
    const double xu = x[u];
    double dot = 0;
    for (ull e = b + lane; e < e1; e += 32) dot += (double)wn[e] * s * xu * lam[adj[e]];
    dot = warp_sum(dot);
    dot = __shfl_sync(FULL, dot, 0);
    const double rs = rowsum[u];
    for (ull e = b + lane; e < e1; e += 32) gw[e] = (float)(((double)s * xu * lam[adj[e]] - dot) / rs);
}
__global__ void k_wgradsum(ull nseg, const ListSeg* seg, const int* adj, const float* wn, const float* x,
                           const float* lam, float s, double* rowdot) {
    const ull i = (blockIdx.x * (ull)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= nseg) return;
    const ListSeg g = seg[i];
    const double xu = x[g.row];
    double dot = 0;
    for (unsigned j = lane; j < g.len; j += 32) dot += (double)wn[g.base + j] * s * xu * lam[adj[g.base + j]];
    dot = warp_sum(dot);
    if (lane == 0) atomicAdd(&rowdot[g.row], dot);
}
__global__ void k_wgradseg(ull nseg, const ListSeg* seg, const int* adj, const double* rowsum, const float* x,
                           const float* lam, float s, const double* rowdot, float* gw) {
    const ull i = (blockIdx.x * (ull)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= nseg) return;
    const ListSeg g = seg[i];
    const double xu = x[g.row], dot = rowdot[g.row], rs = rowsum[g.row];
    for (unsigned j = lane; j < g.len; j += 32)
        gw[g.base + j] = (float)(((double)s * xu * lam[adj[g.base + j]] - dot) / rs);
}

__global__ void k_wscale(int n, const float* in, float f, float* out) {
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x)
        out[v] = f * in[v];
}

// FP64 pull: y_v = c * t_v + s * sum_e wt[e] x[adj[e]] over the lists of v;
// mx[0] = max |y - x|, mx[1] = max |y| as ordered bit patterns.
__global__ void k_wpull64(int n, const ull* idx, const int* adj, const double* wt, const double* x, const float* t,
                          double c, double s, double* y, ull* mx) {
    const long long v = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (v >= n) return;
    double acc = 0;
    for (ull e = idx[v] + lane; e < idx[v + 1]; e += 32) acc += wt[e] * x[adj[e]];
    acc = warp_sum(acc);
    if (lane == 0) {
        const double nv = c * (t ? (double)t[v] : 1.0) + s * acc;
        y[v] = nv;
        atomicMax(&mx[0], (ull)__double_as_longlong(fabs(nv - x[v])));
        atomicMax(&mx[1], (ull)__double_as_longlong(fabs(nv)));
    }
}

__global__ void k_wdot64(int n, const double* x, const float* c, double* out) {
    double a = 0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x)
        a += x[v] * (double)c[v];
    a = warp_sum(a);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, a);
}

__global__ void k_wgrad64(int n, const ull* idx, const int* adj, const double* wn64, const double* rowsum,
                          const double* x, const double* lam, double s, double* gw) {
    const long long u = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (u >= n) return;
    double dot = 0;
    for (ull e = idx[u] + lane; e < idx[u + 1]; e += 32) dot += wn64[e] * s * x[u] * lam[adj[e]];
    dot = warp_sum(dot);
    dot = __shfl_sync(FULL, dot, 0);
    for (ull e = idx[u] + lane; e < idx[u + 1]; e += 32) gw[e] = (s * x[u] * lam[adj[e]] - dot) / rowsum[u];
}

}  // namespace excent

using namespace excent;

struct excent_wgraph {
    int dev = 0, sms = 0, n = 0;
    ull m = 0;
    const ull* d_idx = nullptr;   // caller's forward CSR
    const int* d_adj = nullptr;
    const float* d_wraw = nullptr;
    float* d_wn = nullptr;        // forward order
    double* d_wn64 = nullptr;
    double* d_rowsum = nullptr;
    ull* d_idxT = nullptr;
    int* d_adjT = nullptr;
    unsigned* d_perm = nullptr;   // transposed edge -> forward edge
    unsigned* d_inv = nullptr;    // forward edge -> transposed edge
    float* d_wt = nullptr;        // transposed order
    double* d_wt64 = nullptr;
    float *d_x = nullptr, *d_r = nullptr, *d_lam = nullptr;
    ListSeg* d_rowseg = nullptr;  // the long lists of the forward graph as segments
    ListSeg* d_colseg = nullptr;  // and of the transposed graph
    ull n_rowseg = 0, n_colseg = 0;
    float* d_d = nullptr;         // what a pass has taken
    double* d_rowdot = nullptr;
    WCtrl* d_ctrl = nullptr;
    double *d_v64[2] = {nullptr, nullptr};
    ull* d_mx = nullptr;
    double* d_red = nullptr;
    cudaStream_t st = nullptr;
    bool have_fwd = false;
    bool host_t = false;          // transposed lists and weights in pinned, mapped host memory
    int* h_adjT = nullptr;
    float* h_wt = nullptr;
    double* h_wt64 = nullptr;
    int fwd_kind = -1;
    double fwd_s = 0;
    ull launches = 0;
};

static void wg_free(excent_wgraph* g) {
    cudaSetDevice(g->dev);
    cudaDeviceSynchronize();
    if (g->host_t) {
        cudaFreeHost(g->h_adjT);
        cudaFreeHost(g->h_wt);
        cudaFreeHost(g->h_wt64);
        g->d_adjT = nullptr; g->d_wt = nullptr; g->d_wt64 = nullptr;
    }
    void* ps[] = {g->d_wn, g->d_wn64, g->d_rowsum, g->d_idxT, g->d_adjT, g->d_perm, g->d_inv, g->d_wt, g->d_wt64,
                  g->d_x, g->d_r, g->d_lam, g->d_rowseg, g->d_colseg, g->d_d, g->d_rowdot, g->d_ctrl, g->d_v64[0], g->d_v64[1], g->d_mx,
                  g->d_red};
    for (void* p : ps) if (p) cudaFree(p);
    if (g->st) cudaStreamDestroy(g->st);
    delete g;
}

#define WG_ALLOC(ptr, bytes) do { if (cudaMalloc((void**)&(ptr), (bytes)) != cudaSuccess) { cudaGetLastError(); \
    ::excent::set_error("wgraph: device allocation of %llu bytes failed (%s)", (ull)(bytes), #ptr); return EXCENT_ERR_NOMEM; } } while (0)

static unsigned seg_blocks(const excent_wgraph* g) { return (unsigned)((g->n_rowseg * 32 + WB - 1) / WB); }

static int wg_normalise(excent_wgraph* g) {
    const unsigned wb = (unsigned)(((long long)g->n * 32 + WB - 1) / WB);
    k_wnorm<<<wb, WB, 0, g->st>>>(g->n, g->d_idx, g->d_wraw, g->d_wn, g->d_wn64, g->d_rowsum);
    if (g->n_rowseg) {
        const unsigned sb = seg_blocks(g);
        k_wsegsum<<<sb, WB, 0, g->st>>>(g->n_rowseg, g->d_rowseg, g->d_wraw, g->d_rowsum);
        k_wsegnorm<<<sb, WB, 0, g->st>>>(g->n_rowseg, g->d_rowseg, g->d_wraw, g->d_rowsum, g->d_wn, g->d_wn64);
        g->launches += 2;
    }
    if (g->m) k_wpermute<<<2048, WB, 0, g->st>>>(g->m, g->d_perm, g->d_wn, g->d_wn64, g->d_wt, g->d_wt64);
    g->launches += 2;
    EX_CUDA(cudaGetLastError());
    EX_CUDA(cudaStreamSynchronize(g->st));
    g->have_fwd = false;
    return EXCENT_OK;
}

// The long lists of one direction as segments (once per graph).
static int wg_segments(excent_wgraph* g, const ull* idx, ListSeg** seg, ull* count) {
    WG_ALLOC(*seg, list_seg_cap(g->m) * sizeof(ListSeg));
    EX_CUDA(cudaMemsetAsync(g->d_mx, 0, sizeof(ull), g->st));
    k_list_segs<<<g->sms * 8, WB, 0, g->st>>>(g->n, idx, *seg, g->d_mx);
    EX_CUDA(cudaGetLastError());
    EX_CUDA(cudaMemcpyAsync(count, g->d_mx, sizeof(ull), cudaMemcpyDeviceToHost, g->st));
    EX_CUDA(cudaStreamSynchronize(g->st));
    return EXCENT_OK;
}

static int wg_setup(excent_wgraph* g, int device, int n, ull m, const ull* d_idx, const int* d_adj, const float* d_w) {
    EX_CUDA(cudaSetDevice(device));
    g->dev = device;
    EX_CUDA(cudaDeviceGetAttribute(&g->sms, cudaDevAttrMultiProcessorCount, device));
    EX_CHECK_ARG(m < (1ull << 32), "weighted graphs are limited to 2^32 - 1 edges");
    g->n = n; g->m = m; g->d_idx = d_idx; g->d_adj = d_adj; g->d_wraw = d_w;
    EX_CUDA(cudaStreamCreateWithFlags(&g->st, cudaStreamNonBlocking));
    const size_t me = std::max<ull>(m, 1);
    WG_ALLOC(g->d_wn, me * 4);
    WG_ALLOC(g->d_wn64, me * 8);
    WG_ALLOC(g->d_rowsum, (size_t)n * 8);
    WG_ALLOC(g->d_idxT, ((size_t)n + 1) * 8);
    WG_ALLOC(g->d_adjT, me * 4);
    WG_ALLOC(g->d_perm, me * 4);
    WG_ALLOC(g->d_inv, me * 4);
    WG_ALLOC(g->d_wt, me * 4);
    WG_ALLOC(g->d_wt64, me * 8);
    WG_ALLOC(g->d_x, (size_t)n * 4);
    WG_ALLOC(g->d_r, (size_t)n * 4);
    WG_ALLOC(g->d_lam, (size_t)n * 4);
    WG_ALLOC(g->d_d, (size_t)n * 4);
    WG_ALLOC(g->d_rowdot, (size_t)n * 8);
    WG_ALLOC(g->d_ctrl, sizeof(WCtrl));
    WG_ALLOC(g->d_mx, 2 * sizeof(ull));
    WG_ALLOC(g->d_red, sizeof(double));
    // transpose: sort (dst, src) keys carrying forward edge ids
    int shift = 1;
    while ((1ll << shift) < (long long)n) shift++;
    uint64_t *k0 = nullptr, *k1 = nullptr;
    unsigned *v0 = nullptr;
    void* tmp = nullptr;
    size_t tb = 0;
    int rc = EXCENT_OK;
    do {
        if (cudaMalloc(&k0, me * 8) != cudaSuccess || cudaMalloc(&k1, me * 8) != cudaSuccess ||
            cudaMalloc(&v0, me * 4) != cudaSuccess) {
            cudaGetLastError();
            set_error("wgraph: transpose scratch does not fit");
            rc = EXCENT_ERR_NOMEM;
            break;
        }
        const unsigned wb = (unsigned)(((long long)n * 32 + WB - 1) / WB);
        k_wkeys<<<wb, WB, 0, g->st>>>(n, shift, d_idx, d_adj, k0, v0);
        cub::DeviceRadixSort::SortPairs(nullptr, tb, k0, k1, v0, g->d_perm, (long long)m, 0, 2 * shift, g->st);
        if (cudaMalloc(&tmp, std::max<size_t>(tb, 16)) != cudaSuccess) {
            cudaGetLastError();
            set_error("wgraph: sort scratch does not fit");
            rc = EXCENT_ERR_NOMEM;
            break;
        }
        if (cub::DeviceRadixSort::SortPairs(tmp, tb, k0, k1, v0, g->d_perm, (long long)m, 0, 2 * shift, g->st) !=
            cudaSuccess) {
            set_error("wgraph: transpose sort failed");
            rc = EXCENT_ERR_CUDA;
            break;
        }
        k_wtrans<<<2048, WB, 0, g->st>>>(n, shift, m, k1, g->d_adjT, g->d_idxT);
        if (cudaStreamSynchronize(g->st) != cudaSuccess) { set_error("wgraph: transpose failed"); rc = EXCENT_ERR_CUDA; }
    } while (0);
    if (k0) cudaFree(k0);
    if (k1) cudaFree(k1);
    if (v0) cudaFree(v0);
    if (tmp) cudaFree(tmp);
    if (rc != EXCENT_OK) return rc;
    // inverse permutation (forward edge -> transposed edge), and the long lists of both directions
    if (m) {
        k_winverse<<<2048, WB, 0, g->st>>>(m, g->d_perm, g->d_inv);
        EX_TRY(wg_segments(g, d_idx, &g->d_rowseg, &g->n_rowseg));
        EX_TRY(wg_segments(g, g->d_idxT, &g->d_colseg, &g->n_colseg));
    }
    return wg_normalise(g);
}

extern "C" int excent_wgraph_create(int device, int n, unsigned long long m, const unsigned long long* d_idx,
                                    const int32_t* d_adj, const float* d_w, excent_wgraph** out) {
    EX_CHECK_ARG(out && n >= 1 && d_idx && (m == 0 || (d_adj && d_w)), "bad argument");
    *out = nullptr;
    excent_wgraph* g = new excent_wgraph();
    const int rc = wg_setup(g, device, n, m, d_idx, d_adj, d_w);
    if (rc != EXCENT_OK) {
        std::string msg = get_error();
        wg_free(g);
        set_error("%s", msg.c_str());
        return rc;
    }
    *out = g;
    return EXCENT_OK;
}

extern "C" int excent_wgraph_destroy(excent_wgraph* g) {
    if (g) wg_free(g);
    return EXCENT_OK;
}

extern "C" int excent_wgraph_set_weights(excent_wgraph* g, const float* d_w) {
    EX_CHECK_ARG(g && (d_w || g->m == 0), "bad argument");
    EX_CUDA(cudaSetDevice(g->dev));
    g->d_wraw = d_w;
    return wg_normalise(g);
}

static WArgs wargs(excent_wgraph* g, bool transposed, float s, float eps, float* x, float* r) {
    WArgs a{};
    a.n = g->n; a.m = g->m;
    const WLists fwd{g->d_idx, g->d_adj, g->d_wn, g->d_rowseg, g->n_rowseg};
    const WLists tr{g->d_idxT, g->d_adjT, g->d_wt, g->d_colseg, g->n_colseg};
    a.out = transposed ? tr : fwd;
    a.in = transposed ? fwd : tr;
    // a gather reads every list, at about four times the scatter's rate; where one direction's
    // lists lie in host memory, the solve stays with the other
    a.pull_min = g->host_t ? (transposed ? 0 : ~0ull) : g->m / 4;
    a.s = s; a.eps = a.pull_min <= g->m && 0.5f * eps > 0.f ? 0.5f * eps : eps; a.x = x; a.r = r; a.d = g->d_d;
    a.ctrl = g->d_ctrl;
    return a;
}

// Delta-push to eps of the fixed point x = c0 * seed + s * (op) x; op = W^T
// (forward lists) or W (transposed lists). Result in x.
static int wg_push(excent_wgraph* g, bool transposed, float s, float eps, int max_passes, const float* seed, float c0,
                   float* x, int* passes, ull* pushed) {
    k_wseed<<<g->sms * 8, WB, 0, g->st>>>(g->n, seed, c0, x, g->d_r, g->d_d);
    WCtrl c{};
    c.max_passes = max_passes;
    EX_CUDA(cudaMemcpyAsync(g->d_ctrl, &c, sizeof c, cudaMemcpyHostToDevice, g->st));
    WArgs a = wargs(g, transposed, s, eps, x, g->d_r);
    // one block per SM, fewer where there is not a tile of 32 vertices for each
    const int grid = (int)std::max(1ll, std::min<long long>(g->sms, ((long long)g->n + 31) / 32));
    EX_CUDA(launch_grid(k_wsolve, grid, WP, 0, a, &g->d_ctrl->bar, g->st));
    EX_CUDA(cudaMemcpyAsync(&c, g->d_ctrl, sizeof c, cudaMemcpyDeviceToHost, g->st));
    EX_CUDA(cudaStreamSynchronize(g->st));
    g->launches += 2;
    if (c.bar.failed) EX_FAIL(EXCENT_ERR_STATE, "wgraph: a wait between the blocks of the push timed out");
    if (passes) *passes = c.pass;
    if (pushed) *pushed = c.total_e;
    return EXCENT_OK;
}

extern "C" int excent_wgraph_forward(excent_wgraph* g, int kind, double s, const float* d_t, float eps, int max_passes,
                                     float* d_x_out, int* passes, unsigned long long* pushed) {
    EX_CHECK_ARG(g && (kind == EXCENT_PR || kind == EXCENT_KATZ) && eps > 0 && max_passes >= 1, "bad argument");
    EX_CUDA(cudaSetDevice(g->dev));
    const float c0 = kind == EXCENT_PR ? (float)(1.0 - s) : 1.f;
    EX_TRY(wg_push(g, false, (float)s, eps, max_passes, d_t, c0, g->d_x, passes, pushed));
    if (d_x_out) EX_CUDA(cudaMemcpy(d_x_out, g->d_x, (size_t)g->n * 4, cudaMemcpyDeviceToDevice));
    g->have_fwd = true;
    g->fwd_kind = kind;
    g->fwd_s = s;
    return EXCENT_OK;
}

extern "C" int excent_wgraph_vjp(excent_wgraph* g, const float* d_c, float eps, int max_passes, float* d_grad_t,
                                 float* d_grad_w, int* passes, unsigned long long* pushed) {
    EX_CHECK_ARG(g && d_c && eps > 0 && max_passes >= 1, "bad argument");
    EX_CHECK_ARG(g->have_fwd, "vjp needs a forward solve with the current weights first");
    EX_CUDA(cudaSetDevice(g->dev));
    const float s = (float)g->fwd_s;
    EX_TRY(wg_push(g, true, s, eps, max_passes, d_c, 1.f, g->d_lam, passes, pushed));
    if (d_grad_t) {
        const float f = g->fwd_kind == EXCENT_PR ? (float)(1.0 - g->fwd_s) : 1.f;
        k_wscale<<<g->sms * 8, WB, 0, g->st>>>(g->n, g->d_lam, f, d_grad_t);
        g->launches++;
    }
    if (d_grad_w && g->m) {
        const unsigned wb = (unsigned)(((long long)g->n * 32 + WB - 1) / WB);
        k_wgrad<<<wb, WB, 0, g->st>>>(g->n, g->d_idx, g->d_adj, g->d_wn, g->d_rowsum, g->d_x, g->d_lam, s, d_grad_w,
                                      g->d_rowdot);
        g->launches++;
        if (g->n_rowseg) {
            const unsigned sb = seg_blocks(g);
            k_wgradsum<<<sb, WB, 0, g->st>>>(g->n_rowseg, g->d_rowseg, g->d_adj, g->d_wn, g->d_x, g->d_lam, s,
                                             g->d_rowdot);
            k_wgradseg<<<sb, WB, 0, g->st>>>(g->n_rowseg, g->d_rowseg, g->d_adj, g->d_rowsum, g->d_x, g->d_lam, s,
                                             g->d_rowdot, d_grad_w);
            g->launches += 2;
        }
    }
    EX_CUDA(cudaGetLastError());
    EX_CUDA(cudaStreamSynchronize(g->st));
    return EXCENT_OK;
}

extern "C" int excent_wgraph_lambda(excent_wgraph* g, float* d_out) {
    EX_CHECK_ARG(g && d_out, "bad argument");
    EX_CUDA(cudaSetDevice(g->dev));
    EX_CUDA(cudaMemcpy(d_out, g->d_lam, (size_t)g->n * 4, cudaMemcpyDeviceToDevice));
    return EXCENT_OK;
}

// FP64 Jacobi of x = c0 * t + s * (op) x by pulls: the forward operator pulls
// over the transposed lists, the adjoint over the forward lists.
static int wg_jacobi64(excent_wgraph* g, bool adjoint, double s, double c0, const float* t, double tol, int maxit,
                       double* out_dev_sel) {
    const size_t n = g->n;
    for (auto& p : g->d_v64) if (!p) WG_ALLOC(p, n * 8);
    const unsigned wb = (unsigned)(((long long)n * 32 + WB - 1) / WB);
    // x0 = c0 * t
    EX_CUDA(cudaMemsetAsync(g->d_v64[0], 0, n * 8, g->st));
    double* x = g->d_v64[0];
    double* y = g->d_v64[1];
    const ull* idx = adjoint ? g->d_idx : g->d_idxT;
    const int* adj = adjoint ? g->d_adj : g->d_adjT;
    const double* w = adjoint ? g->d_wn64 : g->d_wt64;
    double rel = 1;
    for (int it = 0; it < maxit && rel > tol; it++) {
        EX_CUDA(cudaMemsetAsync(g->d_mx, 0, 2 * sizeof(ull), g->st));
        k_wpull64<<<wb, WB, 0, g->st>>>(g->n, idx, adj, w, x, t, c0, s, y, g->d_mx);
        ull h[2];
        EX_CUDA(cudaMemcpyAsync(h, g->d_mx, sizeof h, cudaMemcpyDeviceToHost, g->st));
        EX_CUDA(cudaStreamSynchronize(g->st));
        double d, mv;
        memcpy(&d, &h[0], 8);
        memcpy(&mv, &h[1], 8);
        rel = mv > 0 ? d / mv : 0;
        std::swap(x, y);
    }
    if (x != g->d_v64[0]) std::swap(g->d_v64[0], g->d_v64[1]);  // result in d_v64[0]
    (void)out_dev_sel;
    return EXCENT_OK;
}

// Set raw weight of forward edge e to w_e + delta (or restore), renormalising row u in FP64.
static int wg_perturb(excent_wgraph* g, long long e, double delta, int* u_out, std::vector<double>& saved) {
    std::vector<ull> idx(g->n + 1);
    EX_CUDA(cudaMemcpy(idx.data(), g->d_idx, (g->n + 1) * 8, cudaMemcpyDeviceToHost));
    const int u = (int)(std::upper_bound(idx.begin(), idx.end(), (ull)e) - idx.begin()) - 1;
    const ull b = idx[u], d = idx[u + 1] - b;
    std::vector<float> w(d);
    EX_CUDA(cudaMemcpy(w.data(), g->d_wraw + b, d * 4, cudaMemcpyDeviceToHost));
    saved.resize(d);
    EX_CUDA(cudaMemcpy(saved.data(), g->d_wn64 + b, d * 8, cudaMemcpyDeviceToHost));
    std::vector<double> wd(d), q(d);
    double rs = 0;
    for (ull i = 0; i < d; i++) { wd[i] = w[i] + (b + i == (ull)e ? delta : 0.0); rs += wd[i]; }
    for (ull i = 0; i < d; i++) q[i] = wd[i] / rs;
    EX_CUDA(cudaMemcpy(g->d_wn64 + b, q.data(), d * 8, cudaMemcpyHostToDevice));
    std::vector<unsigned> inv(d);
    EX_CUDA(cudaMemcpy(inv.data(), g->d_inv + b, d * 4, cudaMemcpyDeviceToHost));
    for (ull i = 0; i < d; i++) EX_CUDA(cudaMemcpy(g->d_wt64 + inv[i], &q[i], 8, cudaMemcpyDefault));
    *u_out = u;
    return EXCENT_OK;
}

static int wg_restore(excent_wgraph* g, int u, const std::vector<double>& saved) {
    ull b[2];
    EX_CUDA(cudaMemcpy(b, g->d_idx + u, 16, cudaMemcpyDeviceToHost));
    const ull d = b[1] - b[0];
    EX_CUDA(cudaMemcpy(g->d_wn64 + b[0], saved.data(), d * 8, cudaMemcpyHostToDevice));
    std::vector<unsigned> inv(d);
    EX_CUDA(cudaMemcpy(inv.data(), g->d_inv + b[0], d * 4, cudaMemcpyDeviceToHost));
    for (ull i = 0; i < d; i++) EX_CUDA(cudaMemcpy(g->d_wt64 + inv[i], &saved[i], 8, cudaMemcpyDefault));
    return EXCENT_OK;
}

extern "C" int excent_wgraph_loss_fp64(excent_wgraph* g, int kind, double s, const float* d_t, const float* d_c,
                                       long long edge, double delta, double tol, double* loss) {
    EX_CHECK_ARG(g && d_c && loss && (kind == EXCENT_PR || kind == EXCENT_KATZ), "bad argument");
    EX_CHECK_ARG(edge < (long long)g->m, "edge out of range");
    EX_CUDA(cudaSetDevice(g->dev));
    int u = -1;
    std::vector<double> saved;
    if (edge >= 0) EX_TRY(wg_perturb(g, edge, delta, &u, saved));
    const double c0 = kind == EXCENT_PR ? 1.0 - s : 1.0;
    const int rc = wg_jacobi64(g, false, s, c0, d_t, tol, 1000000, nullptr);
    if (edge >= 0) EX_TRY(wg_restore(g, u, saved));
    EX_TRY(rc);
    EX_CUDA(cudaMemsetAsync(g->d_red, 0, 8, g->st));
    k_wdot64<<<g->sms * 8, WB, 0, g->st>>>(g->n, g->d_v64[0], d_c, g->d_red);
    EX_CUDA(cudaMemcpyAsync(loss, g->d_red, 8, cudaMemcpyDeviceToHost, g->st));
    EX_CUDA(cudaStreamSynchronize(g->st));
    return EXCENT_OK;
}

extern "C" int excent_wgraph_grad_fp64(excent_wgraph* g, int kind, double s, const float* d_t, const float* d_c,
                                       double tol, double* grad_t, double* grad_w) {
    EX_CHECK_ARG(g && d_c && (kind == EXCENT_PR || kind == EXCENT_KATZ), "bad argument");
    EX_CUDA(cudaSetDevice(g->dev));
    const size_t n = g->n;
    const double c0 = kind == EXCENT_PR ? 1.0 - s : 1.0;
    EX_TRY(wg_jacobi64(g, false, s, c0, d_t, tol, 1000000, nullptr));
    double* xf = nullptr;
    WG_ALLOC(xf, n * 8);
    EX_CUDA(cudaMemcpy(xf, g->d_v64[0], n * 8, cudaMemcpyDeviceToDevice));
    int rc = wg_jacobi64(g, true, s, 1.0, d_c, tol, 1000000, nullptr);
    double* gw = nullptr;
    if (rc == EXCENT_OK && grad_t) {
        std::vector<double> lam(n);
        cudaMemcpy(lam.data(), g->d_v64[0], n * 8, cudaMemcpyDeviceToHost);
        for (size_t v = 0; v < n; v++) grad_t[v] = (kind == EXCENT_PR ? 1.0 - s : 1.0) * lam[v];
    }
    if (rc == EXCENT_OK && grad_w && g->m) {
        if (cudaMalloc(&gw, g->m * 8) != cudaSuccess) { cudaGetLastError(); set_error("grad buffer"); rc = EXCENT_ERR_NOMEM; }
        else {
            const unsigned wb = (unsigned)(((long long)n * 32 + WB - 1) / WB);
            k_wgrad64<<<wb, WB, 0, g->st>>>(g->n, g->d_idx, g->d_adj, g->d_wn64, g->d_rowsum, xf, g->d_v64[0], s, gw);
            if (cudaMemcpyAsync(grad_w, gw, g->m * 8, cudaMemcpyDeviceToHost, g->st) != cudaSuccess ||
                cudaStreamSynchronize(g->st) != cudaSuccess) { set_error("grad copy failed"); rc = EXCENT_ERR_CUDA; }
        }
    }
    cudaFree(xf);
    if (gw) cudaFree(gw);
    return rc;
}

extern "C" int excent_wgraph_stream(excent_wgraph* g, void** stream) {
    EX_CHECK_ARG(g && stream, "null argument");
    *stream = (void*)g->st;
    return EXCENT_OK;
}

// Move the transposed lists and weights to pinned, device-mapped host memory:
// the adjoint push then reads them in place over the host link (zero copy),
// the way the engine's host cache serves graphs larger than device memory.
extern "C" int excent_wgraph_host_transposed(excent_wgraph* g) {
    EX_CHECK_ARG(g, "null graph");
    if (g->host_t || g->m == 0) return EXCENT_OK;
    EX_CUDA(cudaSetDevice(g->dev));
    EX_CUDA(cudaDeviceSynchronize());
    const unsigned fl = cudaHostAllocMapped | cudaHostAllocPortable;
    int* ha = nullptr;
    float* hw = nullptr;
    double* hw64 = nullptr;
    if (cudaHostAlloc((void**)&ha, g->m * 4, fl) != cudaSuccess || cudaHostAlloc((void**)&hw, g->m * 4, fl) != cudaSuccess ||
        cudaHostAlloc((void**)&hw64, g->m * 8, fl) != cudaSuccess) {
        cudaGetLastError();
        if (ha) cudaFreeHost(ha);
        if (hw) cudaFreeHost(hw);
        if (hw64) cudaFreeHost(hw64);
        EX_FAIL(EXCENT_ERR_NOMEM, "pinned host copy of the transposed graph does not fit");
    }
    EX_CUDA(cudaMemcpy(ha, g->d_adjT, g->m * 4, cudaMemcpyDeviceToHost));
    EX_CUDA(cudaMemcpy(hw, g->d_wt, g->m * 4, cudaMemcpyDeviceToHost));
    EX_CUDA(cudaMemcpy(hw64, g->d_wt64, g->m * 8, cudaMemcpyDeviceToHost));
    cudaFree(g->d_adjT);
    cudaFree(g->d_wt);
    cudaFree(g->d_wt64);
    g->h_adjT = ha; g->h_wt = hw; g->h_wt64 = hw64;
    EX_CUDA(cudaHostGetDevicePointer((void**)&g->d_adjT, ha, 0));
    EX_CUDA(cudaHostGetDevicePointer((void**)&g->d_wt, hw, 0));
    EX_CUDA(cudaHostGetDevicePointer((void**)&g->d_wt64, hw64, 0));
    g->host_t = true;
    return EXCENT_OK;
}
