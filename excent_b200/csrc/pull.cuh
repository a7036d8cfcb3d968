// pull.cuh -- sums over adjacency lists: the gather form of a pass.
//
// Where a pass touches most of the graph, gathering the pushed weights along
// the lists beats scattering them: on a B200 the lists of an R-MAT graph of
// 263M entries gather at 326 G entries/s (279 G/s with a float4 per entry)
// and scatter at 93 (80): reductions to the same few high-degree vertices
// serialise in L2, while gathers of the same vertices hit in L1 and share its
// lookups (lookups alone, one an entry, would be 284 G/s).
#pragma once
#include <cuda_runtime.h>

#include "device.cuh"

namespace excent {

// Longer lists are read as segments, one warp each, of PULL_SEG entries. The
// line lies where a tile of 32 lists cannot hold one warp up: forward and
// adjoint solve of a weighted R-MAT of 16.8M entries took 23.2 + 12.7 ms with
// lists of up to 256 entries left in the tiles, 14.4 + 7.8 with 128, 11.8 + 7.1
// with 64 and 11.6 + 6.8 with 32.
static constexpr unsigned PULL_LONG = 32;
static constexpr unsigned PULL_SEG = 512;

// One stretch of a list longer than PULL_LONG.
struct ListSeg {
    ull base;
    unsigned len, row;
};

// Per warp: the nonempty lists of a tile, compacted.
template <typename T> struct PullScratch {
    ull base[32];
    unsigned ex[32];
    T acc[32];
};

// Each lane's sum of f over its list [b, b + ds), ds <= PULL_LONG. f.key(e)
// loads what entry e names, f.value(key) gathers its value (0 for a default
// key). The tile's lists are laid end to end and every lane takes one entry of
// each 32-entry window, summed per list by a segmented scan, so short lists (5
// entries on average on the R-MAT graphs) keep every lane busy.
template <typename T, typename F>
__device__ __forceinline__ T warp_window_sums(ull b, unsigned ds, const F& f, PullScratch<T>& s, int lane) {
    const unsigned nz = __ballot_sync(FULL, ds != 0);
    if (!nz) return T(0);
    const unsigned incl = warp_incl_scan(ds, lane);
    const unsigned tot = __shfl_sync(FULL, incl, 31);
    const unsigned ex = incl - ds;
    const int rank = __popc(nz & ((1u << lane) - 1u));
    if (ds) { s.base[rank] = b; s.ex[rank] = ex; s.acc[rank] = T(0); }
    __syncwarp();
    const unsigned le = lane == 31 ? FULL : (2u << lane) - 1u;
    constexpr int W = 4;   // windows in flight
    for (unsigned j0 = 0; j0 < tot; j0 += 32 * W) {
        typename F::Key key[W];
        unsigned starts[W];
        int own[W];
#pragma unroll
        for (int q = 0; q < W; q++) {
            const unsigned wb = j0 + 32 * q, j = wb + lane;
            starts[q] = __reduce_or_sync(FULL, (ds && ex >= wb && ex - wb < 32) ? 1u << (ex - wb) : 0u);
            own[q] = __popc(__ballot_sync(FULL, ds && ex <= wb)) - 1 + __popc(starts[q] & le & ~1u);
            key[q] = typename F::Key{};
            if (j < tot) key[q] = f.key(s.base[own[q]] + (j - s.ex[own[q]]));
        }
        T val[W];
#pragma unroll
        for (int q = 0; q < W; q++) val[q] = f.value(key[q]);
#pragma unroll
        for (int q = 0; q < W; q++) {
            const unsigned j = j0 + 32 * q + lane;
            if (j0 + 32 * q >= tot) break;
            const int first = 31 - __clz((starts[q] & le) | 1u);   // where this lane's list starts in the window
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const T up = shfl_up(val[q], o);
                if (lane - o >= first) val[q] += up;
            }
            const bool last = lane == 31 || j + 1 >= tot || ((starts[q] >> (lane + 1)) & 1u);
            if (j < tot && last) s.acc[own[q]] += val[q];
            __syncwarp();
        }
    }
    const T sum = ds ? s.acc[rank] : T(0);
    __syncwarp();
    return sum;
}

// Each lane's sum of f over its list [b, b + ds), ds <= PULL_LONG (TINY: at
// most 8). f.key(e) loads what entry e names, f.value(key) gathers its value (0
// for a default key). Eight lanes walk a list, four lists at a time and R such
// rounds in flight: on lists of 5 to 7 entries that keeps half of the lanes
// busy for less than half the instructions of a segmented scan over the
// concatenated lists (15 shuffles and as many additions per 32 float4
// entries). A batch of 4 R lists takes a gather's latency for every eight
// entries of its longest one, so lists of at most 8 entries go apart.
template <typename T, bool TINY, typename O, typename F>
__device__ __forceinline__ T warp_list_sums(O b, unsigned ds, const F& f, int lane) {
    constexpr int R = TINY ? 8 : 4;
    T mine = T(0);
    if (!__any_sync(FULL, ds)) return mine;
    const int sub = lane >> 3, l8 = lane & 7;
#pragma unroll 1
    for (int t = 0; t < 8; t += R) {   // R rounds of four lists in flight
        O bb[R];
        unsigned dd[R], most = 0;
        T acc[R];
        typename F::Key key[R];
#pragma unroll
        for (int k = 0; k < R; k++) {
            const int src = (t + k) * 4 + sub;
            bb[k] = __shfl_sync(FULL, b, src);
            dd[k] = __shfl_sync(FULL, ds, src);
            most = max(most, dd[k]);
            acc[k] = T(0);
            key[k] = typename F::Key{};
            if ((unsigned)l8 < dd[k]) key[k] = f.key(bb[k] + l8);
        }
        if constexpr (TINY) {
#pragma unroll
            for (int k = 0; k < R; k++) acc[k] = f.value(key[k]);
        } else {
            most = __reduce_max_sync(FULL, most);
            for (unsigned j = 8; j < most + 8; j += 8) {   // the next entries' keys are loaded ahead
                typename F::Key next[R];
#pragma unroll
                for (int k = 0; k < R; k++) {
                    next[k] = typename F::Key{};
                    if (j + l8 < dd[k]) next[k] = f.key(bb[k] + j + l8);
                }
#pragma unroll
                for (int k = 0; k < R; k++) {
                    acc[k] += f.value(key[k]);
                    key[k] = next[k];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < R; k++) {
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) acc[k] += shfl_xor(acc[k], o);
            const T v = shfl(acc[k], (lane & 3) * 8);   // list 4 * (t + k) + s is summed by lanes 8 s .. 8 s + 7
            if ((lane >> 2) == t + k) mine = v;
        }
    }
    return mine;
}

// The warp's sums of f over two segments (valid in lane 0).
template <typename T, typename F>
__device__ __forceinline__ void warp_segment_sums(const ListSeg& g0, const ListSeg& g1, const F& f, int lane, T& a0,
                                                  T& a1) {
    a0 = T(0);
    a1 = T(0);
    for (unsigned j = lane; j < max(g0.len, g1.len); j += 128) {
        typename F::Key k0[4], k1[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            k0[q] = typename F::Key{};
            k1[q] = typename F::Key{};
            if (j + 32 * q < g0.len) k0[q] = f.key(g0.base + j + 32 * q);
            if (j + 32 * q < g1.len) k1[q] = f.key(g1.base + j + 32 * q);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            a0 += f.value(k0[q]);
            a1 += f.value(k1[q]);
        }
    }
    a0 = warp_sum(a0);
    a1 = warp_sum(a1);
}

// One gather phase of a persistent kernel over the lists [idx[v], idx[v + 1])
// of every v < n: add(v, sum) once per short list and once per segment of a
// long one (then from several warps). Blocks share the work in a fixed
// interleaved split, pairs of segments before tiles of 32 short lists, and a
// block's warps claim it from s_next (0 when the phase begins): with a fixed
// split between warps too, a third of all warp time was waiting for the
// slowest at the barrier. A warp loads its next segment records ahead: a
// segment is a chain of three dependent loads.
template <typename T, typename F, typename A>
__device__ __forceinline__ void gather_phase(int n, const ull* idx, const ListSeg* seg, ull nseg, const F& f, const A& add,
                                             unsigned* s_next, PullScratch<T>& S, int lane) {
    const ull npairs = (nseg + 1) / 2, ntiles = ((ull)n + 31) / 32;
    constexpr ListSeg none{0, 0, 0};
    auto claim = [&]() -> ull {
        unsigned k = 0;
        if (lane == 0) k = atomicAdd(s_next, 1u);
        return (ull)__shfl_sync(FULL, k, 0) * gridDim.x + blockIdx.x;
    };
    ull i = claim();
    ListSeg g0 = i < npairs ? seg[2 * i] : none, g1 = 2 * i + 1 < nseg ? seg[2 * i + 1] : none;
    while (i < npairs) {
        const ull next = claim();
        const ListSeg n0 = next < npairs ? seg[2 * next] : none, n1 = 2 * next + 1 < nseg ? seg[2 * next + 1] : none;
        T a0, a1;
        warp_segment_sums<T>(g0, g1, f, lane, a0, a1);
        if (lane == 0) {
            add(g0.row, a0, true);
            if (g1.len) add(g1.row, a1, true);
        }
        i = next; g0 = n0; g1 = n1;
    }
    for (; i - npairs < ntiles; i = claim()) {
        const long long v = (long long)(i - npairs) * 32 + lane;
        ull b = 0;
        unsigned ds = 0;
        if (v < n) {
            b = idx[v];
            const ull dv = idx[v + 1] - b;
            ds = dv > PULL_LONG ? 0u : (unsigned)dv;
        }
        if (!__any_sync(FULL, ds)) continue;
        const T t = warp_window_sums<T>(b, ds, f, S, lane);
        if (ds) add((unsigned)v, t, false);
    }
}

// The lists longer than PULL_LONG as segments, in any order (out null: their number alone).
__global__ void k_list_segs(int n, const ull* idx, ListSeg* out, ull* cnt);
// At most this many segments in a graph of m entries.
static inline ull list_seg_cap(ull m) { return m / PULL_SEG + m / PULL_LONG + 1; }

}  // namespace excent
