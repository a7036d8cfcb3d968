// pull.cu -- the segment table of a graph's long lists (pull.cuh).
#include "pull.cuh"

namespace excent {

__global__ void k_list_segs(int n, const ull* idx, ListSeg* out, ull* cnt) {
    for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < n; u += (long long)gridDim.x * blockDim.x) {
        const ull b = idx[u], deg = idx[u + 1] - b;
        if (deg <= PULL_LONG) continue;
        const ull k = (deg + PULL_SEG - 1) / PULL_SEG, at = atomicAdd(cnt, k);
        if (!out) continue;
        for (ull i = 0; i < k; i++)
            out[at + i] = ListSeg{b + i * PULL_SEG, (unsigned)min((ull)PULL_SEG, deg - i * PULL_SEG), (unsigned)u};
    }
}

}  // namespace excent
