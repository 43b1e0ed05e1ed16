// What the kernels with free-running warps share (solid_patch.cu, solid_geo.cu,
// solid_adjoint.cu): the order in which a block's warps visit the nodes, and the prefetch of
// rows into L2 by cache lines.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "step_core.cuh"

namespace cvfes {

constexpr int kPatchWarps = 16;

// Node order: patches of L x (W / L) nodes, W warps a block, over rows of R nodes after the
// clamped prefix, patch after patch along a strip of W / L rows.
struct PatchMap {
    int R, L, tps, n_strips;
};

// Patch shape for a mesh of this bandwidth: rows of bandwidth - 1 nodes (the distance to
// the next mesh row in a row-by-row numbering).  A strip that the mesh does not fill, or a
// run that a row does not fill, idles warps, so four rows are taken while at most an eighth
// of the places are empty, else two, else runs of W nodes (any numbering; what locality is
// left is that of consecutive nodes).
inline PatchMap patch_map(long long n_free, long long bandwidth, int W = kPatchWarps) {
    PatchMap m;
    const long long R = bandwidth - 1;
    for (int J = 4; J >= 2; J /= 2) {
        const int L = W / J;
        if (R < L || R > n_free / J) continue;
        m.R = (int)R;
        m.L = L;
        m.tps = (int)((R + L - 1) / L);
        m.n_strips = (int)((n_free + J * R - 1) / (J * R));
        if ((long long)m.n_strips * m.tps * W * 8 <= n_free * 9) return m;
    }
    m.R = (int)std::max(n_free, 1LL);
    m.L = W;
    m.tps = (int)((m.R + W - 1) / W);
    m.n_strips = n_free > 0 ? 1 : 0;
    return m;
}

// A warp's walk over its nodes: place (wj, wi) of every patch that its block takes, blocks
// (of one sample chunk) striding over the patches.
struct PatchWalk {
    int strip, tile, dstrip, dtile, wj, wi, J, first, n_nodes;
    __device__ __forceinline__ PatchWalk(const PatchMap& M, int warp, int block, int blocks,
                                         int first_, int n_nodes_, int W = kPatchWarps) {
        J = W / M.L;
        wj = warp / M.L;
        wi = warp - wj * M.L;
        dstrip = blocks / M.tps;
        dtile = blocks - dstrip * M.tps;
        strip = block / M.tps;
        tile = block - strip * M.tps;
        first = first_;
        n_nodes = n_nodes_;
    }
    __device__ __forceinline__ bool more(const PatchMap& M) const { return strip < M.n_strips; }
    __device__ __forceinline__ int node(const PatchMap& M) const {  // -1: none at this place
        const int c = tile * M.L + wi;
        const int b = first + (strip * J + wj) * M.R + c;
        return strip < M.n_strips && c < M.R && b < n_nodes ? b : -1;
    }
    __device__ __forceinline__ void advance(const PatchMap& M) {
        strip += dstrip;
        tile += dtile;
        if (tile >= M.tps) {
            tile -= M.tps;
            ++strip;
        }
    }
};

// Lines of a chunk's rows (32 * V samples): lane l takes line l % kLines of row l / kLines.
template <typename T, int V>
struct RowLines {
    static constexpr int kRow = 32 * V * (int)sizeof(T), kLines = kRow / 128;
    static constexpr int kRows = 32 / kLines;  // rows of one warp-wide prefetch
    int row;
    size_t off;  // byte offset of the lane's line in a row
    bool on;     // the row reaches that far
    __device__ __forceinline__ RowLines(int lane, int chunk, uint32_t rowb) {
        row = lane / kLines;
        off = (size_t)chunk * kRow + (lane % kLines) * 128;
        on = off < rowb;
    }
};

// Slots of node b.  A node with more than the descriptor's max_degree, for which the stages
// are sized, is left out (b = -1) and the warp's flag (shared memory) set: such nodes follow
// after the loop, from global memory.
__device__ __forceinline__ void node_slots(const int32_t* node_ptr, int max_degree, int* flag,
                                           int& b, int& k0, int& n) {
    k0 = n = 0;
    if (b >= 0) {
        k0 = __ldg(node_ptr + b);
        n = __ldg(node_ptr + b + 1) - k0;
        if (n > max_degree) {
            *flag = 1;
            b = -1;
            n = 0;
        }
    }
}

// The launch read again, opaque to the compiler: what follows from it (after a long loop) is
// computed anew and holds no registers during the loop.
struct LaunchAgain {
    int block, blocks, thread;
    __device__ __forceinline__ LaunchAgain() {
        asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(block));
        asm volatile("mov.u32 %0, %%nctaid.x;" : "=r"(blocks));
        asm volatile("mov.u32 %0, %%tid.x;" : "=r"(thread));
    }
};

}  // namespace cvfes
