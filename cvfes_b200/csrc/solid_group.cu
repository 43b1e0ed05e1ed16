// Group step: the template step for few samples or a small wall (step variant 6 where the
// patch kernel of solid_patch.cu would leave most lanes, or most of the chip, idle).
//
// A thread owns one node and V samples; the lanes of a warp hold as many nodes as the
// samples leave room for.  These problems live in L2, so a step costs its chain of
// dependent loads and the launch itself, not bandwidth: slot pointers -> slot records ->
// rows.  The chain is cut in two ways:
//   * everything that the steps do not write (slot pointers, records and stiffness rows
//     into shared memory, then the elements' coefficients and the inverse mass into
//     registers) is read before the kernel waits for the step before it (programmatic
//     dependent launch), under that step's tail;
//   * after the wait all rows of u and u_{n-1} that the node needs are requested at once.
// A block holds 64 threads' nodes; their slots are contiguous, so staging is coalesced.
// The register cost of the burst (up to nine rows of three vectors) allows 1 FP64 or 2
// FP32 samples a thread.  Bits as the other step kernels: the same products in the same
// order.
//
// 64 x 128 wall, 8 samples: FP64 8.4 -> 4.1 us a step, FP32 6.1 -> 3.5 us (graph replays);
// 128 x 400 wall, FP32: 8 samples 14.7 -> 11.1 us, 16 samples 21.5 -> 19.3 us, 3 samples
// 16.5 -> 9.3 us; FP64, 8 samples 48 -> 30 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "step_core.cuh"

namespace cvfes {

constexpr int kGroupThreads = 64;  // FP64 64 x 128 wall, 8 samples: 4.25 us at 128, 4.64 at 256
constexpr int kGroupDegree = 8;  // slots of a node held in registers

template <typename T, int V, bool VEL, int MAXD, bool FULL>
__global__ void __launch_bounds__(kGroupThreads, MAXD <= 6 ? 8 : 6)
    k_step_group(StepArgs<T> A) {
    extern __shared__ __align__(16) unsigned char smem[];
    using P = SlotStage<T, FULL>;
    constexpr int kStep = P::kSlotBytes / (int)sizeof(T);
    const int a0 = blockIdx.x * A.npb, n_nodes = (int)A.n_nodes;
    const int a1 = min(a0 + A.npb, n_nodes);
    const int kb = __ldg(A.node_ptr + a0), nsl = __ldg(A.node_ptr + a1) - kb;
    const int t = threadIdx.x / A.tpn, a = a0 + t;
    const int vec = threadIdx.x - t * A.tpn;
    const bool active = t < A.npb && a < n_nodes;
    int k0 = 0, deg = 0;
    if (active) {
        k0 = __ldg(A.node_ptr + a) - kb;
        deg = __ldg(A.node_ptr + a + 1) - kb - k0;
    }
    // a block whose slots do not fit the stage forms its rows from global memory
    const int all = deg;
    const bool staged = nsl <= A.cap_slots;
    if (!staged) deg = 0;
    int4* const srec = reinterpret_cast<int4*>(smem);
    unsigned char* const sslab = smem + (size_t)A.cap_slots * 16;
    const char* const rec = reinterpret_cast<const char*>(A.rec + kb);
    const char* const slab = reinterpret_cast<const char*>(A.slab + (size_t)kb * kSlabStride);
    for (int q = threadIdx.x; q < nsl && staged; q += kGroupThreads)
        cp_async<16>(smem_u32(srec) + 16 * q, rec + 16 * q);
    cp_async_commit();
    for (int q = threadIdx.x; q < P::kWords * nsl && staged; q += kGroupThreads) {
        const int s = q / P::kWords, w = q - s * P::kWords;
        cp_async<16>(smem_u32(sslab) + 16 * q,
                     slab + s * (kSlabStride * (int)sizeof(T)) + (P::kFirst + w) * 16);
    }
    cp_async_commit();
    grid_dependency_release();
    const uint32_t rowb = (uint32_t)A.S * sizeof(T), nodeb = 3 * rowb;
    const size_t S = (size_t)A.S, col = (size_t)vec * V;
    const bool free_row = active && a >= A.n_clamped;
    Vec<T, V> im = vzero<T, V>();
    T fh[3] = {T(0), T(0), T(0)};
    if (free_row) {
        im = ldg<T, V>(row_at(A.invm + col, a, rowb));
#pragma unroll
        for (int d = 0; d < 3; ++d) fh[d] = __ldg(A.fhat + 4 * (size_t)a + d);
    }
    cp_async_wait_group<1>();
    __syncthreads();
    Vec<T, V> C[MAXD];
    if (free_row) {
#pragma unroll
        for (int j = 0; j < MAXD; ++j)
            if (j < deg) C[j] = ldg<T, V>(row_at(A.coef + col, srec[k0 + j].x, rowb));
    }
    cp_async_wait_all();
    __syncthreads();
    grid_dependency_wait();
    if (!active) return;
    T* const un = row_at(A.un + col, a, nodeb);
    if (!free_row) {
        clamp_store<T, V>(A, S, (size_t)a * 3 * S + col);
        return;
    }
    const T* const u = A.u + col;
    Vec<T, V> ua[3], vo[3], R[MAXD + 1][3], acc[3];
    auto rows = [&](Vec<T, V> (&x)[3], const T* q) {
#pragma unroll
        for (int d = 0; d < 3; ++d) x[d] = ld<T, V>(q + d * S);
    };
    rows(ua, row_at(u, a, nodeb));
    if (deg > 0) rows(R[0], row_at(u, srec[k0].y, nodeb));
#pragma unroll
    for (int j = 0; j < MAXD; ++j)
        if (j < deg) rows(R[j + 1], row_at(u, srec[k0 + j].z, nodeb));
    {
        const T* q = row_at(A.up + col, a, nodeb);
#pragma unroll
        for (int d = 0; d < 3; ++d) vo[d] = ld_state<T, V, true>(q + d * S);
    }
    const T p = step_pressure<T>(A);
    const T* const K = reinterpret_cast<const T*>(sslab) - 16 / (int)sizeof(T) * P::kFirst +
                       (size_t)k0 * kStep;
#pragma unroll
    for (int d = 0; d < 3; ++d) acc[d] = vzero<T, V>();
    if (deg > 0) to_diff<T, V, FULL>(R[0], ua);
#pragma unroll
    for (int j = 0; j < MAXD; ++j) {
        if (j < deg) {
            to_diff<T, V, FULL>(R[j + 1], ua);
            if (j > 0 && !(srec[k0 + j].w & 1)) {  // fan break: a first neighbour of its own
                Vec<T, V> b[3];
                rows(b, row_at(u, srec[k0 + j].y, nodeb));
                to_diff<T, V, FULL>(b, ua);
                slot_fma<T, V, FULL>(K + kStep * j, C[j], b, R[j + 1], ua, acc);
            } else {
                slot_fma<T, V, FULL>(K + kStep * j, C[j], R[j], R[j + 1], ua, acc);
            }
        }
    }
    if (deg > MAXD) {  // the elements that the registers do not hold, one after another
        Vec<T, V> x1[3], x2[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) x1[d] = R[MAXD][d];
        for (int j = MAXD; j < deg; ++j) {
            const int4 r = srec[k0 + j];
            rows(x2, row_at(u, r.z, nodeb));
            const Vec<T, V> c = ldg<T, V>(row_at(A.coef + col, r.x, rowb));
            if (!(r.w & 1)) {
                rows(x1, row_at(u, r.y, nodeb));
                to_diff<T, V, FULL>(x1, ua);
            }
            to_diff<T, V, FULL>(x2, ua);
            slot_fma<T, V, FULL>(K + kStep * j, c, x1, x2, ua, acc);
#pragma unroll
            for (int d = 0; d < 3; ++d) x1[d] = x2[d];
        }
    }
    if (!staged)
        ku_row_unstaged<T, V, FULL>(A.rec + kb + k0, A.slab + (size_t)(kb + k0) * kSlabStride, all, u,
                              A.coef + col, rowb, ua, acc);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        T f = p * fh[d];
        if (A.trac) f += __ldg(A.trac + 4 * (size_t)a + d);
        Vec<T, V> o, vn;
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const T dv = VEL ? vo[d].v[i] : ua[d].v[i] - vo[d].v[i];
            const T w = A.w0 * im.v[i];
            const T v = fma(w, f - acc[d].v[i], fma(-row_eta(A, im.v[i]), dv, dv));
            const bool live = im.v[i] != T(0);
            o.v[i] = live ? ua[d].v[i] + v : T(0);
            vn.v[i] = live ? v : -ua[d].v[i];
        }
        stcs<T, V>(un + d * S, o);
        if constexpr (VEL) stcs<T, V>(row_at(A.vel + col, a, nodeb) + d * S, vn);
    }
}

template <typename T, int V, bool VEL, int MAXD, bool FULL>
static int launch_group_k(const StepArgs<T>& A, bool after_step, cudaStream_t st) {
    auto kernel = k_step_group<T, V, VEL, MAXD, FULL>;
    const size_t smem = (size_t)A.cap_slots * SlotStage<T, FULL>::kBytes;
    int per_sm = 0;  // also sets the shared-memory attribute
    const int rc =
        fanp_blocks_per_sm(reinterpret_cast<const void*>(kernel), kGroupThreads, smem, &per_sm);
    if (rc) return rc;
    const long long blocks = (A.n_nodes + A.npb - 1) / A.npb;
    return launch_step_kernel(kernel, dim3((unsigned)blocks), kGroupThreads, smem, after_step, st, "k_step_group",
                              A);
}

// Taken for at most 16 sample vectors a node (2 FP32 samples each from 8 samples on), or 20
// single samples: there the patch kernel leaves half its lanes idle.  Either side of the
// line, 128 x 400 wall, us a step, group / patch: FP32 16 samples 19.3 / 44.1, 32 samples
// 43.2 / 50.2, 64 samples 87 / 57; FP64 16 samples 55.3 / 67.8, 25 samples 92 / 63.
// Below 8 FP32 samples one a thread is the faster (4 samples: 8.4 against 10.1 us).
// Any number of elements a node: a Delaunay sheet of 20,000 nodes with up to 18, us a step,
// group / patch: FP32 1 sample 5.4 / 21.7, 8 samples 9.5 / 21.3, 32 samples 19.3 / 21.7; FP64
// 8 samples 12.3 / 28.2, 16 samples 20.9 / 28.8.
template <typename T>
int launch_step_group(const cvfes_solid_mesh* m, StepArgs<T> A, int vec_max, bool after_step,
                      cudaStream_t st) {
    const int V = sizeof(T) == 4 && vec_max >= 2 && A.S >= 8 ? 2 : 1;
    const int sv = A.S / V;
    const bool full = mesh_full<T>(m);
    if (m->max_degree <= 0 || sv > (V == 2 ? 16 : 20) || m->n_nodes >= INT32_MAX / 2) return 1;
    A.tpn = sv;
    A.nch = 1;
    // at most 36 KB of slots: six blocks share an SM (one or two samples only).  A few nodes
    // of more elements than the registers hold fit beside the others (six a node on average)
    const int deg = (int)std::min<long long>(m->max_degree, kGroupDegree);
    const int fit = (int)(36 * 1024 / (deg * (full ? SlotStage<T, true>::kBytes : SlotStage<T>::kBytes)));
    A.npb = std::min(kGroupThreads / A.tpn, fit);
    A.cap_slots = A.npb * deg + (int)std::min<long long>(m->max_degree - deg, 24);
#define CVFES_GROUP(VV, FULL)                                                                  \
    if (m->max_degree <= 6)                                                                    \
        return A.vel ? launch_group_k<T, VV, true, 6, FULL>(A, after_step, st)                 \
                     : launch_group_k<T, VV, false, 6, FULL>(A, after_step, st);               \
    return A.vel ? launch_group_k<T, VV, true, kGroupDegree, FULL>(A, after_step, st)          \
                 : launch_group_k<T, VV, false, kGroupDegree, FULL>(A, after_step, st);
    if constexpr (sizeof(T) == 4) {
        if (V == 2) {
            CVFES_GROUP(2, false)
        }
    } else if (full) {
        CVFES_GROUP(1, true)
    }
    CVFES_GROUP(1, false)
#undef CVFES_GROUP
}

template int launch_step_group<float>(const cvfes_solid_mesh*, StepArgs<float>, int, bool,
                                      cudaStream_t);
template int launch_step_group<double>(const cvfes_solid_mesh*, StepArgs<double>, int, bool,
                                       cudaStream_t);

}  // namespace cvfes
