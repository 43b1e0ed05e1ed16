// Discrete adjoint of the explicit membrane time step for a displacement-mismatch
// objective, with respect to per-element, per-sample log E and log h.
//
// Forward step n (n = 0 .. T-1), free rows, W = w0 * inverse lumped mass:
//     u_{n+1} = u_n + (1 - eta)(u_n - u_{n-1}) + W (p_n fhat - K(c) u_n),   K(c) = sum_e c_e Khat_e
// clamped rows hold the clamp value, c_e = E_e h_e, and the objective is
//     J_s = sum_{n in O} sum_{i in obs} |u_n(i) - uobs_n(i)|^2,   O = {n : n % obs_every == 0, n > 0}.
// With chi_n = W mu_n (mu the adjoint of u_n, zero on clamped rows) the reverse
// recursion has the form of the forward step:
//     chi_n = chi_{n+1} + (1 - eta)(chi_{n+1} - chi_{n+2}) - W K chi_{n+1} + W dJ/du_n
// and the gradients are
//     dJ/dlogE_e = -c_e Gamma_e,   Gamma_e = sum_n chi_{n+1,e}^T Khat_e u_{n,e}
//     dJ/dlogh_e = -c_e Gamma_e - h_e sum_{a in e} alpha_{e,a} invm_a G_a,   G_a = sum_n chi_{n+1,a} . r_{n,a}
// with r_n = p_n fhat - K u_n and alpha_{e,a} the element's lumped-mass weight of node a
// (m_a = sum_e h_e alpha_{e,a}).  The damping is mass-proportional, so eta does not
// depend on the material.
//
// States u_n are not stored: the reverse sweep runs the forward step backwards,
//     u_{n-1} = u_n - ((u_{n+1} - u_n) - W r_n) / (1 - eta),
// in the same kernel that advances chi, and replaces the reconstructed pair by the
// exact pair (u_m, u_{m+1}) saved by the forward pass at every checkpoint m (every
// ckpt_every steps), so the reconstruction drift never spans more than one segment.
// Both recursions share one pass over the node's slots: the fan-ordered slot rows of
// Khat are applied to u_n and chi_{n+1}, and the slot of each element's local node 0
// (its owner) also evaluates the element's bilinear form from the difference
// vectors (u_b - u_a, chi_b - chi_a), which needs only the blocks K_b1b1, K_b1b2,
// K_b2b2 of that slot's two neighbours (rigid translations are in Khat's null space).
// Every element and node accumulator is written by one thread: no atomics.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "patch_walk.cuh"
#include "step_core.cuh"

namespace cvfes {

constexpr int kObsChunk = 16;   // observation nodes per block of the mismatch kernel
constexpr int kOwnStride = 28;  // K_b1b1 (9), K_b1b2 (9), K_b2b2 (9), pad

struct MassWeights {
    double w[9];  // w[3a + g]: lumped-mass weight of local node a at quadrature point g
};

// Owner-slot neighbour blocks of every element, in the owner slot's (b1, b2) order,
// stored at the owner slot (the slot of the element's local node 0); the entries of the
// other slots are not used.
template <typename T>
__global__ void k_owner_blocks(long long n_elems, const int32_t* __restrict__ elems,
                               const int32_t* __restrict__ elem_slot,
                               const int32_t* __restrict__ slot_rec, const T* __restrict__ slab,
                               T* __restrict__ own) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= n_elems) return;
    const int s0 = elem_slot[3 * e];
    const int b1 = slot_rec[4 * s0 + 1], b2 = slot_rec[4 * s0 + 2];
    const int l1 = elems[3 * e + 1] == b1 ? 1 : 2;
    const int s1 = elem_slot[3 * e + l1], s2 = elem_slot[3 * e + 3 - l1];
    const int q = slot_rec[4 * s1 + 1] == b2 ? 1 : 2;  // block of b2 in b1's slot
    T* o = own + (size_t)kOwnStride * s0;
    const T* k1 = slab + (size_t)kSlabStride * s1;
    const T* k2 = slab + (size_t)kSlabStride * s2;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        o[i] = k1[i];
        o[9 + i] = k1[9 * q + i];
        o[18 + i] = k2[i];
    }
    o[27] = T(0);
}

// coef = E*h and thickness h from the log-material of each element and sample.
__global__ void k_material_log(long long n, const double* __restrict__ logE,
                               const double* __restrict__ logh, double* __restrict__ coef64,
                               float* __restrict__ coef32, double* __restrict__ thick) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double h = exp(logh[i]);
    const double c = exp(logE[i]) * h;
    if (coef64) coef64[i] = c;
    if (coef32) coef32[i] = (float)c;
    if (thick) thick[i] = h;
}

// Observation step k: either record u at the observation nodes, or add the squared
// mismatch of this block's observation nodes into jpart[k][block][s].
template <typename T>
__global__ void k_obs(int n_obs, int S, const int32_t* __restrict__ obs_nodes,
                      const T* __restrict__ u, T* __restrict__ obs_k, double* __restrict__ jpart_k,
                      int record) {
    const int s = blockIdx.y * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const int i0 = blockIdx.x * kObsChunk;
    const int i1 = min(n_obs, i0 + kObsChunk);
    double acc = 0.0;
    for (int i = i0; i < i1; ++i) {
        const size_t a = (size_t)obs_nodes[i];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const T v = u[(3 * a + c) * S + s];
            const size_t o = ((size_t)i * 3 + c) * S + s;
            if (record) {
                obs_k[o] = v;
            } else {
                const double d = (double)v - (double)obs_k[o];
                acc = fma(d, d, acc);
            }
        }
    }
    if (!record) jpart_k[(size_t)blockIdx.x * S + s] = acc;
}

// J[s] = sum over observation steps and node blocks, in a fixed order: group g of a block adds
// parts g, g + kReduceGroups, ..., the groups' sums are added in order (one thread a sample
// summing all parts took 40 us for 320 parts, one dependent addition after another).
constexpr int kReduceSamples = 32, kReduceGroups = 16;
__global__ void __launch_bounds__(kReduceSamples * kReduceGroups)
    k_obs_reduce(long long n_parts, int S, const double* __restrict__ jpart,
                 double* __restrict__ J) {
    __shared__ double part[kReduceGroups][kReduceSamples];
    const int l = threadIdx.x % kReduceSamples, g = threadIdx.x / kReduceSamples;
    const int s = blockIdx.x * kReduceSamples + l;
    double acc = 0.0;
    if (s < S)
        for (long long k = g; k < n_parts; k += kReduceGroups) acc += jpart[(size_t)k * S + s];
    part[g][l] = acc;
    __syncthreads();
    if (g != 0 || s >= S) return;
    for (int q = 1; q < kReduceGroups; ++q) acc += part[q][l];
    J[s] = acc;
}

// chi_n += W dJ/du_n = W * 2 (u_n - uobs_n) at the free observation nodes.
template <typename T>
__global__ void k_adj_force(int n_obs, int S, const int32_t* __restrict__ obs_nodes,
                            int n_clamped, const T* __restrict__ invm, T w0,
                            const T* __restrict__ u, const T* __restrict__ obs_k, T* __restrict__ chi) {
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long i = g / S;
    if (i >= n_obs) return;
    const int s = (int)(g - i * S);
    const size_t a = (size_t)obs_nodes[i];
    if ((long long)a < n_clamped) return;
    const T w = w0 * invm[a * S + s];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const size_t r = (3 * a + c) * S + s;
        const T d = u[r] - obs_k[((size_t)i * 3 + c) * S + s];
        chi[r] += w * T(2) * d;
    }
}

template <typename T>
struct RevArgs {
    const int32_t* node_ptr;
    const int4* rec;
    const T* slab;
    const T* own;
    const T* fhat;
    const T* coef;
    const T* invm;
    const T* u;    // u_n
    T* uo;         // in: u_{n+1}; out: u_{n-1}
    const T* x;    // chi_{n+1}
    T* xo;         // in: chi_{n+2}; out: chi_n (without the observation forcing)
    T* gam;        // (E, S) Gamma accumulator
    T* gm;         // (N, S) G accumulator, or null
    const double* p;  // pressure of forward step n
    long long n_nodes;
    int S;
    int n_clamped;
    T clamp;
    T eta;
    T inv1meta;
    T w0;
    int tpn;
    int npb;
    int nch;        // sample chunks of 32*VEC per node block (fan kernel)
    int cap_slots;  // slot capacity of the shared-memory stage (fan kernel)
    int* status;    // bit 0: a bounded wait gave up; bit 1: stage too small
    int pf_dist = 0;   // fan kernel: nodes ahead whose rows are prefetched into L2 (0: off)
    int pf_parts = 0;  // bit 0: node rows; bit 1: element coefficient and Gamma rows
    int pf_group = 1;  // node blocks covered by one prefetching block
};

// Prefetch into L2 the rows that nodes a0 .. a0 + n - 1 read in a reverse step: u_n,
// chi_{n+1}, u_{n+1}, chi_{n+2}, inverse mass, the G row, and the coefficient and
// Gamma rows of their elements (found through their slot records).
template <typename T, bool GM>
__device__ __forceinline__ void rev_prefetch(const RevArgs<T>& A, long long a0, int n,
                                             int lane) {
    if (a0 >= A.n_nodes) return;
    const long long a1 = (a0 + n < A.n_nodes) ? a0 + n : A.n_nodes;
    const size_t S = (size_t)A.S;
    const size_t nrow = (size_t)(a1 - a0) * S * sizeof(T);
    if (A.pf_parts & 1) {
        if (lane == 0) bulk_prefetch_l2(A.u + (size_t)a0 * 3 * S, 3 * nrow);
        if (lane == 1) bulk_prefetch_l2(A.x + (size_t)a0 * 3 * S, 3 * nrow);
        if (lane == 2) bulk_prefetch_l2(A.uo + (size_t)a0 * 3 * S, 3 * nrow);
        if (lane == 3) bulk_prefetch_l2(A.xo + (size_t)a0 * 3 * S, 3 * nrow);
        if (lane == 4) bulk_prefetch_l2(A.invm + (size_t)a0 * S, nrow);
        if constexpr (GM) {
            if (lane == 5) bulk_prefetch_l2(A.gm + (size_t)a0 * S, nrow);
        }
    }
    if (!(A.pf_parts & 2)) return;
    const int kb = __ldg(A.node_ptr + a0), ke = __ldg(A.node_ptr + a1);
    for (int k = kb + lane; k < ke; k += 32) {
        const size_t e = (size_t)__ldg(&A.rec[k].x);
        bulk_prefetch_l2(A.coef + e * S, S * sizeof(T));
        bulk_prefetch_l2(A.gam + e * S, S * sizeof(T));
    }
}

template <typename T>
__device__ __forceinline__ void load27(const T* K, T (&kk)[27]) {
    if constexpr (std::is_same<T, float>::value) {
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const float4 t = __ldg(reinterpret_cast<const float4*>(K) + q);
            if (4 * q + 0 < 27) kk[4 * q + 0] = t.x;
            if (4 * q + 1 < 27) kk[4 * q + 1] = t.y;
            if (4 * q + 2 < 27) kk[4 * q + 2] = t.z;
            if (4 * q + 3 < 27) kk[4 * q + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int q = 0; q < 14; ++q) {
            const double2 t = __ldg(reinterpret_cast<const double2*>(K) + q);
            if (2 * q + 0 < 27) kk[2 * q + 0] = t.x;
            if (2 * q + 1 < 27) kk[2 * q + 1] = t.y;
        }
    }
}

// dchi^T Khat_e du for the element owned by this slot: (u1, u2) and (x1, x2) are
// the first and second neighbour rows of u_n and chi_{n+1}, already differences
// u_b - u_a (FULL: the rows themselves).
template <typename T, int V, bool SMEM_OWN = false, bool FULL = false>
__device__ __forceinline__ Vec<T, V> owner_form(const T* own, const Vec<T, V> (&u1)[3],
                                                const Vec<T, V> (&u2)[3],
                                                const Vec<T, V> (&x1)[3],
                                                const Vec<T, V> (&x2)[3],
                                                const Vec<T, V> (&ua)[3],
                                                const Vec<T, V> (&ca)[3]) {
    Vec<T, V> du1[3], du2[3], dy1[3], dy2[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        du1[d] = FULL ? vsub(u1[d], ua[d]) : u1[d];
        du2[d] = FULL ? vsub(u2[d], ua[d]) : u2[d];
        dy1[d] = FULL ? vsub(x1[d], ca[d]) : x1[d];
        dy2[d] = FULL ? vsub(x2[d], ca[d]) : x2[d];
    }
    // own points into global memory (gather kernel) or shared memory (fan kernel, SMEM_OWN):
    // plain generic loads, not the global-only read-only path.  From shared memory they
    // are volatile, so that each of the 27 values is read where it is used instead of all
    // of them being hoisted into registers beside the three rotating neighbour-row sets
    // (the fan kernel spilled at its 128-register cap with them hoisted; it fits without).
    using OwnPtr = typename std::conditional<SMEM_OWN, const volatile T*, const T*>::type;
    const OwnPtr ob = own;
    Vec<T, V> g = vzero<T, V>();
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        Vec<T, V> z1 = vzero<T, V>(), z2 = vzero<T, V>();
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) {
            axpy(z1, ob[3 * i + jj], du1[jj]);       // K_b1b1
            axpy(z1, ob[9 + 3 * i + jj], du2[jj]);   // K_b1b2
            axpy(z2, ob[9 + 3 * jj + i], du1[jj]);   // K_b2b1 = K_b1b2^T
            axpy(z2, ob[18 + 3 * i + jj], du2[jj]);  // K_b2b2
        }
        vfma(g, dy1[i], z1);
        vfma(g, dy2[i], z2);
    }
    return g;
}

// Gamma_e += that form.
template <typename T, int V, bool SMEM_OWN = false, bool FULL = false>
__device__ __forceinline__ void owner_grad(const RevArgs<T>& A, int e, const T* own, size_t S,
                                           size_t col,
                                           const Vec<T, V> (&u1)[3], const Vec<T, V> (&u2)[3],
                                           const Vec<T, V> (&x1)[3], const Vec<T, V> (&x2)[3],
                                           const Vec<T, V> (&ua)[3], const Vec<T, V> (&ca)[3]) {
    const Vec<T, V> g = owner_form<T, V, SMEM_OWN, FULL>(own, u1, u2, x1, x2, ua, ca);
    T* gp = A.gam + (size_t)e * S + col;
    Vec<T, V> gv = ld<T, V>(gp);
#pragma unroll
    for (int q = 0; q < V; ++q) gv.v[q] += g.v[q];
    st<T, V>(gp, gv);
}

// The rows that a free node's update reads besides its own u_n and chi_{n+1}.
template <typename T, int V>
struct RevRows {
    Vec<T, V> u1[3], x2[3], im, gm;
    T f[3];
};
template <typename T, int V, bool GM>
__device__ __forceinline__ void rev_rows(const RevArgs<T>& A, int a, size_t col,
                                         RevRows<T, V>& R) {
    const size_t S = (size_t)A.S;
    const uint32_t rowb = (uint32_t)A.S * sizeof(T), nodeb = 3 * rowb;
    const T* qu = row_at(A.uo + col, a, nodeb);
    const T* qx = row_at(A.xo + col, a, nodeb);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        R.u1[d] = ld<T, V>(qu + d * S);
        R.x2[d] = ld<T, V>(qx + d * S);
        R.f[d] = __ldg(A.fhat + 4 * (size_t)a + d);
    }
    R.im = ldg<T, V>(row_at(A.invm + col, a, rowb));
    if constexpr (GM) R.gm = ld<T, V>(row_at(A.gm + col, a, rowb));
}
// A free node's update from those rows.
template <typename T, int V, bool GM>
__device__ __forceinline__ void rev_update(const RevArgs<T>& A, int a, size_t col,
                                           const Vec<T, V> (&ua)[3], const Vec<T, V> (&ca)[3],
                                           const Vec<T, V> (&accU)[3],
                                           const Vec<T, V> (&accC)[3], RevRows<T, V>& R, bool on) {
    const size_t S = (size_t)A.S;
    const uint32_t rowb = (uint32_t)A.S * sizeof(T), nodeb = 3 * rowb;
    T* uo = row_at(A.uo + col, a, nodeb);
    T* xo = row_at(A.xo + col, a, nodeb);
    const T p = (T)A.p[0];
    Vec<T, V> gacc = vzero<T, V>();
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        Vec<T, V> um, xn;
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const bool live = R.im.v[i] != T(0);
            const T w = A.w0 * R.im.v[i];
            const T r = fma(p, R.f[d], -accU[d].v[i]);
            const T dv = ((R.u1[d].v[i] - ua[d].v[i]) - w * r) * A.inv1meta;
            um.v[i] = live ? ua[d].v[i] - dv : T(0);
            const T dx = ca[d].v[i] - R.x2[d].v[i];
            xn.v[i] = live ? ca[d].v[i] + fma(-A.eta, dx, dx) - w * accC[d].v[i] : T(0);
            if constexpr (GM) gacc.v[i] = fma(ca[d].v[i], r, gacc.v[i]);
        }
        if (on) st<T, V>(uo + d * S, um);
        if (on) st<T, V>(xo + d * S, xn);
    }
    if constexpr (GM) {
#pragma unroll
        for (int q = 0; q < V; ++q) R.gm.v[q] += gacc.v[q];
        if (on) st<T, V>(row_at(A.gm + col, a, rowb), R.gm);
    }
}

// Node update of one reverse step: u_{n-1} (backward step), chi_n, and G += chi_{n+1} . r_n.
template <typename T, int V, bool GM>
__device__ __forceinline__ void rev_epilogue(const RevArgs<T>& A, long long a, size_t S,
                                             size_t col, size_t row, const Vec<T, V> (&ua)[3],
                                             const Vec<T, V> (&ca)[3],
                                             const Vec<T, V> (&accU)[3],
                                             const Vec<T, V> (&accC)[3], bool on = true) {
    if (a < A.n_clamped) {
        const Vec<T, V> cl = vfill<T, V>(A.clamp), z = vzero<T, V>();
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (on) st<T, V>(A.uo + row + d * S, cl);
            if (on) st<T, V>(A.xo + row + d * S, z);
        }
        return;
    }
    RevRows<T, V> R;
    rev_rows<T, V, GM>(A, (int)a, col, R);
    rev_update<T, V, GM>(A, (int)a, col, ua, ca, accU, accC, R, on);
}

// One reverse step for (node a, V samples): reconstruct u_{n-1}, advance chi, accumulate
// Gamma over the elements this node owns and G of this node.  Rows are gathered
// through L1; a fan continuation reuses the previous slot's second neighbour.
template <typename T, int V, bool GM, bool FULL = false>
__global__ void __launch_bounds__(256) k_reverse(RevArgs<T> A) {
    long long a;
    int vec;
    if (!map_row(A.tpn, A.npb, A.n_nodes, A.S / V, a, vec)) return;
    const size_t S = (size_t)A.S;
    const size_t col = (size_t)vec * V;
    const size_t row = (size_t)a * 3 * S + col;
    Vec<T, V> ua[3], ca[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        ua[d] = ldg<T, V>(A.u + row + d * S);
        ca[d] = ldg<T, V>(A.x + row + d * S);
    }
    Vec<T, V> accU[3], accC[3], cu[3], cc[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        accU[d] = vzero<T, V>();
        accC[d] = vzero<T, V>();
        cu[d] = vzero<T, V>();
        cc[d] = vzero<T, V>();
    }
    const int k0 = __ldg(A.node_ptr + a), k1 = __ldg(A.node_ptr + a + 1);
    for (int k = k0; k < k1; ++k) {
        const int4 r = __ldg(A.rec + k);
        Vec<T, V> x1[3], x2[3], y1[3], y2[3];
        if (r.w & 1) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                x1[d] = cu[d];
                y1[d] = cc[d];
            }
        } else {
            const size_t o1 = (size_t)r.y * 3 * S + col;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                x1[d] = ldg<T, V>(A.u + o1 + d * S);
                y1[d] = ldg<T, V>(A.x + o1 + d * S);
                if constexpr (!FULL) x1[d] = vsub(x1[d], ua[d]);
                if constexpr (!FULL) y1[d] = vsub(y1[d], ca[d]);
            }
        }
        const size_t o2 = (size_t)r.z * 3 * S + col;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            x2[d] = ldg<T, V>(A.u + o2 + d * S);
            y2[d] = ldg<T, V>(A.x + o2 + d * S);
            if constexpr (!FULL) x2[d] = vsub(x2[d], ua[d]);
            if constexpr (!FULL) y2[d] = vsub(y2[d], ca[d]);
        }
        const Vec<T, V> c = ldg<T, V>(A.coef + (size_t)r.x * S + col);
        T kk[27];
        load27<T>(A.slab + (size_t)kSlabStride * k, kk);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            Vec<T, V> tu = vzero<T, V>(), tc = vzero<T, V>();
            if constexpr (FULL) {
#pragma unroll
                for (int jj = 0; jj < 3; ++jj) {
                    axpy(tu, kk[3 * i + jj], ua[jj]);
                    axpy(tc, kk[3 * i + jj], ca[jj]);
                }
            }
#pragma unroll
            for (int jj = 0; jj < 3; ++jj) {
                axpy(tu, kk[9 + 3 * i + jj], x1[jj]);
                axpy(tc, kk[9 + 3 * i + jj], y1[jj]);
            }
#pragma unroll
            for (int jj = 0; jj < 3; ++jj) {
                axpy(tu, kk[18 + 3 * i + jj], x2[jj]);
                axpy(tc, kk[18 + 3 * i + jj], y2[jj]);
            }
            vfma(accU[i], c, tu);
            vfma(accC[i], c, tc);
        }
        if (((r.w >> 8) & 3) == 0)
            owner_grad<T, V, false, FULL>(A, r.x, A.own + (size_t)kOwnStride * k, S, col, x1, x2, y1, y2,
                                   ua, ca);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            cu[d] = x2[d];
            cc[d] = y2[d];
        }
    }
    rev_epilogue<T, V, GM>(A, a, S, col, row, ua, ca, accU, accC);
}

// ------------------------------------------------------------ fan-rotation reverse step
// As the forward fan kernel: a warp per node and 32*VEC-sample chunk, the block's slot
// records and stiffness rows bulk-copied (TMA) into shared memory, and the neighbour
// rows of u_n and chi_{n+1} rotating through three register sets so that the loads of
// slot k+1 are in flight while slot k is multiplied.
template <typename T, int V>
__device__ __forceinline__ void load3(Vec<T, V> (&x)[3], const T* __restrict__ base, int node,
                                      size_t S, size_t col) {
    const T* p = base + (size_t)node * 3 * S + col;
#pragma unroll
    for (int d = 0; d < 3; ++d) x[d] = ldg<T, V>(p + d * S);
}
template <typename T, int V, bool FULL = false>
__device__ __forceinline__ void diff3(Vec<T, V> (&x)[3], const Vec<T, V> (&ref)[3]) {
    if constexpr (!FULL) {
#pragma unroll
        for (int d = 0; d < 3; ++d) x[d] = vsub(x[d], ref[d]);
    }
}

// Both row products of one slot from one read of its stiffness rows (shared memory).
template <typename T, int V, bool FULL = false>
__device__ __forceinline__ void slot_fma2(const T* K, const Vec<T, V>& c,
                                          const Vec<T, V> (&u1)[3], const Vec<T, V> (&u2)[3],
                                          const Vec<T, V> (&x1)[3], const Vec<T, V> (&x2)[3],
                                          const Vec<T, V> (&ua)[3], const Vec<T, V> (&ca)[3],
                                          Vec<T, V> (&accU)[3], Vec<T, V> (&accC)[3]) {
    T kk[28];
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int q = 2; q < 7; ++q) {
            const float4 t = reinterpret_cast<const float4*>(K)[q];
            kk[4 * q] = t.x;
            kk[4 * q + 1] = t.y;
            kk[4 * q + 2] = t.z;
            kk[4 * q + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int q = FULL ? 0 : 4; q < 14; ++q) {
            const double2 t = reinterpret_cast<const double2*>(K)[q];
            kk[2 * q] = t.x;
            kk[2 * q + 1] = t.y;
        }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        Vec<T, V> tu = vzero<T, V>(), tc = vzero<T, V>();
        if constexpr (FULL) {
#pragma unroll
            for (int jj = 0; jj < 3; ++jj) {
                axpy(tu, kk[3 * i + jj], ua[jj]);
                axpy(tc, kk[3 * i + jj], ca[jj]);
            }
        }
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) {
            axpy(tu, kk[9 + 3 * i + jj], u1[jj]);
            axpy(tc, kk[9 + 3 * i + jj], x1[jj]);
        }
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) {
            axpy(tu, kk[18 + 3 * i + jj], u2[jj]);
            axpy(tc, kk[18 + 3 * i + jj], x2[jj]);
        }
        vfma(accU[i], c, tu);
        vfma(accC[i], c, tc);
    }
}

template <typename T, int V>
__device__ __forceinline__ void rev_phase(int& k, int k1, const int4* srec, const T* sslab,
                                          const T* sown, const RevArgs<T>& A, size_t S, size_t col,
                                          const Vec<T, V> (&ua)[3], const Vec<T, V> (&ca)[3],
                                          Vec<T, V> (&accU)[3], Vec<T, V> (&accC)[3],
                                          Vec<T, V> (&pu)[3], Vec<T, V> (&px)[3],
                                          Vec<T, V> (&cu)[3], Vec<T, V> (&cx)[3],
                                          const Vec<T, V>& ccur, Vec<T, V> (&nu)[3],
                                          Vec<T, V> (&nx)[3], Vec<T, V>& cnxt) {
    const bool more = k + 1 < k1;
    int4 rn = make_int4(0, 0, 0, 1);
    if (more) {
        rn = srec[k + 1];
        load3<T, V>(nu, A.u, rn.z, S, col);
        load3<T, V>(nx, A.x, rn.z, S, col);
        cnxt = ldg<T, V>(A.coef + (size_t)rn.x * S + col);
    }
    diff3<T, V>(cu, ua);
    diff3<T, V>(cx, ca);
    const int4 r = srec[k];
    slot_fma2<T, V>(sslab + (size_t)kSlabStride * k, ccur, pu, cu, px, cx, ua, ca, accU,
                          accC);
    if (((r.w >> 8) & 3) == 0)
        owner_grad<T, V, true>(A, r.x, sown + (size_t)kOwnStride * k, S, col, pu, cu, px, cx, ua,
                               ca);
    if (more && !(rn.w & 1)) {  // fan break: the next slot's first neighbour is new
        load3<T, V>(cu, A.u, rn.y, S, col);
        load3<T, V>(cx, A.x, rn.y, S, col);
        diff3<T, V>(cu, ua);
        diff3<T, V>(cx, ca);
    }
    ++k;
}

template <typename T, int V, bool GM, int MINB>
__global__ void __launch_bounds__(256, MINB) k_reverse_fan(RevArgs<T> A) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const long long nb = blockIdx.x / A.nch;
    const int chunk = (int)(blockIdx.x - nb * A.nch);
    const long long a0 = nb * A.npb;
    const long long a1 = (a0 + A.npb < A.n_nodes) ? a0 + A.npb : A.n_nodes;
    const int kb = __ldg(A.node_ptr + a0), ke = __ldg(A.node_ptr + a1);
    const int nsl = ke - kb;
    if (nsl > A.cap_slots) {
        if (threadIdx.x == 0 && A.status) atomicOr(A.status, 2);
        return;
    }
    const uint32_t bar = smem_u32(smem);
    int4* srec = reinterpret_cast<int4*>(smem + 16);
    T* sslab = reinterpret_cast<T*>(smem + 16 + (size_t)A.cap_slots * 16);
    T* sown = sslab + (size_t)A.cap_slots * kSlabStride;
    if (threadIdx.x == 0) mbar_init(bar, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t b_rec = (uint32_t)nsl * 16u;
        const uint32_t b_slab = (uint32_t)nsl * (uint32_t)(kSlabStride * sizeof(T));
        mbar_arrive_expect_tx(bar, b_rec + 2 * b_slab);
        if (nsl > 0) {
            bulk_g2s(smem_u32(srec), A.rec + kb, b_rec, bar);
            bulk_g2s(smem_u32(sslab), A.slab + (size_t)kb * kSlabStride, b_slab, bar);
            bulk_g2s(smem_u32(sown), A.own + (size_t)kb * kOwnStride, b_slab, bar);
        }
    }
    const long long a = a0 + warp;
    const bool active = warp < A.npb && a < a1;
    const size_t S = (size_t)A.S;
    const size_t col = ((size_t)chunk * 32 + lane) * V;
    const size_t row = (size_t)a * 3 * S + col;
    Vec<T, V> ua[3], ca[3];
    if (active) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            ua[d] = ldg<T, V>(A.u + row + d * S);
            ca[d] = ldg<T, V>(A.x + row + d * S);
            prefetch_l2(A.uo + row + d * S);
            prefetch_l2(A.xo + row + d * S);
        }
        prefetch_l2(A.invm + (size_t)a * S + col);
    }
    if (A.pf_dist > 0 && chunk == 0 && nb % A.pf_group == 0 && warp == A.npb - 1)
        rev_prefetch<T, GM>(A, a0 + A.pf_dist, A.npb * A.pf_group, lane);
    if (!mbar_wait_bounded(bar, 0, kMaxPolls)) {
        if (lane == 0 && A.status) atomicOr(A.status, 1);
        return;
    }
    if (!active) return;
    Vec<T, V> accU[3], accC[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        accU[d] = vzero<T, V>();
        accC[d] = vzero<T, V>();
    }
    const int k0 = __ldg(A.node_ptr + a) - kb, k1 = __ldg(A.node_ptr + a + 1) - kb;
    if (k0 < k1) {
        Vec<T, V> U0[3], U1[3], U2[3], X0[3], X1[3], X2[3], c0, c1, c2;
        const int4 r0 = srec[k0];
        load3<T, V>(U0, A.u, r0.y, S, col);
        load3<T, V>(X0, A.x, r0.y, S, col);
        load3<T, V>(U1, A.u, r0.z, S, col);
        load3<T, V>(X1, A.x, r0.z, S, col);
        c1 = ldg<T, V>(A.coef + (size_t)r0.x * S + col);
        diff3<T, V>(U0, ua);
        diff3<T, V>(X0, ca);
        int k = k0;
        while (true) {
            rev_phase<T, V>(k, k1, srec, sslab, sown, A, S, col, ua, ca, accU, accC, U0, X0, U1,
                                  X1, c1, U2, X2, c2);
            if (k >= k1) break;
            rev_phase<T, V>(k, k1, srec, sslab, sown, A, S, col, ua, ca, accU, accC, U1, X1, U2,
                                  X2, c2, U0, X0, c0);
            if (k >= k1) break;
            rev_phase<T, V>(k, k1, srec, sslab, sown, A, S, col, ua, ca, accU, accC, U2, X2, U0,
                                  X0, c0, U1, X1, c1);
            if (k >= k1) break;
        }
    }
    rev_epilogue<T, V, GM>(A, a, S, col, row, ua, ca, accU, accC);
}

// ------------------------------------------------------------ patch reverse step
// The reverse step with free-running warps on patches of nodes, as the forward patch kernel
// (solid_patch.cu): 32 * V samples of one node at a time, the next node's slots (records,
// stiffness rows, owner blocks) staged in shared memory and its rows prefetched into L2
// under the current node.  Clamped nodes are walked like the others: they own elements.
// It waits on the gathers of two states a neighbour, so the closed fan of six is unrolled
// (one element ahead; the update's rows in the place of element 7) and an owned element's
// Gamma row is requested before its products.  us a step, fan or persistent fan / this:
// 128 x 400 wall, FP32 64 samples 155 / 116, 128 samples with G 315 / 235; 128 x 320 wall, FP64
// 64 samples with G 267 / 213; 64 x 128 wall, 64 samples FP32 22.4 / 21.3, FP64 54.7 / 46.4.
// Both row products and the Gamma update of a node that is not staged (more slots than the
// descriptor's max_degree), all from global memory, as ku_row_unstaged.
template <typename T, int V, bool FULL>
__device__ __forceinline__ void rev_row_unstaged(const RevArgs<T>& A, int k0, int n, const T* u,
                                                 const T* x, size_t col, uint32_t rowb, bool on,
                                                 const Vec<T, V> (&ua)[3],
                                                 const Vec<T, V> (&ca)[3], Vec<T, V> (&accU)[3],
                                                 Vec<T, V> (&accC)[3]) {
    const size_t S = rowb / sizeof(T);
    Vec<T, V> u1[3], u2[3], x1[3], x2[3];
    auto rows = [&](Vec<T, V> (&p)[3], Vec<T, V> (&q)[3], int b) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            p[d] = ld_state<T, V>(row_at(u, b, 3 * rowb) + d * S);
            q[d] = ld_state<T, V>(row_at(x, b, 3 * rowb) + d * S);
        }
        diff3<T, V, FULL>(p, ua);
        diff3<T, V, FULL>(q, ca);
    };
#pragma unroll 1
    for (int k = k0; k < k0 + n; ++k) {
        const int4 r = __ldg(A.rec + k);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            u1[d] = u2[d];
            x1[d] = x2[d];
        }
        if (k == k0 || !(r.w & 1)) rows(u1, x1, r.y);
        rows(u2, x2, r.z);
        slot_fma2<T, V, FULL>(A.slab + (size_t)kSlabStride * k,
                        ldg<T, V>(row_at(A.coef + col, r.x, rowb)), u1, u2, x1, x2, ua, ca, accU,
                        accC);
        if (((r.w >> 8) & 3) == 0) {
            T* const gp = row_at(A.gam + col, r.x, rowb);
            Vec<T, V> gv = ld<T, V>(gp);
            const Vec<T, V> g =
                owner_form<T, V, false, FULL>(A.own + (size_t)kOwnStride * k, u1, u2, x1, x2, ua, ca);
#pragma unroll
            for (int i = 0; i < V; ++i) gv.v[i] += g.v[i];
            if (on) st<T, V>(gp, gv);
        }
    }
}

template <typename T, int V, bool GM, int W, bool FULL>
__global__ void __launch_bounds__(32 * W, 1)
    k_reverse_patch(RevArgs<T> A, PatchMap M, int max_degree) {
    extern __shared__ __align__(16) unsigned char smem[];
    using P = SlotStage<T, FULL>;
    constexpr int kOwnWords = kOwnStride * (int)sizeof(T) / 16;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t b_rec = 16u * max_degree, b_slab = P::kSlotBytes * max_degree;
    const uint32_t b_stage = b_rec + b_slab + 16u * kOwnWords * max_degree;
    unsigned char* const wb = smem + warp * (2 * b_stage);
    const uint32_t rowb = (uint32_t)A.S * sizeof(T), nodeb = 3 * rowb;
    const int chunk = blockIdx.x % A.nch;
    const int vec = chunk * 32 + lane, last = A.S / V - 1;
    const bool on = vec <= last;
    const size_t S = (size_t)A.S, col = (size_t)(on ? vec : last) * V;
    PatchWalk walk(M, warp, blockIdx.x / A.nch, gridDim.x / A.nch, 0, (int)A.n_nodes, W);
    auto stage = [&](int b, int k0, int n, int sg) {
        if (b >= 0) {
            const uint32_t d = smem_u32(wb + sg * b_stage);
            const char* r = reinterpret_cast<const char*>(A.rec + k0);
            const char* s = reinterpret_cast<const char*>(A.slab + (size_t)k0 * kSlabStride);
            const char* o = reinterpret_cast<const char*>(A.own + (size_t)k0 * kOwnStride);
            for (int q = lane; q < n; q += 32) cp_async<16>(d + 16 * q, r + 16 * q);
            for (int q = lane; q < P::kWords * n; q += 32) {
                const int sl = q / P::kWords, w = q - sl * P::kWords;
                cp_async<16>(d + b_rec + 16 * q,
                             s + sl * (kSlabStride * (int)sizeof(T)) + (P::kFirst + w) * 16);
            }
            for (int q = lane; q < kOwnWords * n; q += 32)
                cp_async<16>(d + b_rec + b_slab + 16 * q, o + 16 * q);
        }
        cp_async_commit();
    };
    __shared__ int unstaged[W];  // a node of the warp was not staged
    if (lane == 0) unstaged[warp] = 0;
    __syncwarp();
    bool more = walk.more(M);
    int a = walk.node(M), n, an, k0, nn;
    node_slots(A.node_ptr, max_degree, unstaged + warp, a, k0, n);
    stage(a, k0, n, 0);
    walk.advance(M);
    an = walk.node(M);
    node_slots(A.node_ptr, max_degree, unstaged + warp, an, k0, nn);
    // line prefetch: rows 0..2 u_n, 3..5 chi_{n+1}, 6..8 u_{n+1}, 9..11 chi_{n+2}, 12 inverse
    // mass, 13 G; then coefficient rows and, by the owner, Gamma rows
    const RowLines<T, V> ln(lane, chunk, rowb);
    auto prefetch_node = [&](int b) {
        if (b < 0 || !ln.on) return;
#pragma unroll
        for (int r0 = 0; r0 < (GM ? 14 : 13); r0 += RowLines<T, V>::kRows) {
            const int r = r0 + ln.row;
            const T* q = r < 3    ? A.u + r * S
                         : r < 6  ? A.x + (r - 3) * S
                         : r < 9  ? A.uo + (r - 6) * S
                         : r < 12 ? A.xo + (r - 9) * S
                         : r < 13 ? A.invm
                                  : A.gm;
            if (r < (GM ? 14 : 13))
                prefetch_l2(reinterpret_cast<const char*>(q) + ln.off +
                            (uint64_t)(uint32_t)b * (r < 12 ? nodeb : rowb));
        }
    };
    grid_dependency_release();
    grid_dependency_wait();
    const T* const u = A.u + col;
    const T* const x = A.x + col;
    const T* const cf = A.coef + col;
    T* const gam = A.gam + col;
    for (int sg = 0; more; sg ^= 1) {
        Vec<T, V> ua[3], ca[3];
        auto rows = [&](Vec<T, V> (&p)[3], Vec<T, V> (&q)[3], int b) {
            const uint64_t o = (uint64_t)(uint32_t)b * nodeb;
            const T* pu = reinterpret_cast<const T*>(reinterpret_cast<const char*>(u) + o);
            const T* px = reinterpret_cast<const T*>(reinterpret_cast<const char*>(x) + o);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                p[d] = ld_state<T, V>(pu + d * S);
                q[d] = ld_state<T, V>(px + d * S);
            }
        };
        if (a >= 0) rows(ua, ca, a);
        cp_async_wait_all();
        __syncwarp();
        const unsigned char* const st = wb + sg * b_stage;
        const int4* const srec = reinterpret_cast<const int4*>(st);
        const T* const K = reinterpret_cast<const T*>(st + b_rec) - 16 / (int)sizeof(T) * P::kFirst;
        const T* const own = reinterpret_cast<const T*>(st + b_rec + b_slab);
        constexpr int kStep = P::kSlotBytes / (int)sizeof(T);
        stage(an, k0, nn, sg ^ 1);
        prefetch_node(an);
        const int nn_cur = nn;
        more = walk.more(M);
        walk.advance(M);
        int ax = walk.node(M);
        node_slots(A.node_ptr, max_degree, unstaged + warp, ax, k0, nn);
        auto prefetch_elems = [&]() {  // coefficient rows and owned Gamma rows of the next node
            cp_async_wait_all();
            __syncwarp();
            const int4* nr = reinterpret_cast<const int4*>(wb + (sg ^ 1) * b_stage);
            constexpr int kHalf = RowLines<T, V>::kRows / 2;
            const int q = ln.row % kHalf;
            if (an >= 0 && ln.on && q < nn_cur) {
                const bool gamma = ln.row >= kHalf;
                const int4 r = nr[q];
                if (!gamma || ((r.w >> 8) & 3) == 0)
                    prefetch_l2(reinterpret_cast<const char*>(gamma ? A.gam : A.coef) + ln.off +
                                (uint64_t)(uint32_t)r.x * rowb);
            }
        };
        if (a >= 0) {
            Vec<T, V> accU[3], accC[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) accU[d] = accC[d] = vzero<T, V>();
            auto element = [&](int k, const int4& r, const Vec<T, V>& c, const Vec<T, V> (&u1)[3],
                               const Vec<T, V> (&u2)[3], const Vec<T, V> (&x1)[3],
                               const Vec<T, V> (&x2)[3]) {
                const bool owner = ((r.w >> 8) & 3) == 0;
                Vec<T, V> gv = vzero<T, V>();
                T* const gp = row_at(gam, r.x, rowb);
                if (owner) gv = ld<T, V>(gp);  // requested before the products
                slot_fma2<T, V, FULL>(K + kStep * k, c, u1, u2, x1, x2, ua, ca, accU, accC);
                if (owner) {
                    const Vec<T, V> g = owner_form<T, V, true, FULL>(own + kOwnStride * k, u1, u2,
                                                                     x1, x2, ua, ca);
#pragma unroll
                    for (int q = 0; q < V; ++q) gv.v[q] += g.v[q];
                    if (on) cvfes::st<T, V>(gp, gv);
                }
            };
            RevRows<T, V> R;
            const int flag = lane < n ? srec[lane].w : 1;
            const bool six = n == 6 && __all_sync(0xffffffffu, (flag & 1) || lane == 0);
            if (six) {  // closed fan: unrolled, the update's rows in the place of element 6
                Vec<T, V> U[8][3], X[8][3], C[7];
                rows(U[0], X[0], srec[0].y);
                rows(U[1], X[1], srec[0].z);
                C[0] = ldg<T, V>(row_at(cf, srec[0].x, rowb));
                diff3<T, V, FULL>(U[0], ua);
                diff3<T, V, FULL>(X[0], ca);
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    if (k < 5) {
                        const int4 rn = srec[k + 1];
                        rows(U[k + 2], X[k + 2], rn.z);
                        C[k + 1] = ldg<T, V>(row_at(cf, rn.x, rowb));
                    } else {
                        if (a >= A.n_clamped) rev_rows<T, V, GM>(A, a, col, R);
                    }
                    if (k == 2) prefetch_elems();
                    diff3<T, V, FULL>(U[k + 1], ua);
                    diff3<T, V, FULL>(X[k + 1], ca);
                    element(k, srec[k], C[k], U[k], U[k + 1], X[k], X[k + 1]);
                    // FP32: keeps the next element's loads from sinking to their uses
                    // (64 x 128 wall, 64 samples: 3.36 ms a gradient of 100 steps, 3.52 without)
                    if constexpr (sizeof(T) == 4) __syncwarp();
                }
            } else if (n > 0) {
                Vec<T, V> U0[3], U1[3], U2[3], X0[3], X1[3], X2[3], c0, c1, c2;
                int4 r = srec[0];
                rows(U0, X0, r.y);
                rows(U1, X1, r.z);
                c1 = ldg<T, V>(row_at(cf, r.x, rowb));
                diff3<T, V, FULL>(U0, ua);
                diff3<T, V, FULL>(X0, ca);
                int k = 0;
                auto phase = [&](Vec<T, V> (&pu)[3], Vec<T, V> (&px)[3], Vec<T, V> (&cu)[3],
                                 Vec<T, V> (&cx)[3], const Vec<T, V>& c, Vec<T, V> (&nu)[3],
                                 Vec<T, V> (&nx)[3], Vec<T, V>& cn) {
                    const bool next = k + 1 < n;
                    int4 rn = make_int4(0, 0, 0, 1);
                    if (next) {
                        rn = srec[k + 1];
                        rows(nu, nx, rn.z);
                        cn = ldg<T, V>(row_at(cf, rn.x, rowb));
                    }
                    diff3<T, V, FULL>(cu, ua);
                    diff3<T, V, FULL>(cx, ca);
                    element(k, r, c, pu, cu, px, cx);
                    if (next && !(rn.w & 1)) {  // fan break: the next first neighbour is new
                        rows(cu, cx, rn.y);
                        diff3<T, V, FULL>(cu, ua);
                        diff3<T, V, FULL>(cx, ca);
                    }
                    r = rn;
                    ++k;
                };
                while (true) {
                    phase(U0, X0, U1, X1, c1, U2, X2, c2);
                    if (k >= n) break;
                    phase(U1, X1, U2, X2, c2, U0, X0, c0);
                    if (k >= n) break;
                    phase(U2, X2, U0, X0, c0, U1, X1, c1);
                    if (k >= n) break;
                }
            }
            if (!six) prefetch_elems();
            if (six && a >= A.n_clamped)
                rev_update<T, V, GM>(A, a, col, ua, ca, accU, accC, R, on);
            else
                rev_epilogue<T, V, GM>(A, a, S, col, (size_t)a * 3 * S + col, ua, ca, accU, accC,
                                       on);
        }
        __syncwarp();
        a = an;
        n = nn_cur;
        an = ax;
    }
    cp_async_wait_all();
    __syncwarp();
    if (!unstaged[threadIdx.x >> 5]) return;
    // the nodes that were not staged, after all others: they cost the loop no registers
    const LaunchAgain L;
    const int vec2 = L.block % A.nch * 32 + (L.thread & 31);
    const bool on2 = vec2 * V < A.S;
    const size_t col2 = (size_t)min(vec2, A.S / V - 1) * V;
    const uint32_t rb = (uint32_t)A.S * sizeof(T);
    PatchWalk again(M, L.thread >> 5, L.block / A.nch, L.blocks / A.nch, 0, (int)A.n_nodes, W);
    for (; again.more(M); again.advance(M)) {
        const int b = again.node(M);
        if (b < 0) continue;
        const int s0 = __ldg(A.node_ptr + b), ns = __ldg(A.node_ptr + b + 1) - s0;
        if (ns <= max_degree) continue;
        Vec<T, V> ua[3], ca[3], accU[3], accC[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            ua[d] = ld_state<T, V>(row_at(A.u + col2, b, 3 * rb) + d * (size_t)A.S);
            ca[d] = ld_state<T, V>(row_at(A.x + col2, b, 3 * rb) + d * (size_t)A.S);
            accU[d] = accC[d] = vzero<T, V>();
        }
        rev_row_unstaged<T, V, FULL>(A, s0, ns, A.u + col2, A.x + col2, col2,
                               rb, on2, ua, ca, accU, accC);
        rev_epilogue<T, V, GM>(A, b, (size_t)A.S, col2, (size_t)b * 3 * A.S + col2, ua, ca, accU,
                               accC, on2);
    }
}

// dJ/dlogE = -c Gamma; dJ/dlogh = -c Gamma - h sum_a alpha_{e,a} G_a / m_a.
template <typename T>
__global__ void k_grad_final(long long n_elems, int S, const int32_t* __restrict__ elems,
                             const double* __restrict__ area, MassWeights mw,
                             const double* __restrict__ lm, const double* __restrict__ logE,
                             const double* __restrict__ logh, const T* __restrict__ gam,
                             const T* __restrict__ gm, double* __restrict__ gE,
                             double* __restrict__ gh) {
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long e = g / S;
    if (e >= n_elems) return;
    const int s = (int)(g - e * S);
    const size_t o = (size_t)e * S + s;
    const double h = exp(logh[o]);
    const double c = exp(logE[o]) * h;
    const double ge = -c * (double)gam[o];
    if (gE) gE[o] = ge;
    if (gh) {
        double m = 0.0;
        if (gm) {
#pragma unroll
            for (int la = 0; la < 3; ++la) {
                const size_t na = (size_t)elems[3 * e + la];
                const double alpha = area[e] * (mw.w[3 * la] + mw.w[3 * la + 1] + mw.w[3 * la + 2]);
                m += alpha * (double)gm[na * S + s] / lm[na * S + s];
            }
        }
        gh[o] = ge - h * m;
    }
}

struct RevTuning {
    int vec;      // samples per thread (upper bound)
    int npb;      // nodes (warps) per block of the fan kernel
    int variant;  // 0: L1-gather kernel; 1: fan-rotation kernel with staged slots;
                  // 2: persistent patch kernel (npb and minb have no effect)
    int minb;     // resident blocks per SM asked of the compiler (fan kernel)
};
// Defaults: the patch kernel, which takes 2 FP32 samples or 1 FP64 sample a thread (figures
// at the kernel).
static RevTuning g_rev32 = {2, 2, 2, 2};
static RevTuning g_rev64 = {1, 4, 2, 2};
template <typename T>
RevTuning& rev_tuning() {
    return sizeof(T) == 4 ? g_rev32 : g_rev64;
}

constexpr size_t kRevMaxStage = 160 * 1024;

template <typename Kern, typename T>
int launch_rev_fan(Kern kernel, unsigned grid, int threads, size_t smem, cudaStream_t st,
                   const RevArgs<T>& A) {
    if (smem > 48 * 1024) {
        cudaError_t e =
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess)
            return fail(CVFES_ERR_CUDA, "k_reverse_fan smem attribute: %s", cudaGetErrorString(e));
    }
    kernel<<<grid, threads, smem, st>>>(A);
    CVFES_LAUNCH_CHECK("k_reverse_fan");
    return CVFES_OK;
}

template <typename T, int V, bool GM>
int launch_rev_fan_m(int minb, unsigned grid, int threads, size_t smem, cudaStream_t st,
                     const RevArgs<T>& A) {
    switch (minb) {
        case 4: return launch_rev_fan(k_reverse_fan<T, V, GM, 4>, grid, threads, smem, st, A);
        case 3: return launch_rev_fan(k_reverse_fan<T, V, GM, 3>, grid, threads, smem, st, A);
        case 2: return launch_rev_fan(k_reverse_fan<T, V, GM, 2>, grid, threads, smem, st, A);
        default: return launch_rev_fan(k_reverse_fan<T, V, GM, 1>, grid, threads, smem, st, A);
    }
}

// The patch kernel (variant 2); returns 1 without launching when a node's slots do not fit.
template <typename T, int V, bool FULL = false>
int launch_rev_patch(const cvfes_solid_mesh* m, RevArgs<T> A, bool after_step, cudaStream_t st) {
    const size_t slot = SlotStage<T, FULL>::kBytes + kOwnStride * sizeof(T);
    // (the slots are staged in 16-byte words)
    if (m->max_degree <= 0 || m->max_degree >= 1024 || A.S >= (1 << 27) ||
        m->n_nodes >= INT32_MAX / 2 || reinterpret_cast<uintptr_t>(A.own) % 16 ||
        reinterpret_cast<uintptr_t>(A.slab) % 16 || reinterpret_cast<uintptr_t>(A.rec) % 16)
        return 1;
    // what the registers allow (single FP32 samples, 128 x 400 wall, 37 samples: 183 us a step
    // at 16 warps, 157 at 24; the others are slower above 16)
    constexpr int W = sizeof(T) == 4 && V == 1 ? 24 : 16;
    const size_t smem = (size_t)W * 2 * slot * m->max_degree;
    if (smem > 160 * 1024) return 1;
    A.nch = (A.S / V + 31) / 32;
    const PatchMap M = patch_map(m->n_nodes, m->bandwidth, W);
    auto kernel = A.gm ? k_reverse_patch<T, V, true, W, FULL> : k_reverse_patch<T, V, false, W, FULL>;
    int per_sm = 0;
    const int rc = fanp_blocks_per_sm(reinterpret_cast<const void*>(kernel), 32 * W, smem, &per_sm);
    if (rc) return rc;
    const long long places = std::max(1LL, (long long)M.n_strips * M.tps);
    const long long per_chunk =
        std::max(1LL, std::min((long long)per_sm * device_sm_count() / A.nch, places));
    return launch_step_kernel(kernel, dim3((unsigned)(per_chunk * A.nch)), 32 * W, smem,
                              after_step, st, "k_reverse_patch", A, M, (int)m->max_degree);
}

template <typename T, int V>
int launch_rev_v(const RevTuning& tu, bool fan, bool gmv, unsigned fan_grid, size_t smem,
                 const RowGrid& rg, cudaStream_t st, const RevArgs<T>& A) {
    if (fan) {
        const int threads = 32 * tu.npb;
        return gmv ? launch_rev_fan_m<T, V, true>(tu.minb, fan_grid, threads, smem, st, A)
                   : launch_rev_fan_m<T, V, false>(tu.minb, fan_grid, threads, smem, st, A);
    }
    if (gmv) k_reverse<T, V, true><<<rg.grid, 256, 0, st>>>(A);
    else k_reverse<T, V, false><<<rg.grid, 256, 0, st>>>(A);
    CVFES_LAUNCH_CHECK("k_reverse");
    return CVFES_OK;
}

template <typename T>
int launch_reverse_step(const cvfes_adjoint_desc* d, const T* u, T* uo, const T* x, T* xo,
                        long long n, bool after_step, cudaStream_t st) {
    const cvfes_solid_mesh* m = &d->mesh;
    RevArgs<T> A;
    A.node_ptr = m->node_ptr;
    A.rec = reinterpret_cast<const int4*>(m->slot_rec);
    A.slab = static_cast<const T*>(m->slot_k);
    A.own = static_cast<const T*>(d->owner_blocks);
    A.fhat = static_cast<const T*>(m->fhat);
    A.coef = static_cast<const T*>(d->coef);
    A.invm = static_cast<const T*>(d->invm);
    A.u = u;
    A.uo = uo;
    A.x = x;
    A.xo = xo;
    A.gam = static_cast<T*>(d->gamma);
    A.gm = static_cast<T*>(d->gmass);
    A.p = d->p_sched + n;
    A.n_nodes = m->n_nodes;
    A.S = (int)m->n_samples;
    A.n_clamped = (int)m->n_clamped;
    A.clamp = (T)m->clamp_value;
    A.status = m->status;
    const double g = 0.5 * d->dt * d->damp;
    const double eta = d->dt * d->damp / (1.0 + g);
    A.eta = (T)eta;
    A.inv1meta = (T)(1.0 / (1.0 - eta));
    A.w0 = (T)(d->dt * d->dt / (1.0 + g));
    RevTuning tu = rev_tuning<T>();
    // rows as given (FP64, slot_form 0): the patch and row-gather kernels have that form
    const bool full = mesh_full<T>(m);
    if (full && tu.variant != 0) tu.variant = 2;
    const Prefetch pf = step_prefetch(sizeof(T) == 4 ? 32 : 64, m->bandwidth);
    A.pf_dist = pf.dist;
    A.pf_parts = pf.parts;
    const void* ptrs[8] = {d->coef, d->invm, u, uo, x, xo, d->gamma, d->gmass};
    int V = (int)(16 / sizeof(T));
    while (V > tu.vec) V /= 2;
    for (; V > 1; V /= 2) {
        bool ok = A.S % V == 0;
        for (int i = 0; i < 8; ++i)
            if (ptrs[i] && reinterpret_cast<uintptr_t>(ptrs[i]) % (V * sizeof(T))) ok = false;
        if (ok) break;
    }
    // below 20 samples most lanes of a patch warp would idle: the row-gather kernel (128 x 400
    // wall, FP32, us a step: 16 samples 69 against about 92, 24 samples 104 / 92)
    if (tu.variant == 2 && A.S >= 20) {
        int prc = 1;
        if constexpr (sizeof(T) == 4) {
            if (V >= 2 && (A.S + 31) / 32 > (A.S / 2 + 31) / 32) prc = launch_rev_patch<T, 2>(m, A, after_step, st);
        }
        if constexpr (sizeof(T) == 8) {
            if (full) prc = launch_rev_patch<T, 1, true>(m, A, after_step, st);
        }
        if (prc == 1 && !full) prc = launch_rev_patch<T, 1>(m, A, after_step, st);
        if (prc <= 0) return prc;
    }
    const RowGrid rg = row_grid(m->n_nodes, A.S / V, 256);
    A.tpn = rg.tpn;
    A.npb = rg.npb;
    A.nch = 1;
    A.cap_slots = 0;
    const long long cap = (long long)tu.npb * m->max_degree;
    const size_t smem = 16 + (size_t)cap * (16 + (kSlabStride + kOwnStride) * sizeof(T));
    const bool fan = (tu.variant == 1 || tu.variant == 2) && !full && m->max_degree > 0 &&
                     (A.S / V) % 32 == 0 && smem <= kRevMaxStage && tu.npb >= 1 && tu.npb <= 8;
    unsigned fan_grid = 0;
    if (fan) {
        A.npb = tu.npb;
        A.tpn = 32;
        A.nch = A.S / V / 32;
        A.pf_group = prefetch_group(A.nch);
        A.pf_parts = prefetch_parts(A.pf_parts, A.nch);
        A.cap_slots = (int)cap;
        fan_grid = (unsigned)(((m->n_nodes + A.npb - 1) / A.npb) * A.nch);
    }
    const bool gmv = d->gmass != nullptr;
    if constexpr (sizeof(T) == 8) {
        if (full) {
            auto kernel = V == 2 ? (gmv ? k_reverse<T, 2, true, true> : k_reverse<T, 2, false, true>)
                                 : (gmv ? k_reverse<T, 1, true, true> : k_reverse<T, 1, false, true>);
            kernel<<<rg.grid, 256, 0, st>>>(A);
            CVFES_LAUNCH_CHECK("k_reverse");
            return CVFES_OK;
        }
    }
    if (V == 4) {
        if constexpr (sizeof(T) == 4)
            return launch_rev_v<T, 4>(tu, fan, gmv, fan_grid, smem, rg, st, A);
        return fail(CVFES_ERR_UNSUPPORTED, "k_reverse: vec 4 is FP32 only");
    }
    if (V == 2) return launch_rev_v<T, 2>(tu, fan, gmv, fan_grid, smem, rg, st, A);
    return launch_rev_v<T, 1>(tu, fan, gmv, fan_grid, smem, rg, st, A);
}

int check_adjoint(const cvfes_adjoint_desc* d, const char* who) {
    if (!d) return fail(CVFES_ERR_ARG, "%s: null descriptor", who);
    const cvfes_solid_mesh* m = &d->mesh;
    if (m->n_nodes <= 0 || m->n_samples <= 0 || m->n_samples > INT32_MAX || !m->node_ptr ||
        !m->slot_rec || !m->slot_k || !m->fhat)
        return fail(CVFES_ERR_ARG, "%s: incomplete mesh descriptor", who);
    if (d->precision != 32 && d->precision != 64)
        return fail(CVFES_ERR_ARG, "%s: precision must be 32 or 64", who);
    if (d->n_steps <= 0 || d->ckpt_every <= 0 || d->obs_every <= 0 || d->n_obs < 0)
        return fail(CVFES_ERR_ARG, "%s: steps, checkpoint and observation intervals must be "
                    "positive", who);
    if (!d->coef || !d->invm || !d->owner_blocks || !d->state[0] || !d->state[1] ||
        !d->state[2] || !d->adj[0] || !d->adj[1] || !d->ckpt || !d->p_sched || !d->clock ||
        !d->J || !d->gamma)
        return fail(CVFES_ERR_ARG, "%s: null buffer", who);
    if (d->n_obs > 0 && (!d->obs_nodes || !d->obs || !d->jpart))
        return fail(CVFES_ERR_ARG, "%s: observation buffers missing", who);
    if (!(d->dt > 0.0)) return fail(CVFES_ERR_ARG, "%s: dt must be positive", who);
    return CVFES_OK;
}

__global__ void k_set_clock(long long* clock, long long n) { clock[0] = n; }

template <typename T>
int adjoint_forward(const cvfes_adjoint_desc* d, int* out_cur, int* out_prev, cudaStream_t st) {
    int rc = check_adjoint(d, "cvfes_adjoint_forward");
    if (rc) return rc;
    const cvfes_solid_mesh* m = &d->mesh;
    const long long S = m->n_samples, N = m->n_nodes, T_ = d->n_steps;
    const long long C = d->ckpt_every, K = d->obs_every;
    const size_t state = (size_t)3 * N * S;
    const size_t sbytes = state * sizeof(T);
    T* buf[3] = {static_cast<T*>(d->state[0]), static_cast<T*>(d->state[1]),
                 static_cast<T*>(d->state[2])};
    T* ck = static_cast<T*>(d->ckpt);
    T* obs = static_cast<T*>(d->obs);
    for (int q = 0; q < 3; ++q) CVFES_CUDA_TRY(cudaMemsetAsync(buf[q], 0, sbytes, st));
    CVFES_CUDA_TRY(cudaMemsetAsync(d->J, 0, S * sizeof(double), st));
    const int nchunk = (d->n_obs + kObsChunk - 1) / kObsChunk;
    int cur = 0, prev = 1, nxt = 2;
    long long n = 0;
    while (n < T_) {
        long long next = T_;
        const long long no = (n / K + 1) * K;
        if (no < next) next = no;
        long long mc = (n / C) * C + 1;
        if (mc <= n) mc += C;
        if (mc < next) next = mc;
        int ci = 0, pi = 1;
        const int order[3] = {cur, prev, nxt};
        if constexpr (sizeof(T) == 8)
            rc = cvfes_solid_advance_f64(m, static_cast<const double*>(d->coef),
                                         static_cast<const double*>(d->invm), buf[cur], buf[prev],
                                         buf[nxt], d->p_sched + n, nullptr, next - n, d->dt, d->damp,
                                         &ci, &pi, st);
        else
            rc = cvfes_solid_advance_f32(m, static_cast<const float*>(d->coef),
                                         static_cast<const float*>(d->invm), buf[cur], buf[prev],
                                         buf[nxt], d->p_sched + n, nullptr, next - n, d->dt, d->damp,
                                         &ci, &pi, st);
        if (rc) return rc;
        cur = order[ci];
        prev = order[pi];
        nxt = 3 - cur - prev;
        n = next;
        if ((n - 1) % C == 0) {
            T* slot = ck + (size_t)((n - 1) / C) * 2 * state;
            CVFES_CUDA_TRY(cudaMemcpyAsync(slot, buf[prev], sbytes, cudaMemcpyDeviceToDevice, st));
            CVFES_CUDA_TRY(
                cudaMemcpyAsync(slot + state, buf[cur], sbytes, cudaMemcpyDeviceToDevice, st));
        }
        if (n % K == 0 && d->n_obs > 0) {
            const long long k = n / K - 1;
            dim3 grid((unsigned)nchunk, (unsigned)((S + 127) / 128));
            k_obs<T><<<grid, 128, 0, st>>>(d->n_obs, (int)S, d->obs_nodes, buf[cur],
                                           obs + (size_t)k * d->n_obs * 3 * S,
                                           d->jpart + (size_t)k * nchunk * S, d->record);
            CVFES_LAUNCH_CHECK("k_obs");
        }
    }
    k_set_clock<<<1, 1, 0, st>>>(reinterpret_cast<long long*>(d->clock), T_);
    CVFES_LAUNCH_CHECK("k_set_clock");
    const long long n_obs_steps = T_ / K;
    if (!d->record && d->n_obs > 0 && n_obs_steps > 0) {
        k_obs_reduce<<<grid_1d(S, kReduceSamples), kReduceSamples * kReduceGroups, 0, st>>>(
            n_obs_steps * nchunk, (int)S, d->jpart, d->J);
        CVFES_LAUNCH_CHECK("k_obs_reduce");
    }
    if (out_cur) *out_cur = cur;
    if (out_prev) *out_prev = prev;
    return CVFES_OK;
}

template <typename T>
int adjoint_force(const cvfes_adjoint_desc* d, const T* u, T* chi, long long k, cudaStream_t st) {
    if (d->n_obs <= 0) return CVFES_OK;
    const long long S = d->mesh.n_samples;
    const double g = 0.5 * d->dt * d->damp;
    const T w0 = (T)(d->dt * d->dt / (1.0 + g));
    k_adj_force<T><<<grid_1d((long long)d->n_obs * S, 256), 256, 0, st>>>(
        d->n_obs, (int)S, d->obs_nodes, (int)d->mesh.n_clamped, static_cast<const T*>(d->invm),
        w0, u, static_cast<const T*>(d->obs) + (size_t)k * d->n_obs * 3 * S, chi);
    CVFES_LAUNCH_CHECK("k_adj_force");
    return CVFES_OK;
}

template <typename T>
int adjoint_reverse(const cvfes_adjoint_desc* d, int cur, int prev, cudaStream_t st) {
    int rc = check_adjoint(d, "cvfes_adjoint_reverse");
    if (rc) return rc;
    if (cur < 0 || cur > 2 || prev < 0 || prev > 2 || cur == prev)
        return fail(CVFES_ERR_ARG, "cvfes_adjoint_reverse: bad final state roles");
    const cvfes_solid_mesh* m = &d->mesh;
    const long long S = m->n_samples, N = m->n_nodes, E = m->n_elems, T_ = d->n_steps;
    const long long C = d->ckpt_every, K = d->obs_every;
    const size_t state = (size_t)3 * N * S;
    const size_t sbytes = state * sizeof(T);
    T* uA = static_cast<T*>(d->state[prev]);  // u_n      (starts at u_{T-1})
    T* uB = static_cast<T*>(d->state[cur]);   // u_{n+1}  (starts at u_T)
    T* xA = static_cast<T*>(d->adj[0]);       // chi_{n+1}
    T* xB = static_cast<T*>(d->adj[1]);       // chi_{n+2}
    const T* ck = static_cast<const T*>(d->ckpt);
    CVFES_CUDA_TRY(cudaMemsetAsync(xA, 0, sbytes, st));
    CVFES_CUDA_TRY(cudaMemsetAsync(xB, 0, sbytes, st));
    CVFES_CUDA_TRY(cudaMemsetAsync(d->gamma, 0, (size_t)E * S * sizeof(T), st));
    if (d->gmass) CVFES_CUDA_TRY(cudaMemsetAsync(d->gmass, 0, (size_t)N * S * sizeof(T), st));
    if (T_ % K == 0) {
        rc = adjoint_force<T>(d, uB, xA, T_ / K - 1, st);
        if (rc) return rc;
    }
    bool after_step = false;  // the launch before is a reverse step: this one may overlap it
    for (long long n = T_ - 1; n >= 0; --n) {
        if (n % C == 0) {
            after_step = false;
            const T* slot = ck + (size_t)(n / C) * 2 * state;
            CVFES_CUDA_TRY(cudaMemcpyAsync(uA, slot, sbytes, cudaMemcpyDeviceToDevice, st));
            CVFES_CUDA_TRY(
                cudaMemcpyAsync(uB, slot + state, sbytes, cudaMemcpyDeviceToDevice, st));
        }
        rc = launch_reverse_step<T>(d, uA, uB, xA, xB, n, after_step, st);
        if (rc) return rc;
        after_step = true;
        T* t = uA;
        uA = uB;
        uB = t;
        t = xA;
        xA = xB;
        xB = t;
        // now uA = u_{n-1}, uB = u_n, xA = chi_n, xB = chi_{n+1}
        if (n > 0 && n % K == 0) {
            rc = adjoint_force<T>(d, uB, xA, n / K - 1, st);
            if (rc) return rc;
            after_step = after_step && d->n_obs <= 0;
        }
    }
    return CVFES_OK;
}

template <typename F>
int capture(F&& issue, cvfes_graph** out) {
    cudaStream_t cs;
    CVFES_CUDA_TRY(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) {
        cudaStreamDestroy(cs);
        return fail(CVFES_ERR_CUDA, "begin capture: %s", cudaGetErrorString(e));
    }
    const int rc = issue(cs);
    cudaGraph_t graph = nullptr;
    e = cudaStreamEndCapture(cs, &graph);
    cudaStreamDestroy(cs);
    if (rc) {
        if (graph) cudaGraphDestroy(graph);
        return rc;
    }
    if (e != cudaSuccess) return fail(CVFES_ERR_CUDA, "end capture: %s", cudaGetErrorString(e));
    cudaGraphExec_t exec = nullptr;
    e = cudaGraphInstantiate(&exec, graph, 0);
    if (e != cudaSuccess) {
        cudaGraphDestroy(graph);
        return fail(CVFES_ERR_CUDA, "graph instantiate: %s", cudaGetErrorString(e));
    }
    *out = new cvfes_graph{graph, exec};
    return CVFES_OK;
}

}  // namespace cvfes

using namespace cvfes;

extern "C" int cvfes_set_adjoint_tuning(int32_t precision, int32_t vec, int32_t npb,
                                        int32_t variant, int32_t minb) {
    if ((precision != 32 && precision != 64) || (vec != 1 && vec != 2 && vec != 4) ||
        (precision == 64 && vec == 4) || npb < 1 || npb > 8 || variant < 0 || variant > 2 ||
        minb < 1 || minb > 4 || (variant == 2 && minb > 3))
        return fail(CVFES_ERR_ARG, "cvfes_set_adjoint_tuning: bad argument");
    RevTuning& t = precision == 32 ? g_rev32 : g_rev64;
    t = RevTuning{vec, npb, variant, minb};
    return CVFES_OK;
}

extern "C" int cvfes_get_adjoint_tuning(int32_t precision, int32_t* vec, int32_t* npb,
                                        int32_t* variant, int32_t* minb) {
    if (precision != 32 && precision != 64)
        return fail(CVFES_ERR_ARG, "cvfes_get_adjoint_tuning: precision must be 32 or 64");
    const RevTuning& t = precision == 32 ? g_rev32 : g_rev64;
    if (vec) *vec = t.vec;
    if (npb) *npb = t.npb;
    if (variant) *variant = t.variant;
    if (minb) *minb = t.minb;
    return CVFES_OK;
}

extern "C" int64_t cvfes_adjoint_ckpt_count(int64_t n_steps, int64_t ckpt_every) {
    if (n_steps <= 0 || ckpt_every <= 0) return 0;
    return (n_steps + ckpt_every - 1) / ckpt_every;
}

extern "C" int64_t cvfes_adjoint_jpart_size(int64_t n_steps, int32_t obs_every, int32_t n_obs,
                                            int64_t n_samples) {
    if (n_steps <= 0 || obs_every <= 0 || n_obs <= 0 || n_samples <= 0) return 0;
    return (n_steps / obs_every) * ((n_obs + kObsChunk - 1) / kObsChunk) * n_samples;
}

extern "C" int cvfes_adjoint_owner_blocks(const cvfes_solid_mesh* mesh, int32_t precision,
                                          const int32_t* elems, const int32_t* elem_slot,
                                          void* out, void* stream) {
    if (!mesh || mesh->n_elems <= 0 || !mesh->slot_rec || !mesh->slot_k || !elems || !elem_slot ||
        !out || (precision != 32 && precision != 64))
        return fail(CVFES_ERR_ARG, "cvfes_adjoint_owner_blocks: bad argument");
    const long long E = mesh->n_elems;
    if (precision == 64)
        k_owner_blocks<double><<<grid_1d(E, 256), 256, 0, (cudaStream_t)stream>>>(
            E, elems, elem_slot, mesh->slot_rec, static_cast<const double*>(mesh->slot_k),
            static_cast<double*>(out));
    else
        k_owner_blocks<float><<<grid_1d(E, 256), 256, 0, (cudaStream_t)stream>>>(
            E, elems, elem_slot, mesh->slot_rec, static_cast<const float*>(mesh->slot_k),
            static_cast<float*>(out));
    CVFES_LAUNCH_CHECK("k_owner_blocks");
    return CVFES_OK;
}

extern "C" int cvfes_adjoint_material(int64_t n_elems, int64_t n_samples, const double* logE,
                                      const double* logh, double* coef64, float* coef32,
                                      double* thick, void* stream) {
    if (n_elems <= 0 || n_samples <= 0 || !logE || !logh || (!coef64 && !coef32 && !thick))
        return fail(CVFES_ERR_ARG, "cvfes_adjoint_material: bad argument");
    const long long n = n_elems * n_samples;
    k_material_log<<<grid_1d(n, 256), 256, 0, (cudaStream_t)stream>>>(n, logE, logh, coef64,
                                                                        coef32, thick);
    CVFES_LAUNCH_CHECK("k_material_log");
    return CVFES_OK;
}

extern "C" int cvfes_adjoint_forward(const cvfes_adjoint_desc* d, int32_t* final_cur,
                                     int32_t* final_prev, void* stream) {
    if (!d) return fail(CVFES_ERR_ARG, "cvfes_adjoint_forward: null descriptor");
    if (d->precision == 64) return adjoint_forward<double>(d, final_cur, final_prev, (cudaStream_t)stream);
    return adjoint_forward<float>(d, final_cur, final_prev, (cudaStream_t)stream);
}

extern "C" int cvfes_adjoint_reverse(const cvfes_adjoint_desc* d, int32_t final_cur,
                                     int32_t final_prev, void* stream) {
    if (!d) return fail(CVFES_ERR_ARG, "cvfes_adjoint_reverse: null descriptor");
    if (d->precision == 64) return adjoint_reverse<double>(d, final_cur, final_prev, (cudaStream_t)stream);
    return adjoint_reverse<float>(d, final_cur, final_prev, (cudaStream_t)stream);
}

extern "C" int cvfes_adjoint_gradients(const cvfes_adjoint_desc* d, const int32_t* elems,
                                       const double* area, const double* mass_weights,
                                       const double* lm, const double* logE, const double* logh,
                                       double* grad_logE, double* grad_logh, void* stream) {
    int rc = check_adjoint(d, "cvfes_adjoint_gradients");
    if (rc) return rc;
    if (!elems || !area || !logE || !logh || (!grad_logE && !grad_logh))
        return fail(CVFES_ERR_ARG, "cvfes_adjoint_gradients: bad argument");
    if (grad_logh && (!d->gmass || !lm || !mass_weights))
        return fail(CVFES_ERR_ARG,
                    "cvfes_adjoint_gradients: the log h gradient needs the G accumulator, the "
                    "lumped mass and the mass weights");
    MassWeights mw{};
    if (mass_weights)
        for (int i = 0; i < 9; ++i) mw.w[i] = mass_weights[i];
    const long long E = d->mesh.n_elems, S = d->mesh.n_samples;
    if (d->precision == 64)
        k_grad_final<double><<<grid_1d(E * S, 256), 256, 0, (cudaStream_t)stream>>>(
            E, (int)S, elems, area, mw, lm, logE, logh, static_cast<const double*>(d->gamma),
            static_cast<const double*>(d->gmass), grad_logE, grad_logh);
    else
        k_grad_final<float><<<grid_1d(E * S, 256), 256, 0, (cudaStream_t)stream>>>(
            E, (int)S, elems, area, mw, lm, logE, logh, static_cast<const float*>(d->gamma),
            static_cast<const float*>(d->gmass), grad_logE, grad_logh);
    CVFES_LAUNCH_CHECK("k_grad_final");
    return CVFES_OK;
}

extern "C" int cvfes_adjoint_capture(const cvfes_adjoint_desc* d, int32_t which, int32_t cur,
                                     int32_t prev, int32_t* final_cur, int32_t* final_prev,
                                     cvfes_graph** out) {
    if (!d || !out || (which != 0 && which != 1))
        return fail(CVFES_ERR_ARG, "cvfes_adjoint_capture: bad argument");
    return capture(
        [&](cudaStream_t cs) -> int {
            if (which == 0) return cvfes_adjoint_forward(d, final_cur, final_prev, cs);
            return cvfes_adjoint_reverse(d, cur, prev, cs);
        },
        out);
}
