// Geometric-update ("updated coordinates") form of the membrane solid step.
//
// The stiffness and the follower pressure load of every element are taken on the
// deformed geometry x + u_g of each sample, as the reference's GPU kernel
// assemble_K_P does every step (physicsSolverSDampGPUs.cl:232-393) and its CPU path
// does every `stiffness_update_interval` steps (OptimizedSolidAssembleUpdate,
// optimizedSolidAssemble.pyx:710-819, triggered at physicsSolver.py:296-324):
//   K(x + u_g) u_n   and   p_n * sum_e (A_e / 3) n_e     over the deformed triangles.
// Nothing per sample is stored: the row of node a is formed matrix-free from the
// slot's reference edge vectors X_b - X_a (exact, precomputed) plus the neighbour
// displacement differences, so the FP32 form never subtracts large coordinates.
// The membrane block of an isotropic sheet does not depend on the local frame, so no frame
// is formed.  With q1, q2 the deformed edges from a to its neighbours, e = q2 - q1, n the
// unit normal of nn = q1 x q2 and h1 = q2 x n, h2 = n x q1 (2 A times the gradients of the
// neighbours' shape functions; a's is -(h1 + h2)), the row applied to the displacement
// differences d1, d2 is
//   -K d = c / (4 A (1 - nu^2)) [ h1 (pe1 (h1.d1 + h2.d1) + nu s) + h2 (pe1 (h1.d2 + h2.d2) + nu s)
//                                 + w + (k - 1) (n.w) n ],
//   s = h1.d1 + h2.d2,  w = pe1 ((q2.e) d1 - (q1.e) d2),  pe1 = (1 - nu) / 2,  k = 5/6,
// (-K d: a's own gradient has the minus sign), and the follower load is nn / 6: 93 operations and one rsqrt a slot
// where the frame form took about 170 with two rsqrt and a division.  Rigid translations
// are in the null space, so the row only needs u_b - u_a.  The update of the state is the
// linear form's.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "patch_walk.cuh"
#include "step_core.cuh"

namespace cvfes {

constexpr int kGeoStride = 8;  // X_b1 - X_a (3), X_b2 - X_a (3), pad (2)

// Reference edge vectors of every slot (a = the slot's own node).
__global__ void k_slot_geometry(long long n_slots, const double* __restrict__ nodes,
                                const int32_t* __restrict__ elems,
                                const int32_t* __restrict__ slot_rec, double* __restrict__ geo64,
                                float* __restrict__ geo32) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= n_slots) return;
    const int e = slot_rec[4 * s], b1 = slot_rec[4 * s + 1], b2 = slot_rec[4 * s + 2];
    const int la = (slot_rec[4 * s + 3] >> 8) & 3;
    const int a = elems[3 * (size_t)e + la];
    double g[kGeoStride];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        g[d] = nodes[3 * (size_t)b1 + d] - nodes[3 * (size_t)a + d];
        g[3 + d] = nodes[3 * (size_t)b2 + d] - nodes[3 * (size_t)a + d];
    }
    g[6] = g[7] = 0.0;
#pragma unroll
    for (int q = 0; q < kGeoStride; ++q) {
        if (geo64) geo64[(size_t)kGeoStride * s + q] = g[q];
        if (geo32) geo32[(size_t)kGeoStride * s + q] = (float)g[q];
    }
}

// Element-wise products and sums of V samples with the roundings written out (FP32 pairs as
// one packed instruction), so that every width rounds alike.
template <typename T, int V, typename F2, typename F1>
__device__ __forceinline__ Vec<T, V> vmap(const F2& f2, const F1& f1) {
    Vec<T, V> r;
    if constexpr (std::is_same<T, float>::value && V % 2 == 0) {
#pragma unroll
        for (int i = 0; i < V; i += 2) {
            const float2 q = f2(i);
            r.v[i] = q.x;
            r.v[i + 1] = q.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < V; ++i) r.v[i] = f1(i);
    }
    return r;
}
template <int V>
__device__ __forceinline__ float2 pair(const Vec<float, V>& a, int i) {
    return make_float2(a.v[i], a.v[i + 1]);
}
template <int V>
__device__ __forceinline__ float2 pair(const Vec<double, V>&, int) {
    return make_float2(0.f, 0.f);
}
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }

template <typename T, int V>
__device__ __forceinline__ Vec<T, V> vmul(const Vec<T, V>& a, const Vec<T, V>& b) {
    return vmap<T, V>([&](int i) { return __fmul2_rn(pair(a, i), pair(b, i)); },
                      [&](int i) { return mul_rn(a.v[i], b.v[i]); });
}
template <typename T, int V>
__device__ __forceinline__ Vec<T, V> vadd(const Vec<T, V>& a, const Vec<T, V>& b) {
    return vmap<T, V>([&](int i) { return __fadd2_rn(pair(a, i), pair(b, i)); },
                      [&](int i) { return add_rn(a.v[i], b.v[i]); });
}
template <typename T, int V>
__device__ __forceinline__ Vec<T, V> vfma3(const Vec<T, V>& a, const Vec<T, V>& b,
                                           const Vec<T, V>& c) {
    return vmap<T, V>([&](int i) { return __ffma2_rn(pair(a, i), pair(b, i), pair(c, i)); },
                      [&](int i) { return fma(a.v[i], b.v[i], c.v[i]); });
}
template <typename T, int V>
__device__ __forceinline__ Vec<T, V> vdot(const Vec<T, V> (&a)[3], const Vec<T, V> (&b)[3]) {
    return vfma3(a[2], b[2], vfma3(a[1], b[1], vmul(a[0], b[0])));
}
// a x b, with na = -a beside a
template <typename T, int V>
__device__ __forceinline__ void vcross(Vec<T, V> (&r)[3], const Vec<T, V> (&a)[3],
                                       const Vec<T, V> (&na)[3], const Vec<T, V> (&b)[3]) {
    r[0] = vfma3(na[2], b[1], vmul(a[1], b[2]));
    r[1] = vfma3(na[0], b[2], vmul(a[2], b[0]));
    r[2] = vfma3(na[1], b[0], vmul(a[0], b[1]));
}

template <typename T>
struct GeoConst {
    T nu;
    T pe1;    // (1 - nu) / 2
    T shear;  // k - 1, k = 5/6 the shear factor
    T half;   // 1 / (2 (1 - nu^2))
};

// A neighbour of a: displacement difference and deformed edge from a.
template <typename T, int V>
struct GeoEdge {
    Vec<T, V> d[3], q[3];
};

// Adds -(row of a) of c_e K_e(x + u_g) applied to (A.d, B.d) to acc and nn to load (the
// pressure load is nn / 6).
// SAFE: det = |nn|^2 is the fourth power of an edge; where that leaves FP32's range (edges below
// some 3e-10 or above 4e9) 1 / |nn| is formed from nn over its largest component.
template <typename T, int V, bool SAFE = false>
__device__ __forceinline__ void geo_row(const GeoEdge<T, V>& A, const GeoEdge<T, V>& B,
                                        const Vec<T, V>& c, const GeoConst<T>& K,
                                        Vec<T, V> (&acc)[3], Vec<T, V> (&load)[3]) {
    Vec<T, V> e[3], ne[3], nn[3], n[3], m[3], h1[3], h2[3], w[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        e[i] = vsub(B.q[i], A.q[i]);
        ne[i] = vsub(A.q[i], B.q[i]);
    }
    // nn = q1 x q2 = q1 x e = -(e x q1)
    vcross(nn, ne, e, A.q);
    const Vec<T, V> det = vdot(nn, nn);
    Vec<T, V> rs, nrs;
#pragma unroll
    for (int i = 0; i < V; ++i) {
        rs.v[i] = rsqrt(det.v[i]);
        if constexpr (SAFE) {
            if (!(det.v[i] > T(1e-36) && det.v[i] < T(1e36))) {
                const T inv = T(1) / fmax(fmax(fabs(nn[0].v[i]), fabs(nn[1].v[i])), fabs(nn[2].v[i]));
                const T a = nn[0].v[i] * inv, b = nn[1].v[i] * inv, c2 = nn[2].v[i] * inv;
                rs.v[i] = rsqrt(fma(a, a, fma(b, b, c2 * c2))) * inv;
            }
        }
        nrs.v[i] = -rs.v[i];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        load[i] = vadd(load[i], nn[i]);
        n[i] = vmul(nn[i], rs);
        m[i] = vmul(nn[i], nrs);
    }
    vcross(h1, m, n, B.q);  // q2 x n = (-n) x q2
    vcross(h2, n, m, A.q);  // n x q1
    const Vec<T, V> pe1 = vfill<T, V>(K.pe1);
    const Vec<T, V> w1 = vmul(vdot(B.q, e), pe1), w2 = vmul(vdot(A.q, ne), pe1);
    const Vec<T, V> a11 = vdot(h1, A.d), a21 = vdot(h2, A.d);
    const Vec<T, V> a12 = vdot(h1, B.d), a22 = vdot(h2, B.d);
    const Vec<T, V> ns = vmul(vadd(a11, a22), vfill<T, V>(K.nu));
    const Vec<T, V> b1 = vfma3(vadd(a11, a21), pe1, ns);
    const Vec<T, V> b2 = vfma3(vadd(a12, a22), pe1, ns);
#pragma unroll
    for (int i = 0; i < 3; ++i) w[i] = vfma3(w2, B.d[i], vmul(w1, A.d[i]));
    const Vec<T, V> sm = vmul(vdot(n, w), vfill<T, V>(K.shear));
    const Vec<T, V> scale = vmul(vmul(c, vfill<T, V>(K.half)), rs);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const Vec<T, V> f = vfma3(h1[i], b1, vfma3(h2[i], b2, vfma3(n[i], sm, w[i])));
        acc[i] = vfma3(scale, f, acc[i]);
    }
}

template <typename T>
struct GeoArgs {
    const T* geo;  // [kGeoStride * n_slots] reference edge vectors
    const T* ug;   // geometry displacement (== the step's u when the geometry is current)
    GeoConst<T> K;
};

// Whether a node's FP32 sums may come from elements outside the range of det (geo_row): the load
// (a sum of nn) leaves [1e-16, 1e17], or the row is not finite.  Such nodes are formed again.
template <typename T, int V>
__device__ __forceinline__ bool geo_suspect(const Vec<T, V> (&acc)[3], const Vec<T, V> (&load)[3]) {
    bool bad = false;
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const T m = fmax(fmax(fabs(load[0].v[i]), fabs(load[1].v[i])), fabs(load[2].v[i]));
            bad = bad || !(m > T(1e-16) && m < T(1e17)) || !(fabs(acc[0].v[i]) < T(INFINITY));
        }
    }
    return bad;
}

// Update of one node row from its -K u (acc) and load sums; p6 = pressure / 6.
template <typename T, int V>
__device__ __forceinline__ void geo_update(const StepArgs<T>& A, int a, size_t col, T p6,
                                           const Vec<T, V> (&ua)[3], const Vec<T, V> (&acc)[3],
                                           const Vec<T, V> (&load)[3], bool on) {
    const size_t S = (size_t)A.S;
    const uint32_t rowb = (uint32_t)A.S * sizeof(T), nodeb = 3 * rowb;
    const Vec<T, V> im = ldcs<T, V>(row_at(A.invm + col, a, rowb));
    const T* const up = row_at(A.up + col, a, nodeb);
    T* const un = row_at(A.un + col, a, nodeb);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const Vec<T, V> vo = ld_state<T, V, true>(up + d * S);
        // nodal traction (calc_u_appTrac, physicsSolverSDampGPUs.cl:436-446), one per node
        const T tr = A.trac ? __ldg(A.trac + 4 * (size_t)a + d) : T(0);
        Vec<T, V> o;
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const T dv = ua[d].v[i] - vo.v[i];
            const T w = mul_rn(A.w0, im.v[i]);
            T f = mul_rn(p6, load[d].v[i]);
            if (A.trac) f = add_rn(f, tr);
            const T v = fma(w, add_rn(f, acc[d].v[i]), fma(-row_eta(A, im.v[i]), dv, dv));
            o.v[i] = (im.v[i] != T(0)) ? add_rn(ua[d].v[i], v) : T(0);
        }
        if (on) stcs<T, V>(un + d * S, o);
    }
}

// The sums of a node with k1 - k0 slots, all from global memory.
template <typename T, int V, bool SAME, bool SAFE>
__device__ __forceinline__ void geo_node_sums(const StepArgs<T>& A, const GeoArgs<T>& G, int a,
                                              int k0, int k1, size_t col, Vec<T, V> (&ua)[3],
                                              Vec<T, V> (&acc)[3], Vec<T, V> (&load)[3]) {
    const size_t S = (size_t)A.S;
    const uint32_t nodeb = 3 * (uint32_t)A.S * sizeof(T);
    Vec<T, V> ga[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        ua[d] = ld<T, V>(row_at(A.u + col, a, nodeb) + d * S);
        ga[d] = ld<T, V>(row_at(G.ug + col, a, nodeb) + d * S);
        acc[d] = load[d] = vzero<T, V>();
    }
    GeoEdge<T, V> one, two;
    auto edge = [&](GeoEdge<T, V>& o, int k, int b, int second) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const Vec<T, V> e = vfill<T, V>(__ldg(G.geo + (size_t)kGeoStride * k + 3 * second + d));
            o.d[d] = vsub(ld<T, V>(row_at(A.u + col, b, nodeb) + d * S), ua[d]);
            if constexpr (SAME)
                o.q[d] = vadd(o.d[d], e);
            else
                o.q[d] = vadd(vsub(ld<T, V>(row_at(G.ug + col, b, nodeb) + d * S), ga[d]), e);
        }
    };
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
        const int4 r = __ldg(A.rec + k);
        one = two;
        if (k == k0 || !(r.w & 1)) edge(one, k, r.y, 0);
        edge(two, k, r.z, 1);
        geo_row<T, V, SAFE>(one, two, ldg<T, V>(A.coef + (size_t)r.x * S + col), G.K, acc, load);
    }
}

// One step: a thread walks its node's fan with the next element's neighbour rows and
// coefficient in flight.  Consecutive elements of a fan share an edge, so one neighbour is
// gathered per element (two were, and their rows were 6 of the 7 gathered).  What bounds it
// is the arithmetic: 93 packed or FP64 operations a slot against one row.
// SAME: the geometry is the current state (ug == u).  MAXT, MINB: threads of a block and
// blocks an SM that the registers must allow (0: no say).
template <typename T, int V, bool SAME, int MAXT = 256, int MINB = 0>
__global__ void __launch_bounds__(MAXT, MINB) k_step_geo(StepArgs<T> A, GeoArgs<T> G) {
    const int t = threadIdx.x / A.tpn;
    const long long a = (long long)blockIdx.x * A.npb + t;
    const int vec = blockIdx.y * A.tpn + (threadIdx.x - t * A.tpn);
    const bool active = t < A.npb && a < A.n_nodes && vec * V < A.S;
    int k = 0, k1 = 0;
    if (active) {
        k = __ldg(A.node_ptr + a);
        k1 = __ldg(A.node_ptr + a + 1);
    }
    grid_dependency_release();
    grid_dependency_wait();
    if (!active) return;
    const size_t S = (size_t)A.S, col = (size_t)vec * V;
    const uint32_t rowb = (uint32_t)A.S * sizeof(T), nodeb = 3 * rowb;
    if (a < A.n_clamped) {
        const Vec<T, V> cl = vfill<T, V>(A.clamp);
#pragma unroll
        for (int d = 0; d < 3; ++d) stcs<T, V>(row_at(A.un + col, (int)a, nodeb) + d * S, cl);
        return;
    }
    const T* const u = A.u + col;
    const T* const ug = G.ug + col;
    Vec<T, V> ua[3], ga[SAME ? 1 : 3], acc[3], load[3];
    auto rows = [&](Vec<T, V> (&x)[3], const T* q) {
#pragma unroll
        for (int d = 0; d < 3; ++d) x[d] = ld<T, V>(q + d * S);
    };
    rows(ua, row_at(u, (int)a, nodeb));
    if constexpr (!SAME) rows(ga, row_at(ug, (int)a, nodeb));
#pragma unroll
    for (int d = 0; d < 3; ++d) acc[d] = load[d] = vzero<T, V>();
    // raw rows of a neighbour, and the reference edge to it (first or second of slot k)
    Vec<T, V> x[3], g[SAME ? 1 : 3], c, cn;
    T E[3];
    auto request = [&](int slot, int b, int second) {
        rows(x, row_at(u, b, nodeb));
        if constexpr (!SAME) rows(g, row_at(ug, b, nodeb));
#pragma unroll
        for (int d = 0; d < 3; ++d) E[d] = __ldg(G.geo + (size_t)kGeoStride * slot + 3 * second + d);
    };
    auto edge = [&](GeoEdge<T, V>& o) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            o.d[d] = vsub(x[d], ua[d]);
            if constexpr (SAME)
                o.q[d] = vadd(o.d[d], vfill<T, V>(E[d]));
            else
                o.q[d] = vadd(vsub(g[d], ga[d]), vfill<T, V>(E[d]));
        }
    };
    if (k < k1) {
        GeoEdge<T, V> P, Q;
        int4 r = __ldg(A.rec + k);
        request(k, r.y, 0);
        edge(P);
        request(k, r.z, 1);
        cn = ldg<T, V>(row_at(A.coef + col, r.x, rowb));
        auto phase = [&](GeoEdge<T, V>& first, GeoEdge<T, V>& second) {
            edge(second);
            c = cn;
            const bool more = k + 1 < k1;
            if (more) {
                r = __ldg(A.rec + k + 1);
                request(k + 1, r.z, 1);
                cn = ldg<T, V>(row_at(A.coef + col, r.x, rowb));
            }
            geo_row<T, V>(first, second, c, G.K, acc, load);
            if (more && !(r.w & 1)) {  // fan break: the next first neighbour is a new one
                request(k + 1, r.y, 0);
                edge(second);
                request(k + 1, r.z, 1);
            }
            ++k;
        };
        while (true) {
            phase(P, Q);
            if (k >= k1) break;
            phase(Q, P);
            if (k >= k1) break;
        }
    }
    const T p6 = step_pressure<T>(A) * T(1.0 / 6.0);
    if (k1 > __ldg(A.node_ptr + a) && geo_suspect<T, V>(acc, load)) {
        const LaunchAgain L;
        const int t2 = L.thread / A.tpn, a2 = L.block * A.npb + t2;
        const size_t col2 = (size_t)(blockIdx.y * A.tpn + (L.thread - t2 * A.tpn)) * V;
        geo_node_sums<T, V, SAME, true>(A, G, a2, __ldg(A.node_ptr + a2),
                                        __ldg(A.node_ptr + a2 + 1), col2, ua, acc, load);
        geo_update<T, V>(A, a2, col2, p6, ua, acc, load, true);
        return;
    }
    geo_update<T, V>(A, (int)a, col, p6, ua, acc, load, true);
}

// The same step with free-running warps on patches of nodes (patch_walk.cuh): 32 * V samples
// of one node at a time, the next node's slots staged in shared memory and its rows
// prefetched into L2 under the current one.  As in the linear step the plain kernel's time
// went into DRAM misses of first-touched rows: 128 x 400 wall, 128 samples, FP32 306 -> 193 us
// a step; 64 samples, FP64 329 -> 232 us.
// Warps of a block (one block an SM): what the registers allow.  FP32 pairs, 128 x 400 wall,
// 128 samples, us a step at 16 / 20 / 24 warps: current geometry 221 / 204 / 193, stored
// geometry - / 236 / 248 (200 bytes spilled).
template <typename T, bool SAME>
struct GeoWarps {
    static constexpr int kWarps = sizeof(T) == 4 ? (SAME ? 24 : 20) : 16;
};
// The nodes of this warp that the patch kernel did not write (more slots than max_degree, or
// sums that geo_suspect points out): after all others, and everything found again from the launch, so that they cost its loop no
// registers (10 steps of the 128 x 400 wall, FP32, 128 samples: 1.97 ms without them, 2.01 with,
// 2.05 with a function call in or after the loop).
template <typename T, int V, bool SAME, int W>
__device__ __forceinline__ void geo_unstaged(const StepArgs<T>& A, const GeoArgs<T>& G,
                                             const PatchMap& M, int max_degree) {
    const LaunchAgain L;
    const int vec = L.block % A.nch * 32 + (L.thread & 31), last = A.S / V - 1;
    const size_t col = (size_t)min(vec, last) * V;
    PatchWalk walk(M, L.thread >> 5, L.block / A.nch, L.blocks / A.nch, A.n_clamped,
                   (int)A.n_nodes, W);
    for (; walk.more(M); walk.advance(M)) {
        const int a = walk.node(M);
        if (a < 0) continue;
        const int k0 = __ldg(A.node_ptr + a), k1 = __ldg(A.node_ptr + a + 1);
        Vec<T, V> ua[3], acc[3], load[3];
        geo_node_sums<T, V, SAME, false>(A, G, a, k0, k1, col, ua, acc, load);
        if (geo_suspect<T, V>(acc, load) && k1 > k0)
            geo_node_sums<T, V, SAME, true>(A, G, a, k0, k1, col, ua, acc, load);
        else if (k1 - k0 <= max_degree)
            continue;  // this lane has written its samples in the loop
        geo_update<T, V>(A, a, col, step_pressure<T>(A) * T(1.0 / 6.0), ua, acc, load,
                         vec <= last);
    }
}

template <typename T, int V, bool SAME>
__global__ void __launch_bounds__(32 * GeoWarps<T, SAME>::kWarps, 1)
    k_step_geo_patch(StepArgs<T> A, GeoArgs<T> G, PatchMap M, int max_degree) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int W = GeoWarps<T, SAME>::kWarps;
    constexpr int kWords = kGeoStride * (int)sizeof(T) / 16;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t b_rec = 16u * max_degree, b_stage = b_rec + 16u * kWords * max_degree;
    unsigned char* const wb = smem + warp * (2 * b_stage);
    const uint32_t rowb = (uint32_t)A.S * sizeof(T), nodeb = 3 * rowb;
    const int chunk = blockIdx.x % A.nch;
    const int vec = chunk * 32 + lane, last = A.S / V - 1;
    const bool on = vec <= last;
    const size_t S = (size_t)A.S, col = (size_t)(on ? vec : last) * V;
    const int bpc = gridDim.x / A.nch;
    PatchWalk walk(M, warp, blockIdx.x / A.nch, bpc, A.n_clamped, (int)A.n_nodes, W);
    auto stage = [&](int b, int k0, int n, int sg) {
        if (b >= 0) {
            const uint32_t d = smem_u32(wb + sg * b_stage);
            const char* r = reinterpret_cast<const char*>(A.rec + k0);
            const char* g = reinterpret_cast<const char*>(G.geo + (size_t)k0 * kGeoStride);
            for (int q = lane; q < n; q += 32) cp_async<16>(d + 16 * q, r + 16 * q);
            for (int q = lane; q < kWords * n; q += 32) cp_async<16>(d + b_rec + 16 * q, g + 16 * q);
        }
        cp_async_commit();
    };
    __shared__ int unstaged[W];  // a node of the warp was not written
    if (lane == 0) unstaged[warp] = 0;
    __syncwarp();
    bool more = walk.more(M);
    int a = walk.node(M), n, an, k0, nn;
    node_slots(A.node_ptr, max_degree, unstaged + warp, a, k0, n);
    stage(a, k0, n, 0);
    walk.advance(M);
    an = walk.node(M);
    node_slots(A.node_ptr, max_degree, unstaged + warp, an, k0, nn);
    const RowLines<T, V> ln(lane, chunk, rowb);
    const char* const obase =
        reinterpret_cast<const char*>(ln.row < 3   ? A.u + (size_t)ln.row * S
                                      : ln.row < 6 ? A.up + (size_t)(ln.row - 3) * S
                                                   : A.invm) + ln.off;
    const uint32_t ostride = ln.row < 6 ? nodeb : rowb;
    const char* const cbase = reinterpret_cast<const char*>(A.coef) + ln.off;
    const T* const u = A.u + col;
    const T* const ug = G.ug + col;
    grid_dependency_release();
    grid_dependency_wait();
    const T p = step_pressure<T>(A) * T(1.0 / 6.0);
    for (int b = blockIdx.x / A.nch * W + warp; b < A.n_clamped; b += bpc * W) {
        const Vec<T, V> cl = vfill<T, V>(A.clamp);
#pragma unroll
        for (int d = 0; d < 3; ++d)
            if (on) stcs<T, V>(row_at(A.un + col, b, nodeb) + d * S, cl);
    }
    for (int sg = 0; more; sg ^= 1) {
        Vec<T, V> ua[3], ga[SAME ? 1 : 3];
        auto rows = [&](Vec<T, V> (&x)[3], const T* q) {
#pragma unroll
            for (int d = 0; d < 3; ++d) x[d] = ld<T, V>(q + d * S);
        };
        if (a >= 0) {
            rows(ua, row_at(u, a, nodeb));
            if constexpr (!SAME) rows(ga, row_at(ug, a, nodeb));
        }
        cp_async_wait_all();
        __syncwarp();
        const unsigned char* const st = wb + sg * b_stage;
        const int4* const srec = reinterpret_cast<const int4*>(st);
        const T* const sgeo = reinterpret_cast<const T*>(st + b_rec);
        stage(an, k0, nn, sg ^ 1);
        if (an >= 0 && ln.row < 7 && ln.on) prefetch_l2(obase + (uint64_t)(uint32_t)an * ostride);
        const int nn_cur = nn;
        more = walk.more(M);
        walk.advance(M);
        int ax = walk.node(M);
        node_slots(A.node_ptr, max_degree, unstaged + warp, ax, k0, nn);
        if (a >= 0) {
            Vec<T, V> acc[3], load[3], x[3], g[SAME ? 1 : 3], c, cn;
            T E[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) acc[d] = load[d] = vzero<T, V>();
            auto request = [&](int slot, int b, int second) {
                rows(x, row_at(u, b, nodeb));
                if constexpr (!SAME) rows(g, row_at(ug, b, nodeb));
#pragma unroll
                for (int d = 0; d < 3; ++d) E[d] = sgeo[kGeoStride * slot + 3 * second + d];
            };
            auto edge = [&](GeoEdge<T, V>& o) {
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    o.d[d] = vsub(x[d], ua[d]);
                    if constexpr (SAME)
                        o.q[d] = vadd(o.d[d], vfill<T, V>(E[d]));
                    else
                        o.q[d] = vadd(vsub(g[d], ga[d]), vfill<T, V>(E[d]));
                }
            };
            if (n > 0) {
                GeoEdge<T, V> P, Q;
                int k = 0;
                request(0, srec[0].y, 0);
                edge(P);
                request(0, srec[0].z, 1);
                cn = ldg<T, V>(row_at(A.coef + col, srec[0].x, rowb));
                auto phase = [&](GeoEdge<T, V>& one, GeoEdge<T, V>& two) {
                    edge(two);
                    c = cn;
                    const bool next = k + 1 < n;
                    int4 r = make_int4(0, 0, 0, 1);
                    if (next) {
                        r = srec[k + 1];
                        request(k + 1, r.z, 1);
                        cn = ldg<T, V>(row_at(A.coef + col, r.x, rowb));
                    }
                    geo_row<T, V>(one, two, c, G.K, acc, load);
                    if (next && !(r.w & 1)) {  // fan break: the next first neighbour is new
                        request(k + 1, r.y, 0);
                        edge(two);
                        request(k + 1, r.z, 1);
                    }
                    ++k;
                };
                while (true) {
                    phase(P, Q);
                    if (k >= n) break;
                    phase(Q, P);
                    if (k >= n) break;
                }
            }
            cp_async_wait_all();
            __syncwarp();
            if (an >= 0 && ln.on && ln.row < nn_cur)
                prefetch_l2(cbase + (uint64_t)(uint32_t)reinterpret_cast<const int4*>(
                                        wb + (sg ^ 1) * b_stage)[ln.row].x * rowb);
            if (geo_suspect<T, V>(acc, load) && n > 0)
                unstaged[threadIdx.x >> 5] = 1;
            else
                geo_update<T, V>(A, a, col, p, ua, acc, load, on);
        }
        __syncwarp();
        a = an;
        n = nn_cur;
        an = ax;
    }
    cp_async_wait_all();
    __syncwarp();
    if (unstaged[threadIdx.x >> 5]) geo_unstaged<T, V, SAME, W>(A, G, M, max_degree);
}

struct GeoTuning {
    int vec;    // samples per thread (upper bound; 4 runs as 2, one packed pair)
    int block;  // threads per block (64, 128 or 256)
};
static GeoTuning g_geo32 = {2, 128};
static GeoTuning g_geo64 = {1, 128};

template <typename T>
int launch_step_geo(const cvfes_solid_mesh* m, const T* coef, const T* invm, const T* geo,
                    const T* u, const T* up, T* un, const T* ug, const double* p_sched,
                    const long long* clock, long long j, double pressure, const T* trac,
                    double nu, double dt, double damp, cudaStream_t st, bool after_step = false) {
    if (!m || m->n_nodes <= 0 || m->n_samples <= 0 || m->n_samples > INT32_MAX || !m->node_ptr ||
        !m->slot_rec || m->n_clamped < 0 || m->n_clamped > m->n_nodes)
        return fail(CVFES_ERR_ARG, "cvfes_solid_step_geo: incomplete mesh descriptor");
    if (!coef || !invm || !geo || !u || !up || !un)
        return fail(CVFES_ERR_ARG, "cvfes_solid_step_geo: null pointer");
    if (!(dt > 0.0) || !(nu > -1.0 && nu < 0.5))
        return fail(CVFES_ERR_ARG, "cvfes_solid_step_geo: dt must be positive and nu in (-1, 0.5)");
    StepArgs<T> A{};
    A.node_ptr = m->node_ptr;
    A.rec = reinterpret_cast<const int4*>(m->slot_rec);
    A.coef = coef;
    A.invm = invm;
    A.u = u;
    A.up = up;
    A.un = un;
    A.p_sched = p_sched;
    A.clock = clock;
    A.j = j;
    A.pressure = pressure;
    A.trac = trac;
    A.n_nodes = m->n_nodes;
    A.S = (int)m->n_samples;
    A.n_clamped = (int)m->n_clamped;
    A.clamp = (T)m->clamp_value;
    const double g = 0.5 * dt * damp;
    if (m->damping_form == 1) {  // damping force per dof: eta = dt damp / m, no LHS term
        A.damp_per_dof = 1;
        A.eta = (T)(dt * damp);
        A.w0 = (T)(dt * dt);
    } else {
        A.eta = (T)(dt * damp / (1.0 + g));
        A.w0 = (T)(dt * dt / (1.0 + g));
    }
    A.status = m->status;
    GeoArgs<T> G;
    G.geo = geo;
    G.ug = ug ? ug : u;
    G.K.nu = (T)nu;
    G.K.pe1 = (T)(0.5 * (1.0 - nu));
    G.K.shear = (T)(5.0 / 6.0 - 1.0);
    G.K.half = (T)(0.5 / (1.0 - nu * nu));
    const bool same = G.ug == u;
    const void* ptrs[6] = {coef, invm, u, up, un, G.ug};
    const GeoTuning& tu = sizeof(T) == 4 ? g_geo32 : g_geo64;
    int V = std::min(2, tu.vec);
    for (; V > 1; V /= 2) {
        bool ok = A.S % V == 0;
        for (int i = 0; i < 6; ++i)
            if (reinterpret_cast<uintptr_t>(ptrs[i]) % (V * sizeof(T))) ok = false;
        if (ok) break;
    }
    if (m->n_samples >= (1 << 27) || m->n_nodes >= INT32_MAX)
        return fail(CVFES_ERR_ARG, "cvfes_solid_step_geo: too many samples or nodes");
    const int W = same ? GeoWarps<T, true>::kWarps : GeoWarps<T, false>::kWarps;
    const size_t stages = (size_t)W * 2 * (16 + kGeoStride * sizeof(T)) * m->max_degree;
    // The patch kernel where the samples fill its warps: at least 3/4 of the lanes, or 9/10
    // when the step's rows (100 MB) fit L2 and there are few DRAM misses to hide.  us a
    // step, plain / patch: 128 x 400 wall, FP32 128 samples 306 / 204, 100 samples (78%
    // filled) 264 / 211, 40 samples (62%) 94 / 109; FP64 64 samples 329 / 232, 50 samples
    // (78%) 285 / 240; 96 x 200 wall (92 MB), FP64 50 samples 88 / 94, 64 samples 109 / 94.
    A.nch = (A.S / V + 31) / 32;
    const double lanes = (double)(A.S / V) / (32.0 * A.nch);
    const bool in_l2 = 12.0 * m->n_nodes * A.S * sizeof(T) < 100e6;
    if ((sizeof(T) == 4 || V == 1) && lanes >= (in_l2 ? 0.9 : 0.75) && m->max_degree > 0 &&
        m->max_degree < 1024 && stages <= 96 * 1024 &&
        reinterpret_cast<uintptr_t>(geo) % 16 == 0) {  // (staged in 16-byte words)
        const PatchMap M = patch_map(m->n_nodes - A.n_clamped, m->bandwidth, W);
        constexpr int V2 = sizeof(T) == 4 ? 2 : 1;  // (FP64 pairs would spill)
        auto kp = V == 2 ? (same ? k_step_geo_patch<T, V2, true> : k_step_geo_patch<T, V2, false>)
                         : (same ? k_step_geo_patch<T, 1, true> : k_step_geo_patch<T, 1, false>);
        int per_sm = 0;
        const int rc = fanp_blocks_per_sm(reinterpret_cast<const void*>(kp), 32 * W, stages, &per_sm);
        if (rc) return rc;
        const long long places =
            std::max<long long>((long long)M.n_strips * M.tps, (A.n_clamped + W - 1) / W);
        const long long per_chunk = std::max(
            1LL, std::min((long long)per_sm * device_sm_count() / A.nch, places));
        return launch_step_kernel(kp, dim3((unsigned)(per_chunk * A.nch)), 32 * W, stages,
                                  after_step, st, "k_step_geo_patch", A, G, M,
                                  (int)m->max_degree);
    }
    // lanes of a node: its sample vectors in equal parts of at most 32 (the whole block where
    // that would make more parts than a grid has rows)
    const int sv = A.S / V, most = sv > 65535 * 32 ? tu.block : 32, parts = (sv + most - 1) / most;
    A.tpn = (sv + parts - 1) / parts;
    A.npb = tu.block / A.tpn;
    const dim3 grid((unsigned)((m->n_nodes + A.npb - 1) / A.npb), (unsigned)parts);
    auto kernel = V == 2 ? (same ? k_step_geo<T, 2, true> : k_step_geo<T, 2, false>)
                         : (same ? k_step_geo<T, 1, true> : k_step_geo<T, 1, false>);
    // On the current geometry FP64 singles and FP32 pairs fit 96 registers, five blocks of 128
    // threads an SM: 96 x 200 wall, FP64 50 samples 88 -> 74 us a step, 128 x 400 wall, FP32 40
    // samples 93 -> 80 (stored geometry at 96 registers: 98 -> 106).
    constexpr int VT = sizeof(T) == 4 ? 2 : 1;
    if (same && V == VT && tu.block <= 128) kernel = k_step_geo<T, VT, true, 128, 5>;
    return launch_step_kernel(kernel, grid, tu.block, 0, after_step, st, "k_step_geo", A, G);
}

__global__ void k_geo_clock_add(long long* clock, long long n) { clock[0] += n; }

// n_steps geometric steps with the reference's update counter: before each step, if
// counter >= interval the geometry becomes the current state (copied into ugeo, or
// read straight from u_n when interval == 1) and counter = 1, else counter += 1.
template <typename T>
int launch_advance_geo(const cvfes_solid_mesh* m, const T* coef, const T* invm, const T* geo,
                       T* b0, T* b1, T* b2, T* ugeo, const double* p_sched, long long* clock,
                       long long n_steps, long long interval, long long* counter, int geo_live,
                       double nu, double dt, double damp, int* cur_idx, int* prev_idx,
                       int* geo_live_out, cudaStream_t st) {
    if (n_steps < 0 || interval < 1 || !counter || !p_sched || !ugeo)
        return fail(CVFES_ERR_ARG, "cvfes_solid_advance_geo: bad argument");
    T* buf[3] = {b0, b1, b2};
    int cur = 0, prev = 1, nxt = 2;
    const size_t bytes = (size_t)3 * m->n_nodes * m->n_samples * sizeof(T);
    long long c = *counter;
    bool live = geo_live != 0;  // geometry is the current state (interval 1 after an update)
    for (long long j = 0; j < n_steps; ++j) {
        bool after_step = j > 0;  // the launch before this one is the previous step
        if (c >= interval) {
            if (interval == 1) {
                live = true;
            } else {
                CVFES_CUDA_TRY(cudaMemcpyAsync(ugeo, buf[cur], bytes, cudaMemcpyDeviceToDevice, st));
                after_step = false;
            }
            c = 1;
        } else {
            c += 1;
        }
        const T* ug = live ? buf[cur] : ugeo;
        int rc = launch_step_geo<T>(m, coef, invm, geo, buf[cur], buf[prev], buf[nxt], ug, p_sched,
                                    clock, j, 0.0, nullptr, nu, dt, damp, st, after_step);
        if (rc) return rc;
        const int old_prev = prev;
        prev = cur;
        cur = nxt;
        nxt = old_prev;
    }
    if (clock && n_steps > 0) {
        k_geo_clock_add<<<1, 1, 0, st>>>(clock, n_steps);
        CVFES_LAUNCH_CHECK("k_geo_clock_add");
    }
    *counter = c;
    if (cur_idx) *cur_idx = cur;
    if (prev_idx) *prev_idx = prev;
    if (geo_live_out) *geo_live_out = live ? 1 : 0;
    return CVFES_OK;
}

}  // namespace cvfes

using namespace cvfes;

extern "C" int cvfes_set_geo_tuning(int32_t precision, int32_t vec, int32_t block) {
    if ((precision != 32 && precision != 64) || (vec != 1 && vec != 2 && vec != 4) ||
        (precision == 64 && vec == 4) || (block != 64 && block != 128 && block != 256))
        return fail(CVFES_ERR_ARG, "cvfes_set_geo_tuning: bad argument");
    GeoTuning& t = precision == 32 ? g_geo32 : g_geo64;
    t = GeoTuning{vec, block};
    return CVFES_OK;
}

extern "C" int cvfes_get_geo_tuning(int32_t precision, int32_t* vec, int32_t* block) {
    if (precision != 32 && precision != 64)
        return fail(CVFES_ERR_ARG, "cvfes_get_geo_tuning: precision must be 32 or 64");
    const GeoTuning& t = precision == 32 ? g_geo32 : g_geo64;
    if (vec) *vec = t.vec;
    if (block) *block = t.block;
    return CVFES_OK;
}

extern "C" int cvfes_solid_slot_geometry_f64(int64_t n_elems, const double* nodes,
                                             const int32_t* elems, const int32_t* slot_rec,
                                             double* geo64, float* geo32, void* stream) {
    if (n_elems <= 0 || !nodes || !elems || !slot_rec || (!geo64 && !geo32))
        return fail(CVFES_ERR_ARG, "cvfes_solid_slot_geometry_f64: bad argument");
    const long long ns = 3 * n_elems;
    k_slot_geometry<<<grid_1d(ns, 256), 256, 0, (cudaStream_t)stream>>>(ns, nodes, elems, slot_rec,
                                                                         geo64, geo32);
    CVFES_LAUNCH_CHECK("k_slot_geometry");
    return CVFES_OK;
}

extern "C" int cvfes_solid_step_geo_f64(const cvfes_solid_mesh* mesh, const double* coef,
                                        const double* invm, const double* slot_geo,
                                        const double* u, const double* up, double* un,
                                        const double* ug, const double* p_sched,
                                        const int64_t* clock, int64_t j, double pressure,
                                        const double* trac, double nu, double dt, double damp,
                                        void* stream) {
    return launch_step_geo<double>(mesh, coef, invm, slot_geo, u, up, un, ug, p_sched,
                                   reinterpret_cast<const long long*>(clock), j, pressure, trac,
                                   nu, dt, damp, (cudaStream_t)stream);
}

extern "C" int cvfes_solid_step_geo_f32(const cvfes_solid_mesh* mesh, const float* coef,
                                        const float* invm, const float* slot_geo, const float* u,
                                        const float* up, float* un, const float* ug,
                                        const double* p_sched, const int64_t* clock, int64_t j,
                                        double pressure, const float* trac, double nu, double dt,
                                        double damp, void* stream) {
    return launch_step_geo<float>(mesh, coef, invm, slot_geo, u, up, un, ug, p_sched,
                                  reinterpret_cast<const long long*>(clock), j, pressure, trac,
                                  nu, dt, damp, (cudaStream_t)stream);
}

extern "C" int cvfes_solid_advance_geo_f64(const cvfes_solid_mesh* mesh, const double* coef,
                                           const double* invm, const double* slot_geo,
                                           double* buf0, double* buf1, double* buf2, double* ugeo,
                                           const double* p_sched, int64_t* clock, int64_t n_steps,
                                           int64_t interval, int64_t* counter, int32_t geo_live,
                                           double nu, double dt, double damp, int32_t* cur_idx,
                                           int32_t* prev_idx, int32_t* geo_live_out,
                                           void* stream) {
    long long c = counter ? *counter : 0;
    const int rc = launch_advance_geo<double>(
        mesh, coef, invm, slot_geo, buf0, buf1, buf2, ugeo, p_sched,
        reinterpret_cast<long long*>(clock), n_steps, interval, counter ? &c : nullptr, geo_live,
        nu, dt, damp, cur_idx, prev_idx, geo_live_out, (cudaStream_t)stream);
    if (!rc && counter) *counter = c;
    return rc;
}

extern "C" int cvfes_solid_advance_geo_f32(const cvfes_solid_mesh* mesh, const float* coef,
                                           const float* invm, const float* slot_geo, float* buf0,
                                           float* buf1, float* buf2, float* ugeo,
                                           const double* p_sched, int64_t* clock, int64_t n_steps,
                                           int64_t interval, int64_t* counter, int32_t geo_live,
                                           double nu, double dt, double damp, int32_t* cur_idx,
                                           int32_t* prev_idx, int32_t* geo_live_out,
                                           void* stream) {
    long long c = counter ? *counter : 0;
    const int rc = launch_advance_geo<float>(
        mesh, coef, invm, slot_geo, buf0, buf1, buf2, ugeo, p_sched,
        reinterpret_cast<long long*>(clock), n_steps, interval, counter ? &c : nullptr, geo_live,
        nu, dt, damp, cur_idx, prev_idx, geo_live_out, (cudaStream_t)stream);
    if (!rc && counter) *counter = c;
    return rc;
}
