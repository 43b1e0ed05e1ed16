// Element stress recovery per sample (OptimizedCalculateStress,
// optimizedSolidAssemble.pyx:1116-1223, called from physicsSolver.py:416-424 at each
// save): on the element frame of the geometry x + u_g, the local displacement
// TT u_e, the five local stresses E * D B lU (membrane xx, yy, xy and transverse
// shear xz, yz; D / (1 - nu^2) with shear factor 5/6), the local tensor
// [[xx, xy, xz], [xy, yy, yz], [xz, yz, 0]] rotated to the global frame (T^T s T),
// and its xx, yy, xy, xz, yz entries.  B annihilates rigid translations, so the
// displacement enters as differences from the element's node 0 (exact in FP32 for
// small relative motion).
//
// On the undeformed wall the frame is the element's, not the sample's, so the five global
// stresses are E times a 5 x 6 matrix of the element applied to (u_1 - u_0, u_2 - u_0): a
// block forms the matrices of its elements (one thread each, FP64), then every thread applies
// one to V samples, 30 products in place of some 150 operations.  What bounds it then is
// the stores (5 of 7 values moved): a warp's results, contiguous in memory but 5 V values
// apart in its lanes, pass through shared memory and leave as whole 16-byte lines.
// 256 x 400 wall, 128 samples, FP32: 365 -> 171 us (0.89 GB, 5.2 TB/s).  With few samples the
// matrices bound it; formed without the frame (stress_matrix) they take some 170 FP64 operations
// and 30 conversions.
// On a deformed wall (ug) the frame is formed per (element, sample), one thread each.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "step_core.cuh"

namespace cvfes {

template <typename T>
__global__ void k_stress(long long n_elems, int S, const double* __restrict__ nodes,
                         const int32_t* __restrict__ elems, const double* __restrict__ young,
                         const T* __restrict__ u, const T* __restrict__ ug, T nu,
                         T* __restrict__ stress) {
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long e = g / S;
    if (e >= n_elems) return;
    const int s = (int)(g - e * S);
    const int n0 = elems[3 * e], n1 = elems[3 * e + 1], n2 = elems[3 * e + 2];
    const int nid[3] = {n0, n1, n2};
    // positions relative to node 0 and displacement differences
    T P[3][3], du[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const size_t rk = (3 * (size_t)nid[k] + d) * S + s;
            const size_t r0 = (3 * (size_t)n0 + d) * S + s;
            const T x = (T)(nodes[3 * (size_t)nid[k] + d] - nodes[3 * (size_t)n0 + d]);
            P[k][d] = k == 0 ? T(0) : x + (ug ? ug[rk] - ug[r0] : T(0));
            du[k][d] = k == 0 ? T(0) : u[rk] - u[r0];
        }
    T ex[3], ey[3], ez[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) ex[d] = P[2][d] - P[1][d];
    T inv = rsqrt(ex[0] * ex[0] + ex[1] * ex[1] + ex[2] * ex[2]);
#pragma unroll
    for (int d = 0; d < 3; ++d) ex[d] *= inv;
#pragma unroll
    for (int d = 0; d < 3; ++d) ey[d] = P[0][d] - P[2][d];
    const T pr = ex[0] * ey[0] + ex[1] * ey[1] + ex[2] * ey[2];
#pragma unroll
    for (int d = 0; d < 3; ++d) ey[d] -= pr * ex[d];
    inv = rsqrt(ey[0] * ey[0] + ey[1] * ey[1] + ey[2] * ey[2]);
#pragma unroll
    for (int d = 0; d < 3; ++d) ey[d] *= inv;
    ez[0] = ex[1] * ey[2] - ex[2] * ey[1];
    ez[1] = ex[2] * ey[0] - ex[0] * ey[2];
    ez[2] = ex[0] * ey[1] - ex[1] * ey[0];
    T lx[3], ly[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lx[k] = P[k][0] * ex[0] + P[k][1] * ex[1] + P[k][2] * ex[2];
        ly[k] = P[k][0] * ey[0] + P[k][1] * ey[1] + P[k][2] * ey[2];
    }
    const T area = T(0.5) * ((lx[1] * ly[2] - lx[2] * ly[1]) - (lx[0] * ly[2] - lx[2] * ly[0]) +
                             (lx[0] * ly[1] - lx[1] * ly[0]));
    const T b[3] = {ly[1] - ly[2], ly[2] - ly[0], ly[0] - ly[1]};
    const T c[3] = {lx[2] - lx[1], lx[0] - lx[2], lx[1] - lx[0]};
    // local strains B lU (B = [b; c] / (2 area))
    T exx = 0, eyy = 0, gxy = 0, gxz = 0, gyz = 0;
#pragma unroll
    for (int k = 1; k < 3; ++k) {
        const T lu = ex[0] * du[k][0] + ex[1] * du[k][1] + ex[2] * du[k][2];
        const T lv = ey[0] * du[k][0] + ey[1] * du[k][1] + ey[2] * du[k][2];
        const T lw = ez[0] * du[k][0] + ez[1] * du[k][1] + ez[2] * du[k][2];
        exx += b[k] * lu;
        eyy += c[k] * lv;
        gxy += c[k] * lu + b[k] * lv;
        gxz += b[k] * lw;
        gyz += c[k] * lw;
    }
    const T inv2a = T(1) / (T(2) * area);
    const T E = (T)young[(size_t)e * S + s];
    const T f = E / (T(1) - nu * nu) * inv2a;
    const T k56 = T(5) / T(6);
    const T sxx = f * (exx + nu * eyy);
    const T syy = f * (nu * exx + eyy);
    const T sxy = f * T(0.5) * (T(1) - nu) * gxy;
    const T sxz = f * T(0.5) * k56 * (T(1) - nu) * gxz;
    const T syz = f * T(0.5) * k56 * (T(1) - nu) * gyz;
    // global tensor G = T^T L T, L = [[sxx, sxy, sxz], [sxy, syy, syz], [sxz, syz, 0]]
    const T L[3][3] = {{sxx, sxy, sxz}, {sxy, syy, syz}, {sxz, syz, T(0)}};
    const T* R[3] = {ex, ey, ez};
    T G[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            T acc = 0;
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int q = 0; q < 3; ++q) acc += R[p][i] * L[p][q] * R[q][j];
            G[i][j] = acc;
        }
    T* o = stress + ((size_t)e * S + s) * 5;
    o[0] = G[0][0];
    o[1] = G[1][1];
    o[2] = G[0][1];
    o[3] = G[0][2];
    o[4] = G[1][2];
}

constexpr int kStressThreads = 128;

// The 5 x 6 matrix of an element with corners P (FP64, rounded once); scale = 1 / (1 - nu^2).
template <typename T>
__device__ __forceinline__ void stress_matrix(const double (&P)[3][3], double nu, double scale,
                                              T* m) {
    // With n the unit normal and h_k the in-plane gradient of node k's shape function, the
    // stress of a displacement e_d of node k is, times E / (1 - nu^2),
    //   nu h_d (1 - n n^T) + (1 - nu) / 2 (h w^T + w h^T),   w = e_d - (1 - k) n_d n,
    // k = 5/6 the shear factor: the isotropic sheet in the frame's own directions, the
    // transverse shear in w.
    double g[3], r[3], n[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        g[d] = P[1][d] - P[0][d];
        r[d] = P[2][d] - P[0][d];
    }
    n[0] = g[1] * r[2] - g[2] * r[1];
    n[1] = g[2] * r[0] - g[0] * r[2];
    n[2] = g[0] * r[1] - g[1] * r[0];
    const double inv = rsqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);  // 1 / (2 area)
#pragma unroll
    for (int d = 0; d < 3; ++d) n[d] *= inv;
    // gradients: n x (opposite edge) / (2 area), the edge of node 1 from 2 to 0, of node 2
    // from 0 to 1
    const double f = inv * scale;
    const double h[2][3] = {{f * (r[1] * n[2] - r[2] * n[1]), f * (r[2] * n[0] - r[0] * n[2]),
                             f * (r[0] * n[1] - r[1] * n[0])},
                            {f * (n[1] * g[2] - n[2] * g[1]), f * (n[2] * g[0] - n[0] * g[2]),
                             f * (n[0] * g[1] - n[1] * g[0])}};
    constexpr int I[5] = {0, 1, 0, 0, 1}, J[5] = {0, 1, 1, 2, 2};  // xx, yy, xy, xz, yz
    const double sh = 0.5 * (1.0 - nu), drop = 1.0 / 6.0;
    double proj[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) proj[q] = nu * ((I[q] == J[q] ? 1.0 : 0.0) - n[I[q]] * n[J[q]]);
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            double w[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) w[i] = sh * ((i == d ? 1.0 : 0.0) - drop * n[d] * n[i]);
#pragma unroll
            for (int q = 0; q < 5; ++q)
                m[6 * q + 3 * k + d] = (T)(h[k][d] * proj[q] + h[k][I[q]] * w[J[q]] +
                                                w[I[q]] * h[k][J[q]]);
        }
}

// One stress per unit E of V samples from its six matrix entries and the differences (r1, r2).
template <typename T, int V>
__device__ __forceinline__ Vec<T, V> stress_of(const T* m, const Vec<T, V> (&r1)[3],
                                               const Vec<T, V> (&r2)[3]) {
    Vec<T, V> t = vzero<T, V>();
#pragma unroll
    for (int d = 0; d < 3; ++d) axpy(t, m[d], r1[d]);
#pragma unroll
    for (int d = 0; d < 3; ++d) axpy(t, m[3 + d], r2[d]);
    return t;
}

// One sample vector an element: one thread an element, the matrix in its registers.
template <typename T, int V>
__global__ void __launch_bounds__(kStressThreads)
    k_stress_undeformed_one(long long n_elems, int S, const double* __restrict__ nodes,
                            const int32_t* __restrict__ elems, const double* __restrict__ young,
                            const T* __restrict__ u, double nu, double scale,
                            T* __restrict__ stress) {
    const long long e = blockIdx.x * (long long)kStressThreads + threadIdx.x;
    if (e >= n_elems) return;
    int n[3];
    double P[3][3];
    Vec<T, V> r0[3], r1[3], r2[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        n[k] = elems[3 * e + k];
#pragma unroll
        for (int d = 0; d < 3; ++d) P[k][d] = nodes[3 * (size_t)n[k] + d];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        r0[d] = ldg<T, V>(u + (3 * (size_t)n[0] + d) * S);
        r1[d] = ldg<T, V>(u + (3 * (size_t)n[1] + d) * S);
        r2[d] = ldg<T, V>(u + (3 * (size_t)n[2] + d) * S);
    }
    T m[30], E[V], o[5 * V];
#pragma unroll
    for (int i = 0; i < V; ++i) E[i] = (T)__ldcs(young + (size_t)e * S + i);
    stress_matrix<T>(P, nu, scale, m);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        r1[d] = vsub(r1[d], r0[d]);
        r2[d] = vsub(r2[d], r0[d]);
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        const Vec<T, V> t = stress_of<T, V>(m + 6 * q, r1, r2);
#pragma unroll
        for (int i = 0; i < V; ++i) o[5 * i + q] = E[i] * t.v[i];
    }
    T* w = stress + (size_t)e * S * 5;
    if constexpr (V * sizeof(T) == 16) {
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            Vec<T, V> x;
#pragma unroll
            for (int c = 0; c < V; ++c) x.v[c] = o[V * i + c];
            stcs<T, V>(w + V * i, x);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 5 * V; ++i) __stcs(w + i, o[i]);
    }
}

// EB elements a block, their matrices through shared memory; gridDim.y parts of the sample
// vectors.
template <typename T, int V, int EB>
__global__ void __launch_bounds__(kStressThreads)
    k_stress_undeformed(long long n_elems, int S, const double* __restrict__ nodes,
                        const int32_t* __restrict__ elems, const double* __restrict__ young,
                        const T* __restrict__ u, double nu, double scale, T* __restrict__ stress) {
    constexpr int kVec = 16 / (int)sizeof(T);
    // [stress][6 displacement differences]: pairs are read as one access, and the rows of up to
    // 16 elements of a warp lie in different banks
    __shared__ __align__(16) T mat[EB][30];
    __shared__ int nid[EB][3];
    __shared__ __align__(16) T out[kStressThreads / 32][32 * 5 * V];
    const long long e0 = (long long)blockIdx.x * EB;
    const int ne = (int)min((long long)EB, n_elems - e0);
    if ((int)threadIdx.x < ne) {
        const int l = threadIdx.x;
        double P[3][3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            nid[l][k] = elems[3 * (e0 + l) + k];
#pragma unroll
            for (int d = 0; d < 3; ++d) P[k][d] = nodes[3 * (size_t)nid[l][k] + d];
        }
        stress_matrix<T>(P, nu, scale, mat[l]);
    }
    __syncthreads();
    // (element, sample vector) pairs of the block in memory order, 32 a warp
    const int sv = S / V, total = ne * sv, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T* const w = out[warp];
    for (int base = (blockIdx.y * (kStressThreads / 32) + warp) * 32; base < total;
         base += kStressThreads * gridDim.y) {
        const int idx = base + lane, n = min(32, total - base);
        if (lane < n) {
            const int l = idx / sv;
            const size_t col = (size_t)(idx - l * sv) * V;
            Vec<T, V> r0[3], r1[3], r2[3], E;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                r0[d] = ldg<T, V>(u + (3 * (size_t)nid[l][0] + d) * S + col);
                r1[d] = ldg<T, V>(u + (3 * (size_t)nid[l][1] + d) * S + col);
                r2[d] = ldg<T, V>(u + (3 * (size_t)nid[l][2] + d) * S + col);
            }
            const double* y = young + (size_t)(e0 + l) * S + col;
#pragma unroll
            for (int i = 0; i < V; ++i) E.v[i] = (T)__ldcs(y + i);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                r1[d] = vsub(r1[d], r0[d]);
                r2[d] = vsub(r2[d], r0[d]);
            }
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                const Vec<T, V> t = stress_of<T, V>(mat[l] + 6 * q, r1, r2);
#pragma unroll
                for (int i = 0; i < V; ++i) w[(lane * V + i) * 5 + q] = E.v[i] * t.v[i];
            }
        }
        __syncwarp();
        T* o = stress + ((size_t)e0 * S + (size_t)base * V) * 5;
        if constexpr (V == kVec) {
            for (int i = lane; i < n * 5; i += 32)
                stcs<T, kVec>(o + kVec * i,
                              lds<T, kVec>(reinterpret_cast<unsigned char*>(w + kVec * i)));
        } else {
            for (int i = lane; i < n * 5 * V; i += 32) __stcs(o + i, w[i]);
        }
        __syncwarp();
    }
}

template <typename T>
int launch_stress(long long n_elems, long long S, const double* nodes, const int32_t* elems,
                  const double* young, const T* u, const T* ug, double nu, T* stress,
                  cudaStream_t st) {
    if (n_elems <= 0 || S <= 0 || S > INT32_MAX || !nodes || !elems || !young || !u || !stress)
        return fail(CVFES_ERR_ARG, "cvfes_solid_stress: bad argument");
    if (!ug && S <= (1 << 24)) {
        int V = (int)(16 / sizeof(T));
        while (V > 1 && (S % V || reinterpret_cast<uintptr_t>(u) % (V * sizeof(T)) ||
                         reinterpret_cast<uintptr_t>(stress) % 16))
            V /= 2;
        // One vector an element: a thread each.  Few vectors: 128 elements a block, so that all
        // its threads form matrices; more: 32, and below eight blocks an SM the vectors in parts
        // (each part forms its elements' matrices again).  us a call back to back, a frame per
        // (element, sample) as on a deformed wall / 32 elements a block whatever the size / this
        // rule: FP32 2,016 elements x 256 samples 10.3 / 16.5 / 6.3; 20,352 x 3 4.5 / 6.2 / 6.2;
        // 204,288 x 1 6.2 / 18.6 / 7.4, x 4 14.4 / 20.6 / 10.4, x 37 111 / 100 / 93; FP64 2,016 x
        // 256 16.5 / 34.9 / 10.4; 204,288 x 1 10.3 / 20.1 / 8.3.  (One to three FP32 samples
        // of large walls pay up to 2 us for the FP64 matrix, whose error is half the frame's.)
        const long long sv = S / V;
        const bool one = sv == 1, few = sv <= 4;
        const int EB = few ? kStressThreads : 32;
        const long long bx = (n_elems + EB - 1) / EB;
        const long long parts = one ? 1 : (EB * sv + kStressThreads - 1) / kStressThreads;
        const long long by =
            std::max(1LL, std::min(std::min(parts, 65535LL), 8LL * device_sm_count() / bx));
        const dim3 grid((unsigned)bx, (unsigned)by);
#define CVFES_STRESS(VV)                                                               \
    (one ? k_stress_undeformed_one<T, VV>                                              \
         : few ? k_stress_undeformed<T, VV, kStressThreads> : k_stress_undeformed<T, VV, 32>) \
        <<<grid, kStressThreads, 0, st>>>(n_elems, (int)S, nodes, elems, young, u, nu, \
                                          1.0 / (1.0 - nu * nu), stress)
        if (V == 4) {
            if constexpr (sizeof(T) == 4) CVFES_STRESS(4);
        } else if (V == 2) {
            CVFES_STRESS(2);
        } else {
            CVFES_STRESS(1);
        }
#undef CVFES_STRESS
        CVFES_LAUNCH_CHECK("k_stress_undeformed");
        return CVFES_OK;
    }
    k_stress<T><<<grid_1d(n_elems * S, 256), 256, 0, st>>>(n_elems, (int)S, nodes, elems, young,
                                                           u, ug, (T)nu, stress);
    CVFES_LAUNCH_CHECK("k_stress");
    return CVFES_OK;
}

}  // namespace cvfes

using namespace cvfes;

extern "C" int cvfes_solid_stress_f64(int64_t n_elems, int64_t n_samples, const double* nodes,
                                      const int32_t* elems, const double* young, const double* u,
                                      const double* ug, double nu, double* stress, void* stream) {
    return launch_stress<double>(n_elems, n_samples, nodes, elems, young, u, ug, nu, stress,
                                 (cudaStream_t)stream);
}

extern "C" int cvfes_solid_stress_f32(int64_t n_elems, int64_t n_samples, const double* nodes,
                                      const int32_t* elems, const double* young, const float* u,
                                      const float* ug, double nu, float* stress, void* stream) {
    return launch_stress<float>(n_elems, n_samples, nodes, elems, young, u, ug, nu, stress,
                                (cudaStream_t)stream);
}
