// Patch-ordered persistent step (step variant 6, the default): the template step of
// solid_step.cu with free-running warps.
//
// A warp owns one node and one chunk of 32 * V samples at a time and walks its own
// sequence of nodes; nothing in the loop waits for another warp.  What bounds the step is
// the latency of its gathers, first of all the DRAM misses of rows that no warp has read
// yet, so the kernel is laid out around those (256x512 tube, FP32, 256 samples; the step
// streams 2.06 GB):
//   * the W warps of a block (16, 20 or 28: PatchBlock) take the 4 x W/4 nodes of a patch
//     (four runs of consecutive nodes, one mesh row apart), so the neighbour and coefficient
//     rows they share are read from L2 once: with 16, L1 hits 50% against 34% for runs of four
//     nodes (the SM <- L2 path saturates near 10 TB/s on this chip, and 27 rows a node make
//     2.7 GB);
//   * while a node is multiplied, the rows of the warp's next node that come from DRAM
//     are prefetched into L2 one 128-byte line per lane: its u, u_{n-1} and inverse mass
//     rows when the node starts, its elements' coefficient rows once its slot records
//     have arrived.  All of them or nothing: 484 us without, 471 with the coefficient rows
//     alone, 494 with the node rows alone, 418 with both;
//   * slot records and stiffness rows of the next node are copied into the warp's own
//     shared-memory stage (cp.async) under the current node: no block barrier;
//   * the closed fan of six elements, the interior node of a triangulated surface, is
//     unrolled with the rows of element k + 2 requested before element k is multiplied,
//     and the epilogue rows in the place of elements 6 and 7: 750 instructions a node
//     against 1036 in the loop form (other fans take a loop, one element ahead).
// Measured there: 582 -> 385 us (5.2 TB/s, 81% of the copy rate; 451 us once the board is at
// its power limit, after some 0.1 s); FP64, 64 samples, previous-displacement form:
// 363 -> 228 us, 210 us in the difference form (242 us a step in a call of 20).  5 blocks of 4
// warps at 96 registers spill and are slower (488 us), as are 8 x 2 and 2 x 8 patches (+10%).
// (These figures are of read-only state loads; ld_state in their place, no warp barriers in the
// fan and one address a neighbour give the same: 256 x 512 wall, FP32, 256 samples, 50 steps
// 22.55 ms before and 22.53 after, FP64, 64 samples, 20 steps 4.85 and 4.85 ms.)
//
// Sample counts that do not fill the last chunk leave its lanes without a store (they
// repeat the last samples' loads).  Nodes of more slots than the stages hold follow after the
// loop, from global memory.  Every product and sum is formed in the order of the other step
// kernels, so the bits are the same.  FULL: FP64 rows applied as given (slot_form 0).
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "patch_walk.cuh"
#include "step_core.cuh"

namespace cvfes {

// One node row's update (increment form) and store; su, sv, nf: its norm terms.
template <typename T, int V, bool VEL, bool NORMS>
__device__ __forceinline__ void patch_epilogue(const StepArgs<T>& A, T* un, T* vel,
                                               const Vec<T, V> (&ua)[3],
                                               const Vec<T, V> (&acc)[3], const T (&f)[3],
                                               const Vec<T, V> (&vo)[3], const Vec<T, V>& im,
                                               bool on, T (&su)[V], T (&sv)[V], int (&nf)[V]) {
    bool live = true;
#pragma unroll
    for (int i = 0; i < V; ++i) live = live && im.v[i] != T(0);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        Vec<T, V> o, vn;
        if constexpr (std::is_same<T, float>::value && V % 2 == 0) {
#pragma unroll
            for (int h = 0; h < V; h += 2) {
                const float2 im2 = make_float2(im.v[h], im.v[h + 1]);
                const float2 ua2 = make_float2(ua[d].v[h], ua[d].v[h + 1]);
                const float2 w = __fmul2_rn(make_float2(A.w0, A.w0), im2);
                float2 dv = make_float2(vo[d].v[h], vo[d].v[h + 1]);
                if constexpr (!VEL) dv = __ffma2_rn(dv, make_float2(-1.f, -1.f), ua2);
                float2 eta = make_float2(-A.eta, -A.eta);
                if (A.damp_per_dof) eta = __fmul2_rn(eta, im2);
                const float2 r =
                    __ffma2_rn(make_float2(acc[d].v[h], acc[d].v[h + 1]), make_float2(-1.f, -1.f),
                               make_float2(f[d], f[d]));
                const float2 v = __ffma2_rn(w, r, __ffma2_rn(eta, dv, dv));
                const float2 s = __fadd2_rn(ua2, v);
                vn.v[h] = v.x;
                vn.v[h + 1] = v.y;
                o.v[h] = s.x;
                o.v[h + 1] = s.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < V; ++i) {
                const T dv = VEL ? vo[d].v[i] : ua[d].v[i] - vo[d].v[i];
                const T w = A.w0 * im.v[i];
                const T v = fma(w, f[d] - acc[d].v[i], fma(-row_eta(A, im.v[i]), dv, dv));
                vn.v[i] = v;
                o.v[i] = ua[d].v[i] + v;
            }
        }
        if (!live) {  // a row without mass: u = 0, the exact increment -u
#pragma unroll
            for (int i = 0; i < V; ++i) {
                if (im.v[i] == T(0)) {
                    o.v[i] = T(0);
                    vn.v[i] = -ua[d].v[i];
                }
            }
        }
        if constexpr (NORMS) {
#pragma unroll
            for (int i = 0; i < V; ++i) {
                const T du = VEL ? vn.v[i] : o.v[i] - ua[d].v[i];
                su[i] = fma(o.v[i], o.v[i], su[i]);
                sv[i] = fma(du, du, sv[i]);
                nf[i] += isfinite(o.v[i]) ? 0 : 1;
            }
        }
        if (on) {
            stcs<T, V>(un + d * (size_t)A.S, o);
            if constexpr (VEL) stcs<T, V>(vel + d * (size_t)A.S, vn);
        }
    }
}

// NORMS: 0 none; 1 the per-sample norms of the new state, each lane's sums in tensor
// memory; 2 the same in shared memory behind the stages.  The grid is a multiple of the
// chunks, so a block keeps one chunk for its whole life and writes one row of partials.
template <typename T, int V, bool VEL, int NORMS, int W, bool FULL>
__global__ void __launch_bounds__(32 * W, 1)
    k_step_patch(StepArgs<T> A, PatchMap M, int max_degree) {
    extern __shared__ __align__(16) unsigned char smem[];
    using P = SlotStage<T, FULL>;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t b_rec = 16u * max_degree, b_stage = b_rec + P::kSlotBytes * max_degree;
    unsigned char* const wb = smem + warp * (2 * b_stage);
    const uint32_t rowb = (uint32_t)A.S * sizeof(T), nodeb = 3 * rowb;
    const int chunk = blockIdx.x % A.nch;
    const int vec = chunk * 32 + lane, last = A.S / V - 1;
    const bool on = vec <= last;
    const size_t col = (size_t)(on ? vec : last) * V;
    const T* const u0 = A.u + col;
    const T* const cf = A.coef + col;
    const int n_nodes = (int)A.n_nodes, first = A.n_clamped;

    const int bpc = gridDim.x / A.nch;  // blocks of a chunk
    PatchWalk walk(M, warp, blockIdx.x / A.nch, bpc, first, n_nodes, W);
    // ---- slot staging: lane l copies word l % kWords of every (32 / kWords)-th slot from
    // l / kWords, or every 32nd word where whole rows are staged (FULL); records one a lane
    const int qs = lane / P::kWords, qw = lane - qs * P::kWords;
    auto stage = [&](int b, int k0, int n, int sg) {
        if (b >= 0) {
            const uint32_t d = smem_u32(wb + sg * b_stage);
            const char* r = reinterpret_cast<const char*>(A.rec + k0);
            const char* s = reinterpret_cast<const char*>(A.slab + (size_t)k0 * kSlabStride);
            for (int q = lane; q < n; q += 32) cp_async<16>(d + 16 * q, r + 16 * q);
            if constexpr (P::kWords < 14) {
                constexpr int kPer = 32 / P::kWords;
                for (int q = qs; q < n && qs < kPer; q += kPer)
                    cp_async<16>(d + b_rec + q * P::kSlotBytes + qw * 16,
                                 s + q * (kSlabStride * (int)sizeof(T)) + (P::kFirst + qw) * 16);
            } else {
                for (int q = lane; q < P::kWords * n; q += 32)
                    cp_async<16>(d + b_rec + 16 * q, s + 16 * q);
            }
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

    // ---- line prefetch: u, u_{n-1} and inverse mass rows of a node; coefficient rows
    const RowLines<T, V> ln(lane, chunk, rowb);
    const char* const obase =
        reinterpret_cast<const char*>(ln.row < 3   ? A.u + (size_t)ln.row * A.S
                                      : ln.row < 6 ? A.up + (size_t)(ln.row - 3) * A.S
                                                   : A.invm) + ln.off;
    const uint32_t ostride = ln.row < 6 ? nodeb : rowb;
    const char* const cbase = reinterpret_cast<const char*>(A.coef) + ln.off;

    grid_dependency_release();
    grid_dependency_wait();
    const T p = step_pressure<T>(A);

    // ---- norm accumulators
    constexpr int kAcc = 4 * V * 32;  // doubles of one warp's sums
    double* const nbase = reinterpret_cast<double*>(smem + W * (2 * b_stage));
    double* const nacc = nbase + warp * kAcc + lane;
    uint32_t tm = 0;
    __shared__ uint32_t tmem_slot;
    if constexpr (NORMS == 1) {
        if (warp == 0) {
            tmem_alloc(&tmem_slot, 32 * (W / 4));
            tmem_relinquish();
        }
        tmem_fence_before_sync();
        __syncthreads();
        tmem_fence_after_sync();
        tm = tmem_slot + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(warp >> 2) * 32u;
        norms_zero<V>(tm);
    }
    if constexpr (NORMS == 2) {
#pragma unroll
        for (int q = 0; q < 4 * V; ++q) nacc[q * 32] = 0.0;
    }
    auto add_norms = [&](const Vec<T, V>& im, const T (&su)[V], const T (&sv)[V],
                         const int (&nf)[V]) {
        if constexpr (NORMS == 1) norms_add<T, V>(tm, im, su, sv, nf);
        if constexpr (NORMS == 2) norms_add_smem<T, V>(nacc, im, su, sv, nf);
    };

    // ---- clamped rows
    for (int b = blockIdx.x / A.nch * W + warp; b < first; b += bpc * W) {
        const Vec<T, V> cl = vfill<T, V>(A.clamp);
        T su[V], sv[V];
        int nf[V];
#pragma unroll
        for (int i = 0; i < V; ++i) {
            su[i] = sv[i] = T(0);
            nf[i] = 0;
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (VEL || NORMS) {
                const Vec<T, V> dv =
                    vsub(cl, ld_state<T, V>(row_at(u0, b, nodeb) + d * (size_t)A.S));
                if (VEL && on) stcs<T, V>(row_at(A.vel + col, b, nodeb) + d * (size_t)A.S, dv);
                if constexpr (NORMS != 0) {
#pragma unroll
                    for (int i = 0; i < V; ++i) {
                        su[i] = fma(cl.v[i], cl.v[i], su[i]);
                        sv[i] = fma(dv.v[i], dv.v[i], sv[i]);
                        nf[i] += isfinite(cl.v[i]) ? 0 : 1;
                    }
                }
            }
            if (on) stcs<T, V>(row_at(A.un + col, b, nodeb) + d * (size_t)A.S, cl);
        }
        if constexpr (NORMS != 0)
            add_norms(ldcs<T, V>(row_at(A.invm + col, b, rowb)), su, sv, nf);
    }

    // ---- free rows
    for (int sg = 0; more; sg ^= 1) {
        Vec<T, V> ua[3];
        if (a >= 0) {
            const T* q = row_at(u0, a, nodeb);
            ua[0] = ld_state<T, V>(q);
            ua[1] = ld_state<T, V>(q + A.S);
            ua[2] = ld_state<T, V>(q + 2 * (size_t)A.S);
        }
        cp_async_wait_all();
        __syncwarp();
        const unsigned char* const st = wb + sg * b_stage;
        const int4* const srec = reinterpret_cast<const int4*>(st);
        const T* const K = reinterpret_cast<const T*>(st + b_rec) - 16 / (int)sizeof(T) * P::kFirst;
        constexpr int kStep = P::kSlotBytes / (int)sizeof(T);
        stage(an, k0, nn, sg ^ 1);
        if (an >= 0 && ln.row < 7 && ln.on) prefetch_l2(obase + (uint64_t)(uint32_t)an * ostride);
        const int nn_cur = nn;
        more = walk.more(M);
        walk.advance(M);
        int ax = walk.node(M);
        node_slots(A.node_ptr, max_degree, unstaged + warp, ax, k0, nn);
        // coefficient rows of the next node's elements (the first kRows of them: a loop
        // over more cost the spill-free allocation, 385 -> 400 us and FP64 228 -> 270 us)
        auto prefetch_coef = [&]() {
            cp_async_wait_all();
            __syncwarp();
            const int4* nr = reinterpret_cast<const int4*>(wb + (sg ^ 1) * b_stage);
            if (an >= 0 && ln.on && ln.row < nn_cur)
                prefetch_l2(cbase + (uint64_t)(uint32_t)nr[ln.row].x * rowb);
        };
        if (a >= 0) {
            // one address and two additions: base pointers for the three rows cost four more
            // registers, which FP32 spills (90 x 301 wall, 100 samples, 24 steps: 1135 us,
            // with them 1166)
            auto rows = [&](Vec<T, V> (&x)[3], int b) {
                const T* q = row_at(u0, b, nodeb);
                x[0] = ld_state<T, V>(q);
                x[1] = ld_state<T, V>(q + A.S);
                x[2] = ld_state<T, V>(q + 2 * (size_t)A.S);
            };
            Vec<T, V> acc[3], vo[3], im;
            T f[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) acc[d] = vzero<T, V>();
            auto epilogue_rows = [&]() {
                node_load<T>(A, a, p, f);
                im = ldcs<T, V>(row_at(A.invm + col, a, rowb));
                const T* q = row_at(A.up + col, a, nodeb);
#pragma unroll
                for (int d = 0; d < 3; ++d) vo[d] = ld_state<T, V, true>(q + d * (size_t)A.S);
            };
            const int flag = lane < n ? srec[lane].w : 1;
            if (n == 6 && __all_sync(0xffffffffu, (flag & 1) || lane == 0)) {
                Vec<T, V> X[7][3], C[6];
                const int4 r0 = srec[0], r1 = srec[1];
                rows(X[0], r0.y);
                rows(X[1], r0.z);
                C[0] = ldg<T, V>(row_at(cf, r0.x, rowb));
                rows(X[2], r1.z);
                C[1] = ldg<T, V>(row_at(cf, r1.x, rowb));
                to_diff<T, V, FULL>(X[0], ua);
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    if (k < 4) {
                        const int4 r = srec[k + 2];
                        rows(X[(k + 3) % 7], r.z);
                        C[(k + 2) % 6] = ldg<T, V>(row_at(cf, r.x, rowb));
                    }
                    if (k == 4) epilogue_rows();
                    if (k == 2) prefetch_coef();
                    to_diff<T, V, FULL>(X[k + 1], ua);
                    slot_fma<T, V, FULL>(K + kStep * k, C[k], X[k], X[k + 1], ua, acc);
                }
            } else {
                if (n > 0) {  // any fan: three buffers rotate, one element ahead
                    Vec<T, V> B0[3], B1[3], B2[3], c0, c1, c2;
                    const int4 r0 = srec[0];
                    rows(B0, r0.y);
                    rows(B1, r0.z);
                    c1 = ldg<T, V>(row_at(cf, r0.x, rowb));
                    to_diff<T, V, FULL>(B0, ua);
                    int k = 0;
                    auto phase = [&](Vec<T, V> (&prev)[3], Vec<T, V> (&cur)[3], const Vec<T, V>& c,
                                     Vec<T, V> (&nx)[3], Vec<T, V>& cn) {
                        const bool next = k + 1 < n;
                        int4 r = make_int4(0, 0, 0, 1);
                        if (next) {
                            r = srec[k + 1];
                            rows(nx, r.z);
                            cn = ldg<T, V>(row_at(cf, r.x, rowb));
                        }
                        to_diff<T, V, FULL>(cur, ua);
                        slot_fma<T, V, FULL>(K + kStep * k, c, prev, cur, ua, acc);
                        if (next && !(r.w & 1)) {  // fan break: a first neighbour of its own
                            rows(cur, r.y);
                            to_diff<T, V, FULL>(cur, ua);
                        }
                        ++k;
                    };
                    while (true) {
                        phase(B0, B1, c1, B2, c2);
                        if (k >= n) break;
                        phase(B1, B2, c2, B0, c0);
                        if (k >= n) break;
                        phase(B2, B0, c0, B1, c1);
                        if (k >= n) break;
                    }
                }
                epilogue_rows();
                prefetch_coef();
            }
            T su[V], sv[V];
            int nf[V];
#pragma unroll
            for (int i = 0; i < V; ++i) {
                su[i] = sv[i] = T(0);
                nf[i] = 0;
            }
            patch_epilogue<T, V, VEL, NORMS != 0>(A, row_at(A.un + col, a, nodeb),
                                                  VEL ? row_at(A.vel + col, a, nodeb) : nullptr,
                                                  ua, acc, f, vo, im, on, su, sv, nf);
            if constexpr (NORMS != 0) add_norms(im, su, sv, nf);
        }
        __syncwarp();
        a = an;
        n = nn_cur;
        an = ax;
    }
    cp_async_wait_all();
    __syncwarp();
    if (unstaged[threadIdx.x >> 5]) {  // after all others, so that they cost the loop no registers
        const LaunchAgain L;
        const int vec2 = L.block % A.nch * 32 + (L.thread & 31);
        const bool on2 = vec2 * V < A.S;
        const size_t S = (size_t)A.S, col2 = (size_t)min(vec2, A.S / V - 1) * V;
        const uint32_t rb = (uint32_t)A.S * sizeof(T);
        const T p2 = step_pressure<T>(A);
        PatchWalk again(M, L.thread >> 5, L.block / A.nch, L.blocks / A.nch, A.n_clamped,
                        (int)A.n_nodes, W);
        for (; again.more(M); again.advance(M)) {
            const int b = again.node(M);
            if (b < 0) continue;
            const int s0 = __ldg(A.node_ptr + b), ns = __ldg(A.node_ptr + b + 1) - s0;
            if (ns <= max_degree) continue;
            Vec<T, V> ua[3], acc[3], vo[3];
            T f[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                ua[d] = ld_state<T, V>(row_at(A.u + col2, b, 3 * rb) + d * S);
                vo[d] = ld_state<T, V, true>(row_at(A.up + col2, b, 3 * rb) + d * S);
                acc[d] = vzero<T, V>();
            }
            ku_row_unstaged<T, V, FULL>(A.rec + s0, A.slab + (size_t)s0 * kSlabStride,
                                  ns, A.u + col2, A.coef + col2, rb, ua,
                                  acc);
            const Vec<T, V> im = ldcs<T, V>(row_at(A.invm + col2, b, rb));
            node_load<T>(A, b, p2, f);
            T su[V], sv[V];
            int nf[V];
#pragma unroll
            for (int i = 0; i < V; ++i) {
                su[i] = sv[i] = T(0);
                nf[i] = 0;
            }
            patch_epilogue<T, V, VEL, NORMS != 0>(A, row_at(A.un + col2, b, 3 * rb),
                                                  VEL ? row_at(A.vel + col2, b, 3 * rb) : nullptr,
                                                  ua, acc, f, vo, im, on2, su, sv, nf);
            if constexpr (NORMS != 0) add_norms(im, su, sv, nf);
        }
    }

    if constexpr (NORMS != 0) {  // the block's row of partials, its warps added in order
        double* const scr = reinterpret_cast<double*>(smem);
        __syncthreads();
        if constexpr (NORMS == 1) {
            for (int w = 0; w < W; ++w) {
                if (warp == w) norms_fold<V>(tm, scr + lane, w == 0);
                __syncthreads();
            }
        }
        const long long prow = blockIdx.x / A.nch;
        for (int t = threadIdx.x; t < kAcc; t += blockDim.x) {
            const int q = t / (32 * V), c = t - q * 32 * V;  // c: sample of the chunk
            const int lane_c = c / V, i = c - lane_c * V;
            double sum = 0.0;
            if constexpr (NORMS == 1) {
                sum = scr[(q * V + i) * 32 + lane_c];
            } else {
                for (int w = 0; w < W; ++w) {
                    const double x = nbase[w * kAcc + (q * V + i) * 32 + lane_c];
                    sum = w == 0 ? x : sum + x;
                }
            }
            const int s = chunk * 32 * V + c;
            if (s < A.S) A.norm_part[((size_t)prow * A.S + s) * 4 + q] = sum;
        }
        if constexpr (NORMS == 1) {
            tmem_fence_before_sync();
            __syncthreads();
            tmem_fence_after_sync();
            if (warp == 0) tmem_dealloc(tmem_slot, 32 * (W / 4));
        }
    }
}

// Warps of a block (one block an SM): what the registers allow.  us a step at 16 / 20 / 24
// (28) warps: FP32 pairs, 256 x 512 wall, 64 samples 142 / 136 / 133, 64 x 128 wall 10.7 /
// 10.7 / 12.2; FP32 singles, 128 x 400 wall, 33 samples 93 / - / 81 (74); FP64 singles, 37
// samples 125 / 128 / 129.  With the norms 16: tensor memory holds the sums of 16 warps in
// 128 columns.
template <typename T, int V, int NORMS>
struct PatchBlock {
    static constexpr int kWarps =
        NORMS || sizeof(T) == 8 || V == 4 ? 16 : (V == 2 ? 20 : 28);
};

template <typename T, int V, bool VEL, int NORMS, bool FULL>
static int launch_patch_k(const StepArgs<T>& A, const cvfes_solid_mesh* m, int max_degree,
                          long long max_rows, long long* rows, bool after_step,
                          cudaStream_t st) {
    constexpr int W = PatchBlock<T, V, NORMS>::kWarps;
    const PatchMap M = patch_map(m->n_nodes - A.n_clamped, m->bandwidth, W);
    auto kernel = k_step_patch<T, V, VEL, NORMS, W, FULL>;
    size_t smem = (size_t)W * 2 * max_degree * SlotStage<T, FULL>::kBytes;
    // Slots of up to 29 (FP64) or 30 to 53 (FP32, by the block's warps) elements a node; 160 KB
    // leave room for the sums of NORMS 2.  Tube closed by a cap of nc elements at its apex, nc
    // x 400 nodes, us a step, patch / fan: FP64 nc 28, 64 samples 26.8 / 38.8; FP32 nc 50, 256
    // samples 80.9 / 125.
    if (smem > 160 * 1024) return 1;
    const size_t sums = (size_t)4 * V * 32 * sizeof(double);
    if (NORMS == 1) smem = std::max(smem, sums);
    if (NORMS == 2) smem += W * sums;
    int per_sm = 0;
    const int rc = fanp_blocks_per_sm(reinterpret_cast<const void*>(kernel), 32 * W,
                                      smem, &per_sm);
    if (rc) return rc;
    // whole rounds of the chunks, so that a block keeps its chunk
    const long long places = std::max<long long>((long long)M.n_strips * M.tps,
                                                 (A.n_clamped + W - 1) / W);
    long long per_chunk = std::max(1LL, (long long)per_sm * device_sm_count() / A.nch);
    per_chunk = std::min(per_chunk, std::max(places, 1LL));
    if (NORMS) {
        per_chunk = std::min(per_chunk, max_rows);
        if (rows) *rows = per_chunk;
    }
    return launch_step_kernel(kernel, dim3((unsigned)(per_chunk * A.nch)), 32 * W, smem, after_step, st,
                              "k_step_patch", A, M, max_degree);
}

// Samples per thread: the narrowest width that needs no more chunks than the widest one
// (a warp's time for a node hardly depends on its width: 750 instructions at 4 FP32
// samples a thread, 600 at one).
static int patch_vec(int S, int vmax) {
    int v = vmax;
    while (v > 1 && (S / (v / 2) + 31) / 32 == (S / v + 31) / 32) v /= 2;
    return v;
}

template <typename T>
int launch_step_patch(const cvfes_solid_mesh* m, StepArgs<T> A, int vec_max, bool after_step,
                      cudaStream_t st, int norms_mode, long long max_rows, long long* rows) {
    const int md = (int)m->max_degree;
    if (m->max_degree <= 0 || m->max_degree >= 1024 || A.S >= (1 << 27) ||
        m->n_nodes >= INT32_MAX / 2)
        return 1;
    const int V = patch_vec(A.S, vec_max);
    A.nch = (A.S / V + 31) / 32;
    const int norms = A.norm_part ? (norms_mode == 0 ? 1 : 2) : 0;
#define CVFES_PATCH(VV, VEL, FULL)                                                             \
    switch (norms) {                                                                           \
        case 1: return launch_patch_k<T, VV, VEL, 1, FULL>(A, m, md, max_rows, rows, false, st); \
        case 2: return launch_patch_k<T, VV, VEL, 2, FULL>(A, m, md, max_rows, rows, false, st); \
        default:                                                                               \
            return launch_patch_k<T, VV, VEL, 0, FULL>(A, m, md, 0, nullptr, after_step, st);  \
    }
#define CVFES_PATCH_V(VV, FULL)         \
    if (A.vel) CVFES_PATCH(VV, true, FULL) \
    CVFES_PATCH(VV, false, FULL)
    if constexpr (sizeof(T) == 8) {
        if (mesh_full<T>(m)) {
            if (V == 2) {
                CVFES_PATCH_V(2, true)
            }
            CVFES_PATCH_V(1, true)
        }
    } else if (V == 4) {
        CVFES_PATCH_V(4, false)
    }
    if (V == 2) {
        CVFES_PATCH_V(2, false)
    }
    CVFES_PATCH_V(1, false)
#undef CVFES_PATCH_V
#undef CVFES_PATCH
}

template int launch_step_patch<float>(const cvfes_solid_mesh*, StepArgs<float>, int, bool,
                                      cudaStream_t, int, long long, long long*);
template int launch_step_patch<double>(const cvfes_solid_mesh*, StepArgs<double>, int, bool,
                                       cudaStream_t, int, long long, long long*);

}  // namespace cvfes
