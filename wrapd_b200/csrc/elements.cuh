// Per-element kernels of the ADMM loop (one thread per tet) and the free-vertex
// vector kernels.  Element arrays are SoA: component k of element e is at
// [k * ne + e], so every load and store of a warp is coalesced.  All state is
// stored in FP64; the local step's SVD and prox can run in FP32 (mixed mode),
// everything else (gradient assembly, reductions, the global step) is FP64.
#pragma once
#include "elem_math.cuh"
#include "elem_types.cuh"
#include "prox_net.cuh"

namespace wrapd {

// Candidate-weight modes of update_all_candidate_weights (src/TetElements.cpp:391-432).
enum { CAND_NONE = 0, CAND_REST = 1, CAND_HESSIAN = 2 };

template <typename T>
__device__ __forceinline__ void load9(const double* a, int ne, int e, T* m) {
#pragma unroll
    for (int k = 0; k < 9; ++k) m[k] = T(a[(size_t)k * ne + e]);
}
template <typename T>
__device__ __forceinline__ void store9(double* a, int ne, int e, const T* m) {
#pragma unroll
    for (int k = 0; k < 9; ++k) a[(size_t)k * ne + e] = double(m[k]);
}

// F = (D_free x_free + D_fix x_fix)^T, src/TetElements.cpp:568-586, computed
// in FP64.  `split` sums free then pinned slots as the reference does for
// partially pinned tets; otherwise the four slots in order (Di * x_local).
__device__ __forceinline__ void deformation(const ElemView& E, int e, const double* __restrict__ x,
                                            const double* __restrict__ xfix, bool split, double* F) {
    const int4 id = E.idx[e];
    const int ids[4] = {id.x, id.y, id.z, id.w};
    double xa[4][3];
    bool fixed[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        fixed[a] = ids[a] < 0;
        const double* p = fixed[a] ? xfix + 3 * (size_t)(-ids[a] - 1) : x + 3 * (size_t)ids[a];
        xa[a][0] = p[0]; xa[a][1] = p[1]; xa[a][2] = p[2];
    }
    const bool any_fixed = fixed[0] || fixed[1] || fixed[2] || fixed[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double d[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) d[a] = E.Di[(size_t)(c + 3 * a) * E.ne + e];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            if (split && any_fixed) {
                double vf = 0.0, vx = 0.0;
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    if (fixed[a]) vx += d[a] * xa[a][r];
                    else vf += d[a] * xa[a][r];
                }
                F[r + 3 * c] = vf + vx;
            } else {
                double v = 0.0;
#pragma unroll
                for (int a = 0; a < 4; ++a) v += d[a] * xa[a][r];
                F[r + 3 * c] = v;
            }
        }
    }
}

// A gradient row (kRow doubles, 32-byte aligned) in one 256-bit access.
__device__ __forceinline__ void store_row(double* p, double a, double b, double c) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(0.0) : "memory");
}
__device__ __forceinline__ void load_row(const double* p, double (&v)[3]) {
    double pad;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(pad) : "l"(p));
}

// potential_energy_x per element (src/TetElements.cpp:598-635) from the
// sign-fixed singular values: NH psi(sigma); ARAP |F - R|^2 / 2 with
// R = U V^T, i.e. sum (sigma_i - 1)^2 / 2 (k = 1).
__device__ __forceinline__ double elastic_energy(const Material& m, const double* s) {
    if (m.model == MODEL_ARAP)
        return 0.5 * ((s[0] - 1.0) * (s[0] - 1.0) + (s[1] - 1.0) * (s[1] - 1.0) + (s[2] - 1.0) * (s[2] - 1.0));
    return NH<double>{m.mu, m.lambda}.psi_plain(s[0], s[1], s[2]);
}

// ---- the defo cache + gradient of the global AL objective -------------------
// update_defo_cache (src/TetElements.cpp:564-596) fused with
// global_obj_grad (src/TetElements.cpp:691-738): F, SVD, symF, Q = V^T P V,
// K + K^T, M = F - U diag(s) (K+K^T) V^T and g_e = w^2 Di^T M^T, plus the AL
// value 0.5 w^2 |symF - P|^2, the potential energy and the inversion count at
// x (src/TetElements.cpp:444-468, 598-635).  Outputs out[0..2] = value, pe, flips.
// SEG: a batch (per-mesh sums); a single mesh takes grid_reduce, the same
// arithmetic.  Register budget: all forms are held to 128 (16 warps per SM) by the
// hint, without which they took 164-168 (the form without U and V, 786k elements:
// 245 -> 160 us).  Launched
// on 256-element tiles (two CTAs per SM).
// UV: 0 = SVD as usual; 1 = also keep U and V of the SVD in uv (U then V, 9 SoA
// components each); 2 = x is the point of the meshes' last UV = 1 launch, so F's
// SVD is that launch's: sig, U, V and symF are read back instead of recomputed
// (the same values, so the same results).
// FAST: the SVD's rotations from rsqrt (svd3_fast).  Mixed precision keeps the
// general form's operations: there the FP32 local step turns a last bit of the
// gradient into 1e-8 of the positions within twenty iterations.
template <bool FAST, bool SEG, int UV = 0>
static __global__ void __launch_bounds__(256, 2) k_grad(ElemView E, Tiles T, const int* on, const double* __restrict__ x,
                                              const double* __restrict__ xfix, Material mat0, int write_gel,
                                              double* partials, unsigned* counters, double* out, int stride,
                                              double* __restrict__ uv = nullptr) {
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    const int e = tl.first + threadIdx.x;
    const Material mat = elem_material(E, mat0, e < tl.end ? e : E.ne);
    double red[3] = {0.0, 0.0, 0.0};
    if (e < tl.end) {
        double Fd[9];
        deformation(E, e, x, xfix, true, Fd);
        double F[9], s[3], Us[9], Vs[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) F[i] = double(Fd[i]);
        double S[9];
        if constexpr (UV == 2) {
            load9(uv, E.ne, e, Us);
            load9(uv + (size_t)9 * E.ne, E.ne, e, Vs);
#pragma unroll
            for (int i = 0; i < 3; ++i) s[i] = E.sig[(size_t)i * E.ne + e];
            load9(E.symF, E.ne, e, S);
        } else {
            svd3_of<FAST>(F, s, Us, Vs);
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    M3(S, r, c) = M3(Vs, r, 0) * s[0] * M3(Vs, c, 0) + M3(Vs, r, 1) * s[1] * M3(Vs, c, 1) +
                                  M3(Vs, r, 2) * s[2] * M3(Vs, c, 2);
            store9(E.symF, E.ne, e, S);
#pragma unroll
            for (int i = 0; i < 3; ++i) E.sig[(size_t)i * E.ne + e] = s[i];
            if constexpr (UV == 1) {
                store9(uv, E.ne, e, Us);
                store9(uv + (size_t)9 * E.ne, E.ne, e, Vs);
            }
        }
        double Zm[9], Um[9], P[9];
        load9(E.Z, E.ne, e, Zm);
        load9(E.U, E.ne, e, Um);
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) M3(P, r, c) = M3(Zm, c, r) - M3(Um, c, r);
        const double w2 = E.w2[e];
        {
            double v = 0.0;
#pragma unroll
            for (int i = 0; i < 9; ++i) { const double d = double(S[i]) - double(P[i]); v += d * d; }
            red[0] = (0.5 * w2) * v;
        }
        red[1] = E.vol[e] * elastic_energy(mat, s);
        red[2] = (s[0] < double(0) || s[1] < double(0) || s[2] < double(0)) ? 1.0 : 0.0;
        if (write_gel) {
            double Tm[9], Q[9], K[9], Mm[9];
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    M3(Tm, r, c) = M3(Vs, 0, r) * M3(P, 0, c) + M3(Vs, 1, r) * M3(P, 1, c) + M3(Vs, 2, r) * M3(P, 2, c);
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    M3(Q, r, c) = M3(Tm, r, 0) * M3(Vs, 0, c) + M3(Tm, r, 1) * M3(Vs, 1, c) + M3(Tm, r, 2) * M3(Vs, 2, c);
            M3(K, 0, 0) = M3(Q, 0, 0) / s[0];
            M3(K, 1, 1) = M3(Q, 1, 1) / s[1];
            M3(K, 2, 2) = M3(Q, 2, 2) / s[2];
            M3(K, 0, 1) = M3(K, 1, 0) = (M3(Q, 0, 1) + M3(Q, 1, 0)) / (s[0] + s[1]);
            M3(K, 0, 2) = M3(K, 2, 0) = (M3(Q, 0, 2) + M3(Q, 2, 0)) / (s[0] + s[2]);
            M3(K, 1, 2) = M3(K, 2, 1) = (M3(Q, 1, 2) + M3(Q, 2, 1)) / (s[1] + s[2]);
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    double v = double(0);
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        const double t = M3(K, a, 0) * M3(Vs, c, 0) + M3(K, a, 1) * M3(Vs, c, 1) + M3(K, a, 2) * M3(Vs, c, 2);
                        v += M3(Us, r, a) * s[a] * t;
                    }
                    M3(Mm, r, c) = F[r + 3 * c] - v;
                }
            const double w2t = double(w2);
            const int4 row = E.row[e];
            const int rows[4] = {row.x, row.y, row.z, row.w};
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                double g[3];
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    double v = double(0);
#pragma unroll
                    for (int c = 0; c < 3; ++c) v += double(E.Di[(size_t)(c + 3 * a) * E.ne + e]) * (w2t * M3(Mm, r, c));
                    g[r] = v;
                }
                if (rows[a] >= 0) store_row(E.gel + (size_t)kRow * rows[a], g[0], g[1], g[2]);
            }
        }
    }
    if constexpr (SEG)
        seg_reduce_out<3>(red, T, tl.mesh, partials, counters, out, stride);
    else
        grid_reduce<3>(red, partials, counters, out);
}

// ---- per-mesh vectors of the global step (MeshCtl, VecPools: elem_types.cuh) --
__device__ __forceinline__ int hist_slot(const MeshCtl& c, int i, int M) { return (c.head + i) % (M + 1); }
__device__ __forceinline__ double* g_cur(const VecPools& P, const MeshCtl& c) { return P.G[c.grot % 3]; }
__device__ __forceinline__ double* g_new(const VecPools& P, const MeshCtl& c) { return P.G[(c.grot + 1) % 3]; }
__device__ __forceinline__ double* g_old(const VecPools& P, const MeshCtl& c) { return P.G[(c.grot + 2) % 3]; }

// A mesh's scalars and the status word to pinned host memory, a store each, with no
// order among them: the host polls every word.
constexpr int kHostLow = 20, kHostHigh = 85, kHostSlots = 26;   // slots [0, 20) and from 85 on
__device__ __forceinline__ void publish_mesh(const HostWords& P, int mesh) {
    volatile unsigned long long* w = P.host + (size_t)mesh * (kHostSlots + 1);
    const double* s = P.scal + (size_t)mesh * P.stride;
    for (int k = threadIdx.x; k <= kHostSlots; k += blockDim.x)
        w[k] = k == kHostSlots ? (unsigned long long)*reinterpret_cast<const volatile unsigned*>(P.status)
                               : (unsigned long long)__double_as_longlong(__ldcg(s + (k < kHostLow ? k : k - kHostLow + kHostHigh)));
}

// Gather modes: at the start of an ADMM iteration the gradient goes to the
// mesh's cur buffer and is compared with old (|grad - grad_old|^2, the early
// return of SplitLBFGS.hpp:138-142); inside the L-BFGS loop it goes to new,
// y = new - cur is staged with <s, y>; GATHER_PLAIN writes `plain` only.
enum { GATHER_START = 0, GATHER_LBFGS = 1, GATHER_PLAIN = 2 };

// Free-vertex gather of the element gradients (atomic-free; each vertex's
// incidences, in element order, are added by eight lanes in a fixed order, so
// the sum is deterministic):
//   grad[i] = sum over (e, a) incident to i of g_e(a, :).
// Tiles of 32 free vertices (eight lanes each).  Per mesh: out[0] = |d|^2 with
// d = grad - gold, out[1] = <s_stage, d> (GATHER_LBFGS), out[2] = |x - xs|^2
// (the x error of AlgorithmData, at the point the gradient was taken; x may be
// null).  The last block of a mesh then hands the mesh's scalars to the host (pub):
// this is the last launch before the host decides.
// Bound by the rows' traffic on a large mesh and by the chain of loads on a small
// one.  The rows lie in the order in which they are added here, each a sector of
// its own: eight lanes read 256 contiguous bytes, no index is read on the way and
// every byte that is fetched is used.  (With the rows in element order, component
// by component, each of a vertex's incidences cost three sectors for 24 bytes.)
// A lane has its first three rows in flight at once (a vertex of the bars' meshes
// has 24 incidences at most): five CTAs of 48 registers on an SM; two rows and six
// or eight CTAs, or four and four, are 1 to 15 % slower.  Per launch: 8x8x32
// 8.1 -> 5.4 us, 16x16x64 11.2 -> 7.8, 32x32x128 57 -> 40, a batch of 16 bars
// 18.9 -> 14.6.
constexpr int kGatherAhead = 3;
static __global__ void __launch_bounds__(256, 5) k_gather(Tiles T, const int* on, int mode, const MeshCtl* __restrict__ ctl,
                                                VecPools P, double* __restrict__ plain, const int* __restrict__ inc_ptr,
                                                const double* __restrict__ gel, const double* __restrict__ x,
                                                const double* __restrict__ xs, double* partials, unsigned* counters,
                                                double* out, int stride, HostWords pub) {
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    // eight lanes per vertex: lane s of the group adds incidences s, s + 8, ...
    // of the vertex, then the group adds its lanes in a fixed xor tree
    const int i = tl.first + (threadIdx.x >> 3), sub = threadIdx.x & 7;
    const bool lead = i < tl.end && sub == 0;
    int t = 0, t1 = 0;
    if (i < tl.end) {
        t = inc_ptr[i] + sub;
        t1 = inc_ptr[i + 1];
    }
    double *grad = plain, *ystage = nullptr;
    const double *gold = nullptr, *sstage = nullptr;
    if (mode != GATHER_PLAIN) {
        const MeshCtl c = ctl[tl.mesh];
        if (mode == GATHER_START) {
            grad = g_cur(P, c);
            gold = g_old(P, c);
        } else {
            grad = g_new(P, c);
            gold = g_cur(P, c);
            ystage = P.Y[c.stage];
            sstage = P.S[c.stage];
        }
    }
    // the lane's first rows and what the vertex's sum is compared with, all on
    // their way before the first is used; lane c < 3 of a group has component c
    double r[kGatherAhead][3];
#pragma unroll
    for (int j = 0; j < kGatherAhead; ++j)
        if (t + 8 * j < t1) load_row(gel + (size_t)kRow * (t + 8 * j), r[j]);
    const size_t at = 3 * (size_t)i + sub;
    const bool comp = i < tl.end && sub < 3;
    const double go = comp && gold ? gold[at] : 0.0;
    const double ss = comp && sstage ? sstage[at] : 0.0;
    const double dx = comp && x ? x[at] - xs[at] : 0.0;
    double g0 = 0.0, g1 = 0.0, g2 = 0.0;
#pragma unroll
    for (int j = 0; j < kGatherAhead; ++j)
        if (t + 8 * j < t1) { g0 += r[j][0]; g1 += r[j][1]; g2 += r[j][2]; }
    for (t += 8 * kGatherAhead; t < t1; t += 8) {
        load_row(gel + (size_t)kRow * t, r[0]);
        g0 += r[0][0]; g1 += r[0][1]; g2 += r[0][2];
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        g0 += __shfl_xor_sync(0xffffffffu, g0, o);
        g1 += __shfl_xor_sync(0xffffffffu, g1, o);
        g2 += __shfl_xor_sync(0xffffffffu, g2, o);
    }
    const double g = sub == 0 ? g0 : sub == 1 ? g1 : g2;   // every lane of the group has the sums
    const double d = g - go;
    if (comp) {
        grad[at] = g;
        if (ystage) ystage[at] = d;
    }
    double red[3] = {0.0, 0.0, 0.0};
    if (gold) {
        const double d1 = __shfl_down_sync(0xffffffffu, d, 1), d2 = __shfl_down_sync(0xffffffffu, d, 2);
        if (lead) red[0] = d * d + d1 * d1 + d2 * d2;
        if (sstage) {
            const double s1 = __shfl_down_sync(0xffffffffu, ss, 1), s2 = __shfl_down_sync(0xffffffffu, ss, 2);
            if (lead) red[1] = ss * d + s1 * d1 + s2 * d2;
        }
    }
    if (x) {
        const double e1 = __shfl_down_sync(0xffffffffu, dx, 1), e2 = __shfl_down_sync(0xffffffffu, dx, 2);
        if (lead) red[2] = dx * dx + e1 * e1 + e2 * e2;
    }
    double tot[3];
    if (!seg_reduce<3>(red, T, tl.mesh, partials, counters, tot)) return;
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < 3; ++k) out[(size_t)tl.mesh * stride + k] = tot[k];
    if (!pub.host) return;
    __syncthreads();
    publish_mesh(pub, tl.mesh);
}

// max_wsq_ratio (src/Elements.hpp:56-69) of one element: max(w2/w2c, w2c/w2).  Per mesh
// the gamma rule (System::possibly_update_weights) takes the max over its own elements.
__device__ __forceinline__ double weight_ratio(double w2, double w2c) {
    const double a = w2 / w2c, b = 1.0 / a;
    return fmax(a, b);
}

// ---- local step ---------------------------------------------------------------
// TetElements::polar_update, NH branch (src/TetElements.cpp:284-346), fused
// per element: S_in = (symF + U)^T, SVD, prox from the last stretches, Z and
// U update, and the candidate weight (src/TetElements.cpp:391-432).  C is the
// arithmetic of the SVD and the prox (double, or float in mixed mode); loads,
// stores, the dual update and every sum are FP64.
// out[0..5] = bef_penalty, aft_penalty, curr_pe, negative-stretch count, prox
// iterations and, with `ratio` (the gamma rule; the candidates are then written), the
// largest weight_ratio.  (8x8x32, per iteration a launch of 4.5 us less for it: 8.36 ->
// 8.06 ms per solve; without the rule the sixth value would cost the step 1 to 5 %.)
// prox_mode 0: the reference's L-BFGS prox; 1: Newton (prox_newton); 2 (NET):
// Newton from the better (lower prox objective) of the last stretches and the
// prox network's prediction.  The FP32 instantiation always uses Newton.
// NET needs dynamic shared memory: the network image plus one scratch per warp.
template <typename C, bool NET>
__global__ void __launch_bounds__(512, 1) k_local(ElemView E, Tiles T, const int* on, Material mat0, int prox_iters,
                                               int cand_mode, int ratio, int prox_mode, const unsigned char* __restrict__ net_img,
                                               double* partials, unsigned* counters, double* out, int stride) {
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    double red[6] = {};
    extern __shared__ __align__(16) unsigned char local_smem[];
    if constexpr (NET) {
        net::load_image(net_img, local_smem);
        __syncthreads();
    }
    const int e = tl.first + threadIdx.x;
    const bool valid = e < tl.end;
    const Material mat = elem_material(E, mat0, valid ? e : E.ne);
    double S[9], Um[9];
    double w2 = 0.0, vol = 1.0;
    C sg[3] = {C(1), C(1), C(1)}, Ue[9], Ve[9];
    if (valid) {
        double Zm[9];
        load9(E.symF, E.ne, e, S);
        load9(E.U, E.ne, e, Um);
        load9(E.Z, E.ne, e, Zm);
        w2 = E.w2[e];
        vol = E.vol[e];
        C Sin[9];
        double bef = 0.0;
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                M3(Sin, r, c) = C(M3(S, c, r) + M3(Um, c, r));
                const double d = M3(S, r, c) - (M3(Zm, r, c) - M3(Um, r, c));
                bef += d * d;
            }
        red[0] += 0.5 * w2 * bef;
        if constexpr (sizeof(C) == sizeof(double)) svd3_fast(Sin, sg, Ue, Ve);
        else svd3(Sin, sg, Ue, Ve);
    }
    Prox<C> P;
    P.nh.mu = C(mat.mu);
    P.nh.lambda = C(mat.lambda);
    P.x0[0] = sg[0]; P.x0[1] = sg[1]; P.x0[2] = sg[2];
    P.wov = C(w2 / vol);
    C xs[3] = {C(1), C(1), C(1)};
    if (valid) {
#pragma unroll
        for (int i = 0; i < 3; ++i) xs[i] = C(E.slast[(size_t)i * E.ne + e]);
    }
    if constexpr (NET) {
        // warp-collective: every lane runs the network, lanes past the end on dummies
        const float sf[3] = {float(sg[0]), float(sg[1]), float(sg[2])};
        float f[net::IN], y[net::OUT], pr[3];
        net::features(sf, valid ? float(w2 / vol) : float(mat.mu), float(mat.mu), float(mat.lambda), f);
        net::warp_forward(local_smem, local_smem + net::IMAGE_BYTES + (threadIdx.x >> 5) * net::WARP_SCRATCH, f,
                          valid, y);
        net::predict_start(local_smem, sf, y, pr);
        if (valid) {
            const C cand[3] = {C(pr[0]), C(pr[1]), C(pr[2])};
            if (isfinite(cand[0]) && isfinite(cand[1]) && isfinite(cand[2]) && P.value(cand) < P.value(xs)) {
                xs[0] = cand[0]; xs[1] = cand[1]; xs[2] = cand[2];
            }
        }
    }
    if (valid) {
        int iters;
        LsPoint<C> end;   // the log term at the solution, where the prox leaves it
        end.ok = false;
        if constexpr (sizeof(C) == sizeof(double)) {
            if (NET || prox_mode == 1) {
                iters = prox_newton(P, xs, prox_iters, C(1e-12));
            } else {
                extern __shared__ double prox_hist[];   // 48 x blockDim doubles
                iters = prox_lbfgs(P, xs, prox_iters, ProxHistory<double>{prox_hist + threadIdx.x, (int)blockDim.x}, &end);
                if (iters < 0) iters = prox_iters;
            }
        } else {
            iters = prox_newton(P, xs, prox_iters, C(8) * Lim<C>::eps());
        }
        if (sizeof(C) < sizeof(double) &&
            !(isfinite(xs[0]) && isfinite(xs[1]) && isfinite(xs[2]) && xs[0] >= C(0) && xs[1] >= C(0) && xs[2] >= C(0))) {
            // FP32 range guard: near a vanishing stretch 1/x overflows in single
            // precision; redo this element's prox in FP64 from the same inputs.
            Prox<double> Pd;
            Pd.nh.mu = mat.mu;
            Pd.nh.lambda = mat.lambda;
            Pd.x0[0] = double(sg[0]); Pd.x0[1] = double(sg[1]); Pd.x0[2] = double(sg[2]);
            Pd.wov = w2 / vol;
            double xd[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) xd[i] = E.slast[(size_t)i * E.ne + e];
            iters += prox_newton(Pd, xd, prox_iters, 1e-12);
#pragma unroll
            for (int i = 0; i < 3; ++i) xs[i] = C(xd[i]);
        }
        red[4] += double(iters);
        double xo[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) { xo[i] = double(xs[i]); E.slast[(size_t)i * E.ne + e] = xo[i]; }
        red[3] += (xo[0] < 0.0 || xo[1] < 0.0 || xo[2] < 0.0) ? 1.0 : 0.0;
        C Soc[9];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                M3(Soc, r, c) = M3(Ve, r, 0) * xs[0] * M3(Ue, c, 0) + M3(Ve, r, 1) * xs[1] * M3(Ue, c, 1) +
                                M3(Ve, r, 2) * xs[2] * M3(Ue, c, 2);
        if (end.ok)
            red[2] += vol * NH<double>{mat.mu, mat.lambda}.psi_log(xo[0], xo[1], xo[2], double(end.lf));
        else
            red[2] += vol * NH<double>{mat.mu, mat.lambda}.psi_plain(xo[0], xo[1], xo[2]);
        double aft = 0.0, Zm[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            const double So = double(Soc[i]);
            const double d = S[i] - (So - Um[i]);
            aft += d * d;
            Zm[i] = So;
            Um[i] = Um[i] + (S[i] - So);
        }
        red[1] += 0.5 * w2 * aft;
        store9(E.Z, E.ne, e, Zm);
        store9(E.U, E.ne, e, Um);
        double cand = 0.0;
        if (cand_mode == CAND_REST) {
            cand = vol * mat.wr;
        } else if (cand_mode == CAND_HESSIAN) {
            const double lm = NH<double>{mat.mu, mat.lambda}.template hess_lmax<sizeof(C) == sizeof(double)>(xo);
            double c = lm;
            if (lm < mat.wmin) c = mat.wmin;
            if (lm > mat.wmax) c = mat.wmax;
            cand = vol * c;
        }
        if (cand_mode != CAND_NONE) E.w2c[e] = cand;
        if (ratio) red[5] = weight_ratio(w2, cand);
    }
    if (ratio) {
        seg_reduce_out<6, 5>(red, T, tl.mesh, partials, counters, out, stride);
    } else {
        const double sums[5] = {red[0], red[1], red[2], red[3], red[4]};
        seg_reduce_out<5>(sums, T, tl.mesh, partials, counters, out, stride);
    }
}

// initialize_dual_vars (src/TetElements.cpp:145-166): Z = (V diag(s) V^T)^T of
// F(X) with all four slots read from X, U = 0; then polar_potential_energy
// (src/TetElements.cpp:638-675) of the new Z.  out[0] = that energy.
template <bool FAST>
static __global__ void __launch_bounds__(128) k_init_dual(ElemView E, Tiles T, const int* on, const double* __restrict__ x,
                                                   const double* __restrict__ xfix, Material mat0,
                                                   double* partials, unsigned* counters, double* out, int stride) {
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    const int e = tl.first + threadIdx.x;
    const Material mat = elem_material(E, mat0, e < tl.end ? e : E.ne);
    double red[1] = {0.0};
    if (e < tl.end) {
        double Fd[9];
        deformation(E, e, x, xfix, false, Fd);
        double F[9], s[3], Us[9], Vs[9], Zm[9], Zt[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) F[i] = double(Fd[i]);
        svd3_of<FAST>(F, s, Us, Vs);
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                M3(Zm, r, c) = M3(Vs, c, 0) * s[0] * M3(Vs, r, 0) + M3(Vs, c, 1) * s[1] * M3(Vs, r, 1) +
                               M3(Vs, c, 2) * s[2] * M3(Vs, r, 2);
        store9(E.Z, E.ne, e, Zm);
        double zero[9] = {};
        store9(E.U, E.ne, e, zero);
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) M3(Zt, r, c) = M3(Zm, c, r);
        if (mat.model == MODEL_ARAP) {
            // ARAP polar_potential_energy (src/TetElements.cpp:640-646): |Z - I|^2 / 2
            double n2 = 0.0;
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c) { const double d = M3(Zm, r, c) - (r == c ? 1.0 : 0.0); n2 += d * d; }
            red[0] = 0.5 * E.vol[e] * n2;
        } else {
            svd3_of<FAST>(Zt, s, Us, Vs);
            red[0] = E.vol[e] * NH<double>{mat.mu, mat.lambda}.psi_plain(double(s[0]), double(s[1]), double(s[2]));
        }
    }
    seg_reduce_out<1>(red, T, tl.mesh, partials, counters, out, stride);
}

// Candidate weights of midupdate_weights (src/TetElements.cpp:360-388): from
// F(X) (from_x = 1) or from the cached singular values.
template <bool FAST>
static __global__ void __launch_bounds__(128) k_mid_candidates(ElemView E, Tiles T, const int* on,
                                                        const double* __restrict__ x, const double* __restrict__ xfix,
                                                        Material mat0, int from_x, int cand_mode) {
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    const int e = tl.first + threadIdx.x;
    if (e >= tl.end) return;
    const Material mat = elem_material(E, mat0, e);
    double s[3];
    if (from_x) {
        double Fd[9];
        deformation(E, e, x, xfix, false, Fd);
        double F[9], st[3], Us[9], Vs[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) F[i] = double(Fd[i]);
        svd3_of<FAST>(F, st, Us, Vs);
        s[0] = st[0]; s[1] = st[1]; s[2] = st[2];
    } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) s[i] = double(E.sig[(size_t)i * E.ne + e]);
    }
    const double vol = E.vol[e];
    if (cand_mode == CAND_HESSIAN) {
        const double lm = NH<double>{mat.mu, mat.lambda}.template hess_lmax<FAST>(s);
        double c = lm;
        if (lm < mat.wmin) c = mat.wmin;
        if (lm > mat.wmax) c = mat.wmax;
        E.w2c[e] = vol * c;
    } else {
        E.w2c[e] = vol * mat.wr;
    }
}

// update_actual_weights (src/TetElements.cpp:435-442), on the meshes that reweight.
static __global__ void __launch_bounds__(256) k_apply_weights(ElemView E, Tiles T, const int* on) {
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    const int e = tl.first + threadIdx.x;
    if (e >= tl.end) return;
    const double r = E.w2[e] / E.w2c[e];
#pragma unroll
    for (int k = 0; k < 9; ++k) E.U[(size_t)k * E.ne + e] = r * E.U[(size_t)k * E.ne + e];
    E.w2[e] = E.w2c[e];
}

// ---- global-step vector kernels (n x 3 FP64, dissection order) ----------------
// Tiles of kVecTile doubles of one mesh's range (thread t takes entries t,
// t + 256, ...).  The two-loop recursion of SplitLBFGS::minimize
// (SplitLBFGS.hpp:152-177) runs as a chain of steps, each an axpy and an inner
// product per mesh; every mesh walks its own history length `it`:
//   first loop, step j = it-1 .. 0: q = g (j = it-1) or q -= alpha_{j+1} y_{j+1};
//     alpha_j = rho_j <s_j, q>;  step -1: q -= alpha_0 y_0 (q = g when it = 0);
//   second loop, step j = 0 .. it-1: q += c_{j-1} s_{j-1} (j > 0);
//     c_j = alpha_j - rho_j <y_j, q>;  step it: q += c_{it-1} s_{it-1};
//     dir = <g, q>.
// A launch serves one step index j for every mesh; meshes whose walk has no
// step j return.  alpha_j, c_j and dir are per mesh in the scalar block
// (scal + mesh * stride + S_ALPHA / S_C / S_DIR).
constexpr int kVecTile = 2048;


static __global__ void __launch_bounds__(256) k_lbfgs_first(Tiles T, const int* on, const MeshCtl* __restrict__ ctl,
                                                     VecPools P, const double* __restrict__ rho,
                                                     double* __restrict__ q, int j, TwoLoopSlots sl, double* partials,
                                                     unsigned* counters, double* scal, int stride) {
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    const MeshCtl c = ctl[tl.mesh];
    if (j >= c.it) return;
    double* sc = scal + (size_t)tl.mesh * stride;
    const bool first = j == c.it - 1;                  // q = g (also j = -1 with it = 0)
    const double* g = g_cur(P, c);
    const double* yv = first ? nullptr : P.Y[hist_slot(c, j + 1, P.M)];
    const double cf = first ? 0.0 : -__ldcg(sc + sl.alpha + j + 1);
    const double* sv = j >= 0 ? P.S[hist_slot(c, j, P.M)] : nullptr;
    double red[1] = {0.0};
    for (int i = tl.first + (int)threadIdx.x; i < tl.end; i += blockDim.x) {
        double qi = first ? g[i] : q[i];
        if (yv) qi = qi + cf * yv[i];
        q[i] = qi;
        if (sv) red[0] += sv[i] * qi;
    }
    if (j < 0) return;
    double tot[1];
    if (seg_reduce<1>(red, T, tl.mesh, partials, counters, tot) && threadIdx.x == 0)
        sc[sl.alpha + j] = rho[(size_t)tl.mesh * kHistSlots + hist_slot(c, j, P.M)] * tot[0];
}

static __global__ void __launch_bounds__(256) k_lbfgs_second(Tiles T, const int* on, const MeshCtl* __restrict__ ctl,
                                                      VecPools P, const double* __restrict__ rho,
                                                      double* __restrict__ q, int j, TwoLoopSlots sl, double* partials,
                                                      unsigned* counters, double* scal, int stride) {
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    const MeshCtl c = ctl[tl.mesh];
    if (j > c.it) return;
    double* sc = scal + (size_t)tl.mesh * stride;
    const double* sv = j > 0 ? P.S[hist_slot(c, j - 1, P.M)] : nullptr;
    const double cf = j > 0 ? __ldcg(sc + sl.c + j - 1) : 0.0;
    const double* w = j < c.it ? P.Y[hist_slot(c, j, P.M)] : g_cur(P, c);
    double red[1] = {0.0};
    for (int i = tl.first + (int)threadIdx.x; i < tl.end; i += blockDim.x) {
        double qi = q[i];
        if (sv) {
            qi = qi + cf * sv[i];
            q[i] = qi;
        }
        red[0] += w[i] * qi;
    }
    double tot[1];
    if (seg_reduce<1>(red, T, tl.mesh, partials, counters, tot) && threadIdx.x == 0) {
        if (j < c.it)
            sc[sl.c + j] = __ldcg(sc + sl.alpha + j) + (-rho[(size_t)tl.mesh * kHistSlots + hist_slot(c, j, P.M)]) * tot[0];
        else
            sc[sl.dir] = tot[0];
    }
}

// ---- the two-loop recursion in one launch per loop -------------------------------
// The M + 1 steps of each loop above, with the vectors' entries in registers or
// walked in place, and the step's inner product exchanged inside the launch.  The
// per-entry operations and the order of every sum are those of the per-step
// launches: the same alpha_i, c_i and decrement, bit for bit, in every CTA.  The
// second loop can end with the step x <- x - q of k_xupdate (`x` given), whose
// restart rule needs the decrement that every CTA then holds: q never goes to memory.
// Us per inner iteration at history 5, first + second loop (+ x step before): a
// barrier of atomics per step or one CTA per small mesh before, now:
//   8x8x32      10.7 + 11.7 + 3.5     7.1 +  9.6
//   16x16x64    13.2 + 15.7 + 4.8    10.0 + 12.7
//   24x24x48    13.7 + 17.1 + 6.1    11.1 + 17.6
//   32x32x128   16.2 + 19.8 + 6.3    14.6 + 20.5
//   16 bars     18 + 18 + 11 per-step launches of 10.5 + 5.5 -> 10 + 14 + 12 + 16
struct TwoLoopArgs {
    const MeshCtl* ctl;
    VecPools P;
    const double* rho;    // per mesh, kHistSlots each
    double* q;
    TwoLoopSlots sl;
    double* scal;
    int stride;
    double* x;            // second loop: x to step, or null (q is stored instead)
};

// x and s = x_new - x_old at entry i (k_xupdate with rate 1).
__device__ __forceinline__ void x_step(const TwoLoopArgs& a, double* s, int i, double step) {
    const double xo = a.x[i];
    const double xn = xo - step;
    s[i] = xn - xo;
    a.x[i] = xn;
}

// Meshes above kTwoLoopMaxN unknowns: a cooperative launch (all CTAs resident).
// Step j's tile sums go to slots[j * count + tile].  In a mesh of at most
// kDirectTiles tiles every CTA polls them (see kUnset) and adds them in
// seg_reduce's order; with more, that many readers of the same few lines slow the
// writers down, so the mesh's first CTA alone does, and hands the total on in
// eight copies.  Each launch unsets the other loop's slots and totals, whose
// launch has ended.  REG: a CTA per tile of any
// mesh, kTwoLoopPT entries of q per thread in registers and the two history vectors
// of the next step loaded before the exchange.  Otherwise one mesh, CTA b taking tiles
// b, b + G, ... with q in memory.
constexpr int kTwoLoopGridThreads = 256;
// Us per inner iteration, first + second loop, polled by all and through the first
// CTA: 9 tiles 10.5 + 12.6, 12.4 + 16.4; 41 to 75 tiles the same within 0.5; 106 tiles 16.8 + 23.2,
// 13.5 + 21.0; 203 tiles 31.9 + 36.0, 16.3 + 23.2.
constexpr int kDirectTiles = 64;
constexpr int kTwoLoopPT = kVecTile / kTwoLoopGridThreads;
static_assert(kVecTile % kTwoLoopGridThreads == 0, "whole entries per thread");

// q <- qs + cf v over a tile (v null: as it is; qd null: not stored), and the threads'
// parts of <w, q> (w null: 0) to `sum`.  Four entries' reads go out together.
template <typename F>
__device__ __forceinline__ void walk_tile(const Tile& tl, const double* qs, double* qd, const double* v, double cf,
                                          const double* w, F&& sum) {
    double red = 0.0;
    constexpr int U = 4;
    for (int i = tl.first + (int)threadIdx.x; i < tl.end; i += U * kTwoLoopGridThreads) {
        double qi[U], vi[U], wi[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = i + u * kTwoLoopGridThreads;
            qi[u] = k < tl.end ? qs[k] : 0.0;
            vi[u] = (v && k < tl.end) ? v[k] : 0.0;
            wi[u] = (w && k < tl.end) ? w[k] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = i + u * kTwoLoopGridThreads;
            if (k >= tl.end) break;
            if (v) qi[u] = qi[u] + cf * vi[u];
            if (qd) qd[k] = qi[u];
            if (w) red += wi[u] * qi[u];
        }
    }
    sum(red);
}

constexpr int kTotalCopies = 8, kTotalPitch = 16;      // copies of a total, a 128-byte line each
constexpr int kTotalSlots = kHistSlots * kTotalCopies * kTotalPitch;   // doubles per mesh
struct GridExchange {
    double* slots;
    double* totals;       // the mesh's
    int count, t0, t1;
    int* status;
    bool lead;            // the mesh's first CTA
    int hold;             // a tile whose sums are not handed on (-1: none): the test of the bounded waits
    // A tile's sum of the threads' v (block_reduce's order), to slot j.  `again`: the
    // second or a later tile of the step.
    __device__ __forceinline__ void put(int j, int tile, double v, bool again = false) {
        __shared__ double sm[kTwoLoopGridThreads / 32];
        if (again) __syncthreads();   // thread 0 has read the tile's before
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            double r = 0.0;
            for (int w = 0; w < kTwoLoopGridThreads / 32; ++w) r += sm[w];
            if (tile != hold) st_relaxed(slots + (size_t)j * count + tile, r);
        }
    }
    // The total of slot j over the mesh's tiles, in every thread; false when a wait gave up.
    __device__ __forceinline__ bool get(int j, double& total) {
        __shared__ double sm[kTwoLoopGridThreads / 32];
        double acc = 0.0;
        bool ok = true;
        unsigned long long since = 0;
        const bool direct = t1 - t0 <= kDirectTiles;
        if (!direct && !lead) {
            if (threadIdx.x == 0) {
                const double* p = totals + (j * kTotalCopies + blockIdx.x % kTotalCopies) * kTotalPitch;
                double v = ld_relaxed(p);
                for (int i = 0; unset(v) && ok; ++i) {
                    ok = look_again(i, since, status);
                    v = ld_relaxed(p);
                }
                sm[0] = v;
            }
            ok = __syncthreads_and(ok);
            total = sm[0];
            return ok;
        }
        for (int b = t0 + (int)threadIdx.x; b < t1; b += kTwoLoopGridThreads) {
            double v = ld_relaxed(slots + (size_t)j * count + b);
            for (int i = 0; unset(v) && ok; ++i) {
                ok = look_again(i, since, status);
                v = ld_relaxed(slots + (size_t)j * count + b);
            }
            acc += v;
        }
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = acc;
        ok = __syncthreads_and(ok);
        double r = 0.0;
        for (int w = 0; w < kTwoLoopGridThreads / 32; ++w) r += sm[w];
        total = r;
        if (!direct && ok && threadIdx.x < kTotalCopies)
            st_relaxed(totals + (j * kTotalCopies + threadIdx.x) * kTotalPitch, r);
        return ok;
    }
};

template <bool SECOND, bool REG>
static __global__ void __launch_bounds__(kTwoLoopGridThreads, REG ? 3 : 4) k_two_loop_grid(Tiles T, const int* on, TwoLoopArgs A,
                                                       double* slots, double* other, int nslots, int* status,
                                                       int hold) {
    const int count = T.count, G = gridDim.x;
    for (int s = threadIdx.x; s < nslots * ((count + G - 1) / G); s += kTwoLoopGridThreads) {
        const int t = blockIdx.x + (s / nslots) * G;
        if (t < count) st_relaxed(other + (size_t)(s % nslots) * count + t, unset_value());
    }
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    const MeshCtl c = A.ctl[tl.mesh];
    const VecPools& P = A.P;
    const double* rho = A.rho + (size_t)tl.mesh * kHistSlots;
    double* scal = A.scal + (size_t)tl.mesh * A.stride;
    const int t0 = T.t ? T.tile0[tl.mesh] : 0;
    const bool first_cta = (int)blockIdx.x == t0;
    const size_t totals = (size_t)kHistSlots * count + (size_t)tl.mesh * kTotalSlots;
    GridExchange X{slots, slots + totals, count, t0, T.t ? T.tile0[tl.mesh + 1] : count, status, first_cta, hold};
    if (first_cta)
        for (int s = threadIdx.x; s < nslots * kTotalCopies; s += kTwoLoopGridThreads)
            st_relaxed(other + totals + s * kTotalPitch, unset_value());
    if constexpr (REG) {
        const int i0 = tl.first + (int)threadIdx.x;
        double qv[kTwoLoopPT], av[kTwoLoopPT], bv[kTwoLoopPT];
        auto load = [&](double (&v)[kTwoLoopPT], const double* src) {
#pragma unroll
            for (int k = 0; k < kTwoLoopPT; ++k) {
                const int i = i0 + k * kTwoLoopGridThreads;
                v[k] = (src && i < tl.end) ? src[i] : 0.0;
            }
        };
        auto store_q = [&]() {
#pragma unroll
            for (int k = 0; k < kTwoLoopPT; ++k) {
                const int i = i0 + k * kTwoLoopGridThreads;
                if (i < tl.end) A.q[i] = qv[k];
            }
        };
        if constexpr (!SECOND) {
            // av: y_{j+1} (the update), bv: s_j (the inner product) of step j
            double alpha_next = 0.0;
            load(qv, g_cur(P, c));
            load(bv, c.it - 1 >= 0 ? P.S[hist_slot(c, c.it - 1, P.M)] : nullptr);
            for (int j = c.it - 1; j >= -1; --j) {
                const bool first = j == c.it - 1;
                const double cf = first ? 0.0 : -alpha_next;
                double red = 0.0;
#pragma unroll
                for (int k = 0; k < kTwoLoopPT; ++k) {
                    if (i0 + k * kTwoLoopGridThreads < tl.end) {
                        double qi = qv[k];
                        if (!first) qi = qi + cf * av[k];
                        qv[k] = qi;
                        if (j >= 0) red += bv[k] * qi;
                    }
                }
                if (j < 0) break;
                X.put(j, blockIdx.x, red);
                load(av, P.Y[hist_slot(c, j, P.M)]);
                load(bv, j - 1 >= 0 ? P.S[hist_slot(c, j - 1, P.M)] : nullptr);
                double tot;
                if (!X.get(j, tot)) return;
                alpha_next = rho[hist_slot(c, j, P.M)] * tot;
                if (first_cta && threadIdx.x == 0) scal[A.sl.alpha + j] = alpha_next;
            }
            store_q();
        } else {
            // av: s_{j-1} (the update), bv: y_j or g (the inner product) of step j
            double c_prev = 0.0, dir = 0.0;
            load(qv, A.q);
            load(bv, 0 < c.it ? P.Y[hist_slot(c, 0, P.M)] : g_cur(P, c));
            for (int j = 0; j <= c.it; ++j) {
                const double cf = j > 0 ? c_prev : 0.0;
                double red = 0.0;
#pragma unroll
                for (int k = 0; k < kTwoLoopPT; ++k) {
                    if (i0 + k * kTwoLoopGridThreads < tl.end) {
                        double qi = qv[k];
                        if (j > 0) {
                            qi = qi + cf * av[k];
                            qv[k] = qi;
                        }
                        red += bv[k] * qi;
                    }
                }
                X.put(j, blockIdx.x, red);
                if (j < c.it) {
                    load(av, P.S[hist_slot(c, j, P.M)]);
                    load(bv, j + 1 < c.it ? P.Y[hist_slot(c, j + 1, P.M)] : g_cur(P, c));
                }
                double tot;
                if (!X.get(j, tot)) return;
                if (j < c.it) {
                    c_prev = __ldcg(scal + A.sl.alpha + j) + (-rho[hist_slot(c, j, P.M)]) * tot;
                    if (first_cta && threadIdx.x == 0) scal[A.sl.c + j] = c_prev;
                } else {
                    dir = tot;
                    if (first_cta && threadIdx.x == 0) scal[A.sl.dir] = tot;
                }
            }
            if (!A.x) { store_q(); return; }
            const bool restart = !(dir > 0.0);   // bv holds g
#pragma unroll
            for (int k = 0; k < kTwoLoopPT; ++k) {
                const int i = i0 + k * kTwoLoopGridThreads;
                if (i < tl.end) x_step(A, P.S[c.stage], i, restart ? bv[k] : qv[k]);
            }
        }
    } else if constexpr (!SECOND) {
        // j = it - 1 .. -1: q = (first ? g : q) - alpha_{j+1} y_{j+1}; alpha_j = rho_j <s_j, q>
        double alpha_next = 0.0;
        for (int j = c.it - 1; j >= -1; --j) {
            const bool first = j == c.it - 1;
            const double* qs = first ? g_cur(P, c) : A.q;
            const double* yv = first ? nullptr : P.Y[hist_slot(c, j + 1, P.M)];
            const double cf = first ? 0.0 : -alpha_next;
            const double* sv = j >= 0 ? P.S[hist_slot(c, j, P.M)] : nullptr;
            for (int t = blockIdx.x; t < count; t += G)
                walk_tile(tile_at(T, t), qs, A.q, yv, cf, sv, [&](double red) { if (j >= 0) X.put(j, t, red, t != (int)blockIdx.x); });
            if (j < 0) break;
            double tot;
            if (!X.get(j, tot)) return;
            alpha_next = rho[hist_slot(c, j, P.M)] * tot;
            if (first_cta && threadIdx.x == 0) scal[A.sl.alpha + j] = alpha_next;
        }
    } else {
        // j = 0 .. it: q += c_{j-1} s_{j-1}; c_j = alpha_j - rho_j <y_j, q>, dir = <g, q>
        double c_prev = 0.0, dir = 0.0;
        for (int j = 0; j <= c.it; ++j) {
            const double* sv = j > 0 ? P.S[hist_slot(c, j - 1, P.M)] : nullptr;
            const double* w = j < c.it ? P.Y[hist_slot(c, j, P.M)] : g_cur(P, c);
            for (int t = blockIdx.x; t < count; t += G)
                walk_tile(tile_at(T, t), A.q, j > 0 ? A.q : nullptr, sv, c_prev, w, [&](double red) { X.put(j, t, red, t != (int)blockIdx.x); });
            double tot;
            if (!X.get(j, tot)) return;
            if (j < c.it) {
                c_prev = __ldcg(scal + A.sl.alpha + j) + (-rho[hist_slot(c, j, P.M)]) * tot;
                if (first_cta && threadIdx.x == 0) scal[A.sl.c + j] = c_prev;
            } else {
                dir = tot;
                if (first_cta && threadIdx.x == 0) scal[A.sl.dir] = tot;
            }
        }
        if (!A.x) return;
        const double* step = !(dir > 0.0) ? g_cur(P, c) : A.q;
        for (int t = blockIdx.x; t < count; t += G) {
            const Tile w = tile_at(T, t);
            for (int i = w.first + (int)threadIdx.x; i < w.end; i += kTwoLoopGridThreads) x_step(A, P.S[c.stage], i, step[i]);
        }
    }
}

// Meshes of at most kTwoLoopMaxN unknowns: a cluster of eight CTAs per mesh, which
// stand for one CTA of 1024 threads (thread v of it is thread v % 128 of CTA v / 128)
// with PT entries of q each in registers.  A step's warp sums go to
// every CTA's shared memory, and after one cluster barrier every thread adds the
// 32 of them in order, as block_reduce does for 1024 threads.  The history vectors of
// the next step are loaded before the exchange.  (One CTA of 1024 threads, the form
// before, reads all vectors through one SM and exchanges behind two barriers.)
constexpr int kTwoLoopCluster = 8;
constexpr int kTwoLoopThreads = 128;       // per CTA
constexpr int kTwoLoopMaxN = kTwoLoopCluster * kTwoLoopThreads * 16;   // PT 16, 8 or 4: see SolverGPU::initialize

__device__ __forceinline__ double cluster_total(double v, double (*sm)[32], int buf, unsigned rank) {
    const int lane = threadIdx.x & 31, vw = rank * (kTwoLoopThreads / 32) + (threadIdx.x >> 5);
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    v = __shfl_sync(0xffffffffu, v, 0);
    if (lane < kTwoLoopCluster) {
        const unsigned local = static_cast<unsigned>(__cvta_generic_to_shared(&sm[buf][vw]));
        unsigned remote;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(lane));
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote), "d"(v) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    double r = 0.0;
#pragma unroll
    for (int w = 0; w < 32; ++w) r += sm[buf][w];
    return r;
}

// Cluster i serves mesh ids[i] (ids null: mesh i).
template <bool SECOND, int PT>
static __global__ void __cluster_dims__(kTwoLoopCluster, 1, 1) __launch_bounds__(kTwoLoopThreads)
    k_two_loop_cluster(const int* __restrict__ ids, const int* on, TwoLoopArgs A) {
    __shared__ double sm[2][32];   // by step parity: a step's barrier ends the reads of the step before the last
    const int m = ids ? ids[blockIdx.x / kTwoLoopCluster] : blockIdx.x / kTwoLoopCluster;
    const unsigned rank = blockIdx.x % kTwoLoopCluster;
    const MeshCtl c = A.ctl[m];
    if (!mesh_on(on, m)) return;   // the whole cluster
    const VecPools& P = A.P;
    const double* rho = A.rho + (size_t)m * kHistSlots;
    double* scal = A.scal + (size_t)m * A.stride;
    constexpr int STEP = kTwoLoopCluster * kTwoLoopThreads;
    const int i0 = c.v0 + (int)(rank * kTwoLoopThreads + threadIdx.x), end = c.v1;
    const bool lead = rank == 0 && threadIdx.x == 0;
    double qv[PT], av[PT], bv[PT];
    auto load = [&](double (&v)[PT], const double* src) {
#pragma unroll
        for (int k = 0; k < PT; ++k) v[k] = i0 + k * STEP < end ? src[i0 + k * STEP] : 0.0;
    };
    // every CTA of the cluster is running before any writes to another's shared memory
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if constexpr (!SECOND) {
        // q = g; for j = it-1 .. 0: alpha_j = rho_j <s_j, q>, q -= alpha_j y_j (SplitLBFGS.hpp:152-158)
        load(qv, g_cur(P, c));
        if (c.it > 0) load(bv, P.S[hist_slot(c, c.it - 1, P.M)]);
        for (int j = c.it - 1; j >= 0; --j) {
            double d = 0.0;
#pragma unroll
            for (int k = 0; k < PT; ++k)
                if (i0 + k * STEP < end) d += bv[k] * qv[k];
            load(av, P.Y[hist_slot(c, j, P.M)]);
            if (j > 0) load(bv, P.S[hist_slot(c, j - 1, P.M)]);
            const double a = rho[hist_slot(c, j, P.M)] * cluster_total(d, sm, j & 1, rank);
            if (lead) scal[A.sl.alpha + j] = a;
#pragma unroll
            for (int k = 0; k < PT; ++k)
                if (i0 + k * STEP < end) qv[k] = qv[k] + (-a) * av[k];
        }
#pragma unroll
        for (int k = 0; k < PT; ++k)
            if (i0 + k * STEP < end) A.q[i0 + k * STEP] = qv[k];
    } else {
        // for j = 0 .. it-1: c_j = alpha_j - rho_j <y_j, q>, q += c_j s_j; then dir = <g, q> (SplitLBFGS.hpp:170-173)
        load(qv, A.q);
        load(bv, 0 < c.it ? P.Y[hist_slot(c, 0, P.M)] : g_cur(P, c));
        for (int j = 0; j < c.it; ++j) {
            double d = 0.0;
#pragma unroll
            for (int k = 0; k < PT; ++k)
                if (i0 + k * STEP < end) d += bv[k] * qv[k];
            load(av, P.S[hist_slot(c, j, P.M)]);
            load(bv, j + 1 < c.it ? P.Y[hist_slot(c, j + 1, P.M)] : g_cur(P, c));
            const double cc = scal[A.sl.alpha + j] + (-rho[hist_slot(c, j, P.M)]) * cluster_total(d, sm, j & 1, rank);
            if (lead) scal[A.sl.c + j] = cc;
#pragma unroll
            for (int k = 0; k < PT; ++k)
                if (i0 + k * STEP < end) qv[k] = qv[k] + cc * av[k];
        }
        double d = 0.0;
#pragma unroll
        for (int k = 0; k < PT; ++k)
            if (i0 + k * STEP < end) {
                if (!A.x) A.q[i0 + k * STEP] = qv[k];
                d += bv[k] * qv[k];
            }
        const double dir = cluster_total(d, sm, c.it & 1, rank);
        if (lead) scal[A.sl.dir] = dir;
        if (!A.x) return;
        const bool restart = !(dir > 0.0);   // bv holds g
#pragma unroll
        for (int k = 0; k < PT; ++k)
            if (i0 + k * STEP < end) x_step(A, P.S[c.stage], i0 + k * STEP, restart ? bv[k] : qv[k]);
    }
}

// x <- x - rate * step with step = q, or grad when the mesh's decrement
// dir <= 0 (the steepest-descent restart of SplitLBFGS.hpp:189-194);
// s = x_new - x_old into the mesh's stage slot.  rate is 1 unless the global
// line search chose another (SplitLBFGS.hpp:196-206).
static __global__ void __launch_bounds__(256) k_xupdate(Tiles T, const int* on, const MeshCtl* __restrict__ ctl,
                                                 VecPools P, double* __restrict__ x, const double* __restrict__ q,
                                                 const double* scal, int dir_slot, int stride, double rate) {
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    const MeshCtl c = ctl[tl.mesh];
    const bool restart = !(__ldcg(scal + (size_t)tl.mesh * stride + dir_slot) > 0.0);
    const double* grad = g_cur(P, c);
    double* s = P.S[c.stage];
    for (int i = tl.first + (int)threadIdx.x; i < tl.end; i += blockDim.x) {
        const double xo = x[i];
        const double xn = fma(-rate, restart ? grad[i] : q[i], xo);
        s[i] = xn - xo;
        x[i] = xn;
    }
}

// grad_old = 0 (SplitLBFGS keeps grad_old across ADMM iterations and zeroes
// it with the history, SplitLBFGS.hpp:118-121) on the meshes that are on.
static __global__ void __launch_bounds__(256) k_zero_old(Tiles T, const int* on, const MeshCtl* __restrict__ ctl,
                                                  VecPools P) {
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    double* g = g_old(P, ctl[tl.mesh]);
    for (int i = tl.first + (int)threadIdx.x; i < tl.end; i += blockDim.x) g[i] = 0.0;
}

// Per mesh |x - xs|^2 (the x error of AlgorithmData::update_per_iter_data).
static __global__ void __launch_bounds__(256) k_xerr(Tiles T, const int* on, const double* __restrict__ x,
                                              const double* __restrict__ xs, double* partials, unsigned* counters,
                                              double* out, int stride) {
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    double red[1] = {0.0};
    for (int i = tl.first + (int)threadIdx.x; i < tl.end; i += blockDim.x) {
        const double d = x[i] - xs[i];
        red[0] += d * d;
    }
    seg_reduce_out<1>(red, T, tl.mesh, partials, counters, out, stride);
}

// Inputs of the global line search (Backtracking::search,
// deps/mcloptlib/include/MCL/Backtracking.hpp:71-98): out[0] = <q, q>,
// out[1] = <grad, grad> (sums), out[2] = max |grad|.
static __global__ void __launch_bounds__(256) k_ls_norms(int n, const double* __restrict__ q,
                                                  const double* __restrict__ grad, double* partials,
                                                  unsigned* counter, double* out) {
    double red[3] = {0.0, 0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        red[0] += q[i] * q[i];
        red[1] += grad[i] * grad[i];
        red[2] = fmax(red[2], fabs(grad[i]));
    }
    grid_reduce<3, 2>(red, partials, counter, out);
}

// Trial point of the line search: xt = x + alpha * p with p = -step; the same
// operation as k_xupdate's, so that an accepted step arrives at the trial's bits.
static __global__ void __launch_bounds__(256) k_ls_trial(int n, double* __restrict__ xt, const double* __restrict__ x,
                                                  const double* __restrict__ step, double alpha) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        xt[i] = fma(-alpha, step[i], x[i]);
}

// ---- ARAP local step (rotation-aware) ------------------------------------------
// polar_update, ARAP branch (src/TetElements.cpp:265-282): S = symF + U (both
// symmetric), Z = (S + I) / 2, U += symF - Z; curr_pe = sum vol |symF - I|^2 / 2.
// out[0..4] as k_local (no prox: [3] = [4] = 0).
static __global__ void __launch_bounds__(128) k_local_arap(ElemView E, Tiles T, const int* on, double* partials,
                                                         unsigned* counters, double* out, int stride) {
    const Tile tl = tile_at(T, blockIdx.x);
    if (!mesh_on(on, tl.mesh)) return;
    const int e = tl.first + threadIdx.x;
    double red[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (e < tl.end) {
        double S[9], Um[9], Zm[9];
        load9(E.symF, E.ne, e, S);
        load9(E.U, E.ne, e, Um);
        load9(E.Z, E.ne, e, Zm);
        const double w2 = E.w2[e], vol = E.vol[e];
        double bef = 0.0, aft = 0.0, n2 = 0.0;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            const double d = S[i] - (Zm[i] - Um[i]);
            bef += d * d;
        }
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            const double id = (i % 4 == 0) ? 1.0 : 0.0;
            const double So = 0.5 * ((S[i] + Um[i]) + id);
            n2 += (S[i] - id) * (S[i] - id);
            const double d = S[i] - (So - Um[i]);
            aft += d * d;
            Zm[i] = So;
            Um[i] = Um[i] + (S[i] - So);
        }
        red[0] = 0.5 * w2 * bef;
        red[1] = 0.5 * w2 * aft;
        red[2] = 0.5 * vol * n2;
        store9(E.Z, E.ne, e, Zm);
        store9(E.U, E.ne, e, Um);
    }
    seg_reduce_out<5>(red, T, tl.mesh, partials, counters, out, stride);
}

// ---- rotation-unaware ADMM (-ra 0) -----------------------------------------------
// initialize_dual_vars, rotation-unaware branch (src/TetElements.cpp:167-181):
// Z = Di x = F^T with all four slots read from X, U = 0.
static __global__ void __launch_bounds__(128) k_init_dual_unaware(ElemView E, const double* __restrict__ x,
                                                                const double* __restrict__ xfix) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E.ne) return;
    double F[9], Zm[9], zero[9] = {};
    deformation(E, e, x, xfix, false, F);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) M3(Zm, r, c) = F[c + 3 * r];
    store9(E.Z, E.ne, e, Zm);
    store9(E.U, E.ne, e, zero);
}

// UnawareGS right-hand side per element (TetElements::add_to_b,
// src/TetElements.cpp:470-481): b_e(a, r) = w^2 sum_c Di(c, a) (Z - U - Dfix xfix)(c, r),
// into the gradient rows gel (the gather adds the free slots).  From the new Z and U in
// the local step's registers: a launch that read them back took 7 us of 105 on 20x18x50
// (7.33 -> 7.19 ms per solve without it).
__device__ __forceinline__ void rhs_rows(const ElemView& E, int e, const double* __restrict__ xfix, double w2,
                                         const double* Zm, const double* Um) {
    double Ffix[9] = {};
    const int4 id = E.idx[e];
    const int s[4] = {id.x, id.y, id.z, id.w};
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (s[a] >= 0) continue;
        const double* p = xfix + 3 * (size_t)(-s[a] - 1);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double d = E.Di[(size_t)(c + 3 * a) * E.ne + e];
#pragma unroll
            for (int r = 0; r < 3; ++r) Ffix[c + 3 * r] += d * p[r];   // (Dfix xfix)(c, r)
        }
    }
    const int4 row = E.row[e];
    const int rows[4] = {row.x, row.y, row.z, row.w};
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (rows[a] < 0) continue;
        double b[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            double v = 0.0;
#pragma unroll
            for (int c = 0; c < 3; ++c)
                v += E.Di[(size_t)(c + 3 * a) * E.ne + e] * (M3(Zm, c, r) - M3(Um, c, r) - Ffix[c + 3 * r]);
            b[r] = w2 * v;
        }
        store_row(E.gel + (size_t)kRow * rows[a], b[0], b[1], b[2]);
    }
}

// TetElements::update (src/TetElements.cpp:193-254) from F at the current x
// (the defo cache): Dx = F^T, F' = (Dx + U)^T; NH: SVD of F', the prox from the
// last stretches, Z = V diag(sigma*) U^T; ARAP: Z = (F' + rot(F'))^T / 2; then
// U += Dx - Z.  C: arithmetic of the SVD and prox as in k_local (float in mixed
// mode, with the same FP64 rescue).  out[0..4] = 0, 0, 0, negative stretches,
// prox iterations.
template <typename C>
__global__ void __launch_bounds__(128, 4) k_local_unaware(ElemView E, const double* __restrict__ x,
                                                       const double* __restrict__ xfix, Material mat0, int prox_iters,
                                                       int cand_mode, int ratio, int prox_mode, double* partials,
                                                       unsigned* counter, double* out) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    double red[6] = {};
    if (e < E.ne) {
        const Material mat = elem_material(E, mat0, e);
        double F[9], Um[9], Zn[9];
        deformation(E, e, x, xfix, true, F);
        load9(E.U, E.ne, e, Um);
        C Fp[9];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) M3(Fp, r, c) = C(F[r + 3 * c] + M3(Um, c, r));   // (F^T + U)^T
        C sg[3], Ue[9], Ve[9];
        if constexpr (sizeof(C) == sizeof(double)) svd3_fast(Fp, sg, Ue, Ve);
        else svd3(Fp, sg, Ue, Ve);
        if (mat.model == MODEL_ARAP) {
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    // rot(F') = Ue Ve^T; Z(r, c) = (F'(c, r) + R(c, r)) / 2
                    const double Rcr = double(M3(Ue, c, 0) * M3(Ve, r, 0) + M3(Ue, c, 1) * M3(Ve, r, 1) +
                                              M3(Ue, c, 2) * M3(Ve, r, 2));
                    M3(Zn, r, c) = 0.5 * (double(M3(Fp, c, r)) + Rcr);
                }
        } else {
            const double w2 = E.w2[e], vol = E.vol[e];
            Prox<C> P;
            P.nh.mu = C(mat.mu);
            P.nh.lambda = C(mat.lambda);
            P.x0[0] = sg[0]; P.x0[1] = sg[1]; P.x0[2] = sg[2];
            P.wov = C(w2 / vol);
            C xs[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) xs[i] = C(E.slast[(size_t)i * E.ne + e]);
            int iters;
            if constexpr (sizeof(C) == sizeof(double)) {
                if (prox_mode != 0) {
                    iters = prox_newton(P, xs, prox_iters, C(1e-12));
                } else {
                    extern __shared__ double prox_hist[];
                    iters = prox_lbfgs(P, xs, prox_iters, ProxHistory<double>{prox_hist + threadIdx.x, (int)blockDim.x});
                    if (iters < 0) iters = prox_iters;
                }
            } else {
                iters = prox_newton(P, xs, prox_iters, C(8) * Lim<C>::eps());
                if (!(isfinite(xs[0]) && isfinite(xs[1]) && isfinite(xs[2]) && xs[0] >= C(0) && xs[1] >= C(0) &&
                      xs[2] >= C(0))) {
                    Prox<double> Pd;
                    Pd.nh.mu = mat.mu;
                    Pd.nh.lambda = mat.lambda;
                    Pd.x0[0] = double(sg[0]); Pd.x0[1] = double(sg[1]); Pd.x0[2] = double(sg[2]);
                    Pd.wov = w2 / vol;
                    double xd[3];
#pragma unroll
                    for (int i = 0; i < 3; ++i) xd[i] = E.slast[(size_t)i * E.ne + e];
                    iters += prox_newton(Pd, xd, prox_iters, 1e-12);
#pragma unroll
                    for (int i = 0; i < 3; ++i) xs[i] = C(xd[i]);
                }
            }
            red[4] = double(iters);
            double xo[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) { xo[i] = double(xs[i]); E.slast[(size_t)i * E.ne + e] = xo[i]; }
            red[3] = (xo[0] < 0.0 || xo[1] < 0.0 || xo[2] < 0.0) ? 1.0 : 0.0;
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    M3(Zn, r, c) = double(M3(Ve, r, 0) * xs[0] * M3(Ue, c, 0) + M3(Ve, r, 1) * xs[1] * M3(Ue, c, 1) +
                                          M3(Ve, r, 2) * xs[2] * M3(Ue, c, 2));
            double cand = 0.0;
            if (cand_mode == CAND_REST) {
                cand = vol * mat.wr;
            } else if (cand_mode == CAND_HESSIAN) {
                const double lm = NH<double>{mat.mu, mat.lambda}.template hess_lmax<sizeof(C) == sizeof(double)>(xo);
                double cnd = lm;
                if (lm < mat.wmin) cnd = mat.wmin;
                if (lm > mat.wmax) cnd = mat.wmax;
                cand = vol * cnd;
            }
            if (cand_mode != CAND_NONE) E.w2c[e] = cand;
            if (ratio) red[5] = weight_ratio(w2, cand);
        }
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) M3(Um, r, c) = M3(Um, r, c) + (F[c + 3 * r] - M3(Zn, r, c));
        store9(E.Z, E.ne, e, Zn);
        store9(E.U, E.ne, e, Um);
        rhs_rows(E, e, xfix, E.w2[e], Zn, Um);
    }
    if (ratio) {
        grid_reduce<6, 5>(red, partials, counter, out);
    } else {
        const double sums[5] = {red[0], red[1], red[2], red[3], red[4]};
        grid_reduce<5>(sums, partials, counter, out);
    }
}

}  // namespace wrapd
