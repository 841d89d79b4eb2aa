// Shared device/host helpers for the wrapd_b200 CUDA library.
#pragma once
#include <cuda_runtime.h>
#include <cfloat>
#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>

#include "../../include/wrapd_gpu.h"

namespace wrapd {

struct CudaError : std::runtime_error {
    int code;
    CudaError(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

#define WRAPD_CUDA(call)                                                                         \
    do {                                                                                         \
        cudaError_t err__ = (call);                                                              \
        if (err__ != cudaSuccess)                                                                \
            throw ::wrapd::CudaError(WRAPD_E_CUDA, std::string(#call " failed: ") +              \
                                                       cudaGetErrorString(err__));               \
    } while (0)

#define WRAPD_LAUNCH_CHECK() WRAPD_CUDA(cudaGetLastError())

template <typename T> struct Lim;
template <> struct Lim<double> {
    __host__ __device__ static constexpr double eps() { return DBL_EPSILON; }
    __host__ __device__ static constexpr double min() { return DBL_MIN; }
};
template <> struct Lim<float> {
    __host__ __device__ static constexpr float eps() { return FLT_EPSILON; }
    __host__ __device__ static constexpr float min() { return FLT_MIN; }
};

// 148 SMs on B200; grids for streaming kernels are sized in multiples of it.
constexpr int kNumSMs = 148;

inline int ceil_div(int64_t a, int64_t b) { return static_cast<int>((a + b - 1) / b); }

// Deterministic block reduction of NV values per thread, sums before M0 and maxima
// from M0 on (blockDim.x a multiple of 32, at most 1024): a shuffle tree per warp, then
// the warps in order.
// Returns the totals in thread 0.  One pair of barriers for all the values: with
// one pair for each, the five sums of the local step took ten barriers, a chain
// that a launch of few CTAs has nothing else to hide behind.
template <int NV, int M0 = NV>
__device__ __forceinline__ void block_reduce(double (&v)[NV]) {
    __shared__ double sm[NV][32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const double w = __shfl_down_sync(0xffffffffu, v[k], o);
            v[k] = k >= M0 ? fmax(v[k], w) : v[k] + w;
        }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();   // the previous call's readers of sm are done
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) sm[k][warp] = v[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        double r[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) r[k] = k >= M0 ? sm[k][0] : 0.0 + sm[k][0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
#pragma unroll
            for (int k = 0; k < NV; ++k) r[k] = k >= M0 ? fmax(r[k], sm[k][w]) : r[k] + sm[k][w];
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] = r[k];
    }
}

// ---- bounded waits between CTAs ----------------------------------------------
// A wait looks at most kWaitPolls times and for one second of the global timer
// (look_again).  One that gives up sets *status to WRAPD_E_TIMEOUT (if it was 0)
// and one that finds *status already set ends at once, so every waiter of a
// failed launch ends.
constexpr unsigned long long kWaitNs = 1000000000ull;
constexpr int kWaitPolls = 1 << 24;

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---- values handed from CTA to CTA by themselves -----------------------------
// An entry that is not yet written holds kUnset; its reader polls the entry itself
// until it holds a value, which thus crosses in one store and one load, with no
// fence, counter or flag between them.  kUnset is a signalling NaN, which no
// arithmetic operation returns, so no result can be mistaken for it.
constexpr unsigned long long kUnset = 0x7ff45a5a5a5a5a5aull;

__device__ __forceinline__ bool unset(double v) {
    return static_cast<unsigned long long>(__double_as_longlong(v)) == kUnset;
}
__device__ __forceinline__ double unset_value() { return __longlong_as_double(static_cast<long long>(kUnset)); }
__device__ __forceinline__ double ld_relaxed(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(double* p, double v) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
// After the i-th look at entries that were not all set (i from 0): whether to
// look again.  The status word and the timer, a round trip to memory each, are
// looked at every sixteenth time only: a hand-over's latency is a few looks.
__device__ __forceinline__ bool look_again(int i, unsigned long long& t0, int* status) {
    if ((i & 15) != 15) return true;
    if (*reinterpret_cast<volatile int*>(status) != 0) return false;
    const unsigned long long now = global_ns();
    if (i == 15) t0 = now;
    if (now - t0 > kWaitNs || i >= kWaitPolls) {
        atomicCAS(status, 0, WRAPD_E_TIMEOUT);
        return false;
    }
    __nanosleep(32);
    return true;
}

static __global__ void k_unset(double* __restrict__ p, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = unset_value();
}
inline void unset_fill(double* p, int64_t n, cudaStream_t st) {
    if (n <= 0) return;
    k_unset<<<ceil_div(n, 256), 256, 0, st>>>(p, n);
    WRAPD_LAUNCH_CHECK();
}

// One block more has written its partials: returns how many had before it.  The
// release orders thread 0's own stores only, and the partials are all that the last
// block reads: the other threads' stores (a gradient's rows) need not be waited for
// (a fence by every thread before the count: 166 -> 160 us for the gradient's
// value alone, 786k elements).
__device__ __forceinline__ unsigned arrive(unsigned* counter) {
    unsigned n;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], 1;" : "=r"(n) : "l"(counter) : "memory");
    return n;
}

// ---- deterministic grid reduction: per-block partials, summed in block order
// by whichever block finishes last. -------------------------------------------
// The sum of the partials of blocks [b0, b1): thread i takes blocks b0 + i,
// b0 + i + blockDim.x, ..., then a block sum.
template <int NV, int M0>
__device__ __forceinline__ void sum_partials(double (&acc)[NV], const double* partials, int b0, int b1) {
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = k >= M0 ? -1.0e308 : 0.0;
    for (int b = b0 + (int)threadIdx.x; b < b1; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const double p = __ldcg(partials + (size_t)b * NV + k);
            acc[k] = k >= M0 ? fmax(acc[k], p) : acc[k] + p;
        }
    block_reduce<NV, M0>(acc);
}

// out[k] = total_k.
template <int NV, int M0 = NV>
__device__ __forceinline__ void grid_reduce(const double (&v)[NV], double* partials, unsigned* counter, double* out) {
    __shared__ bool last;
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = v[k];
    block_reduce<NV, M0>(acc);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) partials[(size_t)blockIdx.x * NV + k] = acc[k];
        last = arrive(counter) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    sum_partials<NV, M0>(acc, partials, 0, (int)gridDim.x);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) out[k] = acc[k];
        *counter = 0u;
    }
}

// ---- launches over a batch of meshes ----------------------------------------
// A launch's blocks are tiles: tile b covers items [first, end) of one mesh
// (elements, free vertices or vector entries; each mesh's items are a
// contiguous range).  With a table (t != null) tile b is t[b] = {mesh, first,
// end}; without one (a single mesh) tile b covers [b * per, (b + 1) * per) of
// [0, n).  Every mesh's tiles start at its own first item, so a mesh's blocks
// in a batch do exactly the work of the same mesh's blocks when it is solved
// alone, and the per-mesh sums below add the same partials in the same order:
// a mesh's results in a batch equal its results alone, bit for bit.
struct Tiles {
    const int4* t;       // per tile {mesh, first, end, 0}, or null (one mesh)
    const int* tile0;    // per mesh its first tile, nm + 1 entries (with t)
    int n, per;          // one mesh: item count and items per tile
    int count;           // tiles of the launch
};
struct Tile {
    int mesh, first, end;
};
__device__ __forceinline__ Tile tile_at(const Tiles& T, int b) {
    if (T.t) {
        const int4 v = T.t[b];
        return {v.x, v.y, v.z};
    }
    return {0, b * T.per, min((b + 1) * T.per, T.n)};
}
// `on` (per mesh, null = all) masks whole meshes out of a launch: their tiles
// return before any work or synchronisation.
__device__ __forceinline__ bool mesh_on(const int* on, int mesh) { return !on || on[mesh] != 0; }

// Per-mesh grid reduction: per-tile partials; the last tile of each mesh to
// finish adds that mesh's partials in tile order (thread i takes tiles i,
// i + blockDim.x, ... of the mesh, then a fixed block sum).  Returns true in
// the last tile of the mesh, with the totals in tot[] of thread 0.  With one
// mesh and no table this is grid_reduce's arithmetic.  counters: one per
// mesh, zero between launches (the last tile resets its mesh's).
template <int NV, int M0 = NV>
__device__ __forceinline__ bool seg_reduce(const double (&v)[NV], const Tiles& T, int mesh, double* partials,
                                           unsigned* counters, double (&tot)[NV]) {
    __shared__ bool last;
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = v[k];
    block_reduce<NV, M0>(acc);
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) partials[(size_t)blockIdx.x * NV + k] = acc[k];
    const int t0 = T.t ? T.tile0[mesh] : 0, t1 = T.t ? T.tile0[mesh + 1] : (int)gridDim.x;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counters + mesh, 1u) == (unsigned)(t1 - t0 - 1);
    __syncthreads();
    if (!last) return false;
    __threadfence();
    sum_partials<NV, M0>(tot, partials, t0, t1);
    if (threadIdx.x == 0) counters[mesh] = 0u;
    return true;
}

// seg_reduce writing the totals to out[mesh * stride + k].
template <int NV, int M0 = NV>
__device__ __forceinline__ void seg_reduce_out(const double (&v)[NV], const Tiles& T, int mesh, double* partials,
                                               unsigned* counters, double* out, int stride) {
    double tot[NV];
    if (seg_reduce<NV, M0>(v, T, mesh, partials, counters, tot) && threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) out[(size_t)mesh * stride + k] = tot[k];
}

}  // namespace wrapd
