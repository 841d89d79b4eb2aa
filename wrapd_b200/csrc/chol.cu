// GPU multifrontal Cholesky and 3-RHS solve; see chol.cuh.
//
// Factorization, per level of the assembly tree (leaves first):
//   assemble     the fronts' entries from A and the children's update matrices;
//   then per panel of NB = 32 columns (right-looking partial Cholesky):
//   panel        every CTA factors the NB x NB diagonal block (four warps; a
//                fifth forms its inverse Li behind the pivots, also stored as a
//                diagonal block of Y), then applies Li to one tile: the panel rows
//                below the block, P <- P Li^T, or the inverse row block
//                Y[p, 0:p0] <- Li Y[p, 0:p0] (FP64 DMMA tiles);
//   update       blocked right-looking: inside the current OB-column block,
//                F[j0:, j0:be] -= P P^T and Y[j0:be, 0:j0] -= P Y[p, 0:j0];
//                after a block's last panel, the deferred trailing update
//                F[be:, be:] -= B B^T and Y[be:, 0:be] -= B Y[block, 0:be] with
//                K = OB (FP64 DMMA tiles, K-looped), so the large trailing
//                matrix is read and written once per OB columns, not per panel;
//   then         W = L_rs Y for the level's fronts (FP64 DMMA, K-looped).
// A's values are computed once per factorization, ahead of the levels.
//
// Every tile product is mma.sync.m8n8k4 f64 (the FP64 tensor-core path of
// sm_100a; tcgen05 has no f64 kind).
#include "chol.cuh"

#include <algorithm>
#include <numeric>
#include <type_traits>

namespace wrapd {

namespace {

constexpr int NB = 32;        // panel width
constexpr int OB = 256;       // outer block: trailing updates beyond it are deferred to one K = OB update
                              // (128: 1.5 % slower on the 3.9M bar; 512: slower on both bars)
constexpr int TL = 64;        // output tile of the DMMA kernels
constexpr int SLD = NB + 4;   // smem row pitch (doubles) for [row][k] operand tiles
constexpr int GEMM_THREADS = 128;
constexpr int kFusedPanelCtas = 4 * 148;   // panel steps up to one wave (4 CTAs per SM) run fused
constexpr int COLS_PER_CTA = 8;    // assembly column groups (one warp each)

// The list item that owns CTA b: the last i < n with prefix[i] <= b.  The lanes of a
// warp look at 32 places at once, so a list of up to 32 items takes one round
// trip to memory and one of 1024 two (a binary search takes five and ten, one
// after the other, before a CTA can load anything).
__device__ __forceinline__ int find_item(const int* prefix, int n, int b) {
    const int lane = threadIdx.x & 31;
    int lo = 0, len = n;
    while (len > 1) {
        const int step = (len + 31) >> 5, o = lane * step;
        const bool le = o < len && __ldg(prefix + lo + o) <= b;
        const int j = 31 - __clz(__ballot_sync(0xffffffffu, le));
        lo += j * step;
        len = min(step, len - j * step);
    }
    return lo;
}

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// S[i][t] = base[i*rs + t*cs] for i < rows, t < K; zero elsewhere (TL x K4).
__device__ __forceinline__ void load_tile(double* S, const double* __restrict__ base, int64_t rs, int64_t cs,
                                          int rows, int K, int K4) {
    const int total = TL * K4;
    if (rs == 1) {
        for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
            const int i = idx % TL, t = idx / TL;
            S[i * SLD + t] = (i < rows && t < K) ? base[i + t * cs] : 0.0;
        }
    } else {
        for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
            const int t = idx % K4, i = idx / K4;
            S[i * SLD + t] = (i < rows && t < K) ? base[i * rs + t * cs] : 0.0;
        }
    }
}

// acc += As * Bs^T over K4 (multiple of 4); 4 warps in a 2x2 grid of 32x32.
__device__ __forceinline__ void tile_mma(const double* As, const double* Bs, int K4, double (&acc)[4][4][2]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = warp & 1, wn = warp >> 1;
    const int r = lane >> 2, c = lane & 3;
    for (int kk = 0; kk < K4; kk += 4) {
        double a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = As[(wm * 32 + i * 8 + r) * SLD + kk + c];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = Bs[(wn * 32 + j * 8 + r) * SLD + kk + c];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
}

// C[row*crs + col*ccs] = acc for row < M, col < N.
__device__ __forceinline__ void tile_store(double* C, int64_t crs, int64_t ccs, int M, int N,
                                           const double (&acc)[4][4][2]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = warp & 1, wn = warp >> 1;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = wm * 32 + i * 8 + (lane >> 2);
                const int col = wn * 32 + j * 8 + 2 * (lane & 3) + h;
                if (row < M && col < N) C[row * crs + col * ccs] = acc[i][j][h];
            }
}

// ---- pipelined GEMM core ------------------------------------------------------
// 64 x 64 tiles of FP64 DMMA, four CTAs of four warps per SM, K in chunks of KC
// columns staged by cp.async, three stages, one barrier per chunk.  Operand tiles
// are staged in one of two layouts, chosen by which index is contiguous in global
// memory so that both the staging writes and the DMMA fragment reads (4 x 4 values
// per half-warp) hit every shared-memory bank evenly:
//   t-major S[t * TP + i] for sources with i contiguous (columns of F); a source
//     that starts on an odd row is staged from the even row before it, shifted by
//     one, so that its copies are 16 bytes wide too;
//   i-major S[i * KC + (t ^ 4 (i % 4))] for sources with t contiguous (row blocks of Y).
// The loop is bound by the DMMA pipe only if little else is issued: a thread's
// copies differ from chunk to chunk by one pointer step, and the k-steps are
// unrolled with constant shared-memory offsets, so a DMMA comes with about two other
// instructions (twelve in the form before, which recomputed every copy's place and
// ran two barriers a chunk).  Rate on the 64x64x160 bar's trailing updates and W
// products: 27 -> 31 to 32.6 of the 37.1 TFLOP/s that the instruction reaches alone.
// Every entry adds its products in ascending k in steps of four, whatever the chunks.
constexpr int KC = 16;                // K columns per staged chunk
constexpr int TP = TL + 4;            // t-major pitch (4 mod 16 doubles)
constexpr int TILE_D = KC * TP;       // doubles per staged operand tile
constexpr int GEMM_STAGES = 3;
constexpr int GEMM_SMEM = GEMM_STAGES * 2 * TILE_D * (int)sizeof(double);   // stages x (A, B)
static_assert(TL * KC <= TILE_D && KC == 16 && GEMM_THREADS == 128, "the staging maps below");

__device__ __forceinline__ void cp_async8(double* s, const double* g, bool valid) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(s));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(g), "r"(valid ? 8 : 0));
}
// 16-byte copy of which the first src_bytes (16, 8 or 0) come from global
// memory and the rest is zero-filled; both addresses 16-byte aligned.
__device__ __forceinline__ void cp_async16(double* s, const double* g, int src_bytes) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(s));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(g), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// One operand of a tile: element (i, t), i < rows, t < K, at base[i + t * ld]
// (TMAJOR) or base[i * ld + t].  TMAJOR: thread copies row pair tid % 32 of columns
// tid / 32 + 4 u; else: column pair tid % 8 of rows tid / 8 + 16 u.  ld is even, and
// an i-major base even too.
template <bool TMAJOR>
struct Operand {
    const double* base;   // a valid address, for copies of nothing
    const double* p;      // this thread's first source of the next chunk
    int64_t step;         // between its copies
    int64_t chunk;        // between chunks
    double* dst;          // within a stage
    int t0;               // its first (TMAJOR) or only t
    int bytes;            // TMAJOR: of the row pair that exist; else: how many of its four rows exist
    int shift;            // TMAJOR: rows the source is shifted by
    bool last;            // TMAJOR, shifted: this thread copies row TL - 1 of column tid

    __device__ __forceinline__ void init(const double* b, int64_t ld, int rows, double* s) {
        const int tid = threadIdx.x;
        base = b;
        if constexpr (TMAJOR) {
            shift = (reinterpret_cast<uintptr_t>(b) >> 3) & 1;
            const int i = 2 * (tid & 31), left = rows + shift - i;
            t0 = tid >> 5;
            bytes = left <= 0 ? 0 : left == 1 ? 8 : 16;
            p = b - shift + (bytes ? i : shift) + (int64_t)t0 * ld;
            step = 4 * ld;
            chunk = KC * ld;
            dst = s + t0 * TP + i;
            last = shift && rows == TL && tid < KC;
        } else {
            const int i = tid >> 3;
            t0 = 2 * (tid & 7);
            bytes = rows <= i ? 0 : (rows - i + 15) >> 4;
            p = b + (int64_t)i * ld + t0;
            step = 16 * ld;
            chunk = KC;
            dst = s + i * KC + (t0 ^ (4 * (i & 3)));
            shift = 0;
            last = false;
        }
    }
    // Copies the chunk that has `left` columns of K left into stage `st`.
    __device__ __forceinline__ void issue(int st, int left) {
        double* d = dst + st * (2 * TILE_D);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if constexpr (TMAJOR) {
                const bool v = t0 + 4 * u < left;
                cp_async16(d + 4 * u * TP, v ? p + u * step : base - shift, v ? bytes : 0);
            } else {
                const int n = u < bytes ? min(max(left - t0, 0), 2) : 0;
                cp_async16(d + 16 * u * KC, n ? p + u * step : base, 8 * n);
            }
        }
        if constexpr (TMAJOR) {
            // row TL - 1 of a shifted source lies in the 33rd pair: its column is this thread's number
            if (last) {
                const bool v = (int)threadIdx.x < left;
                const int64_t ld = step >> 2;
                const double* q = p + (TL - 2 * (int)(threadIdx.x & 31)) + ((int)threadIdx.x - t0) * ld;
                cp_async8(d - (t0 * TP + 2 * (threadIdx.x & 31)) + threadIdx.x * TP + TL, v ? q : base, v);
            }
        }
        p += chunk;
    }
};

// acc += A B'^T over t in [0, K): A(i, t) = A0[i + t * lda] (i < M), B'(j, t) =
// B0[j + t * ldb] when BT, else B0[j * ldb + t] (j < N).  4 warps in a 2 x 2 grid of 32 x 32.
template <bool BT>
__device__ __forceinline__ void gemm_pipelined(const double* A0, int64_t lda, int M, const double* B0, int64_t ldb,
                                               int N, int K, double* smem, double (&acc)[4][4][2]) {
    const int nch = (K + KC - 1) / KC;
    Operand<true> A;
    Operand<BT> B;
    A.init(A0, lda, M, smem);
    B.init(B0, ldb, N, smem + TILE_D);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = warp & 1, wn = warp >> 1, r = lane >> 2, c = lane & 3;
    const double* As = smem + c * TP + wm * 32 + r + A.shift;
    // i-major: (t ^ 4 (i % 4)) with t = kk + c: the k-step kk is swizzled by the row's low bits
    const double* Bs = smem + TILE_D + (BT ? c * TP + wn * 32 + r + B.shift : (wn * 32 + r) * KC + c);
    const int sw = BT ? 0 : 4 * (r & 3);
#pragma unroll
    for (int s = 0; s < GEMM_STAGES - 1; ++s) {
        if (s < nch) {
            A.issue(s, K - s * KC);
            B.issue(s, K - s * KC);
        }
        cp_async_commit();   // an empty group past the last chunk keeps the wait count uniform
    }
    int rd = 0, wr = GEMM_STAGES - 1;
    for (int k = 0; k < nch; ++k) {
        cp_async_wait<GEMM_STAGES - 2>();
        __syncthreads();   // chunk k is there, and stage wr, read for chunk k - 1, is free
        const int left = K - (k + GEMM_STAGES - 1) * KC;
        if (left > 0) {
            A.issue(wr, left);
            B.issue(wr, left);
        }
        cp_async_commit();
        const double* a0 = As + rd * (2 * TILE_D);
        const double* b0 = Bs + rd * (2 * TILE_D);
#pragma unroll
        for (int kk = 0; kk < KC; kk += 4) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = a0[kk * TP + i * 8];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = BT ? b0[kk * TP + j * 8] : b0[j * 8 * KC + (kk ^ sw)];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
        }
        rd = rd + 1 == GEMM_STAGES ? 0 : rd + 1;
        wr = wr + 1 == GEMM_STAGES ? 0 : wr + 1;
    }
    cp_async_wait<0>();
}

// ---- assembly ----------------------------------------------------------------
// The values of A's lower-triangle entries, by front column (see build).
__global__ void k_assemble_A(double* __restrict__ Aval, const int* __restrict__ slot, const int* __restrict__ ptr,
                             const int* __restrict__ con, int nA, const double* __restrict__ w2,
                             const double* __restrict__ Di, int ne) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nA) return;
    double v = 0.0;
    for (int q = ptr[t]; q < ptr[t + 1]; ++q) {
        const int c = con[q];
        const int e = c >> 4, a = (c >> 2) & 3, b = c & 3;
        double d = 0.0;
#pragma unroll
        for (int r = 0; r < 3; ++r) d += Di[(int64_t)(r + 3 * a) * ne + e] * Di[(int64_t)(r + 3 * b) * ne + e];
        v += w2[e] * d;
    }
    Aval[slot[t]] = v;
}

// The front column of entry t of A (at F-pool offset pos[t]): counted, or, with the
// columns' first places ptr, given the next place of its column.
__global__ void k_A_places(int nA, const int64_t* __restrict__ pos, const FrontDesc* __restrict__ desc, int nfronts,
                           const int* __restrict__ ptr, int* cnt, int* __restrict__ slot, int* __restrict__ row) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nA) return;
    int lo = 0, hi = nfronts;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (desc[mid].f_off <= pos[t]) lo = mid; else hi = mid;
    }
    const int64_t o = pos[t] - desc[lo].f_off;
    const int ld = desc[lo].ld, col = desc[lo].first + static_cast<int>(o / ld);
    const int k = atomicAdd(cnt + col, 1);
    if (!ptr) return;
    slot[t] = ptr[col] + k;
    row[ptr[col] + k] = static_cast<int>(o % ld);
}

// The k x k part of every front's Y block: the identity (a warp per column).
__global__ void __launch_bounds__(32 * COLS_PER_CTA) k_y_identity(double* __restrict__ Y, const FrontDesc* __restrict__ desc,
                                                                  WorkList wl) {
    const int item = find_item(wl.d_prefix, wl.n, blockIdx.x);
    const FrontDesc d = desc[wl.d_fronts[item]];
    const int j = (blockIdx.x - wl.d_prefix[item]) * COLS_PER_CTA + (threadIdx.x >> 5);
    if (j >= d.k) return;
    double* Yj = Y + d.y_off + (int64_t)j * d.ldy;
    for (int i = threadIdx.x & 31; i < d.k; i += 32) Yj[i] = i == j ? 1.0 : 0.0;
}

// The fronts of a level: F(i, j), i >= j, = A(i, j) + U_c0(., .) + U_c1(., .), the
// entries of A (front columns only) and of the children's update matrices that
// land there, added in that order; zeros elsewhere.  A warp writes a column, so
// the front is written once and nothing is read but the children's update
// matrices and the row map, which a CTA's eight columns share in L1: 8 bytes
// per front entry and 8 per child entry.  (The form before zeroed whole squares
// and added each child in place, 8 bytes per square entry and 24 per child
// entry: memset and extend-add took 1.72 ms of a factorization of the 32x32x128
// bar and 14.6 ms on the 64x64x160 one, this takes 0.70 and 5.4.)  The strict
// upper triangle is never read; the padding row is, into itself alone, and is
// written as zero.
__global__ void __launch_bounds__(32 * COLS_PER_CTA) k_assemble_front(double* F, const FrontDesc* __restrict__ desc,
                                                                      const int* __restrict__ inv,
                                                                      const double* __restrict__ Aval,
                                                                      const int* __restrict__ Acol,
                                                                      const int* __restrict__ Arow, WorkList wl) {
    const int item = find_item(wl.d_prefix, wl.n, blockIdx.x);
    const FrontDesc d = desc[wl.d_fronts[item]];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = (blockIdx.x - wl.d_prefix[item]) * COLS_PER_CTA + warp;
    const int R = d.k + d.r;
    if (j >= R) return;
    const int2* iv = reinterpret_cast<const int2*>(inv + d.inv_off);
    double* Fj = F + d.f_off + (int64_t)j * d.ld;
    // the children's update columns landing on column j (null: none), indexed by row of U
    const double *C0 = nullptr, *C1 = nullptr;
    const int2 ij = iv[j];
    if (ij.x >= 0) {
        const FrontDesc& c = desc[d.child0];
        const int u0 = static_cast<int>(c.u_off / 3);
        C0 = F + c.f_off + c.k + (int64_t)(c.k + ij.x - u0) * c.ld - u0;
    }
    if (ij.y >= 0) {
        const FrontDesc& c = desc[d.child1];
        const int u0 = static_cast<int>(c.u_off / 3);
        C1 = F + c.f_off + c.k + (int64_t)(c.k + ij.y - u0) * c.ld - u0;
    }
    constexpr int U = 4;   // rows per lane whose reads go out together
    for (int i0 = j + lane; i0 < d.ld; i0 += 32 * U) {
        double c0[U], c1[U];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const int i = i0 + 32 * q;
            const int2 m = (i < R && (C0 || C1)) ? iv[i] : make_int2(-1, -1);
            c0[q] = (C0 && m.x >= 0) ? C0[m.x] : 0.0;
            c1[q] = (C1 && m.y >= 0) ? C1[m.y] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < U; ++q)
            if (i0 + 32 * q < d.ld) Fj[i0 + 32 * q] = c0[q] + c1[q];
    }
    if (j >= d.k) return;
    __syncwarp();   // the column's entries of A over what the loop wrote there
    const int t1 = Acol[d.first + j + 1];
    for (int t = Acol[d.first + j] + lane; t < t1; t += 32) {
        const int i = Arow[t];
        const int2 m = iv[i];
        double v = Aval[t];
        if (C0 && m.x >= 0) v += C0[m.x];
        if (C1 && m.y >= 0) v += C1[m.y];
        Fj[i] = v;
    }
}

// ---- panel factorization -------------------------------------------------------
// Cholesky of the nb x nb (nb <= NB = 32) diagonal block at Fd (column-major,
// lower part read) and its inverse, in shared memory by a CTA of CHOL_THREADS:
// four warps run the pivots, the fifth the inverse, one row behind them.
// Right-looking: at pivot j every thread updates a fixed slice of 8 entries
// of row i = tid % 32 (columns tid / 32 + 4m), with all its operands loaded
// before the first store, so one barrier per pivot is the only serial step.
// Every thread also works out the next pivot, A'(j+1, j+1) less its update, and
// starts its rsqrt before the barrier, whose latency then runs behind the updates
// (the entry itself is left as it is: nobody reads it again).
// L(i, j) = A'(i, j) rsqrt(d) goes to Lsm (pitch lp), rsqrt(d) to D.  The
// inverse is right-looking by rows: lane c of the fifth warp owns
// column c of inv(L), its partial sums P(r, c) in registers; row s of the
// column is (delta(s, c) - P(s, c)) / L(s, s), and the rows below add L(r, s)
// times it (the same fma sequence per entry as a row-by-row sweep; the sums of
// rows past nb are never used and are not guarded: the 496 branches took more
// than half of the inverse's time).  Row s of inv(L) is written to X (pitch xp),
// columns < nb.  A non-positive (or NaN) pivot sets *bad and continues with a unit
// pivot.  A pivot's 320 cycles are its rsqrt and the three operations between
// two of them.  Measured, cycles for a block of 32: pivots 10.4k and inverse
// behind them 0.3k; with the four warps alone, the inverse after the pivots,
// 10.4k + 5.1k (12.0k with its guards).
constexpr int LSP = NB + 1;
constexpr int CHOL_THREADS = GEMM_THREADS + 32;
static_assert(GEMM_THREADS == 128 && NB == 32, "cta_chol_inv maps 128 threads onto 32 rows x 4 column slices");
// A barrier of the CTA's CHOL_THREADS that its warps reach in different loops.
__device__ __forceinline__ void chol_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(CHOL_THREADS) : "memory"); }
__device__ __forceinline__ void cta_chol_inv(const double* __restrict__ Fd, int64_t ld, int nb, double* S,
                                             double* Lsm, int lp, double* D, double* X, int xp, bool* bad) {
    const int tid = threadIdx.x;
    for (int idx = tid; idx < NB * NB; idx += CHOL_THREADS) {
        const int i = idx & 31, c = idx >> 5;
        S[i * LSP + c] = (i < nb && c <= i) ? Fd[i + (int64_t)c * ld] : 0.0;
    }
    __syncthreads();
    bool b = false;
    if (tid < GEMM_THREADS) {
        const int i = tid & 31, q = tid >> 5;
        double piv = S[0];
        if (!(piv > 0.0)) { b = true; piv = 1.0; }
        double rs = rsqrt(piv);
        for (int j = 0; j < nb; ++j) {
            const double sij = S[i * LSP + j];
            const int n = min(j + 1, NB - 1);
            const double nj = S[n * LSP + j], nn = S[n * LSP + n];
            double cj[8], ic[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                cj[m] = S[(q + 4 * m) * LSP + j];
                ic[m] = S[i * LSP + q + 4 * m];
            }
            const double r2 = rs * rs;
            double next = fma(-(nj * r2), nj, nn);
            if (j + 1 < nb && !(next > 0.0)) { b = true; next = 1.0; }
            if (q == 0 && i >= j && i < nb) Lsm[i * lp + j] = i == j ? piv * rs : sij * rs;
            if (tid == 0) D[j] = rs;
            const double t = sij * r2;
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                const int c = q + 4 * m;
                if (c > j && c <= i && i < nb && i > j + 1) S[i * LSP + c] = fma(-t, cj[m], ic[m]);
            }
            piv = next;
            rs = rsqrt(next);
            chol_barrier();
        }
    } else {
        const int c = tid - GEMM_THREADS;
        double P[NB];
#pragma unroll
        for (int r = 0; r < NB; ++r) P[r] = 0.0;
#pragma unroll
        for (int s = 0; s < NB; ++s) {
            if (s < nb) {
                chol_barrier();   // column s of L and D[s] are there
                const double f = (c <= s) ? ((c == s ? 1.0 : 0.0) - P[s]) * D[s] : 0.0;
                if (c < nb) X[s * xp + c] = f;
#pragma unroll
                for (int r = s + 1; r < NB; ++r) P[r] = fma(Lsm[r * lp + s], f, P[r]);
            }
        }
    }
    __syncthreads();
    *bad = b;
}

// Diagonal step alone, for panel steps with many CTAs (where redoing the
// block in every CTA would cost more than a launch): one CTA per front
// factors the block and writes Li as the diagonal block of Y.
__global__ void __launch_bounds__(CHOL_THREADS) k_diag(const double* __restrict__ F, double* __restrict__ Y,
                                                       const FrontDesc* __restrict__ desc, WorkList wl, int p,
                                                       int* __restrict__ status) {
    __shared__ double S[NB * LSP];
    __shared__ double Lsm[NB * LSP];
    __shared__ double X[NB * LSP];
    __shared__ double D[NB];
    const FrontDesc d = desc[wl.d_fronts[blockIdx.x]];
    const int p0 = p * NB, nb = min(NB, d.k - p0);
    if (nb <= 0) return;
    bool bad = false;
    cta_chol_inv(F + d.f_off + p0 + (int64_t)p0 * d.ld, d.ld, nb, S, Lsm, LSP, D, X, LSP, &bad);
    if (bad && threadIdx.x == 0) atomicExch(status, WRAPD_E_NOT_SPD);
    double* Yp = Y + d.y_off + p0;   // row block p of Y (column-major, ld = ldy)
    for (int idx = threadIdx.x; idx < NB * NB; idx += CHOL_THREADS) {
        const int i = idx & 31, c = idx >> 5;
        if (i < nb && c < nb) Yp[i + (int64_t)(p0 + c) * d.ldy] = c <= i ? X[i * LSP + c] : 0.0;
    }
}

// The tiles of a panel step after k_diag: nP panel-row tiles (P <- P Li^T),
// then the inverse row-block tiles Y[p, c0:c0+64] <- Li Y[p, c0:c0+64], with
// Li read back from Y's diagonal block.
__global__ void __launch_bounds__(GEMM_THREADS) k_trsm(double* __restrict__ F, double* __restrict__ Y,
                                                       const FrontDesc* __restrict__ desc, WorkList wl,
                                                       const int* __restrict__ nP_of_item, int p) {
    __shared__ double As[TL * SLD];
    __shared__ double Bs[TL * SLD];
    const int item = find_item(wl.d_prefix, wl.n, blockIdx.x);
    const FrontDesc d = desc[wl.d_fronts[item]];
    const int tile = blockIdx.x - wl.d_prefix[item];
    const int nP = nP_of_item[item];
    const int p0 = p * NB, nb = min(NB, d.k - p0), j0 = p0 + nb;
    if (nb <= 0) return;
    const int K4 = (nb + 3) & ~3;
    const double* Li = Y + d.y_off + p0 + (int64_t)p0 * d.ldy;   // Li(i, t) at Li[i + t ldy]
    double acc[4][4][2] = {};
    if (tile < nP) {
        const int m = min(d.ld - j0 - tile * TL, TL);
        double* A = F + d.f_off + j0 + tile * TL + (int64_t)p0 * d.ld;
        load_tile(As, A, 1, d.ld, m, nb, K4);
        load_tile(Bs, Li, 1, d.ldy, nb, nb, K4);
        __syncthreads();
        tile_mma(As, Bs, K4, acc);
        tile_store(A, 1, d.ld, m, nb, acc);
    } else {
        const int c0 = (tile - nP) * TL;
        if (c0 >= p0) return;
        double* Yr = Y + d.y_off + p0 + (int64_t)c0 * d.ldy;   // Y[p0 + t, c0 + j] at Yr[t + j ldy]
        load_tile(As, Li, 1, d.ldy, nb, nb, K4);
        load_tile(Bs, Yr, d.ldy, 1, min(p0 - c0, TL), nb, K4);
        __syncthreads();
        tile_mma(As, Bs, K4, acc);
        tile_store(Yr, 1, d.ldy, nb, min(p0 - c0, TL), acc);
    }
}

// Panel steps with few CTAs (the upper levels: a few large fronts, where the
// step is latency-bound) run as one launch: every CTA first factors the
// front's NB x NB diagonal block itself (cta_chol_inv) and keeps its
// inverse Li in shared memory, so no separate diagonal launch precedes it.  Items per front: nP
// panel-row tiles (P <- P Li^T below the diagonal block), then the inverse
// row-block tiles Y[p, c0:c0+64] <- Li Y[p, c0:c0+64], c0 < p0; a front with
// neither has one item that only factors.  The front's first item writes Li
// as the diagonal block of Y.  F's diagonal block is read, never written: the
// solve and the later steps use only Y, W and the panels below it.
__global__ void __launch_bounds__(CHOL_THREADS) k_panel(double* __restrict__ F, double* __restrict__ Y,
                                                        const FrontDesc* __restrict__ desc, WorkList wl,
                                                        const int* __restrict__ nP_of_item, int p,
                                                        int* __restrict__ status) {
    __shared__ __align__(16) double As[TL * SLD];
    __shared__ __align__(16) double Bs[TL * SLD];
    __shared__ double S[NB * LSP];
    __shared__ double D[NB];
    const int item = find_item(wl.d_prefix, wl.n, blockIdx.x);
    const FrontDesc d = desc[wl.d_fronts[item]];
    const int tile = blockIdx.x - wl.d_prefix[item];
    const int nP = nP_of_item[item];
    const int p0 = p * NB, nb = min(NB, d.k - p0), j0 = p0 + nb;
    if (nb <= 0) return;
    const int K4 = (nb + 3) & ~3;
    const bool ptile = tile < nP;
    const int c0 = (tile - nP) * TL;
    const bool ytile = !ptile && c0 < p0;
    // The other operand is staged asynchronously while the diagonal block is
    // factored: the panel rows (A(i, t) = P(i, t)) or the Y row block (B'(j, t)
    // = Y(p0 + t, c0 + j)).
    const int tid = threadIdx.x;
    if (ptile) {
        const int m = min(d.ld - j0 - tile * TL, TL);
        const double* A = F + d.f_off + j0 + tile * TL + (int64_t)p0 * d.ld;
        for (int idx = tid; idx < TL * K4; idx += CHOL_THREADS) {
            const int i = idx % TL, t = idx / TL;
            const bool v = i < m && t < nb;
            cp_async8(As + i * SLD + t, v ? A + i + (int64_t)t * d.ld : A, v);
        }
    } else if (ytile) {
        const int n = min(p0 - c0, TL);
        const double* Yr = Y + d.y_off + p0 + (int64_t)c0 * d.ldy;
        for (int idx = tid; idx < TL * K4; idx += CHOL_THREADS) {
            const int t = idx % K4, j = idx / K4;
            const bool v = j < n && t < nb;
            cp_async8(Bs + j * SLD + t, v ? Yr + t + (int64_t)j * d.ldy : Yr, v);
        }
    }
    cp_async_commit();
    // Li lands in the operand slot of the product: B for panel tiles (B'(j, t) =
    // Li(j, t)), A for inverse row-block tiles (A(i, t) = Li(i, t)); rows 32..63
    // of that slot hold L meanwhile and are cleared afterwards.
    double* Ls = ptile ? Bs : As;
    for (int idx = tid; idx < NB * SLD; idx += CHOL_THREADS) Ls[idx] = 0.0;
    bool bad = false;
    cta_chol_inv(F + d.f_off + p0 + (int64_t)p0 * d.ld, d.ld, nb, S, Ls + NB * SLD, SLD, D, Ls, SLD, &bad);
    if (tile == 0) {
        if (bad && tid == 0) atomicExch(status, WRAPD_E_NOT_SPD);
        double* Yp = Y + d.y_off + p0;   // row block p of Y (column-major, ld = ldy)
        for (int idx = tid; idx < NB * NB; idx += CHOL_THREADS) {
            const int i = idx & 31, c = idx >> 5;
            if (i < nb && c < nb) Yp[i + (int64_t)(p0 + c) * d.ldy] = Ls[i * SLD + c];
        }
    }
    __syncthreads();
    for (int idx = tid; idx < NB * SLD; idx += CHOL_THREADS) Ls[NB * SLD + idx] = 0.0;
    cp_async_wait<0>();
    __syncthreads();
    if ((!ptile && !ytile) || tid >= GEMM_THREADS) return;   // the product is the first four warps'
    double acc[4][4][2] = {};
    tile_mma(As, Bs, K4, acc);
    if (ptile) {
        const int m = min(d.ld - j0 - tile * TL, TL);
        tile_store(F + d.f_off + j0 + tile * TL + (int64_t)p0 * d.ld, 1, d.ld, m, nb, acc);
    } else {
        tile_store(Y + d.y_off + p0 + (int64_t)c0 * d.ldy, 1, d.ldy, nb, min(p0 - c0, TL), acc);
    }
}

#ifndef WRAPD_EPI_BATCH
#define WRAPD_EPI_BATCH 8
#endif
constexpr int EPI_BATCH = WRAPD_EPI_BATCH;   // columns per thread whose reads the staged epilogue issues together
constexpr int EPI_P = TL + 2;   // pitch of the staged output tile: lanes' (row, 2-column) fragments hit distinct banks
static_assert(TL * EPI_P <= 2 * GEMM_STAGES * TILE_D, "the staged output tile reuses the operand stages");
static_assert(TL == 2 * 32 && GEMM_THREADS == 2 * TL, "the staged epilogue maps two threads per row");

// C[row + col*ld] -= acc for row < M, col < N and row + diag >= col, through
// shared memory: the fragments go to a column-major tile, then each warp
// updates 32 consecutive rows of a column (coalesced) with EPI_BATCH columns'
// reads in flight before their writes.  Direct read-modify-writes from the
// fragments would be serialised, since a store through C may alias the next
// read as far as the compiler can tell.  `smem` (the operand stages) must have
// no reads pending from other threads; the call's first barrier ensures that.
__device__ __forceinline__ void tile_sub_staged(double* __restrict__ C, int64_t ld, int M, int N, int diag,
                                                const double (&acc)[4][4][2], double* smem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = warp & 1, wn = warp >> 1;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = wm * 32 + i * 8 + (lane >> 2);
                const int col = wn * 32 + j * 8 + 2 * (lane & 3) + h;
                smem[col * EPI_P + row] = acc[i][j][h];
            }
    __syncthreads();
    const int row = threadIdx.x & (TL - 1), cg = threadIdx.x >> 6;
    if (row >= M) return;
    // columns cg, cg + 2, ... below N and with row + diag >= col
    const int cend = min(N, row + diag + 1);
#pragma unroll 1
    for (int c0 = cg; c0 < cend; c0 += 2 * EPI_BATCH) {
        double v[EPI_BATCH];
#pragma unroll
        for (int q = 0; q < EPI_BATCH; ++q) {
            const int col = c0 + 2 * q;
            v[q] = col < cend ? C[row + (int64_t)col * ld] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < EPI_BATCH; ++q) {
            const int col = c0 + 2 * q;
            if (col < cend) C[row + (int64_t)col * ld] = v[q] - smem[col * EPI_P + row];
        }
    }
}

// Tile t of a job: kind 0 enumerates lower tiles (ti >= tj) column by column,
// kind 1 the full rectangle.  Column tj of the lower tiles starts at tile
// tj Tr - tj (tj - 1) / 2; the root of that, corrected, gives tj.
__device__ __forceinline__ void job_tile(const GemmJob& jb, int t, int& ti, int& tj) {
    const int Tr = (jb.rows + TL - 1) / TL, Tc = (jb.cols + TL - 1) / TL;
    if (jb.kind == 1) { ti = t / Tc; tj = t - ti * Tc; return; }
    const float m = 2.0f * Tr + 1.0f;
    tj = static_cast<int>(0.5f * (m - sqrtf(fmaxf(0.0f, m * m - 8.0f * t))));
    tj = max(0, min(tj, Tc - 1));
    auto start = [&](int c) { return c * Tr - (c * (c - 1)) / 2; };
    while (tj > 0 && start(tj) > t) --tj;
    while (tj + 1 < Tc && start(tj + 1) <= t) ++tj;
    ti = tj + t - start(tj);
}

#ifndef WRAPD_GEMM_MINB
#define WRAPD_GEMM_MINB 4
#endif
__global__ void __launch_bounds__(GEMM_THREADS, WRAPD_GEMM_MINB) k_update(double* __restrict__ F, double* __restrict__ Y,
                                                         JobList jl) {
    extern __shared__ __align__(16) double gemm_smem[];
    const int item = find_item(jl.d_prefix, jl.n, blockIdx.x);
    const GemmJob jb = jl.d_jobs[item];
    int ti, tj;
    job_tile(jb, blockIdx.x - jl.d_prefix[item], ti, tj);
    const int r0 = ti * TL, c0 = tj * TL;
    const int M = min(TL, jb.rows - r0), N = min(TL, jb.cols - c0);
    double* C = (jb.kind == 0 ? F : Y) + jb.c + r0 + (int64_t)c0 * jb.ldc;
    // the tile of C that the epilogue reads: towards L2 meanwhile (16 lines of 128 bytes
    // per 4 columns at most; rows past M stay in the pool's next columns)
    for (int q = threadIdx.x; q < 4 * N; q += GEMM_THREADS)
        if (16 * (q & 3) < M) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + 16 * (q & 3) + (int64_t)(q >> 2) * jb.ldc));
    double acc[4][4][2] = {};
    const double* A0 = F + jb.a + r0;
    if (jb.kind == 0)
        gemm_pipelined<true>(A0, jb.lda, M, F + jb.b + c0, jb.lda, N, jb.K, gemm_smem, acc);
    else   // B'(j, t) = Y(k0 + t, c0 + j)
        gemm_pipelined<false>(A0, jb.lda, M, Y + jb.b + (int64_t)c0 * jb.ldc, jb.ldc, N, jb.K, gemm_smem, acc);
    // on tiles of kind 0 crossing the diagonal keep only row >= column (global indices)
    tile_sub_staged(C, jb.ldc, M, N, jb.kind == 0 ? jb.diag + r0 - c0 : TL, acc, gemm_smem);
}

// W = L_rs Y (r x k) with Y lower triangular: tile (ti, tj) of 64 x 64 sums
// t over [64 tj, k) in chunks of KC.
__global__ void __launch_bounds__(GEMM_THREADS) k_wgemm(const double* __restrict__ F, const double* __restrict__ Y,
                                                        double* __restrict__ W, const FrontDesc* __restrict__ desc,
                                                        WorkList wl) {
    extern __shared__ __align__(16) double gemm_smem[];
    const int item = find_item(wl.d_prefix, wl.n, blockIdx.x);
    const FrontDesc d = desc[wl.d_fronts[item]];
    const int t = blockIdx.x - wl.d_prefix[item];
    // column tiles slowest: the tiles with the longest K (c0 = 0) come first in
    // the launch, the short ones fill in behind them
    const int nr = (d.r + TL - 1) / TL;
    const int r0 = (t % nr) * TL, c0 = (t / nr) * TL;
    const int M = min(TL, d.r - r0), N = min(TL, d.k - c0);
    const double* A = F + d.f_off + d.k + r0;   // L_rs(i, t) at A[i + t ld]
    double acc[4][4][2] = {};
    // t over [c0, k): Y(k0 + t, c0 + j) vanishes above the diagonal
    gemm_pipelined<false>(A + (int64_t)c0 * d.ld, d.ld, M, Y + d.y_off + c0 + (int64_t)c0 * d.ldy, d.ldy, N, d.k - c0,
                          gemm_smem, acc);
    tile_store(W + d.y_off + d.k + r0 + (int64_t)c0 * d.ldy, 1, d.ldy, M, N, acc);
}

// ---- solve -----------------------------------------------------------------------
// One launch per direction walks every level of the tree.  The work of a
// direction is one list of items, forward leaves first and backward root first.
// Forward: an item is a band of 64 rows of a front's M = [Y; W] ((k + r) x k,
// leading dimension ldy) times a chunk of its columns (Y rows only up to the
// diagonal): rows < k give z_s = Y t_s, rows >= k give u_s = v_s - W t_s.
// Backward: a band of 64 columns times a chunk of the rows below the diagonal
// and of the W rows: y_s = Y^T z_s - W^T y_rows.
//
// Persistent CTAs take items in list order through an atomic head.  What an
// item reads of other fronts -- forward the children's update entries U,
// backward the ancestors' solution -- it waits for entry by entry: those
// buffers hold the pattern kUnset in every entry not yet written, and a reader
// polls the entry itself until it holds a value.  A value thus crosses from
// its writer to its reader in one store and one load, with no fence, counter
// or flag between them, which is what bounds a system of this kind: a tree
// of ten levels is a chain of ten such hand-overs, each way.  The partial sums
// of a band's chunks are handed to the band's last item the same way and added
// in chunk order, so results do not depend on which CTA takes which item.
// (kUnset, see common.cuh; every value stored in these buffers is the result of
// an arithmetic operation.)
//
// Everything waited for comes from items earlier in the list, which were taken
// by running CTAs, so the earliest unfinished item never waits and the list
// always drains.  Every wait is bounded (kWaitNs, kWaitPolls): one that gives
// up sets *status to WRAPD_E_TIMEOUT and its item is skipped, and waits that
// find *status set return at once.
//
// The buffers are unset again on the way: the forward pass unsets the solution
// buffer, the backward pass U, and a band's last item the partial sums it has
// read; after a failed launch the host refills them (CholGPU::reset_solve).
//
// Measured, us per solve, forward + backward (before: register-staged loads,
// per-front counters raised behind a fence and read by one thread, an arrival
// counter per band, a copy of the right-hand side and a memset per solve):
//   bar          levels  [Y; W]    before          now
//   8x8x32            6    2 MB   25.5 +   21.6   13.8 +   12.0
//   13x11x37          8    7 MB   39.0 +   36.2   23.6 +   22.0
//   16x16x64          9   30 MB   57.4 +   59.2   35.9 +   36.0
//   24x24x48         10   66 MB   92.9 +   84.9   46.8 +   69.4
//   32x32x128        12  490 MB  199.9 +  195.9    133 +    164
//   64x64x160        14  4.5 GB    958 +   1436    957 +   1070   (4.7, 4.2 TB/s)
// The order of every sum is the earlier kernels', so the results are the same
// bit for bit: in mixed precision the rounding of the local step turns a last
// bit here into 1e-8 of the positions within twenty iterations.
constexpr int SCH = 256;              // longest chunk of the streamed dimension
constexpr int SCH_MIN = 64;
constexpr int kSolveItems = 2 * 148;   // items wanted per level (see build and build_queues)
constexpr int kBwdSub = 4;            // narrow backward bands per 64 columns
// Largest [Y; W] of the deep backward ring (see k_bwd_queue).  Us backward, deep and
// not, over compact bars: 564 MB 161, 178; 705 MB 200, 206; 864 MB 261, 235; 1.2 GB 324, 296;
// 2.1 GB 549, 472: they cross at 0.8 GB, so the line is higher than these want it.
constexpr size_t kBwdDeepBytes = (size_t)3 << 29;
// Largest [Y; W] whose items poll their inputs at once (see k_fwd_queue).  Us forward +
// backward, at once and gated: compact bars of 126 MB 139, 145; 208 MB 192, 178; 255 MB 244,
// 184; 363 MB 308, 227; thin bars (4 x 4, 3 x 3) of 218 MB 202, 216; 262 MB 236, 257; batches
// of 50 to 370 MB within 4 % of each other.
constexpr size_t kGateBytes = (size_t)256 << 20;
__device__ __forceinline__ void st_unset3(double* p) {
    st_relaxed(p, unset_value());
    st_relaxed(p + 1, unset_value());
    st_relaxed(p + 2, unset_value());
}

// The rows of three values at p[0 .. N-1] (null: zeros), looked at until all
// of them are set.  False when the wait gave up or the launch had already failed.
template <int N>
__device__ __forceinline__ bool await3(const double* const (&p)[N], double (&v)[N][3], int* status) {
    unsigned long long t0 = 0;
    for (int i = 0;; ++i) {
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int c = 0; c < 3; ++c) v[n][c] = p[n] ? ld_relaxed(p[n] + c) : 0.0;
        bool all = true;
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int c = 0; c < 3; ++c) all = all && !unset(v[n][c]);
        if (all) return true;
        if (!look_again(i, t0, status)) return false;
    }
}

// s <- the sum of row `row`'s partial sums of a band's chunks, in chunk order,
// the last of which is s itself (the caller's); the slots read are unset.
__device__ __forceinline__ bool add_chunks(double* P, int first, int nchunk, int row, double (&s)[3], int* status) {
    constexpr int NB = 6;   // rows looked at together
    double t[3] = {0.0, 0.0, 0.0};
    for (int c = 0; c < nchunk - 1; c += NB) {
        const double* p[NB];
        double v[NB][3];
#pragma unroll
        for (int e = 0; e < NB; ++e) p[e] = c + e < nchunk - 1 ? P + 3 * ((int64_t)(first + c + e) * TL + row) : nullptr;
        if (!await3(p, v, status)) return false;
#pragma unroll
        for (int e = 0; e < NB; ++e)
            if (p[e]) {
                t[0] += v[e][0]; t[1] += v[e][1]; t[2] += v[e][2];
                st_unset3(const_cast<double*>(p[e]));
            }
    }
    s[0] = t[0] + s[0]; s[1] = t[1] + s[1]; s[2] = t[2] + s[2];
    return true;
}

// The CTA's item list position: thread 0 of its last warp takes the ticket of the
// next item and its warp copies that item's record to shared memory while the others
// finish the current one.  Gated items (k_fwd_queue) take it after the gate's wait,
// so that a CTA that waits does not sit on work another could take; the others before
// they poll, which on a small system has CTAs to spare.  Either way a CTA's current
// item comes before the one it holds, so the earliest unfinished item is always
// some CTA's current one.
struct ItemSlot {
    SolveWork it;
    int q;
};
__device__ __forceinline__ void fetch_item(const SolveQueue& Q, int ticket, ItemSlot* slot) {
    const int lane = threadIdx.x & 31;
    const int q = __shfl_sync(0xffffffffu, ticket, 0);
    if (lane == 0) slot->q = q;
    if (q < Q.n && lane < (int)(sizeof(SolveWork) / 16))
        reinterpret_cast<int4*>(&slot->it)[lane] = __ldg(reinterpret_cast<const int4*>(Q.items + q) + lane);
}

// Both directions stream an item's block of [Y; W] through shared memory in
// stages of 16 columns x 64 rows (8 KB) by cp.async, a ring of stages in flight
// per CTA and the first ringful issued before the item's waits ([Y; W] does not
// change during a solve).  Every warp copies exactly the values it will use
// itself, so the stages need no CTA barrier.  Five CTAs of four warps per SM with
// rings of four keep 160 KB in flight per SM, against 128 KB of register loads
// before.  The backward pass has long chunks to stream at every level (a
// front's r rows; forward a chunk is at most the front's k columns), so where a
// level has few items its time is ringfuls: rings of eight with three CTAs per
// SM run it in 19, 64, 168 us on the 8x8x32, 24x24x48, 32x32x128 bars against 30,
// 100, 199 with rings of four and five CTAs, while the 64x64x160 bar has items
// enough and takes 1.14 ms with more CTAs against 1.44 (an earlier form of the
// kernel, 64-column bands throughout).  The line lies between the two last:
// kBwdDeepBytes of [Y; W].
constexpr int SOLVE_WARPS = 4;
constexpr int SOLVE_THREADS = 32 * SOLVE_WARPS;
constexpr int FWD_MINB = 5;           // CTAs per SM
constexpr int FRING = 4;              // stages in flight per CTA
constexpr int ST_C = 16;              // columns of a stage
constexpr int FR = TL;                // doubles per staged column of a warp (4 of the stage's 16 columns)
constexpr int ring_doubles(int stages) { return stages * ST_C * FR; }
constexpr int FWD_RING = ring_doubles(FRING);
constexpr int solve_smem(int stages) { return (ring_doubles(stages) + (SCH + TL) * 3) * (int)sizeof(double); }
static_assert(ST_C % SOLVE_WARPS == 0 && TL == 64 && SOLVE_WARPS == 4, "the warps' shares of a stage");
static_assert(3 * TL <= FRING * (ST_C / SOLVE_WARPS) * FR, "a forward warp's sums reuse its ring");

// Forward: lane l of warp w holds rows b0 + 2l and b0 + 2l + 1 of the band and
// takes columns w, w + 4, ... of the chunk; the warps' sums are added in warp
// order.
__global__ void __launch_bounds__(SOLVE_THREADS, FWD_MINB)
    k_fwd_queue(const double* __restrict__ B, double* __restrict__ Zb, double* __restrict__ Xp, double* U,
                const int* __restrict__ inv, const double* __restrict__ YW, SolveQueue Q, double* P,
                const int* __restrict__ mesh_on) {
    constexpr int NT = SOLVE_THREADS, TPT = SCH / NT, WC = ST_C / SOLVE_WARPS;
    __shared__ __align__(16) ItemSlot slots[2];
    extern __shared__ __align__(16) double ssm[];
    double* tv = ssm + FWD_RING;          // [SCH][3]
    double* vrow = tv + SCH * 3;                 // [TL][3]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    double* ring = ssm + warp * (FRING * WC * FR);
    if (blockIdx.x == 0 && tid == 0) *Q.other_head = 0u;
    if (warp == SOLVE_WARPS - 1) fetch_item(Q, lane == 0 ? (int)atomicAdd(Q.head, 1u) : 0, &slots[0]);
    __syncthreads();
    for (int turn = 0;; turn ^= 1) {
        const int q = slots[turn].q;
        if (q >= Q.n) break;
        const SolveWork& it = slots[turn].it;
        int ticket = 0;
        const bool on = !mesh_on || mesh_on[it.mesh];
        bool ok = true;
        if (on) {
            const int nc = it.hi - it.lo, nst = (nc + ST_C - 1) / ST_C;
            const int64_t ldy = it.ldy;
            const double* M = YW + it.m_off + 2 * lane;
            const bool live = it.b0 + 2 * lane < it.R;
            auto issue = [&](int s) {
                if (s < nst) {
                    double* dst = ring + (s % FRING) * (WC * FR) + 2 * lane;
#pragma unroll
                    for (int u = 0; u < WC; ++u) {
                        const int j = s * ST_C + warp + SOLVE_WARPS * u;
                        const bool v = live && j < nc;
                        cp_async16(dst + u * FR, v ? M + (int64_t)j * ldy : M, v ? 16 : 0);
                    }
                }
                cp_async_commit();
            };
#pragma unroll
            for (int s = 0; s < FRING; ++s) issue(s);
            // the children's entries of the chunk's columns and, in the band's
            // last item, of its rows
            int2 iv[TPT];
            const int2* inv2 = reinterpret_cast<const int2*>(inv) + it.aux;
#pragma unroll
            for (int m = 0; m < TPT; ++m) {
                const int j = tid + m * NT;
                iv[m] = (it.leaf || j >= nc) ? make_int2(-1, -1) : __ldg(inv2 + it.lo + j);
            }
            const bool owner = q == it.first + it.nchunk - 1;
            const int vr = tid - (NT - TL);   // threads NT - TL .. NT - 1: row vr of the band
            int2 ivr = make_int2(-1, -1);
            if (owner && vr >= 0 && it.b0 + vr >= it.k && it.b0 + vr < it.R && !it.leaf) ivr = __ldg(inv2 + it.b0 + vr);
            if (Q.gate && (it.gate0 >= 0 || it.gate1 >= 0)) {
                // a large system: one thread polls until the item's inputs are about
                // there, so that waiting CTAs leave the L2 to the streaming ones; the
                // others poll at once, which saves a round trip per level (forward +
                // backward on the 8x8x32, 16x16x64, 24x24x48, 32x32x128 bars: 31, 72, 103,
                // 313 us polling at once, 35, 81, 115, 309 us gated)
                if (tid == 0) {
                    const double* const p[2] = {it.gate0 >= 0 ? U + 3 * (int64_t)it.gate0 : nullptr,
                                                it.gate1 >= 0 ? U + 3 * (int64_t)it.gate1 : nullptr};
                    double g[2][3];
                    await3(p, g, Q.status);
                }
                __syncthreads();
            }
            if (tid == NT - 32) ticket = (int)atomicAdd(Q.head, 1u);
            {
                const double* p[2 * TPT + 2];
                double c[2 * TPT + 2][3];
#pragma unroll
                for (int m = 0; m < TPT; ++m) {
                    p[2 * m] = iv[m].x >= 0 ? U + 3 * (int64_t)iv[m].x : nullptr;
                    p[2 * m + 1] = iv[m].y >= 0 ? U + 3 * (int64_t)iv[m].y : nullptr;
                }
                p[2 * TPT] = ivr.x >= 0 ? U + 3 * (int64_t)ivr.x : nullptr;
                p[2 * TPT + 1] = ivr.y >= 0 ? U + 3 * (int64_t)ivr.y : nullptr;
                ok = await3(p, c, Q.status);
#pragma unroll
                for (int m = 0; m < TPT; ++m) {
                    const int j = tid + m * NT;
                    double v[3] = {0.0, 0.0, 0.0};
                    if (j < nc && it.lo + j < it.k) {
                        const double* b = B + 3 * ((int64_t)it.col + it.lo + j);
                        v[0] = b[0]; v[1] = b[1]; v[2] = b[2];
                    }
                    if (j < nst * ST_C)
#pragma unroll
                        for (int e = 0; e < 3; ++e) tv[3 * j + e] = v[e] + c[2 * m][e] + c[2 * m + 1][e];
                }
                if (owner && vr >= 0)
#pragma unroll
                    for (int e = 0; e < 3; ++e) vrow[3 * vr + e] = c[2 * TPT][e] + c[2 * TPT + 1][e];
            }
            ok = __syncthreads_and(ok);
            double a0 = 0.0, a1 = 0.0, a2 = 0.0, b0 = 0.0, b1 = 0.0, b2 = 0.0;
            for (int s = 0; s < nst; ++s) {
                cp_async_wait<FRING - 1>();   // own copies only: no barrier
                const double* src = ring + (s % FRING) * (WC * FR) + 2 * lane;
                const double* t = tv + 3 * (s * ST_C + warp);
#pragma unroll
                for (int u = 0; u < WC; ++u) {
                    const double2 m = *reinterpret_cast<const double2*>(src + u * FR);
                    const double t0 = t[12 * u], t1 = t[12 * u + 1], t2 = t[12 * u + 2];
                    a0 = fma(m.x, t0, a0); a1 = fma(m.x, t1, a1); a2 = fma(m.x, t2, a2);
                    b0 = fma(m.y, t0, b0); b1 = fma(m.y, t1, b1); b2 = fma(m.y, t2, b2);
                }
                asm volatile("" ::: "memory");   // the stage is read before it is refilled
                issue(s + FRING);
            }
            cp_async_wait<0>();
            __syncwarp();
            // the warp's sums, in its own ring
            ring[6 * lane] = a0; ring[6 * lane + 1] = a1; ring[6 * lane + 2] = a2;
            ring[6 * lane + 3] = b0; ring[6 * lane + 4] = b1; ring[6 * lane + 5] = b2;
            __syncthreads();
            const int row = tid, i = it.b0 + row;
            if (ok && row < TL && i < it.R) {
                double s[3] = {0.0, 0.0, 0.0};
#pragma unroll
                for (int w = 0; w < SOLVE_WARPS; ++w) {
                    const double* pw = ssm + w * (FRING * WC * FR) + 3 * row;
                    s[0] += pw[0]; s[1] += pw[1]; s[2] += pw[2];
                }
                if (!owner) {
                    double* p = P + 3 * ((int64_t)q * TL + row);
                    st_relaxed(p, s[0]); st_relaxed(p + 1, s[1]); st_relaxed(p + 2, s[2]);
                } else if (it.nchunk == 1 || add_chunks(P, it.first, it.nchunk, row, s, Q.status)) {
                    if (i < it.k) {
                        const int64_t o = 3 * ((int64_t)it.col + i);
                        Zb[o] = s[0]; Zb[o + 1] = s[1]; Zb[o + 2] = s[2];
                        st_unset3(Xp + o);
                    } else if (it.col != Q.hold) {
                        double* u = U + 3 * ((int64_t)it.u_row + i - it.k);
                        st_relaxed(u, vrow[3 * row] - s[0]);
                        st_relaxed(u + 1, vrow[3 * row + 1] - s[1]);
                        st_relaxed(u + 2, vrow[3 * row + 2] - s[2]);
                    }
                }
            }
        } else if (tid == NT - 32) {
            ticket = (int)atomicAdd(Q.head, 1u);
        }
        if (warp == SOLVE_WARPS - 1) fetch_item(Q, ticket, &slots[turn ^ 1]);
        __syncthreads();   // the next record is there; this item's shared memory is free
    }
}

// Backward: warp w takes columns 4 w .. 4 w + 3 of each stage (16 of the band's
// 64 columns, one 64-row block of the chunk; a column group's row blocks follow
// each other).  Lane 8 c + p has column c and row pairs p, p + 8, p + 16, p + 24 of the
// block, a sum for each: the pairs are added as a tree over pair bits 16, 8 (in
// the lane), 4, 2, 1 (across lanes).  The input of row i is z_i for i < k and
// minus the solution at the front's row i - k for i >= k.
template <int BRING, int MINB>
__global__ void __launch_bounds__(SOLVE_THREADS, MINB)
    k_bwd_queue(double* __restrict__ x, const double* __restrict__ Zb, double* Xp, double* __restrict__ U,
                const double* __restrict__ YW, const int* __restrict__ rows, SolveQueue Q, double* P,
                const int* __restrict__ mesh_on) {
    constexpr int NT = SOLVE_THREADS, TPT = SCH / NT, WC = ST_C / SOLVE_WARPS;
    __shared__ __align__(16) ItemSlot slots[2];
    extern __shared__ __align__(16) double ssm[];
    double* in = ssm + BRING * SOLVE_WARPS * WC * FR;   // [SCH][3], zero past the chunk
    double* res = in + SCH * 3;                                // [TL][3]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    double* ring = ssm + warp * (BRING * WC * FR);
    if (blockIdx.x == 0 && tid == 0) *Q.other_head = 0u;
    if (warp == SOLVE_WARPS - 1) fetch_item(Q, lane == 0 ? (int)atomicAdd(Q.head, 1u) : 0, &slots[0]);
    __syncthreads();
    for (int turn = 0;; turn ^= 1) {
        const int q = slots[turn].q;
        if (q >= Q.n) break;
        const SolveWork& it = slots[turn].it;
        int ticket = 0;
        const bool on = !mesh_on || mesh_on[it.mesh];
        bool ok = true;
        if (on) {
            const int nr = it.hi - it.lo, nc = min(it.w, it.k - it.b0);
            const int nrb = (nr + TL - 1) / TL, ng = (nc + ST_C - 1) / ST_C;   // row blocks, column groups
            const int64_t ldy = it.ldy;
            const double* M = YW + it.m_off + 2 * lane + (int64_t)(WC * warp) * ldy;
            // the next stage to copy: its group and row block, its place in the ring
            int ig = 0, irb = 0, is = 0;
            auto issue = [&]() {
                if (ig < ng) {
                    double* dst = ring + is * (WC * FR) + 2 * lane;
                    const double* src = M + irb * TL + (int64_t)(ig * ST_C) * ldy;
                    const bool live = irb * TL + 2 * lane < nr;
#pragma unroll
                    for (int u = 0; u < WC; ++u) {
                        const bool v = live && ig * ST_C + WC * warp + u < nc;
                        cp_async16(dst + u * FR, v ? src + (int64_t)u * ldy : M, v ? 16 : 0);
                    }
                    if (++irb == nrb) { irb = 0; ++ig; }
                    is = is + 1 == BRING ? 0 : is + 1;
                }
                cp_async_commit();
            };
#pragma unroll
            for (int s = 0; s < BRING; ++s) issue();
            const bool owner = q == it.first + it.nchunk - 1;
            int row[TPT];
            double v[TPT][3];
#pragma unroll
            for (int m = 0; m < TPT; ++m) {
                const int t = tid + m * NT, i = it.lo + t;
                row[m] = -1;
                v[m][0] = v[m][1] = v[m][2] = 0.0;
                if (t < nr) {
                    if (i < it.k) {
                        const double* z = Zb + 3 * ((int64_t)it.col + i);
                        v[m][0] = z[0]; v[m][1] = z[1]; v[m][2] = z[2];
                    } else {
                        row[m] = __ldg(rows + it.aux + i - it.k);
                        // the forward pass is done with U: unset it for the next solve
                        if (it.b0 == 0) st_unset3(U + 3 * ((int64_t)it.u_row + i - it.k));
                    }
                }
            }
            if (Q.gate && it.gate0 >= 0) {
                if (tid == 0) {
                    const double* const p[1] = {Xp + 3 * (int64_t)it.gate0};
                    double g[1][3];
                    await3(p, g, Q.status);
                }
                __syncthreads();
            }
            if (tid == NT - 32) ticket = (int)atomicAdd(Q.head, 1u);
            {
                const double* p[TPT];
                double y[TPT][3];
#pragma unroll
                for (int m = 0; m < TPT; ++m) p[m] = row[m] >= 0 ? Xp + 3 * (int64_t)row[m] : nullptr;
                ok = await3(p, y, Q.status);
#pragma unroll
                for (int m = 0; m < TPT; ++m) {
                    const int t = tid + m * NT;
                    if (t < nrb * TL)
#pragma unroll
                        for (int e = 0; e < 3; ++e) in[3 * t + e] = row[m] >= 0 ? -y[m][e] : v[m][e];
                }
            }
            ok = __syncthreads_and(ok);
            const int cl = lane >> 3, pr = lane & 7;
            int cs = 0;   // the stage's place in the ring
            for (int g = 0; g < ng; ++g) {
                double a[4][3];
#pragma unroll
                for (int e = 0; e < 4; ++e) a[e][0] = a[e][1] = a[e][2] = 0.0;
                for (int rb = 0; rb < nrb; ++rb) {
                    cp_async_wait<BRING - 1>();
                    __syncwarp();   // the warp's copies are all there
                    const double* src = ring + cs * (WC * FR) + cl * FR + 2 * pr;
                    const double2* xin = reinterpret_cast<const double2*>(in + 3 * (rb * TL + 2 * pr));
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const double2 m = *reinterpret_cast<const double2*>(src + 16 * e);
                        const double2 x0 = xin[24 * e], x1 = xin[24 * e + 1], x2 = xin[24 * e + 2];   // rows 2l, 2l + 1
                        a[e][0] = fma(m.y, x1.y, fma(m.x, x0.x, a[e][0]));
                        a[e][1] = fma(m.y, x2.x, fma(m.x, x0.y, a[e][1]));
                        a[e][2] = fma(m.y, x2.y, fma(m.x, x1.x, a[e][2]));
                    }
                    cs = cs + 1 == BRING ? 0 : cs + 1;
                    __syncwarp();   // the stage is read
                    issue();
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    double t = (a[0][c] + a[2][c]) + (a[1][c] + a[3][c]);
                    t += __shfl_xor_sync(0xffffffffu, t, 4);
                    t += __shfl_xor_sync(0xffffffffu, t, 2);
                    t += __shfl_xor_sync(0xffffffffu, t, 1);
                    if (pr == 0) res[3 * (g * ST_C + WC * warp + cl) + c] = t;
                }
            }
            __syncthreads();
            const int j = tid;
            if (ok && j < nc) {
                double s[3] = {res[3 * j], res[3 * j + 1], res[3 * j + 2]};
                if (!owner) {
                    double* p = P + 3 * ((int64_t)q * TL + j);
                    st_relaxed(p, s[0]); st_relaxed(p + 1, s[1]); st_relaxed(p + 2, s[2]);
                } else if (it.nchunk == 1 || add_chunks(P, it.first, it.nchunk, j, s, Q.status)) {
                    const int64_t o = 3 * ((int64_t)it.col + it.b0 + j);
                    if (it.col != Q.hold) {
                        st_relaxed(Xp + o, s[0]); st_relaxed(Xp + o + 1, s[1]); st_relaxed(Xp + o + 2, s[2]);
                    }
                    x[o] = s[0]; x[o + 1] = s[1]; x[o + 2] = s[2];
                }
            }
        } else if (tid == NT - 32) {
            ticket = (int)atomicAdd(Q.head, 1u);
        }
        if (warp == SOLVE_WARPS - 1) fetch_item(Q, ticket, &slots[turn ^ 1]);
        __syncthreads();
    }
}

}  // namespace

CholGPU::~CholGPU() {
    if (factor_graph_) cudaGraphExecDestroy(factor_graph_);
    if (solve_graph_) cudaGraphExecDestroy(solve_graph_);
    for (void* p : allocs_) cudaFree(p);
}

void CholGPU::release(void* p) {
    if (!p) return;
    cudaFree(p);
    allocs_.erase(std::remove(allocs_.begin(), allocs_.end(), p), allocs_.end());
}

template <typename X>
X* CholGPU::upload(const std::vector<X>& v, cudaStream_t st) {
    X* p = nullptr;
    const size_t bytes = std::max<size_t>(1, v.size()) * sizeof(X);
    if (cudaMalloc(&p, bytes) != cudaSuccess) { cudaGetLastError(); throw CudaError(WRAPD_E_OOM, "cudaMalloc failed (factor structures)"); }
    allocs_.push_back(p);
    device_bytes += bytes;
    if (!v.empty()) WRAPD_CUDA(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(X), cudaMemcpyHostToDevice, st));
    return p;
}

JobList CholGPU::make_jobs(const std::vector<GemmJob>& jobs, cudaStream_t st) {
    JobList l;
    std::vector<GemmJob> keep;
    std::vector<int> pre(1, 0);
    for (const GemmJob& jb : jobs) {
        const int Tr = ceil_div(jb.rows, TL), Tc = ceil_div(jb.cols, TL);
        if (Tr <= 0 || Tc <= 0 || jb.K <= 0) continue;
        int tiles = 0;
        if (jb.kind == 1) tiles = Tr * Tc;
        else for (int tj = 0; tj < Tc; ++tj) tiles += std::max(0, Tr - tj);
        if (tiles <= 0) continue;
        keep.push_back(jb);
        pre.push_back(pre.back() + tiles);
    }
    l.n = static_cast<int>(keep.size());
    l.total = pre.back();
    if (l.n == 0) return l;
    l.d_jobs = upload(keep, st);
    l.d_prefix = upload(pre, st);
    return l;
}

WorkList CholGPU::make_list(const std::vector<int>& fronts, const std::vector<int>& ctas, cudaStream_t st) {
    WorkList w;
    std::vector<int> f, pre(1, 0);
    for (size_t i = 0; i < fronts.size(); ++i)
        if (ctas[i] > 0) { f.push_back(fronts[i]); pre.push_back(pre.back() + ctas[i]); }
    w.n = static_cast<int>(f.size());
    w.total = pre.back();
    if (w.n == 0) return w;
    w.d_fronts = upload(f, st);
    w.d_prefix = upload(pre, st);
    return w;
}

void CholGPU::build(const Symbolic& S, const std::vector<int64_t>& A_pos, const std::vector<int>& A_ptr,
                    const std::vector<int>& A_contrib, cudaStream_t st) {
    WRAPD_CUDA(cudaFuncSetAttribute(k_update, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM));
    WRAPD_CUDA(cudaFuncSetAttribute(k_wgemm, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM));
    WRAPD_CUDA(cudaFuncSetAttribute(k_fwd_queue, cudaFuncAttributeMaxDynamicSharedMemorySize, solve_smem(FRING)));
    // deep rings for latency, or more CTAs per SM for throughput (see k_bwd_queue)
    const size_t yw_bytes = (size_t)S.y_pool * sizeof(double);
    bwd_smem_ = yw_bytes <= kBwdDeepBytes ? solve_smem(8) : solve_smem(4);
    bwd_fn_ = yw_bytes <= kBwdDeepBytes ? k_bwd_queue<8, 3> : k_bwd_queue<4, 5>;
    solve_gate_ = yw_bytes > kGateBytes;
    WRAPD_CUDA(cudaFuncSetAttribute(bwd_fn_, cudaFuncAttributeMaxDynamicSharedMemorySize, bwd_smem_));
    n = S.n;
    nfronts = static_cast<int>(S.fronts.size());
    nlevels = static_cast<int>(S.levels.size());
    nnz_L = S.nnz_L;
    flops = S.flops;
    if (S.max_children > 2) throw CudaError(WRAPD_E_INPUT, "assembly tree with more than 2 children");
    h_desc_.resize(nfronts);
    std::vector<int> rows;
    int64_t roff = 0, ioff = 0;
    for (int f = 0; f < nfronts; ++f) {
        const Front& F = S.fronts[f];
        FrontDesc& d = h_desc_[f];
        d.first = F.first; d.k = F.ncols; d.r = F.nrows(); d.ld = F.ld();
        d.f_off = F.f_off; d.y_off = F.y_off; d.u_off = F.u_off;
        d.rows_off = roff;
        rows.insert(rows.end(), F.rows.begin(), F.rows.end());
        roff += F.nrows();
        d.inv_off = ioff; ioff += 2 * ((int64_t)d.k + d.r);
        d.nchild = static_cast<int>(F.children.size());
        d.child0 = d.nchild > 0 ? F.children[0] : -1;
        d.child1 = d.nchild > 1 ? F.children[1] : -1;
        d.ldy = static_cast<int>(yw_ld(d.k, d.r));
        d.mesh = front_mesh.empty() ? 0 : front_mesh[f];
    }
    if (S.u_pool / 3 > INT32_MAX) throw CudaError(WRAPD_E_INPUT, "solve update vectors exceed 32-bit row indexes");
    h_inv_.assign(ioff, -1);
    for (int f = 0; f < nfronts; ++f) {
        const Front& F = S.fronts[f];
        for (size_t q = 0; q < F.children.size(); ++q) {
            const Front& C = S.fronts[F.children[q]];
            for (int i = 0; i < C.nrows(); ++i)
                h_inv_[h_desc_[f].inv_off + 2 * (int64_t)S.relmap[C.rel_off + i] + (int64_t)q] =
                    static_cast<int>(C.u_off / 3) + i;
        }
    }
    d_inv_ = upload(h_inv_, st);
    h_rows_ = rows;
    d_desc_ = upload(h_desc_, st);
    d_rows_ = upload(rows, st);
    // A's entries by front column: entry t's place, and each place's row in the
    // front (a counting sort over the columns; the order within a column, which
    // nothing depends on, is left to the atomics)
    nA_ = static_cast<int>(A_pos.size());
    {
        int64_t* pos = upload(A_pos, st);
        int* cnt = upload(std::vector<int>(n, 0), st);
        d_Aslot_ = upload(std::vector<int>(nA_), st);
        d_Arow_ = upload(std::vector<int>(nA_), st);
        std::vector<int> ptr(n + 1, 0);
        if (nA_ > 0) k_A_places<<<ceil_div(nA_, 256), 256, 0, st>>>(nA_, pos, d_desc_, nfronts, nullptr, cnt, nullptr, nullptr);
        WRAPD_LAUNCH_CHECK();
        WRAPD_CUDA(cudaMemcpyAsync(ptr.data() + 1, cnt, n * sizeof(int), cudaMemcpyDeviceToHost, st));
        WRAPD_CUDA(cudaMemsetAsync(cnt, 0, n * sizeof(int), st));
        WRAPD_CUDA(cudaStreamSynchronize(st));
        for (int c = 0; c < n; ++c) ptr[c + 1] += ptr[c];
        d_Acol_ = upload(ptr, st);
        if (nA_ > 0) k_A_places<<<ceil_div(nA_, 256), 256, 0, st>>>(nA_, pos, d_desc_, nfronts, d_Acol_, cnt, d_Aslot_, d_Arow_);
        WRAPD_LAUNCH_CHECK();
        WRAPD_CUDA(cudaStreamSynchronize(st));
        release(pos);
        release(cnt);
        device_bytes -= A_pos.size() * sizeof(int64_t) + n * sizeof(int);
    }
    d_Aptr_ = upload(A_ptr, st);
    d_Acon_ = upload(A_contrib, st);
    f_pool_ = S.f_pool; y_pool_ = S.y_pool; u_pool_ = S.u_pool;
    auto dalloc = [&](size_t count) {
        double* p = nullptr;
        if (cudaMalloc(&p, std::max<size_t>(1, count) * sizeof(double)) != cudaSuccess) {
            cudaGetLastError();
            throw CudaError(WRAPD_E_OOM, "cudaMalloc failed (factor pools)");
        }
        allocs_.push_back(p);
        device_bytes += std::max<size_t>(1, count) * sizeof(double);
        return p;
    };
    d_Aval_ = dalloc(nA_);
    d_F_ = dalloc(f_pool_);
    d_Y_ = dalloc(y_pool_);
    // the padding rows of [Y; W] stay zero; a factorization writes all the rest
    WRAPD_CUDA(cudaMemsetAsync(d_Y_, 0, y_pool_ * sizeof(double), st));
    d_U_ = dalloc(u_pool_);
    d_Xp_ = dalloc(3 * (size_t)n);
    d_Z_ = dalloc(3 * (size_t)n);
    int* st_ptr = nullptr;
    WRAPD_CUDA(cudaMalloc(&st_ptr, sizeof(int)));
    allocs_.push_back(st_ptr);
    d_status = st_ptr;
    WRAPD_CUDA(cudaMemsetAsync(d_status, 0, sizeof(int), st));

    {
        std::vector<int> all(nfronts), cnt(nfronts);
        for (int f = 0; f < nfronts; ++f) { all[f] = f; cnt[f] = ceil_div(h_desc_[f].k, COLS_PER_CTA); }
        y_cols_ = make_list(all, cnt, st);
    }
    levels_.assign(nlevels, Level());
    fused_ctas_ = kFusedPanelCtas;
    for (int l = 0; l < nlevels; ++l) {
        Level& L = levels_[l];
        L.fronts_sorted = S.levels[l];
        std::stable_sort(L.fronts_sorted.begin(), L.fronts_sorted.end(),
                         [&](int a, int b) { return h_desc_[a].k > h_desc_[b].k; });
        const auto& fs = L.fronts_sorted;
        L.kmax = fs.empty() ? 0 : h_desc_[fs[0]].k;
        std::vector<int> cnt(fs.size());
        for (size_t i = 0; i < fs.size(); ++i)
            cnt[i] = ceil_div(h_desc_[fs[i]].k + h_desc_[fs[i]].r, COLS_PER_CTA);
        L.assemble = make_list(fs, cnt, st);
        const int steps = ceil_div(L.kmax, NB);
        for (int p = 0; p < steps; ++p) {
            std::vector<int> act, ct, nP;
            std::vector<GemmJob> jobs;
            for (int f : fs) {
                const FrontDesc& d = h_desc_[f];
                const int p0 = p * NB;
                if (d.k <= p0) continue;
                const int nb = std::min(NB, d.k - p0), j0 = p0 + nb;
                const int m = d.ld - j0;
                const int bs = (p0 / OB) * OB, be = std::min(d.k, bs + OB);
                act.push_back(f);
                nP.push_back(ceil_div(m, TL));
                ct.push_back(ceil_div(m, TL) + ceil_div(p0, TL));
                // F[r0:r1, c0:c1] -= F[r0:r1, k0:k1] F[c0:c1, k0:k1]^T, and
                // Y[r0:r1, c0:c1] -= F[r0:r1, k0:k1] Y[k0:k1, c0:c1]
                auto f_job = [&](int r0, int r1, int c0, int c1, int k0, int k1) {
                    jobs.push_back(GemmJob{d.f_off + r0 + (int64_t)k0 * d.ld, d.f_off + c0 + (int64_t)k0 * d.ld,
                                           d.f_off + r0 + (int64_t)c0 * d.ld, d.ld, d.ld, r1 - r0, c1 - c0, k1 - k0, 0,
                                           r0 - c0, 0});
                };
                auto y_job = [&](int r0, int r1, int c0, int c1, int k0, int k1) {
                    jobs.push_back(GemmJob{d.f_off + r0 + (int64_t)k0 * d.ld, d.y_off + k0 + (int64_t)c0 * d.ldy,
                                           d.y_off + r0 + (int64_t)c0 * d.ldy, d.ld, d.ldy, r1 - r0, c1 - c0, k1 - k0, 1,
                                           0, 0});
                };
                if (j0 < be) {
                    // inside the outer block: only the block's remaining columns, K = this panel
                    f_job(j0, d.ld, j0, be, p0, j0);
                    y_job(j0, be, 0, j0, p0, j0);
                } else {
                    // the block's last panel: the deferred trailing update, K = the whole block
                    f_job(be, d.ld, be, d.ld, bs, be);
                    y_job(be, d.k, 0, be, bs, be);
                }
            }
            // every active front gets at least one item (its diagonal block is factored there)
            for (int& c : ct) c = std::max(c, 1);
            // both forms of the step are kept; factor_launches picks one by the step's size
            L.diag.push_back(make_list(act, std::vector<int>(act.size(), 1), st));
            L.trsm.push_back(make_list(act, ct, st));
            L.trsm_split.push_back(nP);
            L.update.push_back(make_jobs(jobs, st));
        }
        std::vector<int> wg(fs.size());
        for (size_t q = 0; q < fs.size(); ++q) {
            const FrontDesc& d = h_desc_[fs[q]];
            wg[q] = ceil_div(d.r, TL) * ceil_div(d.k, TL);
        }
        // Solve items with chunks of sch_of(front) (<= SCH) along the streamed dimension.
        auto fwd_items = [&](auto sch_of, std::vector<SolveItem>& fwd) {
            fwd.clear();
            for (int f : fs) {
                const int sch = sch_of(f);
                const FrontDesc& d = h_desc_[f];
                const int R = d.k + d.r;
                // forward: row bands; Y bands use columns up to their last row
                for (int b0 = 0; b0 < R; b0 += TL) {
                    const int cend = b0 < d.k ? std::min(d.k, b0 + TL) : d.k;
                    const int nch = ceil_div(cend, sch), first = static_cast<int>(fwd.size());
                    for (int c = 0; c < nch; ++c)
                        fwd.push_back({f, b0, c * sch, std::min(cend, (c + 1) * sch), nch, first});
                }
            }
        };
        auto bwd_items = [&](auto sch_of, std::vector<SolveItem>& bwd) {
            bwd.clear();
            for (int f : fs) {
                const int sch = sch_of(f);
                const FrontDesc& d = h_desc_[f];
                const int R = d.k + d.r;
                // backward: column bands over rows [b0, R) (Y rows below the band, then the W rows)
                for (int b0 = 0; b0 < d.k; b0 += TL) {
                    const int nch = ceil_div(R - b0, sch), first = static_cast<int>(bwd.size());
                    for (int lo = b0; lo < R; lo += sch) bwd.push_back({f, b0, lo, std::min(R, lo + sch), nch, first});
                }
            }
        };
        // Candidate chunk lengths SCH, SCH/2, ..., SCH_MIN.  The fixed rule takes
        // chunks as long as possible (fewer partial sums to hand over) while the
        // level still has kSolveItems items: the levels near the root of a large
        // system hold a few large fronts, and long chunks there leave most SMs
        // idle.  When not even the shortest chunks give that many (a small system)
        // the longest are kept.  The chunks alone decide the order in which a sum
        // is added, so that they are the same for a mesh of a batch as for the mesh
        // alone.  autotune() may pick another candidate by timing.
        std::vector<SolveItem> fwd, bwd;
        L.cfwd = -1;
        L.cbwd = -1;
        // per mesh of a batch: its item counts for each candidate (the rule
        // below applied to the mesh alone)
        const int nmesh = front_mesh.empty() ? 1 : 1 + *std::max_element(front_mesh.begin(), front_mesh.end());
        std::vector<std::vector<int>> mfwd(nmesh), mbwd(nmesh);
        for (int sch = SCH, c = 0; sch >= SCH_MIN; sch /= 2, ++c) {
            fwd_items([&](int) { return sch; }, fwd);
            bwd_items([&](int) { return sch; }, bwd);
            L.cand.push_back({sch, fwd, bwd});
            if (L.cfwd < 0 && (int)fwd.size() >= kSolveItems) L.cfwd = c;
            if (L.cbwd < 0 && (int)bwd.size() >= kSolveItems) L.cbwd = c;
            if (nmesh > 1) {
                for (int m = 0; m < nmesh; ++m) { mfwd[m].push_back(0); mbwd[m].push_back(0); }
                for (const SolveItem& it : fwd) mfwd[front_mesh[it.front]][c]++;
                for (const SolveItem& it : bwd) mbwd[front_mesh[it.front]][c]++;
            }
        }
        if (L.cfwd < 0) L.cfwd = 0;
        if (L.cbwd < 0) L.cbwd = 0;
        if (nmesh > 1) {
            // a batch: every front takes its own mesh's choice
            std::vector<int> sf(nmesh, SCH), sb(nmesh, SCH);
            for (int m = 0; m < nmesh; ++m) {
                int cf = -1, cb = -1;
                for (int c = 0; c < (int)mfwd[m].size(); ++c) {
                    if (cf < 0 && mfwd[m][c] >= kSolveItems) cf = c;
                    if (cb < 0 && mbwd[m][c] >= kSolveItems) cb = c;
                }
                sf[m] = SCH >> std::max(cf, 0);
                sb[m] = SCH >> std::max(cb, 0);
            }
            fwd_items([&](int f) { return sf[front_mesh[f]]; }, fwd);
            bwd_items([&](int f) { return sb[front_mesh[f]]; }, bwd);
            L.cand.push_back({0, fwd, bwd});
            L.cfwd = L.cbwd = static_cast<int>(L.cand.size()) - 1;
        }
        L.wgemm = make_list(fs, wg, st);
    }
    trsm_nP_.clear();
    for (auto& L : levels_) {
        std::vector<int*> w;
        for (auto& nP : L.trsm_split) w.push_back(nP.empty() ? nullptr : upload(nP, st));
        trsm_nP_.push_back(w);
    }
    count_launches();
    d_heads_ = upload(std::vector<unsigned>(2, 0u), st);
    {
        int dev = 0, sms = 0, bf = 0, bb = 0;
        WRAPD_CUDA(cudaGetDevice(&dev));
        WRAPD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        WRAPD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bf, k_fwd_queue, SOLVE_THREADS, solve_smem(FRING)));
        WRAPD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bb, bwd_fn_, SOLVE_THREADS, bwd_smem_));
        qgrid_f_ = std::max(1, bf) * sms;
        qgrid_b_ = std::max(1, bb) * sms;
    }
    build_queues(st);
    WRAPD_CUDA(cudaStreamSynchronize(st));
}

// The chosen candidate of every level, concatenated: forward leaves first,
// backward root first, each item with the front's numbers it needs and the
// entries its first poll looks at: the last of its inputs that each child
// writes (forward), the nearest ancestor's (backward).  Every index of an item is
// checked against its buffer here; the entries of inv and rows that the kernels
// look up are the symbolic analysis'.
void CholGPU::build_queues(cudaStream_t st) {
    std::vector<SolveWork> qf, qb;
    auto work = [&](const SolveItem& g, int first) {
        const FrontDesc& d = h_desc_[g.front];
        SolveWork w{};
        w.ldy = d.ldy; w.k = d.k; w.R = d.k + d.r; w.col = d.first;
        w.b0 = g.b0; w.lo = g.lo; w.hi = g.hi; w.nchunk = g.nchunk; w.w = TL;
        w.first = first; w.gate0 = w.gate1 = -1; w.mesh = d.mesh;
        w.u_row = static_cast<int>(d.u_off / 3);
        w.leaf = d.child0 < 0 && d.child1 < 0;
        return w;
    };
    for (int l = 0; l < nlevels; ++l) {
        const Level& L = levels_[l];
        if (L.cand.empty()) continue;
        const int base = static_cast<int>(qf.size());
        for (const SolveItem& g : L.cand[L.cfwd].fwd) {
            const FrontDesc& d = h_desc_[g.front];
            SolveWork w = work(g, base + g.first);
            w.m_off = d.y_off + g.b0 + (int64_t)g.lo * d.ldy;
            w.aux = d.inv_off / 2;
            for (int i = g.hi - 1; i >= g.lo && !w.leaf && (w.gate0 < 0 || w.gate1 < 0); --i) {
                if (w.gate0 < 0) w.gate0 = h_inv_[d.inv_off + 2 * (int64_t)i];
                if (w.gate1 < 0) w.gate1 = h_inv_[d.inv_off + 2 * (int64_t)i + 1];
            }
            qf.push_back(w);
        }
    }
    for (int l = nlevels - 1; l >= 0; --l) {
        const Level& L = levels_[l];
        if (L.cand.empty()) continue;
        const std::vector<SolveItem>& items = L.cand[L.cbwd].bwd;
        // A level with few items works on bands of 16 columns, four times the items
        // (a column's sum does not depend on its band's width): backward, 8x8x32,
        // 13x11x37, 16x16x64, 24x24x48 and 32x32x128 bars, 12, 22, 36, 69, 164 us
        // against 19, 33, 62, 80, 175 with bands of 64 (32: 14, 25, 45, 71, 165).
        // With the line at twice kSolveItems: 12, 22, 36, 84, 216.
        const int nsub = (int)items.size() < kSolveItems ? kBwdSub : 1, wd = TL / nsub;
        for (size_t i = 0; i < items.size();) {
            const int nch = items[i].nchunk;
            for (int sub = 0; sub < nsub; ++sub) {
                const int first = static_cast<int>(qb.size());
                for (int c = 0; c < nch; ++c) {
                    const SolveItem& g = items[i + c];
                    const FrontDesc& d = h_desc_[g.front];
                    if (g.b0 + sub * wd >= d.k) break;
                    SolveWork w = work(g, first);
                    w.b0 = g.b0 + sub * wd;
                    w.w = wd;
                    w.m_off = d.y_off + g.lo + (int64_t)w.b0 * d.ldy;
                    w.aux = d.rows_off;
                    if (g.hi > d.k) w.gate0 = h_rows_[d.rows_off + std::max(g.lo, d.k) - d.k];
                    qb.push_back(w);
                }
            }
            i += nch;
        }
    }
    auto check = [&](const std::vector<SolveWork>& q, bool fwd) {
        if (q.size() > (size_t)INT32_MAX / (3 * TL)) throw CudaError(WRAPD_E_INPUT, "solve queue too long");
        const int64_t gmax = fwd ? u_pool_ / 3 : n;
        for (size_t i = 0; i < q.size(); ++i) {
            const SolveWork& g = q[i];
            const int64_t last = fwd ? g.m_off + std::min(g.w, g.R - g.b0) - 1 + (int64_t)(g.hi - g.lo - 1) * g.ldy
                                     : g.m_off + (g.hi - g.lo) - 1 + (int64_t)(std::min(g.w, g.k - g.b0) - 1) * g.ldy;
            const bool ok = g.nchunk >= 1 && g.first >= 0 && g.first <= (int)i && (int)i < g.first + g.nchunk &&
                            (int64_t)g.first + g.nchunk <= (int64_t)q.size() && g.lo >= 0 && g.lo < g.hi &&
                            g.hi - g.lo <= SCH && (fwd ? g.hi <= g.k && g.b0 < g.R : g.hi <= g.R && g.b0 < g.k) &&
                            g.m_off >= 0 && last < y_pool_ && (g.m_off & 1) == 0 && (g.ldy & 1) == 0 &&
                            g.gate0 < gmax && g.gate1 < gmax && g.col >= 0 && g.col + g.k <= n &&
                            (int64_t)g.u_row + (g.R - g.k) <= u_pool_ / 3;
            if (!ok) throw CudaError(WRAPD_E_INPUT, "solve queue item out of range");
        }
    };
    check(qf, true);
    check(qb, false);
    // (the buffers grow when the autotuner tries a choice with more items)
    WRAPD_CUDA(cudaStreamSynchronize(st));
    auto grow = [&](auto*& p, int64_t& cap, int64_t want, size_t bytes) {
        if (want <= cap) return;
        release(p);
        device_bytes -= (size_t)cap * bytes;
        p = nullptr;
        cap = 0;
        void* q = nullptr;
        if (cudaMalloc(&q, (size_t)want * bytes) != cudaSuccess) {
            cudaGetLastError();
            throw CudaError(WRAPD_E_OOM, "cudaMalloc failed (solve queues)");
        }
        allocs_.push_back(q);
        p = static_cast<std::remove_reference_t<decltype(p)>>(q);
        cap = want;
        device_bytes += (size_t)cap * bytes;
    };
    grow(d_qf_, qcap_f_, static_cast<int64_t>(qf.size()), sizeof(SolveWork));
    grow(d_qb_, qcap_b_, static_cast<int64_t>(qb.size()), sizeof(SolveWork));
    grow(d_P_, solve_parts_, static_cast<int64_t>(std::max(qf.size(), qb.size())), 3 * TL * sizeof(double));
    reset_solve();
    nqf_ = static_cast<int>(qf.size());
    nqb_ = static_cast<int>(qb.size());
    if (!qf.empty()) WRAPD_CUDA(cudaMemcpyAsync(d_qf_, qf.data(), qf.size() * sizeof(SolveWork), cudaMemcpyHostToDevice, st));
    if (!qb.empty()) WRAPD_CUDA(cudaMemcpyAsync(d_qb_, qb.data(), qb.size() * sizeof(SolveWork), cudaMemcpyHostToDevice, st));
    WRAPD_CUDA(cudaStreamSynchronize(st));   // the host vectors go out of scope
    if (solve_graph_) { cudaGraphExecDestroy(solve_graph_); solve_graph_ = nullptr; }
}

// The state that a solve starts from and leaves behind: every hand-over entry
// unset, both queue heads 0.  Every launch of the queues goes through here first.
void CholGPU::ready_solve(cudaStream_t st) {
    if (!solve_stale_) return;
    unset_fill(d_U_, u_pool_, st);
    unset_fill(d_Xp_, 3 * (int64_t)n, st);
    unset_fill(d_P_, 3 * TL * solve_parts_, st);
    WRAPD_CUDA(cudaMemsetAsync(d_heads_, 0, 2 * sizeof(unsigned), st));
    solve_stale_ = false;
}

void CholGPU::count_launches() {
    launches_factor = 2;   // A's values + identity
    launches_solve = 2;    // the two queue launches
    for (const Level& L : levels_) {
        launches_factor += L.assemble.total ? 1 : 0;
        for (size_t p = 0; p < L.trsm.size(); ++p) {
            if (L.trsm[p].total > fused_ctas_) launches_factor += L.diag[p].n ? 1 : 0;
            launches_factor += (L.trsm[p].total ? 1 : 0) + (L.update[p].total ? 1 : 0);
        }
        launches_factor += L.wgemm.total ? 1 : 0;
    }
}

std::vector<int> CholGPU::tuning() const {
    std::vector<int> t{fused_ctas_, nlevels};
    for (const Level& L : levels_) t.push_back(L.cand.empty() ? 0 : L.cand[L.cfwd].sch);
    for (const Level& L : levels_) t.push_back(L.cand.empty() ? 0 : L.cand[L.cbwd].sch);
    return t;
}

// Each candidate is timed by CUDA events on the handle's stream: one whole
// factorization launched directly (after one untimed at the fixed rule), or,
// level by level, the solves (the mean of three after one untimed) with that
// candidate on the level and the choices so far on the others.  The solves run
// on a scratch vector; the factorizations on the current weights, so the
// factor is valid afterwards whatever the choice.
void CholGPU::autotune(const double* d_w2, const double* d_Di, int ne, cudaStream_t st) {
    struct Scratch {   // freed on every path
        double* x = nullptr;
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        ~Scratch() {
            if (x) cudaFree(x);
            if (e0) cudaEventDestroy(e0);
            if (e1) cudaEventDestroy(e1);
        }
    } s;
    WRAPD_CUDA(cudaEventCreate(&s.e0));
    WRAPD_CUDA(cudaEventCreate(&s.e1));
    auto timed = [&](int reps, auto&& launch) {
        launch();
        WRAPD_CUDA(cudaEventRecord(s.e0, st));
        for (int r = 0; r < reps; ++r) launch();
        WRAPD_CUDA(cudaEventRecord(s.e1, st));
        WRAPD_CUDA(cudaEventSynchronize(s.e1));
        float ms = 0.f;
        WRAPD_CUDA(cudaEventElapsedTime(&ms, s.e0, s.e1));
        return ms / reps;
    };
    const int candidates[] = {0, kNumSMs, kFusedPanelCtas, 4 * kFusedPanelCtas, 1 << 30};
    float best = 1e30f;
    int pick = kFusedPanelCtas;
    fused_ctas_ = kFusedPanelCtas;
    factor_launches(d_w2, d_Di, ne, st);   // untimed first run
    for (int c : candidates) {
        fused_ctas_ = c;
        const float t = timed(1, [&] { factor_launches(d_w2, d_Di, ne, st); });
        if (t < best) { best = t; pick = c; }
    }
    fused_ctas_ = pick;
    count_launches();
    WRAPD_CUDA(cudaMemsetAsync(d_status, 0, sizeof(int), st));
    // (a batch keeps its per-mesh chunk lengths: a mesh's solve stays its own)
    if (front_mesh.empty()) {
        const size_t bytes = 3 * (size_t)n * sizeof(double);
        if (cudaMalloc(&s.x, bytes) != cudaSuccess) {
            cudaGetLastError();
            throw CudaError(WRAPD_E_OOM, "cudaMalloc failed (autotuner)");
        }
        WRAPD_CUDA(cudaMemsetAsync(s.x, 0, bytes, st));
        for (Level& L : levels_) {
            for (int* choice : {&L.cfwd, &L.cbwd}) {
                float best_t = 1e30f;
                int best_c = *choice;
                for (int c = 0; c < (int)L.cand.size(); ++c) {
                    *choice = c;
                    build_queues(st);
                    const float t = timed(3, [&] {   // (the untimed launch finds the buffers unset)
                        ready_solve(st);
                        solve_launches(s.x, st, nullptr);
                    });
                    if (t < best_t) { best_t = t; best_c = c; }
                }
                *choice = best_c;
            }
        }
        build_queues(st);
    }
    WRAPD_CUDA(cudaMemsetAsync(d_status, 0, sizeof(int), st));
    reset_solve();
    WRAPD_CUDA(cudaStreamSynchronize(st));
}

void CholGPU::factor_launches(const double* d_w2, const double* d_Di, int ne, cudaStream_t st) {
    if (nA_ > 0) {
        k_assemble_A<<<ceil_div(nA_, 256), 256, 0, st>>>(d_Aval_, d_Aslot_, d_Aptr_, d_Acon_, nA_, d_w2, d_Di, ne);
        WRAPD_LAUNCH_CHECK();
    }
    k_y_identity<<<y_cols_.total, 32 * COLS_PER_CTA, 0, st>>>(d_Y_, d_desc_, y_cols_);
    WRAPD_LAUNCH_CHECK();
    for (int l = 0; l < nlevels; ++l) {
        Level& L = levels_[l];
        if (L.assemble.total) {
            k_assemble_front<<<L.assemble.total, 32 * COLS_PER_CTA, 0, st>>>(d_F_, d_desc_, d_inv_, d_Aval_, d_Acol_,
                                                                             d_Arow_, L.assemble);
            WRAPD_LAUNCH_CHECK();
        }
        for (size_t p = 0; p < L.trsm.size(); ++p) {
            if (L.trsm[p].total <= fused_ctas_) {
                if (L.trsm[p].total) {
                    k_panel<<<L.trsm[p].total, CHOL_THREADS, 0, st>>>(d_F_, d_Y_, d_desc_, L.trsm[p],
                                                                      trsm_nP_[l][p], (int)p, d_status);
                    WRAPD_LAUNCH_CHECK();
                }
            } else {
                if (L.diag[p].n) {
                    k_diag<<<L.diag[p].n, CHOL_THREADS, 0, st>>>(d_F_, d_Y_, d_desc_, L.diag[p], (int)p, d_status);
                    WRAPD_LAUNCH_CHECK();
                }
                if (L.trsm[p].total) {
                    k_trsm<<<L.trsm[p].total, GEMM_THREADS, 0, st>>>(d_F_, d_Y_, d_desc_, L.trsm[p],
                                                                     trsm_nP_[l][p], (int)p);
                    WRAPD_LAUNCH_CHECK();
                }
            }
            if (L.update[p].total) {
                k_update<<<L.update[p].total, GEMM_THREADS, GEMM_SMEM, st>>>(d_F_, d_Y_, L.update[p]);
                WRAPD_LAUNCH_CHECK();
            }
        }
        if (L.wgemm.total) {
            k_wgemm<<<L.wgemm.total, GEMM_THREADS, GEMM_SMEM, st>>>(d_F_, d_Y_, d_Y_, d_desc_, L.wgemm);
            WRAPD_LAUNCH_CHECK();
        }
    }
}

void CholGPU::factor(const double* d_w2, const double* d_Di, int ne, cudaStream_t st) {
    if (!use_graphs) { factor_launches(d_w2, d_Di, ne, st); return; }
    if (!factor_graph_) {
        cudaGraph_t g;
        WRAPD_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        try {
            factor_launches(d_w2, d_Di, ne, st);
        } catch (...) {
            cudaStreamEndCapture(st, &g);
            throw;
        }
        WRAPD_CUDA(cudaStreamEndCapture(st, &g));
        WRAPD_CUDA(cudaGraphInstantiate(&factor_graph_, g, 0));
        cudaGraphDestroy(g);
    }
    WRAPD_CUDA(cudaGraphLaunch(factor_graph_, st));
}

void CholGPU::solve_launches(double* d_x, cudaStream_t st, const int* mesh_on, int hold) {
    // on buffers that are not unset the waits would take what they hold for values
    if (solve_stale_) throw CudaError(WRAPD_E_STATE, "triangular solve on hand-over buffers that are not unset");
    const int hold_col = hold < 0 ? -1 : h_desc_[hold].first;
    if (nqf_ > 0) {
        const SolveQueue Q{d_qf_, nqf_, d_heads_, d_heads_ + 1, d_status, hold_col, solve_gate_};
        k_fwd_queue<<<std::min(qgrid_f_, nqf_), SOLVE_THREADS, solve_smem(FRING), st>>>(d_x, d_Z_, d_Xp_, d_U_, d_inv_, d_Y_, Q,
                                                                               d_P_, mesh_on);
        WRAPD_LAUNCH_CHECK();
    }
    if (nqb_ > 0) {
        const SolveQueue Q{d_qb_, nqb_, d_heads_ + 1, d_heads_, d_status, hold_col, solve_gate_};
        bwd_fn_<<<std::min(qgrid_b_, nqb_), SOLVE_THREADS, bwd_smem_, st>>>(d_x, d_Z_, d_Xp_, d_U_, d_Y_, d_rows_, Q,
                                                                               d_P_, mesh_on);
        WRAPD_LAUNCH_CHECK();
    }
}

void CholGPU::solve_holding(double* d_x, int hold, cudaStream_t st) {
    if (hold < 0 || hold >= nfronts) throw CudaError(WRAPD_E_INPUT, "front index out of range");
    ready_solve(st);
    solve_launches(d_x, st, nullptr, hold);
    solve_stale_ = true;
}

void CholGPU::solve(double* d_x, cudaStream_t st, const int* mesh_on) {
    ready_solve(st);
    if (!use_graphs) { solve_launches(d_x, st, mesh_on); return; }
    if (!solve_graph_ || solve_graph_x_ != d_x || solve_graph_mask_ != mesh_on) {
        if (solve_graph_) { cudaGraphExecDestroy(solve_graph_); solve_graph_ = nullptr; }
        cudaGraph_t g;
        WRAPD_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        try {
            solve_launches(d_x, st, mesh_on);
        } catch (...) {
            cudaStreamEndCapture(st, &g);
            throw;
        }
        WRAPD_CUDA(cudaStreamEndCapture(st, &g));
        WRAPD_CUDA(cudaGraphInstantiate(&solve_graph_, g, 0));
        cudaGraphDestroy(g);
        solve_graph_x_ = d_x;
        solve_graph_mask_ = mesh_on;
    }
    WRAPD_CUDA(cudaGraphLaunch(solve_graph_, st));
}

}  // namespace wrapd
