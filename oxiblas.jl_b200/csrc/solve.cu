// Triangular solves with the LU factors (ldiv!), column-major factors as the
// caller holds them.
//
// N: X = B[p, :], then L (unit lower) and U solves   (src/api/linalg_api.jl:168-175)
// T: U^T then L^T solves, then X[p, :] = X            (src/api/linalg_api.jl:176-184)
//
// The handle's solves run on the superblock kernels (trsv.cu).  The
// no-allocation entry point has k_trsv2 below: a CTA takes the next 64-row
// block from an atomic ticket (so every block it waits on is already running,
// which rules out deadlock), accumulates the products with the solved blocks as
// their "done" flags appear (bounded spin; a timeout sets an error word and the
// kernel returns), solves its 64 x 64 diagonal block with warp shuffles, and
// publishes its rows.  The factor is read once, coalesced: threads run along
// the contiguous dimension of the factor (rows for L/U, columns for L^T/U^T).
#include <atomic>
#include <mutex>
#include <vector>
#include "oxi_internal.h"
#include "tma_util.cuh"

namespace oxi {

constexpr int SB = 64;        // rows per block
constexpr int SOLVE_NT = 256; // threads per CTA

__device__ __forceinline__ int ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(int *p, int v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// M is the effective triangle: ROWACC ? M(r, j) = A[r*lda + j] : M(r, j) = A[r + j*lda].
// A CTA owns a row block (ticket order); its 8 warps take the solved column
// blocks round-robin, each lane accumulating two rows, so the off-diagonal
// products of one block run with 8-way memory parallelism and no cross-lane
// reductions.  The diagonal block is solved by substitution: no workspace
// beyond the flags.
constexpr int TRSV_WARPS = SOLVE_NT / 32;

template <typename T, int NR>
struct TrsvSmem {
    T x[TRSV_WARPS][SB][NR];     // per-warp staging of solved blocks
    T acc[TRSV_WARPS][SB][NR];   // per-warp partial sums
    T y[SB][NR];                 // right-hand side of the diagonal block
    T x0[SB][NR];                // the critical block's solution
    T part[SOLVE_NT / SB][SB][NR];
    T tile[SB][SB + 1];          // the critical off-diagonal tile, prefetched
    T diag[SB][SB + 1];          // the diagonal block
};

// A solved block is published through its flag (release after the rows are
// stored; consumers acquire it before reading the rows).
template <typename T, bool LOWER, bool UNIT, bool ROWACC, int NR>
__global__ void __launch_bounds__(SOLVE_NT)
k_trsv2(const T *__restrict__ A, i64 lda, T *__restrict__ X, i64 ldx, int n, int *__restrict__ ticket,
        int *__restrict__ flags, int *__restrict__ err) {
    extern __shared__ __align__(16) unsigned char trsv_smem[];
    TrsvSmem<T, NR> &S = *reinterpret_cast<TrsvSmem<T, NR> *>(trsv_smem);
    __shared__ int s_blk;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nb = (n + SB - 1) / SB;
    if (t == 0) s_blk = aborted(err) ? nb : atomicAdd(ticket, 1);  // an aborted call: no block
    __syncthreads();
    const int bi = s_blk;
    if (bi >= nb) return;
    const int b = LOWER ? bi : nb - 1 - bi;
    const int r0 = b * SB;
    const int rows = min(SB, n - r0);
    auto Mv = [&](int r, int j) -> T {
        return ROWACC ? A[(i64)r * lda + j] : A[(i64)r + (i64)j * lda];
    };

    // ---- prefetch (no dependency on other blocks): diagonal block and critical tile ----
    const bool has_crit = bi > 0;
    const int cc = LOWER ? b - 1 : b + 1;  // the last block solved before this one
    const int cc0 = cc * SB, ccols = has_crit ? min(SB, n - cc0) : 0;
    for (int e = t; e < SB * SB; e += SOLVE_NT) {
        // threads run along the contiguous index of the stored factor
        int r, j;
        if (ROWACC) { r = e / SB; j = e % SB; } else { r = e % SB; j = e / SB; }
        S.diag[r][j] = (r < rows && j < rows) ? Mv(r0 + r, r0 + j) : T(0);
        if (has_crit) S.tile[r][j] = (r < rows && j < ccols) ? Mv(r0 + r, cc0 + j) : T(0);
    }

    // ---- products with the other solved blocks (warps round-robin) ----
    // 16-byte row loads only when every row start is 16-byte aligned (the
    // caller's lda need not be even).
    const bool vec_rows = ROWACC && ((lda * (i64)sizeof(T)) % 16 == 0) && ((((uintptr_t)A) & 15) == 0);
    T acc[2][NR];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int k = 0; k < NR; ++k) acc[q][k] = T(0);
    for (int step = warp; step < bi - 1; step += TRSV_WARPS) {
        const int c = LOWER ? step : nb - 1 - step;
        const int c0 = c * SB;
        const int cols = min(SB, n - c0);
        if (lane == 0 && ld_acquire(&flags[c]) == 0) {
            const uint64_t t0 = global_ns();
            uint32_t it = 0;
            while (ld_acquire(&flags[c]) == 0) {
                if (spin_give_up<256>(it, t0, err, 3)) break;
            }
        }
        __syncwarp();
        for (int e = lane; e < SB * NR; e += 32) {
            const int jj = e % SB, k = e / SB;
            S.x[warp][jj][k] = (jj < cols) ? __ldcg(&X[(i64)(c0 + jj) + (i64)k * ldx]) : T(0);
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int r = lane + 32 * q;
            if (r >= rows) continue;
            if (ROWACC) {
                const T *arow = A + (i64)(r0 + r) * lda + c0;
                if (cols == SB && vec_rows) {
#pragma unroll 16
                    for (int jj = 0; jj < SB; jj += 16 / (int)sizeof(T)) {
                        T av[16 / sizeof(T)];
                        *(int4 *)av = *(const int4 *)(arow + jj);
#pragma unroll
                        for (int u = 0; u < (int)(16 / sizeof(T)); ++u)
#pragma unroll
                            for (int k = 0; k < NR; ++k) acc[q][k] = fma(av[u], S.x[warp][jj + u][k], acc[q][k]);
                    }
                } else {
                    for (int jj = 0; jj < cols; ++jj)
#pragma unroll
                        for (int k = 0; k < NR; ++k) acc[q][k] = fma(arow[jj], S.x[warp][jj][k], acc[q][k]);
                }
            } else {
                const T *acol = A + (i64)(r0 + r) + (i64)c0 * lda;
#pragma unroll 16
                for (int jj = 0; jj < cols; ++jj) {
                    const T a = acol[(i64)jj * lda];
#pragma unroll
                    for (int k = 0; k < NR; ++k) acc[q][k] = fma(a, S.x[warp][jj][k], acc[q][k]);
                }
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int k = 0; k < NR; ++k) S.acc[warp][lane + 32 * q][k] = acc[q][k];
    __syncthreads();
    for (int e = t; e < SB * NR; e += SOLVE_NT) {
        const int r = e % SB, k = e / SB;
        T v = T(0);
#pragma unroll
        for (int w = 0; w < TRSV_WARPS; ++w) v += S.acc[w][r][k];
        S.y[r][k] = (r < rows) ? (X[(i64)(r0 + r) + (i64)k * ldx] - v) : T(0);
    }

    // ---- critical path: the block solved just before, then the diagonal ----
    constexpr int SEG = SOLVE_NT / SB, SEGW = SB / SEG;
    const int pr = t % SB, ps = t / SB;
    if (has_crit) {
        if (t == 0 && ld_acquire(&flags[cc]) == 0) {
            const uint64_t t0 = global_ns();
            uint32_t it = 0;
            while (ld_acquire(&flags[cc]) == 0) {
                if (spin_give_up<256>(it, t0, err, 3)) break;
            }
        }
        __syncthreads();
        for (int e = t; e < SB * NR; e += SOLVE_NT) {
            const int jj = e % SB, k = e / SB;
            S.x0[jj][k] = (jj < ccols) ? __ldcg(&X[(i64)(cc0 + jj) + (i64)k * ldx]) : T(0);
        }
        __syncthreads();
        T pv[NR];
#pragma unroll
        for (int k = 0; k < NR; ++k) pv[k] = T(0);
#pragma unroll
        for (int jj = 0; jj < SEGW; ++jj) {
            const T a = S.tile[pr][ps * SEGW + jj];
#pragma unroll
            for (int k = 0; k < NR; ++k) pv[k] = fma(a, S.x0[ps * SEGW + jj][k], pv[k]);
        }
#pragma unroll
        for (int k = 0; k < NR; ++k) S.part[ps][pr][k] = pv[k];
        __syncthreads();
        for (int e = t; e < SB * NR; e += SOLVE_NT) {
            const int r = e % SB, k = e / SB;
            T v = T(0);
#pragma unroll
            for (int q = 0; q < SEG; ++q) v += S.part[q][r][k];
            S.y[r][k] -= v;
        }
    }
    __syncthreads();

    // substitution on the diagonal block: warp k takes right-hand side k
    for (int k = warp; k < NR; k += TRSV_WARPS) {
        T y[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) y[q] = S.y[lane + 32 * q][k];
        for (int st = 0; st < rows; ++st) {
            const int p = LOWER ? st : rows - 1 - st;
            const int hp = p >> 5, lp = p & 31;
            const T yp = __shfl_sync(0xffffffffu, hp ? y[1] : y[0], lp);
            const T xp = UNIT ? yp : yp / S.diag[p][p];
            if (lane == lp) { if (hp) y[1] = xp; else y[0] = xp; }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int r = lane + 32 * q;
                const bool below = LOWER ? (r > p) : (r < p);
                if (below && r < rows) y[q] = fma(-S.diag[r][p], xp, y[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int r = lane + 32 * q;
            if (r < rows) X[(i64)(r0 + r) + (i64)k * ldx] = y[q];
        }
    }
    __threadfence();
    __syncthreads();
    if (t == 0) st_release(&flags[b], 1);
}

template <typename T>
__global__ void k_gather_rows(const T *__restrict__ B, i64 ldb, const int64_t *__restrict__ perm,
                              T *__restrict__ X, i64 ldx, int n, int nrhs, int scatter) {
    const i64 idx = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (i64)n * nrhs) return;
    const int i = (int)(idx % n), k = (int)(idx / n);
    if (!scatter) X[i + (i64)k * ldx] = B[perm[i] + (i64)k * ldb];
    else X[perm[i] + (i64)k * ldx] = B[i + (i64)k * ldb];
}

// UPPER_A / TRANS describe the stored factor as in LAPACK (column-major A,
// op(A) = A or A^T); ROWACC access of the same memory is the transposed view.
template <typename T, bool UPPER_A, bool UNIT, bool TRANS>
static void trsv_launch(const T *A, i64 lda, T *X, i64 ldx, int n, int nrhs, int *ctl, int *err,
                        cudaStream_t s) {
    constexpr bool LOWER = (UPPER_A == TRANS);
    const int nb = (n + SB - 1) / SB;
    ProfScope ps(KC_TRSV, s, (double)n * n * nrhs, (double)n * n * sizeof(T) / 2);
    for (int k0 = 0; k0 < nrhs;) {
        const int left = nrhs - k0;
        OXI_CUDA(cudaMemsetAsync(ctl, 0, sizeof(int) * (nb + 1), s));
        int *ticket = ctl, *flags = ctl + 1;
        T *Xk = X + (i64)k0 * ldx;
#define OXI_TRSV_GO(NRV)                                                                              \
    do {                                                                                             \
        const int smem = (int)sizeof(TrsvSmem<T, NRV>);                                             \
        auto kern = k_trsv2<T, LOWER, UNIT, TRANS, NRV>;                                             \
        OXI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));     \
        kern<<<nb, SOLVE_NT, smem, s>>>(A, lda, Xk, ldx, n, ticket, flags, err);                      \
        k0 += NRV;                                                                                   \
    } while (0)
        if (left >= 8) OXI_TRSV_GO(8);
        else if (left >= 4) OXI_TRSV_GO(4);
        else if (left >= 2) OXI_TRSV_GO(2);
        else OXI_TRSV_GO(1);
#undef OXI_TRSV_GO
        OXI_LAUNCH_CHECK();
    }
}

// Solve with device-resident permutation `perm` (0-based, A[perm,:] = L U).
template <typename T>
void getrs_perm(oxi_handle_s *h, char trans, i64 n, i64 nrhs, const T *LU, i64 lda,
                const int64_t *d_perm, T *B, i64 ldb, int *d_err) {
    cudaStream_t s = h->stream;
    T *X = (T *)h->solve_ws.get(sizeof(T) * (size_t)n * nrhs);
    const i64 tot = n * nrhs;
    const int nt = 256;
    // the two triangles' block inverses, then the solves
    const i64 inv = tri_inverse_elems<T>(n);
    T *P1 = (T *)h->trsv_ws.get(2 * sizeof(T) * (size_t)inv);
    T *P2 = P1 + inv;
    const TriForm form = trans == 'N' ? TriForm::LU_N : (trans == 'T' ? TriForm::LU_T : TriForm::LU_C);
    tri_inverses<T>(h, form, LU, lda, n, P1, P2);
    if (trans == 'N') {
        k_gather_rows<T><<<(unsigned)((tot + nt - 1) / nt), nt, 0, s>>>(B, ldb, d_perm, X, n, (int)n, (int)nrhs, 0);
        OXI_LAUNCH_CHECK();
        tri_solves<T>(h, form, LU, lda, n, X, n, nrhs, d_err, P1, P2);
        OXI_CUDA(cudaMemcpy2DAsync(B, ldb * sizeof(T), X, n * sizeof(T), n * sizeof(T), nrhs,
                                   cudaMemcpyDeviceToDevice, s));
    } else {
        OXI_CUDA(cudaMemcpy2DAsync(X, n * sizeof(T), B, ldb * sizeof(T), n * sizeof(T), nrhs,
                                   cudaMemcpyDeviceToDevice, s));
        tri_solves<T>(h, form, LU, lda, n, X, n, nrhs, d_err, P1, P2);
        k_gather_rows<T><<<(unsigned)((tot + nt - 1) / nt), nt, 0, s>>>(X, n, d_perm, B, ldb, (int)n, (int)nrhs, 1);
        OXI_LAUNCH_CHECK();
    }
}
// Cholesky solve with the column-major lower factor L: L Y = B (non-unit lower),
// then L^T X = Y (its transpose, upper); B overwritten.
template <typename T>
void potrs_colmajor(oxi_handle_s *h, i64 n, i64 nrhs, const T *L, i64 ldl, T *B, i64 ldb, int *d_err) {
    const i64 inv = tri_inverse_elems<T>(n);
    T *P1 = (T *)h->trsv_ws.get(2 * sizeof(T) * (size_t)inv);
    T *P2 = P1 + inv;
    tri_inverses<T>(h, TriForm::CHOLESKY, L, ldl, n, P1, P2);
    tri_solves<T>(h, TriForm::CHOLESKY, L, ldl, n, B, ldb, nrhs, d_err, P1, P2);
}
template void potrs_colmajor<double>(oxi_handle_s *, i64, i64, const double *, i64, double *, i64, int *);

template void getrs_perm<double>(oxi_handle_s *, char, i64, i64, const double *, i64, const int64_t *, double *, i64, int *);
template void getrs_perm<zc64>(oxi_handle_s *, char, i64, i64, const zc64 *, i64, const int64_t *, zc64 *, i64, int *);
template void getrs_perm<float>(oxi_handle_s *, char, i64, i64, const float *, i64, const int64_t *, float *, i64, int *);

// LUFactor.p from the interchange sequence (src/lapack/factorizations.jl:72-75).
void perm_from_ipiv(const int64_t *ipiv, i64 q, i64 m, int64_t *perm) {
    for (i64 i = 0; i < m; ++i) perm[i] = i;
    for (i64 j = 0; j < q; ++j) {
        const i64 p = ipiv[j] - 1;
        const int64_t t = perm[j];
        perm[j] = perm[p];
        perm[p] = t;
    }
}

template <typename T>
static int getrs_entry(oxi_handle_s *h, char trans, i64 n, i64 nrhs, const T *dLU, i64 lda,
                       const int64_t *d_ipiv, T *dB, i64 ldb) {
    if (!h) return OXI_EINVAL;
    if (trans == 'C' && sizeof(T) != sizeof(zc64)) trans = 'T';
    if (trans != 'N' && trans != 'T' && trans != 'C') return OXI_EINVAL;
    if (n < 0 || nrhs < 0 || lda < std::max<i64>(1, n) || ldb < std::max<i64>(1, n)) return OXI_EINVAL;
    if (n == 0 || nrhs == 0) return OXI_OK;
    if (!dLU || !d_ipiv || !dB || n >= (1ll << 31)) return OXI_EINVAL;
    if (sizeof(T) == sizeof(zc64) && ((uintptr_t)dLU % 16 || (uintptr_t)dB % 16)) return OXI_EINVAL;
    try {
        ProfGuard pg(&h->prof);
        OXI_CUDA(cudaSetDevice(h->device));
        // The interchange sequence is inherently sequential: fold it into the
        // permutation once on the host (n int64 each way).
        std::vector<int64_t> ip(n), perm(n);
        OXI_CUDA(cudaMemcpyAsync(ip.data(), d_ipiv, sizeof(int64_t) * n, cudaMemcpyDeviceToHost, h->stream));
        OXI_CUDA(cudaStreamSynchronize(h->stream));
        for (i64 j = 0; j < n; ++j)
            if (ip[j] < 1 || ip[j] > n) return OXI_EINVAL;
        perm_from_ipiv(ip.data(), n, n, perm.data());
        AbortScope ab(h);
        int64_t *dperm = (int64_t *)h->perm_ws.get(sizeof(int64_t) * n);
        int64_t *hperm = (int64_t *)h->host_ws.get(sizeof(int64_t) * (n + 8));
        std::copy(perm.begin(), perm.end(), hperm);
        OXI_CUDA(cudaMemcpyAsync(dperm, hperm, sizeof(int64_t) * n, cudaMemcpyHostToDevice, h->stream));
        getrs_perm<T>(h, trans, n, nrhs, dLU, lda, dperm, dB, ldb, ab.word);
        int *herr = (int *)(hperm + n);
        queue_abort_read(h, herr);
        OXI_CUDA(cudaStreamSynchronize(h->stream));
        return check_abort(h, herr);
    } catch (const CudaError &e) {
        h->last_error = std::string(e.what) + ": " + cudaGetErrorString(e.code);
        return OXI_ECUDA;
    }
}

// ---------------------------------------------------------------------------
// No-allocation FP64 getrs.  Its scratch is one file-scope device array:
//   [0, 4)        abort word of the triangular solves (cleared every call)
//   [4, 8)        invalid-pivot flag (cleared every call)
//   [8, 16)       wait limit of the solves' bounded waits: never written, so
//                 zero (the default, 2 s) from the module's load
//   [256, 4356)   tickets + per-block flags of k_trsv2 (cleared per launch)
//   [8 KiB, +8n)  0-based permutation, int64 (written whole every call)
//   [1 MiB, 8 MiB) the solve vector X, n x nrhs (written before it is read)
constexpr i64 kNaScratchBytes = OXI_NOALLOC_SCRATCH_BYTES;
constexpr i64 kNaCtlOff = 256, kNaPermOff = 8192, kNaXOff = 1 << 20;
constexpr i64 kNaMaxN = OXI_NOALLOC_MAX_N;
constexpr i64 kNaMaxElems = OXI_NOALLOC_MAX_ELEMS;
static_assert(kNaMaxElems * (i64)sizeof(double) == kNaScratchBytes - kNaXOff, "X region");
static_assert(kNaPermOff + 8 * kNaMaxN <= kNaXOff, "permutation region");
static_assert(kNaCtlOff + 4 * (kNaMaxN / SB + 1) <= kNaPermOff, "control region");
constexpr int kNaMaxDevices = 64;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaScratchBytes];

// The interchange sequence folded into a permutation (as perm_from_ipiv) on the
// device: all threads check the pivots and seed the identity, then one thread
// applies the n swaps in shared memory (16-bit rows, n <= 65536), eight pivots
// fetched ahead at a time.  An out-of-range pivot sets *bad and writes nothing.
__global__ void __launch_bounds__(1024) k_perm_from_ipiv_na(const int64_t *__restrict__ ipiv, int n,
                                                            int64_t *__restrict__ perm, int *__restrict__ bad) {
    extern __shared__ uint16_t s_perm[];
    int badl = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int64_t p = ipiv[i];
        badl |= (p < 1 || p > n);
        s_perm[i] = (uint16_t)i;
    }
    if (__syncthreads_or(badl)) {
        if (threadIdx.x == 0) *bad = 1;
        return;
    }
    if (threadIdx.x == 0) {
        for (int j0 = 0; j0 < n; j0 += 8) {
            int p[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) p[u] = (j0 + u < n) ? (int)ipiv[j0 + u] - 1 : j0 + u;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (j0 + u >= n) break;
                const uint16_t a = s_perm[j0 + u], b = s_perm[p[u]];
                s_perm[j0 + u] = b;
                s_perm[p[u]] = a;
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) perm[i] = s_perm[i];
}

template <bool UPPER_A, bool UNIT, bool TRANS>
static void na_load_trsv(cudaFuncAttributes *fa) {
    constexpr bool LOWER = (UPPER_A == TRANS);
    OXI_CUDA(cudaFuncGetAttributes(fa, k_trsv2<double, LOWER, UNIT, TRANS, 1>));
    OXI_CUDA(cudaFuncGetAttributes(fa, k_trsv2<double, LOWER, UNIT, TRANS, 2>));
    OXI_CUDA(cudaFuncGetAttributes(fa, k_trsv2<double, LOWER, UNIT, TRANS, 4>));
    OXI_CUDA(cudaFuncGetAttributes(fa, k_trsv2<double, LOWER, UNIT, TRANS, 8>));
}

// Identity of the current context (cuCtxGetCurrent + cuCtxGetId through the
// runtime's driver entry points): the array's address belongs to the context
// that resolved it.
static unsigned long long current_context_id() {
    using GetCurrent = CUresult (*)(CUcontext *);
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    if (!get_current || !get_id) {
        void *p1 = nullptr, *p2 = nullptr;
        cudaDriverEntryPointQueryResult q1, q2;
        OXI_CUDA(cudaGetDriverEntryPoint("cuCtxGetCurrent", &p1, cudaEnableDefault, &q1));
        OXI_CUDA(cudaGetDriverEntryPoint("cuCtxGetId", &p2, cudaEnableDefault, &q2));
        if (!p1 || !p2 || q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess)
            throw CudaError{cudaErrorNotSupported, "cuCtxGetCurrent / cuCtxGetId unavailable"};
        get_current = (GetCurrent)p1;
        get_id = (GetId)p2;
    }
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (get_current(&ctx) != CUDA_SUCCESS || !ctx) {
        // this host thread has not used the runtime yet: a symbol query makes
        // the device's primary context current (it allocates nothing)
        void *sym = nullptr;
        OXI_CUDA(cudaGetSymbolAddress(&sym, g_noalloc_scratch));
        if (get_current(&ctx) != CUDA_SUCCESS || !ctx) throw CudaError{cudaErrorInvalidResourceHandle, "no current context"};
    }
    if (get_id(ctx, &id) != CUDA_SUCCESS) throw CudaError{cudaErrorInvalidResourceHandle, "cuCtxGetId"};
    return id;
}

// Once per device and context, with that device current: the array's address,
// and the kernels of this path loaded (so no later call loads a module).  A
// device reset or a re-created primary context gives a new context id, and the
// address is resolved again.
static char *noalloc_scratch(int dev) {
    struct Slot {
        std::atomic<char *> ptr{nullptr};
        std::atomic<unsigned long long> ctx{0};
    };
    static Slot slots[kNaMaxDevices];
    static std::mutex mu;
    const unsigned long long ctx = current_context_id();
    Slot &sl = slots[dev];
    char *p = sl.ptr.load(std::memory_order_acquire);
    if (p && sl.ctx.load(std::memory_order_acquire) == ctx) return p;
    std::lock_guard<std::mutex> lk(mu);
    p = sl.ptr.load(std::memory_order_acquire);
    if (p && sl.ctx.load(std::memory_order_acquire) == ctx) return p;
    void *sym = nullptr;
    OXI_CUDA(cudaGetSymbolAddress(&sym, g_noalloc_scratch));
    OXI_CUDA(cudaFuncSetAttribute(k_perm_from_ipiv_na, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(uint16_t) * kNaMaxN)));
    cudaFuncAttributes fa;
    OXI_CUDA(cudaFuncGetAttributes(&fa, k_gather_rows<double>));
    na_load_trsv<false, true, false>(&fa);
    na_load_trsv<true, false, false>(&fa);
    na_load_trsv<true, false, true>(&fa);
    na_load_trsv<false, true, true>(&fa);
    p = (char *)sym;
    sl.ctx.store(ctx, std::memory_order_release);
    sl.ptr.store(p, std::memory_order_release);
    return p;
}

static int getrs_noalloc(cudaStream_t s, char trans, i64 n, i64 nrhs, const double *dLU, i64 lda,
                         const int64_t *d_ipiv, double *dB, i64 ldb) {
    if (trans == 'C') trans = 'T';
    if (trans != 'N' && trans != 'T') return OXI_EINVAL;
    if (n < 0 || nrhs < 0 || lda < std::max<i64>(1, n) || ldb < std::max<i64>(1, n)) return OXI_EINVAL;
    if (n == 0 || nrhs == 0) return OXI_OK;
    if (!dLU || !d_ipiv || !dB) return OXI_EINVAL;
    if (n > kNaMaxN || nrhs > kNaMaxElems || n * nrhs > kNaMaxElems) return OXI_ESCRATCH;
    try {
        int dev = 0;
        OXI_CUDA(cudaGetDevice(&dev));
        if (dev < 0 || dev >= kNaMaxDevices) return OXI_EINVAL;
        char *sc = noalloc_scratch(dev);
        int *err = (int *)sc, *bad = err + 1, *ctl = (int *)(sc + kNaCtlOff);
        int64_t *perm = (int64_t *)(sc + kNaPermOff);
        double *X = (double *)(sc + kNaXOff);
        int hflags[2] = {0, 0};
        OXI_CUDA(cudaMemsetAsync(sc, 0, sizeof(hflags), s));
        k_perm_from_ipiv_na<<<1, 1024, sizeof(uint16_t) * n, s>>>(d_ipiv, (int)n, perm, bad);
        OXI_LAUNCH_CHECK();
        OXI_CUDA(cudaMemcpyAsync(hflags, sc, sizeof(hflags), cudaMemcpyDeviceToHost, s));
        OXI_CUDA(cudaStreamSynchronize(s));
        if (hflags[1]) return OXI_EINVAL;  // B untouched, as oxi_dgetrs
        const i64 tot = n * nrhs;
        const int nt = 256;
        const unsigned gb = (unsigned)((tot + nt - 1) / nt);
        if (trans == 'N') {
            k_gather_rows<double><<<gb, nt, 0, s>>>(dB, ldb, perm, X, n, (int)n, (int)nrhs, 0);
            OXI_LAUNCH_CHECK();
            trsv_launch<double, false, true, false>(dLU, lda, X, n, (int)n, (int)nrhs, ctl, err, s);
            trsv_launch<double, true, false, false>(dLU, lda, X, n, (int)n, (int)nrhs, ctl, err, s);
            OXI_CUDA(cudaMemcpy2DAsync(dB, ldb * sizeof(double), X, n * sizeof(double), n * sizeof(double),
                                       nrhs, cudaMemcpyDeviceToDevice, s));
        } else {
            OXI_CUDA(cudaMemcpy2DAsync(X, n * sizeof(double), dB, ldb * sizeof(double), n * sizeof(double),
                                       nrhs, cudaMemcpyDeviceToDevice, s));
            trsv_launch<double, true, false, true>(dLU, lda, X, n, (int)n, (int)nrhs, ctl, err, s);
            trsv_launch<double, false, true, true>(dLU, lda, X, n, (int)n, (int)nrhs, ctl, err, s);
            k_gather_rows<double><<<gb, nt, 0, s>>>(X, n, perm, dB, ldb, (int)n, (int)nrhs, 1);
            OXI_LAUNCH_CHECK();
        }
        OXI_CUDA(cudaMemcpyAsync(hflags, sc, sizeof(int), cudaMemcpyDeviceToHost, s));
        OXI_CUDA(cudaStreamSynchronize(s));
        return hflags[0] ? OXI_ETIMEOUT : OXI_OK;
    } catch (const CudaError &) {
        return OXI_ECUDA;
    }
}

}  // namespace oxi

extern "C" int oxi_dgetrs_noalloc(void *stream, char trans, int64_t n, int64_t nrhs, const double *dLU,
                                  int64_t lda, const int64_t *d_ipiv, double *dB, int64_t ldb) {
    return oxi::getrs_noalloc((cudaStream_t)stream, trans, n, nrhs, dLU, lda, d_ipiv, dB, ldb);
}

extern "C" int oxi_dgetrs(oxi_handle_t h, char trans, int64_t n, int64_t nrhs, const double *dLU,
                          int64_t lda, const int64_t *d_ipiv, double *dB, int64_t ldb) {
    return oxi::getrs_entry<double>(h, trans, n, nrhs, dLU, lda, d_ipiv, dB, ldb);
}
extern "C" int oxi_sgetrs(oxi_handle_t h, char trans, int64_t n, int64_t nrhs, const float *dLU,
                          int64_t lda, const int64_t *d_ipiv, float *dB, int64_t ldb) {
    return oxi::getrs_entry<float>(h, trans, n, nrhs, dLU, lda, d_ipiv, dB, ldb);
}
extern "C" int oxi_zgetrs(oxi_handle_t h, char trans, int64_t n, int64_t nrhs, const void *dLU, int64_t lda,
                          const int64_t *d_ipiv, void *dB, int64_t ldb) {
    return oxi::getrs_entry<oxi::zc64>(h, trans, n, nrhs, (const oxi::zc64 *)dLU, lda, d_ipiv, (oxi::zc64 *)dB, ldb);
}
