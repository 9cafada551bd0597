// Dense Cholesky factorization A = L L^T (FP64) and its solve.
//
// Replaces cholesky_factor / _cholesky_factor! (src/lapack/factorizations.jl:
// 205-291, LAPACK potrf2 recursion with 64-column leaves) and the solve of a
// CholeskyFactor (:293-305) behind OxiBLAS.cholesky / cholesky! and
// ldiv!(F::Cholesky, B) (src/api/linalg_api.jl:221-290).
//
// Layout: the lower triangle of the caller's column-major A, read with the
// same leading dimension as a ROW-major matrix, is the upper triangle of that
// matrix, and L (column-major, lower) is U = L^T (row-major, upper) in the same
// memory.  So the factorization runs in place, row-oriented, with no copy:
// blocks of NB rows of U, each
//   1. U_kk = chol(A_kk) and the inverses of its four 32 x 32 diagonal blocks,
//      one CTA, the block in shared memory;
//   2. U_k,right = U_kk^-T A_k,right by blocks of 32 rows (products with the
//      diagonal blocks' inverses), into place, into an aligned block row X and
//      into its transpose, one launch;
//   3. A_right,right -= X^T X on the FP64 tensor cores, upper triangle only
//      (tiles wholly below the diagonal skipped, crossing tiles write only on
//      and above it), its left operand the transposed copy so that both
//      operands are K-contiguous.
// The reference solves the block row by substitution (trsm!); the product with
// the inverted 32 x 32 diagonal blocks is the same solve with another
// association of the sums (the diagonal blocks of a positive definite matrix's
// factor are well conditioned: cond(U_kk)^2 <= cond(A)).
// A pivot that is not finite and positive stops the factorization there: info
// is its 1-based column (PosDefException(info)); every later block row X is
// written as zero, so the later updates change nothing, and no block row
// reaches the matrix.
#include <algorithm>
#include <cmath>
#include "oxi_internal.h"
#include "tma_util.cuh"

namespace oxi {

namespace {
constexpr int PO_NB = 128;          // block rows per step
constexpr int PO_SB = 32;           // blocks inside a diagonal block
constexpr int PO_NT = 256;
constexpr int PO_FW = 4;             // diagonal block: warps that factor, the others update
constexpr int PO_DT = 32 * PO_FW + 256;
constexpr int PO_GB = 8;            // rows factored between two updates of the block
// row pitches in shared memory: 4 modulo 16, no conflicts of a DMMA fragment's loads
constexpr int PO_LP = PO_NB + 4, PO_CP = PO_SB + 4;
}  // namespace

// d = sqrt(a), y = 1 / d and z, an approximation of 1 / d that is ready earlier,
// for 2^-900 < a < 2^900: the approximate reciprocal root y0, one step of the
// binomial series of (1 - e)^(-1/2) with e = 1 - a y0^2 (z = y0 (1 + e / 2 + 3 e^2 / 8),
// within an ulp), and each result corrected once by its fused remainder
// (P. Markstein, Computation of elementary functions on the IBM RISC System/6000
// processor, IBM J. Res. Dev. 34, 1990): the latency of one chain instead of a
// square root followed by a division.  What is left before the last rounding is of
// the order of 2^-103 of the result, so it is the rounded root (quotient) but where
// the exact one lies that close to the middle of two numbers; test_kernel_edges_gpu.py
// compares both with sqrt and the division bit for bit.
__device__ __forceinline__ void root_recip(double a, double &d, double &y, double &z) {
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-(a * y), y, 1.0);
    z = fma(y * e, fma(0.375, e, 0.5), y);
    const double g = a * z;
    d = fma(fma(-g, g, a), 0.5 * z, g);
    y = fma(fma(-d, z, 1.0), z, z);
}
__device__ __forceinline__ void root_recip(float a, float &d, float &y, float &z) {
    d = sqrtf(a);
    z = y = 1.0f / d;
}
__device__ __forceinline__ bool root_range(double a) { return a > 0x1p-900 && a < 0x1p900; }
__device__ __forceinline__ bool root_range(float a) { return a > 0.0f && a <= 3.402823466e38f; }
__device__ __forceinline__ bool exp_all_ones(double a) { return (__double2hiint(a) & 0x7ff00000) == 0x7ff00000; }
__device__ __forceinline__ bool exp_all_ones(float a) { return (__float_as_uint(a) & 0x7f800000u) == 0x7f800000u; }

// Rows of an N x N diagonal block (upper, u) with one column x beside it:
// u_cc = sqrt(u_cc), u_cj /= u_cc, x_c /= u_cc, then the rows below take the
// products; sy, if not null, takes the reciprocals of the roots.  FAST has no
// branch: roots and quotients are products with the reciprocal corrected by the
// remainder (see root_recip), and false is returned where a pivot or
// a result leaves the range in which that holds (the caller starts again without
// FAST, which divides).  Returns true with bad = the first pivot that is not
// finite and positive (N: none) otherwise.
template <bool FAST, int N, typename T>
__device__ __forceinline__ bool chol_rows(T (&u)[N][N], T (&x)[N], T *sy, int &bad) {
    bool ok = true;
    bad = N;
#pragma unroll
    for (int c = 0; c < N; ++c) {
        const T a = u[c][c];
        T d, y, z;
        if constexpr (FAST) {
            ok = ok && root_range(a);
            root_recip(a, d, y, z);
        } else {
            if (bad < N) continue;
            if (!(a > T(0)) || exp_all_ones(a)) {
                bad = c;
                continue;
            }
            d = sqrt(a);
            y = T(1) / d;
        }
        if (sy) sy[c] = y;
        u[c][c] = d;
#pragma unroll
        for (int j = c; j < N; ++j) {  // j = c: the column beside the block
            T &v = j == c ? x[c] : u[c][j];
            if constexpr (FAST) {
                const T q = v * z;
                v = fma(fma(-q, d, v), z, q);
            } else {
                v = v / d;
            }
        }
#pragma unroll
        for (int i = c + 1; i < N; ++i) {
#pragma unroll
            for (int k = i; k < N; ++k) u[i][k] = fma(-u[c][i], u[c][k], u[i][k]);
            x[i] = fma(-u[c][i], x[c], x[i]);
        }
    }
    if constexpr (FAST) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            ok = ok && !exp_all_ones(x[i]);
#pragma unroll
            for (int k = i; k < N; ++k) ok = ok && !exp_all_ones(u[i][k]);
        }
    }
    return ok;
}

template <typename T>
__device__ __forceinline__ void copy_async(T *dst, const T *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"((int)sizeof(T)) : "memory");
}

// four neighbours in shared memory, 16-byte aligned
__device__ __forceinline__ void load4(double (&v)[4], const double *p) {
    const double2 a = *(const double2 *)p, b = *(const double2 *)(p + 2);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void load4(float (&v)[4], const float *p) {
    const float4 a = *(const float4 *)p;
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void store4(double *p, const double (&v)[4]) {
    *(double2 *)p = make_double2(v[0], v[1]);
    *(double2 *)(p + 2) = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void store4(float *p, const float (&v)[4]) { *(float4 *)p = make_float4(v[0], v[1], v[2], v[3]); }

// Cholesky of the t x t diagonal block (row-major upper, ld) in shared memory, by
// groups of 8 rows.  Each of the factoring warps that has columns to the right factors
// the group's 8 x 8 diagonal block in registers, each lane the whole of it (no
// exchange between lanes, no barrier before the rows to the right), and takes
// its own column along.  The updating warps then take the rank-8 product for the
// next group's rows, and for the rest while the next group is factored.  These
// are the operations of the reference leaf's column updates
// (src/lapack/factorizations.jl:266-282), read through the transposition.
// Winv: the inverses of a full block's 32 x 32 diagonal blocks, PO_SB x PO_SB
// row-major each (upper), one warp each at the end.
// Bound: latency of the 16 groups, each a chain of eight roots, quotients and
// products (3200 cycles), the next rows' update (250) and two barriers.  Alone on
// one B200: 80000 cycles; 472000 with one warp passing the block's rows by shuffles
// (380000 of them), loads each waiting for the store of the one before (36000)
// and the update between the groups (1500 each).  In the n = 4999 factorization,
// beside the trailing update, 88 -> 53 us; the whole, with small tiles for the next
// block's rows, 5.76 -> 4.06 ms.
template <typename T>
__global__ void __launch_bounds__(PO_DT) k_potrf_diag(T *__restrict__ U, i64 ld, int t, i64 g0,
                                                      int64_t *__restrict__ info, T *__restrict__ Winv) {
    extern __shared__ __align__(16) unsigned char po_smem_raw[];
    T *S = (T *)po_smem_raw;
    __shared__ T s_y[PO_NB];  // 1 / u_ii
    __shared__ __align__(16) T s_d[PO_GB][PO_GB];  // a group's factored diagonal block
    __shared__ int s_fail;            // 1 + the first column of the failing group
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_fail = (*(volatile int64_t *)info != 0) ? 1 : 0;
    __syncthreads();
    if (s_fail) return;  // an earlier block failed
    // the upper triangle, every element's copy in flight at once; identity past t
    for (int e = tid; e < PO_NB * PO_NB; e += PO_DT) {
        const int i = e / PO_NB, j = e % PO_NB;
        if (j < i) continue;
        if (j < t) copy_async(&S[i * PO_LP + j], U + (i64)i * ld + j);
        else S[i * PO_LP + j] = i == j ? T(1) : T(0);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // FP32: the whole of it by 4 x 4 tiles of the upper triangle
    auto update32 = [&](int b0) {
        const int r0 = b0 + PO_GB;
        const int nt4 = (PO_NB - r0) / 4, tasks = nt4 * (nt4 + 1) / 2;
        for (int q = tid; q < tasks; q += PO_DT) {
            int bj = (int)((sqrtf(8.0f * q + 1.0f) - 1.0f) * 0.5f);
            while ((bj + 1) * (bj + 2) / 2 <= q) ++bj;
            while (bj * (bj + 1) / 2 > q) --bj;
            const int bi = q - bj * (bj + 1) / 2;
            const int i = r0 + 4 * bi, j = r0 + 4 * bj;
            T v[4][4];
#pragma unroll
            for (int u = 0; u < 4; ++u) load4(v[u], S + (i + u) * PO_LP + j);
#pragma unroll
            for (int p = 0; p < PO_GB; ++p) {
                const T *row = S + (b0 + p) * PO_LP;
                T ui[4], uj[4];
                load4(ui, row + i);
                load4(uj, row + j);
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int w = 0; w < 4; ++w) v[u][w] = fma(-ui[u], uj[w], v[u][w]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) store4(S + (i + u) * PO_LP + j, v[u]);
        }
    };
    auto bar = [] { asm volatile("bar.sync 1, %0;" ::"n"(PO_DT) : "memory"); };
    // The two roles meet at two barriers a group: the group's rows are factored;
    // the next group's rows are up to date.
    if (warp < PO_FW) {
#pragma unroll 1
        for (int b0 = 0; b0 < t; b0 += PO_GB) {
            const int r0 = b0 + PO_GB;  // the columns to the right
            if (warp == 0 || r0 + 32 * warp < PO_NB) {
                // u: the diagonal block; x: this thread's column,
                // x_i = (a_i - sum_{p<i} u_pi x_p) / u_ii
                const int j = r0 + tid, jc = min(j, PO_NB - 1);
                T u[PO_GB][PO_GB], x[PO_GB];
                int bad;
                auto load = [&]() {
#pragma unroll
                    for (int i = 0; i < PO_GB; ++i) {
                        const T *row = S + (b0 + i) * PO_LP;
#pragma unroll
                        for (int h = 0; h < PO_GB; h += 4)
                            if (h + 3 >= i) {
                                T v[4];
                                load4(v, row + b0 + h);
#pragma unroll
                                for (int c = 0; c < 4; ++c) u[i][h + c] = v[c];
                            }
                        x[i] = row[jc];
                    }
                };
                load();
                if (!__all_sync(0xffffffffu, chol_rows<true>(u, x, tid == 0 ? s_y + b0 : nullptr, bad))) {
                    load();
                    chol_rows<false>(u, x, tid == 0 ? s_y + b0 : nullptr, bad);
                    if (bad < PO_GB && tid == 0) {  // not positive definite at global column g0 + b0 + bad + 1
                        s_fail = b0 + 1;
                        if (*info == 0) *info = g0 + b0 + bad + 1;
                    }
                }
                if (tid == 0) {  // not over the block itself: other warps may still read it
#pragma unroll
                    for (int i = 0; i < PO_GB; ++i) {
#pragma unroll
                        for (int h = 0; h < PO_GB; h += 4)
                            if (h + 3 >= i) {
                                const T v[4] = {u[i][h], u[i][h + 1], u[i][h + 2], u[i][h + 3]};
                                store4(&s_d[i][h], v);
                            }
                    }
                }
                if (j < PO_NB && bad == PO_GB) {
#pragma unroll
                    for (int i = 0; i < PO_GB; ++i) S[(b0 + i) * PO_LP + j] = x[i];
                }
            }
            bar();
            if (s_fail) break;
            if (tid < PO_GB * PO_GB && (tid & 7) >= (tid >> 3))
                S[(b0 + (tid >> 3)) * PO_LP + b0 + (tid & 7)] = s_d[tid >> 3][tid & 7];
            if (sizeof(T) == 4) update32(b0);
            bar();
        }
        if (s_fail && tid < PO_GB * PO_GB && (tid & 7) >= (tid >> 3))  // the failing group's block as far as it got
            S[(s_fail - 1 + (tid >> 3)) * PO_LP + s_fail - 1 + (tid & 7)] = s_d[tid >> 3][tid & 7];
    } else {
        // a_ij -= sum_p u_pi u_pj (r0 <= i <= j).  FP64: the block's 72 tiles of
        // 16 x 8 on and above the diagonal stay in registers as the tensor cores'
        // accumulators, nine a warp of the eight: slot e of warp w is row tile e of
        // column tile w, then row tile e - w / 2 - 1 of column tile 15 - w.
        constexpr int SLOTS = sizeof(T) == 8 ? 9 : 1;
        const int uw = warp - PO_FW;
        const int gid = lane >> 2, tig = lane & 3;
        const int first = uw / 2 + 1;  // slots of the first column tile
        auto tile_row = [&](int e) { return 16 * (e < first ? e : e - first); };
        auto tile_col = [&](int e) { return 8 * (e < first ? uw : 15 - uw); };
        T acc[SLOTS][4];
        // the tiles of row tile lo (rest: below it) take the products of group b0's rows
        // (what a tile holds below the diagonal or of finished rows is never read)
        auto update = [&](int b0, bool rest) {
            if constexpr (sizeof(T) == 8) {
                const int r0 = b0 + PO_GB, lo = r0 & ~15;
                double bf[2][2];
#pragma unroll
                for (int w = 0; w < 2; ++w)
#pragma unroll
                    for (int h = 0; h < 2; ++h) bf[w][h] = S[(b0 + 4 * h + tig) * PO_LP + 8 * (w == 0 ? uw : 15 - uw) + gid];
#pragma unroll
                for (int e = 0; e < SLOTS; ++e) {
                    const int i = tile_row(e);
                    if (tile_col(e) >= r0 && (rest ? i > lo : i == lo)) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const double *row = S + (b0 + 4 * h + tig) * PO_LP + i + gid;
                            asm volatile(
                                "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                                : "+d"(acc[e][0]), "+d"(acc[e][1]), "+d"(acc[e][2]), "+d"(acc[e][3])
                                : "d"(-row[0]), "d"(-row[8]), "d"(e < first ? bf[0][h] : bf[1][h]));
                        }
                    }
                }
            }
        };
        if (sizeof(T) == 8) {
#pragma unroll
            for (int e = 0; e < SLOTS; ++e) {
                const int i = tile_row(e), j = tile_col(e);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const T *p = S + (i + 8 * h + gid) * PO_LP + j + 2 * tig;
                    acc[e][2 * h] = p[0];
                    acc[e][2 * h + 1] = p[1];
                }
            }
        }
#pragma unroll 1
        for (int b0 = 0; b0 < t; b0 += PO_GB) {
            if (b0 > 0) update(b0 - PO_GB, true);  // beside this group's factorization
            bar();
            if (s_fail) {  // the rows below as far as they got
                if constexpr (sizeof(T) == 8) {
#pragma unroll
                    for (int e = 0; e < SLOTS; ++e)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int i = tile_row(e) + 8 * h + gid;
                            if (i >= b0 + PO_GB)
                                *(double2 *)(S + i * PO_LP + tile_col(e) + 2 * tig) =
                                    make_double2(acc[e][2 * h], acc[e][2 * h + 1]);
                        }
                }
                break;
            }
            if constexpr (sizeof(T) == 8) {
                // as far as the next group's rows, which go back to shared memory
                const int r0 = b0 + PO_GB;
                update(b0, false);
#pragma unroll
                for (int e = 0; e < SLOTS; ++e)
                    if (tile_row(e) == (r0 & ~15) && tile_col(e) >= r0) {
                        const int h = (r0 >> 3) & 1;
                        *(double2 *)(S + (r0 + gid) * PO_LP + tile_col(e) + 2 * tig) =
                            h ? make_double2(acc[e][2], acc[e][3]) : make_double2(acc[e][0], acc[e][1]);
                    }
            } else {
                update32(b0);
            }
            bar();
        }
    }
    __syncthreads();
    if (warp < PO_NB / PO_SB && t == PO_NB && !s_fail) {
        // column `lane` of this warp's diagonal block's inverse, eight rows at a time
        const int b0 = warp * PO_SB;
        T w[PO_SB];
#pragma unroll
        for (int i = 0; i < PO_SB; ++i) w[i] = (i == lane) ? T(1) : T(0);
#pragma unroll
        for (int p = PO_SB - 1; p >= 0; --p) {
            w[p] = w[p] * s_y[b0 + p];
#pragma unroll
            for (int i = 0; i < p; ++i) w[i] = fma(-S[(b0 + i) * PO_LP + b0 + p], w[p], w[i]);
        }
#pragma unroll
        for (int i = 0; i < PO_SB; ++i) Winv[(b0 + i) * PO_SB + lane] = w[i];
    }
#pragma unroll 16
    for (int e = tid; e < PO_NB * PO_NB; e += PO_DT) {
        const int i = e / PO_NB, j = e % PO_NB;
        if (j >= i && j < t) U[(i64)i * ld + j] = S[i * PO_LP + j];
    }
}

// The block row right of a full diagonal block: X = U_kk^-T A (128 x N), 32
// columns per CTA, row block by row block: T_k = A_k - sum_{p<k} U_pk^T X_p,
// X_k = W_kk^T T_k with the diagonal block's inverse.  X goes into place (A), into
// the aligned block row X and, transposed, into Xt (N x 128); zeros instead, and
// A untouched, once the factorization has failed.  One launch instead of a
// cleared block row, a product, a copy and a transpose.  FP64 products run on the
// tensor cores.  Bound: latency (the staging, then up to 20 chained DMMAs and
// three barriers per row block).
template <typename T>
struct PoRowSmem {
    T U[PO_NB][PO_LP];
    T W[PO_NB][PO_CP];
    T A[PO_NB][PO_CP];
};

template <typename T>
__global__ void __launch_bounds__(PO_NT) k_potrf_row(const T *__restrict__ Ukk, const T *__restrict__ Winv,
                                                     T *__restrict__ A, i64 ld, i64 N, T *__restrict__ X, i64 ldx,
                                                     T *__restrict__ Xt, const int64_t *__restrict__ info) {
    extern __shared__ __align__(16) unsigned char po_smem_raw[];
    PoRowSmem<T> &S = *reinterpret_cast<PoRowSmem<T> *>(po_smem_raw);
    const int tid = threadIdx.x;
    const i64 c0 = (i64)blockIdx.x * PO_SB;
    const int cols = (int)((N - c0) < PO_SB ? (N - c0) : PO_SB);
    const bool failed = *(volatile const int64_t *)info != 0;
    if (failed) {
        for (int e = tid; e < PO_NB * PO_SB; e += PO_NT) {
            const int i = e / PO_SB, c = e % PO_SB;
            if (c < cols) {
                X[(i64)i * ldx + c0 + c] = T(0);
                Xt[(c0 + c) * PO_NB + i] = T(0);
            }
        }
        return;
    }
    for (int e = tid; e < PO_NB * PO_NB; e += PO_NT) {
        const int i = e / PO_NB, j = e % PO_NB;
        if (j / PO_SB > i / PO_SB) copy_async(&S.U[i][j], Ukk + (i64)i * ld + j);
    }
    for (int e = tid; e < PO_NB * PO_SB; e += PO_NT) {
        const int i = e / PO_SB, c = e % PO_SB;
        copy_async(&S.W[i][c], Winv + e);
        if (c < cols) copy_async(&S.A[i][c], A + (i64)i * ld + c0 + c);
        else S.A[i][c] = T(0);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if constexpr (sizeof(T) == 8) {
        // a 16 x 8 tile of the row block per warp on the tensor cores
        const int lane = tid & 31, warp = tid >> 5, gid = lane >> 2, tig = lane & 3;
        const int m0 = (warp & 1) * 16 + gid, n0 = (warp >> 1) * 8;
        auto products = [&](double (&c)[2][4], const double *Am, int ap, const double *Bm, int K) {  // Am^T Bm
#pragma unroll 4
            for (int k = 0; k < K; k += 8)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int kc = k + 4 * h + tig;
                    asm volatile(
                        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                        : "+d"(c[h][0]), "+d"(c[h][1]), "+d"(c[h][2]), "+d"(c[h][3])
                        : "d"(Am[kc * ap + m0]), "d"(Am[kc * ap + m0 + 8]), "d"(Bm[kc * PO_CP + n0 + gid]));
                }
        };
        for (int b = 0; b < PO_NB; b += PO_SB) {
            if (b > 0) {
                double c[2][4] = {};
                products(c, &S.U[0][b], PO_LP, &S.A[0][0], b);
                // each thread rewrites elements that only it has read in this block
#pragma unroll
                for (int e = 0; e < 4; ++e) S.A[b + m0 + 8 * (e >> 1)][n0 + 2 * tig + (e & 1)] -= c[0][e] + c[1][e];
                __syncthreads();
            }
            double c[2][4] = {};
            products(c, &S.W[b][0], PO_CP, &S.A[b][0], PO_SB);  // W is zero below its diagonal
            __syncthreads();
#pragma unroll
            for (int e = 0; e < 4; ++e) S.A[b + m0 + 8 * (e >> 1)][n0 + 2 * tig + (e & 1)] = c[0][e] + c[1][e];
            __syncthreads();
        }
    } else {
        const int ri = tid >> 3, c4 = (tid & 7) * 4;  // a row, four columns
        for (int b = 0; b < PO_NB; b += PO_SB) {
            T v[4];
            load4(v, &S.A[b + ri][c4]);
            if (b > 0) {
#pragma unroll 8
                for (int p = 0; p < b; ++p) {
                    const T u = S.U[p][b + ri];
                    T x[4];
                    load4(x, &S.A[p][c4]);
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[q] = fma(-u, x[q], v[q]);
                }
                store4(&S.A[b + ri][c4], v);
                __syncthreads();
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = T(0);
#pragma unroll 8
            for (int p = 0; p < PO_SB; ++p) {
                const T w = S.W[b + p][ri];  // zero below the diagonal
                T x[4];
                load4(x, &S.A[b + p][c4]);
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = fma(w, x[q], v[q]);
            }
            __syncthreads();
            store4(&S.A[b + ri][c4], v);
            __syncthreads();
        }
    }
#pragma unroll 4
    for (int e = tid; e < PO_NB * PO_SB; e += PO_NT) {
        const int i = e / PO_SB, c = e % PO_SB;
        if (c < cols) {
            const T x = S.A[i][c];
            A[(i64)i * ld + c0 + c] = x;
            X[(i64)i * ldx + c0 + c] = x;
        }
    }
#pragma unroll 4
    for (int e = tid; e < PO_NB * PO_SB; e += PO_NT) {
        const int c = e / PO_NB, i = e % PO_NB;
        if (c < cols) Xt[(c0 + c) * PO_NB + i] = S.A[i][c];
    }
}

// The strict lower triangle of the row-major view (the strict upper triangle
// of the caller's column-major matrix) set to zero, as the reference does.
template <typename T>
__global__ void k_zero_strict_lower(T *__restrict__ U, i64 ld, int n, const int64_t *__restrict__ info) {
    if (*info != 0) return;  // as the reference: a failed factorization keeps its other triangle
    const i64 idx = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (i64)n * n) return;
    const int i = (int)(idx / n), j = (int)(idx - (i64)i * n);
    if (j < i) U[(i64)i * ld + j] = T(0);
}

// Workspace of one factorization, in elements: Xt (n x NB) and X (NB x ldx), two
// of each (the lookahead's update of block k reads them while block k + 1 writes
// the other pair), and the diagonal blocks' inverses.
size_t potrf_work_elems(i64 n) {
    const i64 ldx = (n + 3) / 4 * 4;
    return 2 * (size_t)n * PO_NB + 2 * (size_t)PO_NB * ldx + (size_t)PO_NB * PO_SB + 64;
}

// The symmetric update A22 -= Xt X, upper triangle of the row-major view: FP64
// on the DMMA tensor-core GEMM; FP32 (the mixed solve's low-precision factor, a
// private copy) in the handle's trailing precision (tcgen05 for the 16-bit
// kinds; the whole square, the other triangle being scratch there).
// rows x N block of the symmetric update whose (0, 0) is on the diagonal
// (M <= N): FP64 only on and above the diagonal
static void po_sym_update(oxi_handle_s *, double *A22, i64 ld, const double *T, int t, const double *X, i64 ldx,
                          i64 M, i64 N, cudaStream_t s) {
    launch_gemm_dmma(A22, ld, T, t, X, ldx, M, N, t, s, /*upper_only=*/true);
}
static void po_sym_update(oxi_handle_s *h, float *A22, i64 ld, const float *T, int t, const float *X, i64 ldx,
                          i64 M, i64 N, cudaStream_t s) {
    if (h->trailing == TRAIL_NATIVE) launch_gemm_simt<float>(A22, ld, T, t, X, ldx, M, N, t, s);
    else gemm_trailing_f32(h, A22, ld, T, t, X, ldx, M, N, t);
}

// One factorization: U in place (row-major view), *d_info set on failure.
// With the lookahead (OXI_OPT_LOOKAHEAD, the reference GEMM mode excluded)
// block k's symmetric update is split: the next block's rows first, on the
// panel stream (they are what block k + 1 needs), the rest on the low-priority
// stream beside block k + 1's diagonal factor and block-row product; the
// next block's rows wait for that rest of block k - 1's update.  Every element
// is updated by the same products in the same order: the factor is the same.
template <typename T>
void potrf_rowmajor(oxi_handle_s *h, T *U, i64 ld, i64 n, int64_t *d_info, T *work) {
    const cudaStream_t caller = h->stream;
    const bool la = h->opt.lookahead && h->opt.gemm == 0 && n > 2 * PO_NB;
    const i64 ldx = (n + 3) / 4 * 4;  // 16-byte rows for the TMA-fed GEMMs
    T *Tt2[2] = {work, work + (size_t)n * PO_NB};
    T *X2[2] = {work + 2 * (size_t)n * PO_NB, work + 2 * (size_t)n * PO_NB + (size_t)PO_NB * ldx};
    T *Winv = X2[1] + (size_t)PO_NB * ldx;
    if (la) {
        ensure_lookahead_streams(h);
        OXI_CUDA(cudaEventRecord(h->la_in, caller));
        OXI_CUDA(cudaStreamWaitEvent(h->la_main, h->la_in, 0));
        h->stream = h->la_main;
    }
    const cudaStream_t s = h->stream;
    bool b_pending = false;
    try {
        for (i64 k0 = 0, kb = 0; k0 < n; k0 += PO_NB, ++kb) {
            const int t = (int)std::min<i64>(PO_NB, n - k0);
            T *Ukk = U + k0 * ld + k0;
            T *Tt = Tt2[kb & 1], *X = X2[kb & 1];
            {
                const int smem = (int)(sizeof(T) * PO_NB * PO_LP);
                set_max_dyn_smem((const void *)k_potrf_diag<T>, smem);
                ProfScope ps(KC_LEAF, s, (double)t * t * t * (2.0 / 3.0), 2.0 * sizeof(T) * t * t);
                k_potrf_diag<T><<<1, PO_DT, smem, s>>>(Ukk, ld, t, k0, d_info, Winv);
                OXI_LAUNCH_CHECK();
            }
            const i64 right = n - k0 - t;
            if (right <= 0) break;
            {
                const int smem = (int)sizeof(PoRowSmem<T>);
                set_max_dyn_smem((const void *)k_potrf_row<T>, smem);
                ProfScope ps(KC_TRSM_LEAF, s, (double)t * t * right, 4.0 * (double)t * right * sizeof(T));
                k_potrf_row<T><<<(unsigned)((right + PO_SB - 1) / PO_SB), PO_NT, smem, s>>>(Ukk, Winv, Ukk + t, ld, right,
                                                                                           X, ldx, Tt, d_info);
                OXI_LAUNCH_CHECK();
            }
            T *A22 = U + (k0 + t) * ld + (k0 + t);
            if (!la) {
                po_sym_update(h, A22, ld, Tt, t, X, ldx, right, right, s);
                continue;
            }
            // the rest of the update needs the block row only (FP32 converts its
            // operands in the handle's buffers, one update after the other)
            if (sizeof(T) == 8) OXI_CUDA(cudaEventRecord(h->la_fork, s));
            // the next block's rows, after the rest of the previous update
            if (b_pending) {
                OXI_CUDA(cudaStreamWaitEvent(s, h->la_join, 0));
                b_pending = false;
            }
            const i64 t2 = std::min<i64>(PO_NB, right);
            po_sym_update(h, A22, ld, Tt, t, X, ldx, t2, right, s);
            if (right > t2) {  // the rest on the low-priority stream
                if (sizeof(T) == 4) OXI_CUDA(cudaEventRecord(h->la_fork, s));
                OXI_CUDA(cudaStreamWaitEvent(h->la_stream, h->la_fork, 0));
                h->stream = h->la_stream;
                h->tc_slot = 1;
                // tcgen05: persistent clusters on every GPC but one, which stays free for
                // the next block's diagonal factor and block-row product
                if constexpr (sizeof(T) == 4) h->gemm_ctas = -64;
                po_sym_update(h, A22 + t2 * ld + t2, ld, Tt + t2 * t, t, X + t2, ldx, right - t2, right - t2,
                              h->la_stream);
                h->stream = s;
                h->tc_slot = 0;
                h->gemm_ctas = 0;
                OXI_CUDA(cudaEventRecord(h->la_join, h->la_stream));
                b_pending = true;
            }
        }
        if (b_pending) OXI_CUDA(cudaStreamWaitEvent(s, h->la_join, 0));
        const i64 tot = n * n;
        k_zero_strict_lower<T><<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(U, ld, (int)n, d_info);
        OXI_LAUNCH_CHECK();
        if (la) {
            OXI_CUDA(cudaEventRecord(h->la_out, s));
            OXI_CUDA(cudaStreamWaitEvent(caller, h->la_out, 0));
        }
        h->stream = caller;
    } catch (...) {
        h->stream = caller;
        h->tc_slot = 0;
        h->gemm_ctas = 0;
        throw;
    }
}
template void potrf_rowmajor<double>(oxi_handle_s *, double *, i64, i64, int64_t *, double *);
template void potrf_rowmajor<float>(oxi_handle_s *, float *, i64, i64, int64_t *, float *);

// ---------------------------------------------------------------------------
// Solves with the factor: L y = b, then L^T x = y (the reference's two
// triangular solves, src/lapack/factorizations.jl:293-305).  L is the caller's
// column-major lower factor: the superblock solve of a non-unit lower triangle and its
// transpose (solve.cu, trsv.cu).
// ---------------------------------------------------------------------------
template <typename T>
void potrs_colmajor(oxi_handle_s *h, i64 n, i64 nrhs, const T *L, i64 ldl, T *B, i64 ldb, int *d_err);

}  // namespace oxi

extern "C" int oxi_dpotrf(oxi_handle_t h, int64_t n, double *dA, int64_t lda, int64_t *h_info) {
    using namespace oxi;
    if (!h || !h_info || n < 0 || lda < std::max<int64_t>(1, n)) return OXI_EINVAL;
    *h_info = 0;
    if (n == 0) return OXI_OK;
    if (!dA || n >= (1ll << 31)) return OXI_EINVAL;
    try {
        ProfGuard pg(&h->prof);
        OXI_CUDA(cudaSetDevice(h->device));
        AbortScope ab(h);
        char *sc = (char *)h->scratch.get(kScratchBytes);
        int64_t *d_info = (int64_t *)sc;
        OXI_CUDA(cudaMemsetAsync(d_info, 0, sizeof(int64_t), h->stream));
        // T (the transposed block row, n x NB) and room for an aligned copy of the block row
        double *work = (double *)h->work.get(sizeof(double) * potrf_work_elems(n));
        potrf_rowmajor<double>(h, dA, lda, n, d_info, work);
        int64_t *hi = (int64_t *)h->host_ws.get(64);
        OXI_CUDA(cudaMemcpyAsync(hi, d_info, sizeof(int64_t), cudaMemcpyDeviceToHost, h->stream));
        queue_abort_read(h, (int *)(hi + 2));
        OXI_CUDA(cudaStreamSynchronize(h->stream));
        *h_info = hi[0];
        const int we = check_abort(h, (const int *)(hi + 2));
        if (we != OXI_OK) return we;
        return hi[0] > 0 ? OXI_ENOTPOSDEF : OXI_OK;
    } catch (const CudaError &e) {
        h->last_error = std::string(e.what) + ": " + cudaGetErrorString(e.code);
        return OXI_ECUDA;
    }
}

extern "C" int oxi_dpotrs(oxi_handle_t h, int64_t n, int64_t nrhs, const double *dL, int64_t ldl, double *dB,
                          int64_t ldb) {
    using namespace oxi;
    if (!h || n < 0 || nrhs < 0 || ldl < std::max<int64_t>(1, n) || ldb < std::max<int64_t>(1, n))
        return OXI_EINVAL;
    if (n == 0 || nrhs == 0) return OXI_OK;
    if (!dL || !dB || n >= (1ll << 31)) return OXI_EINVAL;
    try {
        ProfGuard pg(&h->prof);
        OXI_CUDA(cudaSetDevice(h->device));
        AbortScope ab(h);
        potrs_colmajor<double>(h, n, nrhs, dL, ldl, dB, ldb, ab.word);
        int *he = (int *)h->host_ws.get(64);
        queue_abort_read(h, he);
        OXI_CUDA(cudaStreamSynchronize(h->stream));
        return check_abort(h, he);
    } catch (const CudaError &e) {
        h->last_error = std::string(e.what) + ": " + cudaGetErrorString(e.code);
        return OXI_ECUDA;
    }
}
