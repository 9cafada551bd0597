// Panel-level kernels of the dense LU: layout conversion, the cluster leaf LU,
// row interchanges, the TRSM leaf and the reference-order GEMM.
//
// Storage inside the engine is ROW-major (row i of an m x n matrix is n
// contiguous elements, leading dimension ld).  Row interchanges -- the laswp of
// src/lapack/factorizations.jl:82-88 -- then move contiguous row segments, and
// a panel row (w elements) is one contiguous load.  The C ABI converts from and
// to the caller's column-major layout at entry and exit.
#include <cooperative_groups.h>
#include <algorithm>
#include <climits>
#include <type_traits>
#include "leaf.cuh"
#include "oxi_internal.h"
#include "tma_util.cuh"

namespace cg = cooperative_groups;

namespace oxi {

// ---------------------------------------------------------------------------
// Layout conversion (32 x 32 tiles through shared memory, conflict-free).
// ---------------------------------------------------------------------------
template <typename TS, typename TD>
__global__ void k_cm_to_rm(const TS *__restrict__ A, i64 lda, TD *__restrict__ W, i64 ldw,
                           i64 m, i64 n) {
    __shared__ TD tile[32][33];
    const i64 i0 = (i64)blockIdx.x * 32, j0 = (i64)blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
    for (int r = ty; r < 32; r += 8) {             // read column j0+r, rows i0+tx
        i64 i = i0 + tx, j = j0 + r;
        if (i < m && j < n) tile[r][tx] = (TD)A[i + j * lda];
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {  // write row i0+r, columns j0+tx
        i64 i = i0 + r, j = j0 + tx;
        if (i < m && j < n) W[i * ldw + j] = tile[tx][r];
    }
}

template <typename TS, typename TD>
__global__ void k_rm_to_cm(const TS *__restrict__ W, i64 ldw, TD *__restrict__ A, i64 lda,
                           i64 m, i64 n) {
    __shared__ TD tile[32][33];
    const i64 i0 = (i64)blockIdx.x * 32, j0 = (i64)blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int r = ty; r < 32; r += 8) {  // read row i0+r, columns j0+tx
        i64 i = i0 + r, j = j0 + tx;
        if (i < m && j < n) tile[r][tx] = (TD)W[i * ldw + j];
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {  // write column j0+r, rows i0+tx
        i64 i = i0 + tx, j = j0 + r;
        if (i < m && j < n) A[i + j * lda] = tile[tx][r];
    }
}

template <typename TS, typename TD>
void launch_cm_to_rm(const TS *A, i64 lda, TD *W, i64 ldw, i64 m, i64 n, cudaStream_t s) {
    if (m <= 0 || n <= 0) return;
    dim3 grid((unsigned)((m + 31) / 32), (unsigned)((n + 31) / 32));
    k_cm_to_rm<TS, TD><<<grid, dim3(32, 8), 0, s>>>(A, lda, W, ldw, m, n);
    OXI_LAUNCH_CHECK();
}
template <typename TS, typename TD>
void launch_rm_to_cm(const TS *W, i64 ldw, TD *A, i64 lda, i64 m, i64 n, cudaStream_t s) {
    if (m <= 0 || n <= 0) return;
    dim3 grid((unsigned)((m + 31) / 32), (unsigned)((n + 31) / 32));
    k_rm_to_cm<TS, TD><<<grid, dim3(32, 8), 0, s>>>(W, ldw, A, lda, m, n);
    OXI_LAUNCH_CHECK();
}
template void launch_cm_to_rm<double, double>(const double *, i64, double *, i64, i64, i64, cudaStream_t);
template void launch_cm_to_rm<float, float>(const float *, i64, float *, i64, i64, i64, cudaStream_t);
template void launch_cm_to_rm<double, float>(const double *, i64, float *, i64, i64, i64, cudaStream_t);
template void launch_cm_to_rm<double2, double2>(const double2 *, i64, double2 *, i64, i64, i64, cudaStream_t);
template void launch_rm_to_cm<double, double>(const double *, i64, double *, i64, i64, i64, cudaStream_t);
template void launch_rm_to_cm<float, float>(const float *, i64, float *, i64, i64, i64, cudaStream_t);
template void launch_rm_to_cm<float, double>(const float *, i64, double *, i64, i64, i64, cudaStream_t);

// ---------------------------------------------------------------------------
// Leaf LU: one thread-block cluster (1..16 CTAs of NT threads) holds the m x W
// leaf in REGISTERS, R rows per thread, with implicit pivoting: a row never
// leaves its thread, it carries the position the interchanges have brought it
// to and is stored there at the end.  Column by column, as the leaf loop of
// _lu_panel! (src/lapack/factorizations.jl:116-139):
//   pivot = first position of the largest |a_ij| among positions >= j (_lu_pivot, :92-107);
//   positions j and p change places;
//   zero pivot -> info (first one), skip the column;
//   l_ij = a_ij / a_jj (correctly rounded, as the reference's division);
//   a_ic = muladd(-l_ij, a_jc, a_ic) for c > j.
// The columns go in groups of GW = 8.  A column step updates only the rest of
// its group, so what a CTA publishes per column is its candidate's position
// and live group values.  After the group its GW pivot rows publish their
// multipliers and remaining columns once, every CTA solves the GW x GW unit
// triangle for them, and each row takes the GW updates of its remaining columns
// together.  Every element sees the same fused multiply-adds in the same order
// as in the column-by-column form.
//
// Bound: latency of the column steps.  One step is a warp arg-max (one redux and
// a ballot; ties take two more) with the winner lane's candidate into shared
// memory, one CTA barrier, the arg-max over the warps and, across CTAs, one
// exchange: a few warps push one 16-byte chunk each of the CTA's winner to every
// CTA with st.async, completing on the receiver's mbarrier.  Slots are
// double-buffered by column parity, which makes one exchange per column
// sufficient: a slot is rewritten two columns later, after its receiver has
// pushed the column in between, i.e. after it read the slot.  Measured forms that
// are slower: rolled column loops (1.2-1.5 times a step), one warp reducing for
// the others (two barriers; 1.15 times in FP64), plain stores polled by every
// warp (1.15 times across CTAs).
// Rows travel between global memory and the threads that own them through
// per-warp shared memory, 128 contiguous bytes at a time: one row per lane, 16
// bytes at a time, costs 32 cache lines an instruction.
// ---------------------------------------------------------------------------
constexpr int LEAF_NT = 512;
constexpr int LEAF_MAX_CS = 16;

// The multiplier a / d.  FP64 divides, as the reference (the rounded quotient from
// the pivot's reciprocal by two remainder corrections is the same bits and slower:
// 1043 against 979 cycles a column at 256 rows, 1714 against 1648 at 1024).  FP32 multiplies by the
// pivot's rounded reciprocal (taken while the arg-max picks the pivot) and corrects
// the product by its exact remainder (Markstein's quotient, see potrf.cu); of 4e8
// random |a| <= |d| none differed from the division.  A pivot whose reciprocal
// leaves the normal range divides.
__device__ __forceinline__ double multiplier(double a, double d, double) { return a / d; }
__device__ __forceinline__ float multiplier(float a, float d, float y) {
    const uint32_t u = __float_as_uint(d) & 0x7fffffffu;
    if (u - (67u << 23) > (120u << 23)) return a / d;  // |d| outside [2^-60, 2^60]
    const float q = a * y;
    return fmaf(fmaf(-q, d, a), y, q);
}

// DUAL (FP64, 64 columns): the recursion's step from 32 to 64 columns inside the
// launch, in the reference's order (src/lapack/factorizations.jl:140-150): the
// first 32 columns as a leaf of their own, then the 32 pivot rows go to every
// CTA, each solves U12 by the recursive TRSM's steps (8-row leaves), every row
// below takes C - s with s one fma chain over the 32 columns from zero, and the
// last 32 columns are the second leaf.  It replaces two leaves, a TRSM and a GEMM.
// Bound: latency, as the leaf.
// One B200, launches timed with the profile's events: 256 rows 4 x (31 + 31 + 8
// + 10) us -> 4 x 64 us; the whole FP64 solve of n = 256 591 -> 575 us, n = 3001
// 6.29 -> 6.00 ms, the n = 2048 forward and pullback 4.59 -> 4.35 ms.  Sending
// the pivot rows by 16-byte st.async instead of bulk copies, and the step
// unrolled over its blocks, cost 6 us a leaf more across CTAs.
template <typename T, int W, int R, int NT, bool DUAL>
__global__ void __launch_bounds__(NT, 1)
k_leaf_lu(T *__restrict__ P, i64 ld, int m, int wact, i64 gofs, int64_t *__restrict__ ipiv,
          int64_t *__restrict__ info, int *__restrict__ moves, int *__restrict__ nmoves,
          LeafPanel pn) {
    cg::cluster_group cl = cg::this_cluster();
    const int CS = (int)cl.num_blocks();
    const int cr = (int)cl.block_rank();
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    constexpr int NW = NT / 32;
    constexpr int GW = W < 8 ? W : 8, NGR = W / GW, HW = DUAL ? W / 2 : W, NGRH = HW / GW;
    constexpr int VEC = 16 / sizeof(T);               // elements per 16-byte vector
    constexpr int CW = (VEC + GW + VEC - 1) / VEC * VEC;  // a candidate: position, live group values
    constexpr bool STAGED = (W * sizeof(T)) % 128 == 0;   // rows of whole 128-byte segments
    constexpr int H = STAGED ? (int)(W * sizeof(T) / 128) : 1, CC = 128 / (int)sizeof(T);
    // in-leaf row moves: at most 2W moved rows in a CTA; at most LEAF_MAX_OTHER
    // other panel columns
    constexpr int MOVE_PW = (2 * W + NW - 1) / NW;
    constexpr int MOVE_CH = LEAF_MAX_OTHER / VEC / 32 > 0 ? LEAF_MAX_OTHER / VEC / 32 : 1;
    const int G = CS * NT;
    const int g = cr * NT + t;

    extern __shared__ __align__(16) unsigned char leaf_smem[];  // 32 rows x 144 bytes per warp (STAGED)
    __shared__ __align__(16) T s_cand[2][NW][CW];              // this CTA's warps, by column parity
    __shared__ __align__(16) T s_slot[2][LEAF_MAX_CS][CW];     // every CTA's winner (clusters), by column parity
    __shared__ __align__(16) T s_right[GW][HW];  // the group's pivot rows: group values, columns to the right
    __shared__ __align__(16) T s_stage[GW][HW];
    __shared__ __align__(16) T s_u[GW][HW];            // columns to the right after the unit triangle
    __shared__ __align__(8) uint64_t s_xbar[2];        // exchange barriers, by column parity
    __shared__ __align__(8) uint64_t s_rbar;           // pivot rows of a group
    __shared__ __align__(8) uint64_t s_mbar;           // DUAL: the first half's pivot rows
    __shared__ int s_piv[W];   // pivots and info stay on chip until the end
    __shared__ int s_info;
    __shared__ int s_skip;     // the call was aborted before this launch
    __shared__ int s_mcnt;
    __shared__ int2 s_mv[2 * W];
    if (t == 0) {
        s_info = 0;
        s_mcnt = 0;
        s_skip = aborted(pn.abort) ? 1 : 0;
        mbar_init(&s_xbar[0], 1);
        mbar_init(&s_xbar[1], 1);
        mbar_init(&s_rbar, 1);
        mbar_init(&s_mbar, 1);
        fence_barrier_init();
    }
    constexpr int PERMAX = CW / VEC;   // 16-byte chunks of a candidate

    // ---- load ----
    T r[R][W];
    int pos[R];  // -1: no row
    const bool vec_ok = (wact == W) && ((ld * (i64)sizeof(T)) % 16 == 0) && (((uintptr_t)P) % 16 == 0);
    unsigned char *tr = leaf_smem + warp * (32 * 144);
    const int trow = lane >> 3, tchk = lane & 7;       // staged transfers: four rows an instruction
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int i = k * G + g;
        pos[k] = i < m ? i : -1;
#pragma unroll
        for (int c = 0; c < W; ++c) r[k][c] = T(0);
    }
    if (STAGED && vec_ok) {
        int4 x[R][H][8];
#pragma unroll
        for (int k = 0; k < R; ++k)
#pragma unroll
            for (int hh = 0; hh < H; ++hh)
#pragma unroll
                for (int it = 0; it < 8; ++it) {
                    const int i = k * G + g - lane + it * 4 + trow;
                    x[k][hh][it] = make_int4(0, 0, 0, 0);
                    if (i < m) x[k][hh][it] = *(const int4 *)(P + (i64)i * ld + hh * CC + tchk * VEC);
                }
#pragma unroll
        for (int k = 0; k < R; ++k)
#pragma unroll
            for (int hh = 0; hh < H; ++hh) {
#pragma unroll
                for (int it = 0; it < 8; ++it) *(int4 *)(tr + (it * 4 + trow) * 144 + tchk * 16) = x[k][hh][it];
                __syncwarp();
                load_row<T, W / H>(&r[k][hh * (W / H)], (const T *)(tr + lane * 144));
                __syncwarp();
            }
    } else {
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (pos[k] >= 0) {
                const T *src = P + (i64)pos[k] * ld;
                if (vec_ok) {
                    load_row<T, W>(r[k], src);
                } else {
#pragma unroll
                    for (int c = 0; c < W; ++c)
                        if (c < wact) r[k][c] = src[c];
                }
            }
        }
    }
    if (DUAL) fence_proxy_async();  // the transfer area takes bulk copies later
    // every CTA's barriers exist before any CTA pushes into them, and
    // every row is read before any CTA stores one at its final position
    if (CS > 1) cl.sync();
    else __syncthreads();
    // CTA 0's reading of the abort word decides for the whole cluster (the
    // word may change between the CTAs' own readings)
    const int skip = (CS > 1) ? *cl.map_shared_rank(&s_skip, 0) : s_skip;
    if (skip) {
        if (CS > 1) cl.sync();  // CTA 0's shared memory stays alive until every CTA read it
        return;
    }
    // An exchange wait that gave up (timeout or the call aborted elsewhere):
    // the CTA leaves the column loop together (at its next barrier), stores
    // nothing and emits no moves, but still meets every cluster barrier.
    bool dead = false;

    // a block the previous launch left in a buffer (see LeafPanel): rows above the leaf
    if (pn.u_rows > 0) {
        const T *us = (const T *)pn.u_src;
        T *ud = (T *)pn.u_dst;
        for (int e = g; e < pn.u_rows * pn.u_cols; e += G) ud[(i64)(e / pn.u_cols) * ld + e % pn.u_cols] = us[e];
    }
    const int q = m < wact ? m : wact;
    // the same shared-memory layout in every CTA: one offset per destination
    const int half = lane & 15;
    const uint32_t to_cta = cluster_map_u32(&s_rbar, half < CS ? half : 0) - smem_u32(&s_rbar);

    // The groups are a rolled loop: the registers rotate by GW slots per group,
    // so the active group always sits in slots 0..GW-1, the unfinished columns
    // behind it and the finished ones last; after all groups the row is back in
    // its order.
    uint32_t rphase = 0;  // exchanges of pivot rows so far
#pragma unroll 1
    for (int s = 0; s < NGR; ++s) {
        const int j0 = s * GW;
        uint32_t live = 0;   // columns of the group with a nonzero pivot
#pragma unroll
        for (int jj = 0; jj < GW; ++jj) {
            const int j = j0 + jj;
            if (j >= q) break;
            const int par = jj & 1;
            const int PER = (1 + GW - jj + VEC - 1) / VEC;  // chunks of this column's candidates
            // (a) this thread's best candidate in column j (_lu_pivot starts from row
            // j with strict '>')
            uint64_t bk = step_key(r[0][jj], pos[0], j);
            int bp = pos[0] >= j ? pos[0] : INT_MAX, bs = 0;
#pragma unroll
            for (int k = 1; k < R; ++k) {
                const uint64_t key = step_key(r[k][jj], pos[k], j);
                if (pos[k] >= j && (bp == INT_MAX || key > bk || (key == bk && pos[k] < bp))) {
                    bk = key;
                    bp = pos[k];
                    bs = k;
                }
            }
            // (b) the warp's winner into shared memory: {position, a_pj, a_p,j+1, ...}
            {
                const uint32_t wm = warp_winner<T>(bk, bp);
                if (wm == 0 ? lane == 0 : ((wm >> lane) & 1)) {
                    T row[CW];
                    if constexpr (sizeof(T) == 4) row[0] = __int_as_float(bp);
                    else row[0] = __longlong_as_double((long long)bp);
#pragma unroll
                    for (int e = 1; e < CW; ++e) {
                        row[e] = T(0);
                        if (jj + e - 1 < GW) {
                            const int c = jj + e - 1 < GW ? jj + e - 1 : 0;
                            row[e] = r[0][c];
#pragma unroll
                            for (int k = 1; k < R; ++k)
                                if (k == bs) row[e] = r[k][c];
                        }
                    }
#pragma unroll
                    for (int e = 0; e < PERMAX; ++e)
                        if (e < PER) store_row<T, VEC>(s_cand[par][warp] + e * VEC, row + e * VEC);
                }
            }
            __syncthreads();
            // key, position and value of the candidate whose first chunk is h
            auto cand_key = [&](ulonglong2 h, int &cp, T &cv) -> uint64_t {
                if constexpr (sizeof(T) == 4) {
                    cp = (int)(uint32_t)h.x;
                    cv = __uint_as_float((uint32_t)(h.x >> 32));
                } else {
                    cp = (int)h.x;
                    cv = __longlong_as_double((long long)h.y);
                }
                return step_key(cv, cp, j);
            };
            // the winner of n candidates, lane l looking at the first chunk h of number l
            auto winner = [&](ulonglong2 h, int n, T &cv) -> int {
                uint64_t ck = 0;
                int cp = INT_MAX;
                if (lane < n) ck = cand_key(h, cp, cv);
                const uint32_t wm = warp_winner<T>(ck, cp);
                return wm ? __ffs(wm) - 1 : 0;
            };
            T cv = T(1), v[CW];
            int wq;
            if (CS > 1) {
                // (c) the CTA's winner to every CTA, warp e its chunk e
                if (!dead) {
                    if (t == 0) mbar_arrive_expect_tx(&s_xbar[par], (uint32_t)(CS * 16 * PER));
                    if (warp < PER) {
                        T w0;
                        ulonglong2 h = make_ulonglong2(0, 0);
                        if (lane < NW) h = *reinterpret_cast<const ulonglong2 *>(s_cand[par][lane]);
                        const int w = winner(h, NW, w0);
                        if (lane < CS)
                            for (int e = warp; e < PER; e += NW)
                                st_async_v4(smem_u32(s_slot[par][cr]) + 16u * e + to_cta,
                                            reinterpret_cast<const uint4 *>(s_cand[par][w])[e],
                                            smem_u32(&s_xbar[par]) + to_cta);
                    }
                    if (!mbar_wait(&s_xbar[par], (uint32_t)((j >> 1) & 1), pn.abort, 1)) dead = true;
                }
                // (d) the winner, the same in every CTA, and its row
                ulonglong2 h = make_ulonglong2(0, 0);
                if (lane < CS) h = *reinterpret_cast<const ulonglong2 *>(s_slot[par][lane]);
                wq = winner(h, CS, cv);
#pragma unroll
                for (int e = 0; e < PERMAX; ++e)
                    if (e < PER) load_row<T, VEC>(v + e * VEC, s_slot[par][wq] + e * VEC);
            } else {
                ulonglong2 h = make_ulonglong2(0, 0);
                if (lane < NW) h = *reinterpret_cast<const ulonglong2 *>(s_cand[par][lane]);
                wq = winner(h, NW, cv);
#pragma unroll
                for (int e = 0; e < PERMAX; ++e)
                    if (e < PER) load_row<T, VEC>(v + e * VEC, s_cand[par][wq] + e * VEC);
            }
            T y = T(0);
            if constexpr (sizeof(T) == 4) y = __shfl_sync(0xffffffffu, 1.0f / cv, wq);
            int wp;
            if constexpr (sizeof(T) == 4) wp = __float_as_int(v[0]);
            else wp = (int)__double_as_longlong(v[0]);
            const T d = v[1];
            const bool ok = !is_zero(d);
            live |= ok ? 1u << jj : 0u;
            if (t == 0) {
                s_piv[j] = wp;
                // zero pivot: info, no elimination (the winner is then row j itself)
                if (!ok && s_info == 0) s_info = j + 1;
            }
            // (e) interchange of positions, scaling, update inside the group
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int p = pos[k];
                pos[k] = p == wp ? j : (p == j ? wp : p);
                if (ok && p >= j && p != wp) {
                    const T l = multiplier(r[k][jj], d, y);
                    r[k][jj] = l;
#pragma unroll
                    for (int c = jj + 1; c < GW; ++c) r[k][c] = fma(-l, v[1 + c - jj], r[k][c]);
                }
            }
        }
        if constexpr (NGR > 1) {
            const int np = min(GW, q - j0);            // pivots of this group
            const int nblk = NGRH - 1 - s % NGRH;      // unfinished groups to the right (of this half)
            if (np > 0 && nblk > 0 && j0 + np < wact) {
                const int rem = nblk * GW, nch = (GW + rem) / VEC;
                // (f) the pivot rows' multipliers and remaining columns to every CTA
                if (CS > 1 && t == 0 && !dead) mbar_arrive_expect_tx(&s_rbar, (uint32_t)(np * nch * 16));
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    const int kk = pos[k] - j0;
                    const bool own = pos[k] >= j0 && kk < np;
                    if (own) {
                        T *dst = (CS > 1) ? s_stage[kk] : s_right[kk];
#pragma unroll
                        for (int b = 0; b < NGRH; ++b)
                            if (b <= nblk) store_row<T, GW>(dst + b * GW, &r[k][b * GW]);
                    }
                    if (CS > 1) {
                        uint32_t om = __ballot_sync(0xffffffffu, own);
                        while (om) {
                            const int src = __ffs(om) - 1;
                            om &= om - 1;
                            const int ks = __shfl_sync(0xffffffffu, kk, src);
                            __syncwarp();
                            if (half < CS && !dead)
                                for (int c = lane >> 4; c < nch; c += 2)
                                    st_async_v4(smem_u32(s_right[ks]) + 16u * c + to_cta,
                                                reinterpret_cast<const uint4 *>(s_stage[ks])[c],
                                                smem_u32(&s_rbar) + to_cta);
                        }
                    }
                }
                if (CS > 1) {
                    if (warp == 0 && !dead && !mbar_wait(&s_rbar, rphase & 1u, pn.abort, 1)) dead = true;
                    ++rphase;
                } else {
                    __syncthreads();
                }
                // (g) their unit triangle, one column per lane
                const bool full = live == (1u << GW) - 1;
                if (warp == 0 && lane < rem) {
                    T x[GW];
#pragma unroll
                    for (int k = 0; k < GW; ++k) x[k] = k < np ? s_right[k][GW + lane] : T(0);
                    if (full) {
#pragma unroll
                        for (int p = 0; p < GW; ++p)
#pragma unroll
                            for (int k = p + 1; k < GW; ++k) x[k] = fma(-s_right[k][p], x[p], x[k]);
                    } else {
                        for (int p = 0; p < np; ++p) {
                            if (!((live >> p) & 1)) continue;
#pragma unroll
                            for (int k = 1; k < GW; ++k) {
                                T xp = x[0];
#pragma unroll
                                for (int e = 1; e < GW; ++e) xp = e == p ? x[e] : xp;
                                if (k > p && k < np) x[k] = fma(-s_right[k][p], xp, x[k]);
                            }
                        }
                    }
#pragma unroll
                    for (int k = 0; k < GW; ++k) s_u[k][lane] = x[k];
                }
                __syncthreads();
                // (h) the group's updates of the remaining columns: the rows below the
                // pivots take them all; a pivot row's own are its row of the triangle's
                // solution
                bool act[R];
                bool any = false;
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    act[k] = pos[k] >= j0 + np;
                    any = any || act[k];
                }
                const bool warp_any = __any_sync(0xffffffffu, any);
#pragma unroll
                for (int b = 0; b < NGRH - 1; ++b) {
                    if (b < nblk) {
                        if (warp_any) {
                            T nv[R][GW];
#pragma unroll
                            for (int k = 0; k < R; ++k)
#pragma unroll
                                for (int c = 0; c < GW; ++c) nv[k][c] = r[k][(b + 1) * GW + c];
                            if (full) {
#pragma unroll
                                for (int p = 0; p < GW; ++p) {
                                    T u[GW];
                                    load_row<T, GW>(u, &s_u[p][b * GW]);
#pragma unroll
                                    for (int k = 0; k < R; ++k)
#pragma unroll
                                        for (int c = 0; c < GW; ++c) nv[k][c] = fma(-r[k][p], u[c], nv[k][c]);
                                }
                            } else {
#pragma unroll
                                for (int p = 0; p < GW; ++p) {
                                    if (!((live >> p) & 1)) continue;
                                    T u[GW];
                                    load_row<T, GW>(u, &s_u[p][b * GW]);
#pragma unroll
                                    for (int k = 0; k < R; ++k)
#pragma unroll
                                        for (int c = 0; c < GW; ++c) nv[k][c] = fma(-r[k][p], u[c], nv[k][c]);
                                }
                            }
#pragma unroll
                            for (int k = 0; k < R; ++k)
#pragma unroll
                                for (int c = 0; c < GW; ++c)
                                    if (act[k]) r[k][(b + 1) * GW + c] = nv[k][c];
                        }
#pragma unroll
                        for (int k = 0; k < R; ++k) {
                            const int kk = pos[k] - j0;
                            if (pos[k] >= j0 && kk < np) load_row<T, GW>(&r[k][(b + 1) * GW], &s_u[kk][b * GW]);
                        }
                    }
                }
            }
            // the finished group moves behind the unfinished columns
#pragma unroll
            for (int k = 0; k < R; ++k) {
                T f[GW];
#pragma unroll
                for (int c = 0; c < GW; ++c) f[c] = r[k][c];
#pragma unroll
                for (int c = 0; c < W - GW; ++c) r[k][c] = r[k][c + GW];
#pragma unroll
                for (int c = 0; c < GW; ++c) r[k][W - GW + c] = f[c];
            }
        }
        if constexpr (DUAL) {
            if (s == NGRH - 1) {
                // slots 0..HW-1 hold the second half's columns, slots HW.. the first's.
                // The rows' transfer area is free until the end: X (U12, HW x HW), the
                // pivot rows' multipliers, and the rows on their way out.
                constexpr int LP = HW + 2;
                static_assert(!DUAL || (R == 1 && (2 * HW + LP + HW) * HW * (int)sizeof(T) <= NW * 32 * 144), "mid-step area");
                T *X = (T *)leaf_smem;                 // [HW][HW]
                T *Ls = X + HW * HW;                   // [HW][LP]
                T *st = Ls + HW * LP;                  // [HW][W]
                __syncthreads();
                if (CS > 1 && t == 0 && !dead) mbar_arrive_expect_tx(&s_mbar, (uint32_t)(HW * W * sizeof(T)));
                const int kk = pos[0];
                const bool own = kk >= 0 && kk < HW;
                if (own) {
                    store_row<T, HW>(CS > 1 ? st + kk * W : Ls + kk * LP, &r[0][HW]);
                    store_row<T, HW>(CS > 1 ? st + kk * W + HW : X + kk * HW, &r[0][0]);
                }
                if (CS > 1) {
                    // a row's two halves to every CTA, one bulk copy each
                    uint32_t om = __ballot_sync(0xffffffffu, own);
                    if (own) fence_proxy_async();
                    __syncwarp();
                    while (om) {
                        const int src = __ffs(om) - 1;
                        om &= om - 1;
                        const int ks = __shfl_sync(0xffffffffu, kk, src);
                        const bool lo = lane < 16;
                        if (half < CS && !dead)
                            bulk_to_cluster(smem_u32(lo ? Ls + ks * LP : X + ks * HW) + to_cta,
                                            smem_u32(st + ks * W + (lo ? 0 : HW)), HW * sizeof(T),
                                            smem_u32(&s_mbar) + to_cta);
                    }
                    if (!dead && !mbar_wait(&s_mbar, 0u, pn.abort, 1)) dead = true;
                }
                __syncthreads();
                // U12 in the order of the recursive solve: halves down to 8-row leaves
#pragma unroll 1
                for (int a = 0; a < HW; a += 8) {
                    if (t < HW) {
                        T x[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) x[u] = X[(a + u) * HW + t];
#pragma unroll
                        for (int u = 1; u < 8; ++u)
#pragma unroll
                            for (int p = 0; p < u; ++p) x[u] = fma(-Ls[(a + u) * LP + a + p], x[p], x[u]);
#pragma unroll
                        for (int u = 1; u < 8; ++u) X[(a + u) * HW + t] = x[u];
                    }
                    __syncthreads();
                    // rows [a + 8, hi) -= L[rows, lo:a+8] X[lo:a+8]
                    const int lo = a == 8 ? 0 : a, hi = a == 8 ? HW : a == 24 ? 0 : a + 16;
                    for (int i = a + 8 + t / HW; i < hi; i += NT / HW) {
                        T acc = T(0);
#pragma unroll 8
                        for (int p = lo; p < a + 8; ++p) acc = fma(Ls[i * LP + p], X[p * HW + t % HW], acc);
                        X[i * HW + t % HW] -= acc;
                    }
                    __syncthreads();
                }
                // the rows below: C - s; the pivot rows' own columns are U12's rows
                if (own) {
                    load_row<T, HW>(&r[0][0], X + kk * HW);
                } else {
#pragma unroll 1
                    for (int b = 0; b < NGRH; ++b) {  // rotating, as the groups do
                        T acc[GW];
#pragma unroll
                        for (int c = 0; c < GW; ++c) acc[c] = T(0);
#pragma unroll
                        for (int p = 0; p < HW; ++p) {
                            T u[GW];
                            load_row<T, GW>(u, X + p * HW + b * GW);
#pragma unroll
                            for (int c = 0; c < GW; ++c) acc[c] = fma(r[0][HW + p], u[c], acc[c]);
                        }
#pragma unroll
                        for (int c = 0; c < GW; ++c) acc[c] = r[0][c] - acc[c];
#pragma unroll
                        for (int c = 0; c < HW - GW; ++c) r[0][c] = r[0][c + GW];
#pragma unroll
                        for (int c = 0; c < GW; ++c) r[0][HW - GW + c] = acc[c];
                    }
                }
            }
        }
    }
    // pivots and info, written once
    dead = __syncthreads_or(dead);
    if (!dead && cr == 0 && t < q) ipiv[gofs + t] = gofs + s_piv[t] + 1;
    if (!dead && cr == 0 && t == 0 && s_info != 0 && *info == 0) *info = gofs + s_info;

    // ---- store every row at its final position ----
    const bool inleaf = pn.nother > 0 || pn.map;  // the moves are applied here, not by a later launch
    if (!dead) {
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int i = k * G + g;
            if (pos[k] >= 0 && pos[k] != i) {
                if (inleaf) {
                    const int slot = atomicAdd(&s_mcnt, 1);
                    s_mv[slot] = make_int2(pos[k], i);
                } else {
                    const int slot = atomicAdd(nmoves, 1);
                    moves[2 * slot] = pos[k];
                    moves[2 * slot + 1] = i;
                }
            }
            if (STAGED && vec_ok) {
#pragma unroll
                for (int hh = 0; hh < H; ++hh) {
                    store_row<T, W / H>((T *)(tr + lane * 144), &r[k][hh * (W / H)]);
                    __syncwarp();
#pragma unroll
                    for (int it = 0; it < 8; ++it) {
                        const int dst = __shfl_sync(0xffffffffu, pos[k], it * 4 + trow);
                        if (dst >= 0)
                            *(int4 *)(P + (i64)dst * ld + hh * CC + tchk * VEC) =
                                *(const int4 *)(tr + (it * 4 + trow) * 144 + tchk * 16);
                    }
                    __syncwarp();
                }
            } else if (pos[k] >= 0) {
                T *dst = P + (i64)pos[k] * ld;
                if (vec_ok) {
                    store_row<T, W>(dst, r[k]);
                } else {
#pragma unroll
                    for (int c = 0; c < W; ++c)
                        if (c < wact) dst[c] = r[k][c];
                }
            }
        }
    }
    if (inleaf) {
        // The leaf's row interchanges on the panel's other columns, and on the
        // panel row map, done here rather than by separate launches: each CTA
        // reads the segments of its own moved rows, all CTAs meet, and each
        // writes them at their final positions (one warp per moved row, 16 bytes
        // a lane where the panel's column ranges allow it).
        int mapv[R];
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int i = k * G + g;
            mapv[k] = (!dead && pn.map && pos[k] >= 0 && pos[k] != i) ? pn.map[pn.map_off + i] : 0;
        }
        __syncthreads();
        const int cnt = s_mcnt;
        const int nother = pn.nother;
        T *const base = P - pn.leaf_c0;
        const bool mvec = ((ld * (i64)sizeof(T)) % 16 == 0) && (((uintptr_t)base) % 16 == 0) &&
                          ((pn.left_n | pn.pc_lo | pn.right_lo | nother) % VEC == 0);
        if (mvec) {
            const int nv = nother / VEC;
            int off[MOVE_CH];
#pragma unroll
            for (int ci = 0; ci < MOVE_CH; ++ci) {
                const int oc = (ci * 32 + lane) * VEC;
                off[ci] = ci * 32 + lane >= nv ? -1 : (oc < pn.left_n ? pn.pc_lo + oc : pn.right_lo + (oc - pn.left_n));
            }
            int4 vals[MOVE_PW][MOVE_CH];
#pragma unroll
            for (int mi = 0; mi < MOVE_PW; ++mi) {
                const int mv = warp + mi * NW;
                if (mv < cnt) {
                    const T *srow = base + (i64)s_mv[mv].y * ld;
#pragma unroll
                    for (int ci = 0; ci < MOVE_CH; ++ci)
                        if (off[ci] >= 0) vals[mi][ci] = *(const int4 *)(srow + off[ci]);
                }
            }
            if (CS > 1) cl.sync();
            else __syncthreads();
#pragma unroll
            for (int mi = 0; mi < MOVE_PW; ++mi) {
                const int mv = warp + mi * NW;
                if (mv < cnt) {
                    T *drow = base + (i64)s_mv[mv].x * ld;
#pragma unroll
                    for (int ci = 0; ci < MOVE_CH; ++ci)
                        if (off[ci] >= 0) *(int4 *)(drow + off[ci]) = vals[mi][ci];
                }
            }
        } else {
            constexpr int SCH = LEAF_MAX_OTHER / 32;
            T vals[MOVE_PW][SCH];
#pragma unroll
            for (int mi = 0; mi < MOVE_PW; ++mi) {
                const int mv = warp + mi * NW;
                if (mv < cnt) {
                    const T *srow = base + (i64)s_mv[mv].y * ld;
#pragma unroll
                    for (int ci = 0; ci < SCH; ++ci) {
                        const int oc = ci * 32 + lane;
                        if (oc < nother) vals[mi][ci] = srow[oc < pn.left_n ? pn.pc_lo + oc : pn.right_lo + (oc - pn.left_n)];
                    }
                }
            }
            if (CS > 1) cl.sync();
            else __syncthreads();
#pragma unroll
            for (int mi = 0; mi < MOVE_PW; ++mi) {
                const int mv = warp + mi * NW;
                if (mv < cnt) {
                    T *drow = base + (i64)s_mv[mv].x * ld;
#pragma unroll
                    for (int ci = 0; ci < SCH; ++ci) {
                        const int oc = ci * 32 + lane;
                        if (oc < nother) drow[oc < pn.left_n ? pn.pc_lo + oc : pn.right_lo + (oc - pn.left_n)] = vals[mi][ci];
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int i = k * G + g;
            if (!dead && pn.map && pos[k] >= 0 && pos[k] != i) pn.map[pn.map_off + pos[k]] = mapv[k];
        }
    } else if (CS > 1) {
        // every push into a CTA that gave up has landed before its shared memory goes
        cl.sync();
    }
}


template <typename T> int leaf_width_for(i64 m);
template <> int leaf_width_for<double>(i64 m) {
    const i64 cap = (i64)LEAF_MAX_CS * LEAF_NT;  // rows per slot
    if (m <= cap * 1) return 32;
    if (m <= cap * 2) return 16;
    if (m <= cap * 4) return 8;
    if (m <= cap * 8) return 4;
    return 0;
}
template <> int leaf_width_for<float>(i64 m) {
    const i64 cap = (i64)LEAF_MAX_CS * LEAF_NT;
    if (m <= cap * 2) return 32;
    if (m <= cap * 4) return 16;
    if (m <= cap * 8) return 8;
    return 0;
}

template <typename T, int W, int R, int NT = LEAF_NT, bool DUAL = false>
static void launch_leaf_wr(T *P, i64 ld, i64 m, int w, i64 gofs, int64_t *ipiv, int64_t *info,
                           int *moves, int *nmoves, cudaStream_t s, LeafPanel pn) {
    const i64 per_cta = (i64)NT * R;
    int need = (int)((m + per_cta - 1) / per_cta);
    const int cs = need;
    auto kern = k_leaf_lu<T, W, R, NT, DUAL>;
    if (cs > 8) OXI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(NT);
    constexpr int smem = (W * sizeof(T)) % 128 == 0 ? (NT / 32) * 32 * 144 : 0;
    if (smem > 0) set_max_dyn_smem((const void *)kern, smem);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (pn.nother > LEAF_MAX_OTHER)
        throw CudaError{cudaErrorInvalidValue, "panel too wide for the in-leaf row moves"};
    pn.abort = cur_abort();
    ProfScope ps(KC_LEAF, s, 0.0, 2.0 * (double)m * w * sizeof(T));
    OXI_CUDA(cudaLaunchKernelEx(&cfg, kern, P, ld, (int)m, w, gofs, ipiv, info, moves, nmoves, pn));
    count_launch();
}

// Threads and rows a thread by height, kernel alone, us on one B200: 256 threads of
// one row while 16 CTAs hold the rows (FP64 1024 rows 44 against 52 with 512 threads, 4096 rows 47
// against 54; FP32 256 rows 27 against 33, 4096 rows 41 against 43, with two rows a
// thread 47): fewer warps to reduce over, twice the registers.  Above 4096 rows 512
// threads (8192 rows: FP64 56 against 60 with 256 threads of two rows, FP32 45
// against 50), from 8193 FP32 rows two a thread (16384: 55, 70 with four in 256).
// (257 to 512 rows in one CTA of 512 threads: FP64 39 against 44, FP32 31 against
// 40, and no difference to a whole solve, so no rule of their own.)
// The cluster has as many CTAs as the rows need, not the next power of two: the
// exchange takes 413 cycles among 2 CTAs and 746 among 16.
template <typename T>
void launch_leaf(T *P, i64 ld, i64 m, int w, i64 gofs, int64_t *ipiv, int64_t *info, int *moves,
                 int *nmoves, int leafw, cudaStream_t s, LeafPanel pn) {
    if constexpr (sizeof(T) == 8) {
        if (leafw == 64) launch_leaf_wr<T, 64, 1, 256, true>(P, ld, m, w, gofs, ipiv, info, moves, nmoves, s, pn);
        else if (leafw == 32 && m <= LEAF_MAX_CS * 256) launch_leaf_wr<T, 32, 1, 256>(P, ld, m, w, gofs, ipiv, info, moves, nmoves, s, pn);
        else if (leafw == 32) launch_leaf_wr<T, 32, 1>(P, ld, m, w, gofs, ipiv, info, moves, nmoves, s, pn);
        else if (leafw == 16) launch_leaf_wr<T, 16, 2>(P, ld, m, w, gofs, ipiv, info, moves, nmoves, s, pn);
        else if (leafw == 8) launch_leaf_wr<T, 8, 4>(P, ld, m, w, gofs, ipiv, info, moves, nmoves, s, pn);
        else launch_leaf_wr<T, 4, 8>(P, ld, m, w, gofs, ipiv, info, moves, nmoves, s, pn);
    } else {
        if (leafw == 32) {
            if (m <= LEAF_MAX_CS * 256) launch_leaf_wr<T, 32, 1, 256>(P, ld, m, w, gofs, ipiv, info, moves, nmoves, s, pn);
            else if (m <= LEAF_MAX_CS * LEAF_NT) launch_leaf_wr<T, 32, 1>(P, ld, m, w, gofs, ipiv, info, moves, nmoves, s, pn);
            else launch_leaf_wr<T, 32, 2>(P, ld, m, w, gofs, ipiv, info, moves, nmoves, s, pn);
        } else if (leafw == 16) {
            launch_leaf_wr<T, 16, 4>(P, ld, m, w, gofs, ipiv, info, moves, nmoves, s, pn);
        } else {
            launch_leaf_wr<T, 8, 8>(P, ld, m, w, gofs, ipiv, info, moves, nmoves, s, pn);
        }
    }
}
template void launch_leaf<double>(double *, i64, i64, int, i64, int64_t *, int64_t *, int *, int *, int, cudaStream_t, LeafPanel);
template void launch_leaf<float>(float *, i64, i64, int, i64, int64_t *, int64_t *, int *, int *, int, cudaStream_t, LeafPanel);

// ---------------------------------------------------------------------------
// Row moves: W[r0 + dst][c] <- W[r0 + src][c] for every move, all sources read
// before any destination is written.  One thread per column: the moves of a
// column are private to its thread, so no synchronisation is needed, and a warp
// touches 32 contiguous elements of each row (coalesced).
// ---------------------------------------------------------------------------
constexpr int MAX_MOVES = 64;

template <typename T>
__global__ void k_rowmoves(T *__restrict__ W, i64 ld, i64 r0, const int *__restrict__ moves,
                           const int *__restrict__ nmoves, i64 c_lo, i64 c_hi, i64 skip_lo,
                           i64 skip_hi) {
    const i64 c = c_lo + (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= c_hi || (c >= skip_lo && c < skip_hi)) return;
    const int cnt = min(*nmoves, MAX_MOVES);
    T tmp[MAX_MOVES];
    T *base = W + r0 * ld + c;
#pragma unroll
    for (int e = 0; e < MAX_MOVES; ++e)
        if (e < cnt) tmp[e] = base[(i64)moves[2 * e + 1] * ld];
#pragma unroll
    for (int e = 0; e < MAX_MOVES; ++e)
        if (e < cnt) base[(i64)moves[2 * e] * ld] = tmp[e];
}

template <typename T>
void launch_rowmoves(T *W, i64 ld, i64 r0, const int *moves, const int *nmoves, i64 c_lo, i64 c_hi,
                     i64 skip_lo, i64 skip_hi, cudaStream_t s) {
    if (c_hi <= c_lo) return;
    const int nt = 128;
    const i64 cols = c_hi - c_lo;
    ProfScope ps(KC_ROWMOVES, s, 0.0, 0.0);
    k_rowmoves<T><<<(unsigned)((cols + nt - 1) / nt), nt, 0, s>>>(W, ld, r0, moves, nmoves, c_lo, c_hi,
                                                                   skip_lo, skip_hi);
    OXI_LAUNCH_CHECK();
}
template void launch_rowmoves<double>(double *, i64, i64, const int *, const int *, i64, i64, i64, i64, cudaStream_t);
template void launch_rowmoves<float>(float *, i64, i64, const int *, const int *, i64, i64, i64, i64, cudaStream_t);

// ---------------------------------------------------------------------------
// Panel-level composition of the leaves' row permutations.  map[p] = the row
// (relative to the panel's first row) whose data sits at position p; each
// leaf's moves compose into it, and at the end of the panel the positions with
// map[p] != p form one move list for all the columns outside the panel.
// ---------------------------------------------------------------------------
// identity row map of a panel; also zeroes the panel's move-list count (no
// separate memset on the panel's critical path)
__global__ void k_rowmap_init(int *__restrict__ map, int len, int *__restrict__ listcnt) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < len) map[p] = p;
    if (p == 0) *listcnt = 0;
}
__global__ void k_rowmap_extract(const int *__restrict__ map, int len, int *__restrict__ list,
                                 int *__restrict__ cnt) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= len) return;
    const int src = map[p];
    if (src != p) {
        const int slot = atomicAdd(cnt, 1);
        list[2 * slot] = p;
        list[2 * slot + 1] = src;
    }
}

// All sources of a CTA's column slab are staged in shared memory before any
// destination is written, so cycles of the permutation are safe.  Each thread
// owns one 16-byte vector column of the slab and walks the move list with a
// stride, 8 independent loads in flight.
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) k_rowmoves_big(T *__restrict__ W, i64 ld, i64 r0,
                                                      const int *__restrict__ list,
                                                      const int *__restrict__ cnt_ptr, int maxcnt,
                                                      i64 c_lo, i64 c_hi, int cpc) {
    extern __shared__ __align__(16) unsigned char rm_smem[];
    constexpr int V = VEC ? 16 / (int)sizeof(T) : 1;
    using VT = typename std::conditional<VEC, int4, T>::type;
    VT *buf = reinterpret_cast<VT *>(rm_smem);
    const int cnt = min(*cnt_ptr, maxcnt);
    const i64 cbase = c_lo + (i64)blockIdx.x * cpc;
    const int cols = (int)((c_hi - cbase) < (i64)cpc ? (c_hi - cbase) : (i64)cpc);
    if (cols <= 0 || cnt == 0) return;
    const int nv = cpc / V;                 // vector columns per slab
    const int v = threadIdx.x % nv, g = threadIdx.x / nv, G = blockDim.x / nv;
    const bool full = (v + 1) * V <= cols;  // this thread's vector lies inside the slab
    const bool part = !full && v * V < cols;
    T *base = W + r0 * ld + cbase + (i64)v * V;
#pragma unroll 8
    for (int e = g; e < cnt; e += G) {
        const T *src = base + (i64)list[2 * e + 1] * ld;
        if (full) {
            buf[(i64)e * nv + v] = *reinterpret_cast<const VT *>(src);
        } else if (part) {
            T tmp[V];
            for (int u = 0; u < V; ++u) tmp[u] = (v * V + u < cols) ? src[u] : T(0);
            buf[(i64)e * nv + v] = *reinterpret_cast<VT *>(tmp);
        }
    }
    __syncthreads();
#pragma unroll 8
    for (int e = g; e < cnt; e += G) {
        T *dst = base + (i64)list[2 * e] * ld;
        if (full) {
            *reinterpret_cast<VT *>(dst) = buf[(i64)e * nv + v];
        } else if (part) {
            const VT val = buf[(i64)e * nv + v];
            const T *tv = reinterpret_cast<const T *>(&val);
            for (int u = 0; u < V; ++u)
                if (v * V + u < cols) dst[u] = tv[u];
        }
    }
}

void launch_rowmap_init(int *map, i64 len, int *listcnt, cudaStream_t s) {
    if (len <= 0) return;
    k_rowmap_init<<<(unsigned)((len + 255) / 256), 256, 0, s>>>(map, (int)len, listcnt);
    OXI_LAUNCH_CHECK();
}
void launch_rowmap_extract(const int *map, i64 len, int *list, int *cnt, cudaStream_t s) {
    if (len <= 0) return;
    k_rowmap_extract<<<(unsigned)((len + 255) / 256), 256, 0, s>>>(map, (int)len, list, cnt);
    OXI_LAUNCH_CHECK();
}
template <typename T>
void launch_rowmoves_big(T *W, i64 ld, i64 r0, const int *list, const int *cnt, int maxcnt, i64 c_lo,
                         i64 c_hi, cudaStream_t s) {
    if (c_hi <= c_lo || maxcnt <= 0) return;
    const int V = 16 / (int)sizeof(T);
    const bool vec = ((uintptr_t)W % 16 == 0) && ((ld * (i64)sizeof(T)) % 16 == 0) && (c_lo % V == 0);
    // slab of 64 columns (FP32) / 32 (FP64): 16 or 8 threads per row, 16 or 32 rows at once
    int cpc = vec ? 16 * V : 64;
    while (cpc > V && (size_t)maxcnt * cpc * sizeof(T) > 160 * 1024) cpc /= 2;
    // few columns (the next panel's, on the panels' critical path): slabs down to 64
    // bytes, so that the moves spread over more SMs (n = 16384, 256 columns: 4 CTAs
    // took 30 us)
    while (vec && (c_hi - c_lo + cpc - 1) / cpc < 32 && cpc * (int)sizeof(T) > 64) cpc /= 2;
    const size_t smem = (size_t)maxcnt * cpc * sizeof(T);
    constexpr int kMaxSmem = 200 * 1024;  // the kernel's one limit (see set_max_dyn_smem)
    if (smem > (size_t)kMaxSmem) throw CudaError{cudaErrorInvalidValue, "panel too wide for the row moves"};
    ProfScope ps(KC_ROWMOVES, s, 0.0, 2.0 * maxcnt * (double)(c_hi - c_lo) * sizeof(T));
    const i64 blocks = (c_hi - c_lo + cpc - 1) / cpc;
    if (vec) {
        set_max_dyn_smem((const void *)k_rowmoves_big<T, true>, kMaxSmem);
        k_rowmoves_big<T, true><<<(unsigned)blocks, 256, smem, s>>>(W, ld, r0, list, cnt, maxcnt, c_lo, c_hi, cpc);
    } else {
        set_max_dyn_smem((const void *)k_rowmoves_big<T, false>, kMaxSmem);
        k_rowmoves_big<T, false><<<(unsigned)blocks, 256, smem, s>>>(W, ld, r0, list, cnt, maxcnt, c_lo, c_hi, cpc);
    }
    OXI_LAUNCH_CHECK();
}
template void launch_rowmoves_big<double>(double *, i64, i64, const int *, const int *, int, i64, i64, cudaStream_t);
template void launch_rowmoves_big<float>(float *, i64, i64, const int *, const int *, int, i64, i64, cudaStream_t);

// ---------------------------------------------------------------------------
// TRSM leaf: B (t x N) <- L^-1 B with L unit lower (t <= 32), row-major.  One
// thread per right-hand-side column, L staged in shared memory; the order is
// the reference leaf's (src/blas/level3.jl:309-321): s = b_i, then
// s = muladd(-L_ip, b_p, s) for p = 1..i-1.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_trsm_leaf(const T *__restrict__ L, i64 ldl, T *__restrict__ B, i64 ldb, int t,
                            i64 N) {
    __shared__ T sL[32][33];
    for (int e = threadIdx.x; e < t * t; e += blockDim.x) {
        const int i = e / t, p = e - i * t;
        sL[i][p] = L[(i64)i * ldl + p];
    }
    __syncthreads();
    const i64 c = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= N) return;
    T x[32];
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (i < t) x[i] = B[(i64)i * ldb + c];
#pragma unroll
    for (int i = 1; i < 32; ++i) {
        if (i < t) {
            T s = x[i];
#pragma unroll
            for (int p = 0; p < i; ++p) s = fma(-sL[i][p], x[p], s);
            x[i] = s;
        }
    }
#pragma unroll
    for (int i = 1; i < 32; ++i)
        if (i < t) B[(i64)i * ldb + c] = x[i];
}

// Column-oriented (right-looking) leaf for the tensor-core engine: once x_p is
// final, x_i -= L_ip x_p for all i > p -- t-p independent FMAs per step instead
// of one dependent chain per row.  One right-hand-side column per thread.
template <typename T>
__global__ void k_trsm_leaf_col(const T *__restrict__ L, i64 ldl, T *__restrict__ B, i64 ldb, int t,
                                i64 N) {
    __shared__ T sL[32][33];
    for (int e = threadIdx.x; e < t * t; e += blockDim.x) {
        const int i = e / t, p = e - i * t;
        sL[i][p] = L[(i64)i * ldl + p];
    }
    __syncthreads();
    const i64 c = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= N) return;
    T x[32];
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (i < t) x[i] = B[(i64)i * ldb + c];
#pragma unroll
    for (int p = 0; p < 31; ++p) {
        if (p + 1 < t) {
            const T xp = x[p];
#pragma unroll
            for (int i = p + 1; i < 32; ++i)
                if (i < t) x[i] = fma(-sL[i][p], xp, x[i]);
        }
    }
#pragma unroll
    for (int i = 1; i < 32; ++i)
        if (i < t) B[(i64)i * ldb + c] = x[i];
}

template <typename T>
void launch_trsm_leaf(const T *L, i64 ldl, T *B, i64 ldb, int t, i64 N, cudaStream_t s,
                      bool ref_order) {
    if (t <= 1 || N <= 0) return;  // a unit 1x1 triangle is the identity
    const int nt = 128;
    ProfScope ps(KC_TRSM_LEAF, s, (double)t * t * N, 2.0 * (double)t * N * sizeof(T));
    if (ref_order) {
        k_trsm_leaf<T><<<(unsigned)((N + nt - 1) / nt), nt, 0, s>>>(L, ldl, B, ldb, t, N);
    } else {
        k_trsm_leaf_col<T><<<(unsigned)((N + nt - 1) / nt), nt, 0, s>>>(L, ldl, B, ldb, t, N);
    }
    OXI_LAUNCH_CHECK();
}
// ---------------------------------------------------------------------------
// Fused blocked TRSM (tensor-core engine): B (t x N) <- L^-1 B for a unit lower
// L with t <= 256, one CTA per 32-column strip of B kept in shared memory for
// the whole solve.  Block row I: X_I -= sum_{J<I} L_IJ X_J (L blocks staged
// through shared memory), then the 32 x 32 diagonal block by warp-shuffle
// substitution (lane = row, one warp per 4 columns).  One launch replaces the
// recursive halving's leaves and GEMMs.
// ---------------------------------------------------------------------------
constexpr int TF_TB = 32, TF_TMAX = 256;

// Right-looking: for each 32-row block J, solve its 32 x 32 diagonal block by
// warp-shuffle substitution (lane = row, one warp per CW/8 columns), then update
// all rows below with that block's solution in one pass (L column block staged in
// shared memory, four columns per thread).  CW = 32 columns per CTA for wide
// right-hand sides, 8 for narrow ones (a panel's U12): four times the CTAs, a
// quarter of the dependent chain per CTA.
template <typename T, int CW>
__global__ void __launch_bounds__(256) k_trsm_fused(const T *__restrict__ L, i64 ldl, T *__restrict__ B,
                                                    i64 ldb, int t, i64 N) {
    constexpr int NG = CW / 4, RG = 256 / NG;                 // column groups of 4, row groups
    constexpr int QMAX = (TF_TMAX - TF_TB + RG - 1) / RG;     // rows per thread below a block
    constexpr int CPW = CW / 8;                               // chain columns per warp
    extern __shared__ __align__(16) unsigned char tf_smem[];
    T(*X)[CW + 1] = reinterpret_cast<T(*)[CW + 1]>(tf_smem);
    T(*Lc)[TF_TB + 1] = reinterpret_cast<T(*)[TF_TB + 1]>(tf_smem + sizeof(T) * TF_TMAX * (CW + 1));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const i64 c0 = (i64)blockIdx.x * CW;
    const int cols = (int)((N - c0) < CW ? (N - c0) : CW);
    for (int e = tid; e < t * CW; e += 256) {
        const int i = e / CW, c = e % CW;
        X[i][c] = (c < cols) ? B[(i64)i * ldb + c0 + c] : T(0);
    }
    const int nblk = (t + TF_TB - 1) / TF_TB;
    const int cq = (tid % NG) * 4, rq = tid / NG;  // update mapping: rows rq + RG q, columns cq..cq+3
    for (int J = 0; J < nblk; ++J) {
        const int j0 = J * TF_TB, jrows = min(TF_TB, t - j0);
        const int rb = j0 + jrows, nrem = t - rb;  // rows below the block
        // stage L[j0.., j0..j0+31] (diagonal block first, then the rows below)
        for (int e = tid; e < (t - j0) * TF_TB; e += 256) {
            const int rr = e / TF_TB, pp = e % TF_TB;
            Lc[rr][pp] = (pp < jrows) ? L[(i64)(j0 + rr) * ldl + j0 + pp] : T(0);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < CPW; ++q) {
            const int c = warp * CPW + q;
            T x = (lane < jrows) ? X[j0 + lane][c] : T(0);
            for (int p = 0; p < jrows - 1; ++p) {
                const T xp = __shfl_sync(0xffffffffu, x, p);
                if (lane > p) x = fma(-Lc[lane][p], xp, x);
            }
            if (lane < jrows) X[j0 + lane][c] = x;
        }
        __syncthreads();
        if (nrem > 0) {
            T acc[QMAX][4];
#pragma unroll
            for (int q = 0; q < QMAX; ++q)
#pragma unroll
                for (int u = 0; u < 4; ++u) acc[q][u] = T(0);
#pragma unroll 4
            for (int p = 0; p < jrows; ++p) {
                const T x0 = X[j0 + p][cq], x1 = X[j0 + p][cq + 1], x2 = X[j0 + p][cq + 2], x3 = X[j0 + p][cq + 3];
#pragma unroll
                for (int q = 0; q < QMAX; ++q) {
                    const int r = rq + RG * q;
                    if (r < nrem) {
                        const T l = Lc[TF_TB + r][p];
                        acc[q][0] = fma(l, x0, acc[q][0]);
                        acc[q][1] = fma(l, x1, acc[q][1]);
                        acc[q][2] = fma(l, x2, acc[q][2]);
                        acc[q][3] = fma(l, x3, acc[q][3]);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < QMAX; ++q) {
                const int r = rq + RG * q;
                if (r < nrem) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) X[rb + r][cq + u] -= acc[q][u];
                }
            }
        }
        __syncthreads();
    }
    for (int e = tid; e < t * CW; e += 256) {
        const int i = e / CW, c = e % CW;
        if (c < cols) B[(i64)i * ldb + c0 + c] = X[i][c];
    }
}

// The narrow FP32 solve (a panel's U12 in the mixed factor, on the panels'
// critical path): 8 columns per CTA, all diagonal blocks in shared memory from the
// start, each block column of L requested one block ahead; a block row's solve is
// a substitution, a warp per column with its row of the block in registers.
// Bound: latency of the block rows (a 31-step chain of shuffles, a 32-step one of
// products, three barriers each).  By products with inverted diagonal blocks the
// chain is shorter (the 125 solves of the n = 16384 mixed factor 7.4 ms instead of
// 7.65), but the residual reached 258 roundings where substitution leaves 2
// (restated in NumPy, fourth difference matrix of order 1024).
constexpr int TN_CW = 8;
struct TrsmNarrowSmem {
    float D[TF_TMAX / TF_TB][TF_TB][TF_TB + 1];
    float L[TF_TMAX - TF_TB][TF_TB + 1];
    float X[TF_TMAX][TN_CW];
};
__global__ void __launch_bounds__(256) k_trsm_narrow(const float *__restrict__ L, i64 ldl, float *__restrict__ B, i64 ldb,
                                                  int t, i64 N) {
    extern __shared__ __align__(16) unsigned char tf_smem[];
    TrsmNarrowSmem &S = *reinterpret_cast<TrsmNarrowSmem *>(tf_smem);
    constexpr int PRE = (TF_TMAX - TF_TB) * TF_TB / 256;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const i64 c0 = (i64)blockIdx.x * TN_CW;
    const int cols = (int)((N - c0) < TN_CW ? (N - c0) : TN_CW);
    const int nblk = (t + TF_TB - 1) / TF_TB;
    float pre[PRE];
    auto fetch = [&](int J) {  // L below diagonal block J
        const int rb = (J + 1) * TF_TB;
#pragma unroll
        for (int q = 0; q < PRE; ++q) {
            const int r = warp + 8 * q;
            pre[q] = rb + r < t ? L[(i64)(rb + r) * ldl + J * TF_TB + lane] : 0.f;
        }
    };
    fetch(0);
    if (warp < nblk) {
        float(*D)[TF_TB + 1] = S.D[warp];
        const int d0 = warp * TF_TB;
#pragma unroll
        for (int i = 0; i < TF_TB; ++i)
            D[i][lane] = (d0 + i < t && lane < i) ? L[(i64)(d0 + i) * ldl + d0 + lane] : 0.f;
    }
#pragma unroll
    for (int e = tid; e < TF_TMAX * TN_CW; e += 256) {
        const int i = e / TN_CW, c = e % TN_CW;
        S.X[i][c] = (i < t && c < cols) ? B[(i64)i * ldb + c0 + c] : 0.f;
    }
    for (int J = 0; J < nblk; ++J) {
        const int j0 = J * TF_TB, rem = t - j0 - TF_TB;  // rows below the block
#pragma unroll
        for (int q = 0; q < PRE; ++q) S.L[warp + 8 * q][lane] = pre[q];
        __syncthreads();
        if (J + 1 < nblk) fetch(J + 1);
        {
            float x = S.X[j0 + lane][warp], d[TF_TB];
#pragma unroll
            for (int p = 0; p < TF_TB; ++p) d[p] = S.D[J][lane][p];
#pragma unroll
            for (int p = 0; p < TF_TB - 1; ++p) {
                const float xp = __shfl_sync(0xffffffffu, x, p);
                if (lane > p) x = fmaf(-d[p], xp, x);
            }
            S.X[j0 + lane][warp] = x;
        }
        __syncthreads();
        if (tid < rem) {
            float acc[TN_CW];
#pragma unroll
            for (int c = 0; c < TN_CW; ++c) acc[c] = 0.f;
#pragma unroll 8
            for (int k = 0; k < TF_TB; ++k) {
                const float l = S.L[tid][k];
                const float4 a = *(const float4 *)&S.X[j0 + k][0], b = *(const float4 *)&S.X[j0 + k][4];
                acc[0] = fmaf(l, a.x, acc[0]);
                acc[1] = fmaf(l, a.y, acc[1]);
                acc[2] = fmaf(l, a.z, acc[2]);
                acc[3] = fmaf(l, a.w, acc[3]);
                acc[4] = fmaf(l, b.x, acc[4]);
                acc[5] = fmaf(l, b.y, acc[5]);
                acc[6] = fmaf(l, b.z, acc[6]);
                acc[7] = fmaf(l, b.w, acc[7]);
            }
#pragma unroll
            for (int c = 0; c < TN_CW; ++c) S.X[j0 + TF_TB + tid][c] -= acc[c];
        }
        __syncthreads();
    }
#pragma unroll
    for (int e = tid; e < TF_TMAX * TN_CW; e += 256) {
        const int i = e / TN_CW, c = e % TN_CW;
        if (i < t && c < cols) B[(i64)i * ldb + c0 + c] = S.X[i][c];
    }
}

template <typename T>
void launch_trsm_fused(const T *L, i64 ldl, T *B, i64 ldb, int t, i64 N, cudaStream_t s) {
    if (t <= 1 || N <= 0) return;
    ProfScope ps(KC_TRSM_LEAF, s, (double)t * t * N, 2.0 * (double)t * N * sizeof(T));
    if constexpr (sizeof(T) == 4) {
        if (N <= 2048) {
            set_max_dyn_smem((const void *)k_trsm_narrow, (int)sizeof(TrsmNarrowSmem));
            k_trsm_narrow<<<(unsigned)((N + TN_CW - 1) / TN_CW), 256, sizeof(TrsmNarrowSmem), s>>>(L, ldl, B, ldb, t, N);
            OXI_LAUNCH_CHECK();
            return;
        }
    }
    auto go = [&](auto kern, int cw) {
        const size_t smem = sizeof(T) * ((size_t)TF_TMAX * (cw + 1) + (size_t)TF_TMAX * (TF_TB + 1));
        set_max_dyn_smem((const void *)kern, (int)smem);
        kern<<<(unsigned)((N + cw - 1) / cw), 256, smem, s>>>(L, ldl, B, ldb, t, N);
        OXI_LAUNCH_CHECK();
    };
    if constexpr (sizeof(T) == 8) {
        if (N <= 2048) {
            go(k_trsm_fused<T, 8>, 8);
            return;
        }
    }
    go(k_trsm_fused<T, 32>, 32);
}
// ---------------------------------------------------------------------------
// Reference-order TRSM (FP64, t <= 128): B (t x N) <- L^-1 B for a unit lower
// L, performing element by element the operations of the reference's
// recursive solve (src/blas/level3.jl:338-355, _trsm_blocks_left!): halve the
// triangle (h = t / 2), solve the top half, update the bottom half with one
// fma chain from zero per element followed by a subtraction (the GEMM of
// src/blas/gemm.jl:286-298 / simd.jl:151 for k <= kc), solve the bottom half;
// leaves of <= 8 rows by substitution, s = b; s = fma(-L[i,p], x[p], s) for
// p < i (_trsm_leaf_generic!, level3.jl:309-321).  The host flattens the
// recursion into a list of leaf and update steps in the recursion's order; one
// CTA takes CW columns and runs the list with its columns in shared memory, so
// one launch gives the recursive solve's bits.
// ---------------------------------------------------------------------------
struct TrsmSteps {
    int count;
    int4 step[64];  // {kind (0 leaf, 1 update), a, b, c}: leaf rows [a, b); update rows [b, c) from [a, b)
};

static void trsm_steps_rec(int a, int b, TrsmSteps &st) {
    if (b - a <= 8) {
        st.step[st.count++] = make_int4(0, a, b, 0);
        return;
    }
    const int h = (b - a) / 2;
    trsm_steps_rec(a, a + h, st);
    st.step[st.count++] = make_int4(1, a, a + h, b);
    trsm_steps_rec(a + h, b, st);
}

constexpr int TR_TMAX = 128;
constexpr int TR_LP = TR_TMAX + 1;  // row pitch of the staged triangle

// Bound: latency of the steps, each a barrier, the operands' shared-memory
// loads and one chain of up to 64 dependent FP64 FMAs (t = 128, 8 columns a CTA: 31
// steps 26000 cycles, a leaf 550 to 650, an 8-row update 670, the widest 3300;
// the staging 7300).  The strict lower triangle of L is therefore staged in
// shared memory once per CTA, with everything in flight at once, instead of
// being fetched through L1 in every step.
template <int CW, int CPT>
__global__ void __launch_bounds__(256) k_trsm_refo(const double *__restrict__ L, i64 ldl, double *__restrict__ B,
                                                   i64 ldb, int t, i64 N, const __grid_constant__ TrsmSteps st) {
    extern __shared__ __align__(16) double tr_smem[];
    double *X = tr_smem;                          // t x CW
    double *Ls = tr_smem + (size_t)t * CW;        // t x TR_LP, strict lower triangle
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const i64 c0 = (i64)blockIdx.x * CW;
    const int cols = (int)((N - c0) < CW ? (N - c0) : CW);
    for (int i = warp; i < t; i += 8)
        for (int p = lane; p < i; p += 32) {
            const uint32_t dst = smem_u32(&Ls[i * TR_LP + p]);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(L + (i64)i * ldl + p) : "memory");
        }
#pragma unroll 4
    for (int e = tid; e < t * CW; e += 256) {
        const int i = e / CW, c = e - i * CW;
        X[i * CW + c] = (c < cols) ? B[(i64)i * ldb + c0 + c] : 0.0;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int k = 0; k < st.count; ++k) {
        const int4 o = st.step[k];
        if (o.x == 0) {
            // leaf of nl <= 8 rows, a column per thread: the triangle's loads all
            // issued up front (fully unrolled, predicated)
            if (tid < CW) {
                const int nl = o.z - o.y;
                double xv[8], lv[8][8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    xv[u] = (u < nl) ? X[(o.y + u) * CW + tid] : 0.0;
#pragma unroll
                    for (int pp = 0; pp < u; ++pp) lv[u][pp] = (u < nl) ? Ls[(o.y + u) * TR_LP + o.y + pp] : 0.0;
                }
#pragma unroll
                for (int u = 1; u < 8; ++u)
#pragma unroll
                    for (int pp = 0; pp < u; ++pp) xv[u] = fma(-lv[u][pp], xv[pp], xv[u]);
#pragma unroll
                for (int u = 1; u < 8; ++u)
                    if (u < nl) X[(o.y + u) * CW + tid] = xv[u];
            }
        } else {
            // rows [o.z, o.w) -= L[rows, o.y:o.z] X[o.y:o.z]: a thread takes CPT
            // columns of one row at a time (each element is one fma chain in pp
            // order, then the subtraction)
            constexpr int NG = CW / CPT, RGS = 256 / NG;
            const int cq = (tid % NG) * CPT;
            for (int r = o.z + tid / NG; r < o.w; r += RGS) {
                const double *Lr = Ls + r * TR_LP;
                double a[CPT];
#pragma unroll
                for (int u = 0; u < CPT; ++u) a[u] = 0.0;
#pragma unroll 8
                for (int pp = o.y; pp < o.z; ++pp) {
                    const double l = Lr[pp];
#pragma unroll
                    for (int u = 0; u < CPT; u += 2) {
                        const double2 x2 = *(const double2 *)(X + pp * CW + cq + u);
                        a[u] = fma(l, x2.x, a[u]);
                        a[u + 1] = fma(l, x2.y, a[u + 1]);
                    }
                }
                double *xr = X + r * CW + cq;
#pragma unroll
                for (int u = 0; u < CPT; u += 2) {
                    double2 x2 = *(double2 *)(xr + u);
                    x2.x -= a[u];
                    x2.y -= a[u + 1];
                    *(double2 *)(xr + u) = x2;
                }
            }
        }
        __syncthreads();
    }
#pragma unroll 4
    for (int e = tid; e < t * CW; e += 256) {
        const int i = e / CW, c = e - i * CW;
        if (c < cols) B[(i64)i * ldb + c0 + c] = X[i * CW + c];
    }
}

bool trsm_refo_applicable(int t) { return t >= 2 && t <= TR_TMAX; }

void launch_trsm_refo(const double *L, i64 ldl, double *B, i64 ldb, int t, i64 N, cudaStream_t s) {
    if (t <= 1 || N <= 0) return;
    if (t > TR_TMAX) throw CudaError{cudaErrorInvalidValue, "reference-order TRSM: triangle too large"};
    TrsmSteps st{};
    trsm_steps_rec(0, t, st);
    ProfScope ps(KC_TRSM_LEAF, s, (double)t * t * N, 2.0 * (double)t * N * 8);
    // Narrow strips while they fit one wave (a strip's time is its chain of
    // steps), then wider ones, which read the triangle less often.
    auto go = [&](auto kern, int cw) {
        set_max_dyn_smem((const void *)kern, (int)(sizeof(double) * TR_TMAX * (cw + TR_LP)));
        kern<<<(unsigned)((N + cw - 1) / cw), 256, sizeof(double) * (size_t)t * (cw + TR_LP), s>>>(L, ldl, B, ldb, t, N,
                                                                                                  st);
    };
    if (N <= 8 * 148) go(k_trsm_refo<8, 2>, 8);
    else go(k_trsm_refo<32, 4>, 32);
    OXI_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// Rank-k update in the order of a panel leaf's rank-1 steps (FP64): for every
// element of C (M x N, row-major), s = C; s = fma(-A[r,k], B[k,c], s) for
// k = 0..K-1.  Inside the reference's 32-column leaf (src/lapack/
// factorizations.jl:117-139) the columns right of step k receive exactly this
// sequence, so a leaf narrower than 32 columns followed by this update (and a
// substitution solve of its rows) reproduces the 32-column leaf's bits.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_rankk_seq(double *__restrict__ C, i64 ldc, const double *__restrict__ A,
                                                   i64 lda, const double *__restrict__ B, i64 ldb, int M, int N,
                                                   int K) {
    const i64 idx = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (i64)M * N) return;
    const int r = (int)(idx / N), c = (int)(idx - (i64)r * N);
    const double *a = A + (i64)r * lda;
    double sv = C[(i64)r * ldc + c];
    for (int k = 0; k < K; ++k) sv = fma(-a[k], B[(i64)k * ldb + c], sv);
    C[(i64)r * ldc + c] = sv;
}

void launch_rankk_seq(double *C, i64 ldc, const double *A, i64 lda, const double *B, i64 ldb, i64 M, i64 N,
                      i64 K, cudaStream_t s) {
    if (M <= 0 || N <= 0 || K <= 0) return;
    ProfScope ps(KC_GEMM_REF, s, 2.0 * M * N * K, 8.0 * (2.0 * M * N + M * K + K * N));
    const i64 tot = M * N;
    k_rankk_seq<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(C, ldc, A, lda, B, ldb, (int)M, (int)N, (int)K);
    OXI_LAUNCH_CHECK();
}

template void launch_trsm_fused<double>(const double *, i64, double *, i64, int, i64, cudaStream_t);
template void launch_trsm_fused<float>(const float *, i64, float *, i64, int, i64, cudaStream_t);

template void launch_trsm_leaf<double>(const double *, i64, double *, i64, int, i64, cudaStream_t, bool);
template void launch_trsm_leaf<float>(const float *, i64, float *, i64, int, i64, cudaStream_t, bool);

// ---------------------------------------------------------------------------
// Reference-order GEMM: C <- C - A*B, s_ij = sum_p fma(A_ip, B_pj, s) in p order
// from zero, then C_ij - s_ij -- the arithmetic of src/blas/gemm.jl:286-298 with
// alpha = -1, beta = 1.  64 x 64 tiles, 16-deep k slabs, 4 x 4 per thread.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) k_gemm_ref(T *__restrict__ C, i64 ldc, const T *__restrict__ A,
                                                  i64 lda, const T *__restrict__ B, i64 ldb, i64 M,
                                                  i64 N, i64 K) {
    __shared__ T As[16][64 + 1];
    __shared__ T Bs[16][64 + 1];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const i64 m0 = (i64)blockIdx.y * 64, n0 = (i64)blockIdx.x * 64;
    T acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = T(0);
    for (i64 k0 = 0; k0 < K; k0 += 16) {
        for (int e = threadIdx.x; e < 64 * 16; e += 256) {
            const int r = e >> 4, kk = e & 15;   // A: row r, k kk (k contiguous)
            const i64 gi = m0 + r, gk = k0 + kk;
            As[kk][r] = (gi < M && gk < K) ? A[gi * lda + gk] : T(0);
            const int kr = e >> 6, cc = e & 63;  // B: k kr, col cc (n contiguous)
            const i64 gk2 = k0 + kr, gj = n0 + cc;
            Bs[kr][cc] = (gk2 < K && gj < N) ? B[gk2 * ldb + gj] : T(0);
        }
        __syncthreads();
        const int kmax = (int)((K - k0) < 16 ? (K - k0) : 16);
        for (int p = 0; p < kmax; ++p) {
            T a[4], b[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) a[x] = As[p][ty + 16 * x];
#pragma unroll
            for (int y = 0; y < 4; ++y) b[y] = Bs[p][tx + 16 * y];
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) acc[x][y] = fma(a[x], b[y], acc[x][y]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            const i64 gi = m0 + ty + 16 * x, gj = n0 + tx + 16 * y;
            if (gi < M && gj < N) C[gi * ldc + gj] = C[gi * ldc + gj] - acc[x][y];
        }
}

template <typename T>
void launch_gemm_ref(T *C, i64 ldc, const T *A, i64 lda, const T *B, i64 ldb, i64 M, i64 N, i64 K,
                     cudaStream_t s) {
    if (M <= 0 || N <= 0 || K <= 0) return;
    dim3 grid((unsigned)((N + 63) / 64), (unsigned)((M + 63) / 64));
    ProfScope ps(KC_GEMM_REF, s, 2.0 * M * N * K, (double)sizeof(T) * (2.0 * M * N + M * K + K * N));
    k_gemm_ref<T><<<grid, 256, 0, s>>>(C, ldc, A, lda, B, ldb, M, N, K);
    OXI_LAUNCH_CHECK();
}
// ---------------------------------------------------------------------------
// Register-blocked CUDA-core GEMM for the FP32 panel (C <- C - A*B, row-major):
// 128 x BN tile, 16-deep k slabs double-buffered through registers, 8 x (BN/16)
// outputs per thread (strided so shared-memory reads broadcast or are
// conflict-free).
// ---------------------------------------------------------------------------
template <typename T, int BN>
__global__ void __launch_bounds__(256) k_gemm_simt(T *__restrict__ C, i64 ldc, const T *__restrict__ A,
                                                   i64 lda, const T *__restrict__ B, i64 ldb, i64 M,
                                                   i64 N, i64 K) {
    constexpr int BM = 128, BK = 16, TN = BN / 16;
    __shared__ T As[2][BK][BM + 4];
    __shared__ T Bs[2][BK][BN + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const i64 m0 = (i64)blockIdx.y * BM, n0 = (i64)blockIdx.x * BN;
    T acc[8][TN];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = 0; b < TN; ++b) acc[a][b] = T(0);
    constexpr int AL = BM * BK / 256, BL = BK * BN / 256;
    T ra[AL], rb[BL];
    auto gload = [&](i64 k0) {
#pragma unroll
        for (int q = 0; q < AL; ++q) {
            const int e = threadIdx.x + q * 256;
            const int r = e / BK, kk = e % BK;
            const i64 gi = m0 + r, gk = k0 + kk;
            ra[q] = (gi < M && gk < K) ? A[gi * lda + gk] : T(0);
        }
#pragma unroll
        for (int q = 0; q < BL; ++q) {
            const int e = threadIdx.x + q * 256;
            const int kr = e / BN, cc = e % BN;
            const i64 gk = k0 + kr, gj = n0 + cc;
            rb[q] = (gk < K && gj < N) ? B[gk * ldb + gj] : T(0);
        }
    };
    auto sstore = [&](int buf) {
#pragma unroll
        for (int q = 0; q < AL; ++q) {
            const int e = threadIdx.x + q * 256;
            As[buf][e % BK][e / BK] = ra[q];
        }
#pragma unroll
        for (int q = 0; q < BL; ++q) {
            const int e = threadIdx.x + q * 256;
            Bs[buf][e / BN][e % BN] = rb[q];
        }
    };
    gload(0);
    sstore(0);
    __syncthreads();
    int buf = 0;
    for (i64 k0 = 0; k0 < K; k0 += BK) {
        const bool more = k0 + BK < K;
        if (more) gload(k0 + BK);
#pragma unroll
        for (int p = 0; p < BK; ++p) {
            T a[8], b[TN];
#pragma unroll
            for (int x = 0; x < 8; ++x) a[x] = As[buf][p][ty + 16 * x];
#pragma unroll
            for (int y = 0; y < TN; ++y) b[y] = Bs[buf][p][tx + 16 * y];
#pragma unroll
            for (int x = 0; x < 8; ++x)
#pragma unroll
                for (int y = 0; y < TN; ++y) acc[x][y] = fma(a[x], b[y], acc[x][y]);
        }
        if (more) {
            sstore(buf ^ 1);
            __syncthreads();
            buf ^= 1;
        }
    }
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        const i64 gi = m0 + ty + 16 * x;
        if (gi >= M) continue;
#pragma unroll
        for (int y = 0; y < TN; ++y) {
            const i64 gj = n0 + tx + 16 * y;
            if (gj < N) C[gi * ldc + gj] -= acc[x][y];
        }
    }
}

template <typename T>
void launch_gemm_simt(T *C, i64 ldc, const T *A, i64 lda, const T *B, i64 ldb, i64 M, i64 N, i64 K,
                      cudaStream_t s) {
    if (M <= 0 || N <= 0 || K <= 0) return;
    ProfScope ps(KC_GEMM_REF, s, 2.0 * M * N * K, (double)sizeof(T) * (2.0 * M * N + M * K + K * N));
    if (N <= 64) {
        dim3 grid((unsigned)((N + 63) / 64), (unsigned)((M + 127) / 128));
        k_gemm_simt<T, 64><<<grid, 256, 0, s>>>(C, ldc, A, lda, B, ldb, M, N, K);
    } else {
        dim3 grid((unsigned)((N + 127) / 128), (unsigned)((M + 127) / 128));
        k_gemm_simt<T, 128><<<grid, 256, 0, s>>>(C, ldc, A, lda, B, ldb, M, N, K);
    }
    OXI_LAUNCH_CHECK();
}
template void launch_gemm_simt<float>(float *, i64, const float *, i64, const float *, i64, i64, i64, i64, cudaStream_t);

// ---------------------------------------------------------------------------
// Right-looking step inside an FP32 panel, after a KW-wide leaf:
//   U12 <- L11^-1 A12     (L11 the leaf's KW x KW unit lower block, A12 the
//                          panel's N columns right of the leaf in those rows)
//   A22 <- A22 - L21 U12  (L21 the leaf's M rows below L11)
// in ONE launch.  Every CTA solves the 64-column slice of U12 it needs (a
// KW-step substitution, one thread per column, L11 from shared memory), the
// CTAs of the first row tile write it to ubuf (the next leaf, or a copy,
// moves it into place once no CTA reads A12 any more), and each CTA then
// updates its 128 x 64 tile of A22 (K = KW).
// ---------------------------------------------------------------------------
// Bound: latency of one CTA's stages (operands, U12's chain, products) and the
// panel's L2 round trip.  The tile of A22 is requested with the operands, before
// U12's chain; a thread owns 8 rows x 4 adjacent columns, so the products read
// shared memory 16 bytes at a time (three loads per 32 FMAs).
template <int KW>
__global__ void __launch_bounds__(256, 2) k_panel_rl(float *__restrict__ P, i64 ld, int M, int N,
                                                  float *__restrict__ ubuf) {
    constexpr int BM = 128, BN = 64, AP = KW + 4, UP = BN + 4;
    __shared__ float Ls[KW][KW + 1];
    __shared__ __align__(16) float Us[KW][UP];
    __shared__ __align__(16) float As[BM][AP];  // the L21 tile
    const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const bool vec = (ld % 4 == 0) && ((uintptr_t)P % 16 == 0);
    constexpr int KV = KW / 4, AL = BM * KV / 256;
    float4 av[AL];
#pragma unroll
    for (int q = 0; q < AL; ++q) {
        const int e = t + 256 * q, r = e / KV, k = 4 * (e % KV);
        av[q] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m0 + r < M) {
            const float *src = P + (i64)(KW + m0 + r) * ld + k;
            if (vec) av[q] = *(const float4 *)src;
            else av[q] = make_float4(src[0], src[1], src[2], src[3]);
        }
    }
    constexpr int UL = KW * BN / 256;
    float uv[UL];
#pragma unroll
    for (int q = 0; q < UL; ++q) {
        const int e = t + 256 * q, i = e / BN, j = e % BN;
        uv[q] = (n0 + j < N) ? P[(i64)i * ld + KW + n0 + j] : 0.f;
    }
    constexpr int LL = (KW * KW + 255) / 256;
    float lv[LL];
#pragma unroll
    for (int q = 0; q < LL; ++q) {
        const int e = t + 256 * q;
        lv[q] = e < KW * KW ? P[(i64)(e / KW) * ld + e % KW] : 0.f;
    }
    // this thread's elements of A22: rows ty 8 .., columns tx 4 ..
    float c[8][4];
    const int col = n0 + tx * 4;
    const bool whole = vec && col + 3 < N;
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        const int r = m0 + ty * 8 + x;
        const float *src = P + (i64)(KW + r) * ld + KW + col;
        if (r < M && whole) {
            const float4 v = *(const float4 *)src;
            c[x][0] = v.x; c[x][1] = v.y; c[x][2] = v.z; c[x][3] = v.w;
        } else {
#pragma unroll
            for (int y = 0; y < 4; ++y) c[x][y] = (r < M && col + y < N) ? src[y] : 0.f;
        }
    }
#pragma unroll
    for (int q = 0; q < LL; ++q) {
        const int e = t + 256 * q;
        if (e < KW * KW) Ls[e / KW][e % KW] = lv[q];
    }
#pragma unroll
    for (int q = 0; q < UL; ++q) {
        const int e = t + 256 * q;
        Us[e / BN][e % BN] = uv[q];
    }
#pragma unroll
    for (int q = 0; q < AL; ++q) {
        const int e = t + 256 * q;
        *(float4 *)&As[e / KV][4 * (e % KV)] = av[q];
    }
    __syncthreads();
    if (t < BN) {
        float x[KW];
#pragma unroll
        for (int i = 0; i < KW; ++i) x[i] = Us[i][t];
#pragma unroll
        for (int p = 0; p < KW; ++p)
#pragma unroll
            for (int i = p + 1; i < KW; ++i) x[i] = fmaf(-Ls[i][p], x[p], x[i]);
#pragma unroll
        for (int i = 0; i < KW; ++i) Us[i][t] = x[i];
        if (blockIdx.y == 0 && n0 + t < N) {  // not into A12: other CTAs may still read it
#pragma unroll
            for (int i = 0; i < KW; ++i) ubuf[(i64)i * N + n0 + t] = x[i];
        }
    }
    __syncthreads();
#pragma unroll 2
    for (int k = 0; k < KW; k += 4) {
        float4 a[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) a[x] = *(const float4 *)&As[ty * 8 + x][k];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const float4 b = *(const float4 *)&Us[k + kk][tx * 4];
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                const float ak = kk == 0 ? a[x].x : (kk == 1 ? a[x].y : (kk == 2 ? a[x].z : a[x].w));
                c[x][0] = fmaf(-ak, b.x, c[x][0]);
                c[x][1] = fmaf(-ak, b.y, c[x][1]);
                c[x][2] = fmaf(-ak, b.z, c[x][2]);
                c[x][3] = fmaf(-ak, b.w, c[x][3]);
            }
        }
    }
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        const int r = m0 + ty * 8 + x;
        float *dst = P + (i64)(KW + r) * ld + KW + col;
        if (r < M && whole) {
            *(float4 *)dst = make_float4(c[x][0], c[x][1], c[x][2], c[x][3]);
        } else {
#pragma unroll
            for (int y = 0; y < 4; ++y)
                if (r < M && col + y < N) dst[y] = c[x][y];
        }
    }
}

void launch_panel_rl(float *P, i64 ld, int kw, i64 M, i64 N, float *ubuf, cudaStream_t s) {
    if (N <= 0) return;
    dim3 grid((unsigned)((N + 63) / 64), (unsigned)std::max<i64>(1, (M + 127) / 128));
    ProfScope ps(KC_GEMM_REF, s, 2.0 * (double)std::max<i64>(M, 0) * N * kw + (double)kw * kw * N,
                 4.0 * (2.0 * std::max<i64>(M, 0) * N + (double)(M + kw) * kw + 2.0 * kw * N));
    if (kw == 32) k_panel_rl<32><<<grid, 256, 0, s>>>(P, ld, (int)M, (int)N, ubuf);
    else if (kw == 16) k_panel_rl<16><<<grid, 256, 0, s>>>(P, ld, (int)M, (int)N, ubuf);
    else if (kw == 8) k_panel_rl<8><<<grid, 256, 0, s>>>(P, ld, (int)M, (int)N, ubuf);
    else throw CudaError{cudaErrorInvalidValue, "right-looking panel step: leaf width 8, 16 or 32"};
    OXI_LAUNCH_CHECK();
}

template void launch_gemm_ref<double>(double *, i64, const double *, i64, const double *, i64, i64, i64, i64, cudaStream_t);
template void launch_gemm_ref<float>(float *, i64, const float *, i64, const float *, i64, i64, i64, i64, cudaStream_t);

}  // namespace oxi
