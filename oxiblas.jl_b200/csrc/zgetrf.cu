// Complex (ComplexF64) partial-pivoted LU and its solves.
//
// Replaces _lu_factor! / _lu_panel! for Complex{Float64} (src/lapack/
// factorizations.jl:30-152: blocked right-looking with nb = 128, recursive
// panel with 16-column leaves for complex types (:113), the complex pivot rule
// of _lu_pivot (:92-107): the largest abs2, strict '>' so the first row wins,
// redone with abs when the largest square is not finite) and ldiv! with
// trans 'N' / 'T' / 'C' (src/api/linalg_api.jl:168-184).
//
// Layout: the caller's interleaved column-major A is split into two row-major
// FP64 planes (real, imaginary) in the handle's working matrix, so that a row
// interchange moves contiguous segments and the trailing update is one launch of
// real products on the FP64 tensor cores (k_zgemm_dmma), four per element:
//   Cr -= Ar Br;  Cr -= (-Ai) Bi;  Ci -= Ar Bi;  Ci -= Ai Br.
// (At an odd column offset, which TMA cannot take: four launches on the planes,
// with a negated copy of the panel's imaginary one.)  A panel's leaves of 16
// columns hold their rows in the registers of a cluster of up to 16 CTAs
// (k_zleaf_reg) and apply their interchanges to the panel's other columns; the
// columns outside the panel get the panel's composed interchanges once.  Above
// 8192 rows the leaf keeps its rows in the cluster's shared memory (k_zleaf_cl), above
// 12288 in global memory with one CTA (k_zleaf), and each leaf's interchanges go
// to all other columns right after it (k_zlaswp).  The U block row is solved by a
// unit-lower substitution kernel.
#include <cooperative_groups.h>
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>
#include "leaf.cuh"
#include "oxi_internal.h"
#include "tma_util.cuh"

namespace oxi {

namespace {
constexpr int ZLEAF = 16;      // complex leaf (the reference's _lu_leaf for complex types)
constexpr int ZLEAF_NT = 1024;
inline i64 zrup(i64 x, i64 a) { return (x + a - 1) / a * a; }
}  // namespace

struct zd {
    double r, i;
};
__device__ __forceinline__ zd zmul(zd a, zd b) { return {a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r}; }
// c - a b: the product, then the difference (muladd(-a, b, c) of the reference)
__device__ __forceinline__ zd zmsub(zd c, zd a, zd b) {
    return {c.r - (a.r * b.r - a.i * b.i), c.i - (a.r * b.i + a.i * b.r)};
}
// c - a b on double2
__device__ __forceinline__ double2 zmsub2(double2 c, double2 a, double2 b) {
    return make_double2(fma(a.y, b.y, fma(-a.x, b.x, c.x)), fma(-a.y, b.x, fma(-a.x, b.y, c.y)));
}

// 1 / b = conj(b) / |b|^2, b scaled by the power of two of the larger of |b.r|,
// |b.i| (exact, and |b|^2 stays far from over- and underflow): one division instead of
// the four of scaling by the component itself, which a column step waits for.
// Errors of 3e6 random ones, normwise in units of 2^-53: root mean square 0.81,
// largest 3.0 (four divisions: 0.83 and 2.5).
__device__ __forceinline__ zd zrecip(zd b) {
    const double m = fmax(fabs(b.r), fabs(b.i));
    if (m > 0x1p-1000 && m < 0x1p1000) {
        const int e = (__double2hiint(m) >> 20) - 1023;
        const double s = __hiloint2double((1023 - e) << 20, 0);  // 2^-e
        const double br = b.r * s, bi = b.i * s;                 // the larger in [1, 2)
        const double y = 1.0 / fma(br, br, bi * bi);
        return {br * y * s, -(bi * y) * s};
    }
    const double s = m == 0.0 ? 1.0 : m;
    const double br = b.r / s, bi = b.i / s;
    const double den = (br * br + bi * bi) * s;
    return {br / den, -bi / den};
}

// (key, position) argmax over the CTA: the largest key, the smallest position
// among equal keys; keys are non-negative doubles (NaN never enters).
__device__ __forceinline__ void cta_argmax(double &key, int &pos, double *s_key, int *s_pos) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int off = 16; off > 0; off >>= 1) {
        const double ok = __shfl_xor_sync(0xffffffffu, key, off);
        const int op = __shfl_xor_sync(0xffffffffu, pos, off);
        if (ok > key || (ok == key && op < pos)) { key = ok; pos = op; }
    }
    if (lane == 0) { s_key[warp] = key; s_pos[warp] = pos; }
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        key = lane < nw ? s_key[lane] : -1.0;
        pos = lane < nw ? s_pos[lane] : INT_MAX;
        for (int off = 16; off > 0; off >>= 1) {
            const double ok = __shfl_xor_sync(0xffffffffu, key, off);
            const int op = __shfl_xor_sync(0xffffffffu, pos, off);
            if (ok > key || (ok == key && op < pos)) { key = ok; pos = op; }
        }
        if (lane == 0) { s_key[0] = key; s_pos[0] = pos; }
    }
    __syncthreads();
    key = s_key[0];
    pos = s_pos[0];
    __syncthreads();
}

// Leaf: the m x w (w <= 16) block at (Wr, Wi) (row-major planes, ld), one CTA.
// Column j: the pivot row (largest abs2 among rows >= j; with abs when that
// square is not finite; the row itself when nothing beats it), the interchange
// within the leaf's columns, the multipliers l = a / d and the rank-1 update of
// the leaf's later columns.  ipiv gets gofs + p + 1, info the first zero pivot.
__global__ void __launch_bounds__(ZLEAF_NT) k_zleaf(double *__restrict__ Wr, double *__restrict__ Wi, i64 ld, int m,
                                                    int w, i64 gofs, int64_t *__restrict__ ipiv,
                                                    int64_t *__restrict__ info) {
    __shared__ double s_key[32];
    __shared__ int s_pos[32];
    __shared__ zd s_prow[ZLEAF];
    const int tid = threadIdx.x;
    const int q = m < w ? m : w;
    for (int j = 0; j < q; ++j) {
        // candidates by abs2
        double key = -1.0;
        int pos = INT_MAX;
        bool nonfinite = false;
        for (int i = j + tid; i < m; i += ZLEAF_NT) {
            const double ar = Wr[(i64)i * ld + j], ai = Wi[(i64)i * ld + j];
            const double v = ar * ar + ai * ai;
            if (v == v && v > key) { key = v; pos = i; }
        }
        // the reference starts from row j: a NaN there keeps row j
        {
            const double ar = Wr[(i64)j * ld + j], ai = Wi[(i64)j * ld + j];
            const double v0 = ar * ar + ai * ai;
            if (v0 != v0) { key = (tid == 0) ? INFINITY : -1.0; pos = (tid == 0) ? j : INT_MAX; }
        }
        cta_argmax(key, pos, s_key, s_pos);
        nonfinite = !(key < INFINITY);
        if (nonfinite) {  // redo with abs (hypot) when the largest square overflowed
            double k2 = -1.0;
            int p2 = INT_MAX;
            for (int i = j + tid; i < m; i += ZLEAF_NT) {
                const double v = hypot(Wr[(i64)i * ld + j], Wi[(i64)i * ld + j]);
                if (v == v && v > k2) { k2 = v; p2 = i; }
            }
            const double v0 = hypot(Wr[(i64)j * ld + j], Wi[(i64)j * ld + j]);
            if (v0 != v0) { k2 = (tid == 0) ? INFINITY : -1.0; p2 = (tid == 0) ? j : INT_MAX; }
            cta_argmax(k2, p2, s_key, s_pos);
            pos = p2;
        }
        const int p = (pos == INT_MAX) ? j : pos;
        if (tid == 0) ipiv[gofs + j] = gofs + p + 1;
        if (p != j && tid < w) {  // the interchange within the leaf's columns
            const double tr = Wr[(i64)j * ld + tid], ti = Wi[(i64)j * ld + tid];
            Wr[(i64)j * ld + tid] = Wr[(i64)p * ld + tid];
            Wi[(i64)j * ld + tid] = Wi[(i64)p * ld + tid];
            Wr[(i64)p * ld + tid] = tr;
            Wi[(i64)p * ld + tid] = ti;
        }
        __syncthreads();
        if (tid < w) s_prow[tid] = {Wr[(i64)j * ld + tid], Wi[(i64)j * ld + tid]};
        __syncthreads();
        const zd d = s_prow[j];
        if (d.r == 0.0 && d.i == 0.0) {
            if (tid == 0 && *info == 0) *info = gofs + j + 1;
            continue;
        }
        // the multipliers a / d as a times the reciprocal of d, formed once per
        // column (the reference divides each element; the results agree to
        // rounding)
        const zd dinv = zrecip(d);
        for (int i = j + 1 + tid; i < m; i += ZLEAF_NT) {
            double *rr = Wr + (i64)i * ld, *ri = Wi + (i64)i * ld;
            const zd l = zmul({rr[j], ri[j]}, dinv);
            rr[j] = l.r;
            ri[j] = l.i;
            for (int c = j + 1; c < w; ++c) {
                const zd v = zmsub({rr[c], ri[c]}, l, s_prow[c]);
                rr[c] = v.r;
                ri[c] = v.i;
            }
        }
        __syncthreads();
    }
}

// The same leaf on a cluster of CS CTAs (1..16) that hold the panel's rows in
// shared memory (CTA r: rows [r RP, (r + 1) RP), both planes, 16 columns), so a
// column step reads no global memory: each CTA's candidate (the largest abs2
// and, for the overflow rule, the largest abs, of its rows below j, first index
// on ties), one cluster barrier, every CTA picks the same pivot from the CS
// candidates and |a_jj| (row j lives in CTA 0: j < 16 <= RP), reads the pivot
// row and row j through distributed shared memory, a second barrier, the two
// owners write the interchanged rows, then each CTA eliminates its own rows.
// Cluster barriers are hardware barriers every CTA meets the same number of
// times; there is no spin wait.
namespace cgz = cooperative_groups;
constexpr int ZCL_NT = 512;
constexpr int ZCL_MAXRP = 768;  // rows per CTA (192 KB of shared memory)
struct ZCand {
    double k2, kh;  // largest abs2 / abs among the CTA's rows below j (-1: none)
    int p2, ph;     // their rows (INT_MAX: none)
};
__device__ __forceinline__ void zcand_combine(double &k, int &p, double k2, int p2) {
    if (k2 > k || (k2 == k && p2 < p)) { k = k2; p = p2; }
}
__global__ void __launch_bounds__(ZCL_NT, 1) k_zleaf_cl(double *__restrict__ Wr, double *__restrict__ Wi, i64 ld, int m,
                                                         int w, int RP, i64 gofs, int64_t *__restrict__ ipiv,
                                                         int64_t *__restrict__ info) {
    cgz::cluster_group cl = cgz::this_cluster();
    const int CS = (int)cl.num_blocks(), cr = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    extern __shared__ double2 zcl[];  // [RP][ZLEAF] complex
    __shared__ ZCand s_cand[2];
    __shared__ double s_rk[ZCL_NT / 32][2];
    __shared__ int s_rp[ZCL_NT / 32][2];
    __shared__ zd s_prow[ZLEAF], s_jrow[ZLEAF];
    __shared__ int s_piv[ZLEAF], s_info;
    const int r0 = cr * RP;
    const int nr = max(0, min(m - r0, RP));
    if (tid == 0) s_info = 0;
    for (int e = tid; e < nr * ZLEAF; e += ZCL_NT) {
        const int li = e / ZLEAF, c = e - li * ZLEAF;
        const i64 g = (i64)(r0 + li) * ld + c;
        zcl[e] = (c < w) ? make_double2(Wr[g], Wi[g]) : make_double2(0.0, 0.0);
    }
    __syncthreads();
    const int q = m < w ? m : w;
    for (int j = 0; j < q; ++j) {
        const int par = j & 1;
        // (1) this CTA's candidates among its rows below j
        double k2 = -1.0, kh = -1.0;
        int p2 = INT_MAX, ph = INT_MAX;
        for (int li = max(0, j + 1 - r0) + tid; li < nr; li += ZCL_NT) {
            const double2 a = zcl[li * ZLEAF + j];
            const double v2 = a.x * a.x + a.y * a.y, vh = hypot(a.x, a.y);
            if (v2 == v2 && v2 > k2) { k2 = v2; p2 = r0 + li; }  // rows ascend per thread: first maximum
            if (vh == vh && vh > kh) { kh = vh; ph = r0 + li; }
        }
        for (int off = 16; off > 0; off >>= 1) {
            zcand_combine(k2, p2, __shfl_xor_sync(0xffffffffu, k2, off), __shfl_xor_sync(0xffffffffu, p2, off));
            zcand_combine(kh, ph, __shfl_xor_sync(0xffffffffu, kh, off), __shfl_xor_sync(0xffffffffu, ph, off));
        }
        if (lane == 0) { s_rk[warp][0] = k2; s_rp[warp][0] = p2; s_rk[warp][1] = kh; s_rp[warp][1] = ph; }
        __syncthreads();
        if (tid == 0) {
            for (int wv = 1; wv < ZCL_NT / 32; ++wv) {
                zcand_combine(k2, p2, s_rk[wv][0], s_rp[wv][0]);
                zcand_combine(kh, ph, s_rk[wv][1], s_rp[wv][1]);
            }
            s_cand[par] = ZCand{k2, kh, p2, ph};
        }
        cl.sync();  // (2) every CTA's candidate is published
        // (3) the pivot, identical in every CTA: _lu_pivot's abs2 scan from row j
        // with strict '>', redone with abs when that square is not finite
        double b2 = -1.0, bh = -1.0;
        int q2 = INT_MAX, qh = INT_MAX;
        for (int rr = 0; rr < CS; ++rr) {
            const ZCand cd = *cl.map_shared_rank(&s_cand[par], rr);
            zcand_combine(b2, q2, cd.k2, cd.p2);
            zcand_combine(bh, qh, cd.kh, cd.ph);
        }
        const double2 ajj = *cl.map_shared_rank(&zcl[j * ZLEAF + j], 0);
        const double v2 = ajj.x * ajj.x + ajj.y * ajj.y;
        int p = j;
        double best = v2;
        if (q2 != INT_MAX && b2 > v2) { best = b2; p = q2; }
        if (!(best < INFINITY)) {  // NaN start or an overflowing square: the abs scan
            const double vh = hypot(ajj.x, ajj.y);
            p = (qh != INT_MAX && bh > vh) ? qh : j;
        }
        // (4) the pivot row and row j through distributed shared memory
        const int cp = p / RP;
        if (tid < ZLEAF) {
            const double2 pv = *cl.map_shared_rank(&zcl[(p - cp * RP) * ZLEAF + tid], cp);
            s_prow[tid] = {pv.x, pv.y};
            const double2 jv = *cl.map_shared_rank(&zcl[j * ZLEAF + tid], 0);
            s_jrow[tid] = {jv.x, jv.y};
        }
        if (cr == 0 && tid == 0) s_piv[j] = p;
        cl.sync();  // (5) every CTA has read both rows before they are rewritten
        if (p != j && tid < ZLEAF) {
            if (cr == 0) zcl[j * ZLEAF + tid] = make_double2(s_prow[tid].r, s_prow[tid].i);
            if (cr == cp) zcl[(p - r0) * ZLEAF + tid] = make_double2(s_jrow[tid].r, s_jrow[tid].i);
        }
        __syncthreads();
        // (6) elimination of this CTA's rows below j
        const zd d = s_prow[j];
        if (d.r == 0.0 && d.i == 0.0) {
            if (cr == 0 && tid == 0 && s_info == 0) s_info = j + 1;
            continue;
        }
        const zd dinv = zrecip(d);
        for (int li = max(0, j + 1 - r0) + tid; li < nr; li += ZCL_NT) {
            double2 *row = zcl + li * ZLEAF;
            const double2 a = row[j];
            const zd l = zmul({a.x, a.y}, dinv);
            row[j] = make_double2(l.r, l.i);
            for (int c = j + 1; c < w; ++c) {
                const double2 b = row[c];
                const zd v = zmsub({b.x, b.y}, l, s_prow[c]);
                row[c] = make_double2(v.r, v.i);
            }
        }
        __syncthreads();
    }
    cl.sync();  // no CTA leaves while another may still read its rows
    for (int e = tid; e < nr * ZLEAF; e += ZCL_NT) {
        const int li = e / ZLEAF, c = e - li * ZLEAF;
        if (c < w) {
            const i64 g = (i64)(r0 + li) * ld + c;
            Wr[g] = zcl[e].x;
            Wi[g] = zcl[e].y;
        }
    }
    if (cr == 0) {
        if (tid < q) ipiv[gofs + tid] = gofs + s_piv[tid] + 1;
        if (tid == 0 && s_info != 0 && *info == 0) *info = gofs + s_info;
    }
}

// The leaf of up to 8192 rows, in the form of the real one (leaf.cuh, lu_kernels.cu):
// a cluster holds the rows in registers, one per thread, with implicit
// pivoting; columns in groups of ZGW = 4, whose pivot rows publish their other
// columns once per group.  A candidate is {position, key}, a_pj, a_p,j+1, ...
// with the key abs2; a column whose largest abs2 is not finite repeats its search
// with abs (_lu_pivot, src/lapack/factorizations.jl:92-107).  Bound: latency of
// the column steps, as the real leaf.
constexpr int ZGW = 4, ZNG = ZLEAF / ZGW;
template <int NT>
__global__ void __launch_bounds__(NT, 1)
k_zleaf_reg(double *__restrict__ Wr, double *__restrict__ Wi, i64 ld, int m, int w, i64 gofs,
            int64_t *__restrict__ ipiv, int64_t *__restrict__ info, LeafPanel pn) {
    cgz::cluster_group cl = cgz::this_cluster();
    const int CS = (int)cl.num_blocks(), cr = (int)cl.block_rank();
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, half = lane & 15;
    constexpr int NW = NT / 32, PERMAX = 1 + ZGW;
    constexpr int MOVE_PW = (2 * ZLEAF + NW - 1) / NW, MOVE_CH = LEAF_MAX_OTHER / 32;
    extern __shared__ __align__(16) unsigned char zl_smem[];  // 32 rows x 144 bytes per warp
    __shared__ double2 s_cand[2][NW][PERMAX];
    __shared__ double2 s_slot[2][16][PERMAX];
    __shared__ double2 s_right[ZGW][ZLEAF], s_stage[ZGW][ZLEAF], s_u[ZGW][ZLEAF];
    __shared__ __align__(8) uint64_t s_xbar[2], s_rbar;
    __shared__ int s_piv[ZLEAF], s_info, s_skip, s_mcnt;
    __shared__ int2 s_mv[2 * ZLEAF];
    if (t == 0) {
        s_info = 0;
        s_mcnt = 0;
        s_skip = aborted(pn.abort) ? 1 : 0;
        mbar_init(&s_xbar[0], 1);
        mbar_init(&s_xbar[1], 1);
        mbar_init(&s_rbar, 1);
        fence_barrier_init();
    }
    const int G = CS * NT, i0 = cr * NT + t;
    int pos = i0 < m ? i0 : -1;
    double2 r[ZLEAF];
#pragma unroll
    for (int c = 0; c < ZLEAF; ++c) r[c] = make_double2(0.0, 0.0);
    const bool vec_ok = w == ZLEAF && ld % 2 == 0 && (((uintptr_t)Wr | (uintptr_t)Wi) % 16 == 0);
    unsigned char *tr = zl_smem + warp * (32 * 144);
    const int trow = lane >> 3, tchk = lane & 7;
    if (vec_ok) {
        double2 x[2][8];
#pragma unroll
        for (int pl = 0; pl < 2; ++pl)
#pragma unroll
            for (int it = 0; it < 8; ++it) {
                const int i = i0 - lane + it * 4 + trow;
                x[pl][it] = make_double2(0.0, 0.0);
                if (i < m) x[pl][it] = *(const double2 *)((pl ? Wi : Wr) + (i64)i * ld + 2 * tchk);
            }
#pragma unroll
        for (int pl = 0; pl < 2; ++pl) {
#pragma unroll
            for (int it = 0; it < 8; ++it) *(double2 *)(tr + (it * 4 + trow) * 144 + tchk * 16) = x[pl][it];
            __syncwarp();
#pragma unroll
            for (int c = 0; c < ZLEAF; c += 2) {
                const double2 v = *(const double2 *)(tr + lane * 144 + c * 8);
                if (pl == 0) { r[c].x = v.x; r[c + 1].x = v.y; }
                else { r[c].y = v.x; r[c + 1].y = v.y; }
            }
            __syncwarp();
        }
    } else if (pos >= 0) {
#pragma unroll
        for (int c = 0; c < ZLEAF; ++c)
            if (c < w) r[c] = make_double2(Wr[(i64)i0 * ld + c], Wi[(i64)i0 * ld + c]);
    }
    // barriers exist, and every row is read, before any CTA pushes or stores
    if (CS > 1) cl.sync();
    else __syncthreads();
    const int skip = (CS > 1) ? *cl.map_shared_rank(&s_skip, 0) : s_skip;
    if (skip) {
        if (CS > 1) cl.sync();
        return;
    }
    bool dead = false;  // an exchange wait gave up: nothing is stored, every cluster barrier still met
    const int q = m < w ? m : w;
    const uint32_t to_cta = cluster_map_u32(&s_xbar[0], half < CS ? half : 0) - smem_u32(&s_xbar[0]);
    int xc = 0;         // exchanges so far
#pragma unroll 1
    for (int s = 0; s < ZNG; ++s) {
        const int j0 = s * ZGW;
        uint32_t live = 0;
#pragma unroll
        for (int jj = 0; jj < ZGW; ++jj) {
            const int j = j0 + jj;
            if (j >= q) break;
            const int PER = 1 + ZGW - jj;
            const double2(*cand)[PERMAX] = nullptr;
            int wq = 0;
            double2 cy;   // this lane's candidate's reciprocal
#pragma unroll 1
            for (int round = 0; round < 2; ++round, ++xc) {
                const int par = xc & 1;
                const double2 a = r[jj];
                const double key = round == 0 ? a.x * a.x + a.y * a.y : hypot(a.x, a.y);
                const uint64_t kb = step_key(key, pos, j);
                {
                    const uint32_t wm = warp_winner<double>(kb, pos >= j ? pos : INT_MAX);
                    if (wm == 0 ? lane == 0 : ((wm >> lane) & 1)) {
                        double2 *c = s_cand[par][warp];
                        c[0] = make_double2(__hiloint2double(0, wm ? pos : INT_MAX), __longlong_as_double((long long)kb));
#pragma unroll
                        for (int e = jj; e < ZGW; ++e) c[1 + e - jj] = r[e];
                    }
                }
                __syncthreads();
                auto list_winner = [&](const double2(*l)[PERMAX], int n, uint64_t &ck) -> int {
                    int cp = INT_MAX;
                    ck = 0;
                    if (lane < n) {
                        const double2 h = l[lane][0];
                        cp = __double2loint(h.x);
                        ck = (uint64_t)__double_as_longlong(h.y);
                    }
                    const uint32_t wm = warp_winner<double>(ck, cp);
                    return wm ? __ffs(wm) - 1 : 0;
                };
                uint64_t ck;
                if (CS > 1 && !dead) {
                    if (t == 0) mbar_arrive_expect_tx(&s_xbar[par], (uint32_t)(CS * 16 * PER));
                    if (warp < PER) {
                        const int wn = list_winner(s_cand[par], NW, ck);
                        if (lane < CS)
                            st_async_v4(smem_u32(s_slot[par][cr]) + 16u * warp + to_cta,
                                        reinterpret_cast<const uint4 *>(s_cand[par][wn])[warp],
                                        smem_u32(&s_xbar[par]) + to_cta);
                    }
                    if (!mbar_wait(&s_xbar[par], (uint32_t)((xc >> 1) & 1), pn.abort, 1)) dead = true;
                }
                cand = (CS > 1) ? s_slot[par] : s_cand[par];
                const int nc = CS > 1 ? CS : NW;
                zd rec = zrecip(lane < nc ? zd{cand[lane][1].x, cand[lane][1].y} : zd{1.0, 0.0});
                cy = make_double2(rec.r, rec.i);
                wq = list_winner(cand, nc, ck);
                const uint64_t best = (uint64_t)__double_as_longlong(cand[wq][0].y);
                // the CTA decides together: after a wait that gave up its warps may
                // have read different slots
                if (!__syncthreads_or(round == 0 && best >= 0x7ff0000000000000ull)) {
                    ++xc;
                    break;
                }
            }
            const double2 dinv = make_double2(__shfl_sync(0xffffffffu, cy.x, wq), __shfl_sync(0xffffffffu, cy.y, wq));
            const int wp = __double2loint(cand[wq][0].x);
            double2 v[ZGW];
#pragma unroll
            for (int c = jj; c < ZGW; ++c) v[c] = cand[wq][1 + c - jj];
            const bool ok = !(is_zero(v[jj].x) && is_zero(v[jj].y));
            if (ok) live |= 1u << jj;
            if (t == 0) {
                s_piv[j] = wp;
                if (!ok && s_info == 0) s_info = j + 1;
            }
            const int p = pos;
            pos = p == wp ? j : (p == j ? wp : p);
            if (ok && p >= j && p != wp) {
                const zd l = zmul({r[jj].x, r[jj].y}, {dinv.x, dinv.y});
                r[jj] = make_double2(l.r, l.i);
#pragma unroll
                for (int c = jj + 1; c < ZGW; ++c) r[c] = zmsub2(r[c], r[jj], v[c]);
            }
        }
        const int np = min(ZGW, q - j0), nblk = ZNG - 1 - s;
        if (np > 0 && nblk > 0 && j0 + np < w) {
            const int rem = nblk * ZGW, nch = ZGW + rem;
            if (CS > 1 && t == 0 && !dead) mbar_arrive_expect_tx(&s_rbar, (uint32_t)(np * nch * 16));
            const int kk = pos - j0;
            const bool own = pos >= j0 && kk < np;
            if (own) {
                double2 *dst = (CS > 1) ? s_stage[kk] : s_right[kk];
#pragma unroll
                for (int b = 0; b < ZNG; ++b)
                    if (b <= nblk)
#pragma unroll
                        for (int c = 0; c < ZGW; ++c) dst[b * ZGW + c] = r[b * ZGW + c];
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
                                        reinterpret_cast<const uint4 *>(s_stage[ks])[c], smem_u32(&s_rbar) + to_cta);
                }
                if (warp == 0 && !dead && !mbar_wait(&s_rbar, (uint32_t)(s & 1), pn.abort, 1)) dead = true;
            } else {
                __syncthreads();
            }
            const bool full = live == (1u << ZGW) - 1;
            if (warp == 0 && lane < rem) {
                double2 x[ZGW];
#pragma unroll
                for (int k = 0; k < ZGW; ++k) x[k] = k < np ? s_right[k][ZGW + lane] : make_double2(0.0, 0.0);
#pragma unroll
                for (int p = 0; p < ZGW; ++p)
#pragma unroll
                    for (int k = p + 1; k < ZGW; ++k)
                        if (full || (((live >> p) & 1) && k < np)) x[k] = zmsub2(x[k], s_right[k][p], x[p]);
#pragma unroll
                for (int k = 0; k < ZGW; ++k) s_u[k][lane] = x[k];
            }
            __syncthreads();
            const bool act = pos >= j0 + np;
#pragma unroll
            for (int b = 0; b < ZNG - 1; ++b) {
                if (b < nblk) {
                    if (act) {
#pragma unroll
                        for (int p = 0; p < ZGW; ++p)
                            if ((live >> p) & 1)
#pragma unroll
                                for (int c = 0; c < ZGW; ++c)
                                    r[(b + 1) * ZGW + c] = zmsub2(r[(b + 1) * ZGW + c], r[p], s_u[p][b * ZGW + c]);
                    } else if (own) {
#pragma unroll
                        for (int c = 0; c < ZGW; ++c) r[(b + 1) * ZGW + c] = s_u[kk][b * ZGW + c];
                    }
                }
            }
        }
        // the finished group moves behind the unfinished columns
        double2 f[ZGW];
#pragma unroll
        for (int c = 0; c < ZGW; ++c) f[c] = r[c];
#pragma unroll
        for (int c = 0; c < ZLEAF - ZGW; ++c) r[c] = r[c + ZGW];
#pragma unroll
        for (int c = 0; c < ZGW; ++c) r[ZLEAF - ZGW + c] = f[c];
    }
    dead = __syncthreads_or(dead);
    if (!dead && cr == 0) {
        if (t < q) ipiv[gofs + t] = gofs + s_piv[t] + 1;
        if (t == 0 && s_info != 0 && *info == 0) *info = gofs + s_info;
    }
    const bool moved = !dead && pos >= 0 && pos != i0;
    if (!dead) {
        if (moved && pn.map) {
            const int slot = atomicAdd(&s_mcnt, 1);
            s_mv[slot] = make_int2(pos, i0);
        }
        if (vec_ok) {
#pragma unroll
            for (int pl = 0; pl < 2; ++pl) {
#pragma unroll
                for (int c = 0; c < ZLEAF; c += 2)
                    *(double2 *)(tr + lane * 144 + c * 8) =
                        pl == 0 ? make_double2(r[c].x, r[c + 1].x) : make_double2(r[c].y, r[c + 1].y);
                __syncwarp();
#pragma unroll
                for (int it = 0; it < 8; ++it) {
                    const int dst = __shfl_sync(0xffffffffu, pos, it * 4 + trow);
                    if (dst >= 0)
                        *(double2 *)((pl ? Wi : Wr) + (i64)dst * ld + 2 * tchk) =
                            *(const double2 *)(tr + (it * 4 + trow) * 144 + tchk * 16);
                }
                __syncwarp();
            }
        } else if (pos >= 0) {
#pragma unroll
            for (int c = 0; c < ZLEAF; ++c)
                if (c < w) {
                    Wr[(i64)pos * ld + c] = r[c].x;
                    Wi[(i64)pos * ld + c] = r[c].y;
                }
        }
    }
    if (pn.map) {
        // the interchanges on the panel's other columns and on its row map, as
        // the real leaf: read, meet, write
        const int mapv = moved ? pn.map[pn.map_off + i0] : 0;
        __syncthreads();
        const int cnt = s_mcnt, nother = pn.nother;
        double *const br = Wr - pn.leaf_c0, *const bi = Wi - pn.leaf_c0;
        int off[MOVE_CH];
#pragma unroll
        for (int ci = 0; ci < MOVE_CH; ++ci) {
            const int oc = ci * 32 + lane;
            off[ci] = oc >= nother ? -1 : (oc < pn.left_n ? pn.pc_lo + oc : pn.right_lo + (oc - pn.left_n));
        }
        double2 vals[MOVE_PW][MOVE_CH];
#pragma unroll
        for (int mi = 0; mi < MOVE_PW; ++mi) {
            const int mv = warp + mi * NW;
            if (mv < cnt) {
                const i64 src = (i64)s_mv[mv].y * ld;
#pragma unroll
                for (int ci = 0; ci < MOVE_CH; ++ci)
                    if (off[ci] >= 0) vals[mi][ci] = make_double2(br[src + off[ci]], bi[src + off[ci]]);
            }
        }
        if (CS > 1) cl.sync();
        else __syncthreads();
#pragma unroll
        for (int mi = 0; mi < MOVE_PW; ++mi) {
            const int mv = warp + mi * NW;
            if (mv < cnt) {
                const i64 dst = (i64)s_mv[mv].x * ld;
#pragma unroll
                for (int ci = 0; ci < MOVE_CH; ++ci)
                    if (off[ci] >= 0) {
                        br[dst + off[ci]] = vals[mi][ci].x;
                        bi[dst + off[ci]] = vals[mi][ci].y;
                    }
            }
        }
        if (moved) pn.map[pn.map_off + pos] = mapv;
    } else if (CS > 1) {
        cl.sync();  // every push into a CTA that gave up has landed before its shared memory goes
    }
}

// laswp: the interchanges ipiv[k0 .. k0+cnt) (global 1-based rows, cnt <= 16)
// on columns [c_lo, c_hi) of both planes.  Their net effect is at most 2 cnt
// row moves (dst <- src); thread 0 of each CTA folds the sequence into that
// list, then every thread moves its column: all sources read, then all
// destinations written (one round trip instead of cnt dependent swaps).
constexpr int ZSWP_MAX = 2 * ZLEAF;
__global__ void k_zlaswp(double *__restrict__ Wr, double *__restrict__ Wi, i64 ld, const int64_t *__restrict__ ipiv,
                         i64 k0, int cnt, i64 c_lo, i64 c_hi, i64 skip_lo, i64 skip_hi) {
    __shared__ i64 s_dst[ZSWP_MAX], s_src[ZSWP_MAX];
    __shared__ int s_n;
    if (threadIdx.x == 0) {
        i64 key[ZSWP_MAX], val[ZSWP_MAX];  // position -> row now there (absent: itself)
        int nk = 0;
        auto find = [&](i64 x) {
            for (int q = 0; q < nk; ++q)
                if (key[q] == x) return q;
            key[nk] = x;
            val[nk] = x;
            return nk++;
        };
        for (int t = 0; t < cnt; ++t) {
            const i64 j = k0 + t, p = ipiv[j] - 1;
            if (p == j) continue;
            const int a = find(j), b = find(p);
            const i64 tmp = val[a];
            val[a] = val[b];
            val[b] = tmp;
        }
        int nm = 0;
        for (int q = 0; q < nk; ++q)
            if (val[q] != key[q]) {
                s_dst[nm] = key[q];
                s_src[nm] = val[q];
                ++nm;
            }
        s_n = nm;
    }
    __syncthreads();
    const int nm = s_n;
    const i64 c = c_lo + (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (nm == 0 || c >= c_hi || (c >= skip_lo && c < skip_hi)) return;
    double vr[ZSWP_MAX], vi[ZSWP_MAX];
#pragma unroll
    for (int q = 0; q < ZSWP_MAX; ++q)
        if (q < nm) {
            vr[q] = Wr[s_src[q] * ld + c];
            vi[q] = Wi[s_src[q] * ld + c];
        }
#pragma unroll
    for (int q = 0; q < ZSWP_MAX; ++q)
        if (q < nm) {
            Wr[s_dst[q] * ld + c] = vr[q];
            Wi[s_dst[q] * ld + c] = vi[q];
        }
}

// B (t x N at (Br, Bi), ld) <- L^-1 B, L the unit lower t x t block at (Lr, Li),
// t <= ZT_MAXT: a CTA per ZT_CW columns, its columns and L's strict lower
// triangle in shared memory (loaded once, everything in flight together).  By
// blocks of 8 rows: the block by substitution, a column per thread, then its
// products subtracted from the rows below.  Bound: latency of the 2 t / 8 steps.
constexpr int ZT_NT = 256, ZT_CW = 16, ZT_MAXT = 64, ZT_RB = 8;
__global__ void __launch_bounds__(ZT_NT) k_ztrsm_lunit(const double *__restrict__ Lr, const double *__restrict__ Li,
                                                       double *__restrict__ Br, double *__restrict__ Bi, i64 ld,
                                                       int t, i64 N) {
    extern __shared__ double2 zt[];  // [t][ZT_CW], then L [t][ZT_MAXT + 1]
    double2 *Ls = zt + t * ZT_CW;
    constexpr int LP = ZT_MAXT + 1;
    const int tid = threadIdx.x, cl = tid % ZT_CW, rg = tid / ZT_CW;
    constexpr int RG = ZT_NT / ZT_CW;
    const i64 c0 = (i64)blockIdx.x * ZT_CW;
    const bool live = c0 + cl < N;
#pragma unroll 8
    for (int e = tid; e < t * ZT_MAXT; e += ZT_NT) {
        const int i = e / ZT_MAXT, p = e % ZT_MAXT;
        if (p < i) Ls[i * LP + p] = make_double2(Lr[(i64)i * ld + p], Li[(i64)i * ld + p]);
    }
#pragma unroll 4
    for (int r = rg; r < t; r += RG)
        zt[r * ZT_CW + cl] = live ? make_double2(Br[(i64)r * ld + c0 + cl], Bi[(i64)r * ld + c0 + cl])
                                  : make_double2(0.0, 0.0);
    __syncthreads();
    for (int b = 0; b < t; b += ZT_RB) {
        if (tid < ZT_CW) {
            double2 x[ZT_RB];
#pragma unroll
            for (int i = 0; i < ZT_RB; ++i) x[i] = b + i < t ? zt[(b + i) * ZT_CW + tid] : make_double2(0.0, 0.0);
#pragma unroll
            for (int p = 0; p < ZT_RB; ++p)
#pragma unroll
                for (int i = p + 1; i < ZT_RB; ++i)
                    if (b + i < t) x[i] = zmsub2(x[i], Ls[(b + i) * LP + b + p], x[p]);
#pragma unroll
            for (int i = 1; i < ZT_RB; ++i)
                if (b + i < t) zt[(b + i) * ZT_CW + tid] = x[i];
        }
        __syncthreads();
        for (int r = b + ZT_RB + rg; r < t; r += RG) {
            double2 v = zt[r * ZT_CW + cl];
#pragma unroll
            for (int p = 0; p < ZT_RB; ++p) v = zmsub2(v, Ls[r * LP + b + p], zt[(b + p) * ZT_CW + cl]);
            zt[r * ZT_CW + cl] = v;
        }
        __syncthreads();
    }
    if (live)
        for (int r = rg + (rg == 0 ? RG : 0); r < t; r += RG) {  // row 0 is unchanged
            const double2 v = zt[r * ZT_CW + cl];
            Br[(i64)r * ld + c0 + cl] = v.x;
            Bi[(i64)r * ld + c0 + cl] = v.y;
        }
}

// dst = -src (rows x cols, row-major, lds / ldd)
__global__ void k_negate(const double *__restrict__ src, i64 lds, double *__restrict__ dst, i64 ldd, i64 rows,
                         i64 cols) {
    const i64 idx = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= rows * cols) return;
    const i64 r = idx / cols, c = idx - r * cols;
    dst[r * ldd + c] = -src[r * lds + c];
}

// interleaved column-major (m x n, lda) <-> two row-major planes (ld)
__global__ void k_z_split(const double2 *__restrict__ A, i64 lda, double *__restrict__ Wr, double *__restrict__ Wi,
                          i64 ld, i64 m, i64 n) {
    __shared__ double2 tile[32][33];
    const i64 i0 = (i64)blockIdx.x * 32, j0 = (i64)blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int r = ty; r < 32; r += 8) {
        const i64 i = i0 + tx, j = j0 + r;
        if (i < m && j < n) tile[r][tx] = A[i + j * lda];
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const i64 i = i0 + r, j = j0 + tx;
        if (i < m && j < n) {
            const double2 v = tile[tx][r];
            Wr[i * ld + j] = v.x;
            Wi[i * ld + j] = v.y;
        }
    }
}
__global__ void k_z_merge(const double *__restrict__ Wr, const double *__restrict__ Wi, i64 ld, double2 *__restrict__ A,
                          i64 lda, i64 m, i64 n) {
    __shared__ double2 tile[32][33];
    const i64 i0 = (i64)blockIdx.x * 32, j0 = (i64)blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int r = ty; r < 32; r += 8) {
        const i64 i = i0 + r, j = j0 + tx;
        if (i < m && j < n) tile[r][tx] = make_double2(Wr[i * ld + j], Wi[i * ld + j]);
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const i64 i = i0 + tx, j = j0 + r;
        if (i < m && j < n) A[i + j * lda] = tile[tx][r];
    }
}

struct ZRun {
    oxi_handle_s *h;
    double *Wr, *Wi;
    i64 ld, m, n;
    int64_t *ipiv, *info;
    double *neg;  // -Ai scratch (m x (nb + 2))
    i64 nb;       // panel width (lu_factor's blocksize, 128 by default)
    // the current panel [pf, pl) and its row map (null: every leaf's interchanges
    // go to all other columns at once)
    i64 pf = 0, pl = 0;
    int *map = nullptr, *list = nullptr, *listcnt = nullptr;
};

// C -= A B on complex planes (row-major, common ld).
static void zgemm_minus(ZRun &R, i64 cr, i64 cc, i64 ar, i64 ac, i64 br, i64 bc, i64 M, i64 N, i64 K) {
    if (M <= 0 || N <= 0 || K <= 0) return;
    cudaStream_t s = R.h->stream;
    const i64 ld = R.ld;
    double *Cr = R.Wr + cr * ld + cc, *Ci = R.Wi + cr * ld + cc;
    const double *Ar = R.Wr + ar * ld + ac, *Ai = R.Wi + ar * ld + ac;
    const double *Bre = R.Wr + br * ld + bc, *Bim = R.Wi + br * ld + bc;
    if (zgemm_dmma_applicable(Ar, Ai, Bre, Bim, ld)) {
        launch_zgemm_dmma(Cr, Ci, Ar, Ai, Bre, Bim, ld, M, N, K, s);
        return;
    }
    // an odd column offset (an odd panel width): the plain kernel, plane by plane
    const i64 ldn = zrup(K, 2);
    k_negate<<<(unsigned)((M * K + 255) / 256), 256, 0, s>>>(Ai, ld, R.neg, ldn, M, K);
    OXI_LAUNCH_CHECK();
    launch_gemm_dmma(Cr, ld, Ar, ld, Bre, ld, M, N, K, s);
    launch_gemm_dmma(Cr, ld, R.neg, ldn, Bim, ld, M, N, K, s);
    launch_gemm_dmma(Ci, ld, Ar, ld, Bim, ld, M, N, K, s);
    launch_gemm_dmma(Ci, ld, Ai, ld, Bre, ld, M, N, K, s);
}

static void ztrsm(ZRun &R, i64 r0, i64 c0, int t, i64 bc, i64 N) {
    if (t <= 1 || N <= 0) return;
    const i64 ld = R.ld;
    if (t > ZT_MAXT) {  // a wider block: the top rows, their update of the rest, the rest
        const int h = ZT_MAXT;
        ztrsm(R, r0, c0, h, bc, N);
        zgemm_minus(R, r0 + h, bc, r0 + h, c0, r0, bc, t - h, N, h);
        ztrsm(R, r0 + h, c0 + h, t - h, bc, N);
        return;
    }
    const int smem = (int)(sizeof(double2) * t * (ZT_CW + ZT_MAXT + 1));
    set_max_dyn_smem((const void *)k_ztrsm_lunit, (int)(sizeof(double2) * ZT_MAXT * (ZT_CW + ZT_MAXT + 1)));
    k_ztrsm_lunit<<<(unsigned)((N + ZT_CW - 1) / ZT_CW), ZT_NT, smem, R.h->stream>>>(
        R.Wr + r0 * ld + c0, R.Wi + r0 * ld + c0, R.Wr + r0 * ld + bc, R.Wi + r0 * ld + bc, ld, t, N);
    OXI_LAUNCH_CHECK();
}

static void zlaswp(ZRun &R, i64 k0, int cnt, i64 c_lo, i64 c_hi, i64 skip_lo, i64 skip_hi) {
    if (c_hi <= c_lo || cnt <= 0) return;
    if (cnt > ZLEAF) throw CudaError{cudaErrorInvalidValue, "more interchanges than a complex leaf makes"};
    const i64 cols = c_hi - c_lo;
    k_zlaswp<<<(unsigned)((cols + 127) / 128), 128, 0, R.h->stream>>>(R.Wr, R.Wi, R.ld, R.ipiv, k0, cnt, c_lo, c_hi,
                                                                        skip_lo, skip_hi);
    OXI_LAUNCH_CHECK();
}

constexpr i64 ZREG_MAXM = 16 * 512;  // rows of the register leaf
template <int NT>
static void launch_zleaf_reg(ZRun &R, i64 c0, i64 mrows, int nc, LeafPanel pn) {
    const int cs = (int)((mrows + NT - 1) / NT);
    auto kern = k_zleaf_reg<NT>;
    constexpr int smem = (NT / 32) * 32 * 144;
    set_max_dyn_smem((const void *)kern, smem);
    if (cs > 8) OXI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = R.h->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    ProfScope ps(KC_LEAF, R.h->stream, 0.0, 32.0 * (double)mrows * nc);
    OXI_CUDA(cudaLaunchKernelEx(&cfg, kern, R.Wr + c0 * R.ld + c0, R.Wi + c0 * R.ld + c0, R.ld, (int)mrows, nc, c0, R.ipiv,
                                R.info, pn));
    count_launch();
}

// _lu_panel! on columns [c0, c0+nc), rows [c0, m).  With a row map (R.map) the leaf
// moves the panel's other columns and the caller the columns outside it; without,
// its interchanges go to every other column right after it.  Either way each
// column receives the reference's sequence.
static void zpanel(ZRun &R, i64 c0, i64 nc) {
    const i64 mrows = R.m - c0;
    if (mrows <= 0 || nc <= 0) return;
    if (nc <= ZLEAF && mrows <= ZREG_MAXM) {
        LeafPanel pn;
        if (R.map) {
            pn.left_n = (int)(c0 - R.pf);
            pn.nother = (int)((c0 - R.pf) + (R.pl - c0 - nc));
            pn.pc_lo = (int)R.pf;
            pn.right_lo = (int)(c0 + nc);
            pn.leaf_c0 = (int)c0;
            pn.map = R.map;
            pn.map_off = (int)(c0 - R.pf);
        }
        pn.abort = cur_abort();
        if (mrows <= 16 * 256) launch_zleaf_reg<256>(R, c0, mrows, (int)nc, pn);
        else launch_zleaf_reg<512>(R, c0, mrows, (int)nc, pn);
        if (!R.map) zlaswp(R, c0, (int)std::min<i64>(nc, mrows), 0, R.n, c0, c0 + nc);
        return;
    }
    if (nc <= ZLEAF) {
        if (mrows <= (i64)ZCL_MAXRP * 16) {
            // rows over a cluster of up to 16 CTAs, in shared memory
            int cs = (int)std::min<i64>(16, std::max<i64>(1, (mrows + 511) / 512));
            int rp = (int)((mrows + cs - 1) / cs);
            while (rp > ZCL_MAXRP) rp = (int)((mrows + (++cs) - 1) / cs);
            const size_t smem = sizeof(double2) * (size_t)rp * ZLEAF;
            set_max_dyn_smem((const void *)k_zleaf_cl, (int)(sizeof(double2) * ZCL_MAXRP * ZLEAF));
            if (cs > 8) OXI_CUDA(cudaFuncSetAttribute(k_zleaf_cl, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(cs);
            cfg.blockDim = dim3(ZCL_NT);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = R.h->stream;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = cs;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            OXI_CUDA(cudaLaunchKernelEx(&cfg, k_zleaf_cl, R.Wr + c0 * R.ld + c0, R.Wi + c0 * R.ld + c0, R.ld,
                                        (int)mrows, (int)nc, rp, c0, R.ipiv, R.info));
        } else {
            k_zleaf<<<1, ZLEAF_NT, 0, R.h->stream>>>(R.Wr + c0 * R.ld + c0, R.Wi + c0 * R.ld + c0, R.ld, (int)mrows,
                                                     (int)nc, c0, R.ipiv, R.info);
        }
        OXI_LAUNCH_CHECK();
        const int cnt = (int)std::min<i64>(nc, mrows);
        zlaswp(R, c0, cnt, 0, R.n, c0, c0 + nc);
        return;
    }
    const i64 h = nc / 2;
    zpanel(R, c0, h);
    ztrsm(R, c0, c0, (int)h, c0 + h, nc - h);
    if (mrows > h) {
        zgemm_minus(R, c0 + h, c0 + h, c0 + h, c0, c0, c0 + h, mrows - h, nc - h, h);
        zpanel(R, c0 + h, nc - h);
    }
}

static void zgetrf_planes(ZRun &R) {
    const i64 q = std::min(R.m, R.n);
    int *map0 = nullptr;
    if (R.nb <= LEAF_MAX_OTHER) {
        map0 = (int *)R.h->rowmap_ws.get(sizeof(int) * (size_t)(R.m + 4 * R.nb + 64));
        R.list = map0 + R.m;
        R.listcnt = R.list + 4 * R.nb;
    }
    for (i64 f = 0; f < q; f += R.nb) {
        const i64 l = std::min(q, f + R.nb);
        // a panel of register leaves applies its interchanges to the columns
        // outside it once, composed
        int *const map = R.m - f <= ZREG_MAXM ? map0 : nullptr;
        R.map = map;
        R.pf = f;
        R.pl = l;
        if (map) launch_rowmap_init(map, R.m - f, R.listcnt, R.h->stream);
        zpanel(R, f, l - f);
        if (map) {
            launch_rowmap_extract(map, R.m - f, R.list, R.listcnt, R.h->stream);
            const int maxcnt = (int)std::min<i64>(2 * (l - f), R.m - f);
            for (double *W : {R.Wr, R.Wi}) {
                launch_rowmoves_big<double>(W, R.ld, f, R.list, R.listcnt, maxcnt, 0, f, R.h->stream);
                launch_rowmoves_big<double>(W, R.ld, f, R.list, R.listcnt, maxcnt, l, R.n, R.h->stream);
            }
        }
        if (l >= R.n) continue;
        ztrsm(R, f, f, (int)(l - f), l, R.n - l);
        if (l >= R.m) continue;
        zgemm_minus(R, l, l, l, f, f, l, R.m - l, R.n - l, l - f);
    }
}

}  // namespace oxi

extern "C" int oxi_zgetrf(oxi_handle_t h, int64_t m, int64_t n, void *dA, int64_t lda, int64_t *d_ipiv,
                          int64_t *h_info) {
    using namespace oxi;
    if (!h || !h_info || m < 0 || n < 0 || lda < std::max<int64_t>(1, m)) return OXI_EINVAL;
    *h_info = 0;
    if (m == 0 || n == 0) return OXI_OK;
    if (!dA || !d_ipiv || m >= (1ll << 31) || n >= (1ll << 31)) return OXI_EINVAL;
    if ((uintptr_t)dA % 16) return OXI_EINVAL;  // ComplexF64 elements are 16-byte aligned
    try {
        ProfGuard pg(&h->prof);
        OXI_CUDA(cudaSetDevice(h->device));
        AbortScope ab(h);
        const i64 ld = zrup(n, 32), nb = std::max<i64>(1, h->opt.blocksize);
        double *W = (double *)h->work.get(sizeof(double) * (2 * (size_t)m * ld + (size_t)m * (nb + 2) + 64));
        ZRun R{h, W, W + (size_t)m * ld, ld, m, n, d_ipiv, nullptr, W + 2 * (size_t)m * ld, nb};
        char *sc = (char *)h->scratch.get(kScratchBytes);
        R.info = (int64_t *)sc;
        cudaStream_t s = h->stream;
        OXI_CUDA(cudaMemsetAsync(R.info, 0, sizeof(int64_t), s));
        dim3 g((unsigned)((m + 31) / 32), (unsigned)((n + 31) / 32));
        k_z_split<<<g, dim3(32, 8), 0, s>>>((const double2 *)dA, lda, R.Wr, R.Wi, ld, m, n);
        OXI_LAUNCH_CHECK();
        zgetrf_planes(R);
        k_z_merge<<<g, dim3(32, 8), 0, s>>>(R.Wr, R.Wi, ld, (double2 *)dA, lda, m, n);
        OXI_LAUNCH_CHECK();
        int64_t *hi = (int64_t *)h->host_ws.get(64);
        OXI_CUDA(cudaMemcpyAsync(hi, R.info, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
        queue_abort_read(h, (int *)(hi + 2));
        OXI_CUDA(cudaStreamSynchronize(s));
        *h_info = hi[0];
        const int we = check_abort(h, (const int *)(hi + 2));
        if (we != OXI_OK) return we;
        return hi[0] > 0 ? OXI_ESINGULAR : OXI_OK;
    } catch (const CudaError &e) {
        h->last_error = std::string(e.what) + ": " + cudaGetErrorString(e.code);
        return OXI_ECUDA;
    }
}
