// Triangular solves with up to 16 right-hand sides per launch (ldiv!, the
// refinement's corrections, Cholesky's two solves).
//
// A triangle is taken in solve order: M(i, j) = a[i rs + j cs] is lower
// triangular, an upper one being read from its last row and column with
// negated strides.  Its rows form superblocks of SP = 256, each of NS = 8 strips
// of ST = 32 rows.  For superblock B
//     x_B = Inv_B (b_B - sum_{C < B} M(B, C) x_C),   Inv_B = M(B, B)^-1,
// the inverses computed once per factor (k_tri_inv).  k_tri_solve is ONE launch
// per triangle: a cluster of NS CTAs takes the next superblock from a ticket
// (everything it waits on is already running), one strip per CTA.  Each CTA
// accumulates its strip's products with the solved superblocks as they
// appear, the strips meet at a cluster barrier and read each other's
// right-hand sides through distributed shared memory, and each multiplies by
// its strip of Inv_B and publishes its 32 rows.
//
// A product with an inverse is not backward stable: its error grows with the
// condition of the block, that of substitution does not.  k_tri_inv therefore
// leaves an estimate E of the inverse's quality with each strip, the largest row
// sum of |Inv||M| times that of the 32 x 32 diagonal blocks (whose explicit
// inverses the strip's rows are made with), and a superblock is solved by its
// largest E:
//   E <= kTriPlain: the product as it is (errors within a few roundings of
//     substitution's);
//   E <= tri_limit: one correction with the triangle itself, x += Inv (r - M x);
//   beyond, and where a right-hand side or the product is not finite:
//     substitution, the strips in turn.
// Backward errors max|b - A x| / (|A||x| + |b|) of a solve by this rule's three forms,
// in units of n eps (substitution / product / corrected), b = A * ones, kernels
// exp(-((i-j)/w)^2) of order 512 restated in NumPy with these kernels' association:
//   FP64 w = 1.4 (E = 60): 3e-3 / 5e-3 / 1e-3;  w = 2.2 (4e7): 2e-3 / 3e1 / 1e-3;
//   w = 2.6 (2e11): 3e-3 / 1e5 / 2e-3;  w = 2.8 (6e13): 3e-3 / 5e7 / 2e1, and beyond
//   that the correction fails altogether: the limit lies at 2^38 = 3e11;
//   FP32 w = 2 (1e6): 3e-3 / 3 / 2e-3;  w = 2.1 (1e7): 3e-3 / 2e1 / 2e-3;  w = 2.2 (4e7):
//   2e-3 / 1e1 / 5e-3;  w = 2.4 (6e9): 3e-3 / 4e2 / 3e1: 2^25 = 3e7.
// Factors of random matrices have E of 4e5 to 4e7 and are corrected: 1e-2 / 5e-2 /
// 1e-2 at order 1024.
//
// Bound: for one right-hand side of a large system the single pass over the
// factor, otherwise the chain of superblocks: one hop through L2, the 32 x SP product
// with the last superblock solved, then three 32 x SP products (with 8 FP64 right-hand
// sides 2300 cycles each, 750 of them the other strips' values) and three cluster
// barriers (950 each) per SP rows.  Measured on one B200 against
// the form it replaces (64-row blocks, a hop through L2 per block): see the
// figures at trsv_pair.
//
// A solved value is its own flag: the exchange buffer starts as all-ones words
// (one memset per launch pair, the tickets included), which no published value
// equals, and a reader polls the data itself.
#include <cooperative_groups.h>
#include <algorithm>
#include <type_traits>
#include "oxi_internal.h"
#include "tma_util.cuh"

namespace cg = cooperative_groups;

namespace oxi {

namespace {
constexpr int ST = 32;
// rows of a superblock: half as many for complex elements, whose inverse's strip
// would not fit shared memory otherwise
template <typename T> constexpr int SP_ = sizeof(T) == 16 ? 128 : 256;
constexpr int INV_NT = 256;
// The estimates up to which a superblock's product stands as it is, and with one
// correction (see above).
constexpr double kTriPlain = 64.0;
template <typename T> constexpr double tri_limit = sizeof(T) == 4 ? 0x1p25 : 0x1p38;

// One effective triangle in solve order.
template <typename T>
struct TriView {
    const T *a;
    i64 rs, cs;
    int n;
    int unit;  // unit diagonal, not stored
    int rev;   // solve order runs from the last row to the first
    int conj;  // complex elements conjugated
};

// c + a b
__device__ __forceinline__ float mad(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ zc64 mad(zc64 a, zc64 b, zc64 c) {
    return zc64(fma(-a.y, b.y, fma(a.x, b.x, c.x)), fma(a.y, b.x, fma(a.x, b.y, c.y)));
}
__device__ __forceinline__ float shfl_xor(float v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ double shfl_xor(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ zc64 shfl_xor(zc64 v, int o) {
    return zc64(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
__device__ __forceinline__ float shfl(float v, int l) { return __shfl_sync(0xffffffffu, v, l); }
__device__ __forceinline__ double shfl(double v, int l) { return __shfl_sync(0xffffffffu, v, l); }
__device__ __forceinline__ zc64 shfl(zc64 v, int l) {
    return zc64(__shfl_sync(0xffffffffu, v.x, l), __shfl_sync(0xffffffffu, v.y, l));
}
// size of an element (complex: within sqrt(2)), and whether it is finite
__device__ __forceinline__ float mag(float v) { return fabsf(v); }
__device__ __forceinline__ double mag(double v) { return fabs(v); }
__device__ __forceinline__ double mag(zc64 v) { return fabs(v.x) + fabs(v.y); }
__device__ __forceinline__ bool is_finite(float v) { return isfinite(v); }
__device__ __forceinline__ bool is_finite(double v) { return isfinite(v); }
__device__ __forceinline__ bool is_finite(zc64 v) { return isfinite(v.x) && isfinite(v.y); }
// the estimate beside the inverses, stored as an element
__device__ __forceinline__ double est_value(float v) { return v; }
__device__ __forceinline__ double est_value(double v) { return v; }
__device__ __forceinline__ double est_value(zc64 v) { return v.x; }
__device__ __forceinline__ float conj_if(float v, int) { return v; }
__device__ __forceinline__ double conj_if(double v, int) { return v; }
__device__ __forceinline__ zc64 conj_if(zc64 v, int c) { return zc64(v.x, c ? -v.y : v.y); }

template <typename T>
TriView<T> tri_view(const T *A, i64 lda, i64 n, bool lower, bool unit, bool rowacc, bool conj = false) {
    TriView<T> v{A, rowacc ? lda : 1, rowacc ? 1 : lda, (int)n, unit ? 1 : 0, lower ? 0 : 1, conj ? 1 : 0};
    if (!lower) {
        v.a = A + (n - 1) * (v.rs + v.cs);
        v.rs = -v.rs;
        v.cs = -v.cs;
    }
    return v;
}
}  // namespace

// ---------------------------------------------------------------------------
// Strip s of every superblock's inverse, one CTA per strip and triangle: the
// row strip Y of L^-1 solves Y L = E_s, from the diagonal to the left:
// Y_s = L_ss^-1, Y_t = -(sum_{t < u <= s} Y_u L_ut) L_tt^-1, with the 32 x 32
// diagonal inverses by substitution, one warp each, the column of a lane in its
// registers.  Each block column's elements are requested before the products
// of the one before it.  FP64 products run on the tensor cores, a 16 x 8 tile
// per warp.  Written column by column, P[(strip * SP + c) * ST + r], zero to the
// right of the diagonal; rows past n are those of the identity; behind them the
// strips' estimates (see the head of the file).  Bound: latency
// of the block columns' steps (up to seven, each two barriers and a chain of
// up to 64 DMMAs); both triangles of a factor are one launch.
// 62000 cycles for the longest strip (32000 of them DMMAs and their loads, 21000
// the fetches, 12000 the diagonal inverses), 71000 before a diagonal block's
// loads were issued together, and about 5000 for the estimate.
// ---------------------------------------------------------------------------
template <typename T>
struct TriInvSmem {
    static constexpr int SP = SP_<T>, NS = SP / ST;
    static constexpr int DP = ST + 4, YP = SP + 4;  // FP64: 4 modulo 16, no conflicts of a DMMA fragment's loads
    T D[NS][ST][DP];
    T L[(NS - 1) * ST][DP];
    T Z[ST][DP];
    T Y[ST][YP];
};

// a / d from d's reciprocal, corrected by the remainder; the division where that
// leaves the finite numbers
template <typename T>
__device__ __forceinline__ T quotient(T a, T d, T r) {
    const T q = a * r;
    const T l = mad(mad(-q, d, a), r, q);
    return isfinite(l) ? l : a / d;
}

// out (32 x 32) = +-A (32 x K, pitch ap) B (K x 32, pitch bp), one call by the CTA
template <typename T>
__device__ __forceinline__ void inv_product(const T *A, int ap, const T *B, int bp, int K, T *out, int op, bool neg) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if constexpr (sizeof(T) == 8) {
        const int m0 = (warp & 1) * 16, n0 = (warp >> 1) * 8, gid = lane >> 2, tig = lane & 3;
        double c[2][4] = {};  // two chains of products
#pragma unroll 4
        for (int k = 0; k < K; k += 8) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int kc = k + 4 * h + tig;
                const double a0 = A[(m0 + gid) * ap + kc], a1 = A[(m0 + gid + 8) * ap + kc], b = B[kc * bp + n0 + gid];
                asm volatile(
                    "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                    : "+d"(c[h][0]), "+d"(c[h][1]), "+d"(c[h][2]), "+d"(c[h][3])
                    : "d"(a0), "d"(a1), "d"(b));
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const double v = c[0][e] + c[1][e];
            out[(m0 + gid + 8 * (e >> 1)) * op + n0 + 2 * tig + (e & 1)] = neg ? -v : v;
        }
    } else {
        const int row = t >> 3, c4 = (t & 7) * 4;
        T z[4] = {T(0), T(0), T(0), T(0)};
        const T *y = A + row * ap;
#pragma unroll 8
        for (int k = 0; k < K; ++k) {
            const T yv = y[k];
#pragma unroll
            for (int u = 0; u < 4; ++u) z[u] = mad(yv, B[k * bp + c4 + u], z[u]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) out[row * op + c4 + u] = neg ? -z[u] : z[u];
    }
}

template <typename T>
__global__ void __launch_bounds__(INV_NT, 1) k_tri_inv(const TriView<T> v0, const TriView<T> v1, T *__restrict__ P0,
                                                    T *__restrict__ P1) {
    constexpr int SP = SP_<T>, NS = SP / ST, DP = TriInvSmem<T>::DP, YP = TriInvSmem<T>::YP;
    constexpr int PRE = (NS - 1) * ST * ST / INV_NT;
    extern __shared__ __align__(16) unsigned char tri_smem[];
    TriInvSmem<T> &S = *reinterpret_cast<TriInvSmem<T> *>(tri_smem);
    const TriView<T> &v = blockIdx.y ? v1 : v0;
    T *P = blockIdx.y ? P1 : P0;
    using R = decltype(mag(T()));
    __shared__ R s_w[SP];          // row sums of |M|, rows up to this strip's
    __shared__ R s_k[NS], s_e[INV_NT / 32];  // |D^-1||D| of the diagonal blocks, |Y||M| of a warp's rows
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int g = blockIdx.x, s = g % NS;
    auto larger = [](R a, R b) { return (a >= b || a != a) ? a : b; };  // keeps a NaN
    // sum of |row| over ST columns, from the lane's own on (no bank conflicts), four
    // chains of additions
    auto row_sum = [&](const T *row) {
        R a[4] = {R(0), R(0), R(0), R(0)};
#pragma unroll
        for (int e = 0; e < ST; ++e) a[e & 3] += mag(row[(e + lane) & 31]);
        return (a[0] + a[1]) + (a[2] + a[3]);
    };
    const i64 r0 = (i64)(g / NS) * SP;  // the superblock's first row
    const bool rowacc = v.cs == 1 || v.cs == -1;
    const T *base = v.a + r0 * (v.rs + v.cs);
    const int nrow = (int)(v.n - r0 < SP ? v.n - r0 : SP);
    // the elements below diagonal block b: K = (s - b) ST rows, ST columns
    T pre[PRE];
    auto place = [&](int q, int &i, int &j) {  // element q of this thread
        const int e = t + INV_NT * q;
        i = rowacc ? e / ST : (e / (ST * ST)) * ST + e % ST;
        j = rowacc ? e % ST : (e / ST) % ST;
    };
    auto fetch = [&](int b) {
#pragma unroll
        for (int q = 0; q < PRE; ++q) {
            int i, j;
            place(q, i, j);
            const int gi = (b + 1) * ST + i;
            pre[q] = (i < (s - b) * ST && gi < nrow) ? base[gi * v.rs + (b * ST + j) * v.cs] : T(0);
        }
    };
    if (s > 0) fetch(s - 1);
    if (warp <= s) {
        T(*D)[DP] = S.D[warp];
        const int d0 = warp * ST;
        // the loads in flight together: into registers before the first one is stored
        T xd[ST];
        const int ds = d0 + ST <= nrow ? ST : nrow - d0;  // the block's rows (<= 0: none)
#pragma unroll
        for (int e = 0; e < ST; ++e) {
            const int i = rowacc ? e : lane, j = rowacc ? lane : e;
            xd[e] = (i < ds && j < ds) ? base[(d0 + i) * v.rs + (d0 + j) * v.cs] : T(0);
        }
#pragma unroll
        for (int e = 0; e < ST; ++e) {
            const int i = rowacc ? e : lane, j = rowacc ? lane : e;
            D[i][j] = (i < ds && (j < i || (j == i && !v.unit))) ? conj_if(xd[e], v.conj) : i == j ? T(1) : T(0);
        }
        __syncwarp();
        const R wsum = row_sum(D[lane]);
        s_w[d0 + lane] = wsum;
        // column `lane` of the inverse, eight rows at a time (rolled: unrolled over
        // the 32 rows the code outgrows the instruction cache it runs through once):
        // the rows by substitution in registers, their products off the rows below.
        // The finished rows replace the block's, which no later step reads.
        const T rd = (v.unit || sizeof(T) == 16) ? T(1) : T(1) / D[lane][lane];
        T xr[ST / 8][8];
#pragma unroll
        for (int b = 0; b < ST / 8; ++b)
#pragma unroll
            for (int u = 0; u < 8; ++u) xr[b][u] = (8 * b + u == lane) ? T(1) : T(0);
#pragma unroll 1
        for (int b = 0; b < ST / 8; ++b) {
            T x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = xr[0][u];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const T *row = &D[8 * b + u][8 * b];
#pragma unroll
                for (int p = 0; p < u; ++p) x[u] = mad(-row[p], x[p], x[u]);
                if (!v.unit) {
                    if constexpr (sizeof(T) == 16) x[u] = x[u] / row[u];
                    else x[u] = quotient(x[u], row[u], __shfl_sync(0xffffffffu, rd, 8 * b + u));
                }
            }
#pragma unroll
            for (int q = 1; q < ST / 8; ++q) {
                if (b + q < ST / 8) {
#pragma unroll
                    for (int w = 0; w < 8; ++w) {
                        const T *row = &D[8 * (b + q) + w][8 * b];
#pragma unroll
                        for (int u = 0; u < 8; ++u) xr[q][w] = mad(-row[u], x[u], xr[q][w]);
                    }
                }
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 8; ++u) D[8 * b + u][lane] = x[u];
#pragma unroll
            for (int q = 0; q < ST / 8 - 1; ++q)
#pragma unroll
                for (int u = 0; u < 8; ++u) xr[q][u] = xr[q + 1][u];
        }
        __syncwarp();
        R k4[4] = {R(0), R(0), R(0), R(0)};
#pragma unroll
        for (int e = 0; e < ST; ++e) k4[e & 3] += mag(D[lane][(e + lane) & 31]) * s_w[d0 + ((e + lane) & 31)];
        R k = (k4[0] + k4[1]) + (k4[2] + k4[3]);
        // an inverse near or among the subnormal numbers has lost digits
        constexpr R tiny = sizeof(R) == 4 ? R(0x1p-102) : R(0x1p-969);
        if (!(mag(D[lane][lane]) >= tiny)) k = R(INFINITY);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) k = larger(k, shfl_xor(k, o));
        if (lane == 0) s_k[warp] = k;
    }
    __syncthreads();
    for (int e = t; e < ST * SP; e += INV_NT) {
        const int r = e / SP, c = e % SP;
        S.Y[r][c] = (c / ST == s) ? S.D[s][r][c % ST] : T(0);
    }
    for (int b = s - 1; b >= 0; --b) {
        const int K = (s - b) * ST;  // rows of the block column below its diagonal block
#pragma unroll
        for (int q = 0; q < PRE; ++q) {
            int i, j;
            place(q, i, j);
            if (i < K) S.L[i][j] = conj_if(pre[q], v.conj);
        }
        __syncthreads();
        if (b > 0) fetch(b - 1);
        if (t < K) s_w[(b + 1) * ST + t] += row_sum(S.L[t]);
        inv_product<T>(&S.Y[0][(b + 1) * ST], YP, &S.L[0][0], DP, K, &S.Z[0][0], DP, true);
        __syncthreads();
        inv_product<T>(&S.Z[0][0], DP, &S.D[b][0][0], DP, ST, &S.Y[0][b * ST], YP, false);
        __syncthreads();
    }
    __syncthreads();
    T *Pg = P + (i64)g * SP * ST;
#pragma unroll 4
    for (int e = t; e < SP * ST; e += INV_NT) {  // a warp: eight rows of four columns
        const int l = e & 31, q = e >> 5, r = (l & 7) + 8 * (q & 3), c = (l >> 3) + 4 * (q >> 2);
        Pg[c * ST + r] = S.Y[r][c];
    }
    // the strip's estimate, behind the inverses: eight lanes a row
    R e4[4] = {R(0), R(0), R(0), R(0)};
    for (int c = t & 7; c < (s + 1) * ST; c += 32)
#pragma unroll
        for (int u = 0; u < 4; ++u) e4[u] += mag(S.Y[t >> 3][c + 8 * u]) * s_w[c + 8 * u];
    R e = (e4[0] + e4[1]) + (e4[2] + e4[3]);
    e += shfl_xor(e, 1);
    e += shfl_xor(e, 2);
    e += shfl_xor(e, 4);
    e = larger(e, shfl_xor(e, 8));
    e = larger(e, shfl_xor(e, 16));
    if (lane == 0) s_e[warp] = e;
    __syncthreads();
    if (t == 0) {
        R k = s_k[0];
        for (int q = 1; q < INV_NT / 32; ++q) e = larger(e, s_e[q]);
        for (int q = 1; q <= s; ++q) k = larger(k, s_k[q]);
        const R est = e * k;
        P[(i64)((v.n + SP - 1) / SP) * SP * SP + g] = T(est == est ? est : R(INFINITY));
    }
}

// ---------------------------------------------------------------------------
// The solve.  ROWACC: the factor's unit stride runs along M's rows.
// ---------------------------------------------------------------------------
// An exchange word: the value's bits; all ones means "not there yet", and a
// value that has those bits (a NaN) is published as another NaN.
template <typename T>
struct ExchWord {  // double, and complex as two words
    using U = unsigned long long;
    static constexpr int W = (int)(sizeof(T) / sizeof(U));
    static __device__ __forceinline__ U load(const U *p) {
        U v;
        asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
        return v;
    }
    static __device__ __forceinline__ void load2(const U *p, U &a, U &b) {
        asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    }
    static __device__ __forceinline__ U bits1(double v) {
        const U u = (U)__double_as_longlong(v);
        return u == ~U(0) ? u ^ 1u : u;
    }
    static __device__ __forceinline__ T value(const U *u) {
        if constexpr (W == 2) return T(__longlong_as_double((long long)u[0]), __longlong_as_double((long long)u[1]));
        else return __longlong_as_double((long long)u[0]);
    }
    static __device__ __forceinline__ void publish(U *p, T v) {
        if constexpr (W == 2) {
            *(volatile U *)p = bits1(v.x);
            *(volatile U *)(p + 1) = bits1(v.y);
        } else {
            *(volatile U *)p = bits1(v);
        }
    }
};
template <> struct ExchWord<float> {
    using U = unsigned int;
    static constexpr int W = 1;
    static __device__ __forceinline__ U load(const U *p) {
        U v;
        asm volatile("ld.volatile.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        return v;
    }
    static __device__ __forceinline__ void load2(const U *p, U &a, U &b) {
        asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "l"(p) : "memory");
    }
    static __device__ __forceinline__ float value(const U *u) { return __uint_as_float(u[0]); }
    static __device__ __forceinline__ void publish(U *p, float v) {
        const U u = __float_as_uint(v);
        *(volatile U *)p = u == ~U(0) ? u ^ 1u : u;
    }
};

// Sum V values over the 32 lanes by halving: V - 1 exchanges for V <= 32, and
// lane l ends with the sums of value indexes lane_value(l) .. + max(V / 32, 1).
template <typename T, int V, int OFF>
__device__ __forceinline__ void lane_sums(T (&a)[V], int lane) {
    if constexpr (OFF > 0) {
        if constexpr (V > 1) {
            constexpr int HV = V / 2;
            const bool up = lane & OFF;
            T h[HV];
#pragma unroll
            for (int i = 0; i < HV; ++i) {
                const T send = up ? a[i] : a[i + HV], keep = up ? a[i + HV] : a[i];
                h[i] = keep + shfl_xor(send, OFF);
            }
            lane_sums<T, HV, OFF / 2>(h, lane);
#pragma unroll
            for (int i = 0; i < HV; ++i) a[i] = h[i];
        } else {
            a[0] += shfl_xor(a[0], OFF);
            lane_sums<T, 1, OFF / 2>(a, lane);
        }
    }
}
template <int V>
__device__ __forceinline__ int lane_value(int lane) {
    int idx = 0;
#pragma unroll
    for (int h = V / 2, off = 16; h >= 1 && off > 0; h /= 2, off /= 2) idx += (lane & off) ? h : 0;
    return idx;
}

// NR values of one row: 16-byte accesses where they fill one
template <typename T, int NR>
__device__ __forceinline__ void get_row(T (&v)[NR], const T *p) {
    constexpr int VEC = 16 / (int)sizeof(T);
    if constexpr (NR % VEC == 0 && VEC > 1) {
#pragma unroll
        for (int k = 0; k < NR; k += VEC) {
            const int4 x = *reinterpret_cast<const int4 *>(p + k);
            const T *xx = reinterpret_cast<const T *>(&x);
#pragma unroll
            for (int u = 0; u < VEC; ++u) v[k + u] = xx[u];
        }
    } else {
#pragma unroll
        for (int k = 0; k < NR; ++k) v[k] = p[k];
    }
}
template <typename T, int NR>
__device__ __forceinline__ void put_row(T *p, const T (&v)[NR]) {
    constexpr int VEC = 16 / (int)sizeof(T);
    if constexpr (NR % VEC == 0 && VEC > 1) {
#pragma unroll
        for (int k = 0; k < NR; k += VEC) {
            int4 x;
            T *xx = reinterpret_cast<T *>(&x);
#pragma unroll
            for (int u = 0; u < VEC; ++u) xx[u] = v[k + u];
            *reinterpret_cast<int4 *>(p + k) = x;
        }
    } else {
#pragma unroll
        for (int k = 0; k < NR; ++k) p[k] = v[k];
    }
}

template <typename T, int NR>
struct TriSolveSmem {
    static constexpr int SP = SP_<T>, NS = SP / ST;
    // pitch of a row's values: 16 bytes more keep eight lanes' 16-byte reads of
    // eight rows free of bank conflicts, 32 bytes a DMMA fragment's loads
    static constexpr int XP = NR * (int)sizeof(T) >= 32 ? NR + (sizeof(T) == 8 && NR == 8 ? 32 : 16) / (int)sizeof(T) : NR;
    // a column's pitch: 16-byte rows, and 4 modulo 16 for the DMMA fragments
    static constexpr int MP = ST + 4;
    T inv[SP][MP];       // this strip of the superblock's inverse, by columns
    T m[SP][MP];         // this strip of the superblock's triangle, by columns
    T xs[2][SP * XP];    // solved values being multiplied, double-buffered
    T part[NS][NR][MP];  // per-warp partial sums (the sums read rows of all right-hand sides)
    // read by the other strips: the strip's right-hand side, its product with the
    // inverse (or its solution), the residual of that
    T r[ST][NR], x[ST][NR], d[ST][NR];
    int bad[2];          // values of r, of x, that are not finite
};

template <typename T, bool ROWACC, int NR>
__global__ void __cluster_dims__(SP_<T> / ST, 1, 1) __launch_bounds__(SP_<T>, 1)
k_tri_solve(const TriView<T> v, const T *__restrict__ P, T *__restrict__ X, i64 ldx, int *__restrict__ ticket,
            typename ExchWord<T>::U *__restrict__ exch, int *__restrict__ err) {
    using EW = ExchWord<T>;
    using U = typename EW::U;
    constexpr int SP = SP_<T>, NS = SP / ST, TRI_NT = SP, TW = EW::W;
    constexpr int RPW = ST / NS, CPL = SP / 32;  // ROWACC: rows per warp, columns per lane
    // the next tile is loaded ahead where two fit the registers
    constexpr bool AHEAD = sizeof(T) <= 8;
    constexpr int XP = TriSolveSmem<T, NR>::XP, MP = TriSolveSmem<T, NR>::MP;
    extern __shared__ __align__(16) unsigned char tri_smem[];
    TriSolveSmem<T, NR> &S = *reinterpret_cast<TriSolveSmem<T, NR> *>(tri_smem);
    __shared__ int s_blk;
    cg::cluster_group cl = cg::this_cluster();
    const int s = (int)cl.block_rank();
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int n = v.n, nsb = (n + SP - 1) / SP;
    // the ticket counts from -1 (cleared with the exchange words); an aborted call takes no block
    if (s == 0 && t == 0) s_blk = aborted(err) ? nsb : atomicAdd(ticket, 1) + 1;
    if (t < 2) S.bad[t] = 0;
    cl.sync();
    const int B = *cl.map_shared_rank(&s_blk, 0);
    if (B >= nsb) {
        cl.sync();
        return;
    }
    const int g = B * NS + s;
    const i64 r0 = (i64)B * SP + s * ST;
    const int rows = (int)(n - r0 < 0 ? 0 : (n - r0 < ST ? n - r0 : ST));

    // ---- no dependency on other superblocks: the inverse's strip, the right-hand side ----
    if (warp <= s && rows > 0) {
        const T *Pg = P + (i64)g * SP * ST;
#pragma unroll
        for (int c = 0; c < ST; ++c) S.inv[warp * ST + c][lane] = Pg[(warp * ST + c) * ST + lane];
    }
    // how the superblock is solved (the same in all its strips): 0 the product, 1
    // with a correction, 2 substitution
    int mode;
    {
        double est = 0.0;
        if (lane < NS && (i64)B * SP + lane * ST < n) est = est_value(P[(i64)nsb * SP * SP + B * NS + lane]);
#pragma unroll
        for (int o = NS / 2; o > 0; o >>= 1) est = fmax(est, shfl_xor(est, o));
        est = shfl(est, 0);
        mode = est <= kTriPlain ? 0 : (est <= tri_limit<T> ? 1 : 2);
    }
    // the strip of the triangle: warp w its block of columns w
    auto load_triangle = [&]() {
        if (warp > s || rows <= 0) return;
        const T *p = v.a + r0 * v.rs + ((i64)B * SP + warp * ST) * v.cs;
        T a[ST];
#pragma unroll
        for (int e = 0; e < ST; ++e) {
            const int i = ROWACC ? e : lane, j = ROWACC ? lane : e;
            a[e] = (i < rows && (warp < s || j < i || (j == i && !v.unit))) ? conj_if(p[i * v.rs + j * v.cs], v.conj)
                                                                            : T(warp == s && i == j ? 1 : 0);
        }
#pragma unroll
        for (int e = 0; e < ST; ++e) S.m[warp * ST + (ROWACC ? lane : e)][ROWACC ? e : lane] = a[e];
    };
    if (mode > 0) load_triangle();
    constexpr int V = ROWACC ? RPW * NR : NR;             // accumulators per lane
    constexpr int OUT = (ST * NR + TRI_NT - 1) / TRI_NT;  // outputs per thread
    // outputs of the first product: (row, rhs) of thread t's q-th value
    auto r_out = [&](int q, int &row, int &k) -> bool {
        if constexpr (ROWACC) {
            const int idx = lane_value<V>(lane) + q;
            row = warp * RPW + idx / NR;
            k = idx % NR;
            return V >= 32 || (lane & (32 / (V < 32 ? V : 32) - 1)) == 0;
        } else {
            const int o = t + TRI_NT * q;
            row = o % ST;
            k = o / ST;
            return o < ST * NR;
        }
    };
    auto xrow = [&](i64 i) -> i64 { return v.rev ? n - 1 - i : i; };
    T bv[OUT];
#pragma unroll
    for (int q = 0; q < OUT; ++q) {
        int row, k;
        bv[q] = T(0);
        if (r_out(q, row, k) && row < rows) bv[q] = X[xrow(r0 + row) + (i64)k * ldx];
    }

    // ---- products with the superblocks before this one ----
    T acc[V];
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = T(0);
    auto load_tile = [&](int C, T (&a)[32]) {
        const i64 c0 = (i64)C * SP;
        if constexpr (ROWACC) {
#pragma unroll
            for (int i = 0; i < RPW; ++i) {
                const int row = warp * RPW + i;
                const T *p = v.a + (r0 + row) * v.rs + (c0 + lane) * v.cs;
#pragma unroll
                for (int u = 0; u < CPL; ++u) a[i * CPL + u] = row < rows ? conj_if(p[32 * u * v.cs], v.conj) : T(0);
            }
        } else {
            const T *p = v.a + (r0 + lane) * v.rs + (c0 + warp * ST) * v.cs;
#pragma unroll
            for (int c = 0; c < 32; ++c) a[c] = lane < rows ? conj_if(p[c * v.cs], v.conj) : T(0);
        }
    };
    U xw[NR * TW];
    const U *myx = exch + (i64)t * (NR * TW);
    auto load_x = [&](int C) {
        const U *p = myx + (i64)C * SP * (NR * TW);
        if constexpr (NR * TW == 1) {
            xw[0] = EW::load(p);
        } else {
#pragma unroll
            for (int k = 0; k < NR * TW; k += 2) EW::load2(p + k, xw[k], xw[k + 1]);
        }
    };
    auto x_ready = [&]() -> bool {
        bool ok = true;
#pragma unroll
        for (int k = 0; k < NR * TW; ++k) ok = ok && xw[k] != ~U(0);
        return ok;
    };
    auto step = [&](int C, T (&a)[32], T (&next)[32]) {
        if (!AHEAD) {
            load_tile(C, a);
            load_x(C);
        }
        if (!x_ready()) {
            const uint64_t t0 = global_ns();
            uint32_t it = 0;
            for (;;) {
                load_x(C);
                if (x_ready()) break;
                if (spin_give_up<256>(it, t0, err, 3)) break;
            }
        }
        T *xs = S.xs[C & 1];
        {
            T x[NR];
#pragma unroll
            for (int k = 0; k < NR; ++k) x[k] = EW::value(xw + k * TW);
            put_row<T, NR>(xs + t * XP, x);
        }
        if (AHEAD && C + 1 < B) {
            load_tile(C + 1, next);
            load_x(C + 1);
        }
        if constexpr (ROWACC) {
            __syncthreads();
#pragma unroll
            for (int u = 0; u < CPL; ++u) {
                T x[NR];
                get_row<T, NR>(x, xs + (lane + 32 * u) * XP);
#pragma unroll
                for (int k = 0; k < NR; ++k)
#pragma unroll
                    for (int i = 0; i < RPW; ++i) acc[i * NR + k] = mad(a[i * CPL + u], x[k], acc[i * NR + k]);
            }
        } else {
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 32; ++c) {
                T x[NR];
                get_row<T, NR>(x, xs + (warp * ST + c) * XP);
#pragma unroll
                for (int k = 0; k < NR; ++k) acc[k] = mad(a[c], x[k], acc[k]);
            }
            __syncwarp();
        }
    };
    if (B > 0 && rows > 0) {
        T a0[32];
        if constexpr (AHEAD) {
            T a1[32];
            load_tile(0, a0);
            load_x(0);
            for (int C = 0; C < B; C += 2) {
                step(C, a0, a1);
                if (C + 1 < B) step(C + 1, a1, a0);
            }
        } else {
            for (int C = 0; C < B; ++C) step(C, a0, a0);
        }
    }
    // ---- the strip's right-hand side, to the whole superblock ----
    if constexpr (ROWACC) {
        lane_sums<T, V, 16>(acc, lane);
    } else {
#pragma unroll
        for (int k = 0; k < NR; ++k) S.part[warp][k][lane] = acc[k];
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < OUT; ++q) {
        int row, k;
        if (r_out(q, row, k)) {
            T sum;
            if constexpr (ROWACC) {
                sum = acc[q < V ? q : 0];
            } else {
                sum = T(0);
#pragma unroll
                for (int w = 0; w < NS; ++w) sum += S.part[w][k][row];
            }
            const T v0 = bv[q] - sum;
            S.r[row][k] = v0;
            if (!is_finite(v0)) S.bad[0] = 1;
        }
    }
    cl.sync();

    // ---- the superblock's own triangle ----
    auto any_bad = [&](int i) -> bool {
        const int b = lane < NS ? *cl.map_shared_rank(&S.bad[i], lane) : 0;
        return __any_sync(0xffffffffu, b != 0);
    };
    auto publish = [&](int row, int k, T x) {
        if (row < rows) {
            EW::publish(exch + ((r0 + row) * NR + k) * TW, x);
            X[xrow(r0 + row) + (i64)k * ldx] = x;
        }
    };
    // the strips' values of src, strip w to warp w: 16 contiguous bytes a lane at a time
    // (of a row each, 64-byte strides, 16 KB take 1700 cycles)
    constexpr int XB = NR * (int)sizeof(T), CPR = XB >= 16 ? XB / 16 : NR;  // a row's bytes, its chunks
    using Chunk = typename std::conditional<(XB >= 16), int4, T>::type;
    struct Chunks {
        Chunk c[CPR];
    } xv;
    auto fetch = [&](T *src) {
        if (warp <= s && rows > 0) {
            const Chunk *p = reinterpret_cast<const Chunk *>(cl.map_shared_rank(src, warp));
#pragma unroll
            for (int i = 0; i < CPR; ++i) xv.c[i] = p[i * 32 + lane];
        }
    };
    auto keep = [&]() {  // into the warp's rows of xs
#pragma unroll
        for (int i = 0; i < CPR; ++i) {
            const int c = i * 32 + lane;
            *reinterpret_cast<Chunk *>(S.xs[0] + (warp * ST + c / CPR) * XP + c % CPR * (NR / CPR)) = xv.c[i];
        }
    };
    // The strip's rows of Mat times those values, warp w strip w's 32 columns, then
    // sink(row, rhs, sum).  With a lane per row, 16-byte loads of a row's values (the
    // same for all lanes, and yet four passes of the shared memory each) bound the
    // product: 5200 cycles with 8 FP64 values, 6000 with 16 FP32 ones.  So FP64 runs
    // on the tensor cores from 4 right-hand sides on, and FP32 by tiles of 4 rows from
    // 8 on.
    auto multiply = [&](const T *Mat, auto &&sink) {
        const bool mine = warp <= s && rows > 0;
        __syncwarp();
        if (mine) keep();
        __syncwarp();
        const T *A = Mat + warp * ST * MP, *xs = S.xs[0] + warp * ST * XP;
        if constexpr (sizeof(T) == 8 && NR >= 4) {
            const int gid = lane >> 2, tig = lane & 3;
            double c[2][4] = {};
            if (mine)
#pragma unroll
                for (int kk = 0; kk < ST; kk += 4) {
                    const double xb = gid < NR ? xs[(kk + tig) * XP + (gid < NR ? gid : 0)] : 0.0;
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        asm volatile(
                            "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                            : "+d"(c[h][0]), "+d"(c[h][1]), "+d"(c[h][2]), "+d"(c[h][3])
                            : "d"(A[(kk + tig) * MP + 16 * h + gid]), "d"(A[(kk + tig) * MP + 16 * h + gid + 8]), "d"(xb));
                }
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (2 * tig + (e & 1) < NR) S.part[warp][2 * tig + (e & 1)][16 * h + gid + 8 * (e >> 1)] = c[h][e];
        } else if constexpr (sizeof(T) == 4 && NR >= 8) {
            constexpr int KW = NR / 4;
            const int r4 = (lane & 7) * 4, k0 = (lane >> 3) * KW;
            T o[KW][4];
#pragma unroll
            for (int k = 0; k < KW; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i) o[k][i] = T(0);
            if (mine)
#pragma unroll 8
                for (int c = 0; c < ST; ++c) {
                    T m[4], x[KW];
                    get_row<T, 4>(m, A + c * MP + r4);
                    if constexpr (KW == 4) get_row<T, 4>(x, xs + c * XP + k0);
                    else *(float2 *)x = *(const float2 *)(xs + c * XP + k0);
#pragma unroll
                    for (int k = 0; k < KW; ++k)
#pragma unroll
                        for (int i = 0; i < 4; ++i) o[k][i] = mad(m[i], x[k], o[k][i]);
                }
#pragma unroll
            for (int k = 0; k < KW; ++k) put_row<T, 4>(&S.part[warp][k0 + k][r4], o[k]);
        } else {
            T o[NR];
#pragma unroll
            for (int k = 0; k < NR; ++k) o[k] = T(0);
            if (mine)
#pragma unroll
                for (int c = 0; c < ST; ++c) {
                    const T mv = A[c * MP + lane];
                    T x[NR];
                    get_row<T, NR>(x, xs + c * XP);
#pragma unroll
                    for (int k = 0; k < NR; ++k) o[k] = mad(mv, x[k], o[k]);
                }
#pragma unroll
            for (int k = 0; k < NR; ++k) S.part[warp][k][lane] = o[k];
        }
        __syncthreads();
        for (int e = t; e < ST * NR; e += TRI_NT) {
            const int row = e / NR, k = e % NR;
            T x = T(0);
#pragma unroll
            for (int w = 0; w < NS; ++w) x += S.part[w][k][row];
            sink(row, k, x);
        }
    };
    const int planned = mode;
    fetch(&S.r[0][0]);
    if (any_bad(0)) mode = 2;
    if (mode == 0) {
        multiply(&S.inv[0][0], publish);
    } else if (mode == 1) {
        multiply(&S.inv[0][0], [&](int row, int k, T x) {
            S.x[row][k] = x;
            if (!is_finite(x)) S.bad[1] = 1;
        });
        cl.sync();
        fetch(&S.x[0][0]);
        if (any_bad(1)) {
            mode = 2;
        } else {
            multiply(&S.m[0][0], [&](int row, int k, T x) { S.d[row][k] = S.r[row][k] - x; });
            cl.sync();
            fetch(&S.d[0][0]);
            multiply(&S.inv[0][0], [&](int row, int k, T x) { publish(row, k, S.x[row][k] + x); });
        }
    }
    if (mode == 2) {
        // the strips in turn, a right-hand side per warp
        if (planned == 0) load_triangle();
        __syncthreads();
        for (int q = 0; q < NS; ++q) {
            if (s == q) {
                for (int k = warp; k < NR; k += NS) {
                    T y = S.r[lane][k];
                    for (int p = 0; p < rows; ++p) {
                        T xp = shfl(y, p);
                        if (!v.unit) xp = xp / S.m[s * ST + p][p];
                        if (lane > p) y = mad(-S.m[s * ST + p][lane], xp, y);
                        else if (lane == p) y = xp;
                    }
                    S.x[lane][k] = y;
                    publish(lane, k, y);
                }
            }
            cl.sync();
            if (s > q && rows > 0) {
                T *xq = S.xs[0];
                const T *src = cl.map_shared_rank(&S.x[0][0], q);
                for (int e = t; e < ST * NR; e += TRI_NT) xq[e] = src[e];
                __syncthreads();
                for (int e = t; e < ST * NR; e += TRI_NT) {
                    const int row = e % ST, k = e / ST;
                    T y = S.r[row][k];
#pragma unroll 8
                    for (int p = 0; p < ST; ++p) y = mad(-S.m[q * ST + p][row], xq[p * NR + k], y);
                    S.r[row][k] = y;
                }
                __syncthreads();
            }
        }
    }
    cl.sync();  // the other strips have read this one's values
}

template <typename T>
i64 tri_inverse_elems(i64 n) {
    return (n + SP_<T> - 1) / SP_<T> * (SP_<T> * (i64)SP_<T> + SP_<T> / ST);  // the inverses, an estimate a strip
}
template i64 tri_inverse_elems<float>(i64);
template i64 tri_inverse_elems<double>(i64);
template i64 tri_inverse_elems<zc64>(i64);

// Exchange words and tickets of one launch pair: a ticket per triangle, then
// their words.
template <typename T>
static i64 exch_words(i64 n, int nr) {
    return (n + SP_<T> - 1) / SP_<T> * SP_<T> * (i64)nr * ExchWord<T>::W;
}

template <typename T>
static void tri_inv_launch(const TriView<T> &v0, const TriView<T> &v1, T *P0, T *P1, cudaStream_t s) {
    const int smem = (int)sizeof(TriInvSmem<T>);
    set_max_dyn_smem((const void *)k_tri_inv<T>, smem);
    const unsigned strips = (unsigned)((v0.n + ST - 1) / ST);
    constexpr double SP = SP_<T>;
    ProfScope ps(KC_TRSV, s, 2.0 * 2.0 * v0.n * SP * SP / 3.0, 2.0 * (double)v0.n * SP * 1.5 * sizeof(T));
    k_tri_inv<T><<<dim3(strips, 2), INV_NT, smem, s>>>(v0, v1, P0, P1);
    OXI_LAUNCH_CHECK();
}

// First triangle, then the second, on X (n x nrhs, in place), by chunks of right-hand
// sides.  Measured on one B200, us, in 64-row blocks -> superblocks by the product
// alone -> by the rule at the head of the file (all of these corrected): inverses and
// pair of FP64 solves, n = 256, one right-hand side 330 -> 66 -> 80; n = 4096, transposed,
// 8 right-hand sides 2090 -> 250 -> 321 (243 the solves); FP32 pairs of the refinement at
// n = 8192 with 16 right-hand sides 15400 -> 2130 -> 3090 in all; complex n = 2048 about
// 8000 (substitution, a column at a time) -> 224 -> 290.  By substitution, n = 2048, one
// right-hand side: 406, complex 1290 (130 and 290 by corrected products).
template <typename T, bool ROWACC0, bool ROWACC1>
static void trsv_pair(oxi_handle_s *h, const TriView<T> &v0, const TriView<T> &v1, const T *P0, const T *P1, T *X,
                      i64 ldx, i64 nrhs, int *err) {
    using U = typename ExchWord<T>::U;
    cudaStream_t s = h->stream;
    const i64 n = v0.n;
    constexpr int SP = SP_<T>, TRI_NT = SP;
    const unsigned grid = (unsigned)((n + SP - 1) / SP * (SP / ST));
    constexpr int NRX = sizeof(T) == 4 ? 16 : (sizeof(T) == 8 ? 8 : 4);
    for (i64 k0 = 0; k0 < nrhs;) {
        const i64 left = nrhs - k0;
        const int nr = left >= 16 && NRX == 16 ? 16 : left >= 8 && NRX >= 8 ? 8 : left >= 4 ? 4 : left >= 2 ? 2 : 1;
        const size_t words = (size_t)exch_words<T>(n, nr);
        const size_t bytes = 256 + 2 * words * sizeof(U);
        char *ws = (char *)h->xtag_ws.get(256 + 2 * (size_t)exch_words<T>(n, NRX) * sizeof(U));
        int *tickets = (int *)ws;
        U *e0 = (U *)(ws + 256), *e1 = e0 + words;
        ProfScope ps(KC_TRSV, s, 2.0 * (double)n * n * nr, (double)n * n * sizeof(T));
        OXI_CUDA(cudaMemsetAsync(ws, 0xff, bytes, s));
        T *Xk = X + k0 * ldx;
#define OXI_TRI_GO(NRV)                                                                                   \
    do {                                                                                                  \
        const int smem = (int)sizeof(TriSolveSmem<T, NRV>);                                               \
        set_max_dyn_smem((const void *)k_tri_solve<T, ROWACC0, NRV>, smem);                               \
        set_max_dyn_smem((const void *)k_tri_solve<T, ROWACC1, NRV>, smem);                               \
        k_tri_solve<T, ROWACC0, NRV><<<grid, TRI_NT, smem, s>>>(v0, P0, Xk, ldx, tickets, e0, err);       \
        OXI_LAUNCH_CHECK();                                                                               \
        k_tri_solve<T, ROWACC1, NRV><<<grid, TRI_NT, smem, s>>>(v1, P1, Xk, ldx, tickets + 1, e1, err);   \
        OXI_LAUNCH_CHECK();                                                                               \
    } while (0)
        if constexpr (NRX == 16) {
            if (nr == 16) OXI_TRI_GO(16);
        }
        if constexpr (NRX >= 8) {
            if (nr == 8) OXI_TRI_GO(8);
        }
        if (nr == 4) OXI_TRI_GO(4);
        else if (nr == 2) OXI_TRI_GO(2);
        else if (nr == 1) OXI_TRI_GO(1);
#undef OXI_TRI_GO
        k0 += nr;
    }
}

// The four forms: LU solves with a column-major factor (N: L, U; T: U^T, L^T),
// with a row-major one, and the two solves of a column-major lower Cholesky factor.
template <typename T>
static void tri_views(TriForm form, const T *A, i64 lda, i64 n, TriView<T> &v0, TriView<T> &v1) {
    switch (form) {
    case TriForm::LU_N:
        v0 = tri_view(A, lda, n, true, true, false);
        v1 = tri_view(A, lda, n, false, false, false);
        break;
    case TriForm::LU_T:
    case TriForm::LU_C:
        v0 = tri_view(A, lda, n, true, false, true, form == TriForm::LU_C);
        v1 = tri_view(A, lda, n, false, true, true, form == TriForm::LU_C);
        break;
    case TriForm::LU_ROWMAJOR:
        v0 = tri_view(A, lda, n, true, true, true);
        v1 = tri_view(A, lda, n, false, false, true);
        break;
    case TriForm::CHOLESKY:
        v0 = tri_view(A, lda, n, true, false, false);
        v1 = tri_view(A, lda, n, false, false, true);
        break;
    }
}

template <typename T>
void tri_inverses(oxi_handle_s *h, TriForm form, const T *A, i64 lda, i64 n, T *P0, T *P1) {
    TriView<T> v0, v1;
    tri_views(form, A, lda, n, v0, v1);
    tri_inv_launch<T>(v0, v1, P0, P1, h->stream);
}
template <typename T>
void tri_solves(oxi_handle_s *h, TriForm form, const T *A, i64 lda, i64 n, T *X, i64 ldx, i64 nrhs, int *err,
                const T *P0, const T *P1) {
    TriView<T> v0, v1;
    tri_views(form, A, lda, n, v0, v1);
    if (form == TriForm::LU_N) trsv_pair<T, false, false>(h, v0, v1, P0, P1, X, ldx, nrhs, err);
    else if (form == TriForm::CHOLESKY) trsv_pair<T, false, true>(h, v0, v1, P0, P1, X, ldx, nrhs, err);
    else trsv_pair<T, true, true>(h, v0, v1, P0, P1, X, ldx, nrhs, err);
}
template void tri_inverses<zc64>(oxi_handle_s *, TriForm, const zc64 *, i64, i64, zc64 *, zc64 *);
template void tri_solves<zc64>(oxi_handle_s *, TriForm, const zc64 *, i64, i64, zc64 *, i64, i64, int *, const zc64 *,
                               const zc64 *);
template void tri_inverses<float>(oxi_handle_s *, TriForm, const float *, i64, i64, float *, float *);
template void tri_inverses<double>(oxi_handle_s *, TriForm, const double *, i64, i64, double *, double *);
template void tri_solves<float>(oxi_handle_s *, TriForm, const float *, i64, i64, float *, i64, i64, int *,
                                const float *, const float *);
template void tri_solves<double>(oxi_handle_s *, TriForm, const double *, i64, i64, double *, i64, i64, int *,
                                 const double *, const double *);

}  // namespace oxi
