// FP64 trailing-update GEMM on the tensor cores: C <- C - A*B, row-major.
//
// sm_100a has no FP64 kind for tcgen05.mma; the FP64 tensor path is DMMA
// (mma.sync.aligned.m16n8k4 .f64), which this kernel feeds from TMA.
// CTA tile 128 x 64 (64 x 32 where those are few), k slab 16, 4-stage mbarrier pipeline, 8 warps in a 4 x 2 grid,
// 32 x 32 per warp (2 x 4 MMAs per k4; 16 x 16 and 1 x 2).  Thread 0 issues the TMA loads: a slot is
// refilled one slab after its own, when every warp has left it.  (A producer warp
// of its own costs the others registers: nine warps a CTA, two CTAs an SM,
// leave 96 a thread, eight leave 128, which the epilogue's loads in flight need.)
// The C tile is prefetched into L2 while the slabs run, and read in two batches.
// A stage holds A[128 x 16] with the 128-byte swizzle (conflict-free fragment
// loads) and B[16 x 64] as eight 16 x 8 boxes laid side by side (each k row of a
// box is 64 contiguous bytes, so a fragment load reads 256 contiguous bytes).
// The product s = A*B is accumulated from zero and subtracted at the end, the
// form of the reference's gemm!(C, A, B, -1, 1) (src/blas/gemm.jl:286-298).
#include "tma_util.cuh"

namespace oxi {

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        OXI_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
        if (!p || q != cudaDriverEntryPointSuccess)
            throw CudaError{cudaErrorNotSupported, "cuTensorMapEncodeTiled unavailable"};
        fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

void make_tmap_2d(CUtensorMap *tm, CUtensorMapDataType dt, int esize, const void *base, i64 cols,
                  i64 rows, i64 ld, int box_cols, int box_rows, CUtensorMapSwizzle swz) {
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)(ld * esize)};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = tensor_map_encoder()(tm, dt, 2, const_cast<void *>(base), dims, strides, box, estr,
                                      CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw CudaError{cudaErrorInvalidValue, "cuTensorMapEncodeTiled"};
}

namespace {
constexpr int BK = 16, STAGES = 4;
constexpr int NCONSUMER_WARPS = 8;
constexpr int NTHREADS = NCONSUMER_WARPS * 32;
constexpr i64 DMMA_SMALL_MAX = 104;  // large tiles up to which small ones are taken
constexpr int smem_bytes(int bm, int bn) { return STAGES * (bm + bn) * BK * 8 + 1024 /*align*/ + 256 /*barriers*/; }
}  // namespace

// A warp leaves a slab; thread 0 refills the slot when every warp has.  The slab
// was read through the generic proxy and the refill writes through the
// asynchronous one: an arrival releases the reads to other generic accesses only,
// so each lane orders its own reads before later asynchronous writes with the
// proxy fence, and lane 0 arrives for the warp.  Without the fence a refill could
// overtake a load that was issued but not done: with 64 x 32 tiles one n = 2048
// factorization in 350 (one in 64 with an arrival by every lane, which releases no
// more and adds traffic to the barrier) took a few operands of the slab four
// further on.
__device__ __forceinline__ void leave_slab(uint64_t *bar, int lane) {
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

template <int BM, int BN>
__global__ void __launch_bounds__(NTHREADS, 2)
k_gemm_dmma(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
            double *__restrict__ C, i64 ldc, int M, int N, int K, int *__restrict__ ab, int upper_only) {
    constexpr int A_STAGE_BYTES = BM * BK * 8, STAGE_BYTES = (BM + BN) * BK * 8;
    constexpr int WM = BM / 4, WN = BN / 2, MT = WM / 16, NT = WN / 8;  // a warp's rows, columns, MMA tiles
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~uintptr_t(1023));
    uint64_t *full = (uint64_t *)(smem + STAGES * STAGE_BYTES);
    uint64_t *empty = full + STAGES;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    // upper_only (a symmetric rank-k update of the upper triangle): tiles that
    // lie wholly below the diagonal are not computed
    if (upper_only && m0 > n0 + BN - 1) return;
    const int KT = (K + BK - 1) / BK;

    __shared__ int s_skip;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], NCONSUMER_WARPS);
        }
        s_skip = aborted(ab) ? 1 : 0;  // one reading for the whole CTA
        fence_barrier_init();
    }
    __syncthreads();
    if (s_skip) return;  // the call was aborted by an earlier wait

    auto issue = [&](int kt) {  // thread 0: slab kt into its slot
        const int s = kt % STAGES;
        uint8_t *sa = smem + s * STAGE_BYTES;
        uint8_t *sb = sa + A_STAGE_BYTES;
        mbar_arrive_expect_tx(&full[s], STAGE_BYTES);
        tma_load_2d(sa, &tmA, &full[s], kt * BK, m0);
#pragma unroll
        for (int g = 0; g < BN / 8; ++g)
            tma_load_2d(sb + g * (BK * 8 * 8), &tmB, &full[s], n0 + 8 * g, kt * BK);
    };
    if (threadIdx.x == 0) {
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
        for (int kt = 0; kt < KT && kt < STAGES; ++kt) issue(kt);
    }
    {
        // the C tile towards L2, 128-byte lines
#pragma unroll
        for (int e = threadIdx.x; e < BM * BN / 16; e += NTHREADS) {
            const int r = m0 + e / (BN / 16), c = n0 + e % (BN / 16) * 16;
            if (r < M && c < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + (i64)r * ldc + c));
        }
    }

    const int wm = warp & 3, wn = warp >> 2;  // 4 x 2 warps
    const int gid = lane >> 2, tig = lane & 3;
    double acc[MT][NT][4];
#pragma unroll
    for (int a = 0; a < MT; ++a)
#pragma unroll
        for (int b = 0; b < NT; ++b)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.0;

    for (int kt = 0; kt < KT; ++kt) {
        const int s = kt % STAGES;
        if (!mbar_wait<false>(&full[s], (kt / STAGES) & 1, ab, 2)) return;
        const uint8_t *sa = smem + s * STAGE_BYTES;
        const uint8_t *sb = sa + A_STAGE_BYTES;
#pragma unroll
        for (int k4 = 0; k4 < BK / 4; ++k4) {
            double af[MT][2], bf[NT];
            const int kc = k4 * 4 + tig;  // k column within the slab
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = wm * WM + mt * 16 + gid + 8 * h;
                    // 128B swizzle: 16-byte chunk index XOR (row mod 8)
                    const int off = r * 128 + ((((kc * 8) >> 4) ^ (r & 7)) << 4) + ((kc * 8) & 15);
                    af[mt][h] = *(const double *)(sa + off);
                }
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int g = (wn * WN + nt * 8) >> 3;
                bf[nt] = *(const double *)(sb + g * (BK * 64) + kc * 64 + gid * 8);
            }
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
                    asm volatile(
                        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, "
                        "{%6}, {%0,%1,%2,%3};"
                        : "+d"(acc[mt][nt][0]), "+d"(acc[mt][nt][1]), "+d"(acc[mt][nt][2]),
                          "+d"(acc[mt][nt][3])
                        : "d"(af[mt][0]), "d"(af[mt][1]), "d"(bf[nt]));
        }
        leave_slab(&empty[s], lane);
        if (threadIdx.x == 0 && kt >= 1 && kt - 1 + STAGES < KT) {  // refill the slab before's slot
            const int pt = kt - 1;
            // (on a wait that gave up nothing is issued: every warp's next wait gives up too)
            if (mbar_wait<false>(&empty[pt % STAGES], (pt / STAGES) & 1, ab, 2)) issue(pt + STAGES);
        }
        __syncwarp();
    }

    // epilogue: C -= acc.  The C pairs of two rows are loaded before any is
    // used so their round trips overlap (16-byte accesses when aligned).  A
    // symmetric update's tile that crosses the diagonal writes only the
    // elements on and above it (the other triangle stays as it was).
    const bool vec2 = ((ldc & 1) == 0) && ((((uintptr_t)C) & 15) == 0) && !(upper_only && m0 + BM - 1 > n0);
    const int cmin_row = upper_only ? 1 : 0;  // 1: column c is written only when c >= r
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        double2 cv[2][NT];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = m0 + wm * WM + mt * 16 + gid + 8 * h;
            const double *crow = C + (i64)r * ldc;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int c = n0 + wn * WN + nt * 8 + 2 * tig;
                if (r < M && c + 1 < N && vec2) cv[h][nt] = __ldcs((const double2 *)(crow + c));
                else {
                    cv[h][nt].x = (r < M && c < N && (!cmin_row || c >= r)) ? crow[c] : 0.0;
                    cv[h][nt].y = (r < M && c + 1 < N && (!cmin_row || c + 1 >= r)) ? crow[c + 1] : 0.0;
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = m0 + wm * WM + mt * 16 + gid + 8 * h;
            if (r >= M) continue;
            double *crow = C + (i64)r * ldc;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int c = n0 + wn * WN + nt * 8 + 2 * tig;
                double2 v;
                v.x = cv[h][nt].x - acc[mt][nt][2 * h];
                v.y = cv[h][nt].y - acc[mt][nt][2 * h + 1];
                if (c + 1 < N && vec2) __stcs((double2 *)(crow + c), v);
                else {
                    if (c < N && (!cmin_row || c >= r)) crow[c] = v.x;
                    if (c + 1 < N && (!cmin_row || c + 1 >= r)) crow[c + 1] = v.y;
                }
            }
        }
    }
}

template <int BM, int BN>
static void launch_dmma_tile(double *C, i64 ldc, const double *A, i64 lda, const double *B, i64 ldb, i64 M, i64 N,
                             i64 K, cudaStream_t s, bool upper_only) {
    CUtensorMap tmA, tmB;
    make_tmap_2d(&tmA, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, A, K, M, lda, BK, BM,
                 CU_TENSOR_MAP_SWIZZLE_128B);
    make_tmap_2d(&tmB, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, B, N, K, ldb, 8, BK,
                 CU_TENSOR_MAP_SWIZZLE_NONE);
    set_max_dyn_smem((const void *)k_gemm_dmma<BM, BN>, smem_bytes(BM, BN));
    dim3 grid((unsigned)((N + BN - 1) / BN), (unsigned)((M + BM - 1) / BM));
    k_gemm_dmma<BM, BN><<<grid, NTHREADS, smem_bytes(BM, BN), s>>>(tmA, tmB, C, ldc, (int)M, (int)N, (int)K, cur_abort(),
                                                                   upper_only ? 1 : 0);
    OXI_LAUNCH_CHECK();
}

void launch_gemm_dmma(double *C, i64 ldc, const double *A, i64 lda, const double *B, i64 ldb, i64 M,
                      i64 N, i64 K, cudaStream_t s, bool upper_only) {
    if (M <= 0 || N <= 0 || K <= 0) return;
    const bool aligned = ((uintptr_t)A % 16 == 0) && ((uintptr_t)B % 16 == 0) && (lda % 2 == 0) &&
                         (ldb % 2 == 0) && M < (1 << 30) && N < (1 << 30) && K < (1 << 30);
    if (!aligned) {  // TMA needs 16-byte aligned bases and pitches (the whole block: same results)
        if (upper_only)  // the plain kernel would write both triangles; callers align first
            throw CudaError{cudaErrorInvalidValue, "symmetric update needs 16-byte aligned operands"};
        launch_gemm_ref<double>(C, ldc, A, lda, B, ldb, M, N, K, s);
        return;
    }
    ProfScope ps(KC_GEMM_DMMA, s, (upper_only ? 1.0 : 2.0) * M * N * K, 8.0 * (2.0 * M * N + M * K + K * N));
    // Small tiles while the large ones leave SMs without one: a tile's time is its
    // chain of products on one SM, whatever the other SMs do.  Large against small,
    // us, by number of large tiles: 8 (960 x 64 x 64) 13.0, 10.1; 48 (3000 x 128 x
    // 128) 18.7, 14.5; 96 (6144 x 128 x 128) 19.1, 18.5; 98 (896 x 896 x 128) 18.9,
    // 18.7; 126 (8064 x 128 x 128) 19.7, 21.5; 148: 20.1, 23.1.
    const i64 large = ((M + 127) / 128) * ((N + 63) / 64);
    if (large <= DMMA_SMALL_MAX) launch_dmma_tile<64, 32>(C, ldc, A, lda, B, ldb, M, N, K, s, upper_only);
    else launch_dmma_tile<128, 64>(C, ldc, A, lda, B, ldb, M, N, K, s, upper_only);
}

// ---------------------------------------------------------------------------
// The complex update C -= A B on real and imaginary planes (row-major, one ld),
// one launch: 64 x 64 tile, k slab 16, 3 stages of the four operand planes, the
// two accumulators of a C element in registers, four DMMAs per fragment pair
// (Cr: Ar Br, then (-Ai) Bi; Ci: Ar Bi, then Ai Br; the negation is a sign bit
// of the fragment).  Against four launches of k_gemm_dmma and a negated copy
// of Ai it loads each fragment once for two products and moves C once.
// ---------------------------------------------------------------------------
namespace {
constexpr int ZM = 64, ZN = 64, ZST = 3;
constexpr int ZPLANE = ZM * BK * 8;            // 8 KB: a plane of A or of B
constexpr int ZSTAGE = 4 * ZPLANE;
constexpr int ZSMEM = ZST * ZSTAGE + 1024 + 256;
}  // namespace

__device__ __forceinline__ void dmma_16x8x4(double (&c)[4], double a0, double a1, double b) {
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                 : "d"(a0), "d"(a1), "d"(b));
}

__global__ void __launch_bounds__(NTHREADS, 2)
k_zgemm_dmma(const __grid_constant__ CUtensorMap tmAr, const __grid_constant__ CUtensorMap tmAi,
             const __grid_constant__ CUtensorMap tmBr, const __grid_constant__ CUtensorMap tmBi,
             double *__restrict__ Cr, double *__restrict__ Ci, i64 ldc, int M, int N, int K, int *__restrict__ ab) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~uintptr_t(1023));
    uint64_t *full = (uint64_t *)(smem + ZST * ZSTAGE);
    uint64_t *empty = full + ZST;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * ZM, n0 = blockIdx.x * ZN;
    const int KT = (K + BK - 1) / BK;
    __shared__ int s_skip;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ZST; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], NCONSUMER_WARPS);
        }
        s_skip = aborted(ab) ? 1 : 0;  // one reading for the whole CTA
        fence_barrier_init();
    }
    __syncthreads();
    if (s_skip) return;

    auto issue = [&](int kt) {
        const int s = kt % ZST;
        uint8_t *sa = smem + s * ZSTAGE;
        mbar_arrive_expect_tx(&full[s], ZSTAGE);
        tma_load_2d(sa, &tmAr, &full[s], kt * BK, m0);
        tma_load_2d(sa + ZPLANE, &tmAi, &full[s], kt * BK, m0);
#pragma unroll
        for (int g = 0; g < ZN / 8; ++g) {
            tma_load_2d(sa + 2 * ZPLANE + g * (BK * 64), &tmBr, &full[s], n0 + 8 * g, kt * BK);
            tma_load_2d(sa + 3 * ZPLANE + g * (BK * 64), &tmBi, &full[s], n0 + 8 * g, kt * BK);
        }
    };
    if (threadIdx.x == 0)
        for (int kt = 0; kt < KT && kt < ZST; ++kt) issue(kt);

    const int wm = warp & 3, wn = warp >> 2;  // 4 x 2 warps: 16 rows x 32 columns each
    const int gid = lane >> 2, tig = lane & 3;
    double cr[4][4], ci[4][4];
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int c = 0; c < 4; ++c) cr[b][c] = ci[b][c] = 0.0;
    for (int kt = 0; kt < KT; ++kt) {
        const int s = kt % ZST;
        if (!mbar_wait<false>(&full[s], (kt / ZST) & 1, ab, 2)) return;
        const uint8_t *sa = smem + s * ZSTAGE;
#pragma unroll
        for (int k4 = 0; k4 < BK / 4; ++k4) {
            const int kc = k4 * 4 + tig;
            double ar[2], ai[2];
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int r = wm * 16 + gid + 8 * hh;
                const int off = r * 128 + ((((kc * 8) >> 4) ^ (r & 7)) << 4) + ((kc * 8) & 15);
                ar[hh] = *(const double *)(sa + off);
                ai[hh] = *(const double *)(sa + ZPLANE + off);
            }
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const int off = (wn * 4 + nt) * (BK * 64) + kc * 64 + gid * 8;
                const double br = *(const double *)(sa + 2 * ZPLANE + off);
                const double bi = *(const double *)(sa + 3 * ZPLANE + off);
                dmma_16x8x4(cr[nt], ar[0], ar[1], br);
                dmma_16x8x4(ci[nt], ar[0], ar[1], bi);
                dmma_16x8x4(cr[nt], -ai[0], -ai[1], bi);
                dmma_16x8x4(ci[nt], ai[0], ai[1], br);
            }
        }
        leave_slab(&empty[s], lane);
        if (threadIdx.x == 0 && kt >= 1 && kt - 1 + ZST < KT) {
            const int pt = kt - 1;
            // (on a wait that gave up nothing is issued: every warp's next wait gives up too)
            if (mbar_wait<false>(&empty[pt % ZST], (pt / ZST) & 1, ab, 2)) issue(pt + ZST);
        }
        __syncwarp();
    }

    const bool vec2 = ((ldc & 1) == 0) && ((((uintptr_t)Cr) & 15) == 0) && ((((uintptr_t)Ci) & 15) == 0);
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        const int r = m0 + wm * 16 + gid + 8 * hh;
        if (r >= M) continue;
#pragma unroll
        for (int pl = 0; pl < 2; ++pl) {
            double *crow = (pl ? Ci : Cr) + (i64)r * ldc;
            double2 cv[4];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const int c = n0 + wn * 32 + nt * 8 + 2 * tig;
                if (c + 1 < N && vec2) cv[nt] = *(const double2 *)(crow + c);
                else {
                    cv[nt].x = c < N ? crow[c] : 0.0;
                    cv[nt].y = c + 1 < N ? crow[c + 1] : 0.0;
                }
            }
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const int c = n0 + wn * 32 + nt * 8 + 2 * tig;
                double2 v;
                v.x = cv[nt].x - (pl ? ci[nt][2 * hh] : cr[nt][2 * hh]);
                v.y = cv[nt].y - (pl ? ci[nt][2 * hh + 1] : cr[nt][2 * hh + 1]);
                if (c + 1 < N && vec2) *(double2 *)(crow + c) = v;
                else {
                    if (c < N) crow[c] = v.x;
                    if (c + 1 < N) crow[c + 1] = v.y;
                }
            }
        }
    }
}

bool zgemm_dmma_applicable(const double *Ar, const double *Ai, const double *Br, const double *Bi, i64 ld) {
    return (((uintptr_t)Ar | (uintptr_t)Ai | (uintptr_t)Br | (uintptr_t)Bi) % 16 == 0) && ld % 2 == 0;
}
void launch_zgemm_dmma(double *Cr, double *Ci, const double *Ar, const double *Ai, const double *Br, const double *Bi,
                       i64 ld, i64 M, i64 N, i64 K, cudaStream_t s) {
    if (M <= 0 || N <= 0 || K <= 0) return;
    constexpr i64 rows_max = 65535ll * ZM;  // a grid's rows of tiles (a tall matrix may have more)
    for (; M > rows_max; M -= rows_max, Ar += rows_max * ld, Ai += rows_max * ld, Cr += rows_max * ld, Ci += rows_max * ld)
        launch_zgemm_dmma(Cr, Ci, Ar, Ai, Br, Bi, ld, rows_max, N, K, s);
    CUtensorMap tm[4];
    make_tmap_2d(&tm[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, Ar, K, M, ld, BK, ZM, CU_TENSOR_MAP_SWIZZLE_128B);
    make_tmap_2d(&tm[1], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, Ai, K, M, ld, BK, ZM, CU_TENSOR_MAP_SWIZZLE_128B);
    make_tmap_2d(&tm[2], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, Br, N, K, ld, 8, BK, CU_TENSOR_MAP_SWIZZLE_NONE);
    make_tmap_2d(&tm[3], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, Bi, N, K, ld, 8, BK, CU_TENSOR_MAP_SWIZZLE_NONE);
    set_max_dyn_smem((const void *)k_zgemm_dmma, ZSMEM);
    dim3 grid((unsigned)((N + ZN - 1) / ZN), (unsigned)((M + ZM - 1) / ZM));
    ProfScope ps(KC_GEMM_DMMA, s, 8.0 * M * N * K, 16.0 * (2.0 * M * N + M * K + K * N));
    k_zgemm_dmma<<<grid, NTHREADS, ZSMEM, s>>>(tm[0], tm[1], tm[2], tm[3], Cr, Ci, ld, (int)M, (int)N, (int)K,
                                               cur_abort());
    OXI_LAUNCH_CHECK();
}

}  // namespace oxi
