// FP32-class GEMM on the fifth-generation tensor cores for the trailing updates of the mixed-precision bordered LU
// (the reference factors with LAPACK's dgetrf, src/assembly/solve.jl:54,84): C -= A B with A (m x k), B (k x n) and C
// FP32, column-major.
//
// Each FP32 operand is split into three bf16 pieces, x = x1 + x2 + x3, each piece the bf16 rounding of what the
// previous ones leave (3 x 8 significant bits cover FP32's 24). The six products whose orders reach FP32's precision,
// A1B1 + A1B2 + A2B1 + A1B3 + A2B2 + A3B1, are accumulated in FP32 in tensor memory (the dropped A2B3, A3B2, A3B3 lie
// below 2^-24 |A||B|), so the factors keep FP32 accuracy and the FP64 refinement converges as with FP32 factors. A1B1
// and the five smaller products go to two accumulators, added in the epilogue, so that the small terms are not
// rounded against the large sum at every step.
//
// Layout: a split kernel writes the pieces K-major (A3[p][row][k], B3[p][col][k], bf16, k padded to 64, rows to
// 128). One CTA per 128 x 128 tile of C, 128 threads:
//   - thread 0 stages 64-wide k-slices of the six operand tiles with TMA (cp.async.bulk.tensor, 128-byte swizzle, this
//     GPU's own memory, no multicast) into two shared-memory stages of 96 KB, paced by mbarriers;
//   - thread 32 issues tcgen05.mma (kind::f16, bf16 operands, M 128, N 128, K 16) into two 128-column FP32
//     accumulators in TMEM, 24 per k-slice, and frees each stage with tcgen05.commit;
//   - the four warps read the accumulators back with tcgen05.ld (warp w holds rows 32w..32w+31) and subtract their
//     sum from C (coalesced along C's columns).
// Every mbarrier wait has an iteration limit: a wait that gives up sets the error word, the CTA skips the rest of its
// work and still frees its TMEM; the host reports VP_ERR_TIMEOUT.
//
// FP64 (vp_tc_gemm_sub64, the trailing updates of the FP64 LU): the same tensor cores through exact integer products
// (Ozaki, Ogita, Oishi and Rump's error-free splitting, Numer. Algorithms 59, 2012; its fixed-point form on low-precision
// tensor cores). Each row of A and column of B is scaled by a power of two to |x| <= 1 and rounded to 62 bits, cut into
// nine signed 7-bit digits d_p (x = sum d_p 2^(-6-7p), |d_p| <= 64), bf16 integers. The products of digits p and q are
// integers of at most 2^12; those of equal p + q = s are summed in one FP32 accumulator, exactly while 9 k 2^12 < 2^24,
// k <= 448 (longer sums go in slices). The 45 products with s <= 8 are kept: what is dropped is below 2^-59 of
// |A_i||B_j| (the row's and the column's largest), so that sums whose terms are far below that still come out at DGEMM's
// accuracy (eight digits were measured 10 times worse than DGEMM on rows graded over five decades, nine are better than
// it there and elsewhere). The nine accumulators (48 columns each) are combined in FP64 at the end: 11 FP64 instructions
// an element whatever k, where the FP64 pipe takes k.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>

#include "vp_internal.h"

namespace {

constexpr int TC_BM = 128, TC_BN = 128, TC_BK = 64;
constexpr int TC_PIECES = 3, TC_STAGES = 2, TC_THREADS = 128;
constexpr int TC_TILE_BYTES = TC_BM * TC_BK * 2;                       // 16 KB: one 128 x 64 bf16 tile
constexpr int TC_STAGE_BYTES = 2 * TC_PIECES * TC_TILE_BYTES;          // 96 KB: three A and three B tiles
constexpr int TC_SMEM = TC_STAGES * TC_STAGE_BYTES + 1024;             // + alignment to 1024 bytes
constexpr int TC_TMEM_COLS = 256;  // two FP32 accumulators of 128 lanes x 128 columns: A1B1, and the five small products
constexpr long long TC_WAIT_LIMIT = 1LL << 22;                         // iterations of a bounded mbarrier wait

// the six products (A piece, B piece) of the three-piece split that reach FP32's precision
__constant__ int c_prod_a[6] = {0, 0, 1, 0, 1, 2};
__constant__ int c_prod_b[6] = {0, 1, 0, 2, 1, 0};

__device__ __forceinline__ void split3(float x, __nv_bfloat16& a, __nv_bfloat16& b, __nv_bfloat16& c) {
    a = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(a);  // exact: a is x rounded to 8 significant bits
    b = __float2bfloat16_rn(r1);
    const float r2 = r1 - __bfloat162float(b);
    c = __float2bfloat16_rn(r2);
}

// A (m x k, column-major, lda) -> three K-major pieces dst[p][row][kk] (rows_pad x k_pad each), through a 32 x 32
// shared-memory transpose so that both the reads (along rows) and the writes (along k) are coalesced; zero padding
__global__ void split_a_kernel(int m, int k, const float* __restrict__ A, int lda, int rows_pad, int k_pad,
                               __nv_bfloat16* __restrict__ dst) {
    __shared__ float t[32][33];
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    for (int yy = ty; yy < 32; yy += 8) {
        const int r = r0 + tx, c = c0 + yy;
        t[yy][tx] = (r < m && c < k) ? A[size_t(c) * lda + r] : 0.f;
    }
    __syncthreads();
    const size_t plane = size_t(rows_pad) * k_pad;
    for (int yy = ty; yy < 32; yy += 8) {
        const int r = r0 + yy, c = c0 + tx;
        __nv_bfloat16 a, b, cc;
        split3(t[tx][yy], a, b, cc);
        const size_t o = size_t(r) * k_pad + c;
        dst[o] = a;
        dst[plane + o] = b;
        dst[2 * plane + o] = cc;
    }
}

// B (k x n, column-major, ldb: k contiguous) -> three K-major pieces dst[p][col][kk] (cols_pad x k_pad each)
__global__ void split_b_kernel(int k, int n, const float* __restrict__ B, int ldb, int cols_pad, int k_pad,
                               __nv_bfloat16* __restrict__ dst) {
    const size_t plane = size_t(cols_pad) * k_pad;
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= plane) return;
    const int j = int(i / k_pad), kk = int(i % k_pad);
    const float x = (j < n && kk < k) ? B[size_t(j) * ldb + kk] : 0.f;
    __nv_bfloat16 a, b, c;
    split3(x, a, b, c);
    dst[i] = a;
    dst[plane + i] = b;
    dst[2 * plane + i] = c;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// wait for the phase of the given parity to complete, at most TC_WAIT_LIMIT tries; false (and the error word set)
// when it gives up
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* err) {
    for (long long i = 0; i < TC_WAIT_LIMIT; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    atomicExch(err, 1);
    return false;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// shared-memory matrix descriptor of a K-major bf16 tile in the 128-byte swizzled layout TMA writes: rows of 128 bytes,
// 8-row groups 1024 bytes apart (stride byte offset), descriptor version 1, swizzle mode 128B
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= uint64_t((addr & 0x3FFFF) >> 4);
    d |= uint64_t(16 >> 4) << 16;    // leading byte offset (not used by the swizzled K-major layout)
    d |= uint64_t(1024 >> 4) << 32;  // stride byte offset
    d |= uint64_t(1) << 46;          // version
    d |= uint64_t(2) << 61;          // 128-byte swizzle
    return d;
}

// instruction descriptor of tcgen05.mma kind::f16: FP32 accumulator, bf16 A and B, both K-major, N = 128, M = 128
constexpr uint32_t TC_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(TC_BN >> 3) << 17) | (uint32_t(TC_BM >> 4) << 24);

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem), "l"(ad), "l"(bd), "r"(TC_IDESC), "r"(acc)
        : "memory");
}

// 32 consecutive FP32 columns of this warp's 32 TMEM lanes (one row per thread)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__global__ void __launch_bounds__(TC_THREADS, 1)
    tc_gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, int m, int n,
                   int ktiles, int m_pad, int n_pad, float* __restrict__ C, int ldc, int* err) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[TC_STAGES], empty_bar[TC_STAGES], done_bar;
    __shared__ uint32_t tmem_holder;
    __shared__ int s_fail;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * TC_BM, n0 = blockIdx.y * TC_BN;
    const uint32_t sbase = smem_u32(smem);
    auto tileA = [&](int s, int p) { return sbase + uint32_t(s * TC_STAGE_BYTES + p * TC_TILE_BYTES); };
    auto tileB = [&](int s, int p) { return sbase + uint32_t(s * TC_STAGE_BYTES + (TC_PIECES + p) * TC_TILE_BYTES); };
    if (threadIdx.x == 0) {
        for (int s = 0; s < TC_STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        mbar_init(smem_u32(&done_bar), 1);
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                     "r"(TC_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_holder;

    if (threadIdx.x == 0) {  // TMA producer
        for (int kt = 0; kt < ktiles; ++kt) {
            const int s = kt % TC_STAGES;
            if (kt >= TC_STAGES && !mbar_wait(smem_u32(&empty_bar[s]), uint32_t((kt / TC_STAGES - 1) & 1), err)) {
                s_fail = 1;
                break;
            }
            const uint32_t fb = smem_u32(&full_bar[s]);
            mbar_expect_tx(fb, TC_STAGE_BYTES);
            for (int p = 0; p < TC_PIECES; ++p) {
                tma_load_2d(tileA(s, p), &mapA, kt * TC_BK, p * m_pad + m0, fb);
                tma_load_2d(tileB(s, p), &mapB, kt * TC_BK, p * n_pad + n0, fb);
            }
        }
    } else if (threadIdx.x == 32) {  // MMA issuer
        int issued_hi = 0, issued_lo = 0;
        for (int kt = 0; kt < ktiles; ++kt) {
            const int s = kt % TC_STAGES;
            if (!mbar_wait(smem_u32(&full_bar[s]), uint32_t((kt / TC_STAGES) & 1), err)) {
                s_fail = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int kk = 0; kk < TC_BK / 16; ++kk)
                for (int q = 0; q < 6; ++q) {
                    const uint64_t ad = smem_desc(tileA(s, c_prod_a[q]) + uint32_t(kk * 32));
                    const uint64_t bd = smem_desc(tileB(s, c_prod_b[q]) + uint32_t(kk * 32));
                    if (q == 0)
                        mma_bf16(tmem, ad, bd, issued_hi++ > 0 ? 1u : 0u);
                    else
                        mma_bf16(tmem + uint32_t(TC_BN), ad, bd, issued_lo++ > 0 ? 1u : 0u);
                }
            mma_commit(smem_u32(&empty_bar[s]));
        }
        mma_commit(smem_u32(&done_bar));  // arrives when every MMA issued above has completed
    }
    __syncwarp();
    // epilogue: the accumulator back from TMEM, C -= D
    const bool done = mbar_wait(smem_u32(&done_bar), 0u, err);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    if (done && !s_fail) {
        const int row = m0 + warp * 32 + lane;
        for (int c0 = 0; c0 < TC_BN; c0 += 32) {
            uint32_t v[32], u[32];
            const uint32_t taddr = tmem + (uint32_t(warp * 32) << 16) + uint32_t(c0);
            tmem_ld32(taddr, v);
            tmem_ld32(taddr + uint32_t(TC_BN), u);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (row < m)
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const int col = n0 + c0 + j;
                    if (col < n) C[size_t(col) * ldc + row] -= __uint_as_float(v[j]) + __uint_as_float(u[j]);
                }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM_COLS) : "memory");
}

// ---- FP64 ------------------------------------------------------------------------------------------------------------

constexpr int TD_BN = 48, TD_BK = 32, TD_DIGITS = 9, TD_PAIRS = (TD_DIGITS + 1) / 2, TD_STAGES = 2;
constexpr int TD_A_BYTES = TC_BM * 128, TD_B_BYTES = TD_BN * 128;  // a tile of two digits of 32 k: rows of 128 bytes
constexpr int TD_STAGE_BYTES = TD_PAIRS * (TD_A_BYTES + TD_B_BYTES);  // 110 KB
constexpr int TD_SMEM = TD_STAGES * TD_STAGE_BYTES + 1024;
constexpr int TD_KMAX = 448;       // exact integer sums in FP32
constexpr int TD_TMEM_COLS = 512;  // nine accumulators of 48 columns
constexpr int TD_EMID = 400;       // scales within 2^+-this combine in one factor

// the largest exponent field of every row of A (m x k, column-major), or (rows = 0) of every column: into ex (zeroed).
// Exponent fields order as the numbers; 2047 marks an infinity or NaN.
__global__ void row_exp_kernel(int m, int k, const double* __restrict__ A, int lda, int* __restrict__ ex) {
    const int r = blockIdx.x * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
    int e = 0;
    if (r < m)
        for (int c = blockIdx.y * 64 + w; c < min(k, int(blockIdx.y) * 64 + 64); c += 8)
            e = max(e, (__double2hiint(A[size_t(c) * lda + r]) >> 20) & 2047);
    __shared__ int s[8][32];
    s[w][threadIdx.x & 31] = e;
    __syncthreads();
    if (w == 0 && r < m) {
        for (int q = 1; q < 8; ++q) e = max(e, s[q][threadIdx.x]);
        atomicMax(ex + r, e);
    }
}
__global__ void col_exp_kernel(int k, int n, const double* __restrict__ B, int ldb, int* __restrict__ ex) {
    const int c = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (c >= n) return;
    int e = 0;
    for (int r = lane; r < k; r += 32) e = max(e, (__double2hiint(B[size_t(c) * ldb + r]) >> 20) & 2047);
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) ex[c] = e;
}

// 2^e for the exponents of normal numbers
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }
// |x| < 2^this for every x of the field (-1021 to 1024; 1025 for an infinity or NaN)
__device__ __forceinline__ int scale_exp(int field) { return max(field, 1) - 1022; }
// the scale 2^e of a row or column, or NaN (nan: it holds an infinity or NaN); 1 outside 2^+-TD_EMID, where the epilogue takes
// the exponents: as factors cut at 2^-900, they lost the digits of smaller entries
__device__ __forceinline__ double scale_of(int e, bool nan) {
    return nan ? __longlong_as_double(0x7ff8000000000000LL) : (abs(e) <= TD_EMID ? pow2(e) : 1.0);
}

// x 2^(62 - e) where the factor is no normal number (out of line: the digit kernels are bound by their instructions)
__device__ __noinline__ double digits_tiny(double x, int e) { return (x * pow2(1000)) * pow2(62 - 1000 - e); }

// the digits of x, |x| < 2^e, to dst[q * plane + par * 32], digit 2 q + par
__device__ __forceinline__ void put_digits(double x, int e, __nv_bfloat16* dst, size_t plane) {
    long long u = __double2ll_rn(e < 62 - 1000 ? digits_tiny(x, e) : x * pow2(62 - e));
#pragma unroll
    for (int p = TD_DIGITS - 1; p >= 0; --p) {
        const int d = p ? (int(u + 64) & 127) - 64 : int(u);
        dst[(p >> 1) * plane + (p & 1) * 32] = __float2bfloat16_rn(float(d));
        u = (u - d) >> 7;
    }
}

// A (m x k, column-major) -> digits dst[q][row][k / 32][digit parity][k % 32] (TD_PAIRS planes q of rows_pad rows of 2 k_pad
// elements), through a 32 x 32 shared-memory transpose; the odd place of the last pair stays unwritten and unread
__global__ void digits_a_kernel(int m, int k, const double* __restrict__ A, int lda, int rows_pad, int k_pad,
                                const int* __restrict__ ex, __nv_bfloat16* __restrict__ dst) {
    __shared__ double t[32][33];
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    for (int yy = ty; yy < 32; yy += 8) {
        const int r = r0 + tx, c = c0 + yy;
        t[yy][tx] = (r < m && c < k) ? A[size_t(c) * lda + r] : 0.0;
    }
    __syncthreads();
    const size_t plane = size_t(rows_pad) * 2 * k_pad;
    for (int yy = ty; yy < 32; yy += 8) {
        const int r = r0 + yy;
        put_digits(t[tx][yy], r < m ? scale_exp(ex[r]) : 0, dst + size_t(r) * 2 * k_pad + 2 * c0 + tx, plane);
    }
}
// B (k x n, column-major) -> digits dst[q][column][..] in the same layout
__global__ void digits_b_kernel(int k, int n, const double* __restrict__ B, int ldb, int cols_pad, int k_pad,
                                const int* __restrict__ ex, __nv_bfloat16* __restrict__ dst) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= size_t(cols_pad) * k_pad) return;
    const int j = int(i / k_pad), kk = int(i % k_pad);
    const double x = (j < n && kk < k) ? B[size_t(j) * ldb + kk] : 0.0;
    put_digits(x, j < n ? scale_exp(ex[j]) : 0, dst + size_t(j) * 2 * k_pad + 2 * (kk & ~31) + (kk & 31),
               size_t(cols_pad) * 2 * k_pad);
}

constexpr uint32_t TD_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(TD_BN >> 3) << 17) | (uint32_t(TC_BM >> 4) << 24);

__device__ __forceinline__ void mma_digits(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem), "l"(ad), "l"(bd), "r"(TD_IDESC), "r"(acc)
        : "memory");
}

// 8 consecutive FP32 columns of this warp's 32 TMEM lanes (one row per thread)
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}

// C (m x n) -= A B for one slice of k <= TD_KMAX: one CTA per 128 x 48 tile of C, as tc_gemm_kernel
__global__ void __launch_bounds__(TC_THREADS, 1)
    tc_gemm64_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, int m, int n,
                     int ktiles, int m_pad, int n_pad, const int* __restrict__ exA, const int* __restrict__ exB,
                     double* __restrict__ C, int ldc, int* err) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[TD_STAGES], empty_bar[TD_STAGES], done_bar;
    __shared__ uint32_t tmem_holder;
    __shared__ int s_fail;
    __shared__ double s_scale[TD_BN];
    __shared__ int s_exp[TD_BN];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * TC_BM, n0 = blockIdx.y * TD_BN;
    const uint32_t sbase = smem_u32(smem);
    auto tileA = [&](int s, int q) { return sbase + uint32_t(s * TD_STAGE_BYTES + q * TD_A_BYTES); };
    auto tileB = [&](int s, int q) { return sbase + uint32_t(s * TD_STAGE_BYTES + TD_PAIRS * TD_A_BYTES + q * TD_B_BYTES); };
    if (threadIdx.x == 0) {
        for (int s = 0; s < TD_STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        mbar_init(smem_u32(&done_bar), 1);
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // the columns' scales 2^(e - 68), which a row's 2^e makes C's
    bool cfar = false;
    for (int j = threadIdx.x; j < TD_BN; j += TC_THREADS) {
        const int f = n0 + j < n ? exB[n0 + j] : 1022, e = scale_exp(f) - 68;
        s_exp[j] = e;
        s_scale[j] = scale_of(e, f == 2047);
        cfar |= f < 2047 && abs(e) > TD_EMID;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                     "r"(TD_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cfar = __syncthreads_or(cfar) != 0;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_holder;

    if (threadIdx.x == 0) {  // TMA producer
        for (int kt = 0; kt < ktiles; ++kt) {
            const int s = kt % TD_STAGES;
            if (kt >= TD_STAGES && !mbar_wait(smem_u32(&empty_bar[s]), uint32_t((kt / TD_STAGES - 1) & 1), err)) {
                s_fail = 1;
                break;
            }
            const uint32_t fb = smem_u32(&full_bar[s]);
            mbar_expect_tx(fb, TD_STAGE_BYTES);
            for (int q = 0; q < TD_PAIRS; ++q) {
                tma_load_2d(tileA(s, q), &mapA, kt * 2 * TD_BK, q * m_pad + m0, fb);
                tma_load_2d(tileB(s, q), &mapB, kt * 2 * TD_BK, q * n_pad + n0, fb);
            }
        }
    } else if (threadIdx.x == 32) {  // MMA issuer
        for (int kt = 0; kt < ktiles; ++kt) {
            const int s = kt % TD_STAGES;
            if (!mbar_wait(smem_u32(&full_bar[s]), uint32_t((kt / TD_STAGES) & 1), err)) {
                s_fail = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int kk = 0; kk < TD_BK / 16; ++kk)
                for (int g = 0; g < TD_DIGITS; ++g)
                    for (int p = 0; p <= g; ++p) {
                        const int q = g - p;
                        const uint64_t ad = smem_desc(tileA(s, p >> 1) + uint32_t((p & 1) * 64 + kk * 32));
                        const uint64_t bd = smem_desc(tileB(s, q >> 1) + uint32_t((q & 1) * 64 + kk * 32));
                        mma_digits(tmem + uint32_t(g * TD_BN), ad, bd, (kt | kk | p) ? 1u : 0u);
                    }
            mma_commit(smem_u32(&empty_bar[s]));
        }
        mma_commit(smem_u32(&done_bar));  // arrives when every MMA issued above has completed
    }
    __syncwarp();
    // epilogue: the accumulators (integers) combined, C -= D
    const bool done = mbar_wait(smem_u32(&done_bar), 0u, err);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    if (done && !s_fail) {
        const int row = m0 + warp * 32 + lane;
        const int f = row < m ? exA[row] : 1022, er = scale_exp(f);
        const double sr = scale_of(er, f == 2047);
        const bool far = cfar || (f < 2047 && abs(er) > TD_EMID);
        for (int c0 = 0; c0 < TD_BN; c0 += 8) {
            uint32_t v[TD_DIGITS][8];
            const uint32_t taddr = tmem + (uint32_t(warp * 32) << 16) + uint32_t(c0);
#pragma unroll
            for (int g = 0; g < TD_DIGITS; ++g) tmem_ld8(taddr + uint32_t(g * TD_BN), v[g]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            auto value = [&](int j) {
                int t[4];  // groups 2 h and 2 h + 1: below 2^31 (group g is at most (g + 1) 448 2^12)
#pragma unroll
                for (int h = 0; h < 4; ++h)
                    t[h] = __float2int_rn(__uint_as_float(v[2 * h][j])) * 128 + __float2int_rn(__uint_as_float(v[2 * h + 1][j]));
                double x = double(t[0]);
                x = fma(x, 16384.0, double(t[1]));
                x = fma(x, 16384.0, double(t[2]));
                x = fma(x, 16384.0, double(t[3]));
                return fma(x, 128.0, double(__uint_as_float(v[8][j])));
            };
            if (row < m && !far) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int col = n0 + c0 + j;
                    const double x = value(j);
                    if (col < n) {
                        double* c = C + size_t(col) * ldc + row;
                        *c = fma(-x, sr * s_scale[c0 + j], *c);
                    }
                }
            } else if (row < m) {  // 2^(row + column) in two factors
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int col = n0 + c0 + j, e = er + s_exp[c0 + j], h = max(e / 2, -1022);
                    const double x = value(j), s = sr * s_scale[c0 + j];
                    if (col < n) {
                        double* c = C + size_t(col) * ldc + row;
                        *c = isnan(s) ? s : fma(-(x * pow2(h)), pow2(max(e - h, -1022)), *c);
                    }
                }
            }
            __syncwarp();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TD_TMEM_COLS) : "memory");
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// the tensor map of `planes` stacked K-major planes (rows_pad rows of `cols` bf16 each), box 64 x box_rows, 128-byte
// swizzle
bool make_map(CUtensorMap* map, void* base, int planes, int rows_pad, int cols, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t gdim[2] = {cuuint64_t(cols), cuuint64_t(planes) * cuuint64_t(rows_pad)};
    const cuuint64_t gstride[1] = {cuuint64_t(cols) * 2};
    const cuuint32_t box[2] = {64, cuuint32_t(box_rows)};
    const cuuint32_t estride[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
           CUDA_SUCCESS;
}

}  // namespace

bool vp_tc_gemm_enabled() {
    const char* e = std::getenv("VP_LU_TENSOR_CORES");
    return !(e && e[0] == '0');
}

bool vp_tc_gemm_fits(int m, int n, int k) { return m >= TC_BM && n >= TC_BN && k >= TC_BK; }

void vp_tc_work_free(TcWork* w) {
    if (w->pieces) cudaFree(w->pieces);
    if (w->exps) cudaFree(w->exps);
    if (w->err) cudaFree(w->err);
    *w = TcWork();
}

namespace {

// room for `elems` bf16 elements and `nexp` exponents, and the error word (kept as it is when the rest grows)
int tc_reserve(vp_ctx* ctx, size_t elems, size_t nexp) {
    TcWork* w = &ctx->tc;
    int r;
    if (!w->err) {
        if ((r = vp_alloc(ctx, &w->err, 1))) return r;
        VP_CUDA(ctx, cudaMemsetAsync(w->err, 0, sizeof(int), ctx->stream));
    }
    if (elems > w->cap) {
        if (w->pieces) cudaFree(w->pieces);
        w->pieces = nullptr;
        w->cap = 0;
        __nv_bfloat16* p = nullptr;
        if ((r = vp_alloc(ctx, &p, elems))) return r;
        w->pieces = p;
        w->cap = elems;
    }
    if (nexp > w->nexp) {
        if (w->exps) cudaFree(w->exps);
        w->exps = nullptr;
        w->nexp = 0;
        if ((r = vp_alloc(ctx, &w->exps, nexp))) return r;
        w->nexp = nexp;
    }
    return VP_OK;
}

}  // namespace

// k >= 64, and enough work: below about 16M multiply-adds the five launches (58 us) take longer than cuBLAS's DGEMM
// (1000 x 64 x 64: 58 against 25 us; 6000 x 64 x 64: 63 against 81; 6000 x 128 x 128: 70 against 226)
bool vp_tc_gemm64_fits(int m, int n, int k) {
    return m >= TC_BM && n >= TD_BN && k >= 64 && double(m) * n * k >= 1.6e7;
}

int vp_tc_gemm_sub64(vp_ctx* ctx, int m, int n, int k, const double* A, int lda, const double* B, int ldb, double* C,
                     int ldc) {
    if (m <= 0 || n <= 0 || k <= 0) return VP_OK;
    const int m_pad = (m + TC_BM - 1) / TC_BM * TC_BM, n_pad = (n + TD_BN - 1) / TD_BN * TD_BN;
    const int kc = std::min(k, TD_KMAX), kc_pad = (kc + TD_BK - 1) / TD_BK * TD_BK;
    const size_t na = size_t(2 * TD_PAIRS) * m_pad * kc_pad, nb = size_t(2 * TD_PAIRS) * n_pad * kc_pad;
    int r = tc_reserve(ctx, na + nb, size_t(m_pad) + n_pad);
    if (r) return r;
    TcWork* w = &ctx->tc;
    if (!w->attr64_set) {
        VP_CUDA(ctx, cudaFuncSetAttribute(tc_gemm64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TD_SMEM));
        w->attr64_set = true;
    }
    __nv_bfloat16* da = static_cast<__nv_bfloat16*>(w->pieces);
    __nv_bfloat16* db = da + na;
    int *ea = w->exps, *eb = w->exps + m_pad;
    for (int k0 = 0; k0 < k; k0 += TD_KMAX) {
        const int kk = std::min(TD_KMAX, k - k0), k_pad = (kk + TD_BK - 1) / TD_BK * TD_BK;
        const double *a = A + size_t(k0) * lda, *b = B + k0;
        VP_CUDA(ctx, cudaMemsetAsync(ea, 0, sizeof(int) * m_pad, ctx->stream));
        row_exp_kernel<<<dim3(m_pad / 32, (kk + 63) / 64), 256, 0, ctx->stream>>>(m, kk, a, lda, ea);
        col_exp_kernel<<<(n + 7) / 8, 256, 0, ctx->stream>>>(kk, n, b, ldb, eb);
        digits_a_kernel<<<dim3(m_pad / 32, k_pad / 32), 256, 0, ctx->stream>>>(m, kk, a, lda, m_pad, k_pad, ea, da);
        digits_b_kernel<<<int((size_t(n_pad) * k_pad + 255) / 256), 256, 0, ctx->stream>>>(kk, n, b, ldb, n_pad, k_pad, eb, db);
        CUtensorMap ma, mb;
        if (!make_map(&ma, da, TD_PAIRS, m_pad, 2 * k_pad, TC_BM) || !make_map(&mb, db, TD_PAIRS, n_pad, 2 * k_pad, TD_BN))
            return vp_fail(ctx, VP_ERR_CUDA, "cuTensorMapEncodeTiled failed");
        tc_gemm64_kernel<<<dim3(m_pad / TC_BM, n_pad / TD_BN), TC_THREADS, TD_SMEM, ctx->stream>>>(
            ma, mb, m, n, k_pad / TD_BK, m_pad, n_pad, ea, eb, C, ldc, w->err);
        ctx->launches += 5;
    }
    VP_CUDA(ctx, cudaGetLastError());
    return VP_OK;
}

int vp_tc_gemm_sub(vp_ctx* ctx, int m, int n, int k, const float* A, int lda, const float* B, int ldb, float* C,
                   int ldc) {
    if (m <= 0 || n <= 0 || k <= 0) return VP_OK;
    TcWork* w = &ctx->tc;
    const int m_pad = (m + TC_BM - 1) / TC_BM * TC_BM, n_pad = (n + TC_BN - 1) / TC_BN * TC_BN;
    const int k_pad = (k + TC_BK - 1) / TC_BK * TC_BK;
    const size_t na = size_t(TC_PIECES) * m_pad * k_pad, nb = size_t(TC_PIECES) * n_pad * k_pad;
    int r = tc_reserve(ctx, na + nb, 0);
    if (r) return r;
    if (!w->attr_set) {
        VP_CUDA(ctx, cudaFuncSetAttribute(tc_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM));
        w->attr_set = true;
    }
    __nv_bfloat16* a3 = static_cast<__nv_bfloat16*>(w->pieces);
    __nv_bfloat16* b3 = a3 + na;
    split_a_kernel<<<dim3(m_pad / 32, k_pad / 32), 256, 0, ctx->stream>>>(m, k, A, lda, m_pad, k_pad, a3);
    split_b_kernel<<<int((size_t(n_pad) * k_pad + 255) / 256), 256, 0, ctx->stream>>>(k, n, B, ldb, n_pad, k_pad, b3);
    CUtensorMap ma, mb;
    if (!make_map(&ma, a3, TC_PIECES, m_pad, k_pad, TC_BM) || !make_map(&mb, b3, TC_PIECES, n_pad, k_pad, TC_BN))
        return vp_fail(ctx, VP_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    tc_gemm_kernel<<<dim3(m_pad / TC_BM, n_pad / TC_BN), TC_THREADS, TC_SMEM, ctx->stream>>>(
        ma, mb, m, n, k_pad / TC_BK, m_pad, n_pad, C, ldc, w->err);
    ctx->launches += 3;
    VP_CUDA(ctx, cudaGetLastError());
    return VP_OK;
}

int vp_tc_gemm_check(vp_ctx* ctx) {
    TcWork* w = &ctx->tc;
    if (!w->err) return VP_OK;
    int e = 0;
    VP_CUDA(ctx, vp_d2h(ctx, &e, w->err, sizeof(int)));
    VP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (e) {
        cudaMemsetAsync(w->err, 0, sizeof(int), ctx->stream);
        return vp_fail(ctx, VP_ERR_TIMEOUT, "tensor-core GEMM: a bounded wait gave up");
    }
    return VP_OK;
}

extern "C" int vp_gemm_sub_f32(vp_ctx* ctx, int m, int n, int k, const float* A, int lda, const float* B, int ldb,
                               float* C, int ldc) {
    if (!ctx || m <= 0 || n <= 0 || k <= 0 || !A || !B || !C || lda < m || ldb < k || ldc < m)
        return vp_fail(ctx, VP_ERR_ARG, "bad argument");
    DeviceGuard dg;
    if (dg.set(ctx->device) != cudaSuccess) return vp_fail(ctx, VP_ERR_CUDA, "cudaSetDevice");
    float *dA, *dB, *dC;
    int r;
    if ((r = vp_upload(ctx, &dA, A, size_t(lda) * k))) return r;
    if ((r = vp_upload(ctx, &dB, B, size_t(ldb) * n))) {
        cudaFree(dA);
        return r;
    }
    if ((r = vp_upload(ctx, &dC, C, size_t(ldc) * n))) {
        cudaFree(dA);
        cudaFree(dB);
        return r;
    }
    r = vp_tc_gemm_sub(ctx, m, n, k, dA, lda, dB, ldb, dC, ldc);
    if (!r) r = vp_tc_gemm_check(ctx);
    if (!r) {
        cudaError_t e = vp_d2h(ctx, C, dC, sizeof(float) * size_t(ldc) * n);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) r = vp_fail(ctx, VP_ERR_CUDA, std::string("vp_gemm_sub_f32: ") + cudaGetErrorString(e));
    }
    cudaFree(dA);
    cudaFree(dB);
    cudaFree(dC);
    return r;
}
