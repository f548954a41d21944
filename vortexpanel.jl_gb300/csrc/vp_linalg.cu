// Bordered dense solve on the GPU: factorize_galerkin / solve_galerkin of src/assembly/solve.jl:15-115 over the
// Galerkin reduction C' A [C; W] of src/dofmap/system.jl:141-165.
//
//  - reduction + border: one kernel gathers M = C' A Cf (A row-major FP64, C and Cf sparse) into a column-major FP64
//    matrix through a shared-memory transpose, then the border rows/columns (scaled to the mean |diagonal|) are set;
//  - LU with partial pivoting (the reference calls LAPACK dgetrf): recursive (left half, swap, TRSM, GEMM, right
//    half). Its leaf panels (m x 16 columns) are factored by one thread-block cluster (1 to 16 CTAs) that holds the panel in
//    registers: per column, every CTA sends its pivot candidate's row to all, every thread picks the pivot, swaps and
//    updates its rows; panels of 64 columns are factored leaf by leaf with swap and update kernels of their own. The
//    trailing updates run on the tensor cores (vp_tcgemm.cu): VP_MIXED by
//    three-piece bf16 splits (FP32-class), VP_FP64 by exact products of 7-bit digits (FP64-class), for updates of at
//    least a tile of the kernels, cuBLAS for the smaller ones; TRSM is cuBLAS, in FP64 on 64 x 64 diagonal blocks only;
//  - VP_MIXED keeps the FP64 bordered matrix and refines every solve with FP64 residuals (iterative refinement) to
//    FP64 accuracy;
//  - the 1-norm condition estimate of dgecon (Hager/Higham, as LAPACK dlacn2) from solves with M and M'.
#include <cooperative_groups.h>

#include <algorithm>
#include <climits>
#include <cmath>

#include "vp_internal.h"

namespace cg = cooperative_groups;

namespace {

constexpr int LU_CL = 8;       // CTAs per cluster of the leaf kernel
constexpr int LU_THREADS = 512;
// right hand sides from which the FP64 residual is one product on the tensor cores: its cost hardly depends on them (the
// digits of M), a matrix-vector product takes 0.1 ms each at 6.6k unknowns: 64 of them 6.9 ms an iteration, one product 2
constexpr int RES_TC = 24;

// M(q, q') = sum_{i in C[:,q]} C[i,q] sum_{j in Cf[:,q']} A[i, j] Cf[j,q'], written column-major (ld n)
__global__ void reduce_kernel(int nq, int n, const double* __restrict__ A, long long lda, const int* __restrict__ ctp,
                              const int* __restrict__ cti, const double* __restrict__ ctv,
                              const int* __restrict__ cfp, const int* __restrict__ cfi,
                              const double* __restrict__ cfv, double* __restrict__ M) {
    __shared__ double tile[32][33];
    const int q0 = blockIdx.y * 32, p0 = blockIdx.x * 32;  // q rows of M, p columns of M
    const int tx = threadIdx.x, ty = threadIdx.y;          // 32 x 8
    for (int yy = ty; yy < 32; yy += 8) {
        int q = q0 + yy, p = p0 + tx;
        double acc = 0;
        if (q < nq && p < nq) {
            for (int u = ctp[q]; u < ctp[q + 1]; ++u) {
                const double* Ar = A + size_t(cti[u]) * size_t(lda);
                double part = 0;
                for (int v = cfp[p]; v < cfp[p + 1]; ++v) part += Ar[cfi[v]] * cfv[v];
                acc += ctv[u] * part;
            }
        }
        tile[yy][tx] = acc;
    }
    __syncthreads();
    for (int yy = ty; yy < 32; yy += 8) {
        int p = p0 + yy, q = q0 + tx;
        if (q < nq && p < nq) M[size_t(p) * n + q] = tile[tx][yy];
    }
}

__global__ void border_kernel(int nq, int n, int nb, const double* __restrict__ ecol, const double* __restrict__ crow,
                              double* __restrict__ M) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int k = 0; k < nb; ++k) {
        // column nq+k: se_k e_k on the unknowns, 0 on the border rows; row nq+k: scaled c_k, 0 in the corner
        M[size_t(nq + k) * n + i] = i < nq ? ecol[size_t(k) * nq + i] : 0.0;
        if (i < nq) M[size_t(i) * n + nq + k] = crow[size_t(k) * nq + i];
    }
}

template <class T>
__global__ void col_abs_sum_kernel(int n, const T* __restrict__ M, double* __restrict__ out) {
    __shared__ double red[256];
    int c = blockIdx.x;
    double s = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += fabs(double(M[size_t(c) * n + i]));
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[c] = red[0];
}

// |v| as an unsigned key that orders as the magnitudes (above the infinity's: NaN)
__device__ __forceinline__ unsigned mag_key(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ unsigned long long mag_key(double v) {
    return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}
__device__ __forceinline__ bool key_nan(unsigned k) { return k > 0x7f800000u; }
__device__ __forceinline__ bool key_nan(unsigned long long k) { return k > 0x7ff0000000000000ull; }

// the index of the largest key of a warp's candidates (key, i), the smallest index on ties; INT_MAX: no candidate
__device__ __forceinline__ int warp_best(unsigned key, int i) {
    const unsigned m = __reduce_max_sync(0xffffffffu, i == INT_MAX ? 0u : key);
    return __reduce_min_sync(0xffffffffu, key == m ? i : INT_MAX);
}
__device__ __forceinline__ int warp_best(unsigned long long key, int i) {
    const unsigned hi = unsigned(key >> 32), lo = unsigned(key);
    const unsigned mh = __reduce_max_sync(0xffffffffu, i == INT_MAX ? 0u : hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh && i != INT_MAX ? lo : 0u);
    return __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? i : INT_MAX);
}

// a CTA's pivot candidate of a column: its row, the reciprocal of its pivot (FP64), its index (INT_MAX: none)
template <class T, int W>
struct alignas(16) LeafCand {
    T row[W];
    T rcp;
    int idx;
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return unsigned(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ unsigned cluster_addr(unsigned a, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// 16 bytes to another CTA's shared memory, counted on its mbarrier
__device__ __forceinline__ void send16(unsigned dst, uint4 v, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
                 : "memory");
}

constexpr long long LEAF_WAIT_LIMIT = 1LL << 20;  // tries of a bounded wait

// LU leaf: rows [c0, c0 + m) x columns [c0, c0 + w) (w <= W) of the column-major matrix (ld lda), partial pivoting, by a
// cluster of CL CTAs. Rows are split over the CTAs (R each) and stay in registers for the whole panel, RPT rows a
// thread. A column is one chain of latencies - search, exchange, elimination - so what bounds a leaf is the steps in
// that chain: each warp finds its candidate and writes that row to shared memory, one warp picks the CTA's and sends it
// to every CTA's shared memory, where an mbarrier counts the bytes; all threads wait for the candidates on their own
// mbarrier, pick the pivot, swap and eliminate. (With the panel in shared memory, reads from the other CTAs after a
// cluster barrier and three more block barriers a column took 7 us; now 2.9 us at 8 CTAs and 4.0 at 16, in a launch list of
// the 12.8k mixed system.) A panel that one CTA holds needs block barriers only. FP64 multiplies by the pivot's reciprocal, computed once
// by the CTA that sends it: a division per row is ten FP64 instructions of each warp.
template <class T, int W, int RPT, int CL, int NT>
__global__ void __launch_bounds__(NT)
    lu_leaf_kernel(T* A, long long lda, int c0, int m, int w, int R, int* __restrict__ ipiv,
                   int* __restrict__ info) {
    cg::cluster_group cl = cg::this_cluster();
    const int rank = CL > 1 ? (int)cl.block_rank() : 0;
    constexpr int NV = sizeof(LeafCand<T, W>) / 16, NR = W * sizeof(T) / 16;
    __shared__ LeafCand<T, W> s_cand[2][CL];         // written by every CTA of the cluster
    __shared__ alignas(16) T s_rowj[2][W];           // row j, written by its owner
    __shared__ LeafCand<T, W> s_warp[NT / 32];
    __shared__ alignas(16) T s_mine[W];
    __shared__ alignas(8) unsigned long long s_bar[2];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nt = blockDim.x, nw = nt >> 5;
    const int row0 = rank * R;
    const int nloc = max(0, min(R, m - row0));
    if (CL > 1) {
        if (tid == 0) {
            for (int b = 0; b < 2; ++b) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s_bar[b])) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        cl.sync();
    }
    T a[RPT][W];
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        const int li = tid + r * nt;
#pragma unroll
        for (int k = 0; k < W; ++k)
            a[r][k] = li < nloc && k < w ? A[size_t(c0 + k) * size_t(lda) + size_t(c0 + row0 + li)] : T(0);
    }
    bool lost = false;
#pragma unroll
    for (int j = 0; j < W; ++j) {
        if (j >= w) break;
        const int buf = j & 1;
        if (CL > 1 && tid == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&s_bar[buf])),
                         "r"(unsigned(CL * sizeof(LeafCand<T, W>) + W * sizeof(T)))
                         : "memory");
        // 1. this warp's candidate: the largest |a(i, j)| over its rows i >= j (smallest index on ties)
        decltype(mag_key(T(0))) bk = 0;
        int bi = INT_MAX;
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            const int li = tid + r * nt, i = row0 + li;
            const auto k = mag_key(a[r][j]);
            if (li < nloc && i >= j && !key_nan(k) && (k > bk || bi == INT_MAX)) {
                bk = k;
                bi = i;
            }
        }
        const int wi = warp_best(bk, bi);
        if (wi == INT_MAX) {
            if (lane == 0) s_warp[wid].idx = INT_MAX;
        } else if (bi == wi) {
            s_warp[wid].idx = wi;
#pragma unroll
            for (int r = 0; r < RPT; ++r)
                if (row0 + tid + r * nt == wi)
#pragma unroll
                    for (int k = 0; k < W; ++k) s_warp[wid].row[k] = a[r][k];
        }
        const bool own_j = j >= row0 && j < row0 + nloc;
        if (own_j)
#pragma unroll
            for (int r = 0; r < RPT; ++r)
                if (row0 + tid + r * nt == j)
#pragma unroll
                    for (int k = 0; k < W; ++k) (CL > 1 ? s_mine : s_rowj[buf])[k] = a[r][k];
        __syncthreads();
        // 2. the CTA's candidate, to every CTA of the cluster, and row j
        if (wid == 0) {
            const int ix = lane < nw ? s_warp[lane].idx : INT_MAX;
            const int ci = warp_best(ix != INT_MAX ? mag_key(s_warp[lane].row[j]) : 0, ix);
            const unsigned who = __ballot_sync(0xffffffffu, ix == ci);
            LeafCand<T, W>* c = &s_warp[__ffs(who) - 1];
            if (sizeof(T) == 8) {
                const T rc = ci != INT_MAX ? T(1) / c->row[j] : T(0);
                if (lane == 0) c->rcp = rc;
                __syncwarp();
            }
            const uint4* src = reinterpret_cast<const uint4*>(c);
            if (CL > 1) {
                for (int e = lane; e < CL * NV; e += 32) {
                    const int dst = e / NV, k = e - dst * NV;
                    send16(cluster_addr(smem_addr(&s_cand[buf][rank]) + 16 * k, dst), src[k],
                           cluster_addr(smem_addr(&s_bar[buf]), dst));
                }
                if (own_j)
                    for (int e = lane; e < CL * NR; e += 32) {
                        const int dst = e / NR, k = e - dst * NR;
                        send16(cluster_addr(smem_addr(&s_rowj[buf][0]) + 16 * k, dst), reinterpret_cast<const uint4*>(s_mine)[k],
                               cluster_addr(smem_addr(&s_bar[buf]), dst));
                    }
            } else {
                for (int k = lane; k < NV; k += 32) reinterpret_cast<uint4*>(&s_cand[buf][0])[k] = src[k];
            }
        }
        if (CL > 1) {
            unsigned done = 0;
            for (long long t = 0; t < LEAF_WAIT_LIMIT && !done && !lost; ++t)
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                    "selp.u32 %0, 1, 0, p;\n\t}"
                    : "=r"(done)
                    : "r"(smem_addr(&s_bar[buf])), "r"(unsigned(j >> 1) & 1u)
                    : "memory");
            if (!done) lost = true;  // the loop goes on without waits, so that the other barriers end; the factors are dropped
        } else {
            __syncthreads();
        }
        // 3. the pivot over the cluster
        decltype(mag_key(T(0))) gk = 0;
        int p = INT_MAX, pr = 0;
#pragma unroll
        for (int r = 0; r < CL; ++r) {
            const int ix = s_cand[buf][r].idx;
            const auto k = mag_key(s_cand[buf][r].row[j]);
            if (ix != INT_MAX && (k > gk || p == INT_MAX || (k == gk && ix < p))) {
                gk = k;
                p = ix;
                pr = r;
            }
        }
        if (gk == 0 || lost) {
            if (lost) atomicExch(info, -1);
            if (rank == 0 && tid == 0) {
                if (*info == 0) *info = c0 + j + 1;
                ipiv[c0 + j] = c0 + j;
            }
            continue;
        }
        if (rank == 0 && tid == 0) ipiv[c0 + j] = c0 + p;
        const T* piv = s_cand[buf][pr].row;
        // 4. swap rows j and p, eliminate below the pivot (l = 0 leaves a row alone)
        const T pj = piv[j], rj = s_cand[buf][pr].rcp;
        const bool mul = sizeof(T) == 8 && fabs(double(pj)) > 1e-300;
        T l[RPT];
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            const int li = tid + r * nt, i = row0 + li;
            if (i == p && p != j && li < nloc)
#pragma unroll
                for (int k = 0; k < W; ++k) a[r][k] = s_rowj[buf][k];
            if (i == j && li < nloc)
#pragma unroll
                for (int k = 0; k < W; ++k) a[r][k] = piv[k];
            l[r] = T(0);
            if (i > j && li < nloc) a[r][j] = l[r] = mul ? a[r][j] * rj : a[r][j] / pj;
        }
#pragma unroll
        for (int k = 0; k < W; ++k)
            if (k > j) {
                const T pk = piv[k];
#pragma unroll
                for (int r = 0; r < RPT; ++r) a[r][k] -= l[r] * pk;
            }
    }
    asm volatile("" : "+l"(A));  // the store addresses computed anew, not kept in registers since the loads
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        const int li = tid + r * nt;
#pragma unroll
        for (int k = 0; k < W; ++k)
            if (li < nloc && k < w) A[size_t(c0 + k) * size_t(lda) + size_t(c0 + row0 + li)] = a[r][k];
    }
    if (CL > 1) cl.sync();  // no CTA leaves while another may still write its shared memory
}

// The LU leaf for panels too tall for the cluster's registers (over 16,384 rows, or where only clusters of 8 CTAs are to be
// had): the panel in shared memory.
template <class T, int W>
__global__ void __cluster_dims__(LU_CL, 1, 1) __launch_bounds__(LU_THREADS)
    lu_leaf_tall_kernel(T* __restrict__ A, long long lda, int c0, int m, int w, int R, int* __restrict__ ipiv,
                   int* __restrict__ info) {
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    extern __shared__ __align__(16) unsigned char smraw[];
    T* pan = reinterpret_cast<T*>(smraw);  // R x W, row-major
    __shared__ T s_cval[2];
    __shared__ int s_cidx[2];
    __shared__ T s_crow[2][W];
    __shared__ T s_rowj[2][W];
    __shared__ T s_piv[W];
    __shared__ T red_v[LU_THREADS / 32];
    __shared__ int red_i[LU_THREADS / 32];
    __shared__ int s_p;
    __shared__ T s_gbest;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int row0 = rank * R;
    const int nloc = max(0, min(R, m - row0));
    for (int k = 0; k < W; ++k)
        for (int li = tid; li < nloc; li += LU_THREADS)
            pan[li * W + k] = k < w ? A[size_t(c0 + k) * size_t(lda) + size_t(c0 + row0 + li)] : T(0);
    __syncthreads();
    for (int j = 0; j < w; ++j) {
        const int buf = j & 1;
        // 1. this CTA's candidate: the largest |a(i, j)| over its rows i >= j (smallest index on ties)
        T best = T(-1);
        int bi = INT_MAX;
        for (int li = tid; li < nloc; li += LU_THREADS) {
            int i = row0 + li;
            if (i >= j) {
                T v = fabs(pan[li * W + j]);
                if (v > best || (v == best && i < bi)) {
                    best = v;
                    bi = i;
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            T ov = __shfl_xor_sync(0xffffffffu, best, o);
            int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) {
                best = ov;
                bi = oi;
            }
        }
        if (lane == 0) {
            red_v[wid] = best;
            red_i[wid] = bi;
        }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < LU_THREADS / 32; ++w)
                if (red_v[w] > best || (red_v[w] == best && red_i[w] < bi)) {
                    best = red_v[w];
                    bi = red_i[w];
                }
            s_cval[buf] = best;
            s_cidx[buf] = bi;
            if (bi != INT_MAX)
                for (int k = 0; k < W; ++k) s_crow[buf][k] = pan[(bi - row0) * W + k];
            if (j >= row0 && j < row0 + nloc)
                for (int k = 0; k < W; ++k) s_rowj[buf][k] = pan[(j - row0) * W + k];
        }
        __syncthreads();
        cl.sync();
        // 2. the pivot over the cluster, its row, and the old row j
        if (tid == 0) {
            T gb = T(-1);
            int gi = INT_MAX;
            for (int r = 0; r < LU_CL; ++r) {
                T v = *cl.map_shared_rank(&s_cval[buf], r);
                int ix = *cl.map_shared_rank(&s_cidx[buf], r);
                if (ix != INT_MAX && (v > gb || (v == gb && ix < gi))) {
                    gb = v;
                    gi = ix;
                }
            }
            s_p = gi;
            s_gbest = gb;
        }
        __syncthreads();
        const int p = s_p;
        const bool zero = !(s_gbest > T(0)) || p == INT_MAX;
        if (zero) {
            if (rank == 0 && tid == 0) {
                if (*info == 0) *info = c0 + j + 1;
                ipiv[c0 + j] = c0 + j;
            }
        } else {
            const int cp = p / R, cj = j / R;
            if (tid < W) {
                T pv = *cl.map_shared_rank(&s_crow[buf][tid], cp);
                T rj = *cl.map_shared_rank(&s_rowj[buf][tid], cj);
                s_piv[tid] = pv;
                if (rank == cj) pan[(j - row0) * W + tid] = pv;
                if (rank == cp && p != j) pan[(p - row0) * W + tid] = rj;
            }
            if (rank == 0 && tid == 0) ipiv[c0 + j] = c0 + p;
            __syncthreads();
            // 3. eliminate below the pivot
            const T pj = s_piv[j];
            for (int li = tid; li < nloc; li += LU_THREADS) {
                int i = row0 + li;
                if (i > j) {
                    T l = pan[li * W + j] / pj;
                    pan[li * W + j] = l;
#pragma unroll
                    for (int k = 0; k < W; ++k)
                        if (k > j) pan[li * W + k] -= l * s_piv[k];
                }
            }
        }
        __syncthreads();
    }
    for (int k = 0; k < w; ++k)
        for (int li = tid; li < nloc; li += LU_THREADS)
            A[size_t(c0 + k) * size_t(lda) + size_t(c0 + row0 + li)] = pan[li * W + k];
    cl.sync();  // no CTA leaves while another may still read its shared memory
}

// apply the row swaps ipiv[j0..j1) (in order) to the columns [cs, ce). The swaps go in groups of 16: a group touches at
// most 32 rows (its own 16 and their partners), and one thread works out which row each of them ends up with; then a warp
// takes a column at a time, a lane a row: one load and one store, where a thread that swaps along its column waits for
// one swap after another (and reads a 32-byte sector per element).
constexpr int SWAP_G = 16, SWAP_WARPS = 8;
constexpr int PANEL_W = 64;  // columns of a panel that is factored leaf by leaf

// one warp: the rows that the ng swaps ipiv[g..g + ng) touch (g .. g + ng - 1 in places 0 .. ng - 1, then the partners
// outside that range, each once; -1 in the other places), and the row whose value each of them ends up with
__device__ __forceinline__ void swap_rows(const int* __restrict__ ipiv, int g, int ng, int lane, int* s_row, int* s_src,
                                          int* s_n) {
    const int p = lane < ng ? ipiv[g + lane] : -1;
    int row = lane < ng ? g + lane : -1, n = ng;
    for (int k = 0; k < ng; ++k) {
        const int pk = __shfl_sync(0xffffffffu, p, k);
        if (!__any_sync(0xffffffffu, row == pk)) {
            if (lane == n) row = pk;
            ++n;
        }
    }
    int src = row;
    for (int k = 0; k < ng; ++k) {
        const int pk = __shfl_sync(0xffffffffu, p, k);
        const int at = __ffs(__ballot_sync(0xffffffffu, row == pk)) - 1;
        const int a = __shfl_sync(0xffffffffu, src, k), b = __shfl_sync(0xffffffffu, src, at);
        if (lane == k) src = b;
        else if (lane == at) src = a;
    }
    s_row[lane] = row;
    s_src[lane] = src;
    if (lane == 0) *s_n = n;
}

template <class T>
__global__ void __launch_bounds__(32 * SWAP_WARPS) laswp_kernel(T* __restrict__ A, long long lda, int cs, int ce, int j0, int j1,
                                                              const int* __restrict__ ipiv) {
    __shared__ int s_row[2 * SWAP_G], s_src[2 * SWAP_G], s_n;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int g = j0; g < j1; g += SWAP_G) {
        const int ng = min(SWAP_G, j1 - g);
        if (w == 0) swap_rows(ipiv, g, ng, lane, s_row, s_src, &s_n);
        __syncthreads();
        const int row = s_row[lane], src = s_src[lane];
        const bool on = lane < s_n && src != row;
        for (int c = cs + blockIdx.x * SWAP_WARPS + w; c < ce; c += gridDim.x * SWAP_WARPS) {
            T* col = A + size_t(c) * size_t(lda);
            const T v = on ? col[src] : T(0);
            __syncwarp();
            if (on) col[row] = v;
            __syncwarp();
        }
        __syncthreads();
    }
}

// x(i, k) = b(perm[i], k) (forward) or x(perm[i], k) = b(i, k) (inverse); column-major n x nrhs
template <class T>
__global__ void permute_kernel(int n, int nrhs, const int* __restrict__ perm, int inverse, const T* __restrict__ b,
                               T* __restrict__ x) {
    size_t idx = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (idx >= size_t(n) * nrhs) return;
    int i = int(idx % n), k = int(idx / n);
    if (inverse)
        x[size_t(k) * n + perm[i]] = b[idx];
    else
        x[idx] = b[size_t(k) * n + perm[i]];
}

// rhs = [C' b; 0] for nrhs columns (b: nslot x nrhs column-major)
__global__ void ctb_kernel(int nq, int n, int nslot, int nrhs, const int* __restrict__ ctp, const int* __restrict__ cti,
                           const double* __restrict__ ctv, const double* __restrict__ b, double* __restrict__ rhs) {
    size_t idx = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (idx >= size_t(n) * nrhs) return;
    int q = int(idx % n), k = int(idx / n);
    double s = 0;
    if (q < nq)
        for (int u = ctp[q]; u < ctp[q + 1]; ++u) s += ctv[u] * b[size_t(k) * nslot + cti[u]];
    rhs[idx] = s;
}

template <class A_, class B_>
__global__ void convert_kernel(size_t n, const A_* __restrict__ a, B_* __restrict__ b) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        b[i] = B_(a[i]);
}

__global__ void axpy_f2d_kernel(size_t n, const float* __restrict__ d, double* __restrict__ x) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        x[i] += double(d[i]);
}

// ------------------------------------------------------------------------------------------------------------------
// host drivers

template <class T>
int gemm_sub(vp_ctx* ctx, int m, int n, int k, const T* A, int lda, const T* B, int ldb, T* C, int ldc);
template <>
int gemm_sub<double>(vp_ctx* ctx, int m, int n, int k, const double* A, int lda, const double* B, int ldb, double* C,
                     int ldc) {
    if (vp_tc_gemm_enabled() && vp_tc_gemm64_fits(m, n, k)) return vp_tc_gemm_sub64(ctx, m, n, k, A, lda, B, ldb, C, ldc);
    const double one = 1.0, mone = -1.0;
    VP_BLAS(ctx, cublasDgemm(ctx->blas, CUBLAS_OP_N, CUBLAS_OP_N, m, n, k, &mone, A, lda, B, ldb, &one, C, ldc));
    return VP_OK;
}
template <>
int gemm_sub<float>(vp_ctx* ctx, int m, int n, int k, const float* A, int lda, const float* B, int ldb, float* C,
                    int ldc) {
    // the trailing updates large enough for a 128 x 128 tile run on the tensor cores (three-piece bf16 split, FP32
    // accumulation in TMEM: FP32-class products); the small ones on cuBLAS
    if (vp_tc_gemm_enabled() && vp_tc_gemm_fits(m, n, k)) return vp_tc_gemm_sub(ctx, m, n, k, A, lda, B, ldb, C, ldc);
    const float one = 1.0f, mone = -1.0f;
    VP_BLAS(ctx, cublasSgemm(ctx->blas, CUBLAS_OP_N, CUBLAS_OP_N, m, n, k, &mone, A, lda, B, ldb, &one, C, ldc));
    return VP_OK;
}

template <class T>
int trsm(vp_ctx* ctx, cublasFillMode_t uplo, cublasOperation_t op, cublasDiagType_t diag, int m, int n, const T* A,
         int lda, T* B, int ldb);
template <>
int trsm<double>(vp_ctx* ctx, cublasFillMode_t uplo, cublasOperation_t op, cublasDiagType_t diag, int m, int n,
                 const double* A, int lda, double* B, int ldb) {
    const double one = 1.0;
    VP_BLAS(ctx, cublasDtrsm(ctx->blas, CUBLAS_SIDE_LEFT, uplo, op, diag, m, n, &one, A, lda, B, ldb));
    return VP_OK;
}
template <>
int trsm<float>(vp_ctx* ctx, cublasFillMode_t uplo, cublasOperation_t op, cublasDiagType_t diag, int m, int n,
                const float* A, int lda, float* B, int ldb) {
    const float one = 1.0f;
    VP_BLAS(ctx, cublasStrsm(ctx->blas, CUBLAS_SIDE_LEFT, uplo, op, diag, m, n, &one, A, lda, B, ldb));
    return VP_OK;
}

// X = L^-1 B for the factorization's unit lower triangle L (m x m), in place of B (m x n). FP64: recursive, so that the
// products go to gemm_sub (tensor cores); cuBLAS's DTRSM, at the FP64 pipe's rate, keeps the 64 x 64 diagonal blocks
template <class T>
int trsm_lower(vp_ctx* ctx, int m, int n, const T* L, int ldl, T* B, int ldb) {
    if (sizeof(T) == 4 || m <= 64 || !vp_tc_gemm64_fits(m, n, m / 2))
        return trsm<T>(ctx, CUBLAS_FILL_MODE_LOWER, CUBLAS_OP_N, CUBLAS_DIAG_UNIT, m, n, L, ldl, B, ldb);
    const int h = (m / 2 + 31) / 32 * 32;
    int r;
    if ((r = trsm_lower<T>(ctx, h, n, L, ldl, B, ldb))) return r;
    if ((r = gemm_sub<T>(ctx, m - h, n, h, L + h, ldl, B, ldb, B + h, ldb))) return r;
    return trsm_lower<T>(ctx, m - h, n, L + size_t(h) * ldl + h, ldl, B + h, ldb);
}

template <class T>
int leaf_width(int m) {
    // FP64: the widest leaf that a cluster of 16 holds in registers (16 columns up to 8,192 rows, 8 up to 16,384); else,
    // and in FP32, the widest whose panel fits the shared memory of 8 CTAs (200 KB each)
    int R = (m + LU_CL - 1) / LU_CL;
    if (sizeof(T) == 8 && m <= 32 * LU_THREADS) return m <= 16 * LU_THREADS ? 16 : 8;
    for (int w : {16, 8, 4})
        if (size_t(R) * w * sizeof(T) <= 200 * 1024) return w;
    return 0;
}

template <class T, int W>
int launch_leaf_tall(vp_ctx* ctx, T* A, int lda, int c0, int m, int w, int* ipiv, int* info) {
    int R = (m + LU_CL - 1) / LU_CL;
    size_t smem = size_t(R) * W * sizeof(T);
    if (smem > 227 * 1024) return vp_fail(ctx, VP_ERR_ARG, "LU leaf panel does not fit shared memory");
    VP_CUDA(ctx, cudaFuncSetAttribute(lu_leaf_tall_kernel<T, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    lu_leaf_tall_kernel<T, W><<<LU_CL, LU_THREADS, smem, ctx->stream>>>(A, lda, c0, m, w, R, ipiv, info);
    ctx->launches++;
    VP_CUDA(ctx, cudaGetLastError());
    return VP_OK;
}

// rows a thread holds at most: 32 words of panel a row pair fit its 128 registers
template <class T, int W>
constexpr int leaf_rpt_max = W * sizeof(T) <= 64 ? 2 : 1;

template <class T, int W, int RPT, int CL, int NT>
int launch_leaf_cl(vp_ctx* ctx, T* A, int lda, int c0, int m, int w, int* ipiv, int* info) {
    auto kern = lu_leaf_kernel<T, W, RPT, CL, NT>;
    const int R = (m + CL - 1) / CL, nt = std::min(NT, ((R + RPT - 1) / RPT + 31) / 32 * 32);
    if (CL > 8) VP_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(CL);
    cfg.blockDim = dim3(nt);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = CL;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    VP_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, A, (long long)lda, c0, m, w, R, ipiv, info));
    ctx->launches++;
    return VP_OK;
}

// whether the device places clusters of 16 CTAs (above the portable 8: 16 free SMs of one GPC) of this leaf kernel
template <class T, int W>
bool leaf16_fits(vp_ctx* ctx) {
    signed char& fits = ctx->leaf16[sizeof(T) == 4][W == 16 ? 0 : (W == 8 ? 1 : 2)];
    if (fits < 0) {
        auto kern = lu_leaf_kernel<T, W, leaf_rpt_max<T, W>, 16, LU_THREADS>;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(16);
        cfg.blockDim = dim3(LU_THREADS);
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = 16;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess;
        if (!ok) cudaGetLastError();  // the device does not take the size: not an error of the factorization
        fits = ok && n > 0;
    }
    return fits != 0;
}

// The smallest cluster that holds the panel, as fewer CTAs exchange faster: FP32, one CTA up to 1,024 rows, 8 CTAs up to
// 8,192, 16 (the largest) up to 16,384; FP64, whose elimination is bound by each SM's two FP64 operations a clock, one CTA
// up to 256 rows, 8 up to 2,048, then 16; the tall kernel beyond, and where clusters of 16 do not fit the device or are not
// allowed: 131 KB of shared memory a CTA at the most rows that 16 CTAs take, for every width.
template <class T, int W>
int launch_leaf(vp_ctx* ctx, T* A, int lda, int c0, int m, int w, int* ipiv, int* info) {
    if (w < 1 || w > W || w > m) return vp_fail(ctx, VP_ERR_ARG, "LU leaf width out of range");
    constexpr int RM = leaf_rpt_max<T, W>;
    if (ctx->lu_cluster < LU_CL) return launch_leaf_tall<T, W>(ctx, A, lda, c0, m, w, ipiv, info);
    if constexpr (sizeof(T) == 4) {
        if (m <= 1024) return launch_leaf_cl<T, W, 1, 1, 1024>(ctx, A, lda, c0, m, w, ipiv, info);
        if (m <= 8 * RM * LU_THREADS) return launch_leaf_cl<T, W, RM, 8, LU_THREADS>(ctx, A, lda, c0, m, w, ipiv, info);
    } else {
        if (m <= 256) return launch_leaf_cl<T, W, 1, 1, 256>(ctx, A, lda, c0, m, w, ipiv, info);
        if (m <= 2048) return launch_leaf_cl<T, W, 1, 8, 256>(ctx, A, lda, c0, m, w, ipiv, info);
    }
    if (m <= 16 * RM * LU_THREADS && ctx->lu_cluster >= 16 && leaf16_fits<T, W>(ctx))
        return launch_leaf_cl<T, W, RM, 16, LU_THREADS>(ctx, A, lda, c0, m, w, ipiv, info);
    return launch_leaf_tall<T, W>(ctx, A, lda, c0, m, w, ipiv, info);
}

// factor a leaf of w columns with the smallest kernel instance that holds it
template <class T>
int leaf(vp_ctx* ctx, T* A, int lda, int c0, int w, int m, int* ipiv, int* info) {
    if (w > 8) return launch_leaf<T, 16>(ctx, A, lda, c0, m, w, ipiv, info);
    if (w > 4) return launch_leaf<T, 8>(ctx, A, lda, c0, m, w, ipiv, info);
    return launch_leaf<T, 4>(ctx, A, lda, c0, m, w, ipiv, info);
}

__global__ void iota_kernel(int n, int* __restrict__ a) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = i;
}

template <class T>
int laswp(vp_ctx* ctx, T* A, int lda, int cs, int ce, int j0, int j1, const int* ipiv) {
    if (ce <= cs || j1 <= j0) return VP_OK;
    int nc = ce - cs;
    laswp_kernel<T><<<std::min((nc + SWAP_WARPS - 1) / SWAP_WARPS, 8 * ctx->nsm), 32 * SWAP_WARPS, 0, ctx->stream>>>(
        A, lda, cs, ce, j0, j1, ipiv);
    ctx->launches++;
    VP_CUDA(ctx, cudaGetLastError());
    return VP_OK;
}

// After a leaf of the columns [j0, j1) inside the panel [c0, c1): its row swaps on the panel's other columns and, for those
// to its right, U = L^-1 A of the leaf's rows (L: its unit lower triangle). A warp takes a column, a lane one of the at
// most 32 rows that the swaps touch (as laswp_kernel); the first j1 - j0 lanes then hold the column's leaf rows and solve
// by shuffles.
template <class T>
__global__ void __launch_bounds__(32 * SWAP_WARPS) panel_swap_kernel(T* __restrict__ A, long long lda, int c0, int c1, int j0,
                                                                   int j1, const int* __restrict__ ipiv) {
    __shared__ int s_row[2 * SWAP_G], s_src[2 * SWAP_G], s_n;
    __shared__ T s_L[SWAP_G][SWAP_G + 1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, ng = j1 - j0;
    if (w == 0) swap_rows(ipiv, j0, ng, lane, s_row, s_src, &s_n);
    for (int e = threadIdx.x; e < ng * ng; e += blockDim.x) {
        const int i = e % ng, k = e / ng;
        s_L[i][k] = i > k ? A[size_t(j0 + k) * size_t(lda) + j0 + i] : T(0);
    }
    __syncthreads();
    const int row = s_row[lane], src = s_src[lane];
    const bool on = lane < s_n;
    for (int q = blockIdx.x * SWAP_WARPS + w; q < c1 - c0 - ng; q += gridDim.x * SWAP_WARPS) {
        const int c = c0 + q < j0 ? c0 + q : c0 + q + ng;
        T* col = A + size_t(c) * size_t(lda);
        T v = on ? col[src] : T(0);
        if (c >= j1)
            for (int k = 0; k < ng; ++k) {
                const T x = __shfl_sync(0xffffffffu, v, k);
                if (lane > k && lane < ng) v -= s_L[lane][k] * x;
            }
        __syncwarp();
        if (on) col[row] = v;
        __syncwarp();
    }
}

// C -= L U for the panel's columns [j1, c1) and the rows below the leaf: L = A(j1.., j0..j1), U = A(j0..j1, j1..c1). A thread
// takes a row: its ng values of L in registers, U in shared memory; the row's columns are read and written once.
template <class T>
__global__ void __launch_bounds__(128) panel_update_kernel(T* __restrict__ A, long long lda, int n, int c1, int j0, int j1) {
    __shared__ T s_U[PANEL_W][SWAP_G];
    const int ng = j1 - j0, nc = c1 - j1;
    for (int e = threadIdx.x; e < nc * SWAP_G; e += blockDim.x) {
        const int k = e % SWAP_G, c = e / SWAP_G;
        s_U[c][k] = k < ng ? A[size_t(j1 + c) * size_t(lda) + j0 + k] : T(0);
    }
    const int i = j1 + blockIdx.x * blockDim.x + threadIdx.x;
    T l[SWAP_G];
#pragma unroll
    for (int k = 0; k < SWAP_G; ++k) l[k] = k < ng && i < n ? A[size_t(j0 + k) * size_t(lda) + i] : T(0);
    __syncthreads();
    if (i >= n) return;
    // blockIdx.y: every gridDim.y-th column
    for (int c = blockIdx.y; c < nc; c += gridDim.y) {
        T* x = A + size_t(j1 + c) * size_t(lda) + i;
        T v = T(0);
#pragma unroll
        for (int k = 0; k < SWAP_G; ++k) v += l[k] * s_U[c][k];
        *x -= v;
    }
}

// LU of a panel of at most PANEL_W columns [c0, c0 + w): leaf by leaf, each followed by its swaps, triangular solve and
// update inside the panel. Three launches a leaf of 16 columns, where the recursion down to leaves takes a leaf, two row
// swap kernels, a cuBLAS TRSM and a cuBLAS GEMM (of 28 us each at 6,600 rows). With the leaf's exchange by mbarriers: LU
// 99.6 -> 75.3 ms at 6.6k unknowns FP64, 78 -> 68 at 12.8k mixed, 4.4 -> 3.2 at 643 FP64.
template <class T>
int panel(vp_ctx* ctx, T* A, int n, int c0, int w, int lw, int* ipiv, int* info) {
    const int c1 = c0 + w;
    int r;
    for (int j0 = c0; j0 < c1; j0 += lw) {
        const int j1 = std::min(j0 + lw, c1);
        if ((r = leaf<T>(ctx, A, n, j0, j1 - j0, n - j0, ipiv, info))) return r;
        if (w == j1 - j0) break;
        panel_swap_kernel<T><<<(w - (j1 - j0) + SWAP_WARPS - 1) / SWAP_WARPS, 32 * SWAP_WARPS, 0, ctx->stream>>>(A, n, c0, c1,
                                                                                                                j0, j1, ipiv);
        ctx->launches++;
        if (j1 < c1 && j1 < n) {
            const int gx = (n - j1 + 127) / 128, gy = std::max(1, std::min(c1 - j1, 4 * ctx->nsm / gx));
            panel_update_kernel<T><<<dim3(gx, gy), 128, 0, ctx->stream>>>(A, n, n, c1, j0, j1);
            ctx->launches++;
        }
    }
    VP_CUDA(ctx, cudaGetLastError());
    return VP_OK;
}

// recursive LU of the columns [c0, c0 + w) (rows c0..n-1)
template <class T>
int rgetrf(vp_ctx* ctx, T* A, int n, int c0, int w, int lw, int* ipiv, int* info) {
    int r;
    if (w <= PANEL_W) return panel<T>(ctx, A, n, c0, w, lw, ipiv, info);
    int w1 = ((w / 2 + PANEL_W - 1) / PANEL_W) * PANEL_W;
    if (w1 >= w) w1 = w - PANEL_W;
    int w2 = w - w1;
    if ((r = rgetrf<T>(ctx, A, n, c0, w1, lw, ipiv, info))) return r;
    if ((r = laswp<T>(ctx, A, n, c0 + w1, c0 + w, c0, c0 + w1, ipiv))) return r;
    if ((r = trsm_lower<T>(ctx, w1, w2, A + size_t(c0) * n + c0, n, A + size_t(c0 + w1) * n + c0, n))) return r;
    if (n - c0 - w1 > 0 &&
        (r = gemm_sub<T>(ctx, n - c0 - w1, w2, w1, A + size_t(c0) * n + (c0 + w1), n, A + size_t(c0 + w1) * n + c0, n,
                         A + size_t(c0 + w1) * n + (c0 + w1), n)))
        return r;
    if ((r = rgetrf<T>(ctx, A, n, c0 + w1, w2, lw, ipiv, info))) return r;
    return laswp<T>(ctx, A, n, c0, c0 + w1, c0 + w1, c0 + w, ipiv);
}

// out[2 k], out[2 k + 1] = the largest |r|, |x| of column k (n rows): one CTA a column, all columns in one launch and one
// copy to the host (cuBLAS IDAMAX and two copies a column, each with its synchronization, took 60 us a column)
__global__ void __launch_bounds__(512) col_max_kernel(int n, const double* __restrict__ r, const double* __restrict__ x,
                                                      double* __restrict__ out) {
    __shared__ unsigned long long s_m[2][16];
    const size_t o = size_t(blockIdx.x) * n;
    unsigned long long m[2] = {0, 0};
    for (int i = threadIdx.x; i < n; i += 512) {
        m[0] = max(m[0], mag_key(r[o + i]));
        m[1] = max(m[1], mag_key(x[o + i]));
    }
    for (int d = 16; d; d >>= 1)
        for (int k = 0; k < 2; ++k) m[k] = max(m[k], __shfl_xor_sync(0xffffffffu, m[k], d));
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 2; ++k) s_m[k][threadIdx.x >> 5] = m[k];
    __syncthreads();
    if (threadIdx.x < 2) {
        unsigned long long v = 0;
        for (int w = 0; w < 16; ++w) v = max(v, s_m[threadIdx.x][w]);
        out[2 * size_t(blockIdx.x) + threadIdx.x] = __longlong_as_double((long long)v);
    }
}

// solve with the factors: op = N: M x = b; op = T: M' x = b (b, x: n x nrhs column-major, device; may alias)
template <class T>
int lu_solve(vp_ctx* ctx, const vp_factor* F, const T* LU, const int* d_perm, int nrhs, T* b, T* work, bool trans) {
    int n = F->n, r;
    size_t tot = size_t(n) * nrhs;
    int nb = int((tot + 255) / 256);
    if (!trans) {
        permute_kernel<T><<<nb, 256, 0, ctx->stream>>>(n, nrhs, d_perm, 0, b, work);
        ctx->launches++;
        if ((r = trsm<T>(ctx, CUBLAS_FILL_MODE_LOWER, CUBLAS_OP_N, CUBLAS_DIAG_UNIT, n, nrhs, LU, n, work, n))) return r;
        if ((r = trsm<T>(ctx, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_N, CUBLAS_DIAG_NON_UNIT, n, nrhs, LU, n, work, n))) return r;
        VP_CUDA(ctx, cudaMemcpyAsync(b, work, sizeof(T) * tot, cudaMemcpyDeviceToDevice, ctx->stream));
    } else {
        if ((r = trsm<T>(ctx, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_T, CUBLAS_DIAG_NON_UNIT, n, nrhs, LU, n, b, n))) return r;
        if ((r = trsm<T>(ctx, CUBLAS_FILL_MODE_LOWER, CUBLAS_OP_T, CUBLAS_DIAG_UNIT, n, nrhs, LU, n, b, n))) return r;
        permute_kernel<T><<<nb, 256, 0, ctx->stream>>>(n, nrhs, d_perm, 1, b, work);
        ctx->launches++;
        VP_CUDA(ctx, cudaMemcpyAsync(b, work, sizeof(T) * tot, cudaMemcpyDeviceToDevice, ctx->stream));
    }
    VP_CUDA(ctx, cudaGetLastError());
    return VP_OK;
}

}  // namespace

int vp_lu_factor(vp_ctx* ctx, int precision, int n, double* M64, vp_factor* F) {
    int r;
    int* d_info;
    if ((r = vp_alloc(ctx, &d_info, 1))) return r;
    VP_CUDA(ctx, cudaMemsetAsync(d_info, 0, sizeof(int), ctx->stream));
    if ((r = vp_alloc(ctx, &F->ipiv, size_t(n)))) return r;
    iota_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(n, F->ipiv);  // every swap index valid from the start
    ctx->launches++;
    if (precision == VP_FP64) {
        if ((r = vp_alloc(ctx, &F->LU64, size_t(n) * n))) return r;
        VP_CUDA(ctx, cudaMemcpyAsync(F->LU64, M64, sizeof(double) * size_t(n) * n, cudaMemcpyDeviceToDevice, ctx->stream));
        int lw = leaf_width<double>(n);
        if (!lw) return vp_fail(ctx, VP_ERR_ARG, "matrix too large for the LU panel");
        r = rgetrf<double>(ctx, F->LU64, n, 0, n, lw, F->ipiv, d_info);
        if (!r) r = vp_tc_gemm_check(ctx);
    } else {
        if ((r = vp_alloc(ctx, &F->LU32, size_t(n) * n))) return r;
        convert_kernel<double, float><<<4 * ctx->nsm, 256, 0, ctx->stream>>>(size_t(n) * n, M64, F->LU32);
        ctx->launches++;
        int lw = leaf_width<float>(n);
        if (!lw) return vp_fail(ctx, VP_ERR_ARG, "matrix too large for the LU panel");
        r = rgetrf<float>(ctx, F->LU32, n, 0, n, lw, F->ipiv, d_info);
        if (!r) r = vp_tc_gemm_check(ctx);
    }
    if (r) {
        cudaFree(d_info);
        return r;
    }
    int info = 0;
    F->h_ipiv.resize(n);
    VP_CUDA(ctx, vp_d2h(ctx, &info, d_info, sizeof(int)));
    VP_CUDA(ctx, vp_d2h(ctx, F->h_ipiv.data(), F->ipiv, sizeof(int) * n));
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    cudaFree(d_info);
    if (e != cudaSuccess) return vp_fail(ctx, VP_ERR_CUDA, std::string("LU: ") + cudaGetErrorString(e));
    if (info < 0) return vp_fail(ctx, VP_ERR_TIMEOUT, "LU leaf: a bounded wait gave up");
    if (info > 0) return vp_fail(ctx, VP_ERR_SINGULAR, "zero pivot in column " + std::to_string(info));
    return VP_OK;
}

// ------------------------------------------------------------------------------------------------------------------

static int solve_core(vp_ctx* ctx, const vp_factor* F, int nrhs, double* x, bool trans, int* iters,
                      SolveWork* ws = nullptr);

extern "C" int vp_factorize(vp_ctx* ctx, const vp_system* sys, int precision, int nq, const int* C_rowptr,
                            const int* C_col, const double* C_val, int nwake, const int* W_rowptr, const int* W_col,
                            const double* W_val, int nbody, const int* q_body, const double* slot_area,
                            const int* slot_body, vp_factor** out, double* cond) {
    if (!ctx || !sys || !C_rowptr || !C_col || !C_val || !out || !q_body || !slot_area || !slot_body)
        return vp_fail(ctx, VP_ERR_ARG, "null argument");
    *out = nullptr;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return vp_fail(ctx, VP_ERR_CUDA, "cudaSetDevice");
    if (precision != VP_FP64 && precision != VP_MIXED) return vp_fail(ctx, VP_ERR_ARG, "unknown precision");
    const int nslot = sys->nslot;
    if (nwake != sys->nwnode)
        return vp_fail(ctx, VP_ERR_ARG, "A is " + std::to_string(nslot) + "x" + std::to_string(sys->ncols) +
                                            ", expected " + std::to_string(nslot) + "x" + std::to_string(nslot + nwake));
    if (nq <= 0 || nbody < 0) return vp_fail(ctx, VP_ERR_ARG, "nq must be positive");
    // C' and Cf' = [C; W]' as CSR over the unknowns
    std::vector<std::vector<std::pair<int, double>>> ct(nq), cft(nq);
    for (int i = 0; i < nslot; ++i)
        for (int u = C_rowptr[i]; u < C_rowptr[i + 1]; ++u) {
            int q = C_col[u];
            if (q < 0 || q >= nq) return vp_fail(ctx, VP_ERR_ARG, "C column out of range");
            ct[q].push_back({i, C_val[u]});
            cft[q].push_back({i, C_val[u]});
        }
    for (int i = 0; i < nwake; ++i)
        for (int u = W_rowptr[i]; u < W_rowptr[i + 1]; ++u) {
            int q = W_col[u];
            if (q < 0 || q >= nq) return vp_fail(ctx, VP_ERR_ARG, "W column out of range");
            cft[q].push_back({nslot + i, W_val[u]});
        }
    auto csr = [](const std::vector<std::vector<std::pair<int, double>>>& rows, std::vector<int>& p, std::vector<int>& c,
                  std::vector<double>& v) {
        p.assign(1, 0);
        for (auto& r : rows) {
            for (auto& e : r) {
                c.push_back(e.first);
                v.push_back(e.second);
            }
            p.push_back((int)c.size());
        }
        if (c.empty()) {
            c.push_back(0);
            v.push_back(0);
        }
    };
    std::vector<int> ctp, cti, cfp, cfi;
    std::vector<double> ctv, cfv;
    csr(ct, ctp, cti, ctv);
    csr(cft, cfp, cfi, cfv);
    const int nb = nbody;
    const int n = nq + nb;
    vp_factor* F = new vp_factor();
    F->n = n;
    F->nq = nq;
    F->nb = nb;
    F->nslot = nslot;
    F->ncols = sys->ncols;
    F->precision = precision;
    int r;
    auto fail = [&](int code) {
        vp_factor_free(F);
        return code;
    };
    int *d_cfp, *d_cfi;
    double* d_cfv;
    if ((r = vp_upload(ctx, &F->Ct_ptr, ctp.data(), ctp.size())) || (r = vp_upload(ctx, &F->Ct_col, cti.data(), cti.size())) ||
        (r = vp_upload(ctx, &F->Ct_val, ctv.data(), ctv.size())))
        return fail(r);
    if ((r = vp_upload(ctx, &d_cfp, cfp.data(), cfp.size()))) return fail(r);
    if ((r = vp_upload(ctx, &d_cfi, cfi.data(), cfi.size()))) { cudaFree(d_cfp); return fail(r); }
    if ((r = vp_upload(ctx, &d_cfv, cfv.data(), cfv.size()))) { cudaFree(d_cfp); cudaFree(d_cfi); return fail(r); }
    if ((r = vp_alloc(ctx, &F->M, size_t(n) * n))) { cudaFree(d_cfp); cudaFree(d_cfi); cudaFree(d_cfv); return fail(r); }
    vp_phase_begin(ctx, PH_REDUCE);
    VP_CUDA(ctx, cudaMemsetAsync(F->M, 0, sizeof(double) * size_t(n) * n, ctx->stream));
    dim3 grid((nq + 31) / 32, (nq + 31) / 32), block(32, 8);
    reduce_kernel<<<grid, block, 0, ctx->stream>>>(nq, n, sys->A, sys->ncols, F->Ct_ptr, F->Ct_col, F->Ct_val, d_cfp,
                                                   d_cfi, d_cfv, F->M);
    ctx->launches++;
    VP_CUDA(ctx, cudaGetLastError());
    // border (bordered_matrix, solve.jl:23-38): scale = mean |diag|, e_k and c_k scaled to 2-norm = scale
    std::vector<double> diag(nq);
    vp_phase_end(ctx);
    VP_CUDA(ctx, cudaMemcpy2DAsync(diag.data(), sizeof(double), F->M, sizeof(double) * (size_t(n) + 1), sizeof(double), nq,
                                   cudaMemcpyDeviceToHost, ctx->stream));
    VP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    cudaFree(d_cfp);
    cudaFree(d_cfi);
    cudaFree(d_cfv);
    double scale = 0;
    for (double d : diag) scale += std::fabs(d);
    scale /= nq;
    F->h_se.assign(nb, 0.0);
    if (nb > 0) {
        std::vector<double> ecol(size_t(nb) * nq, 0.0), crow(size_t(nb) * nq, 0.0);
        for (int k = 0; k < nb; ++k) {
            double ne = 0, nc = 0;
            std::vector<double> c(nq, 0.0);
            for (int q = 0; q < nq; ++q) {
                if (q_body[q] == k + 1) ne += 1;
                for (auto& e : ct[q])
                    if (slot_body[e.first] == k + 1) c[q] += e.second * slot_area[e.first];
            }
            for (int q = 0; q < nq; ++q) nc += c[q] * c[q];
            ne = std::sqrt(ne);
            nc = std::sqrt(nc);
            if (!(ne > 0) || !(nc > 0)) return fail(vp_fail(ctx, VP_ERR_ARG, "a body has no unknowns"));
            F->h_se[k] = scale / ne;
            for (int q = 0; q < nq; ++q) {
                ecol[size_t(k) * nq + q] = q_body[q] == k + 1 ? F->h_se[k] : 0.0;
                crow[size_t(k) * nq + q] = c[q] * (scale / nc);
            }
        }
        double *d_e, *d_c;
        if ((r = vp_upload(ctx, &d_e, ecol.data(), ecol.size()))) return fail(r);
        if ((r = vp_upload(ctx, &d_c, crow.data(), crow.size()))) { cudaFree(d_e); return fail(r); }
        border_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(nq, n, nb, d_e, d_c, F->M);
        ctx->launches++;
        VP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        cudaFree(d_e);
        cudaFree(d_c);
    }
    // norms of M (1-norm for the condition estimate, inf-norm for the refinement test)
    {
        double* d_cs;
        if ((r = vp_alloc(ctx, &d_cs, size_t(n)))) return fail(r);
        col_abs_sum_kernel<double><<<n, 256, 0, ctx->stream>>>(n, F->M, d_cs);
        ctx->launches++;
        std::vector<double> cs(n);
        VP_CUDA(ctx, vp_d2h(ctx, cs.data(), d_cs, sizeof(double) * n));
        VP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        cudaFree(d_cs);
        F->norm1 = *std::max_element(cs.begin(), cs.end());
    }
    vp_phase_begin(ctx, PH_LU);
    r = vp_lu_factor(ctx, precision, n, F->M, F);
    vp_phase_end(ctx);
    if (r) return fail(r);
    // permutation from the sequential swaps
    std::vector<int> perm(n);
    for (int i = 0; i < n; ++i) perm[i] = i;
    for (int j = 0; j < n; ++j) std::swap(perm[j], perm[F->h_ipiv[j]]);
    if ((r = vp_upload(ctx, &F->perm, perm.data(), perm.size()))) return fail(r);
    if (!F->h_se.empty() && (r = vp_upload(ctx, &F->se, F->h_se.data(), F->h_se.size()))) return fail(r);
    // 1-norm condition estimate (LAPACK dgecon / dlacn2: Hager's method with Higham's refinements)
    {
        vp_phase_begin(ctx, PH_COND);
        std::vector<double> hx(n), hy(n);
        double *dx;
        if ((r = vp_alloc(ctx, &dx, size_t(n)))) return fail(r);
        auto solve1 = [&](bool trans) -> int {
            VP_CUDA(ctx, vp_h2d(ctx, dx, hx.data(), sizeof(double) * n));
            int rr = solve_core(ctx, F, 1, dx, trans, nullptr);
            if (rr) return rr;
            VP_CUDA(ctx, vp_d2h(ctx, hy.data(), dx, sizeof(double) * n));
            VP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            return VP_OK;
        };
        auto sgn = [](double v) { return v >= 0 ? 1.0 : -1.0; };
        for (int i = 0; i < n; ++i) hx[i] = 1.0 / n;
        if ((r = solve1(false))) { cudaFree(dx); return fail(r); }
        double est = 0;
        for (double v : hy) est += std::fabs(v);
        std::vector<double> xi(n);
        for (int i = 0; i < n; ++i) xi[i] = sgn(hy[i]);
        hx = xi;
        if ((r = solve1(true))) { cudaFree(dx); return fail(r); }
        int jmax = 0;
        for (int i = 1; i < n; ++i)
            if (std::fabs(hy[i]) > std::fabs(hy[jmax])) jmax = i;
        for (int iter = 2; iter <= 5; ++iter) {
            std::fill(hx.begin(), hx.end(), 0.0);
            hx[jmax] = 1.0;
            if ((r = solve1(false))) { cudaFree(dx); return fail(r); }
            double old = est;
            est = 0;
            for (double v : hy) est += std::fabs(v);
            bool same = true;
            for (int i = 0; i < n && same; ++i) same = sgn(hy[i]) == xi[i];
            if (same || est <= old) break;
            for (int i = 0; i < n; ++i) xi[i] = sgn(hy[i]);
            hx = xi;
            if ((r = solve1(true))) { cudaFree(dx); return fail(r); }
            int jlast = jmax;
            jmax = 0;
            for (int i = 1; i < n; ++i)
                if (std::fabs(hy[i]) > std::fabs(hy[jmax])) jmax = i;
            if (std::fabs(hy[jlast]) == std::fabs(hy[jmax])) break;
        }
        double altsgn = 1;
        for (int i = 0; i < n; ++i) {
            hx[i] = altsgn * (1.0 + double(i) / std::max(n - 1, 1));
            altsgn = -altsgn;
        }
        if ((r = solve1(false))) { cudaFree(dx); return fail(r); }
        double temp = 0;
        for (double v : hy) temp += std::fabs(v);
        temp = 2 * temp / (3.0 * n);
        if (temp > est) est = temp;
        cudaFree(dx);
        vp_phase_end(ctx);
        F->cond = est * F->norm1;
    }
    if (cond) *cond = F->cond;
    *out = F;
    return VP_OK;
}

int vp_solve_work_alloc(vp_ctx* ctx, const vp_factor* F, SolveWork* w) {
    const size_t n = size_t(F->n);
    int r;
    w->n = F->n;
    if ((r = vp_alloc(ctx, &w->work64, n)) || (r = vp_alloc(ctx, &w->rhs, n)) || (r = vp_alloc(ctx, &w->res, n)) ||
        (r = vp_alloc(ctx, &w->f, n)) || (r = vp_alloc(ctx, &w->fw, n)) || (r = vp_alloc(ctx, &w->norms, 2))) {
        vp_solve_work_free(w);
        return r;
    }
    return VP_OK;
}

void vp_solve_work_free(SolveWork* w) {
    cudaFree(w->work64);
    cudaFree(w->rhs);
    cudaFree(w->res);
    cudaFree(w->f);
    cudaFree(w->fw);
    cudaFree(w->norms);
    *w = SolveWork();
}

// solve in place (x holds the right hand side on entry); VP_MIXED refines with FP64 residuals of M. With ws (one
// right hand side) its buffers are used and nothing is allocated.
static int solve_core(vp_ctx* ctx, const vp_factor* F, int nrhs, double* x, bool trans, int* iters, SolveWork* ws) {
    const int n = F->n;
    const int* d_perm = F->perm;
    const double norm1 = F->norm1;
    const size_t tot = size_t(n) * nrhs;
    int r;
    if (ws && (nrhs != 1 || ws->n != n)) return vp_fail(ctx, VP_ERR_ARG, "solve workspace does not fit");
    if (F->precision == VP_FP64) {
        double* work;
        if (ws) {
            work = ws->work64;
        } else if ((r = vp_alloc(ctx, &work, tot))) {
            return r;
        }
        r = lu_solve<double>(ctx, F, F->LU64, d_perm, nrhs, x, work, trans);
        if (!ws) cudaFree(work);
        if (iters) *iters = 1;
        return r;
    }
    // mixed: x0 = LU32^-1 rhs; r = rhs - M x; x += LU32^-1 r until the residual is at FP64 rounding level
    double *rhs, *res, *norms;
    float *f, *fw;
    if (ws) {
        norms = ws->norms;
        rhs = ws->rhs;
        res = ws->res;
        f = ws->f;
        fw = ws->fw;
    } else {
        if ((r = vp_alloc(ctx, &rhs, tot))) return r;
        if ((r = vp_alloc(ctx, &res, tot))) { cudaFree(rhs); return r; }
        if ((r = vp_alloc(ctx, &f, tot))) { cudaFree(rhs); cudaFree(res); return r; }
        if ((r = vp_alloc(ctx, &fw, tot))) { cudaFree(rhs); cudaFree(res); cudaFree(f); return r; }
        if ((r = vp_alloc(ctx, &norms, 2 * size_t(nrhs)))) { cudaFree(rhs); cudaFree(res); cudaFree(f); cudaFree(fw); return r; }
    }
    auto cleanup = [&]() {
        if (ws) return;
        cudaFree(rhs);
        cudaFree(res);
        cudaFree(f);
        cudaFree(fw);
        cudaFree(norms);
    };
    VP_CUDA(ctx, cudaMemcpyAsync(rhs, x, sizeof(double) * tot, cudaMemcpyDeviceToDevice, ctx->stream));
    int g = std::min<int>(4 * ctx->nsm, int((tot + 255) / 256));
    convert_kernel<double, float><<<g, 256, 0, ctx->stream>>>(tot, rhs, f);
    ctx->launches++;
    if ((r = lu_solve<float>(ctx, F, F->LU32, d_perm, nrhs, f, fw, trans))) { cleanup(); return r; }
    convert_kernel<float, double><<<g, 256, 0, ctx->stream>>>(tot, f, x);
    ctx->launches++;
    const double one = 1.0, mone = -1.0;
    const cublasOperation_t op = trans ? CUBLAS_OP_T : CUBLAS_OP_N;
    std::vector<double> mx(2 * size_t(nrhs));
    int it = 0;
    bool conv = false, lost = false;
    double prev = INFINITY;
    // columns whose right hand side holds an infinity or NaN: their solutions do too, as in VP_FP64, and the others go on
    // without them. Looked for once, when a column's numbers are not finite.
    std::vector<char> skip;
    auto not_finite = [&](int k) { return !std::isfinite(mx[2 * size_t(k)]) || !std::isfinite(mx[2 * size_t(k) + 1]); };
    auto find_skipped = [&]() -> int {
        std::vector<double> m(2 * size_t(nrhs));
        col_max_kernel<<<nrhs, 512, 0, ctx->stream>>>(n, rhs, rhs, norms);
        ctx->launches++;
        VP_CUDA(ctx, vp_d2h(ctx, m.data(), norms, sizeof(double) * 2 * nrhs));
        VP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        skip.assign(nrhs, 0);
        for (int k = 0; k < nrhs; ++k) skip[k] = !std::isfinite(m[2 * size_t(k)]);
        return VP_OK;
    };
    for (it = 1; it <= 30; ++it) {
        VP_CUDA(ctx, cudaMemcpyAsync(res, rhs, sizeof(double) * tot, cudaMemcpyDeviceToDevice, ctx->stream));
        // one product on the tensor cores (nine-digit FP64) from RES_TC columns on, below and for M' a matrix-vector product
        // per column: each reads M once at the HBM rate (a DGEMM with a few columns takes a tile shape that reads it far
        // slower, with many it runs at the FP64 pipe's rate)
        const bool tc = nrhs >= RES_TC && !trans && vp_tc_gemm_enabled() && n >= 1024;
        if (tc && (r = vp_tc_gemm_sub64(ctx, n, nrhs, n, F->M, n, x, n, res, n))) { cleanup(); return r; }
        for (int k = 0; k < nrhs && !tc; ++k)
            VP_BLAS(ctx, cublasDgemv(ctx->blas, op, n, n, &mone, F->M, n, x + size_t(k) * n, 1, &one,
                                     res + size_t(k) * n, 1));
        // convergence: every column's residual at FP64 rounding of |M| |x|
        col_max_kernel<<<nrhs, 512, 0, ctx->stream>>>(n, res, x, norms);
        ctx->launches++;
        VP_CUDA(ctx, vp_d2h(ctx, mx.data(), norms, sizeof(double) * 2 * nrhs));
        if (tc && (r = vp_tc_gemm_check(ctx))) { cleanup(); return r; }
        VP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        bool ok = true;
        double worst = 0;
        for (int k = 0; k < nrhs; ++k) {
            if (not_finite(k)) {
                if (skip.empty() && (r = find_skipped())) { cleanup(); return r; }
                if (skip[k]) continue;
                lost = true;  // an overflow of the FP32 factors or solves: more steps do not bring it back
            }
            const double ratio = mx[2 * size_t(k)] / (norm1 * mx[2 * size_t(k) + 1] + 1e-300);
            worst = std::max(worst, ratio);
            if (!(ratio <= 4 * std::sqrt(double(n)) * 1.1102230246251565e-16)) ok = false;
        }
        if (lost) break;
        if (ok) {
            conv = true;
            break;
        }
        if (it > 3 && worst > 0.5 * prev) break;  // stagnation
        prev = worst;
        convert_kernel<double, float><<<g, 256, 0, ctx->stream>>>(tot, res, f);
        ctx->launches++;
        if ((r = lu_solve<float>(ctx, F, F->LU32, d_perm, nrhs, f, fw, trans))) { cleanup(); return r; }
        axpy_f2d_kernel<<<g, 256, 0, ctx->stream>>>(tot, f, x);
        ctx->launches++;
    }
    cleanup();
    if (iters) *iters = it;
    if (lost) return vp_fail(ctx, VP_ERR_NOCONV, "iterative refinement: a solution overflowed FP32");
    if (!conv) {
        // stagnated at a level the FP32 factors cannot improve: accept when already tiny, else report
        return vp_fail(ctx, VP_ERR_NOCONV, "iterative refinement did not converge");
    }
    return VP_OK;
}

int vp_solve_dev(vp_ctx* ctx, const vp_factor* F, const double* d_b, double* d_x, SolveWork* w) {
    const int n = F->n;
    ctb_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(F->nq, n, F->nslot, 1, F->Ct_ptr, F->Ct_col, F->Ct_val, d_b, d_x);
    ctx->launches++;
    VP_CUDA(ctx, cudaGetLastError());
    return solve_core(ctx, F, 1, d_x, false, nullptr, w);
}

extern "C" int vp_solve(vp_ctx* ctx, const vp_factor* F, int nrhs, const double* b, double* q, double* lambda) {
    if (!ctx || !F || !b || !q || nrhs <= 0) return vp_fail(ctx, VP_ERR_ARG, "null argument");
    const int n = F->n, nq = F->nq, nb = F->nb, nslot = F->nslot;
    const size_t tot = size_t(n) * nrhs;
    int r;
    double *db, *x;
    if ((r = vp_alloc(ctx, &db, size_t(nslot) * nrhs))) return r;
    if ((r = vp_alloc(ctx, &x, tot))) { cudaFree(db); return r; }
    VP_CUDA(ctx, vp_h2d(ctx, db, b, sizeof(double) * size_t(nslot) * nrhs));
    ctb_kernel<<<int((tot + 255) / 256), 256, 0, ctx->stream>>>(nq, n, nslot, nrhs, F->Ct_ptr, F->Ct_col, F->Ct_val, db, x);
    ctx->launches++;
    vp_phase_begin(ctx, PH_SOLVE);
    r = solve_core(ctx, F, nrhs, x, false, nullptr);
    vp_phase_end(ctx);
    if (!r) {
        std::vector<double> hx(tot);
        vp_d2h(ctx, hx.data(), x, sizeof(double) * tot);
        cudaError_t e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) r = vp_fail(ctx, VP_ERR_CUDA, cudaGetErrorString(e));
        for (int k = 0; k < nrhs && !r; ++k) {
            for (int i = 0; i < nq; ++i) q[size_t(k) * nq + i] = hx[size_t(k) * n + i];
            if (lambda)
                for (int i = 0; i < nb; ++i) lambda[size_t(k) * nb + i] = F->h_se[i] * hx[size_t(k) * n + nq + i];
        }
    }
    cudaFree(db);
    cudaFree(x);
    return r;
}

// the adjoint's transposed solve: M' [xi; eta] = [g; 0]
extern "C" int vp_solve_transposed(vp_ctx* ctx, const vp_factor* F, int nrhs, const double* g, double* xi) {
    if (!ctx || !F || !g || !xi || nrhs <= 0) return vp_fail(ctx, VP_ERR_ARG, "null argument");
    if (cudaSetDevice(ctx->device) != cudaSuccess) return vp_fail(ctx, VP_ERR_CUDA, "cudaSetDevice");
    const int n = F->n, nq = F->nq;
    const size_t tot = size_t(n) * nrhs;
    std::vector<double> hx(tot, 0.0);
    for (int k = 0; k < nrhs; ++k)
        for (int i = 0; i < nq; ++i) hx[size_t(k) * n + i] = g[size_t(k) * nq + i];
    double* x;
    int r;
    if ((r = vp_upload(ctx, &x, hx.data(), tot))) return r;
    vp_phase_begin(ctx, PH_ADJ_SOLVE);
    r = solve_core(ctx, F, nrhs, x, true, nullptr);
    vp_phase_end(ctx);
    if (!r) {
        cudaError_t e = vp_d2h(ctx, hx.data(), x, sizeof(double) * tot);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) r = vp_fail(ctx, VP_ERR_CUDA, cudaGetErrorString(e));
        for (int k = 0; k < nrhs && !r; ++k)
            for (int i = 0; i < nq; ++i) xi[size_t(k) * nq + i] = hx[size_t(k) * n + i];
    }
    cudaFree(x);
    return r;
}

extern "C" int vp_solve_system(vp_ctx* ctx, const vp_factor* F, const vp_system* sys, double* q, double* lambda,
                               double* residual) {
    if (!ctx || !F || !sys) return vp_fail(ctx, VP_ERR_ARG, "null argument");
    if (sys->nslot != F->nslot) return vp_fail(ctx, VP_ERR_ARG, "system and factorization do not match");
    const int n = F->n, nq = F->nq, nb = F->nb;
    int r;
    double *x, *rhs;
    if ((r = vp_alloc(ctx, &x, size_t(n)))) return r;
    if ((r = vp_alloc(ctx, &rhs, size_t(n)))) { cudaFree(x); return r; }
    ctb_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(nq, n, F->nslot, 1, F->Ct_ptr, F->Ct_col, F->Ct_val, sys->b, x);
    ctx->launches++;
    VP_CUDA(ctx, cudaMemcpyAsync(rhs, x, sizeof(double) * n, cudaMemcpyDeviceToDevice, ctx->stream));
    vp_phase_begin(ctx, PH_SOLVE);
    r = solve_core(ctx, F, 1, x, false, nullptr);
    vp_phase_end(ctx);
    if (!r) {
        std::vector<double> hx(n);
        vp_d2h(ctx, hx.data(), x, sizeof(double) * n);
        if (residual) {
            double nr = 0, nrhs = 0;
            cublasDnrm2(ctx->blas, n, rhs, 1, &nrhs);
            const double one = 1.0, mone = -1.0;
            cublasDgemv(ctx->blas, CUBLAS_OP_N, n, n, &mone, F->M, n, x, 1, &one, rhs, 1);
            cublasDnrm2(ctx->blas, n, rhs, 1, &nr);
            *residual = nrhs > 0 ? nr / nrhs : nr;
        }
        cudaError_t e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) r = vp_fail(ctx, VP_ERR_CUDA, cudaGetErrorString(e));
        if (q)
            for (int i = 0; i < nq; ++i) q[i] = hx[i];
        if (lambda)
            for (int i = 0; i < nb; ++i) lambda[i] = F->h_se[i] * hx[nq + i];
    }
    cudaFree(x);
    cudaFree(rhs);
    return r;
}

extern "C" int vp_factor_info(const vp_factor* F, int* n, double* cond) {
    if (!F) return VP_ERR_ARG;
    if (n) *n = F->n;
    if (cond) *cond = F->cond;
    return VP_OK;
}

extern "C" void vp_factor_free(vp_factor* F) {
    if (!F) return;
    cudaFree(F->perm);
    cudaFree(F->M);
    cudaFree(F->LU64);
    cudaFree(F->LU32);
    cudaFree(F->ipiv);
    cudaFree(F->se);
    cudaFree(F->Ct_ptr);
    cudaFree(F->Ct_col);
    cudaFree(F->Ct_val);
    delete F;
}
