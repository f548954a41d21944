// Galerkin assembly on the GPU: assemble(g, dm, els, σ, V∞; opts, wake) of src/assembly/assemble.jl:377-447.
//
// A_ij = ∫ψ_i n·u[φ_j] dA, b_i = -∫ψ_i n·(V∞ + u_σ) dA over all (test, source) triangle pairs, each pair's 3x3 block
// and 3-vector computed with the quadrature tier of pair_rule (assemble.jl:266-282).
//
// Pipeline (one CUDA stream):
//   1. classification: for every test triangle, the sources that are NOT in the far tier (far test of
//      assemble.jl:269, FP32 with an exact FP64 fallback near the threshold), compacted in source order;
//   2. far tier: tile kernel, one CTA per tile of TT test triangles, one thread per source of a 128-source tile;
//      the far rule's points of the test tile sit in shared memory, each thread keeps its source in registers,
//      evaluates w analytically (FP32 with double-float offsets in VP_MIXED, FP64 in VP_FP64), contracts it into
//      the 3x3 hat block and gathers the tile's blocks into the slots of A in a fixed order. Test tiles are coloured
//      so that no two tiles of one launch share a row slot: the scatter needs no atomics and A is reproducible bit
//      for bit;
//   3. near, touching and contact tiers: the near pairs one per lane in chunks of 32, the others (self, edge, vertex
//      with wide-corner wedges, contact splits) one warp per pair with the reference's rules, all test triangles in one
//      launch each. Every pair's block goes to the pair's own place in a workspace, and one kernel adds the blocks to
//      A row by row, each column's in a fixed order. FP64 for the touching and contact tiers, FP32 or FP64 for the near
//      tier, FP64 for the wake's tip filaments.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>
#include <numeric>
#include <unordered_map>

#include "vp_pairs.cuh"

namespace {

// ------------------------------------------------------------------------------------------------------------------
// device: the far tier
template <class T, int TT>
__device__ __forceinline__ void far_body(const FarArgs& a, const int tile) {
    __shared__ FarTest<T> ts[TT];
    __shared__ T blk[TT][FAR_NT][9];
    __shared__ T rbsum[TT * 3][FAR_NT / 32];
    __shared__ int s_cols[3 * FAR_NT];
    __shared__ short s_cptr[3 * FAR_NT + 1];
    __shared__ short s_cent[3 * FAR_NT];
    __shared__ int s_rows[3 * TT];
    __shared__ short s_rptr[3 * TT + 1];
    __shared__ short s_rent[3 * TT];
    __shared__ int s_ncol, s_nrow;

    const int tid = threadIdx.x;
    // the test tile
    for (int i = tid; i < TT; i += FAR_NT) {
        int t = tile * TT + i;
        FarTest<T>& q = ts[i];
        q.valid = t < a.ntest;
        if (q.valid) {
            const TriGeo& g = a.tgeo[t];
            for (int p = 0; p < a.nq; ++p)
                for (int k = 0; k < 3; ++k) {
                    double x = a.tq[(size_t(t) * NQMAX + p) * 3 + k];
                    T h = T(x);
                    q.xh[p][k] = h;
                    q.xl[p][k] = T(x - double(h));
                    q.wpsi[p][k] = T(a.tw[(size_t(t) * NQMAX + p) * 3 + k]);
                }
            for (int k = 0; k < 3; ++k) {
                q.n[k] = T(g.n[k]);
                q.c64[k] = g.c[k];
            }
            q.diam64 = g.diam;
            q.cf = a.tcent[t];
        }
    }
    if (tid < 3 * TT) s_rows[tid] = a.trow[size_t(tile) * 3 * TT + tid];
    if (tid <= 3 * TT) s_rptr[tid] = a.trptr[size_t(tile) * (3 * TT + 1) + tid];
    if (tid < 3 * TT) s_rent[tid] = a.trent[size_t(tile) * 3 * TT + tid];
    if (tid == 0) s_nrow = a.tnrow[tile];
    __syncthreads();

    T rb[TT][3];
#pragma unroll
    for (int i = 0; i < TT; ++i) rb[i][0] = rb[i][1] = rb[i][2] = T(0);

    for (int set = 0; set < a.nset; ++set) {
        const T* soa = (const T*)a.soa[set];
        const int pad = a.pad[set];
        for (int st = 0; st < a.ntile[set]; ++st) {
            const int s = st * FAR_NT + tid;
            const bool sv = s < a.nsrc[set];
            // the source in registers
            SrcKern<T> S;
            v3<T> ch, cl, gam[3];
            T sig = T(0);
            CentF scf;
            if (sv) {
#define F(f) soa[size_t(f) * pad + s]
                ch = mk3(F(0), F(1), F(2));
                cl = mk3(F(3), F(4), F(5));
                S.diam = F(6);
                S.area = F(7);
                sig = F(8);
                for (int k = 0; k < 3; ++k) {
                    S.d[k] = mk3(F(9 + 3 * k), F(10 + 3 * k), F(11 + 3 * k));
                    S.nu[k] = mk3(F(18 + 3 * k), F(19 + 3 * k), F(20 + 3 * k));
                    S.len[k] = F(27 + k);
                    gam[k] = mk3(F(33 + 3 * k), F(34 + 3 * k), F(35 + 3 * k));
                }
                S.n = mk3(F(30), F(31), F(32));
#undef F
                scf = a.scent[set][s];
            }
#pragma unroll
            for (int i = 0; i < TT; ++i) {
                T out[9];
#pragma unroll
                for (int k = 0; k < 9; ++k) out[k] = T(0);
                const FarTest<T>& q = ts[i];
                bool far = false;
                if (sv && q.valid) {
                    int f = far_test32(q.cf, scf, a.ratio32);
                    if (f < 0) f = far_exact64(q.c64, q.diam64, a.sgeo[set][s].c, a.sgeo[set][s].diam, a.ratio);
                    far = f == 1;
                }
                if (far) {
                    v3<T> P[3] = {mk3(T(0), T(0), T(0)), mk3(T(0), T(0), T(0)), mk3(T(0), T(0), T(0))};
                    for (int p = 0; p < a.nq; ++p) {
                        v3<T> r = mk3((q.xh[p][0] - ch.x) + (q.xl[p][0] - cl.x), (q.xh[p][1] - ch.y) + (q.xl[p][1] - cl.y),
                                      (q.xh[p][2] - ch.z) + (q.xl[p][2] - cl.z));
                        v3<T> w = sv_rel(S, r, 0, T(a.kernel_far), T(1e-12));
                        P[0] += q.wpsi[p][0] * w;
                        P[1] += q.wpsi[p][1] * w;
                        P[2] += q.wpsi[p][2] * w;
                    }
                    v3<T> nT = mk3(q.n[0], q.n[1], q.n[2]);
                    if constexpr (sizeof(T) == 8) {  // P.(n x gam_b) = gam_b.(P x n), and the gam_b sum to zero
#pragma unroll
                        for (int aa = 0; aa < 3; ++aa) {
                            const v3<T> C = cross(P[aa], nT);
                            out[3 * aa] = dot(C, gam[0]);
                            out[3 * aa + 1] = dot(C, gam[1]);
                            out[3 * aa + 2] = -(out[3 * aa] + out[3 * aa + 1]);
                        }
                    } else {
#pragma unroll
                        for (int bb = 0; bb < 3; ++bb) {
                            v3<T> m = cross(nT, gam[bb]);
                            out[0 * 3 + bb] = dot(P[0], m);
                            out[1 * 3 + bb] = dot(P[1], m);
                            out[2 * 3 + bb] = dot(P[2], m);
                        }
                    }
                    rb[i][0] -= sig * dot(P[0], nT);
                    rb[i][1] -= sig * dot(P[1], nT);
                    rb[i][2] -= sig * dot(P[2], nT);
                }
#pragma unroll
                for (int k = 0; k < 9; ++k) blk[i][tid][k] = out[k];
            }
            // the source tile's unique columns
            const size_t tb = size_t(st);
            for (int k = tid; k < 3 * FAR_NT; k += FAR_NT) {
                s_cols[k] = a.tile_cols[set][tb * 3 * FAR_NT + k];
                s_cent[k] = a.tile_cent[set][tb * 3 * FAR_NT + k];
            }
            for (int k = tid; k <= 3 * FAR_NT; k += FAR_NT) s_cptr[k] = a.tile_cptr[set][tb * (3 * FAR_NT + 1) + k];
            if (tid == 0) s_ncol = a.tile_ncol[set][tb];
            __syncthreads();
            // gather into A in a fixed order: cell (r, c) = sum over the test corners of row r and the source corners
            // of column c; rows are this CTA's alone in this launch
            const int nrow = s_nrow, ncol = s_ncol;
            for (int cell = tid; cell < nrow * ncol; cell += FAR_NT) {
                int r = cell / ncol, c = cell - r * ncol;
                double acc = 0;
                for (int u = s_rptr[r]; u < s_rptr[r + 1]; ++u) {
                    int ti = s_rent[u] / 3, ta = s_rent[u] - 3 * ti;
                    T part = T(0);
                    for (int v = s_cptr[c]; v < s_cptr[c + 1]; ++v) {
                        int sj = s_cent[v] / 3, sb = s_cent[v] - 3 * sj;
                        part += blk[ti][sj][ta * 3 + sb];
                    }
                    acc += double(part);
                }
                double* dst = a.A + size_t(s_rows[r]) * size_t(a.lda) + a.col_off[set] + s_cols[c];
                *dst += acc;
            }
            __syncthreads();
        }
    }
    // right hand side: fixed-order block reduction of the per-thread partial sums
    const int lane = tid & 31, wid = tid >> 5;
#pragma unroll
    for (int i = 0; i < TT; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            T v = rb[i][k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) rbsum[i * 3 + k][wid] = v;
        }
    __syncthreads();
    if (tid < s_nrow) {
        double acc = 0;
        for (int u = s_rptr[tid]; u < s_rptr[tid + 1]; ++u) {
            T v = T(0);
            for (int w = 0; w < FAR_NT / 32; ++w) v += rbsum[s_rent[u]][w];
            acc += double(v);
        }
        a.b[s_rows[tid]] += acc;
    }
}

// one system: block b takes test tile a.tiles[b]
template <class T, int TT>
__global__ void __launch_bounds__(FAR_NT) far_kernel(FarArgs a) {
    far_body<T, TT>(a, a.tiles[blockIdx.x]);
}

// a batch of systems in one launch: block b takes test tile work[b].y of system work[b].x
template <class T, int TT>
__global__ void __launch_bounds__(FAR_NT) far_kernel_batch(const FarArgs* __restrict__ sys,
                                                          const int2* __restrict__ work) {
    const int2 wk = work[blockIdx.x];
    far_body<T, TT>(sys[wk.x], wk.y);
}

// ---- the near tier, one pair per lane ---------------------------------------------------------------------------
// A warp takes a chunk of up to 32 consecutive sources of its test triangle at once. Each lane decides its own pair's
// tier (exactly as pair_rule / wake_pair_rule) and, for a pair in the near tier, walks near_pieces' quadtree to its
// leaves. The warp then evaluates all leaves' points of the 32 pairs together, one point per lane (FP32, guarded;
// flagged points are queued and evaluated 32 at a time in FP64), reduces them per pair in a fixed order and writes
// each pair's block to the pair's place in blk. Pairs of the other tiers are appended to the rest list.
//
// Chunks are independent (nothing is added to A here), so a test triangle's chunks go to several warps and all test
// triangles to one launch. When one warp took a whole test triangle, one launch per colour, and added its blocks to A
// pair by pair, the kernel ran ~1 warp per SM on a 1,676-triangle wing (348 ms in FP64) and waited on a
// read-modify-write of A per pair.
struct NearChunkSh {
    NearPlanSh pl;         // the pairs' leaves and FP32 frames
    double acc[32][9];     // per pair: sum of W psi_a w (FP64 evaluations)
    float accf[32][9];     // per pair: the same sums of the FP32 evaluations
    int off[33];           // points before each pair
    int qp[64], qk[64];    // queued FP64 points (mixed): pair, point within the pair
    unsigned char nz[32];  // the pairs with points, in order
};

constexpr int BLK_B = 12, BLK_W = 9;  // doubles of a pair's block: body pairs carry their right hand side terms

// the FP64 evaluation of point k of pair p (queued by the FP32 guard): contributions in v
__device__ void near_point64(const NearArgs& a, const TriGeo& T, const TriGeo& S, const NearChunkSh& ns, int p, int k,
                             double* v) {
    const int nr = a.nrule[R_NEAR];
    int leaf = k / nr, q = k - leaf * nr;
    float bf[9];
    leaf_corners32(ns.pl.leaf[p][leaf], bf);
    double b[9];
    for (int z = 0; z < 9; ++z) b[z] = double(bf[z]);
    RulePt m = a.rule[R_NEAR][q];
    double l0 = m.l0 * b[0] + m.l1 * b[3] + m.l2 * b[6];
    double l1 = m.l0 * b[1] + m.l1 * b[4] + m.l2 * b[7];
    double l2 = m.l0 * b[2] + m.l1 * b[5] + m.l2 * b[8];
    int level = ns.pl.leaf[p][leaf] >> 6;
    double W = (m.w * ldexp(1.0, -2 * level)) * T.area;
    v3<double> x = mk3(l0 * T.x[0] + l1 * T.x[3] + l2 * T.x[6], l0 * T.x[1] + l1 * T.x[4] + l2 * T.x[7],
                       l0 * T.x[2] + l1 * T.x[5] + l2 * T.x[8]);
    v3<double> ra = mk3(l0 * (T.x[0] - S.x[0]) + l1 * (T.x[3] - S.x[0]) + l2 * (T.x[6] - S.x[0]),
                        l0 * (T.x[1] - S.x[1]) + l1 * (T.x[4] - S.x[1]) + l2 * (T.x[7] - S.x[1]),
                        l0 * (T.x[2] - S.x[2]) + l1 * (T.x[5] - S.x[2]) + l2 * (T.x[8] - S.x[2]));
    v3<double> rb = mk3(l0 * (T.x[0] - S.x[3]) + l1 * (T.x[3] - S.x[3]) + l2 * (T.x[6] - S.x[3]),
                        l0 * (T.x[1] - S.x[4]) + l1 * (T.x[4] - S.x[4]) + l2 * (T.x[7] - S.x[4]),
                        l0 * (T.x[2] - S.x[5]) + l1 * (T.x[5] - S.x[5]) + l2 * (T.x[8] - S.x[5]));
    v3<double> rc = mk3(l0 * (T.x[0] - S.x[6]) + l1 * (T.x[3] - S.x[6]) + l2 * (T.x[6] - S.x[6]),
                        l0 * (T.x[1] - S.x[7]) + l1 * (T.x[4] - S.x[7]) + l2 * (T.x[7] - S.x[7]),
                        l0 * (T.x[2] - S.x[8]) + l1 * (T.x[5] - S.x[8]) + l2 * (T.x[8] - S.x[8]));
    v3<double> r = x - ld3(S.c);
    SrcKern<double> K;
    for (int z = 0; z < 3; ++z) {
        K.d[z] = mk3(S.x[3 * z] - S.c[0], S.x[3 * z + 1] - S.c[1], S.x[3 * z + 2] - S.c[2]);
        K.nu[z] = ld3(S.nu + 3 * z);
        K.len[z] = S.len[z];
    }
    K.n = ld3(S.n);
    K.area = S.area;
    K.diam = S.diam;
    double fd = a.kernel_far * K.diam;
    v3<double> w = dot(r, r) > fd * fd ? sv_far(K, r) : sv_exact3(K, ra, rb, rc, r, 0, 1e-12);
    v3<double> psi = test_weights(a.test_mode, l0, l1, l2);
    double ps[3] = {W * psi.x, W * psi.y, W * psi.z};
    for (int ai = 0; ai < 3; ++ai) {
        v[3 * ai + 0] = ps[ai] * w.x;
        v[3 * ai + 1] = ps[ai] * w.y;
        v[3 * ai + 2] = ps[ai] * w.z;
    }
}

// FP64 path: the nr points of leaf `code` of a pair with frame E (x_T,k - v_S,a), summed: P[3a + z] = sum W psi_a w_z
__device__ __forceinline__ void near_leaf64(const NearArgs& a, const TriGeo& T, const TriGeo& S, const double* E, int code,
                                            double* P) {
    float bf[9];
    leaf_corners32(code, bf);
    double b[9];
    for (int z = 0; z < 9; ++z) b[z] = double(bf[z]);
    SrcKern<double> K;
    const v3<double> c = ld3(S.c);
    for (int z = 0; z < 3; ++z) {
        K.d[z] = ld3(S.x + 3 * z) - c;
        K.nu[z] = ld3(S.nu + 3 * z);
        K.len[z] = S.len[z];
    }
    K.n = ld3(S.n);
    K.area = S.area;
    K.diam = S.diam;
    const double fd = a.kernel_far * K.diam, fd2 = fd * fd, frac = ldexp(1.0, -2 * (code >> 6)) * T.area;
    const int nr = a.nrule[R_NEAR];
#pragma unroll 1
    for (int q = 0; q < nr; ++q) {
        const RulePt m = a.rule[R_NEAR][q];
        const double l0 = m.l0 * b[0] + m.l1 * b[3] + m.l2 * b[6];
        const double l1 = m.l0 * b[1] + m.l1 * b[4] + m.l2 * b[7];
        const double l2 = m.l0 * b[2] + m.l1 * b[5] + m.l2 * b[8];
        const v3<double> ra = l0 * ld3(E + 0) + l1 * ld3(E + 9) + l2 * ld3(E + 18);
        const v3<double> rb = l0 * ld3(E + 3) + l1 * ld3(E + 12) + l2 * ld3(E + 21);
        const v3<double> rc = l0 * ld3(E + 6) + l1 * ld3(E + 15) + l2 * ld3(E + 24);
        const v3<double> r = ra + K.d[0];
        const v3<double> w = dot(r, r) > fd2 ? sv_far(K, r) : sv_exact3(K, ra, rb, rc, r, 0, 1e-12);
        const v3<double> psi = test_weights(a.test_mode, l0, l1, l2);
        const double W = m.w * frac, ps[3] = {W * psi.x, W * psi.y, W * psi.z};
        for (int ai = 0; ai < 3; ++ai) {
            P[3 * ai + 0] += ps[ai] * w.x;
            P[3 * ai + 1] += ps[ai] * w.y;
            P[3 * ai + 2] += ps[ai] * w.z;
        }
    }
}

// list: the chunk's sources, p0 the first one's place in nf_src / wf_src; returns the lanes of the rest pairs
template <bool MIXED>
__device__ unsigned near_chunk(PairCtx& pc, NearChunkSh& ns, int t, const int* list, int cnt, bool wake, long long p0,
                               unsigned long long* P, unsigned long long* Q, unsigned long long& Q64) {
    const NearArgs& a = *pc.a;
    const TriGeo& T = *pc.T;
    const int lane = pc.lane;
    const unsigned FULL = 0xffffffffu;
    const bool valid = lane < cnt;
    const int s = valid ? list[lane] : 0;
    const TriGeo& S = wake ? a.wtri[s] : a.tri[s];
    int nleaf = 0;
    bool near = near_plan(pc, ns.pl, t, S, s, valid, wake, nleaf);
    for (int k = 0; k < 9; ++k) {
        ns.acc[lane][k] = 0.0;
        ns.accf[lane][k] = 0.f;
    }
    const int nr = a.nrule[R_NEAR];
    int incl = near ? nleaf * nr : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += y;
    }
    ns.off[lane + 1] = incl;
    if (lane == 0) ns.off[0] = 0;
    const int total = __shfl_sync(FULL, incl, 31);
    const unsigned nearmask = __ballot_sync(FULL, near);
    __syncwarp();
    // 3. every leaf point of the chunk, one per lane
    const float kf = float(a.kernel_far), areaT = float(T.area);
    const Fp32Guard g{PAIR_GUARD};
    int nq = 0;
    unsigned long long n64 = 0;
    if constexpr (!MIXED) {  // FP64: a lane takes a whole leaf, whose points' sums are added to the pair's once
        for (int i0 = 0; i0 < total; i0 += 32 * nr) {
            const int i = i0 + lane * nr;
            int p = 32 + lane;
            double P64[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            if (i < total) {
                int lo = 0, hi = 31;
                while (lo < hi) {
                    int mid = (lo + hi + 1) >> 1;
                    if (ns.off[mid] <= i) lo = mid;
                    else hi = mid - 1;
                }
                p = lo;
                near_leaf64(a, T, wake ? a.wtri[list[p]] : a.tri[list[p]], ns.pl.E64(p),
                            ns.pl.leaf[p][(i - ns.off[p]) / nr], P64);
            }
            seg_accumulate<9>(ns.accf, ns.acc, lane, p, P64);
        }
        n64 = (unsigned long long)total;
    }
    PointWalk wk{};
    if (MIXED) {
        wk = point_walk(incl - (near ? nleaf * nr : 0), near ? nleaf * nr : 0, lane, ns.nz);
        __syncwarp();
    }
    for (int i0 = 0; MIXED && i0 < total; i0 += 32) {
        const int i = i0 + lane;
        const bool v = i < total;
        const int pw = walk_point(wk, i0, lane, ns.nz);
        int p = 32 + lane, k = 0;
        float vals[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        bool need = false;
        if (v) {
            p = pw;
            k = i - ns.off[p];
            int leaf = k / nr, q = k - leaf * nr;
            int code = ns.pl.leaf[p][leaf];
            const float4 m = a.leafpt[leaf_node(code) * nr + q];
            const float l0 = m.x, l1 = m.y, l2 = m.z, W = m.w * areaT;
            const float* E = ns.pl.E32[p];
            const float* Dp = ns.pl.D32[p];
            const float* Sf = ns.pl.S32[p];
            SrcKern<float> K;
            for (int z = 0; z < 3; ++z) {
                K.d[z] = mk3(Sf[3 * z], Sf[3 * z + 1], Sf[3 * z + 2]);
                K.nu[z] = mk3(Sf[9 + 3 * z], Sf[10 + 3 * z], Sf[11 + 3 * z]);
                K.len[z] = Sf[18 + z];
            }
            K.n = mk3(Sf[21], Sf[22], Sf[23]);
            K.area = Sf[24];
            K.diam = Sf[25];
            v3<float> r = l0 * mk3(Dp[0], Dp[1], Dp[2]) + l1 * mk3(Dp[3], Dp[4], Dp[5]) + l2 * mk3(Dp[6], Dp[7], Dp[8]);
            v3<float> w;
            float fd = kf * K.diam;
            bool ok = true;
            if (dot(r, r) > fd * fd) {
                w = sv_far(K, r);
            } else {
                v3<float> ra = l0 * mk3(E[0], E[1], E[2]) + l1 * mk3(E[9], E[10], E[11]) + l2 * mk3(E[18], E[19], E[20]);
                v3<float> rb = l0 * mk3(E[3], E[4], E[5]) + l1 * mk3(E[12], E[13], E[14]) + l2 * mk3(E[21], E[22], E[23]);
                v3<float> rc = l0 * mk3(E[6], E[7], E[8]) + l1 * mk3(E[15], E[16], E[17]) + l2 * mk3(E[24], E[25], E[26]);
                ok = sv_exact3_guarded(K, ra, rb, rc, 0, g, w);
            }
            if (ok) {
                v3<float> psi = a.test_mode == 0 ? mk3(l0, l1, l2) : mk3(1.f, 1.f, 1.f);
                float ps[3] = {W * psi.x, W * psi.y, W * psi.z};
                for (int ai = 0; ai < 3; ++ai) {
                    vals[3 * ai + 0] = ps[ai] * w.x;
                    vals[3 * ai + 1] = ps[ai] * w.y;
                    vals[3 * ai + 2] = ps[ai] * w.z;
                }
            } else {
                need = true;
            }
        }
        seg_accumulate<9>(ns.accf, ns.acc, lane, p, vals);  // flagged points add zero here, their FP64 value when drained
        unsigned m = __ballot_sync(FULL, need);
        if (m) {
            int pos = nq + __popc(m & ((1u << lane) - 1u));
            if (need) {
                ns.qp[pos] = p;
                ns.qk[pos] = k;
            }
            nq += __popc(m);
            __syncwarp();
        }
        while (nq >= 32 || (nq > 0 && i0 + 32 >= total)) {
            const int take = nq < 32 ? nq : 32;
            int qpair = 32 + lane;
            double qv[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            if (lane < take) {
                qpair = ns.qp[lane];
                const TriGeo& Sq = wake ? a.wtri[list[qpair]] : a.tri[list[qpair]];
                near_point64(a, T, Sq, ns, qpair, ns.qk[lane], qv);
            }
            seg_accumulate<9>(ns.accf, ns.acc, lane, qpair, qv);
            const int rest = nq - take;
            int mp = 0, mk = 0;
            if (lane < rest) {
                mp = ns.qp[take + lane];
                mk = ns.qk[take + lane];
            }
            __syncwarp();
            if (lane < rest) {
                ns.qp[lane] = mp;
                ns.qk[lane] = mk;
            }
            __syncwarp();
            nq = rest;
            n64 += take;
        }
    }
    __syncwarp();
    // 4. the pairs' blocks
    if (near) {
        double Pp[9], blk[BLK_B];
        for (int k = 0; k < 9; ++k) Pp[k] = ns.acc[lane][k] + double(ns.accf[lane][k]);
        v3<double> nT = ld3(T.n);
        for (int bb = 0; bb < 3; ++bb) {
            v3<double> mv = cross(nT, ld3(S.gam + 3 * bb));
            for (int ai = 0; ai < 3; ++ai) blk[3 * ai + bb] = Pp[3 * ai] * mv.x + Pp[3 * ai + 1] * mv.y + Pp[3 * ai + 2] * mv.z;
        }
        const int nb = wake ? BLK_W : BLK_B;
        if (!wake)
            for (int ai = 0; ai < 3; ++ai)
                blk[9 + ai] = S.sigma * (Pp[3 * ai] * nT.x + Pp[3 * ai + 1] * nT.y + Pp[3 * ai + 2] * nT.z);
        double* dst = a.blk[wake ? 1 : 0] + size_t(p0 + lane - a.blk0[wake ? 1 : 0]) * nb;
#pragma unroll
        for (int k = 0; k < BLK_B; ++k)
            if (k < nb) dst[k] = blk[k];
    }
    P[TIER_NEAR] += __popc(nearmask);
    Q[TIER_NEAR] += (unsigned long long)total;
    Q64 += n64;
    return __ballot_sync(FULL, valid && !near);
}

// near tier, one pair per lane; the other pairs are listed for near_kernel_pairs. Warp w of nw of test triangle t: every
// nw-th chunk of its body and wake lists.
template <bool MIXED>
__device__ __forceinline__ void near_lanes_body(const NearArgs& a, const int t, const int w, const int nw,
                                                NearChunkSh& sh) {
    const int lane = threadIdx.x & 31;
    const TriGeo& T = a.tri[t];
    PairCtx pc;
    pc.a = &a;
    pc.T = &T;
    pc.sh = nullptr;
    pc.lane = lane;
    unsigned long long P[6] = {0, 0, 0, 0, 0, 0}, Q[6] = {0, 0, 0, 0, 0, 0}, Q64 = 0;
    const long long b0 = a.nf_ptr[t], nb = a.nf_ptr[t + 1] - b0, w0 = a.wf_ptr[t], nwk = a.wf_ptr[t + 1] - w0;
    const int cb = int((nb + 31) >> 5), cw = int((nwk + 31) >> 5);
    for (int c = w; c < cb + cw; c += nw) {
        const bool wake = c >= cb;
        const long long e = 32LL * (wake ? c - cb : c), n = (wake ? nwk : nb) - e, p0 = (wake ? w0 : b0) + e;
        const int cnt = int(n < 32 ? n : 32);
        const unsigned m = near_chunk<MIXED>(pc, sh, t, (wake ? a.wf_src : a.nf_src) + p0, cnt, wake, p0, P, Q, Q64);
        rest_append(a, 2 * t + (wake ? 1 : 0), p0, m, lane);
        __syncwarp();
    }
    if (lane == 0) {
        for (int k = 0; k < 6; ++k) {
            if (P[k]) atomicAdd(a.stats + k, P[k]);
            if (Q[k]) atomicAdd(a.stats + 6 + k, Q[k]);
        }
        if (Q64) atomicAdd(a.stats + 12, Q64);
    }
}

// the kernels of the non-far tiers take one system's arguments by value, or (BATCH) those of system work[i].x from sys.
// MIXED or FP64 by template: with both paths in one kernel the mixed one ran at 216 registers instead of 168 (near
// phase 64 ms instead of 50 on five wings of 900 to 4,000 triangles, before the leaf table). Ten CTAs an SM (168 registers,
// at most 96 bytes of them spilled in mixed precision): near phase 91 ms on a 25k wing; before the leaf table 106, 110 with
// twelve, 127 with eight, 135 with sixteen.
template <bool BATCH, bool MIXED>
__global__ void __launch_bounds__(32, 10) near_kernel_lanes(NearArgs a, const NearArgs* __restrict__ sys,
                                                                  const int2* __restrict__ work) {
    __shared__ NearChunkSh sh;
    const int2 wk = work[blockIdx.x];
    near_lanes_body<MIXED>(BATCH ? sys[wk.x] : a, wk.y, blockIdx.y, gridDim.y, sh);
}

// the block of one pair: the per-lane sums reduced and contracted with n_T x gamma_b (9 values, row-major), and the
// source part of the right hand side sigma_S (P_a . n_T) (3 values, subtracted when the pair is added)
__device__ __forceinline__ void pair_block_out(PairCtx& pc, FwdAcc& acc, const TriGeo& S, double* out, bool with_rhs) {
    fold32(acc);
    double P[9];
    for (int a = 0; a < 3; ++a) {
        P[3 * a + 0] = warp_sum(acc.P[a].x);
        P[3 * a + 1] = warp_sum(acc.P[a].y);
        P[3 * a + 2] = warp_sum(acc.P[a].z);
    }
    const TriGeo& T = *pc.T;
    v3<double> nT = ld3(T.n);
    if (pc.lane < 9) {
        int ai = pc.lane / 3, bb = pc.lane % 3;
        v3<double> m = cross(nT, ld3(S.gam + 3 * bb));
        out[pc.lane] = P[3 * ai] * m.x + P[3 * ai + 1] * m.y + P[3 * ai + 2] * m.z;
    } else if (with_rhs && pc.lane < 12) {
        int ai = pc.lane - 9;
        out[pc.lane] = S.sigma * (P[3 * ai] * nT.x + P[3 * ai + 1] * nT.y + P[3 * ai + 2] * nT.z);
    }
    __syncwarp();
}

// the mixed path's rare FP64 points, out of line: the multipole form, and the exact form in FP64 geometry with FP32-based
// functions where the split evaluation leaves FP32's range
__device__ __noinline__ v3<double> far64_sh(const WarpSh& sh, v3<double> r) { return sv_far(src64(sh), r); }
__device__ __noinline__ v3<double> exact64_sh(const WarpSh& sh, v3<double> ra, v3<double> rb, v3<double> rc, v3<double> r,
                                              int side) {
    return sv_exact3<double, KMathHyb>(src64(sh), ra, rb, rc, r, side, 1e-12);
}

// one FP64 point of a triangle pair: every point of the FP64 path, the points the FP32 guard refuses of the mixed one
template <bool MIXED>
__device__ __forceinline__ void fwd_point64(const PairCtx& pc, FwdAcc& acc, double l0, double l1, double l2, double W) {
    const WarpSh& sh = *pc.sh;
    const v3<double> ra = l0 * ld3(sh.E + 0) + l1 * ld3(sh.E + 9) + l2 * ld3(sh.E + 18);
    const v3<double> rb = l0 * ld3(sh.E + 3) + l1 * ld3(sh.E + 12) + l2 * ld3(sh.E + 21);
    const v3<double> rc = l0 * ld3(sh.E + 6) + l1 * ld3(sh.E + 15) + l2 * ld3(sh.E + 24);
    const SrcKern<double> S = src64(sh);
    const v3<double> r = ra + S.d[0];
    const double fd = pc.a->kernel_far * S.diam;
    const bool far = dot(r, r) > fd * fd;
    v3<double> w;
    if constexpr (MIXED) {
        v3<float> wf;
        if (far)
            w = far64_sh(sh, r);
        else if (sv_exact3_split(sh.Snu, sh.Slen, S.n, S.area, S.diam, ra, rb, rc, r, pc.side, 1e-12, wf))
            w = mk3(double(wf.x), double(wf.y), double(wf.z));
        else
            w = exact64_sh(sh, ra, rb, rc, r, pc.side);
    } else {
        w = far ? sv_far(S, r) : sv_exact3(S, ra, rb, rc, r, pc.side, 1e-12);
    }
    const v3<double> psi = test_weights(pc.a->test_mode, l0, l1, l2);
    acc.P[0] += (W * psi.x) * w;
    acc.P[1] += (W * psi.y) * w;
    acc.P[2] += (W * psi.z) * w;
}

// the records of a pair (walk_pair by one lane) evaluated by the warp. The buffer of leaves fills across the pair's pieces
// and is evaluated when full, a rule piece at once, as when the walkers give the pieces to emit_leaf and emit_rule.
// MIXED: a point is evaluated in FP32 under the guard; those it refuses are queued and evaluated 32 at a time.
template <bool MIXED>
__device__ __forceinline__ void eval_records(PairCtx& pc, FwdAcc& acc, const PieceRec* rec, int nrec,
                                             const unsigned* leaf) {
    WarpSh& sh = *pc.sh;
    const int lane = pc.lane;
    const double areaT = pc.T->area;
    int ri = 0, lpos = 0, nl = 0;
    for (;;) {
        int rid = -1, slot0 = 0, nslot = 0;
        while (ri < nrec) {
            const PieceRec& r = rec[ri];
            const int k = r.rid & (REC_DEP - 1);
            if (k != R_NEAR) {
                if (lane < 10) {
                    const double v = lane < 9 ? r.b[lane] : r.frac;
                    sh.leaf[LEAFBUF][lane] = v;
                    sh.leaff[LEAFBUF][lane] = lane < 9 ? float(v) : float(v * areaT);
                }
                rid = k;
                slot0 = LEAFBUF;
                nslot = 1;
                ++ri;
                break;
            }
            const int take = min(LEAFBUF - nl, r.nleaf - lpos);
            if (lane < take) {
                const unsigned code = leaf[r.leaf0 + lpos + lane];
                const int level = int(code >> LEAF_LEVEL);
                double b[9];
                quad_corners(r.b, level, code & ((1u << LEAF_LEVEL) - 1), b);
                for (int z = 0; z < 9; ++z) {
                    sh.leaf[nl + lane][z] = b[z];
                    sh.leaff[nl + lane][z] = float(b[z]);
                }
                const double fr = r.frac * ldexp(1.0, -2 * level);
                sh.leaf[nl + lane][9] = fr;
                sh.leaff[nl + lane][9] = float(fr * areaT);
            }
            nl += take;
            lpos += take;
            if (lpos == r.nleaf) {
                ++ri;
                lpos = 0;
            }
            if (nl == LEAFBUF) break;
        }
        if (rid < 0) {
            if (nl == 0) break;
            rid = R_NEAR;
            nslot = nl;
            nl = 0;
        }
        __syncwarp();
        const int n = pc.a->nrule[rid], tot = nslot * n;
        const RulePt* R = pc.a->rule[rid];
        const float4* Rf = pc.a->rulef[rid];
        int nq = 0;
        for (int i0 = 0; i0 < tot; i0 += 32) {
            const int i = i0 + lane, k = nslot > 1 ? i / n : 0, q = i - k * n, lf = slot0 + k;
            if constexpr (MIXED) {
                bool need = false;
                if (i < tot) {
                    const float4 m = Rf[q];
                    const float* bf = sh.leaff[lf];
                    const float l0 = m.x * bf[0] + m.y * bf[3] + m.z * bf[6];
                    const float l1 = m.x * bf[1] + m.y * bf[4] + m.z * bf[7];
                    const float l2 = m.x * bf[2] + m.y * bf[5] + m.z * bf[8];
                    need = !fwd_point32(pc, acc, l0, l1, l2, m.w * bf[9]);
                }
                const unsigned msk = __ballot_sync(0xffffffffu, need);
                if (need) {
                    const int pos = nq + __popc(msk & ((1u << lane) - 1u));
                    sh.qi[pos] = q;
                    sh.ql[pos] = lf;
                }
                nq += __popc(msk);
                while (nq >= 32 || (nq > 0 && i0 + 32 >= tot)) {
                    __syncwarp();
                    const int take = nq < 32 ? nq : 32;
                    if (lane < take) {
                        const RulePt m = R[sh.qi[lane]];
                        const double* b = sh.leaf[sh.ql[lane]];
                        const double l0 = m.l0 * b[0] + m.l1 * b[3] + m.l2 * b[6];
                        const double l1 = m.l0 * b[1] + m.l1 * b[4] + m.l2 * b[7];
                        const double l2 = m.l0 * b[2] + m.l1 * b[5] + m.l2 * b[8];
                        fwd_point64<true>(pc, acc, l0, l1, l2, (m.w * b[9]) * areaT);
                    }
                    nq -= take;
                    int mi = 0, ml = 0;
                    if (lane < nq) {
                        mi = sh.qi[take + lane];
                        ml = sh.ql[take + lane];
                    }
                    __syncwarp();
                    if (lane < nq) {
                        sh.qi[lane] = mi;
                        sh.ql[lane] = ml;
                    }
                    pc.n64 += take;
                }
            } else {
                if (i < tot) {
                    const RulePt m = R[q];
                    const double* b = sh.leaf[lf];
                    const double l0 = m.l0 * b[0] + m.l1 * b[3] + m.l2 * b[6];
                    const double l1 = m.l0 * b[1] + m.l1 * b[4] + m.l2 * b[7];
                    const double l2 = m.l0 * b[2] + m.l1 * b[5] + m.l2 * b[8];
                    fwd_point64<false>(pc, acc, l0, l1, l2, (m.w * b[9]) * areaT);
                }
            }
        }
        pc.npts += tot;
        __syncwarp();
    }
    if (!MIXED) pc.n64 = pc.npts;
}

// a pair whose records do not fit, walked and evaluated piece by piece: its block to out; returns the tier
__device__ __noinline__ int pair_direct(const NearArgs& a, WarpSh& sh, int t, int s, bool wake, double* out,
                                        long long* npts, long long* n64) {
    PairCtx pc;
    pc.a = &a;
    pc.T = &a.tri[t];
    pc.sh = &sh;
    pc.lane = threadIdx.x & 31;
    pc.kind = 0;
    pc.npts = pc.n64 = 0;
    pc.nleaf = pc.nq64 = 0;
    FwdAcc acc = {};
    const int tier = tri_pair(pc, acc, t, s, wake);
    pair_block_out(pc, acc, wake ? a.wtri[s] : a.tri[s], out, !wake);
    *npts = pc.npts;
    *n64 = pc.n64;
    return tier;
}

// The self, touching and contact pairs: a persistent grid whose warps take the next pairs of the list from a counter, so
// that test triangles with many contact pairs (thin panels at a sharp trailing edge) do not hold a launch. Each lane
// walks one pair into records (in the warp's part of recs and leaves), then the warp evaluates the pairs one by one;
// each block goes to its pair's place in blk. Mixed, 25k wing (1.1M pairs, 1.97G points): 150 ms, 358 ms when the warp
// walked and evaluated piece by piece.
template <bool BATCH, bool MIXED>
__global__ void __launch_bounds__(32 * NEAR_WARPS, 3) near_kernel_pairs(NearArgs a1, const NearArgs* __restrict__ sys,
                                                                     PieceRec* recs, unsigned* leaves, int gmax) {
    __shared__ WarpSh shm[NEAR_WARPS];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long total = (long long)*a1.rest_n;
    const int warp = blockIdx.x * NEAR_WARPS + w;
    recs += size_t(warp) * gmax * REC_MAX;
    leaves += size_t(warp) * gmax * REC_LEAVES;
    PairCtx pc;
    pc.sh = &shm[w];
    pc.lane = lane;
    pc.kind = 0;
    unsigned long long P[6] = {0, 0, 0, 0, 0, 0}, Q[6] = {0, 0, 0, 0, 0, 0}, Q64 = 0;
    auto flush = [&](const NearArgs& a) {  // the counts of system a so far
        if (lane == 0) {
            for (int k = 0; k < 6; ++k) {
                if (P[k]) atomicAdd(a.stats + k, P[k]);
                if (Q[k]) atomicAdd(a.stats + 6 + k, Q[k]);
            }
            if (Q64) atomicAdd(a.stats + 12, Q64);
        }
        for (int k = 0; k < 6; ++k) P[k] = Q[k] = 0;
        Q64 = 0;
    };
    for (;;) {
        int cnt;
        const long long idx0 = next_rest_pairs(a1, total, gmax, lane, cnt);
        if (cnt == 0) break;
        // each lane walks its pair
        unsigned long long item = 0;
        int sy = 0, s = 0, tier = 0;
        RecAcc ra;
        ra.n = ra.nleaf = 0;
        ra.over = false;
        if (lane < cnt) {
            item = a1.rest_item[idx0 + lane];
            if (BATCH) sy = a1.rest_sys[idx0 + lane];
            const NearArgs& a = BATCH ? sys[sy] : a1;
            const int g = int(item >> REST_SHIFT), t = g >> 1;
            const bool wake = (g & 1) != 0;
            s = (wake ? a.wf_src : a.nf_src)[item & ((1ull << REST_SHIFT) - 1)];
            PairCtx wc;
            wc.a = &a;
            wc.T = &a.tri[t];
            wc.lane = 0;
            ra.rec = recs + lane * REC_MAX;
            ra.leaf = leaves + lane * REC_LEAVES;
            ra.dep = ra.moves = false;
            if (MIXED || wake || s != t) tier = walk_pair(wc, ra, t, s, wake ? a.wtri[s] : a.tri[s], wake);
        }
        __syncwarp();
        for (int q = 0; q < cnt; ++q) {
            const unsigned long long it = __shfl_sync(0xffffffffu, item, q);
            const NearArgs& a = BATCH ? sys[__shfl_sync(0xffffffffu, sy, q)] : a1;
            const int sq = __shfl_sync(0xffffffffu, s, q), nrec = __shfl_sync(0xffffffffu, ra.n, q);
            const bool over = __shfl_sync(0xffffffffu, int(ra.over), q) != 0;
            int tq = __shfl_sync(0xffffffffu, tier, q);
            const int g = int(it >> REST_SHIFT), t = g >> 1;
            const bool wake = (g & 1) != 0;
            const long long p = (long long)(it & ((1ull << REST_SHIFT) - 1));
            if (!MIXED && !wake && sq == t) continue;  // near_kernel_self64's
            const TriGeo& S = wake ? a.wtri[sq] : a.tri[sq];
            double* out = a.blk[wake ? 1 : 0] + size_t(p - a.blk0[wake ? 1 : 0]) * (wake ? BLK_W : BLK_B);
            pc.npts = 0;
            pc.n64 = 0;
            if (over) {
                long long np, n64;
                tq = pair_direct(a, shm[w], t, sq, wake, out, &np, &n64);
                pc.npts = np;
                pc.n64 = n64;
            } else {
                pc.a = &a;
                pc.T = &a.tri[t];
                setup_tri_source(pc, S);
                pc.side = (!wake && sq == t) ? 1 : 0;
                FwdAcc acc = {};
                eval_records<MIXED>(pc, acc, recs + q * REC_MAX, nrec, leaves + q * REC_LEAVES);
                pair_block_out(pc, acc, S, out, !wake);
            }
            P[tq] += 1;
            Q[tq] += pc.npts;
            Q64 += pc.n64;
            if (BATCH) flush(a);
        }
        __syncwarp();
    }
    if (!BATCH) flush(a1);
}

// The self pairs in FP64, a CTA a test triangle: the rule's points over its warps, whose sums are added in warp order (one
// warp took the 4,500 points in 142 rounds, which held an 80-triangle sphere at 1.97 ms: 1.19 so, 9.1 -> 8.4 ms on a
// 1,280-triangle one). Every system and batch takes them so, as their sums' order shows in the last bits. Mixed sums in
// FP32, whose order stays.
constexpr int SELF_WARPS = 8;
template <bool BATCH>
__global__ void __launch_bounds__(32 * SELF_WARPS) near_kernel_self64(NearArgs a1, const NearArgs* __restrict__ sys,
                                                                    const int2* __restrict__ work) {
    __shared__ WarpSh shm;
    __shared__ double s_P[SELF_WARPS][9];
    const int2 wk = work[blockIdx.x];
    const NearArgs& a = BATCH ? sys[wk.x] : a1;
    const int t = wk.y, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const TriGeo& T = a.tri[t];
    // the pair's place: the test triangle among its own sources, which are in order; none in an assembly of wake columns only
    const long long e = a.nf_ptr[t + 1];
    long long lo = a.nf_ptr[t], hi = e;
    while (hi - lo > 1) {
        const long long mid = (lo + hi) >> 1;
        if (a.nf_src[mid] <= t) lo = mid;
        else hi = mid;
    }
    if (lo >= e || a.nf_src[lo] != t) return;
    PairCtx pc;
    pc.a = &a;
    pc.T = &T;
    pc.sh = &shm;
    pc.lane = lane;
    pc.kind = 0;
    pc.side = 1;
    pc.fp32 = 0;
    if (w == 0) setup_tri_source(pc, T);
    __syncthreads();
    const int n = a.nrule[R_SELF];
    FwdAcc acc = {};
    for (int i = threadIdx.x; i < n; i += 32 * SELF_WARPS) {
        const RulePt m = a.rule[R_SELF][i];
        fwd_point64<false>(pc, acc, m.l0, m.l1, m.l2, m.w * T.area);
    }
    for (int k = 0; k < 3; ++k) {
        const v3<double> P = mk3(warp_sum(acc.P[k].x), warp_sum(acc.P[k].y), warp_sum(acc.P[k].z));
        if (lane == 0) {
            s_P[w][3 * k] = P.x;
            s_P[w][3 * k + 1] = P.y;
            s_P[w][3 * k + 2] = P.z;
        }
    }
    __syncthreads();
    if (w > 0) return;
    acc = {};
    if (lane == 0)
        for (int k = 0; k < 3; ++k)
            for (int c = 0; c < SELF_WARPS; ++c) acc.P[k] += mk3(s_P[c][3 * k], s_P[c][3 * k + 1], s_P[c][3 * k + 2]);
    __syncwarp();
    pair_block_out(pc, acc, T, a.blk[0] + size_t(lo - a.blk0[0]) * BLK_B, true);
    if (lane == 0) {
        atomicAdd(a.stats + TIER_SELF, 1ull);
        atomicAdd(a.stats + 6 + TIER_SELF, (unsigned long long)n);
        atomicAdd(a.stats + 12, (unsigned long long)n);
    }
}

// one far tip filament of test triangle T, summed by one lane: segment_block (assemble.jl:312-321) with the far rule
// (the columns of the filament's two end nodes, ca and cb, per test function)
__device__ void far_filament_fwd(const NearArgs& a, const TriGeo& T, v3<double> fa, v3<double> fb, double* ca,
                                 double* cb) {
    const RulePt* R = a.rule[R_FAR];
    const v3<double> n = ld3(T.n);
    v3<double> Ea[3], Eb[3];
    for (int k = 0; k < 3; ++k) {
        Ea[k] = ld3(T.x + 3 * k) - fa;
        Eb[k] = ld3(T.x + 3 * k) - fb;
    }
    for (int i = 0; i < a.nrule[R_FAR]; ++i) {
        const RulePt m = R[i];
        const double W = m.w * T.area;
        const v3<double> ra = m.l0 * Ea[0] + m.l1 * Ea[1] + m.l2 * Ea[2];
        const v3<double> rb = m.l0 * Eb[0] + m.l1 * Eb[1] + m.l2 * Eb[2];
        v3<double> va, vb;
        segment_velocity(ra, rb, va, vb);
        const v3<double> psi = test_weights(a.test_mode, m.l0, m.l1, m.l2);
        const double da = dot(va, n) * W, db = dot(vb, n) * W;
        ca[0] += da * psi.x;
        ca[1] += da * psi.y;
        ca[2] += da * psi.z;
        cb[0] += db * psi.x;
        cb[1] += db * psi.y;
        cb[2] += db * psi.z;
    }
}

// the tip filaments (assemble.jl:344-354): segment_rule (:299-306) and segment_block (:312-321), FP64. A warp takes 32
// filaments of one test triangle: a far one (the far rule's few points) is summed by its own lane, the others by the
// whole warp. Every (test triangle, filament) writes the columns of its two ends to fil_out; near_kernel_gather adds
// them.
template <bool BATCH>
__global__ void __launch_bounds__(32 * NEAR_WARPS, 3) near_kernel_filaments(NearArgs a1, const NearArgs* __restrict__ sys,
                                                                         const int2* __restrict__ work, int nwork) {
    __shared__ WarpSh shm[NEAR_WARPS];
    const int idx = blockIdx.x * NEAR_WARPS + (threadIdx.x >> 5);
    if (idx >= nwork) return;
    const int2 wk = work[idx];
    const NearArgs& a = BATCH ? sys[wk.x] : a1;
    const int f0 = blockIdx.y * 32;
    if (f0 >= a.nfil) return;
    const int t = wk.y;
    const int lane = threadIdx.x & 31;
    const TriGeo& T = a.tri[t];
    PairCtx pc;
    pc.a = &a;
    pc.T = &T;
    pc.sh = &shm[threadIdx.x >> 5];
    pc.lane = lane;
    pc.nleaf = 0;
    pc.nq64 = 0;
    pc.fp32 = 0;
    unsigned long long P[6] = {0, 0, 0, 0, 0, 0}, Q[6] = {0, 0, 0, 0, 0, 0}, Q64 = 0;
    const double corners[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
    double* out = a.fil_out + 6 * (size_t(t - a.t0) * a.nfil + f0);
    const int cnt = a.nfil - f0 < 32 ? a.nfil - f0 : 32;
    bool mfar = false;
    if (lane < cnt) {
        const v3<double> fa = ld3(a.wx + 3 * a.fil[2 * (f0 + lane)]), fb = ld3(a.wx + 3 * a.fil[2 * (f0 + lane) + 1]);
        mfar = vnorm((fa + fb) / 2.0 - ld3(T.c)) > a.far_ratio * fmax(T.diam, vnorm(fb - fa));
        if (mfar) {
            double mca[3] = {0, 0, 0}, mcb[3] = {0, 0, 0};
            far_filament_fwd(a, T, fa, fb, mca, mcb);
            for (int k = 0; k < 3; ++k) {
                out[6 * lane + k] = mca[k];
                out[6 * lane + 3 + k] = mcb[k];
            }
        }
    }
    const unsigned farmask = __ballot_sync(0xffffffffu, mfar);
    P[TIER_FAR] += __popc(farmask);
    Q[TIER_FAR] += (unsigned long long)__popc(farmask) * a.nrule[R_FAR];
    for (int q = 0; q < cnt; ++q) {
        if ((farmask >> q) & 1u) continue;
        // near and vertex filaments, the whole warp
        const v3<double> fa = ld3(a.wx + 3 * a.fil[2 * (f0 + q)]), fb = ld3(a.wx + 3 * a.fil[2 * (f0 + q) + 1]);
        if (lane == 0) {
            for (int k = 0; k < 3; ++k) {
                pc.sh->E[9 * k + 0] = T.x[3 * k + 0] - fa.x;
                pc.sh->E[9 * k + 1] = T.x[3 * k + 1] - fa.y;
                pc.sh->E[9 * k + 2] = T.x[3 * k + 2] - fa.z;
                pc.sh->E[9 * k + 3] = T.x[3 * k + 0] - fb.x;
                pc.sh->E[9 * k + 4] = T.x[3 * k + 1] - fb.y;
                pc.sh->E[9 * k + 5] = T.x[3 * k + 2] - fb.z;
            }
        }
        __syncwarp();
        FwdAcc acc = {};
        pc.kind = 1;
        pc.npts = 0;
        pc.n64 = 0;
        pc.side = 0;
        pc.fp32 = 0;
        int tier, kv = -1;
        for (int k = 0; k < 3 && kv < 0; ++k)
            if (fmin(vnorm(ld3(T.x + 3 * k) - fa), vnorm(ld3(T.x + 3 * k) - fb)) <= 1e-12 * T.diam) kv = k;
        if (kv >= 0) {
            tier = TIER_VERTEX;
            vertex_rule(pc, acc, kv);
        } else {
            tier = TIER_NEAR;
            SrcRef src{1, nullptr, fa, fb};
            near_pieces(pc, acc, src, corners, 1.0, a.near_depth);
            flush_leaves(pc, acc);
        }
        double ca[3], cb[3];
        for (int k = 0; k < 3; ++k) {
            ca[k] = warp_sum(acc.ca[k]);
            cb[k] = warp_sum(acc.cb[k]);
        }
        if (lane == 0)
            for (int k = 0; k < 3; ++k) {
                out[6 * q + k] = ca[k];
                out[6 * q + 3 + k] = cb[k];
            }
        __syncwarp();
        P[tier] += 1;
        Q[tier] += pc.npts;
        Q64 += pc.n64;
    }
    if (lane == 0) {
        for (int k = 0; k < 6; ++k) {
            if (P[k]) atomicAdd(a.stats + k, P[k]);
            if (Q[k]) atomicAdd(a.stats + 6 + k, Q[k]);
        }
        if (Q64) atomicAdd(a.stats + 12, Q64);
    }
}

// the place of source s in the ascending list of n sources, or -1
__device__ __forceinline__ int find_source(const int* list, int n, int s) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (list[mid] < s) lo = mid + 1;
        else hi = mid;
    }
    return lo < n && list[lo] == s ? lo : -1;
}

constexpr int GATHER_NT = 128;
constexpr int GATHER_LIST = 2048;  // sources of a list staged in shared memory (8 KB); longer lists are searched in place

// One CTA per row slot: the blocks of its triangles' non-far pairs and their filaments' columns added to its row of A, its
// right hand side to b, in a fixed order. Per triangle, a thread takes a (pair, source corner) and adds its column's
// whole sum if no earlier pair of the list has that column: the pairs with the column are those of the column's
// triangles that binary search finds in the list. Latency of the searches and of the row's read-modify-writes bounds
// it, so all rows share one launch (one CTA per test triangle, a launch per colour: 2.0 ms on a 1,676-triangle wing).
template <bool BATCH>
__global__ void __launch_bounds__(GATHER_NT) near_kernel_gather(NearArgs a1, const NearArgs* __restrict__ sys,
                                                              const int2* __restrict__ work) {
    __shared__ int s_list[GATHER_LIST];
    __shared__ double red[GATHER_NT];
    const int2 wk = work[blockIdx.x];
    const NearArgs& a = BATCH ? sys[wk.x] : a1;
    const int slot = wk.y, tid = threadIdx.x;
    double* row = a.A + size_t(slot) * size_t(a.lda);
    double rb = 0, free = 0;
    for (int ue = a.col_ptr[0][slot]; ue < a.col_ptr[0][slot + 1]; ++ue) {
        const int et = a.col_ent[0][ue], t = et / 3, ta = et - 3 * t;
        if (t < a.t0 || t >= a.t1) continue;
        const TriGeo& T = a.tri[t];
        for (int set = 0; set < 2; ++set) {
            const long long p0 = (set ? a.wf_ptr : a.nf_ptr)[t];
            const int n = int((set ? a.wf_ptr : a.nf_ptr)[t + 1] - p0);
            if (n == 0) continue;
            const int* src = (set ? a.wf_src : a.nf_src) + p0;
            const int nb = set ? BLK_W : BLK_B;
            const double* blk = a.blk[set] + size_t(p0 - a.blk0[set]) * nb + 3 * ta;
            const int col0 = set ? a.nslot : 0;
            const int *slots = a.slots[set], *ptr = a.col_ptr[set], *ent = a.col_ent[set];
            const bool staged = n <= GATHER_LIST;
            __syncthreads();
            if (staged)
                for (int i = tid; i < n; i += GATHER_NT) s_list[i] = src[i];
            __syncthreads();
            const int* list = staged ? s_list : src;
            for (int i = tid; i < 3 * n; i += GATHER_NT) {
                const int p = i / 3, b = i - 3 * p, s = list[p], c = slots[3 * s + b];
                double v = 0;
                bool own = false;
                for (int u = ptr[c]; u < ptr[c + 1]; ++u) {
                    const int e = ent[u], se = e / 3, be = e - 3 * se;
                    const bool me = e == 3 * s + b;
                    const int q = me ? p : find_source(list, n, se);
                    if (q < 0) continue;
                    if (!me && !own) break;  // an earlier pair has this column
                    own = true;
                    v += blk[size_t(q) * nb + be];
                }
                if (own) row[col0 + c] += v;
            }
            if (!set)
                for (int p = tid; p < n; p += GATHER_NT) rb -= blk[size_t(p) * nb + 9 - 2 * ta];
        }
        if (a.nfil > 0) {
            __syncthreads();  // the wake's columns are the filaments' too
            const double* fo = a.fil_out + 6 * size_t(t - a.t0) * a.nfil + ta;
            for (int i = tid; i < a.nfnode; i += GATHER_NT) {
                double v = 0;
                for (int u = a.fnode_ptr[i]; u < a.fnode_ptr[i + 1]; ++u) v += fo[3 * a.fnode_ent[u]];
                row[a.nslot + a.fnode[i]] += v;
            }
        }
        // the freestream, exact (assemble.jl:422)
        free += (a.vinf[0] * T.n[0] + a.vinf[1] * T.n[1] + a.vinf[2] * T.n[2]) * T.area * a.tint[ta];
    }
    red[tid] = rb;
    for (int o = GATHER_NT / 2; o > 0; o >>= 1) {
        __syncthreads();
        if (tid < o) red[tid] += red[tid + o];
    }
    if (tid == 0) a.b[slot] += red[0] - free;
}

// ------------------------------------------------------------------------------------------------------------------
// host: one system's assembly, prepared (classification, pair lists, far tiles and their colours, near colours) and
// then launched; a batch prepares every system and launches each phase once over all of them

// the far tier's test tiles of TT triangles: their unique row slots, uploaded; the tiles grouped by colour (no two
// tiles of a colour share a row slot)
template <int TT>
int far_prepare(vp_ctx* ctx, FarArgs& fa, int nt, const int* cslot, int nslot, DevList& dl,
                std::vector<std::vector<int>>& colours) {
    int ntiles = (nt + TT - 1) / TT;
    std::vector<int> trow(size_t(ntiles) * 3 * TT), tnrow(ntiles);
    std::vector<short> trptr(size_t(ntiles) * (3 * TT + 1)), trent(size_t(ntiles) * 3 * TT);
    std::vector<std::vector<int>> groups(ntiles);
    for (int k = 0; k < ntiles; ++k) {
        std::vector<int> cs(3 * TT, -1);
        for (int i = 0; i < TT; ++i) {
            int t = k * TT + i;
            if (t < nt)
                for (int a = 0; a < 3; ++a) cs[3 * i + a] = cslot[3 * t + a];
        }
        unique_map(cs, 3 * TT, &trow[size_t(k) * 3 * TT], tnrow[k], &trptr[size_t(k) * (3 * TT + 1)],
                   &trent[size_t(k) * 3 * TT]);
        for (int j = 0; j < tnrow[k]; ++j) groups[k].push_back(trow[size_t(k) * 3 * TT + j]);
    }
    colours = colour_groups(groups, nslot);
    int *d_trow, *d_tnrow;
    short *d_trptr, *d_trent;
    int r;
    if ((r = dl.up(ctx, &d_trow, trow)) || (r = dl.up(ctx, &d_tnrow, tnrow)) || (r = dl.up(ctx, &d_trptr, trptr)) ||
        (r = dl.up(ctx, &d_trent, trent)))
        return r;
    fa.trow = d_trow;
    fa.tnrow = d_tnrow;
    fa.trptr = d_trptr;
    fa.trent = d_trent;
    return VP_OK;
}

// one system of an assembly between its phases
struct AsmJob {
    PairInput in;
    int tt = 8;  // test triangles per far tile
    PairSetup ps;
    vp_system* sys = nullptr;
    FarArgs fa{};
    std::vector<std::vector<int>> far_col;   // far test tiles, per colour
    NearArgs na{};
    unsigned long long* d_stats = nullptr;
    std::chrono::steady_clock::time_point t0;
    ~AsmJob() {
        if (sys) vp_system_free(sys);
    }
};

// classification, pair lists, the zeroed system, the far tier's source tiles and arrays, its test tiles and their
// colours, the near tier's arguments
int job_prepare(vp_ctx* ctx, AsmJob& j) {
    j.t0 = std::chrono::steady_clock::now();
    const PairInput& in = j.in;
    const vp_assembly_options* o = in.o;
    int r = setup_pairs(ctx, in, PH_SETUP, PH_CLASSIFY, j.ps);
    if (r) return r;
    PairSetup& ps = j.ps;
    DevList& dl = ps.dl;
    const int ntri = in.ntri, nslot = in.nslot, nwtri = in.nwtri, ncols = ps.ncols;
    vp_system* sys = new vp_system();
    j.sys = sys;
    sys->nslot = nslot;
    sys->ncols = ncols;
    sys->nwnode = in.nwnode;
    if ((r = vp_alloc(ctx, &sys->A, size_t(nslot) * ncols)) || (r = vp_alloc(ctx, &sys->b, size_t(nslot)))) return r;
    VP_CUDA(ctx, cudaMemsetAsync(sys->A, 0, sizeof(double) * size_t(nslot) * ncols, ctx->stream));
    VP_CUDA(ctx, cudaMemsetAsync(sys->b, 0, sizeof(double) * nslot, ctx->stream));
    // far tier
    FarArgs& fa = j.fa;
    fa.ntest = ntri;
    fa.nq = ps.nq;
    fa.test_mode = o->test;
    fa.tq = ps.d_tq;
    fa.tw = ps.d_tw;
    fa.tgeo = ps.d_tg;
    fa.tcent = ps.d_tc;
    fa.nset = nwtri > 0 ? 2 : 1;
    fa.A = sys->A;
    fa.lda = ncols;
    fa.b = sys->b;
    fa.ratio32 = ps.ratio32;
    fa.ratio = o->far_ratio;
    fa.kernel_far = o->kernel_far;
    const std::vector<TriGeo>* sets[2] = {&ps.tg, &ps.wg};
    int nsrc[2] = {in.body_sources ? ntri : 0, nwtri};
    for (int set = 0; set < fa.nset; ++set) {
        std::vector<TriGeo> g(sets[set]->begin(), sets[set]->begin() + nsrc[set]);
        SrcTiles st = make_src_tiles(g);
        int *d_cols, *d_ncol;
        short *d_cptr, *d_cent;
        if ((r = dl.up(ctx, &d_cols, st.cols)) || (r = dl.up(ctx, &d_ncol, st.ncol)) ||
            (r = dl.up(ctx, &d_cptr, st.cptr)) || (r = dl.up(ctx, &d_cent, st.cent)))
            return r;
        fa.nsrc[set] = nsrc[set];
        fa.ntile[set] = st.ntile;
        fa.col_off[set] = set == 0 ? 0 : nslot;
        fa.scent[set] = set == 0 ? ps.d_tc : ps.d_wc;
        fa.sgeo[set] = set == 0 ? ps.d_tg : ps.d_wg;
        fa.tile_cols[set] = d_cols;
        fa.tile_ncol[set] = d_ncol;
        fa.tile_cptr[set] = d_cptr;
        fa.tile_cent[set] = d_cent;
        if (ps.mixed) {
            std::vector<float> soa;
            float* d;
            fill_soa(g, soa, fa.pad[set]);
            if ((r = dl.up(ctx, &d, soa))) return r;
            fa.soa[set] = d;
        } else {
            std::vector<double> soa;
            double* d;
            fill_soa(g, soa, fa.pad[set]);
            if ((r = dl.up(ctx, &d, soa))) return r;
            fa.soa[set] = d;
        }
    }
    j.tt = ctx->far_tile[ps.mixed ? 1 : 0];
    switch (j.tt) {
        case 1: r = far_prepare<1>(ctx, fa, ntri, in.corner_slot, nslot, dl, j.far_col); break;
        case 2: r = far_prepare<2>(ctx, fa, ntri, in.corner_slot, nslot, dl, j.far_col); break;
        case 4: r = far_prepare<4>(ctx, fa, ntri, in.corner_slot, nslot, dl, j.far_col); break;
        case 8: r = far_prepare<8>(ctx, fa, ntri, in.corner_slot, nslot, dl, j.far_col); break;
        default: return vp_fail(ctx, VP_ERR_ARG, "far tile must be 1, 2, 4 or 8 test triangles");
    }
    if (r) return r;
    // near, touching and contact tiers
    if ((r = dl.alloc(ctx, &j.d_stats, 13))) return r;
    VP_CUDA(ctx, cudaMemsetAsync(j.d_stats, 0, sizeof(unsigned long long) * 13, ctx->stream));
    j.na = near_args(ps, in);
    j.na.A = sys->A;
    j.na.b = sys->b;
    j.na.stats = j.d_stats;
    // the columns' triangles (and corners), the filaments' nodes
    std::vector<int> wslots(3 * size_t(nwtri));
    for (int t = 0; t < nwtri; ++t)
        for (int k = 0; k < 3; ++k) wslots[3 * size_t(t) + k] = ps.wg[t].slot[k];
    auto csr = [](const int* key, int n, int nkey, std::vector<int>& ptr, std::vector<int>& ent) {
        ptr.assign(size_t(nkey) + 1, 0);
        ent.assign(std::max(n, 1), 0);
        for (int i = 0; i < n; ++i) ptr[key[i] + 1]++;
        for (int c = 0; c < nkey; ++c) ptr[c + 1] += ptr[c];
        std::vector<int> at(ptr.begin(), ptr.end() - 1);
        for (int i = 0; i < n; ++i) ent[at[key[i]]++] = i;
    };
    const int* keys[2] = {in.corner_slot, wslots.data()};
    const int nel[2] = {ntri, nwtri}, nkey[2] = {nslot, in.nwnode};
    for (int set = 0; set < 2; ++set) {
        std::vector<int> ptr, ent, sl(keys[set], keys[set] + 3 * size_t(nel[set]));
        csr(keys[set], 3 * nel[set], nkey[set], ptr, ent);
        int *d_sl, *d_ptr, *d_ent;
        if ((r = dl.up(ctx, &d_sl, sl)) || (r = dl.up(ctx, &d_ptr, ptr)) || (r = dl.up(ctx, &d_ent, ent))) return r;
        j.na.slots[set] = d_sl;
        j.na.col_ptr[set] = d_ptr;
        j.na.col_ent[set] = d_ent;
    }
    if (in.nfil > 0) {
        std::vector<int> ptr, ent, node, nptr{0};
        csr(in.fil, 2 * in.nfil, in.nwnode, ptr, ent);
        for (int i = 0; i < in.nwnode; ++i)
            if (ptr[i + 1] > ptr[i]) {
                node.push_back(i);
                nptr.push_back(ptr[i + 1]);
            }
        int *d_node, *d_ptr, *d_ent;
        if ((r = dl.up(ctx, &d_node, node)) || (r = dl.up(ctx, &d_ptr, nptr)) || (r = dl.up(ctx, &d_ent, ent))) return r;
        j.na.nfnode = int(node.size());
        j.na.fnode = d_node;
        j.na.fnode_ptr = d_ptr;
        j.na.fnode_ent = d_ent;
    }
    return VP_OK;
}

// the statistics and the system of a finished job (the stream is synchronised)
int job_finish(vp_ctx* ctx, AsmJob& j, vp_system** out, vp_assembly_stats* stats) {
    unsigned long long hs[13];
    VP_CUDA(ctx, vp_d2h(ctx, hs, j.d_stats, sizeof(hs)));
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return vp_fail(ctx, VP_ERR_CUDA, std::string("assembly kernels: ") + cudaGetErrorString(e));
    if (stats) {
        const PairInput& in = j.in;
        long long total = (long long)in.ntri * (in.ntri + in.nwtri) + (long long)in.ntri * in.nfil;
        long long nonfar = 0;
        for (int k = 0; k < 6; ++k) {
            stats->pairs[k] = (long long)hs[k];
            stats->points[k] = (long long)hs[6 + k];
            if (k != TIER_FAR) nonfar += (long long)hs[k];
        }
        long long far_fil = (long long)hs[TIER_FAR];
        long long far_tri = total - nonfar - far_fil;
        stats->pairs[TIER_FAR] = far_tri + far_fil;
        stats->points[TIER_FAR] = (long long)hs[6 + TIER_FAR] + far_tri * j.ps.nq;
        stats->points_fp64 = (long long)hs[12] + (j.ps.mixed ? 0 : far_tri * j.ps.nq);
        stats->time_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - j.t0).count();
    }
    *out = j.sys;
    j.sys = nullptr;
    return VP_OK;
}

// one system: the far tiles of a colour per launch
template <class T, int TT>
int far_launch(vp_ctx* ctx, AsmJob& j) {
    std::vector<int> all;
    std::vector<int> off{0};
    for (auto& c : j.far_col) {
        all.insert(all.end(), c.begin(), c.end());
        off.push_back((int)all.size());
    }
    int* d_tiles;
    int r;
    if ((r = j.ps.dl.up(ctx, &d_tiles, all))) return r;
    FarArgs fa = j.fa;
    vp_phase_begin(ctx, PH_FAR);
    for (size_t c = 0; c < j.far_col.size(); ++c) {
        fa.tiles = d_tiles + off[c];
        int nb = off[c + 1] - off[c];
        if (nb) {
            far_kernel<T, TT><<<nb, FAR_NT, 0, ctx->stream>>>(fa);
            ctx->launches++;
        }
    }
    vp_phase_end(ctx);
    VP_CUDA(ctx, cudaGetLastError());
    return VP_OK;
}

// a batch: colour c's far tiles of every system in one launch
template <class T, int TT>
int far_launch_batch(vp_ctx* ctx, std::vector<std::unique_ptr<AsmJob>>& jobs, DevList& dl) {
    std::vector<FarArgs> args;
    size_t ncol = 0;
    for (auto& j : jobs) {
        args.push_back(j->fa);
        ncol = std::max(ncol, j->far_col.size());
    }
    FarArgs* d_args;
    int r;
    if ((r = dl.up(ctx, &d_args, args))) return r;
    vp_phase_begin(ctx, PH_FAR);
    for (size_t c = 0; c < ncol; ++c) {
        std::vector<int2> work;
        for (size_t k = 0; k < jobs.size(); ++k)
            if (c < jobs[k]->far_col.size())
                for (int tile : jobs[k]->far_col[c]) work.push_back(make_int2(int(k), tile));
        if (work.empty()) continue;
        int2* d_work;
        if ((r = dl.up(ctx, &d_work, work))) return r;
        far_kernel_batch<T, TT><<<int(work.size()), FAR_NT, 0, ctx->stream>>>(d_args, d_work);
        ctx->launches++;
    }
    vp_phase_end(ctx);
    VP_CUDA(ctx, cudaGetLastError());
    return VP_OK;
}

// the pair blocks' workspace of one pass over test triangles, at most (a pass holds at least one test triangle)
constexpr size_t NEAR_PASS_BYTES = size_t(1) << 30;

// The non-far tiers of the jobs (one: BATCH false). The test triangles go in passes whose pair blocks fit the workspace;
// a pass is: the lanes kernel over all its test triangles (blocks of the near pairs, the list of the rest), the
// persistent pair kernel (blocks of the rest), the filaments, and the kernel that adds the blocks to A's rows.
template <bool BATCH>
int near_launch(vp_ctx* ctx, const std::vector<AsmJob*>& jobs, DevList& dl) {
    int r;
    const int nsys = int(jobs.size());
    struct Range {
        int sys, t0, t1;
    };
    std::vector<std::vector<Range>> passes;
    size_t used = 0, most = 0, most_items = 0, items = 0, most_fil = 0, fil = 0;
    long long max_pairs = 0;
    auto close = [&]() {
        most = std::max(most, used);
        most_items = std::max(most_items, items);
        most_fil = std::max(most_fil, fil);
        used = items = fil = 0;
    };
    for (int k = 0; k < nsys; ++k) {
        const AsmJob& j = *jobs[k];
        const int nfil = j.in.nfil;
        for (int t = 0; t < j.in.ntri; ++t) {
            const size_t nb = size_t(j.ps.nfptr[t + 1] - j.ps.nfptr[t]), nw = size_t(j.ps.wfptr[t + 1] - j.ps.wfptr[t]);
            const size_t need = 8 * (BLK_B * nb + BLK_W * nw + 6 * size_t(nfil)) + 8 * (nb + nw);
            max_pairs = std::max(max_pairs, (long long)std::max(nb, nw));
            if (passes.empty() || (used > 0 && used + need > NEAR_PASS_BYTES)) {
                close();
                passes.emplace_back();
            }
            auto& p = passes.back();
            if (p.empty() || p.back().sys != k) p.push_back({k, t, t});
            p.back().t1 = t + 1;
            used += need;
            items += nb + nw;
            fil += 6 * size_t(nfil);
        }
    }
    close();
    double *d_blk, *d_fil;
    unsigned long long *d_items, *d_cnt;
    int* d_sysof = nullptr;
    if ((r = dl.alloc(ctx, &d_blk, size_t(BLK_B) * most_items)) || (r = dl.alloc(ctx, &d_fil, most_fil)) ||
        (r = dl.alloc(ctx, &d_items, most_items)) || (r = dl.alloc(ctx, &d_cnt, 2)) ||
        (BATCH && (r = dl.alloc(ctx, &d_sysof, most_items))))
        return r;
    auto lanes = jobs[0]->ps.mixed ? near_kernel_lanes<BATCH, true> : near_kernel_lanes<BATCH, false>;
    auto pairs = jobs[0]->ps.mixed ? near_kernel_pairs<BATCH, true> : near_kernel_pairs<BATCH, false>;
    const int npb = persistent_blocks(ctx, pairs, 32 * NEAR_WARPS, 0);
    // pairs a warp walks at once: no more than there can be for every warp
    const int gmax = int(std::max<size_t>(1, std::min<size_t>(32, most_items / (size_t(npb) * NEAR_WARPS))));
    PieceRec* d_recs;
    unsigned* d_leaves;
    if ((r = dl.alloc(ctx, &d_recs, size_t(npb) * NEAR_WARPS * gmax * REC_MAX)) ||
        (r = dl.alloc(ctx, &d_leaves, size_t(npb) * NEAR_WARPS * gmax * REC_LEAVES)))
        return r;
    for (auto& pass : passes) {
        // the systems' places in the workspace, the work lists: all test triangles, then all rows
        std::vector<NearArgs> args(nsys);
        std::vector<int2> work;
        size_t at = 0, fat = 0;
        int nfil = 0;
        for (const Range& g : pass) {
            AsmJob& j = *jobs[g.sys];
            NearArgs& na = j.na;
            na.sys = g.sys;
            na.rest_item = d_items;
            na.rest_sys = d_sysof;
            na.rest_n = d_cnt;
            na.next = d_cnt + 1;
            na.blk0[0] = j.ps.nfptr[g.t0];
            na.blk0[1] = j.ps.wfptr[g.t0];
            na.blk[0] = d_blk + at;
            at += size_t(BLK_B) * size_t(j.ps.nfptr[g.t1] - j.ps.nfptr[g.t0]);
            na.blk[1] = d_blk + at;
            at += size_t(BLK_W) * size_t(j.ps.wfptr[g.t1] - j.ps.wfptr[g.t0]);
            na.fil_out = d_fil + fat;
            na.t0 = g.t0;
            na.t1 = g.t1;
            fat += 6 * size_t(na.nfil) * size_t(g.t1 - g.t0);
            nfil = std::max(nfil, na.nfil);
            args[g.sys] = na;
            for (int t = g.t0; t < g.t1; ++t) work.push_back(make_int2(g.sys, t));
        }
        const int ntests = int(work.size());
        for (const Range& g : pass)
            for (int i = 0; i < jobs[g.sys]->in.nslot; ++i) work.push_back(make_int2(g.sys, i));
        const int nrows = int(work.size()) - ntests;
        int2* d_work;
        NearArgs* d_args = nullptr;
        if ((r = dl.up(ctx, &d_work, work)) || (BATCH && (r = dl.up(ctx, &d_args, args)))) return r;
        const NearArgs& a1 = args[pass[0].sys];
        VP_CUDA(ctx, cudaMemsetAsync(d_cnt, 0, 2 * sizeof(unsigned long long), ctx->stream));
        vp_phase_begin(ctx, PH_NEAR);
        const int lw = lane_warps(ctx, ntests, max_pairs);
        lanes<<<dim3(ntests, lw), 32, 0, ctx->stream>>>(a1, d_args, d_work);
        ctx->launches++;
        if (nfil > 0) {
            near_kernel_filaments<BATCH><<<dim3((ntests + NEAR_WARPS - 1) / NEAR_WARPS, (nfil + 31) / 32), 32 * NEAR_WARPS, 0,
                                           ctx->stream>>>(a1, d_args, d_work, ntests);
            ctx->launches++;
        }
        vp_phase_end(ctx);
        vp_phase_begin(ctx, PH_NEAR_PAIRS);
        if (!jobs[0]->ps.mixed) {
            near_kernel_self64<BATCH><<<ntests, 32 * SELF_WARPS, 0, ctx->stream>>>(a1, d_args, d_work);
            ctx->launches++;
        }
        pairs<<<npb, 32 * NEAR_WARPS, 0, ctx->stream>>>(a1, d_args, d_recs, d_leaves, gmax);
        ctx->launches++;
        vp_phase_end(ctx);
        vp_phase_begin(ctx, PH_NEAR);
        near_kernel_gather<BATCH><<<nrows, GATHER_NT, 0, ctx->stream>>>(a1, d_args, d_work + ntests);
        ctx->launches++;
        vp_phase_end(ctx);
        VP_CUDA(ctx, cudaGetLastError());
    }
    return VP_OK;
}

// the far launches of the job's precision and tile (FP64: 1, 2 or 4 test triangles per tile, mixed: 2, 4 or 8)
int far_dispatch(vp_ctx* ctx, AsmJob& j) {
    if (j.ps.mixed) {
        if (j.tt == 2) return far_launch<float, 2>(ctx, j);
        if (j.tt == 4) return far_launch<float, 4>(ctx, j);
        if (j.tt == 8) return far_launch<float, 8>(ctx, j);
    } else {
        if (j.tt == 1) return far_launch<double, 1>(ctx, j);
        if (j.tt == 2) return far_launch<double, 2>(ctx, j);
        if (j.tt == 4) return far_launch<double, 4>(ctx, j);
    }
    return vp_fail(ctx, VP_ERR_ARG, "far tile not built for this precision");
}
int far_dispatch_batch(vp_ctx* ctx, std::vector<std::unique_ptr<AsmJob>>& jobs, DevList& dl) {
    const bool mixed = jobs[0]->ps.mixed;
    const int tt = jobs[0]->tt;
    for (auto& j : jobs)
        if (j->ps.mixed != mixed) return vp_fail(ctx, VP_ERR_ARG, "one precision for the whole batch");
    if (mixed) {
        if (tt == 2) return far_launch_batch<float, 2>(ctx, jobs, dl);
        if (tt == 4) return far_launch_batch<float, 4>(ctx, jobs, dl);
        if (tt == 8) return far_launch_batch<float, 8>(ctx, jobs, dl);
    } else {
        if (tt == 1) return far_launch_batch<double, 1>(ctx, jobs, dl);
        if (tt == 2) return far_launch_batch<double, 2>(ctx, jobs, dl);
        if (tt == 4) return far_launch_batch<double, 4>(ctx, jobs, dl);
    }
    return vp_fail(ctx, VP_ERR_ARG, "far tile not built for this precision");
}

}  // namespace

// body_sources = 0: the columns of the wake's sheets and filaments alone (explicit_rhs); A's body columns stay zero
int vp_assemble_impl(vp_ctx* ctx, const vp_assembly_options* o, int nnode, const double* x, int ntri, const int* tris,
                     const int* corner_slot, int nslot, int ntouch, const int* touch_pairs, const double* sigma,
                     const double* vinf, int nwnode, const double* wx, int nwtri, const int* wtris, int nfil,
                     const int* fil, vp_system** out, vp_assembly_stats* stats, int body_sources) {
    if (!out) return vp_fail(ctx, VP_ERR_ARG, "null argument");
    *out = nullptr;
    AsmJob j;
    j.in = PairInput{o,     nnode, x,     ntri, tris,  corner_slot, nslot, ntouch, touch_pairs,
                     sigma, vinf,  nwnode, wx,  nwtri, wtris,       nfil,  fil,   body_sources != 0};
    int r;
    if ((r = job_prepare(ctx, j)) || (r = far_dispatch(ctx, j)) || (r = near_launch<false>(ctx, {&j}, j.ps.dl))) return r;
    return job_finish(ctx, j, out, stats);
}

// the batch: every system prepared, then each phase launched once over all of them (one precision for all)
int vp_assemble_batch_impl(vp_ctx* ctx, const vp_assembly_options* o, int nsys, const vp_assembly_input* in,
                           vp_system** out, vp_assembly_stats* stats) {
    if (!out || !in || !o || nsys < 1) return vp_fail(ctx, VP_ERR_ARG, "null argument or empty batch");
    for (int k = 0; k < nsys; ++k) out[k] = nullptr;
    std::vector<std::unique_ptr<AsmJob>> jobs;
    DevList dl;
    int r;
    for (int k = 0; k < nsys; ++k) {
        const vp_assembly_input& w = in[k];
        jobs.emplace_back(new AsmJob());
        jobs.back()->in = PairInput{o,       w.nnode,  w.x,      w.ntri,  w.tris, w.corner_slot, w.nslot,
                                    w.ntouch, w.touch_pairs, w.sigma, w.vinf, w.nwnode, w.wx, w.nwtri,
                                    w.wtris, w.nfil,   w.fil,    true};
        if ((r = job_prepare(ctx, *jobs.back()))) return r;
    }
    std::vector<AsmJob*> all;
    for (auto& j : jobs) all.push_back(j.get());
    if ((r = far_dispatch_batch(ctx, jobs, dl)) || (r = near_launch<true>(ctx, all, dl))) return r;
    for (int k = 0; k < nsys; ++k)
        if ((r = job_finish(ctx, *jobs[k], &out[k], stats ? stats + k : nullptr))) {
            for (int i = 0; i < k; ++i) {
                vp_system_free(out[i]);
                out[i] = nullptr;
            }
            return r;
        }
    return VP_OK;
}
