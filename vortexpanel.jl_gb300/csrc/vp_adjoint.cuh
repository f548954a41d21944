// Reverse-mode derivatives of the pair-integral kernels for the adjoint (templated on float / double).
//
// A quadrature point contributes W nu(q) s, s = w(x)·m, with w the unit source-triangle velocity
// (src/kernels/source_triangle.jl:75-138) and m a per-pair vector. w depends on the point only through the offsets
// r_a = x - v_a to the source's corners, and on the source's shape through its edge normals nu_e, edge lengths, unit
// normal n (exact form) or its corner offsets d_a and area (multipole form). The functions below return s, the
// derivative of s with respect to the offsets at fixed shape, and the per-point factors of the shape derivatives,
// which the caller sums over the points of a pair and turns into corner derivatives once per pair.
#pragma once
#include "vp_math.cuh"

// shape factors of one exact-kernel point: s depends on the shape through
//   sum_e L_e (nu_e·m)/4pi + Omega (n·m)/4pi, with L_e depending on the edge length through num_e = r_i + r_j + len_e
template <class T>
struct ExactShape {
    T L[3];      // edge logs
    T dLdlen[3]; // dL_e / d len_e = 2 / num_e
    T Om;        // solid angle
};

// sv_exact_vjp in FP64 by few FP64 instructions (vp_f64.cuh): one reciprocal of each denominator, the inverse lengths
// from the square roots' reciprocal square roots
__device__ __forceinline__ double sv_exact_vjp_f64(const SrcKern<double>& S, v3<double> r0, v3<double> r1, v3<double> r2,
                                                   v3<double> r, v3<double> m, int side, double plane_tol,
                                                   v3<double>& g0, v3<double>& g1, v3<double>& g2,
                                                   ExactShape<double>& sh) {
    const double i4pi = 1.0 / (4.0 * vp_pi<double>());
    const v3<double> R[3] = {r0, r1, r2};
    double l[3], il[3], p[3], lbar[3] = {0, 0, 0}, s = 0;
    v3<double> gr[3] = {mk3(0.0, 0.0, 0.0), mk3(0.0, 0.0, 0.0), mk3(0.0, 0.0, 0.0)};
#pragma unroll
    for (int a = 0; a < 3; ++a) l[a] = f64::sqrt_inv(dot(R[a], R[a]), il[a]);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const int i = e, j = (e + 1) % 3;
        const v3<double> ri = R[i], rj = R[j];
        p[e] = dot(ri, rj);
        const double num = l[i] + l[j] + S.len[e], n2 = 2.0 * f64::rcp(num);
        const double coef = dot(S.nu[e], m) * i4pi;
        double rden, L;
        if (p[e] < 0.0) {
            const v3<double> c = cross(ri, rj);
            const double den = l[i] * l[j] - p[e], rc2 = f64::rcp(norm2(c));
            rden = f64::rcp(den);
            L = f64::log<-1>(num * num * (den * rc2));
            // d log q: li -> lj/den, lj -> li/den, p -> -1/den, c2 -> -1/c2; c2 = |ri x rj|^2: d/dri = 2 rj x c
            const double k2 = (-2.0 * coef) * rc2;
            gr[i] += k2 * cross(rj, c);
            gr[j] += k2 * cross(c, ri);
            lbar[i] += coef * (n2 + l[j] * rden);
            lbar[j] += coef * (n2 + l[i] * rden);
        } else {
            rden = f64::rcp(l[i] * l[j] + p[e]);
            L = f64::log<-1>(num * num * rden);
            lbar[i] += coef * (n2 - l[j] * rden);
            lbar[j] += coef * (n2 - l[i] * rden);
        }
        const double cp = -coef * rden;
        gr[i] += cp * rj;
        gr[j] += cp * ri;
        s += L * coef;
        sh.L[e] = L;
        sh.dLdlen[e] = n2;
    }
    const double nm = dot(S.n, m) * i4pi;
    const v3<double> c12 = cross(r1, r2);
    const double N = dot(r0, c12);
    const double D = l[0] * l[1] * l[2] + p[0] * l[2] + p[2] * l[1] + p[1] * l[0];
    if (fabs(dot(r, S.n)) <= plane_tol * S.diam) {
        const v3<double> q[3] = {-r0, -r1, -r2};
        sh.Om = side == 0 ? 0.0 : double(side) * 2.0 * vp_pi<double>() * inplane_fraction_rel(q, S.n, S.area, plane_tol);
    } else {
        sh.Om = 2.0 * f64::atan2(N, D);
    }
    // as in the general form: the in-plane branch keeps the one-sided limit of the derivative along the normal
    const double nd2 = N * N + D * D;
    if (nd2 > 0.0) {
        const double h = 2.0 * f64::rcp(nd2);
        const double Nb = nm * D * h, Db = -nm * N * h;
        gr[0] += Nb * c12;
        gr[1] += Nb * cross(r2, r0);
        gr[2] += Nb * cross(r0, r1);
        lbar[0] += Db * (l[1] * l[2] + p[1]);
        lbar[1] += Db * (l[0] * l[2] + p[2]);
        lbar[2] += Db * (l[0] * l[1] + p[0]);
        const double b0 = Db * l[0], b1 = Db * l[1], b2 = Db * l[2];
        gr[0] += b2 * r1 + b1 * r2;
        gr[1] += b2 * r0 + b0 * r2;
        gr[2] += b1 * r0 + b0 * r1;
    }
    s += sh.Om * nm;
#pragma unroll
    for (int a = 0; a < 3; ++a) gr[a] += (lbar[a] * il[a]) * R[a];
    g0 = gr[0];
    g1 = gr[1];
    g2 = gr[2];
    return s;
}

// s = w·m of the exact kernel at fixed shape (nu, len, n from the source) and ds/dr_a.
template <class T, class M = KMath<T>>
__device__ __forceinline__ T sv_exact_vjp(const SrcKern<T>& S, v3<T> r0, v3<T> r1, v3<T> r2, v3<T> r, v3<T> m,
                                          int side, T plane_tol, v3<T>& g0, v3<T>& g1, v3<T>& g2, ExactShape<T>& sh) {
    if constexpr (kPlain64<T, M>) return sv_exact_vjp_f64(S, r0, r1, r2, r, m, side, plane_tol, g0, g1, g2, sh);
    const T i4pi = T(1) / (T(4) * vp_pi<T>());
    const v3<T> R[3] = {r0, r1, r2};
    T l[3] = {M::sqrt(dot(r0, r0)), M::sqrt(dot(r1, r1)), M::sqrt(dot(r2, r2))};
    v3<T> gr[3] = {mk3(T(0), T(0), T(0)), mk3(T(0), T(0), T(0)), mk3(T(0), T(0), T(0))};
    T lbar[3] = {T(0), T(0), T(0)};
    T s = T(0);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const int i = e, j = (e + 1) % 3;
        v3<T> ri = R[i], rj = R[j];
        T p = dot(ri, rj);
        T num = l[i] + l[j] + S.len[e];
        T L, dLdli, dLdlj, dLdp;
        v3<T> c = cross(ri, rj);
        T c2 = norm2(c);
        if (p < T(0)) {
            T den = l[i] * l[j] - p;
            T q = M::div(den, T(2) * c2);
            L = M::log(num * num * q);
            // d log q: li -> lj/den, lj -> li/den, p -> -1/den, c2 -> -1/c2
            dLdli = M::div(T(2), num) + M::div(l[j], den);
            dLdlj = M::div(T(2), num) + M::div(l[i], den);
            dLdp = M::div(-T(1), den);
            T dLdc2 = M::div(-T(1), c2);
            T coef = dot(S.nu[e], m) * i4pi;
            // c2 = |ri x rj|^2: d/dri = 2 rj x c, d/drj = 2 c x ri
            gr[i] += (coef * dLdc2 * T(2)) * cross(rj, c);
            gr[j] += (coef * dLdc2 * T(2)) * cross(c, ri);
        } else {
            T den = l[i] * l[j] + p;
            if constexpr (M::hybrid)
                L = M::log1p(M::div(S.len[e] * num, den));
            else
                L = sizeof(T) == 4 ? T(log1pf(float(S.len[e] * num / den))) : vlog(num * num / (T(2) * den));
            dLdli = M::div(T(2), num) - M::div(l[j], den);
            dLdlj = M::div(T(2), num) - M::div(l[i], den);
            dLdp = M::div(-T(1), den);
        }
        T coef = dot(S.nu[e], m) * i4pi;
        s += L * coef;
        lbar[i] += coef * dLdli;
        lbar[j] += coef * dLdlj;
        gr[i] += (coef * dLdp) * rj;
        gr[j] += (coef * dLdp) * ri;
        sh.L[e] = L;
        sh.dLdlen[e] = M::div(T(2), num);
    }
    T z = dot(r, S.n);
    T nm = dot(S.n, m) * i4pi;
    T N = dot(r0, cross(r1, r2));
    T D = l[0] * l[1] * l[2] + dot(r0, r1) * l[2] + dot(r0, r2) * l[1] + dot(r1, r2) * l[0];
    if (fabs(z) <= plane_tol * S.diam) {
        v3<T> q[3] = {-r0, -r1, -r2};
        sh.Om = side == 0 ? T(0) : T(side) * T(2) * vp_pi<T>() * inplane_fraction_rel(q, S.n, S.area, plane_tol);
    } else {
        sh.Om = T(2) * M::atan2(N, D);
    }
    // 2 atan2(N, D) is smooth across the plane away from the triangle's edges (N = 0, D != 0): in the plane its
    // derivative along the normal is the one-sided limit of the general formula, which the in-plane branch keeps
    if (N * N + D * D > T(0)) {
        T h = M::div(T(2), N * N + D * D);
        T Nb = nm * D * h, Db = -nm * N * h;
        gr[0] += Nb * cross(r1, r2);
        gr[1] += Nb * cross(r2, r0);
        gr[2] += Nb * cross(r0, r1);
        lbar[0] += Db * (l[1] * l[2] + dot(r1, r2));
        lbar[1] += Db * (l[0] * l[2] + dot(r0, r2));
        lbar[2] += Db * (l[0] * l[1] + dot(r0, r1));
        gr[0] += Db * (l[2] * r1 + l[1] * r2);
        gr[1] += Db * (l[2] * r0 + l[0] * r2);
        gr[2] += Db * (l[1] * r0 + l[0] * r1);
    }
    s += sh.Om * nm;
#pragma unroll
    for (int a = 0; a < 3; ++a) gr[a] += M::div(lbar[a], l[a]) * R[a];
    g0 = gr[0];
    g1 = gr[1];
    g2 = gr[2];
    return s;
}

// The mixed adjoint's two evaluators of the touching and contact pairs with the three edges as a loop, their operands rotated
// in registers, the edge's constants read from shared memory (nu: 3 x 3, len: 3). A warp alternates between the two, and
// with the edges unrolled their code (75 KB) did not stay in the instruction caches: 13 of 20 cycles per issue were "no
// instruction". The operations of a point, their order and their fusing (written out where the compiler has a choice) are
// those of the unrolled forms.

// sv_exact_vjp in FP32 under the guard (fp32_guard_ok); false where it refuses
__device__ __forceinline__ bool sv_exact_vjp32(const float* __restrict__ snu, const float* __restrict__ slen, v3<float> n,
                                               float area, float diam, v3<float> r0, v3<float> r1, v3<float> r2,
                                               v3<float> r, v3<float> m, int side, float plane_tol, const Fp32Guard& gd,
                                               float& so, v3<float>& g0, v3<float>& g1, v3<float>& g2,
                                               ExactShape<float>& sh) {
    using M = KMath<float>;
    const float i4pi = 1.f / (4.f * vp_pi<float>());
    float l0 = M::sqrt(dot(r0, r0)), l1 = M::sqrt(dot(r1, r1)), l2 = M::sqrt(dot(r2, r2));
    if (fminf(l0, fminf(l1, l2)) < gd.corner * diam) return false;
    const float N = dot(r0, cross(r1, r2));
    const float l01 = __fmul_rn(l0, l1), P3 = l01 * l2, d01 = dot(r0, r1);
    const float D = fmaf(dot(r1, r2), l0, fmaf(dot(r0, r2), l1, fmaf(l01, l2, __fmul_rn(d01, l2))));
    if (side == 0) {
        if (fabsf(N) < gd.plane * P3 && (D < 0.f || fabsf(D) < gd.plane * P3)) return false;
    }
    g0 = g1 = g2 = mk3(0.f, 0.f, 0.f);
    float b0 = 0.f, b1 = 0.f, b2 = 0.f, s = 0.f;
#pragma unroll 1
    for (int e = 0; e < 3; ++e) {  // the edge from corner offset r0 to r1
        const v3<float> nu = mk3(snu[3 * e], snu[3 * e + 1], snu[3 * e + 2]);
        const float len = slen[e];
        const float p = dot(r0, r1);
        const float num = l0 + l1 + len;
        const float coef = dot(nu, m) * i4pi;
        float L, dLdli, dLdlj, dLdp;
        if (p < 0.f) {
            const v3<float> c = cross(r0, r1);
            const float c2 = norm2(c);
            if (c2 < gd.edge_sin2 * (l0 * l0) * (l1 * l1)) return false;
            const float den = l0 * l1 - p;
            const float q = M::div(den, 2.f * c2);
            L = M::log(num * num * q);
            dLdli = M::div(2.f, num) + M::div(l1, den);
            dLdlj = M::div(2.f, num) + M::div(l0, den);
            dLdp = M::div(-1.f, den);
            const float dLdc2 = M::div(-1.f, c2);
            g0 += (coef * dLdc2 * 2.f) * cross(r1, c);
            g1 += (coef * dLdc2 * 2.f) * cross(c, r0);
        } else {
            const float den = l0 * l1 + p;
            L = log1pf(len * num / den);
            dLdli = M::div(2.f, num) - M::div(l1, den);
            dLdlj = M::div(2.f, num) - M::div(l0, den);
            dLdp = M::div(-1.f, den);
        }
        s += L * coef;
        b0 += coef * dLdli;
        b1 += coef * dLdlj;
        g0 += (coef * dLdp) * r1;
        g1 += (coef * dLdp) * r0;
        sh.L[0] = sh.L[1];
        sh.L[1] = sh.L[2];
        sh.L[2] = L;
        sh.dLdlen[0] = sh.dLdlen[1];
        sh.dLdlen[1] = sh.dLdlen[2];
        sh.dLdlen[2] = M::div(2.f, num);
        const v3<float> tr = r0, tg = g0;
        const float tl = l0, tb = b0;
        r0 = r1, r1 = r2, r2 = tr;
        g0 = g1, g1 = g2, g2 = tg;
        l0 = l1, l1 = l2, l2 = tl;
        b0 = b1, b1 = b2, b2 = tb;
    }
    const float z = dot(r, n);
    const float nm = dot(n, m) * i4pi;
    if (fabs(z) <= plane_tol * diam) {
        const v3<float> q[3] = {-r0, -r1, -r2};
        sh.Om = side == 0 ? 0.f : float(side) * 2.f * vp_pi<float>() * inplane_fraction_rel(q, n, area, plane_tol);
    } else {
        sh.Om = 2.f * M::atan2(N, D);
    }
    auto lin = [](float a, v3<float> x, float b, v3<float> y) {
        return mk3(fmaf(a, x.x, __fmul_rn(b, y.x)), fmaf(a, x.y, __fmul_rn(b, y.y)), fmaf(a, x.z, __fmul_rn(b, y.z)));
    };
    const float nd = fmaf(N, N, __fmul_rn(D, D));
    if (nd > 0.f) {
        const float h = M::div(2.f, nd);
        const float Nb = nm * D * h, Db = -nm * N * h;
        g0 += Nb * cross(r1, r2);
        g1 += Nb * cross(r2, r0);
        g2 += Nb * cross(r0, r1);
        b0 += Db * fmaf(l1, l2, dot(r1, r2));
        b1 += Db * fmaf(l0, l2, dot(r0, r2));
        b2 += Db * __fadd_rn(l01, d01);
        g0 += Db * lin(l2, r1, l1, r2);
        g1 += Db * lin(l2, r0, l0, r2);
        g2 += Db * lin(l1, r0, l0, r1);
    }
    s += sh.Om * nm;
    g0 += M::div(b0, l0) * r0;
    g1 += M::div(b1, l1) * r1;
    g2 += M::div(b2, l2) * r2;
    so = s;
    return true;
}

// The mixed path's FP64 points (where FP32 cancels), split by what cancels: the offsets' lengths, the edges' dot and
// cross products, the stable forms l_i l_j + r_i.r_j, the solid angle's numerator and denominator and the vectors
// l_k r_j + l_j r_k are formed in FP64 (with KMathHyb's square root), and the functions and the derivative algebra on
// them run in FP32, where no difference of nearly equal terms is left. The same s, ds/dr_a and shape factors as
// sv_exact_vjp<double, KMathHyb>, at FP32 accuracy, with about a quarter of its FP64 work. Returns false, with the
// outputs unset, for a point so near a corner or an edge's line that the terms leave FP32's range (a corner offset
// under 1e-10, an edge cross product |c|^2 under 1e-30); the caller takes that point wholly in FP64.
__device__ __forceinline__ bool sv_exact_vjp_split(const double* __restrict__ snu, const double* __restrict__ slen,
                                                   v3<double> n, double area, double diam, v3<double> r0, v3<double> r1,
                                                   v3<double> r2, v3<double> r, v3<float> m, int side, double plane_tol,
                                                   float& svo, v3<float>& g0, v3<float>& g1, v3<float>& g2,
                                                   ExactShape<float>& sh) {
    double L0 = KMathHyb::sqrt(dot(r0, r0)), L1 = KMathHyb::sqrt(dot(r1, r1)), L2 = KMathHyb::sqrt(dot(r2, r2));
    if (!(fmin(L0, fmin(L1, L2)) > 1e-10)) return false;
    const double N64 = dot(r0, cross(r1, r2));
    const double D64 = L0 * L1 * L2 + dot(r0, r1) * L2 + dot(r0, r2) * L1 + dot(r1, r2) * L0;
    const v3<float> V0 = f3(L2 * r1 + L1 * r2), V1 = f3(L2 * r0 + L0 * r2), V2 = f3(L1 * r0 + L0 * r1);
    const double z = dot(r, n);
    const float N = float(N64), D = float(D64);
    // the solid angle's derivative factors 2 (D, N) / (N^2 + D^2), formed in FP64: the squares of N and D leave
    // FP32's range where the offsets are small
    const double nd2 = N64 * N64 + D64 * D64;
    const double hnd = nd2 > 0.0 ? KMathHyb::div(2.0, nd2) : 0.0;
    const float hD = float(hnd * D64), hN = float(hnd * N64);
    const float i4pi = 1.f / (4.f * vp_pi<float>());
    float b0 = 0.f, b1 = 0.f, b2 = 0.f, sv = 0.f, t0 = 0.f, t1 = 0.f, t2 = 0.f;
    v3<float> h0 = mk3(0.f, 0.f, 0.f), h1 = h0, h2 = h0, c0 = h0, c1 = h0, c2 = h0;
#pragma unroll 1
    for (int e = 0; e < 3; ++e) {  // the edge from corner offset r0 to r1
        const double pe = dot(r0, r1);
        const v3<double> ce = cross(r0, r1);
        const double lilj = L0 * L1;
        // l_i l_j + p without cancellation: |c|^2 / (l_i l_j - p) where p < 0
        const double c2e = norm2(ce);
        if (pe < 0.0 && !(c2e > 1e-30)) return false;
        const double se = pe < 0.0 ? KMathHyb::div(c2e, lilj - pe) : lilj + pe;
        const float cc = float(c2e), p = float(pe), st = float(se), li = float(L0), lj = float(L1);
        const v3<float> c = f3(ce), ri = f3(r0), rj = f3(r1);
        // FP32 from here
        const float len = float(slen[e]);
        const float num = li + lj + len;
        const v3<float> nu = mk3(float(snu[3 * e]), float(snu[3 * e + 1]), float(snu[3 * e + 2]));
        const float coef = dot(nu, m) * i4pi;
        float L, dLdli, dLdlj, dLdp;
        if (p < 0.f) {
            const float den = li * lj - p;
            L = logf(num * num * (den / (2.f * cc)));
            dLdli = 2.f / num + lj / den;
            dLdlj = 2.f / num + li / den;
            dLdp = -1.f / den;
            const float k2 = coef * (-1.f / cc) * 2.f;
            h0 += k2 * cross(rj, c);
            h1 += k2 * cross(c, ri);
        } else {
            const float den = st;
            L = log1pf(len * num / den);
            dLdli = 2.f / num - lj / den;
            dLdlj = 2.f / num - li / den;
            dLdp = -1.f / den;
        }
        sv += L * coef;
        b0 += coef * dLdli;
        b1 += coef * dLdlj;
        h0 += (coef * dLdp) * rj;
        h1 += (coef * dLdp) * ri;
        sh.L[0] = sh.L[1];
        sh.L[1] = sh.L[2];
        sh.L[2] = L;
        sh.dLdlen[0] = sh.dLdlen[1];
        sh.dLdlen[1] = sh.dLdlen[2];
        sh.dLdlen[2] = 2.f / num;
        const v3<double> tr = r0;
        const v3<float> th = h0;
        const double tl = L0;
        const float tb = b0;
        r0 = r1, r1 = r2, r2 = tr;
        h0 = h1, h1 = h2, h2 = th;
        L0 = L1, L1 = L2, L2 = tl;
        b0 = b1, b1 = b2, b2 = tb;
        c0 = c1, c1 = c2, c2 = c;
        t0 = t1, t1 = t2, t2 = st;
    }
    const float nm = dot(f3(n), m) * i4pi;
    if (fabs(z) <= plane_tol * diam)
        sh.Om = side == 0 ? 0.f : float(side) * 2.f * vp_pi<float>() * inplane_fraction32(r0, r1, r2, n, area, plane_tol);
    else
        sh.Om = 2.f * atan2f(N, D);
    if (nd2 > 0.0) {
        const float Nb = nm * hD, Db = -nm * hN;
        h0 += Nb * c1;
        h1 += Nb * c2;
        h2 += Nb * c0;
        b0 += Db * t1;
        b1 += Db * t2;
        b2 += Db * t0;
        h0 += Db * V0;
        h1 += Db * V1;
        h2 += Db * V2;
    }
    sv += sh.Om * nm;
    h0 += (b0 / float(L0)) * f3(r0);
    h1 += (b1 / float(L1)) * f3(r1);
    h2 += (b2 / float(L2)) * f3(r2);
    if (!(isfinite(sv) && isfinite(h0.x + h0.y + h0.z + h1.x + h1.y + h1.z + h2.x + h2.y + h2.z))) return false;
    svo = sv;
    g0 = h0;
    g1 = h1;
    g2 = h2;
    return true;
}

// The multipole form in FP64 with its derivatives, by few FP64 instructions (as sv_far_f64): with F·m = A r·m + sum_a c_a
// d_a·m, everything unscaled by the area's factor k = area / 4pi, which is returned: w = k wu, s = k su, ds/dr = k gu,
// ds/dd_a = k gdu_a, ds/darea = su / 4pi. e_a = dF·m/d(d_a·r) serves both ds/dr and ds/dd_a.
__device__ __forceinline__ double sv_far_vjp_f64(const SrcKern<double>& S, v3<double> r, v3<double> m, v3<double>& wu,
                                                 double& su, v3<double>& gu, v3<double>* gdu) {
    double iR2, iR3;
    inv_r23(dot(r, r), iR2, iR3);
    const double iR5 = iR3 * iR2, iR7 = iR5 * iR2, iR9 = iR7 * iR2, iR11 = iR9 * iR2;
    const double rm = dot(r, m);
    double dr[3] = {dot(S.d[0], r), dot(S.d[1], r), 0}, dm[3] = {dot(S.d[0], m), dot(S.d[1], m), 0};
    dr[2] = -(dr[0] + dr[1]);
    dm[2] = -(dm[0] + dm[1]);
    double S2 = 0, S3 = 0, T1 = 0, Sd = 0, B = 0, c[3], e[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double dd = dot(S.d[a], S.d[a]), dr2 = dr[a] * dr[a];
        S2 += dr2;
        S3 += dr2 * dr[a];
        T1 += dd * dr[a];
        Sd += dd;
        const double q = dd * (1.0 / 20) - 0.25 * dr[a], u = iR7 * dr[a];
        c[a] = iR5 * q - (0.25 * iR7) * dr2;
        e[a] = rm * (1.25 * u - 0.25 * iR7 * dd + (1.75 * iR9) * dr2) - dm[a] * (0.25 * iR5 + 0.5 * u);
        const double gdd2 = dm[a] * (0.1 * iR5) - rm * (0.25 * iR5 + 0.5 * u);  // 2 dF·m/d dd_a
        B += dm[a] * ((0.875 * iR9) * dr2 - 2.5 * iR7 * q);
        gdu[a] = e[a] * r + gdd2 * S.d[a] + c[a] * m;
    }
    const double P = 0.625 * S2 - 0.25 * T1, S7 = (7.0 / 12) * S3;
    const double A = iR3 - iR5 * (Sd * 0.125) + iR7 * P + iR9 * S7;
    B += rm * (-1.5 * iR5 + iR7 * (0.3125 * Sd) - 3.5 * iR9 * P - 4.5 * iR11 * S7);
    wu = A * r + (c[0] - c[2]) * S.d[0] + (c[1] - c[2]) * S.d[1];
    gu = A * m + (e[0] - e[2]) * S.d[0] + (e[1] - e[2]) * S.d[1] + (2.0 * B) * r;
    su = A * rm + (c[0] - c[2]) * dm[0] + (c[1] - c[2]) * dm[1];
    return S.area * (1.0 / (4.0 * vp_pi<double>()));
}

// s = w·m of the multipole form (source_triangle.jl:100-119) and its derivatives with respect to r = x - c, to the
// corner offsets d_a (gd) and the area (ga)
template <class T>
__device__ __forceinline__ T sv_far_vjp(const SrcKern<T>& S, v3<T> r, v3<T> m, v3<T>& gr, v3<T>* gd, T& ga) {
    if constexpr (sizeof(T) == 8) {
        v3<double> w;
        double su;
        const double k = sv_far_vjp_f64(S, r, m, w, su, gr, gd);
        gr = k * gr;
        for (int a = 0; a < 3; ++a) gd[a] = k * gd[a];
        ga = su * (1.0 / (4.0 * vp_pi<double>()));
        return k * su;
    }
    const T k = S.area / (T(4) * vp_pi<T>());
    T R2 = dot(r, r);
    T iR2, iR3;
    inv_r23(R2, iR2, iR3);
    T iR5 = iR3 * iR2, iR7 = iR5 * iR2, iR9 = iR7 * iR2, iR11 = iR9 * iR2;
    T rm = dot(r, m);
    // F·m = iR3 rm + sum_a g_a(dr, dd, rm, dm, R2)
    T Fm = iR3 * rm;
    v3<T> gF = iR3 * m;  // d(F·m)/dr, accumulated
    T dR2 = T(-1.5) * iR5 * rm;  // d(F·m)/dR2
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        v3<T> d = S.d[a];
        T dr = dot(d, r), dd = dot(d, d), dm = dot(d, m);
        // quad·m / 24 - oct·m / 180
        T g = (T(15) * dr * dr * iR7 * rm - T(6) * dr * iR5 * dm - T(3) * dd * iR5 * rm) / T(24) -
              (T(45) * dr * dr * iR7 * dm - T(105) * dr * dr * dr * iR9 * rm - T(9) * dd * iR5 * dm +
               T(45) * dd * dr * iR7 * rm) / T(180);
        Fm += g;
        T g_dr = (T(30) * dr * iR7 * rm - T(6) * iR5 * dm) / T(24) -
                 (T(90) * dr * iR7 * dm - T(315) * dr * dr * iR9 * rm + T(45) * dd * iR7 * rm) / T(180);
        T g_dd = (-T(3) * iR5 * rm) / T(24) - (-T(9) * iR5 * dm + T(45) * dr * iR7 * rm) / T(180);
        T g_rm = (T(15) * dr * dr * iR7 - T(3) * dd * iR5) / T(24) -
                 (-T(105) * dr * dr * dr * iR9 + T(45) * dd * dr * iR7) / T(180);
        T g_dm = (-T(6) * dr * iR5) / T(24) - (T(45) * dr * dr * iR7 - T(9) * dd * iR5) / T(180);
        // iR_k = R2^(-k/2): d/dR2 = -(k/2) iR_(k+2)
        T g_R2 = (T(15) * dr * dr * (T(-3.5) * iR9) * rm - T(6) * dr * (T(-2.5) * iR7) * dm -
                  T(3) * dd * (T(-2.5) * iR7) * rm) / T(24) -
                 (T(45) * dr * dr * (T(-3.5) * iR9) * dm - T(105) * dr * dr * dr * (T(-4.5) * iR11) * rm -
                  T(9) * dd * (T(-2.5) * iR7) * dm + T(45) * dd * dr * (T(-3.5) * iR9) * rm) / T(180);
        gF += g_dr * d + g_rm * m;
        dR2 += g_R2;
        gd[a] = k * (g_dr * r + (T(2) * g_dd) * d + g_dm * m);
    }
    gF += (T(2) * dR2) * r;
    gr = k * gF;
    ga = Fm / (T(4) * vp_pi<T>());
    return k * Fm;
}

// the two end parts of a filament (segment.jl:15-25) contracted with ca, cb: s = ca (va·n) + cb (vb·n), and its
// derivatives with respect to ra = x - a and rb = x - b
template <class T>
__device__ __forceinline__ T seg_vjp(v3<T> ra, v3<T> rb, v3<T> n, T ca, T cb, v3<T>& ga, v3<T>& gb) {
    T Ra = vnorm(ra), Rb = vnorm(rb);
    v3<T> c = cross(ra, rb);
    T p = dot(ra, rb);
    T den, c2 = norm2(c);
    bool neg = p < T(0);
    den = neg ? c2 / (Ra * Rb - p) : Ra * Rb + p;
    ga = mk3(T(0), T(0), T(0));
    gb = ga;
    if (den == T(0) || Ra == T(0) || Rb == T(0)) return T(0);
    const T i4pi = T(1) / (T(4) * vp_pi<T>());
    T cn = dot(c, n);
    T wsum = ca / Ra + cb / Rb;
    T s = cn * i4pi / den * wsum;
    // s = cn * i4pi * wsum / den
    T s_cn = i4pi * wsum / den;
    T s_den = -s / den;
    T s_Ra = -cn * i4pi / den * ca / (Ra * Ra);
    T s_Rb = -cn * i4pi / den * cb / (Rb * Rb);
    // cn = (ra x rb)·n: d/dra = rb x n, d/drb = n x ra
    ga += s_cn * cross(rb, n);
    gb += s_cn * cross(n, ra);
    if (neg) {  // den = c2 / (Ra Rb - p)
        T q = Ra * Rb - p;
        T d_c2 = T(1) / q, d_q = -c2 / (q * q);
        ga += (s_den * d_c2 * T(2)) * cross(rb, c);
        gb += (s_den * d_c2 * T(2)) * cross(c, ra);
        s_Ra += s_den * d_q * Rb;
        s_Rb += s_den * d_q * Ra;
        ga += (-s_den * d_q) * rb;
        gb += (-s_den * d_q) * ra;
    } else {  // den = Ra Rb + p
        s_Ra += s_den * Rb;
        s_Rb += s_den * Ra;
        ga += s_den * rb;
        gb += s_den * ra;
    }
    ga += (s_Ra / Ra) * ra;
    gb += (s_Rb / Rb) * rb;
    return s;
}
