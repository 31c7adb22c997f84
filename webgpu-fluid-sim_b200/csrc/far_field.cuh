// far_field.cuh -- local (Taylor) expansions of far multipoles for the group
// walk (extension; no reference counterpart).
//
// The group walk evaluates every accepted node at each of the group's bodies
// (a multipole-to-body interaction per body).  A node that is far from the
// group compared with the group's size -- group half-diagonal r_g < alpha R,
// R = |c - x_g| from the group's centre x_g to the node's COM c -- is instead
// turned once into the coefficients of a local expansion of its potential
// about x_g, summed over all such nodes, and the sum is evaluated at each body
// (Cartesian "multipole-to-local" + "local-to-body").
//
// Potential of a node (mass M, second moments S about its COM; G applied by
// the caller), with the Plummer-softened kernel g(R) = (|R|^2 + eps^2)^-1/2:
//     Phi(x) = -[ M g(R) + 1/2 (Sxx g_xx + 2 Sxy g_xy + Syy g_yy) ],  R = x - c.
// Derivatives of g (Faa di Bruno for g = h(|R|^2), h(u) = (u + eps^2)^-1/2):
//     d^(a,b) g = s^(a+b+1) P_ab(rho),  s = (|R|^2 + eps^2)^-1/2,  rho = s R,
//     P_ab = sum_{i<=a/2, j<=b/2} c(a,i) c(b,j) rho_x^(a-2i) rho_y^(b-2j) w(a+b-i-j),
//     c(a,i) = a! / (i! (a-2i)! 2^i),  w(m) = (-1)^m (2m-1)!!
// (evaluated order by order with a recurrence, far_next).
// With the length scale lambda = r_g and t = lambda s (< alpha for a far node)
// the scaled coefficients of orders 1..4 (kFarCoeffs of them) are
//     C_ab = lambda^(a+b) d^(a,b) Phi(x_g)
//          = -s t^(a+b) [ M P_ab + 1/2 (S'xx P_(a+2)b + 2 S'xy P_(a+1)(b+1) + S'yy P_a(b+2)) ],
//     S' = s^2 S,
// all bounded by M s (no overflow for close, dense groups).  At a body
// x = x_g + lambda d (|d| <= 1) the force of all far nodes is the gradient of
// the local expansion truncated at order 4 (cubic in d):
//     a_x = -(1/lambda) sum_{a+b<=3} C_(a+1)b d_x^a d_y^b / (a! b!),
//     a_y = -(1/lambda) sum_{a+b<=3} C_a(b+1) d_x^a d_y^b / (a! b!).
// The truncation error of a node's force is about (r_g / R)^4 of it; with
// alpha = 0.25 a prototype on the 100k colliding disks moved the median
// force error against the FP64 direct sum from 3.8e-4 to 4.2e-4 while 64% of
// the accepted nodes took this path.
#pragma once

#include "bh_internal.cuh"
#include "packed.cuh"

namespace bh {

constexpr int kFarCoeffs = 14;  // potential coefficients of orders 1..4

// Coefficient index of (a, b), 1 <= a + b <= 4: by order, then by b.
__host__ __device__ constexpr int far_idx(int a, int b) {
    return (a + b - 1) * (a + b + 2) / 2 + b;
}
// P_ab of the next order from the two orders below it (prev: order N - 1 by b,
// last: order N), for two nodes at once.  From u dg/dx = -x g, u = |R|^2 + eps^2,
// differentiated a - 1 times in x and b times in y and scaled as above:
//     P_ab = -[ (2a-1) rho_x P_(a-1)b + (a-1)^2 P_(a-2)b
//               + 2b rho_y P_a(b-1) + b(b-1) P_a(b-2) ]        (a >= 1)
// and the same with x and y exchanged for a = 0.  Two to four fused
// multiply-adds per value, half of what the closed sums take.
template <int N>
__device__ __forceinline__ void far_next(f2x (&next)[N + 2], const f2x (&last)[N + 1],
                                         const f2x* prev, f2x rhx, f2x rhy) {
    auto c2 = [](float v) { return pk(v, v); };
#pragma unroll
    for (int b = 0; b <= N; ++b) {
        const int a = N + 1 - b;
        f2x v = mul2(mul2(rhx, last[b]), c2(-(float)(2 * a - 1)));  // P_(a-1)b
        if (a >= 2 && N >= 1) v = fma2(prev[b], c2(-(float)((a - 1) * (a - 1))), v);      // P_(a-2)b
        if (b >= 1) v = fma2(mul2(rhy, last[b - 1]), c2(-(float)(2 * b)), v);             // P_a(b-1)
        if (b >= 2) v = fma2(prev[b - 2], c2(-(float)(b * (b - 1))), v);                  // P_a(b-2)
        next[b] = v;
    }
    f2x v = mul2(mul2(rhy, last[N]), c2(-(float)(2 * N + 1)));
    if (N >= 1) v = fma2(prev[N - 1], c2(-(float)(N * N)), v);
    next[N + 1] = v;
}

// Add the coefficients of order N of two nodes to acc: st = s t^N, p / q = P
// of order N / N + 2, hxx = S'xx / 2, qxy = S'xy, hyy = S'yy / 2.
template <int N>
__device__ __forceinline__ void far_order(float (&acc)[kFarCoeffs], const f2x (&p)[N + 1],
                                          const f2x (&q)[N + 3], f2x m, f2x hxx, f2x qxy, f2x hyy,
                                          f2x st) {
#pragma unroll
    for (int b = 0; b <= N; ++b) {
        const f2x v = fma2(m, p[b], fma2(hxx, q[b], fma2(qxy, q[b + 1], mul2(hyy, q[b + 2]))));
        acc[far_idx(N - b, b)] -= sum_halves(mul2(st, v));
    }
}

// Add the scaled local coefficients (about x_g, length scale lambda) of two
// nodes, one per half, to acc[kFarCoeffs].  R = x_g - c.  A half with m = S = 0
// (and any finite R) adds nothing.
__device__ __forceinline__ void far_node_coeffs(float (&acc)[kFarCoeffs], f2x rx, f2x ry, f2x m,
                                                f2x sxx, f2x sxy, f2x syy, float lambda,
                                                float eps2) {
    const f2x u = fma2(rx, rx, fma2(ry, ry, pk(eps2, eps2)));
    f2x s = rsqrt2(u);
    // One Newton step: s is good to half a unit in the last place or so.  (An
    // overflowed u leaves s = 0 and adds nothing, hence the finite bound.)
    const f2x half = pk(0.5f, 0.5f);
    float u0, u1;
    upk(u, u0, u1);
    const f2x nu = pk(-fminf(u0, 3.0e38f), -fminf(u1, 3.0e38f));
    s = fma2(mul2(s, half), fma2(mul2(nu, s), s, pk(1.f, 1.f)), s);
    const f2x rhx = mul2(rx, s), rhy = mul2(ry, s), s2 = mul2(s, s), t = mul2(pk(lambda, lambda), s);
    const f2x hxx = mul2(mul2(s2, sxx), half), qxy = mul2(s2, sxy), hyy = mul2(mul2(s2, syy), half);
    f2x p0[1] = {pk(1.f, 1.f)}, p1[2], p2[3], p3[4], p4[5], p5[6], p6[7];
    far_next<0>(p1, p0, nullptr, rhx, rhy);
    far_next<1>(p2, p1, p0, rhx, rhy);
    far_next<2>(p3, p2, p1, rhx, rhy);
    f2x st = mul2(s, t);
    far_order<1>(acc, p1, p3, m, hxx, qxy, hyy, st);
    far_next<3>(p4, p3, p2, rhx, rhy);
    st = mul2(st, t);
    far_order<2>(acc, p2, p4, m, hxx, qxy, hyy, st);
    far_next<4>(p5, p4, p3, rhx, rhy);
    st = mul2(st, t);
    far_order<3>(acc, p3, p5, m, hxx, qxy, hyy, st);
    far_next<5>(p6, p5, p4, rhx, rhy);
    st = mul2(st, t);
    far_order<4>(acc, p4, p6, m, hxx, qxy, hyy, st);
}

// Force of the local expansion at offset d = (x - x_g) / lambda:
// (ax, ay) without the factor -1/lambda (the caller applies it).
__device__ __forceinline__ void far_eval(const float* C, float dx, float dy, float& ax, float& ay) {
    const float dxx = __fmul_rn(dx, dx), dxy = __fmul_rn(dx, dy), dyy = __fmul_rn(dy, dy);
    // sum_{a+b<=3} C_(a+1)b d^(a,b) / (a! b!) and C_a(b+1) likewise
    float x = C[far_idx(1, 0)];
    x = __fmaf_rn(C[far_idx(2, 0)], dx, x);
    x = __fmaf_rn(C[far_idx(1, 1)], dy, x);
    x = __fmaf_rn(0.5f * C[far_idx(3, 0)], dxx, x);
    x = __fmaf_rn(C[far_idx(2, 1)], dxy, x);
    x = __fmaf_rn(0.5f * C[far_idx(1, 2)], dyy, x);
    x = __fmaf_rn((1.f / 6.f) * C[far_idx(4, 0)], __fmul_rn(dxx, dx), x);
    x = __fmaf_rn(0.5f * C[far_idx(3, 1)], __fmul_rn(dxx, dy), x);
    x = __fmaf_rn(0.5f * C[far_idx(2, 2)], __fmul_rn(dx, dyy), x);
    x = __fmaf_rn((1.f / 6.f) * C[far_idx(1, 3)], __fmul_rn(dyy, dy), x);
    float y = C[far_idx(0, 1)];
    y = __fmaf_rn(C[far_idx(1, 1)], dx, y);
    y = __fmaf_rn(C[far_idx(0, 2)], dy, y);
    y = __fmaf_rn(0.5f * C[far_idx(2, 1)], dxx, y);
    y = __fmaf_rn(C[far_idx(1, 2)], dxy, y);
    y = __fmaf_rn(0.5f * C[far_idx(0, 3)], dyy, y);
    y = __fmaf_rn((1.f / 6.f) * C[far_idx(3, 1)], __fmul_rn(dxx, dx), y);
    y = __fmaf_rn(0.5f * C[far_idx(2, 2)], __fmul_rn(dxx, dy), y);
    y = __fmaf_rn(0.5f * C[far_idx(1, 3)], __fmul_rn(dx, dyy), y);
    y = __fmaf_rn((1.f / 6.f) * C[far_idx(0, 4)], __fmul_rn(dyy, dy), y);
    ax = x;
    ay = y;
}

}  // namespace bh
