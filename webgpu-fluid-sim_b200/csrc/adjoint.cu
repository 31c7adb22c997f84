// adjoint.cu -- vector-Jacobian product of the group-walk force and the
// reverse sweep of a kick-drift-kick rollout (extension, no reference
// counterpart).
//
// Force of one interaction (r = c - x, q = r.r + eps^2, s = q^-1/2, G
// applied by the caller):
//     a = m r s^3 - Q'r s^5 + 5/2 (r.Q'r) r s^7          (Q' = 3S - tr(S) I)
// For an upstream adjoint abar (ab) the VJP is
//     mbar  = (ab.r) s^3
//     Q'bar = d(ab.a)/d(q'xx, q'xy, q'yy)
//           = (-ab_x r_x s^5 + 5/2 r_x^2 (ab.r) s^7,
//              -(ab_x r_y + ab_y r_x) s^5 + 5 r_x r_y (ab.r) s^7,
//              -ab_y r_y s^5 + 5/2 r_y^2 (ab.r) s^7)
//     rbar  = m (s^3 ab - 3 s^5 (ab.r) r)
//           - s^5 Q'ab + 5 s^7 (ab.Q'r) r
//           + 5 s^7 (ab.r) Q'r + 5/2 s^7 (r.Q'r) ab - 35/2 s^9 (r.Q'r)(ab.r) r
// and since r = c - x:  xbar -= rbar,  cbar += rbar.  A body-body
// interaction is the monopole case with the source body's position and mass.
//
// Node adjoints go to bodies through the node moments M = sum m_j,
// c = sum m_j x_j / M, S = sum m_j d_j d_j^T (d_j = x_j - c, so dS/dc = 0):
//     xbar_j += m_j cbar_n / M_n + 2 m_j G_n d_jn
//     mbar_j += mbar_n + cbar_n.d_jn / M_n + d_jn^T G_n d_jn
// with G_n the symmetric matrix of dL/dS_n (Sxx, Sxy, Syy from
// Q'xx = 2Sxx - Syy, Q'xy = 3Sxy, Q'yy = 2Syy - Sxx).  Summed over the
// ancestors n of body j these are polynomials in x_j whose coefficients are
// ten path sums; vjp_push_kernel climbs each leaf's ancestors to form them.
#include "bh_internal.cuh"
#include "packed.cuh"

namespace bh {

constexpr int kVjpWarps = 4;
constexpr int kVjpStack = 320;
constexpr int kVjpDfsAt = kVjpStack - 128;  // as in the walk: >= 32 + 96 below the capacity

// A warp's shared memory.  The group's bodies in pairs, read by every lane:
// {x, x', y, y'} and the upstream adjoints {ax, ax', ay, ay'}; their position
// adjoints, as 8 sums for every 4 bodies {x0, x1, x2, x3, y0, y1, y2, y3}.
// Groups per SM below which a block's warps share one (a rollout's gradient,
// limit 1 / 8 / 16 / 32: 65k bodies, 10 groups per SM, 10.9 / 10.9 / 9.67 /
// 9.59 ms; 32k 8.63 / 7.07 / 7.08 / 7.05 ms; 16k 8.09 / 6.60 / 6.61 / 6.57).
constexpr int kVjpSplit = 16;
constexpr int kVjpPairs = 64;  // 128 bodies
struct VjpSmem {
    uint32_t stack[kVjpStack];
    float4 body[kVjpPairs][2];
    float xbar[kVjpPairs / 2][8];
    uint32_t near[64];        // nodes (a step adds at most 32 to fewer than 32)
    uint32_t first[64];       // ranges of bodies: first slot,
    unsigned char count[64];  // and how many
    uint32_t slot[32 * kGroupMaxLeaf];
};

// Warp sums of 8 values by recursive halving: 4 + 2 + 1 exchanges split the
// values between lane halves, 2 more finish the sum.  Afterwards lanes 4k..4k+3
// hold the sum of v[k] (9 shuffles instead of 8 x 5).
__device__ __forceinline__ float warp_reduce_scatter8(float v[8]) {
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
    float a[4], b[2];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float keep = h4 ? v[j + 4] : v[j], send = h4 ? v[j] : v[j + 4];
        a[j] = keep + __shfl_xor_sync(FULL, send, 16);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const float keep = h3 ? a[j + 2] : a[j], send = h3 ? a[j] : a[j + 2];
        b[j] = keep + __shfl_xor_sync(FULL, send, 8);
    }
    float c;
    {
        const float keep = h2 ? b[1] : b[0], send = h2 ? b[0] : b[1];
        c = keep + __shfl_xor_sync(FULL, send, 4);
    }
    c += __shfl_xor_sync(FULL, c, 2);
    c += __shfl_xor_sync(FULL, c, 1);
    return c;
}

// node_adj: 8 floats per internal node {cbar.x, cbar.y, mbar, Q'bar xx | xy, yy, -, -}
//
// A lane owns one list entry (a node or a source body) of a batch of 32 and
// runs over the group's bodies, two per packed instruction: the entry's six
// adjoints are plain sums in its registers, one reduction of the body adjoints
// serves 4 bodies x 32 entries, and only the bodies there are cost anything.
// (One body per lane and one entry at a time, every entry paid a reduction of
// its six adjoints over the warp and a partly filled group its empty lanes:
// 65k bodies in 64-body groups 239 us a launch, 103 us now, both with the
// block's warps sharing a group; bound by latency at that size.)
template <int MP>
__global__ void __launch_bounds__(kVjpWarps * 32)
vjp_group_kernel(const GNode* __restrict__ gnode, const float4* __restrict__ node4,
                 const uint2* __restrict__ groups, const uint32_t* __restrict__ ids,
                 const float2* __restrict__ abar, float* __restrict__ node_adj,
                 float2* __restrict__ xbar_slot, float* __restrict__ mbar_slot,
                 const WalkParams P, uint32_t* __restrict__ err) {
    __shared__ VjpSmem smem[kVjpWarps];
    __shared__ uint32_t s_group;
    if (step_failed(err)) return;  // the tree at these positions was not built
    const int lane = threadIdx.x & 31;
    VjpSmem& S = smem[threadIdx.x >> 5];
    const unsigned FULL = 0xFFFFFFFFu;
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t n = P.n, nm1 = n - 1;
    const uint32_t ngroups = P.group_ctr[1];
    const float th2 = __fmul_rn(P.theta, P.theta);
    const float eps2 = P.eps2, G = P.g;
    const f2x E2 = pk(eps2, eps2), CM3 = pk(-3.0f, -3.0f), CM1 = pk(-1.0f, -1.0f);
    const f2x C5 = pk(5.0f, 5.0f), C25 = pk(2.5f, 2.5f), CM175 = pk(-17.5f, -17.5f);
    const f2x ZERO = pk(0.f, 0.f);
    const int turn_mask = P.split ? kVjpWarps - 1 : 0;
    const int my_turn = P.split ? (int)(threadIdx.x >> 5) : 0;

    while (true) {
        uint32_t g = 0;
        if (P.split) {  // the block's warps share a group, batch by batch
            __syncthreads();
            if (threadIdx.x == 0) s_group = atomicAdd(P.group_ctr, 1u);
            __syncthreads();
            g = s_group;
        } else {
            if (lane == 0) g = atomicAdd(P.group_ctr, 1u);
            g = __shfl_sync(FULL, g, 0);
        }
        if (g >= ngroups) break;
        const uint2 grp = __ldg(&groups[g]);
        const uint32_t base = grp.x, nvalid = grp.y;
        const int quads = (int)((nvalid + 3u) / 4u);
        // ---- stage the bodies; past the end, one far away with a zero adjoint,
        // which adds exactly zero everywhere
        float glox = INFINITY, gloy = INFINITY, ghix = -INFINITY, ghiy = -INFINITY;
        for (int rel = lane; rel < 4 * quads; rel += 32) {
            float2 r = make_float2(-kFarAway, -kFarAway), a = make_float2(0.f, 0.f);
            if ((uint32_t)rel < nvalid) {
                const uint32_t sl = base + (uint32_t)rel;
                const float4 o = __ldg(&node4[nm1 + sl]);
                r = make_float2(o.x, o.y);
                a = __ldg(&abar[__ldg(&ids[sl])]);
                glox = fminf(glox, r.x); gloy = fminf(gloy, r.y);
                ghix = fmaxf(ghix, r.x); ghiy = fmaxf(ghiy, r.y);
            }
            float* const d = reinterpret_cast<float*>(&S.body[rel >> 1][0]) + (rel & 1);
            d[0] = r.x;
            d[2] = r.y;
            d[4] = G * a.x;  // the force carries G
            d[6] = G * a.y;
            S.xbar[rel >> 2][rel & 3] = 0.f;
            S.xbar[rel >> 2][4 + (rel & 3)] = 0.f;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            glox = fminf(glox, __shfl_xor_sync(FULL, glox, o));
            gloy = fminf(gloy, __shfl_xor_sync(FULL, gloy, o));
            ghix = fmaxf(ghix, __shfl_xor_sync(FULL, ghix, o));
            ghiy = fmaxf(ghiy, __shfl_xor_sync(FULL, ghiy, o));
        }
        __syncwarp();

        // Add the warp's sums of rbar of 4 bodies (two pairs) to their adjoints.
        auto add_quad = [&](int quad, f2x x0, f2x y0, f2x x1, f2x y1) {
            float v[8];
            upk(x0, v[0], v[1]);
            upk(x1, v[2], v[3]);
            upk(y0, v[4], v[5]);
            upk(y1, v[6], v[7]);
            const float tot = warp_reduce_scatter8(v);  // lanes 4k.. hold the sum of v[k]
            if ((lane & 3) == 0) S.xbar[quad][lane >> 2] -= tot;
        };
        // One node per lane (lane < cnt).
        auto eval_nodes = [&](int cnt) {
            const uint32_t v = lane < cnt ? S.near[lane] : 0u;
            float4 mom = make_float4(kFarAway, kFarAway, 0.f, 0.f), tail = make_float4(0.f, 0.f, 0.f, 0.f);
            if (lane < cnt) ldg_half(&gnode[v].mom, mom, tail);  // {com, mass, Sxx}, {Sxy, Syy}
            const float sxx = mom.w, sxy = tail.x, syy = tail.y, tr = sxx + syy;  // Q' = 3S - tr(S) I
            const f2x CX = pk(mom.x, mom.x), CY = pk(mom.y, mom.y), M = pk(mom.z, mom.z);
            const f2x QXX = pk(3.0f * sxx - tr, 3.0f * sxx - tr), QXY = pk(3.0f * sxy, 3.0f * sxy);
            const f2x QYY = pk(3.0f * syy - tr, 3.0f * syy - tr);
            f2x CB_X = ZERO, CB_Y = ZERO, MB = ZERO, GXX = ZERO, GXY = ZERO, GYY = ZERO;
            auto pair = [&](int p, f2x& rbx, f2x& rby) {
                const float4 b0 = S.body[p][0], b1 = S.body[p][1];
                const f2x PAX = ld_pair(b1, 0), PAY = ld_pair(b1, 1);
                const f2x rx = sub2(CX, ld_pair(b0, 0)), ry = sub2(CY, ld_pair(b0, 1));
                const f2x sv = rsqrt2(fma2(rx, rx, fma2(ry, ry, E2)));
                const f2x s2 = mul2(sv, sv), s3 = mul2(sv, s2), s5 = mul2(s3, s2);
                const f2x ar = fma2(PAX, rx, mul2(PAY, ry));
                const f2x tn = mul2(mul2(s5, ar), CM3);  // -3 s^5 (ab.r)
                rbx = mul2(M, fma2(s3, PAX, mul2(tn, rx)));
                rby = mul2(M, fma2(s3, PAY, mul2(tn, ry)));
                MB = fma2(ar, s3, MB);
                if (MP >= 2) {
                    const f2x s7 = mul2(s5, s2), s9 = mul2(s7, s2), s5n = mul2(s5, CM1);
                    const f2x qrx = fma2(QXX, rx, mul2(QXY, ry));
                    const f2x qry = fma2(QXY, rx, mul2(QYY, ry));
                    const f2x qax = fma2(QXX, PAX, mul2(QXY, PAY));
                    const f2x qay = fma2(QXY, PAX, mul2(QYY, PAY));
                    const f2x rqr = fma2(rx, qrx, mul2(ry, qry));
                    const f2x aqr = fma2(PAX, qrx, mul2(PAY, qry));
                    const f2x f7 = mul2(C5, s7), h7 = mul2(C25, s7);
                    const f2x c1 = fma2(f7, aqr, mul2(mul2(CM175, s9), mul2(rqr, ar)));
                    const f2x f7ar = mul2(f7, ar), h7ar = mul2(h7, ar), h7rqr = mul2(h7, rqr);
                    rbx = fma2(s5n, qax, rbx);
                    rbx = fma2(c1, rx, rbx);
                    rbx = fma2(f7ar, qrx, rbx);
                    rbx = fma2(h7rqr, PAX, rbx);
                    rby = fma2(s5n, qay, rby);
                    rby = fma2(c1, ry, rby);
                    rby = fma2(f7ar, qry, rby);
                    rby = fma2(h7rqr, PAY, rby);
                    GXX = fma2(mul2(PAX, rx), s5n, fma2(mul2(rx, rx), h7ar, GXX));
                    GXY = fma2(fma2(PAX, ry, mul2(PAY, rx)), s5n, fma2(mul2(rx, ry), f7ar, GXY));
                    GYY = fma2(mul2(PAY, ry), s5n, fma2(mul2(ry, ry), h7ar, GYY));
                }
                CB_X = add2(CB_X, rbx);
                CB_Y = add2(CB_Y, rby);
            };
#pragma unroll 1
            for (int q = 0; q < quads; ++q) {
                f2x x0, y0, x1, y1;
                pair(2 * q, x0, y0);
                pair(2 * q + 1, x1, y1);
                add_quad(q, x0, y0, x1, y1);
            }
            if (lane < cnt) {
                float4* const na = reinterpret_cast<float4*>(node_adj + 8 * (size_t)v);
                atomicAdd(na, make_float4(sum_halves(CB_X), sum_halves(CB_Y), sum_halves(MB),
                                          MP >= 2 ? sum_halves(GXX) : 0.f));
                if (MP >= 2)
                    atomicAdd(reinterpret_cast<float2*>(na + 1),
                              make_float2(sum_halves(GXY), sum_halves(GYY)));
            }
            __syncwarp();
        };
        // One source body per lane (lane < cnt): slots S.slot[c0 + lane].
        auto eval_bodies = [&](int c0, int cnt) {
            const uint32_t sj = lane < cnt ? S.slot[c0 + lane] : kSentinel;
            float4 o = make_float4(kFarAway, kFarAway, 0.f, 0.f);
            if (lane < cnt) o = __ldg(&node4[nm1 + sj]);
            const f2x CX = pk(o.x, o.x), CY = pk(o.y, o.y), M = pk(o.z, o.z);
            f2x CB_X = ZERO, CB_Y = ZERO, MB = ZERO;
            auto pair = [&](int p, f2x& rbx, f2x& rby) {
                const float4 b0 = S.body[p][0], b1 = S.body[p][1];
                const f2x PAX = ld_pair(b1, 0), PAY = ld_pair(b1, 1);
                // a body does not pull itself: seen from far away it adds nothing
                const uint32_t at = base + 2u * (uint32_t)p;
                float r0, r1;
                upk(sub2(CX, ld_pair(b0, 0)), r0, r1);
                const f2x rx = pk(sj == at ? kFarAway : r0, sj == at + 1u ? kFarAway : r1);
                const f2x ry = sub2(CY, ld_pair(b0, 1));
                const f2x sv = rsqrt2(fma2(rx, rx, fma2(ry, ry, E2)));
                const f2x s2 = mul2(sv, sv), s3 = mul2(sv, s2);
                const f2x ar = fma2(PAX, rx, mul2(PAY, ry));
                const f2x tn = mul2(mul2(mul2(s3, s2), ar), CM3);
                rbx = mul2(M, fma2(s3, PAX, mul2(tn, rx)));
                rby = mul2(M, fma2(s3, PAY, mul2(tn, ry)));
                MB = fma2(ar, s3, MB);
                CB_X = add2(CB_X, rbx);
                CB_Y = add2(CB_Y, rby);
            };
#pragma unroll 1
            for (int q = 0; q < quads; ++q) {
                f2x x0, y0, x1, y1;
                pair(2 * q, x0, y0);
                pair(2 * q + 1, x1, y1);
                add_quad(q, x0, y0, x1, y1);
            }
            if (lane < cnt) {
                atomicAdd(&xbar_slot[sj], make_float2(sum_halves(CB_X), sum_halves(CB_Y)));
                atomicAdd(&mbar_slot[sj], sum_halves(MB));
            }
            __syncwarp();
        };

        // Same traversal as walk_group_kernel: identical interaction lists.
        int sp = 0, nn = 0, nr = 0;
        int turn = 0;  // batches so far; a split group's are dealt to its warps
        if (n > 1) {
            if (lane == 0) S.stack[0] = 0u;
            sp = 1;
        }
        __syncwarp();
        while (sp > 0) {
            int k = sp < 32 ? sp : 32;
            if (sp > kVjpDfsAt) k = 1;
            const bool has = lane < k;
            const uint32_t v = has ? S.stack[sp - k + lane] : 0u;
            sp -= k;
            const bool inner = has & (v < nm1), leaf = has & (v >= nm1);
            float4 box, tr;
            ldg_half(&gnode[inner ? v : 0u].box, box, tr);
            const uint32_t link = __float_as_uint(tr.z), small = __float_as_uint(tr.w);
            const bool ok = inner & group_accepts(box, tr.x, tr.y, glox, gloy, ghix, ghiy, th2);
            const bool bucket = inner & !ok & ((small & 255u) <= (uint32_t)P.leaf_size);
            const bool push = inner & !ok & !bucket;
            const bool range = bucket | leaf;
            const unsigned mp = __ballot_sync(FULL, push);
            const unsigned mr = __ballot_sync(FULL, range);
            const unsigned mn = __ballot_sync(FULL, ok);
            int npush = 2 * __popc(mp);
            if (sp + npush > kVjpStack) {  // never expected
                if (lane == 0) atomicOr(err, kErrGroupStack);
                npush = 0;
            } else if (push) {
                const int p = sp + 2 * __popc(mp & lt);
                S.stack[p] = link_right(link, nm1);
                S.stack[p + 1] = link_left(link, nm1);
            }
            sp += npush;
            if (ok) S.near[nn + __popc(mn & lt)] = v;
            if (range) {
                const int p = nr + __popc(mr & lt);
                S.first[p] = leaf ? v - nm1 : link_gamma(link) + 1u - (small >> 8);
                S.count[p] = (unsigned char)(leaf ? 1u : small);
            }
            nn += __popc(mn);
            nr += __popc(mr);
            __syncwarp();
            const bool last = sp == 0;
            if (!last & (nn < 32) & (nr < 32)) continue;
            if (nn >= 32 || (last && nn > 0)) {
                // the first 32; the rest (fewer than 32) moves to the front
                while (nn >= 32 || (last && nn > 0)) {
                    const int cnt = nn < 32 ? nn : 32;
                    if ((turn++ & turn_mask) == my_turn) eval_nodes(cnt);
                    const uint32_t rest = cnt + lane < nn ? S.near[cnt + lane] : 0u;
                    __syncwarp();
                    nn -= cnt;
                    if (lane < nn) S.near[lane] = rest;
                    __syncwarp();
                }
            }
            while (nr >= 32 || (last && nr > 0)) {
                // the bodies of up to 32 ranges: one exclusive scan of their counts
                const int cnt = nr < 32 ? nr : 32;
                nr -= cnt;
                const uint32_t f = lane < cnt ? S.first[nr + lane] : 0u;
                const uint32_t c = lane < cnt ? S.count[nr + lane] : 0u;
                uint32_t incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += t;
                }
                const int ns = (int)__shfl_sync(FULL, incl, 31);
                for (uint32_t u = 0; u < c; ++u) S.slot[incl - c + u] = f + u;
                __syncwarp();
                for (int c0 = 0; c0 < ns; c0 += 32)
                    if ((turn++ & turn_mask) == my_turn) eval_bodies(c0, ns - c0 < 32 ? ns - c0 : 32);
                __syncwarp();
            }
        }
        __syncwarp();
        for (uint32_t rel = (uint32_t)lane; rel < nvalid; rel += 32u) {
            const float* const xb = S.xbar[rel >> 2];
            atomicAdd(&xbar_slot[base + rel], make_float2(xb[rel & 3u], xb[4u + (rel & 3u)]));
        }
        __syncwarp();
    }
}

// Push node adjoints down to bodies and add the per-slot adjoints; writes
// xbar/mbar in original body order (accumulating: +=).
__global__ void __launch_bounds__(256)
vjp_push_kernel(const GNode* __restrict__ gnode, const float4* __restrict__ node4,
                const uint32_t* __restrict__ parent, const uint32_t* __restrict__ ids,
                const float* __restrict__ node_adj, const float2* __restrict__ xbar_slot,
                const float* __restrict__ mbar_slot, float2* __restrict__ xbar,
                float* __restrict__ mbar, uint32_t n, int mp) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t nm1 = n - 1;
    // path sums over the ancestors
    double sm = 0, ux = 0, uy = 0, w = 0, gxx = 0, gxy = 0, gyy = 0, gcx = 0, gcy = 0, cgc = 0;
    uint32_t v = (n > 1) ? __ldg(&parent[nm1 + j]) : kSentinel;
    uint32_t guard = 0;
    while (v != kSentinel && v < nm1 && guard++ < 4096u) {
        const float4 mom = __ldg(&gnode[v].mom);
        const float4 na4 = __ldg(reinterpret_cast<const float4*>(node_adj + 8 * (size_t)v));
        const float4 nb4 = __ldg(reinterpret_cast<const float4*>(node_adj + 8 * (size_t)v) + 1);
        const float na[6] = {na4.x, na4.y, na4.z, na4.w, nb4.x, nb4.y};
        const double cx = mom.x, cy = mom.y, M = mom.z;
        sm += na[2];
        if (M > 0.0) {
            ux += na[0] / M;
            uy += na[1] / M;
            w += (na[0] * cx + na[1] * cy) / M;
        }
        if (mp >= 2) {
            // dL/dS from dL/dQ': Q'xx = 2Sxx - Syy, Q'xy = 3Sxy, Q'yy = 2Syy - Sxx
            const double sxx = 2.0 * na[3] - na[5], sxy = 3.0 * na[4], syy = 2.0 * na[5] - na[3];
            // G = [[sxx, sxy/2], [sxy/2, syy]]
            const double hxy = 0.5 * sxy;
            gxx += sxx;
            gxy += hxy;
            gyy += syy;
            const double tx = sxx * cx + hxy * cy, ty = hxy * cx + syy * cy;
            gcx += tx;
            gcy += ty;
            cgc += cx * tx + cy * ty;
        }
        v = __ldg(&parent[v]);
    }
    const float4 me = __ldg(&node4[nm1 + j]);
    const double x = me.x, y = me.y, m = me.z;
    const double gx = gxx * x + gxy * y - gcx, gy = gxy * x + gyy * y - gcy;  // G x - G c
    const double xb_x = m * ux + 2.0 * m * gx;
    const double xb_y = m * uy + 2.0 * m * gy;
    const double mb = sm + (x * ux + y * uy - w) + (x * (gxx * x + gxy * y) + y * (gxy * x + gyy * y)) -
                      2.0 * (x * gcx + y * gcy) + cgc;
    const uint32_t b = __ldg(&ids[j]);
    const float2 xs = xbar_slot[j];
    float2 acc = xbar[b];
    acc.x += (float)(xb_x + xs.x);
    acc.y += (float)(xb_y + xs.y);
    xbar[b] = acc;
    mbar[b] += (float)(mb + mbar_slot[j]);
}

// ---- elementwise steps of the reverse sweep (original body order) ---------
__global__ void adj_init_kernel(const float2* __restrict__ pos, const float2* __restrict__ target,
                                uint32_t n, float2* __restrict__ xbar, float2* __restrict__ vbar,
                                float* __restrict__ mbar, float2* __restrict__ apend,
                                double* __restrict__ loss) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    double part = 0.0;
    if (i < n) {
        const float dx = pos[i].x - target[i].x, dy = pos[i].y - target[i].y;
        const float sc = 2.0f / (float)n;
        xbar[i] = make_float2(sc * dx, sc * dy);
        vbar[i] = make_float2(0.f, 0.f);
        mbar[i] = 0.f;
        apend[i] = make_float2(0.f, 0.f);
        part = ((double)dx * dx + (double)dy * dy) / (double)n;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xFFFFFFFFu, part, o);
    if ((threadIdx.x & 31) == 0 && part != 0.0) atomicAdd(loss, part);
}

// abar = apend + h vbar   (closing kick of the step that ends at this point)
__global__ void adj_pre_kernel(const float2* __restrict__ apend, const float2* __restrict__ vbar,
                               float h, uint32_t n, float2* __restrict__ abar) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    abar[i] = make_float2(apend[i].x + h * vbar[i].x, apend[i].y + h * vbar[i].y);
}

// drift and opening kick: vbar += dt xbar; apend = h vbar
__global__ void adj_post_kernel(const float2* __restrict__ xbar, float2* __restrict__ vbar,
                                float2* __restrict__ apend, float dt, float h, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float2 v = vbar[i];
    v.x += dt * xbar[i].x;
    v.y += dt * xbar[i].y;
    vbar[i] = v;
    apend[i] = make_float2(h * v.x, h * v.y);
}

// ---- launchers -----------------------------------------------------------------
template <int MP>
static void vjp_launch_t(const DeviceBuffers& b, const WalkParams& p, const float2* abar,
                         float* node_adj, float2* xbar_slot, float* mbar_slot, cudaStream_t s) {
    static int bps_cache[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    int& bps = bps_cache[dev & 63];
    if (bps == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, vjp_group_kernel<MP>, kVjpWarps * 32, 0);
        if (bps < 1) bps = 1;
    }
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    uint32_t blocks = (uint32_t)(sms * bps);
    WalkParams q = p;
    q.split = split_groups(b.n, 32u * (uint32_t)p.bpl, sms, kVjpSplit);
    const uint32_t need = q.split ? b.n : (b.n + kVjpWarps - 1) / kVjpWarps;
    if (blocks > need) blocks = need;
    if (blocks < 1) blocks = 1;
    vjp_group_kernel<MP><<<blocks, kVjpWarps * 32, 0, s>>>(
        b.gnode, b.node4, b.groups, b.ids, abar, node_adj, xbar_slot, mbar_slot, q, b.err);
}

void launch_force_vjp(const DeviceBuffers& b, const WalkParams& p, const float2* abar,
                      float* node_adj, float2* xbar_slot, float* mbar_slot, float2* xbar,
                      float* mbar, cudaStream_t s) {
    if (b.n == 0) return;
    if (b.n > 1) cudaMemsetAsync(node_adj, 0, sizeof(float) * 8 * (size_t)(b.n - 1), s);
    cudaMemsetAsync(xbar_slot, 0, sizeof(float2) * (size_t)b.n, s);
    cudaMemsetAsync(mbar_slot, 0, sizeof(float) * (size_t)b.n, s);
    if (p.multipole >= 2) vjp_launch_t<2>(b, p, abar, node_adj, xbar_slot, mbar_slot, s);
    else vjp_launch_t<1>(b, p, abar, node_adj, xbar_slot, mbar_slot, s);
    const int blocks = (int)((b.n + 255) / 256);
    vjp_push_kernel<<<blocks, 256, 0, s>>>(b.gnode, b.node4, b.parent, b.ids, node_adj, xbar_slot,
                                          mbar_slot, xbar, mbar, b.n, p.multipole);
}

void launch_adj_init(const float2* pos, const float2* target, uint32_t n, float2* xbar,
                     float2* vbar, float* mbar, float2* apend, double* loss, cudaStream_t s) {
    cudaMemsetAsync(loss, 0, sizeof(double), s);
    adj_init_kernel<<<(n + 255) / 256, 256, 0, s>>>(pos, target, n, xbar, vbar, mbar, apend, loss);
}

void launch_adj_pre(const float2* apend, const float2* vbar, float h, uint32_t n, float2* abar,
                    cudaStream_t s) {
    adj_pre_kernel<<<(n + 255) / 256, 256, 0, s>>>(apend, vbar, h, n, abar);
}

void launch_adj_post(const float2* xbar, float2* vbar, float2* apend, float dt, float h, uint32_t n,
                     cudaStream_t s) {
    adj_post_kernel<<<(n + 255) / 256, 256, 0, s>>>(xbar, vbar, apend, dt, h, n);
}

}  // namespace bh
