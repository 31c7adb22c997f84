// walk.cu -- theta-criterion tree walk with the integrator fused in.
//
// Reference: bh_vel_step_main (barnes_hut.wgsl:48-111) + bh_pos_step_main
// (barnes_hut.wgsl:113-120).  Per body the reference pops nodes from a private
// 256-entry stack, skips its own leaf, softens with
// eps = epsMult*sqrt(G*max(m1,m2)*dt), and accepts a node when it is a leaf or
// length/sqrt(d^2+eps^2) < theta; otherwise it pushes both children (dropped
// if the stack is full).
//
// Here one warp walks the tree for T consecutive sorted slots (spatially
// coherent after the Morton sort).  The warp's stack holds {node, the set of
// its bodies that still need the node}.  A step takes the top 32 B / T entries;
// the T / B lanes that share an entry load that node, apply each of their B
// bodies' own criterion to it, add the node's pull on the bodies that accept
// it to their own partial sums, and push the children for the bodies that open
// it.  The lanes' sums are added across the warp at the end.  Every body
// therefore meets exactly the nodes of the reference's per-body walk, each
// with the reference's arithmetic; only the order of the summation differs
// (32 B / T partial sums instead of one running sum).
//
// What bounds it, and why these shapes.  With one body per lane and one node
// per step the walk was a serial chain of dependent loads for few bodies (2k
// bodies: 70 us on 64 warps) and bound by instruction issue for many (800k
// bodies, theta 0.5: 1.09 ms, 81% of the issue slots, 1138 warp instructions
// a body, most of them stack and mask handling).  Several nodes per step cut
// the chain, and B bodies share a step's handling; two bodies share each
// packed FP32 instruction.  Walk stage, B200, start -> T4 B2 / T16 B8 (us):
//   2k 70 -> 16 / 21, 8k 83 -> 19 / 24, 16k 87 -> 20.5 / 24.5,
//   32k 80 -> 28 / 25.5, 64k 63 -> 37 / 30, 50k planetary disk 159 -> 47 / 39,
//   800k theta 0.5: 1090 -> 953 / 555, theta 0.7: 623 -> 600 / 355.
// Also measured at 800k, theta 0.5 (us): T8 B8 586, T8 B4 682, T16 B4 713,
// T32 B8 595, T32 B4 808.  T8 B4 is 2 us better than T16 B8 at 32k, no more.
//
// Own-body data comes from the sorted leaf records (node4[n-1+slot]), which
// the fill wrote from pos/mass at the start of the step, so the drift can
// write pos[] in the same kernel without racing other warps' reads.
//
// Extension: leaf buckets.  With leaf_size L > 1 an opened node of <= L bodies
// is summed directly over its contiguous sorted slots instead of being
// descended (more accurate than the monopoles it would otherwise accept).
#include "bh_internal.cuh"
#include "packed.cuh"

namespace bh {

constexpr int kExactWarps = 4;
// Per-warp stack entries.  Above kExactDfsAt the warp pops one node per step
// (plain depth-first), which adds one entry per level: trees are at most 96
// levels deep (64 key bits + 32 index bits), so the stack stays in bounds.
constexpr int kExactStack = 320;
constexpr int kExactDfsAt = kExactStack - 128;

// A body set of a stack entry, one bit per body of the warp.
template <int T>
struct MaskOf { using type = unsigned char; };
template <>
struct MaskOf<16> { using type = unsigned short; };

// Sums over groups of W consecutive lanes of V values per lane: log2(V)
// exchange steps split the values between lane halves, the rest finish the
// sum.  Lane r of a group ends with the sum of v[r / (W / V)].
template <int V, int W>
__device__ __forceinline__ float lanes_reduce_scatter(float (&v)[V]) {
    static_assert(V <= W, "at least one lane per value");
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int h = V / 2, o = W / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int j = 0; j < h; ++j) {
            const float keep = up ? v[j + h] : v[j], send = up ? v[j] : v[j + h];
            v[j] = keep + __shfl_xor_sync(FULL, send, o);
        }
    }
    float s = v[0];
#pragma unroll
    for (int o = W / V / 2; o >= 1; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
    return s;
}

// T: bodies per warp; B: bodies per lane (T / B lanes share a node, each for
// its own B bodies; NPS = 32 B / T nodes per step).  COUNT: the instrumented
// walk of bh_walk_stats (node visits and interactions, per body).
template <int MODE, bool PLUMMER, bool BUCKETS, int T, int B, bool COUNT>
__global__ void __launch_bounds__(kExactWarps * 32)
walk_kernel(const float4* __restrict__ node4, const uint2* __restrict__ children,
            const uint2* __restrict__ range, const uint32_t* __restrict__ ids,
            float2* __restrict__ pos, float2* __restrict__ vel, float2* __restrict__ acc,
            const WalkParams P, uint32_t* __restrict__ err) {
    constexpr int NP = B / 2, NPS = 32 * B / T;
    using Mask = typename MaskOf<T>::type;
    __shared__ uint32_t s_node[kExactWarps][kExactStack];
    __shared__ Mask s_mask[kExactWarps][kExactStack];
    wait_previous_kernel();
    if (step_failed(err)) return;  // the tree of this step was not built
    const int stack_cap = (P.stack_cap > 0 && P.stack_cap < kExactStack) ? P.stack_cap : kExactStack;
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int part = lane / NPS, item = lane % NPS;  // bodies [part B, part B + B); entry of the step
    const uint32_t n = P.n, nm1 = n - 1;
    const uint32_t slot0 = (blockIdx.x * kExactWarps + (uint32_t)w) * T;
    if (slot0 >= n) return;
    const uint32_t cnt = n - slot0 < (uint32_t)T ? n - slot0 : (uint32_t)T;
    const uint32_t mine0 = slot0 + (uint32_t)(part * B);  // first slot of the lane's bodies
    uint32_t* const stk = s_node[w];
    Mask* const stm = s_mask[w];

    // The lane's bodies, in pairs (one past the end repeats the last body; its
    // bit is in no mask).
    f2x X[NP], Y[NP], AX[NP], AY[NP];
    float bm[B];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        const float4 a = __ldg(&node4[nm1 + min(mine0 + 2u * q, nm1)]);
        const float4 b = __ldg(&node4[nm1 + min(mine0 + 2u * q + 1u, nm1)]);
        X[q] = pk(a.x, b.x);
        Y[q] = pk(a.y, b.y);
        bm[2 * q] = a.z;
        bm[2 * q + 1] = b.z;
        AX[q] = pk(0.f, 0.f);
        AY[q] = pk(0.f, 0.f);
    }
    const f2x E2 = pk(P.eps2, P.eps2), EC = pk(P.eps_coef, P.eps_coef);
    uint32_t n_vis = 0, n_node = 0, n_body = 0;  // instrumented launch only

    // Distance terms of pair q to a node: rx, ry and 1/sqrt(r.r + eps^2).
    auto pair_terms = [&](int q, const float4& nd, f2x& rx, f2x& ry) -> f2x {
        rx = sub2(pk(nd.x, nd.x), X[q]);
        ry = sub2(pk(nd.y, nd.y), Y[q]);
        const f2x d2 = fma2(rx, rx, mul2(ry, ry));
        if (PLUMMER) return rsqrt2(add2(d2, E2));
        return rsqrt2(fma2(EC, pk(fmaxf(bm[2 * q], nd.z), fmaxf(bm[2 * q + 1], nd.z)), d2));
    };
    // Add the pull of mass gm = G m on the bodies of pair q whose bits are set.
    auto pair_add = [&](int q, f2x rx, f2x ry, f2x inv, float gm, unsigned bits) {
        const f2x f = mul2(pk(gm, gm), mul2(mul2(inv, inv), inv));
        float f0, f1;
        upk(f, f0, f1);
        f0 = (bits >> (2 * q)) & 1u ? f0 : 0.0f;
        f1 = (bits >> (2 * q + 1)) & 1u ? f1 : 0.0f;
        const f2x g = pk(f0, f1);
        AX[q] = fma2(g, rx, AX[q]);
        AY[q] = fma2(g, ry, AY[q]);
    };

    if (lane == 0) {
        stk[0] = 0u;
        stm[0] = (Mask)((1u << cnt) - 1u);
    }
    int sp = 1;
    __syncwarp();
    while (sp > 0) {
        int k = sp < NPS ? sp : NPS;
        if (sp > kExactDfsAt) k = 1;
        sp -= k;
        unsigned open = 0u;
        uint2 ch = make_uint2(0u, 0u);
        if (item < k) {
            const uint32_t node = stk[sp + item];
            const unsigned need = ((unsigned)stm[sp + item] >> (part * B)) & ((1u << B) - 1u);
            const bool leaf = node >= nm1;
            const float4 nd = __ldg(&node4[node]);
            uint2 rg = make_uint2(0u, 0u);
            if (!leaf) {
                ch = __ldg(&children[node]);
                if (BUCKETS) rg = __ldg(&range[node]);
            }
            const float gm = P.g * nd.z;
            // a body does not pull itself
            const uint32_t own = node - nm1 - mine0;
            const unsigned others = leaf && own < (uint32_t)B ? ~(1u << own) : ~0u;
            unsigned far = 0u;
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                f2x rx, ry;
                const f2x inv = pair_terms(q, nd, rx, ry);
                float i0, i1;
                upk(inv, i0, i1);
                unsigned ok = (nd.w * i0 < P.theta ? 1u : 0u) | (nd.w * i1 < P.theta ? 2u : 0u);
                if (leaf) ok = 3u;
                ok &= need >> (2 * q);
                far |= ok << (2 * q);
                pair_add(q, rx, ry, inv, gm, (ok << (2 * q)) & others);
            }
            open = need & ~far;
            if (COUNT) {
                n_vis += __popc(need);
                if (leaf) n_body += __popc(need & others);
                else n_node += __popc(far);
            }
            if (BUCKETS && open && rg.y - rg.x < (uint32_t)P.leaf_size) {
                for (uint32_t s = rg.x; s <= rg.y; ++s) {
                    const float4 bj = __ldg(&node4[nm1 + s]);
                    const uint32_t self = s - mine0;
                    const unsigned bits = self < (uint32_t)B ? open & ~(1u << self) : open;
                    const float gj = P.g * bj.z;
#pragma unroll
                    for (int q = 0; q < NP; ++q) {
                        f2x rx, ry;
                        const f2x inv = pair_terms(q, bj, rx, ry);
                        pair_add(q, rx, ry, inv, gj, bits);
                    }
                    if (COUNT) n_body += __popc(bits);
                }
                open = 0u;
            }
        }
        // the bodies of all parts that open the lane's node
        unsigned opened = open << (part * B);
#pragma unroll
        for (int o = NPS; o < 32; o <<= 1) opened |= __shfl_xor_sync(FULL, opened, o);
        unsigned mp = __ballot_sync(FULL, opened != 0u);
        if (NPS < 32) mp &= (1u << NPS) - 1u;  // one bit per node
        const int npush = 2 * __popc(mp);
        if (sp + npush <= stack_cap) {
            if (opened != 0u && part == 0) {
                const int p = sp + 2 * __popc(mp & ((1u << item) - 1u));
                stk[p] = ch.x;
                stk[p + 1] = ch.y;
                stm[p] = (Mask)opened;
                stm[p + 1] = (Mask)opened;
            }
            sp += npush;
        } else if (lane == 0) {
            atomicOr(err, kErrStackOverflow);  // barnes_hut.wgsl:100 drops them silently
        }
        __syncwarp();
    }
    if (COUNT) {
        unsigned long long v = n_vis, nd = n_node, bd = n_body;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v += __shfl_xor_sync(FULL, v, o);
            nd += __shfl_xor_sync(FULL, nd, o);
            bd += __shfl_xor_sync(FULL, bd, o);
        }
        if (lane == 0) {
            atomicAdd(&P.counters[0], v);
            atomicAdd(&P.counters[1], nd);
            atomicAdd(&P.counters[2], bd);
        }
    }
    float vx[B], vy[B];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        upk(AX[q], vx[2 * q], vx[2 * q + 1]);
        upk(AY[q], vy[2 * q], vy[2 * q + 1]);
    }
    const float ax = lanes_reduce_scatter<B, NPS>(vx), ay = lanes_reduce_scatter<B, NPS>(vy);
    constexpr int L = NPS / B;  // lane part NPS + L k finishes the part's body k
    const uint32_t slot = mine0 + (uint32_t)(item / L);
    if (item % L != 0 || slot >= n) return;
    const uint32_t b = __ldg(&ids[slot]);
    if (MODE == kWalkForces) {
        acc[b] = make_float2(ax, ay);
    } else if (MODE == kWalkEulerKickDrift) {
        // barnes_hut.wgsl:110 then :120
        const float4 me = __ldg(&node4[nm1 + slot]);
        float2 v = vel[b];
        v.x = __fadd_rn(v.x, __fmul_rn(ax, P.dt));
        v.y = __fadd_rn(v.y, __fmul_rn(ay, P.dt));
        vel[b] = v;
        pos[b] = make_float2(__fadd_rn(me.x, __fmul_rn(v.x, P.dt)),
                             __fadd_rn(me.y, __fmul_rn(v.y, P.dt)));
    } else {
        const float hdt = 0.5f * P.dt;
        float2 v = vel[b];
        v.x = __fadd_rn(v.x, __fmul_rn(ax, hdt));
        v.y = __fadd_rn(v.y, __fmul_rn(ay, hdt));
        vel[b] = v;
        acc[b] = make_float2(ax, ay);
    }
}

template <int MODE, int T, int B, bool COUNT>
static void launch_tb(const DeviceBuffers& b, const WalkParams& p, cudaStream_t s) {
    const bool buckets = p.leaf_size > 1;
    constexpr uint32_t per_block = kExactWarps * T;
    const uint32_t blocks = (b.n + per_block - 1) / per_block;
#define BH_WALK(PL, BK)                                                                      \
    launch_chained(walk_kernel<MODE, PL, BK, T, B, COUNT>, blocks, kExactWarps * 32, 0, s,    \
        b.node4, b.children, b.range, b.ids, b.pos, b.vel, b.acc, p, b.err)
    if (p.plummer) {
        if (buckets) BH_WALK(true, true); else BH_WALK(true, false);
    } else {
        if (buckets) BH_WALK(false, true); else BH_WALK(false, false);
    }
#undef BH_WALK
}

// Few bodies: many warps of 4 bodies, 16 nodes a step (latency); from
// kExactMany bodies: 16 bodies a warp (fewer instructions).  The two measure
// equal near 24k bodies (figures above).
constexpr uint32_t kExactMany = 24576;
template <int MODE, bool COUNT>
static void launch_mode(const DeviceBuffers& b, const WalkParams& p, cudaStream_t s) {
    if (b.n >= kExactMany) launch_tb<MODE, 16, 8, COUNT>(b, p, s);
    else launch_tb<MODE, 4, 2, COUNT>(b, p, s);
}

void launch_walk(const DeviceBuffers& b, const WalkParams& p, int block, cudaStream_t s) {
    (void)block;
    if (b.n == 0) return;
    switch (p.mode) {
        case kWalkForces:
            if (p.count) launch_mode<kWalkForces, true>(b, p, s);
            else launch_mode<kWalkForces, false>(b, p, s);
            break;
        case kWalkEulerKickDrift: launch_mode<kWalkEulerKickDrift, false>(b, p, s); break;
        default: launch_mode<kWalkKdkClose, false>(b, p, s); break;
    }
}

}  // namespace bh
