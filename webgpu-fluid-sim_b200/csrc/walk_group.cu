// walk_group.cu -- group tree walk with quadrupole moments (extension).
//
// No reference counterpart as a whole: it replaces bh_vel_step_main
// (barnes_hut.wgsl:48-111) + bh_pos_step_main (:113-120) when the
// configuration asks for the group walk.  The reference's per-body monopole
// walk has a median relative force error of order 1e-2 at theta = 0.5 in 2D;
// this walk reaches <= 1e-3 at the same theta.
//
// One warp owns a group: a maximal subtree of at most G = 32 x BPL bodies, so
// its bodies are contiguous sorted slots inside one Morton cell (the build
// kernel lists the groups).  Fixed runs of G slots would not do: a run that
// straddles a jump of the Z curve has a box spanning far-apart regions and
// opens nearly every node.  (Cutting maximal 2G-body subtrees into G-slot
// runs fills more lanes but opens more nodes; measured slower.  So did
// stack entries that stand for both children of an opened node -- adjacent
// in the Karras numbering, one round trip for the pair -- which halve the
// dependent steps but double the emission work per step and the registers.)  The group
// accepts a node when
//     L^2 < theta^2 d^2,  L = longest side of the node's box,
//     d = distance from the group's box to the node's COM,
// and the node's box lies apart from the group's box (group_accepts); then
// every body of the group meets the per-body test length / |com - x| <
// theta.  Other nodes are opened.  Accepted nodes act through their monopole and
// (multipole order 2) quadrupole about the COM,
//     a = G [ M r/|r|^3 - Q'r/|r|^5 + 5/2 (r.Q'r) r/|r|^7 ],  Q' = 3S - tr(S) I,
// with r = com - x and |r|^2 = r.r + eps^2 (S = second moments about the COM).
// Leaves, and opened nodes of <= leaf_size bodies, are summed body by body.
//
// Traversal: a per-warp stack in shared memory.  Every step each lane takes
// one of the top 32 stack entries, loads the half record the decision needs
// with one 256-bit load, decides without branching (a step is a chain of
// dependent instructions), and the warp compacts the outcomes by ballots into
// a node list, a far list, a list of body ranges and the stack.  A list is
// evaluated when it holds 32 entries (far: 64): nodes and bodies are staged in
// shared memory 32 at a time by the 32 lanes in parallel, then every lane
// runs every entry for its BPL bodies (shared-memory broadcasts, no
// divergence).
// Above kWalkDfsAt entries the warp pops one node per step (plain DFS), which
// keeps the stack below kWalkStack for any tree of depth <= 96; a push that
// would not fit raises kErrGroupStack instead of writing out of bounds.
// Groups are taken from an atomic counter (the walk is persistent).  (Taking
// the next group early, to hide that round trip, lengthened the drain: 800k
// walk 359 -> 395 us.  Sharing one traversal among the groups of a larger
// subtree, through lists in global memory, was twice as slow: the groups'
// union of nodes is 1.7 times one group's, and a list step of one warp takes
// as long as a traversal step here.)
//
// Packed arithmetic: each lane evaluates two interactions per instruction with
// the sm_100 packed FP32 instructions (add/sub/mul/fma .rn.f32x2).  Sub-slots
// (32 bodies, one per lane) go two to a pair; staged entries then hold every
// value twice ({cx,cx,cy,cy}, ...), so a 128-bit shared load yields ready
// operand pairs.  An odd sub-slot takes two list entries per instruction
// instead, from a second staged copy ({cx_j,cx_j+1, ...}): groups of 65..96
// bodies cost 1.5 pairs an entry, not 2 (15% fewer evaluations at 800k).  The
// quadrupole is stored negated so every accumulation is a plain fused
// multiply-add.  With eps^2 > 0 a body's own leaf adds exactly zero (r = 0),
// so no self test is needed.
//
// Far field (far_alpha > 0, extension): an accepted node whose COM lies far
// from the group compared with the group's size (r_g < far_alpha R, r_g the
// group box's half-diagonal, R the distance from the box centre to the COM)
// is not evaluated body by body.  Lanes turn 64 such nodes at a time, two
// each, into the coefficients of a local expansion about the box centre, each
// lane summing its own; at the end of the group the lanes' sums are reduced
// and every body evaluates the expansion once (far_field.cuh).
//
// What bounds it (B200, 800k colliding disks, 128-body groups, leaf 4): 167M
// warp instructions at 58% of the issue slots, 20 warps per SM; the last 14% of
// the launch is the drain of the last groups.  Walk stage before the branch-free
// step, id lists, packed far batches, passes over one loop and the top in one
// step -> now: 800k 389 -> 293 us, 16.8M 7.61 -> 5.53 ms, 64-body groups
// (ensemble of 64 systems, 1.2M bodies) 584 -> 386 us.
#include "bh_internal.cuh"
#include "far_field.cuh"
#include "packed.cuh"

namespace bh {

// Per-warp stack entries.  256 entries were slower (0.391 -> 0.407 ms at 800k):
// more warps reach the one-node-per-step depth guard.
constexpr int kWalkStack = 320;
constexpr int kWalkDfsAt = kWalkStack - 128;  // >= 32 + 96 below the capacity

// A warp's shared memory.  The lists hold node ids and body ranges: a step adds
// at most 32 to fewer than 32 kept ones (far: 64).  32 ranges at a time are
// expanded to slots; nodes and bodies are staged 32 at a time for their
// evaluation.
struct GroupSmem {
    uint32_t stack[kWalkStack];
    // staged nodes, as operand pairs: ent[j][0] = {cx, cx, cy, cy},
    // ent[j][1] = {m, m, -Q'xx, -Q'xx}, ent[j][2] = {-Q'xy, -Q'xy, -Q'yy, -Q'yy};
    // ent2: the same with nodes 2j and 2j + 1 in the two places of each value
    // (never staged at the same time as the leaf records: every bit of shared
    // memory saved is L1 for the node records)
    struct Nodes {
        float4 ent[32][3];
        float4 ent2[16][3];
    };
    // staged leaf records: {x, x, y, y}, {m, m, slot bits, slot bits}; body2: two per entry
    struct Bodies {
        float4 body[32][2];
        float4 body2[16][2];
    };
    union {
        Nodes nodes;
        Bodies bodies;
    };
    uint32_t near[64];         // nodes to evaluate at each body
    uint32_t far[96];          // nodes for the group's local expansion (evaluated 64 at a time)
    uint32_t first[64];        // ranges of bodies to sum one by one: first slot,
    unsigned char count[64];   // and how many
    uint32_t slot[32 * kGroupMaxLeaf];
};

// Far list: two nodes per lane (ids[lane], ids[32 + lane], below cnt <= 64)
// added to the lane's local-expansion sums, both in one packed instruction
// stream.  Not inlined: the coefficient arithmetic is the walk's register peak
// (inlined: 800k 316 against 305 us, 16.8M 6.03 / 5.80 ms; 32 nodes a batch
// instead of 64: 317 us, 6.13 ms).
__device__ __noinline__ void far_batch(const GNode* __restrict__ gnode, const uint32_t* ids,
                                       float (&cacc)[kFarCoeffs], int lane, int cnt, float gcx,
                                       float gcy, float rg2, float eps2) {
    if (lane < cnt) {
        const float lam = __fsqrt_rn(rg2);  // the expansion's length scale
        // (two 128-bit loads: with a 256-bit one in a called function ptxas 12.9 crashes)
        const GNode* gp = &gnode[ids[lane]];
        const float4 a = __ldg(&gp->mom), b = __ldg(&gp->tail);
        float4 c = make_float4(a.x, a.y, 0.f, 0.f), d = make_float4(0.f, 0.f, 0.f, 0.f);
        if (lane + 32 < cnt) {
            const GNode* gq = &gnode[ids[lane + 32]];
            c = __ldg(&gq->mom);
            d = __ldg(&gq->tail);
        }
        far_node_coeffs(cacc, pk(__fsub_rn(gcx, a.x), __fsub_rn(gcx, c.x)),
                        pk(__fsub_rn(gcy, a.y), __fsub_rn(gcy, c.y)), pk(a.z, c.z), pk(a.w, c.w),
                        pk(b.x, d.x), pk(b.y, d.y), lam, eps2);
    }
    __syncwarp();
}

// Register budget: launch bounds for blocks of up to 256 threads with 3
// resident per SM for groups of <= 64 bodies (at most 85 registers, the
// budget of 6 resident 128-thread blocks); for 128-body groups blocks of up
// to 128 threads with 5 resident (96 registers, no spills; with 6 the
// far-field walk spills: 800k 313 against 305 us, 16.8M 5.85 / 5.80 ms; 7 and
// 8 were slower still).  The bound does not depend on the block shape chosen
// at launch (walk_block: 64, 128 or, for groups of <= 64 bodies, 256
// threads), so the shape leaves the warps resident per SM unchanged.
constexpr int walk_max_threads(int bpl) { return bpl >= 4 ? 128 : 256; }
#ifndef BH_WALK_MIN_BLOCKS_128
#define BH_WALK_MIN_BLOCKS_128 5
#endif
constexpr int walk_min_blocks(int bpl) { return bpl >= 4 ? BH_WALK_MIN_BLOCKS_128 : 3; }

// FAR: the far-field variant (Plummer softening, quadrupoles); the other
// instantiations carry none of its code or registers.  COUNT: the
// instrumented walk of bh_walk_stats, which also counts node visits and
// interactions; the stepping walk carries no counters (as a runtime switch
// their four 64-bit sums held 8 registers through the whole traversal and
// cost 5% at 800k and 16.8M bodies, 8% for 64-body groups).  Shared memory:
// one GroupSmem per warp, dynamic (the block shape is chosen at
// launch).
template <int BPL, int MP, bool PLUMMER, bool FAR, bool COUNT, bool SPLIT>
__global__ void __launch_bounds__(walk_max_threads(BPL), walk_min_blocks(BPL))
walk_group_kernel(const GNode* __restrict__ gnode, const float4* __restrict__ node4,
                  const uint2* __restrict__ groups, const uint32_t* __restrict__ ids,
                  float2* __restrict__ pos, float2* __restrict__ vel, float2* __restrict__ acc,
                  const WalkParams P, uint32_t* __restrict__ err) {
    constexpr int NP = (BPL + 1) / 2;  // packed pairs per lane
    extern __shared__ __align__(16) unsigned char walk_smem[];
    GroupSmem* smem = reinterpret_cast<GroupSmem*>(walk_smem);
    wait_previous_kernel();
    if (step_failed(err)) return;  // the tree of this step was not built
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    GroupSmem& S = smem[warp];
    const unsigned FULL = 0xFFFFFFFFu;
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t n = P.n, nm1 = n - 1;
    // SPLIT (few groups): the block's warps walk one group together.  Each
    // does the whole traversal, and evaluates every turn_mask+1-th batch.
    const int turn_mask = SPLIT ? (int)(blockDim.x >> 5) - 1 : 0;
    const int my_turn = SPLIT ? warp : 0;
    const uint32_t ngroups = P.group_ctr[1];  // written by the build kernel
    const float th2 = __fmul_rn(P.theta, P.theta);
    const float eps2 = P.eps2, ecoef = P.eps_coef;
    // With a positive softening the own-leaf term is exactly zero.
    const bool self_test = !(PLUMMER && eps2 > 0.0f);
    constexpr bool counting = COUNT;
    unsigned long long c_vis = 0, c_node = 0, c_body = 0, c_far = 0;
    const int stack_cap = (P.stack_cap > 0 && P.stack_cap < kWalkStack) ? P.stack_cap : kWalkStack;

    // The tree's top five levels in heap order (lane L: heap index L + 1), found
    // once per block: a group's first step takes them together, not one level
    // a step with 1, 2, 4, ... lanes at work (800k step, three handles in
    // rotation, 352 -> 349 us, 16.8M 8.16 -> 8.04 ms).  Not for ensembles, whose
    // groups start at different roots.
    __shared__ uint32_t top[32];
    const bool use_top = P.num_systems == 0;
    if (use_top && warp == 0) {
        const uint32_t j = (uint32_t)lane + 1u;
        uint32_t v = n > 1 && j < 32u ? 0u : kSentinel;
        for (int b = 30 - __clz(j); b >= 0; --b) {
            if (v >= nm1) v = kSentinel;  // below a leaf
            else {
                const uint32_t link = __float_as_uint(__ldg(&gnode[v].trav).z);
                v = (j >> b) & 1u ? link_right(link, nm1) : link_left(link, nm1);
            }
        }
        top[lane] = v;
    }
    __syncthreads();

    while (true) {
        uint32_t g = 0;
        if (SPLIT) {
            __syncthreads();  // the previous group's sums have been read
            if (threadIdx.x == 0) S.slot[0] = atomicAdd(P.group_ctr, 1u);
            __syncthreads();
            g = smem[0].slot[0];
            __syncthreads();
        } else {
            if (lane == 0) g = atomicAdd(P.group_ctr, 1u);
            g = __shfl_sync(FULL, g, 0);
        }
        if (g >= ngroups) break;
        // A group is a subtree of <= 32 x BPL bodies: contiguous sorted slots
        // inside one Morton cell, so its box stays compact.
        const uint2 grp = __ldg(&groups[g]);
        if (grp.x < P.slot_lo || grp.x >= P.slot_hi) continue;  // another shard's group (uniform)
        const uint32_t base = grp.x, nvalid = grp.y;
        const int kmax = (int)((nvalid + 31u) / 32u);  // sub-slots in use (uniform)
        // Ensemble: start at the root of the group's own system.  The system id
        // tops every key, so a system is one subtree, whose Karras index is its
        // first or its last slot.  (Started at the common root, with every node
        // tested against the system's slot range: 435 us, now 388, 64 systems of
        // 1.2M bodies.)
        uint32_t root = 0;
        if (P.num_systems > 0) {
            const uint32_t sys = (uint32_t)(__ldg(&P.sys_keys[base]) >> 32);
            const uint32_t lo = __ldg(&P.sys_off[sys]), hi = __ldg(&P.sys_off[sys + 1]);
            const float4 tail = __ldg(&gnode[lo].tail);  // (a system has at least 256 bodies: inner)
            const bool first = __float_as_uint(tail.z) == lo && __float_as_uint(tail.w) == hi - lo;
            root = first ? lo : hi - 1u;
        }
        float bx[BPL], by[BPL], bm[BPL];
        float glox = INFINITY, gloy = INFINITY, ghix = -INFINITY, ghiy = -INFINITY;
#pragma unroll
        for (int k = 0; k < BPL; ++k) {
            float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
            if ((uint32_t)k * 32u + (uint32_t)lane < nvalid) {
                r = __ldg(&node4[nm1 + base + (uint32_t)k * 32u + (uint32_t)lane]);
                glox = fminf(glox, r.x); gloy = fminf(gloy, r.y);
                ghix = fmaxf(ghix, r.x); ghiy = fmaxf(ghiy, r.y);
            }
            bx[k] = r.x; by[k] = r.y; bm[k] = r.z;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            glox = fminf(glox, __shfl_xor_sync(FULL, glox, o));
            gloy = fminf(gloy, __shfl_xor_sync(FULL, gloy, o));
            ghix = fmaxf(ghix, __shfl_xor_sync(FULL, ghix, o));
            ghiy = fmaxf(ghiy, __shfl_xor_sync(FULL, ghiy, o));
        }
        // Far field: box centre, squared half-diagonal and its square root
        // (the expansion's length scale); off for a group of coincident bodies.
        const float gcx = __fmul_rn(0.5f, __fadd_rn(glox, ghix));
        const float gcy = __fmul_rn(0.5f, __fadd_rn(gloy, ghiy));
        const float ghx = __fsub_rn(ghix, glox), ghy = __fsub_rn(ghiy, gloy);
        const float rg2 = __fmul_rn(0.25f, __fadd_rn(__fmul_rn(ghx, ghx), __fmul_rn(ghy, ghy)));
        // (infinite: no node is far)
        const float far_rg2 = FAR && PLUMMER && P.far_alpha2 > 0.0f && rg2 > 0.0f ? rg2 : INFINITY;
        bool far_used = false;
        float cacc[kFarCoeffs];  // this lane's local-expansion sums
#pragma unroll
        for (int k = 0; k < kFarCoeffs; ++k) cacc[k] = 0.0f;
        // The lane's bodies in packed pairs: pair q holds sub-slots 2q and 2q+1.
        // With an odd number of sub-slots in use the last one is held twice in
        // the last pair, whose halves take alternate list entries.
        const bool odd = kmax & 1;
        const int full = kmax >> 1;  // pairs of two sub-slots
        f2x X[NP], Y[NP], AX[NP], AY[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            X[q] = pk(bx[2 * q], bx[BPL > 1 ? 2 * q + 1 : 0]);
            Y[q] = pk(by[2 * q], by[BPL > 1 ? 2 * q + 1 : 0]);
            AX[q] = pk(0.f, 0.f);
            AY[q] = pk(0.f, 0.f);
        }
        float odd_m = bm[0];
        if (BPL > 1 && odd) {
            constexpr int k2 = BPL > 2 ? 2 : 0;
            const bool third = kmax == 3;
            const float ox = third ? bx[k2] : bx[0], oy = third ? by[k2] : by[0];
            X[NP - 1] = pk(ox, ox);
            Y[NP - 1] = pk(oy, oy);
            odd_m = third ? bm[k2] : bm[0];
        }
        const f2x E2 = pk(eps2, eps2);
        const f2x M25 = pk(-2.5f, -2.5f);

        // The lists are evaluated in passes, one per pair in use: the pairs of
        // two sub-slots over ent / body, the odd one over ent2 / body2 (half as
        // many entries).  All passes run the same loop: the kernel's code has
        // to stay small (with a loop for each case the instruction cache
        // thrashed: 4.1 of 9.7 stall cycles an issue, 800k walk 378 us).
        const int passes = full + (odd ? 1 : 0);
        // squared softening of a pair of interactions
        auto soft = [&](f2x M, float ma, float mb) -> f2x {
            if (PLUMMER) return E2;
            float lo, hi;
            upk(M, lo, hi);
            return pk(ecoef * fmaxf(ma, lo), ecoef * fmaxf(mb, hi));
        };
        auto for_passes = [&](auto&& body) {
#pragma unroll 1
            for (int ps = 0; ps < passes; ++ps) {
                const bool is_odd = ps == full;
                const bool lastp = NP > 1 && (ps == NP - 1 || is_odd);  // which register pair
                const f2x x = lastp ? X[NP - 1] : X[0], y = lastp ? Y[NP - 1] : Y[0];
                f2x ax2 = lastp ? AX[NP - 1] : AX[0], ay2 = lastp ? AY[NP - 1] : AY[0];
                // masses and slots of the two bodies (softening by mass, self test)
                const float ma = is_odd ? odd_m : (lastp ? bm[BPL > 2 ? 2 : 0] : bm[0]);
                const float mb = is_odd ? odd_m : (lastp ? bm[BPL > 2 ? 3 : 0] : bm[BPL > 1 ? 1 : 0]);
                const uint32_t sa = base + (uint32_t)lane + (is_odd ? 32u * (uint32_t)(kmax - 1) : 64u * (uint32_t)ps);
                const uint32_t sb = is_odd ? sa : sa + 32u;
                body(is_odd, x, y, ax2, ay2, ma, mb, sa, sb);
                if (lastp) {
                    AX[NP - 1] = ax2;
                    AY[NP - 1] = ay2;
                } else {
                    AX[0] = ax2;
                    AY[0] = ay2;
                }
            }
        };
        // The staged nodes: multipole interactions.
        auto eval_nodes = [&](int cnt) {
            for_passes([&](bool is_odd, f2x x, f2x y, f2x& ax2, f2x& ay2, float ma, float mb, uint32_t, uint32_t) {
                const float4(*e)[3] = is_odd ? S.nodes.ent2 : S.nodes.ent;
                const int m = is_odd ? (cnt + 1) >> 1 : cnt;
#pragma unroll 4  // four independent entries in flight per lane (measured best)
                for (int j = 0; j < m; ++j) {
                    const float4 e0 = e[j][0], e1 = e[j][1];
                    const f2x M = ld_pair(e1, 0);
                    const f2x rx = sub2(ld_pair(e0, 0), x), ry = sub2(ld_pair(e0, 1), y);
                    const f2x r2 = fma2(rx, rx, fma2(ry, ry, soft(M, ma, mb)));
                    const f2x inv = rsqrt2(r2);
                    const f2x inv2 = mul2(inv, inv);
                    const f2x inv3 = mul2(inv, inv2);
                    if (MP >= 2) {
                        const float4 e2 = e[j][2];
                        const f2x NQXX = ld_pair(e1, 1), NQXY = ld_pair(e2, 0), NQYY = ld_pair(e2, 1);
                        const f2x nqrx = fma2(NQXX, rx, mul2(NQXY, ry));  // -(Q'r)_x
                        const f2x nqry = fma2(NQXY, rx, mul2(NQYY, ry));  // -(Q'r)_y
                        const f2x nrqr = fma2(rx, nqrx, mul2(ry, nqry));  // -r.Q'r
                        const f2x inv5 = mul2(inv3, inv2);
                        // f = m / |r|^3 + 5/2 r.Q'r / |r|^7
                        const f2x f = fma2(mul2(nrqr, M25), mul2(inv5, inv2), mul2(M, inv3));
                        ax2 = fma2(nqrx, inv5, fma2(f, rx, ax2));
                        ay2 = fma2(nqry, inv5, fma2(f, ry, ay2));
                    } else {
                        const f2x mi3 = mul2(M, inv3);
                        ax2 = fma2(mi3, rx, ax2);
                        ay2 = fma2(mi3, ry, ay2);
                    }
                }
            });
        };
        // The bodies listed in S.slot: point masses.  32 leaf records at a time
        // are loaded by the 32 lanes in parallel into shared memory.
        auto eval_bodies = [&](int total) {
            for (int c0 = 0; c0 < total; c0 += 32) {
                const int cnt = (total - c0) < 32 ? (total - c0) : 32;
                __syncwarp();
                {
                    float4 o = make_float4(kFarAway, kFarAway, 0.f, 0.f);
                    float sl = __uint_as_float(kSentinel);
                    if (lane < cnt) {
                        const uint32_t slot = S.slot[c0 + lane];
                        o = __ldg(&node4[nm1 + slot]);
                        sl = __uint_as_float(slot);
                    }
                    if (full > 0) {
                        S.bodies.body[lane][0] = make_float4(o.x, o.x, o.y, o.y);
                        S.bodies.body[lane][1] = make_float4(o.z, o.z, sl, sl);
                    }
                    if (odd) {
                        float* const d = reinterpret_cast<float*>(&S.bodies.body2[lane >> 1][0]) + (lane & 1);
                        d[0] = o.x;
                        d[2] = o.y;
                        d[4] = o.z;
                        d[6] = sl;
                    }
                }
                __syncwarp();
                for_passes([&](bool is_odd, f2x x, f2x y, f2x& ax2, f2x& ay2, float ma, float mb, uint32_t sa, uint32_t sb) {
                    const float4(*e)[2] = is_odd ? S.bodies.body2 : S.bodies.body;
                    const int m = is_odd ? (cnt + 1) >> 1 : cnt;
#pragma unroll 4
                    for (int j = 0; j < m; ++j) {
                        const float4 p0 = e[j][0], p1 = e[j][1];
                        const f2x OM = ld_pair(p1, 0);
                        const f2x rx = sub2(ld_pair(p0, 0), x), ry = sub2(ld_pair(p0, 1), y);
                        const f2x r2 = fma2(rx, rx, fma2(ry, ry, soft(OM, ma, mb)));
                        const f2x inv = rsqrt2(r2);
                        f2x f = mul2(OM, mul2(inv, mul2(inv, inv)));
                        if (self_test) {
                            float f0, f1;
                            upk(f, f0, f1);
                            f = pk(__float_as_uint(p1.z) == sa ? 0.0f : f0,
                                   __float_as_uint(p1.w) == sb ? 0.0f : f1);
                        }
                        ax2 = fma2(f, rx, ax2);
                        ay2 = fma2(f, ry, ay2);
                    }
                });
            }
            __syncwarp();
        };
        int sp = 0, nn = 0, nr = 0, nf = 0;
        int turn = 0;  // batches so far
        if (n > 1) {
            S.stack[lane] = use_top ? top[lane] : root;
            sp = use_top ? 31 : 1;
        }
        bool start = use_top;
        __syncwarp();
        while (sp > 0) {
            int k = sp < 32 ? sp : 32;
            if (sp > kWalkDfsAt) k = 1;
            const uint32_t v = lane < k ? S.stack[sp - k + lane] : kSentinel;
            const bool has = v != kSentinel;
            sp -= k;
            // Without branches: a step is a chain of dependent instructions
            // (~1300 cycles with them), and its lanes differ in what they find.
            const bool inner = has & (v < nm1), leaf = has & (v >= nm1);
            float4 box, tr;
            ldg_half(&gnode[inner ? v : 0u].box, box, tr);
            const uint32_t link = __float_as_uint(tr.z), small = __float_as_uint(tr.w);
            bool ok = inner & group_accepts(box, tr.x, tr.y, glox, gloy, ghix, ghiy, th2);
            bool away = false;
            if (FAR) {
                // far from the group: to its local expansion
                const float rx = __fsub_rn(tr.x, gcx), ry = __fsub_rn(tr.y, gcy);
                const float R2 = __fadd_rn(__fmul_rn(rx, rx), __fmul_rn(ry, ry));
                away = ok & (far_rg2 < __fmul_rn(P.far_alpha2, R2));
            }
            const bool bucket = inner & !ok & ((small & 255u) <= (uint32_t)P.leaf_size);
            bool push = inner & !ok & !bucket;
            bool range = bucket | leaf;
            if (start) {
                // the whole top at once: a node counts if all above it are opened
                const unsigned open = __ballot_sync(FULL, push);
                bool reached = true;
#pragma unroll
                for (int up = 1; up < 5; ++up) {
                    const uint32_t j = ((uint32_t)lane + 1u) >> up;  // ancestor
                    reached &= j == 0u || ((open >> (j - 1u)) & 1u);
                }
                ok &= reached;
                away &= reached;
                range &= reached;
                push &= reached & (lane >= 15);
                if (counting) k = __popc(__ballot_sync(FULL, has & reached));
                start = false;
            }
            const unsigned mp = __ballot_sync(FULL, push);
            const unsigned mr = __ballot_sync(FULL, range);
            const unsigned mn = __ballot_sync(FULL, ok & !away);
            const unsigned mf = FAR ? __ballot_sync(FULL, away) : 0u;
            int npush = 2 * __popc(mp);
            if (sp + npush > stack_cap) {  // never expected
                if (lane == 0) atomicOr(err, kErrGroupStack);
                npush = 0;
            } else if (push) {
                // right child below, left child on top
                const int p = sp + 2 * __popc(mp & lt);
                S.stack[p] = link_right(link, nm1);
                S.stack[p + 1] = link_left(link, nm1);
            }
            sp += npush;
            if (ok) {
                if (FAR && away) S.far[nf + __popc(mf & lt)] = v;
                else S.near[nn + __popc(mn & lt)] = v;
            }
            if (range) {
                const int p = nr + __popc(mr & lt);
                S.first[p] = leaf ? v - nm1 : link_gamma(link) + 1u - (small >> 8);
                S.count[p] = (unsigned char)(leaf ? 1u : small);
            }
            nn += __popc(mn);
            nr += __popc(mr);
            nf += __popc(mf);
            if (counting) c_vis += (unsigned long long)k;
            __syncwarp();
            // Lists are evaluated when full, and whatever they hold once the
            // stack is empty; one call site each keeps the kernel's code
            // (and its instruction-cache footprint) small.
            const bool last = sp == 0;
            if (!last & (nn < 32) & (nr < 32) & (!FAR | (nf < 64))) continue;
            while (nn >= 32 || (last && nn > 0)) {
                const int cnt = nn < 32 ? nn : 32;
                nn -= cnt;
                if (SPLIT && (turn++ & turn_mask) != my_turn) continue;
                float4 mom = make_float4(kFarAway, kFarAway, 0.f, 0.f), tail = make_float4(0.f, 0.f, 0.f, 0.f);
                if (lane < cnt) ldg_half(&gnode[S.near[nn + lane]].mom, mom, tail);
                // {com, mass, Sxx}, {Sxy, Syy}: -Q' = tr(S) I - 3S
                const float sxx = mom.w, sxy = tail.x, syy = tail.y, trS = sxx + syy;
                const float nxx = trS - 3.0f * sxx, nxy = -3.0f * sxy, nyy = trS - 3.0f * syy;
                if (full > 0) {
                    S.nodes.ent[lane][0] = make_float4(mom.x, mom.x, mom.y, mom.y);
                    S.nodes.ent[lane][1] = make_float4(mom.z, mom.z, nxx, nxx);
                    if (MP >= 2) S.nodes.ent[lane][2] = make_float4(nxy, nxy, nyy, nyy);
                }
                if (odd) {
                    float* const d = reinterpret_cast<float*>(&S.nodes.ent2[lane >> 1][0]) + (lane & 1);
                    d[0] = mom.x;
                    d[2] = mom.y;
                    d[4] = mom.z;
                    if (MP >= 2) {
                        d[6] = nxx;
                        d[8] = nxy;
                        d[10] = nyy;
                    }
                }
                __syncwarp();
                eval_nodes(cnt);
                if (counting) c_node += (unsigned long long)cnt * nvalid;
                __syncwarp();
            }
            while (nr >= 32 || (last && nr > 0)) {
                // the bodies of up to 32 ranges: one exclusive scan of their counts
                const int cnt = nr < 32 ? nr : 32;
                nr -= cnt;
                if (SPLIT && (turn++ & turn_mask) != my_turn) continue;
                const uint32_t first = lane < cnt ? S.first[nr + lane] : 0u;
                const uint32_t c = lane < cnt ? S.count[nr + lane] : 0u;
                uint32_t incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += t;
                }
                const int ns = (int)__shfl_sync(FULL, incl, 31);
                for (uint32_t u = 0; u < c; ++u) S.slot[incl - c + u] = first + u;
                if (counting) c_body += (unsigned long long)ns * nvalid;
                eval_bodies(ns);
            }
            if constexpr (FAR) {
                while (nf >= 64 || (last && nf > 0)) {
                    const int cnt = nf < 64 ? nf : 64;
                    nf -= cnt;
                    if (SPLIT && (turn++ & turn_mask) != my_turn) continue;
                    far_batch(gnode, S.far + nf, cacc, lane, cnt, gcx, gcy, far_rg2, eps2);
                    if (counting) c_far += (unsigned long long)cnt;
                    far_used = true;
                }
            }
        }
        if (counting && n > 1) c_body -= nvalid;  // each body met its own leaf once
        __syncwarp();
        // The bodies' positions out of the pairs (nothing else keeps them).
#pragma unroll
        for (int k = 0; k < BPL; ++k) {
            float lo, hi, hi2;
            upk(X[k / 2], lo, hi);
            bx[k] = k & 1 ? hi : lo;
            upk(X[NP - 1], lo, hi2);
            if (odd && k == kmax - 1) bx[k] = lo;
            upk(Y[k / 2], lo, hi);
            by[k] = k & 1 ? hi : lo;
            upk(Y[NP - 1], lo, hi2);
            if (odd && k == kmax - 1) by[k] = lo;
        }
        // Far field: reduce the lane columns (every lane gets the sums) and
        // evaluate the local expansion at each of the lane's bodies.
        float fx[BPL], fy[BPL];
#pragma unroll
        for (int k = 0; k < BPL; ++k) {
            fx[k] = 0.0f;
            fy[k] = 0.0f;
        }
        if (far_used) {
            float c[kFarCoeffs];
#pragma unroll
            for (int k = 0; k < kFarCoeffs; ++k) {
                float v = cacc[k];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
                c[k] = v;
            }
            const float inv_lam = __fdiv_rn(1.0f, __fsqrt_rn(far_rg2));
#pragma unroll
            for (int k = 0; k < BPL; ++k) {
                if ((uint32_t)k * 32u + (uint32_t)lane >= nvalid) continue;
                const float dx = __fmul_rn(__fsub_rn(bx[k], gcx), inv_lam);
                const float dy = __fmul_rn(__fsub_rn(by[k], gcy), inv_lam);
                float ex, ey;
                far_eval(c, dx, dy, ex, ey);
                fx[k] = -__fmul_rn(ex, inv_lam);
                fy[k] = -__fmul_rn(ey, inv_lam);
            }
        }
        __syncwarp();

        // Integrate (same modes as the exact walk).
        float ax[BPL], ay[BPL];
        {
            const float ox = sum_halves(AX[NP - 1]), oy = sum_halves(AY[NP - 1]);
#pragma unroll
            for (int k = 0; k < BPL; ++k) {
                float lo, hi;
                upk(AX[k / 2], lo, hi);
                ax[k] = k & 1 ? hi : lo;
                upk(AY[k / 2], lo, hi);
                ay[k] = k & 1 ? hi : lo;
                if (odd && k == kmax - 1) {
                    ax[k] = ox;
                    ay[k] = oy;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < BPL; ++k) {
            ax[k] = far_used ? __fadd_rn(ax[k], fx[k]) : ax[k];
            ay[k] = far_used ? __fadd_rn(ay[k], fy[k]) : ay[k];
        }
        if (SPLIT) {
            // the warps' shares, added in warp order by the first one
            float2* const mine = reinterpret_cast<float2*>(&S.nodes);
#pragma unroll
            for (int k = 0; k < BPL; ++k) mine[32 * k + lane] = make_float2(ax[k], ay[k]);
            __syncthreads();
            if (warp > 0) continue;
            for (int w = 1; w <= turn_mask; ++w) {
                const float2* const other = reinterpret_cast<const float2*>(&smem[w].nodes);
#pragma unroll
                for (int k = 0; k < BPL; ++k) {
                    ax[k] += other[32 * k + lane].x;
                    ay[k] += other[32 * k + lane].y;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < BPL; ++k) {
            const uint32_t s = base + (uint32_t)k * 32u + (uint32_t)lane;
            if ((uint32_t)k * 32u + (uint32_t)lane >= nvalid) continue;
            const float gx = P.g * ax[k], gy = P.g * ay[k];
            const uint32_t b = __ldg(&ids[s]);
            if (P.mode == kWalkForces) {
                acc[b] = make_float2(gx, gy);
            } else if (P.mode == kWalkEulerKickDrift) {
                float2 vv = vel[b];
                vv.x = __fadd_rn(vv.x, __fmul_rn(gx, P.dt));
                vv.y = __fadd_rn(vv.y, __fmul_rn(gy, P.dt));
                vel[b] = vv;
                pos[b] = make_float2(__fadd_rn(bx[k], __fmul_rn(vv.x, P.dt)),
                                     __fadd_rn(by[k], __fmul_rn(vv.y, P.dt)));
            } else {
                const float hdt = 0.5f * P.dt;
                float2 vv = vel[b];
                vv.x = __fadd_rn(vv.x, __fmul_rn(gx, hdt));
                vv.y = __fadd_rn(vv.y, __fmul_rn(gy, hdt));
                vel[b] = vv;
                acc[b] = make_float2(gx, gy);
            }
        }
    }
    if (counting && lane == 0) {
        atomicAdd(&P.counters[0], c_vis);
        atomicAdd(&P.counters[1], c_node);
        atomicAdd(&P.counters[2], c_body);
        atomicAdd(&P.counters[3], c_far);
    }
}

// Warps per block the group walk may run with (walk_block / 32).
constexpr int kWalkShapes[3] = {2, 4, 8};
constexpr int kWalkDefaultWarps = 4;

static int shape_index(int warps) { return warps == 2 ? 0 : (warps == 8 ? 2 : 1); }

template <int BPL, int MP, bool PL, bool FAR>
static cudaError_t set_walk_attributes() {
    const int smem = (int)(walk_max_threads(BPL) / 32 * sizeof(GroupSmem));
    cudaError_t e = cudaFuncSetAttribute(walk_group_kernel<BPL, MP, PL, FAR, false, false>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(walk_group_kernel<BPL, MP, PL, FAR, false, true>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(walk_group_kernel<BPL, MP, PL, FAR, true, false>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

// Largest walk block for bodies_per_lane `bpl` (its launch bound).
int walk_group_max_block(int bpl) { return walk_max_threads(bpl >= 4 ? 4 : 2); }

// With few groups the walk lasts as long as its longest one (100k bodies: 1.1k
// groups for 2,960 resident warps), so a block's warps walk a group together:
// below 8 groups per SM (a group holds about 0.7 of its limit).  Walk stage,
// one warp / one block per group: 16k bodies in 64-body groups 36.7 / 28.5 us,
// 32k 40.3 / 32.9, 65k (10 groups per SM) 52.3 / 55.3; 128-body groups without
// the far field, 50k 157 / 77, 100k (8 per SM) 199 / 121, 200k 221 / 208; with
// it 50k 104 / 60, 100k 114 / 98, 200k 121 / 160.
// From there to 16 groups per SM two warps share one, but only where the caller
// waits for the result (p.latency): 65k leapfrog 53 -> 47 us, forces of 120k
// bodies 205 -> 130, 200k 221 -> 180, a 65k rollout's gradient 8.29 -> 7.57 ms;
// with other work on the GPU the second traversal costs more than it saves
// (65k steps of three handles in rotation 42 -> 47 us each).
bool split_groups(uint32_t n, uint32_t gmax, int sms, int per_sm) {
    return (double)n < 0.7 * gmax * per_sm * sms;
}

template <int BPL, int MP, bool PL, bool FAR, bool COUNT, bool SPLIT>
static void launch_c(const DeviceBuffers& b, const WalkParams& p, int warps, int dev, int sms,
                     cudaStream_t s) {
    static int blocks_per_sm[64][3] = {};
    const size_t smem = (size_t)warps * sizeof(GroupSmem);
    int& bps = blocks_per_sm[dev & 63][shape_index(warps)];
    if (bps == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &bps, walk_group_kernel<BPL, MP, PL, FAR, COUNT, SPLIT>, warps * 32, smem);
        if (bps < 1) bps = 1;
    }
    // Persistent grid; the number of groups (<= n) is only known on the device.
    uint32_t blocks = (uint32_t)(sms * bps);
    const uint32_t need = SPLIT ? b.n : (b.n + warps - 1) / warps;
    if (blocks > need) blocks = need;
    if (blocks < 1) blocks = 1;
    launch_chained(walk_group_kernel<BPL, MP, PL, FAR, COUNT, SPLIT>, blocks, warps * 32, smem, s,
                   b.gnode, b.node4, b.groups, b.ids, b.pos, b.vel, b.acc, p, b.err);
}

// The counting walk only when bh_walk_stats asks for it (p.count).
template <int BPL, int MP, bool PL, bool FAR = false>
static void launch_t(const DeviceBuffers& b, const WalkParams& p, int warps, cudaStream_t s) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (p.count) launch_c<BPL, MP, PL, FAR, true, false>(b, p, warps, dev, sms, s);
    else if (split_groups(b.n, 32u * BPL, sms, 8))
        launch_c<BPL, MP, PL, FAR, false, true>(b, p, warps, dev, sms, s);
    else if (p.latency && split_groups(b.n, 32u * BPL, sms, 16))
        launch_c<BPL, MP, PL, FAR, false, true>(b, p, 2, dev, sms, s);
    else launch_c<BPL, MP, PL, FAR, false, false>(b, p, warps, dev, sms, s);
}

template <int BPL>
static void launch_bpl(const DeviceBuffers& b, const WalkParams& p, int warps, cudaStream_t s) {
    if (p.multipole >= 2) {
        if (p.plummer && p.far_alpha2 > 0.0f) launch_t<BPL, 2, true, true>(b, p, warps, s);
        else if (p.plummer) launch_t<BPL, 2, true>(b, p, warps, s);
        else launch_t<BPL, 2, false>(b, p, warps, s);
    } else {
        if (p.plummer) launch_t<BPL, 1, true>(b, p, warps, s);
        else launch_t<BPL, 1, false>(b, p, warps, s);
    }
}

template <int BPL>
static cudaError_t set_bpl_attributes() {
    cudaError_t e;
    if ((e = set_walk_attributes<BPL, 2, true, true>()) != cudaSuccess) return e;
    if ((e = set_walk_attributes<BPL, 2, true, false>()) != cudaSuccess) return e;
    if ((e = set_walk_attributes<BPL, 2, false, false>()) != cudaSuccess) return e;
    if ((e = set_walk_attributes<BPL, 1, true, false>()) != cudaSuccess) return e;
    return set_walk_attributes<BPL, 1, false, false>();
}

// Allow every walk variant the dynamic shared memory of its largest block
// shape on the current device (once per device, before any launch or
// capture).
cudaError_t walk_init_attributes() {
    cudaError_t e;
    if ((e = set_bpl_attributes<1>()) != cudaSuccess) return e;
    if ((e = set_bpl_attributes<2>()) != cudaSuccess) return e;
    return set_bpl_attributes<4>();
}

void launch_walk_group(const DeviceBuffers& b, const WalkParams& p, int block, cudaStream_t s) {
    if (b.n == 0) return;
    int warps = block / 32;
    if (warps != 2 && warps != 4 && warps != 8) warps = kWalkDefaultWarps;
    if (warps * 32 > walk_group_max_block(p.bpl)) warps = walk_group_max_block(p.bpl) / 32;
    switch (p.bpl) {
        case 1: launch_bpl<1>(b, p, warps, s); break;
        case 4: launch_bpl<4>(b, p, warps, s); break;
        default: launch_bpl<2>(b, p, warps, s); break;
    }
}

}  // namespace bh
