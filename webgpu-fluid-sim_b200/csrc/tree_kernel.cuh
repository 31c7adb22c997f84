// tree_kernel.cuh -- the fused bottom-up hierarchy build + mass / centre-of-mass
// / AABB fill kernel (included by tree.cu, which launches it for the engine).
//
// Reference: build_lbvh_main (lbvh.wgsl:85-165, Karras 2012 fig. 4) followed by
// fill_lbvh_main (lbvh.wgsl:168-232).  The reference builds top-down with one
// thread per internal node and binary searches, then climbs from the leaves
// with arrival counters but no memory fences, which its README calls a race.
//
// Here one thread per sorted slot climbs from its leaf and creates each
// internal node when it is the second child to arrive (agglomerative build,
// Apetrei 2014), using the same delta(i, j) as lbvh.wgsl:72-83:
//   delta = clz(k_i ^ k_j), or key_bits + clz(i ^ j) for equal keys, -1 outside.
// A node covering sorted slots [l, r] is the left child of its parent when
// delta(r, r+1) > delta(l-1, l), and the parent's split is then r; otherwise it
// is the right child and the split is l-1.  Karras numbers an internal node by
// the end of its range next to its parent's split (a left child by its last
// slot, a right child by its first slot, the root is 0), and its children are
// gamma / gamma+1, or the leaves n-1+gamma / n+gamma when a side holds one slot
// (lbvh.wgsl:141-152).  Computing those indices here gives the same
// left/right/parent arrays as the reference's top-down build, bit for bit.
//
// Synchronisation: the two children of a split gamma meet at its slot with
// atomic exchanges of their records; the first arriver (by the range ends'
// word) stops, the second has the other's record from the same exchanges.
// No other data passes between threads, so there are no fences.  A word of
// the sibling that has not landed yet is awaited (bounded; its exchange was
// issued before).  The second arriver empties the slot (all ones between steps).
//
// Two phases per climb.  A CTA owns B consecutive slots (128 in the fused
// build, 512 in the split build's local phase).  A node whose
// range lies inside those slots ("local") is combined through shared memory:
// its split's exchange slot is a shared-memory word, the sibling's record is
// read from shared memory, and block-scope fences suffice.  Which splits are
// local follows from the boundary deltas alone: the node split at boundary g
// spans from just after the nearest boundary on its left with a smaller
// delta to the nearest one on its right with a smaller delta (the hierarchy
// is the Cartesian tree of the boundary deltas, whose values are distinct
// between two smaller ones), so it is local when both of those boundaries
// are among the CTA's own, i.e. when the prefix and suffix minima of the
// CTA's deltas around g are below delta(g).  A climb leaves the local phase
// at the first split that is not local and continues with the device-scope
// protocol above.  Local nodes hold < B < 1024 bodies, so they all take the
// f32 path below.
//
// Mass / COM: small nodes use the reference's f32 formula
//   M = m_l + m_r;  com = (c_l m_l + c_r m_r) / M  (0 if M <= 0)   (lbvh.wgsl:216-224)
// and nodes of >= kFp64MinBodies bodies aggregate {m, m x, m y} in FP64.
// AABB and length = longest side are exact (lbvh.wgsl:212-213,227-228).
#pragma once

#include <cuda/atomic>

#include "bh_internal.cuh"

namespace bh {

// a / b correctly rounded, given r = 1/b correctly rounded (__frcp_rn): one
// correction of the product a r by its exact residual a - b (a r) (an FMA),
// P. Markstein's final step for IEEE division (IBM J. Res. Dev. 34(1), 1990):
// with r within half an ulp of 1/b and q within an ulp of a/b, q + (a - b q) r
// rounds to a/b.  Operands here are normal-range masses and mass moments
// (b > 0); the build divides two numerators by one mass, so the reciprocal
// is shared and each quotient costs a multiply and two FMAs.
__device__ __forceinline__ float div_by(float a, float b, float r) {
    const float q = __fmul_rn(a, r);
    const float e = __fmaf_rn(-q, b, a);
    return __fmaf_rn(e, r, q);
}

template <typename K>
__device__ __forceinline__ int delta_at(const K* __restrict__ keys, uint32_t i, uint32_t j) {
    K a = __ldg(&keys[i]), b = __ldg(&keys[j]);
    if (a == b) return (int)(8 * sizeof(K)) + __clz((int)(i ^ j));
    if (sizeof(K) == 8) return __clzll((long long)(a ^ b));
    return __clz((int)(uint32_t)(a ^ b));
}

template <typename K>
__device__ __forceinline__ int delta_keys(K a, K b, uint32_t i, uint32_t j) {
    if (a == b) return (int)(8 * sizeof(K)) + __clz((int)(i ^ j));
    if (sizeof(K) == 8) return __clzll((long long)(a ^ b));
    return __clz((int)(uint32_t)(a ^ b));
}

// Kernel arguments (device pointers; gnode / groups / group_count are null
// when the caller needs no group-walk records).
template <typename K>
struct BuildArgs {
    const K* keys;
    const uint32_t* ids;
    const float* mass;
    const float2* pos;
    float4* node4;
    uint2* children;
    uint32_t* parent;
    float4* aabb;
    uint2* range;
    MeetSlot* slots;
    uint32_t n;
    int fp64;
    GNode* gnode;
    uint2* groups;
    unsigned int* group_count;
    uint32_t gmax;
    // Split build only: nodes whose parent split is not local, as {first
    // slot, last slot}, and their count (zero before the local phase).
    uint2* frontier = nullptr;
    unsigned int* frontier_count = nullptr;
    // {x, y, m, 0} per body in original order, when the encode wrote them:
    // one gather per slot instead of a position and a mass
    const float4* xm = nullptr;
    // The step's device error word: when an earlier stage of the step failed
    // (kErrSkipMask), the build does nothing; a bounded wait that gives up sets
    // kErrTreeSpin.  Null: no such check.
    uint32_t* err = nullptr;
};

// One thread per sorted slot climbs from its leaf; the lanes of a warp start
// at adjacent leaves, so the low levels they create are adjacent in memory.
// (A persistent variant that hands each finished lane a new leaf measured
// slower at 16M bodies: its lanes drift apart and its node writes scatter.)
// Slots per CTA (tree stage, before the packing below): the fused build, 64 /
// 128 / 256: 800k bodies 102 / 93 / 96 us, 1.5M 170 / 154 / 160, 16k and fewer
// equal; the split build's local phase takes large ones (16.8M, 256 / 512: 1.52
// / 1.43 ms; 4.2M 356 / 374 us).  The frontier climb keeps 256 threads per CTA.
#ifndef BH_BUILD_BLOCK_FUSED
#define BH_BUILD_BLOCK_FUSED 128
#endif
#ifndef BH_BUILD_BLOCK_SPLIT
#define BH_BUILD_BLOCK_SPLIT 512
#endif
constexpr int kBuildBlockFused = BH_BUILD_BLOCK_FUSED;
constexpr int kBuildBlockSplit = BH_BUILD_BLOCK_SPLIT;
constexpr int kClimbBlock = 256;
template <bool SPLIT>
constexpr int build_block() { return SPLIT ? kBuildBlockSplit : kBuildBlockFused; }
// Resident CTAs per SM the launch bounds ask for: 3 for the split build's local
// phase (39 registers, no spills; 4: 16.8M bodies 1.53 against 1.43 ms), the
// compiler's choice (0) for the fused build.
#ifndef BH_BUILD_MIN_BLOCKS_SPLIT
#define BH_BUILD_MIN_BLOCKS_SPLIT 3
#endif
template <bool SPLIT>
constexpr int build_min_blocks() { return SPLIT ? BH_BUILD_MIN_BLOCKS_SPLIT : 0; }
// A block's climbers stop after kPackAfter levels and go on in its first warps:
// after two levels about 5 of a warp's 32 lanes still climb, and every warp went
// through ~15 levels with them (9-12 lanes an instruction, 43 warp instructions
// a body).  Tree stage, packed after 1 / 2 / 3 levels / never: 800k bodies 91 /
// 88 / 88 / 94 us, 4.2M 348 / 345 / 362 / 373, 16.8M 1.35 / 1.36 / 1.39 / 1.44 ms;
// after 2 / never: 400k 57 / 61 us, 150k 37 / 38, 100k 35 / 35, 70k 35 / 33.  In
// rotation on three handles the step is 1.5% (800k) and 1% (16.8M) shorter.
// Below kPackMin the packing's two barriers only lengthen the chain; a runtime
// switch in one kernel costs that too (16k 25.7 -> 26.2 us a step).
constexpr int kPackAfter = 2;
constexpr uint32_t kPackMin = 131072;
static_assert(kFp64MinBodies > kBuildBlockFused && kFp64MinBodies > kBuildBlockSplit,
              "local nodes must all take the f32 path");

// The block-local shared state of the local phase (B slots per CTA).
template <typename K, int B>
struct BuildShared {
    K key[B + 2];           // keys of slots B0-1 .. B0+B
    int d[B + 1];           // delta at boundary g = B0-1+q (between slots g, g+1)
    int wmin[2][B / 32];    // per-warp minima for the two scans
    int suf[B];             // suf[q] = min of d[q+1..B]
    unsigned char local[B + 1];
    uint32_t bound[B + 1];  // exchange slots of the local splits
    float4 leaf[B];         // {x, y, m, 0} by slot - B0
    // local internal nodes by index - B0: {cx, cy, m, link bits}, box,
    // {Sxx, Sxy, Syy, body count bits (0: no such node)}, and first slot - B0
    float4 mom[B], box[B], quad[B];
    unsigned short first[B];
    unsigned short open[B];  // nodes that climb on after the packing (a leaf: B + slot)
    uint32_t num_open;
};

// The node a climbing thread currently owns: its slot range, the deltas at
// the range's two boundaries, and its record.
struct Climb {
    uint32_t l, r;
    int dl, dr;
    float cm, cx, cy;
    float lox, loy, hix, hiy;
    float sxx, sxy, syy;       // second moments about the COM (group walk)
    double dm, dmx, dmy;       // valid when the node has >= kFp64MinBodies bodies
};

// Mass, centre and second moments of the parent of two nodes (f32 path):
//   M = m_a + m_b;  com = (c_a m_a + c_b m_b) / M  (0 if M <= 0)   (lbvh.wgsl:216-224)
//   S = sum_c S_c + m_c d_c d_c^T, d_c = c_c - com (leaves: S_c = 0).
// Each sum joins two terms with one IEEE addition, which is commutative, so
// the children need no ordering.
__device__ __forceinline__ void join_centres(float ma, float ax, float ay, float mb, float bx,
                                             float by, float& tm, float& cx, float& cy) {
    tm = __fadd_rn(ma, mb);
    cx = 0.0f;
    cy = 0.0f;
    if (tm > 0.0f) {
        const float inv = __frcp_rn(tm);
        cx = div_by(__fadd_rn(__fmul_rn(ax, ma), __fmul_rn(bx, mb)), tm, inv);
        cy = div_by(__fadd_rn(__fmul_rn(ay, ma), __fmul_rn(by, mb)), tm, inv);
    }
}
__device__ __forceinline__ void join_moments(float ma, float ax, float ay, float mb, float bx,
                                             float by, float cx, float cy, const float4& sq,
                                             float& sxx, float& sxy, float& syy) {
    const float dax = __fsub_rn(ax, cx), day = __fsub_rn(ay, cy);
    const float dbx = __fsub_rn(bx, cx), dby = __fsub_rn(by, cy);
    const float madx = __fmul_rn(ma, dax), mady = __fmul_rn(ma, day);
    const float mbdx = __fmul_rn(mb, dbx), mbdy = __fmul_rn(mb, dby);
    sxx = __fadd_rn(__fmaf_rn(madx, dax, sxx), __fmaf_rn(mbdx, dbx, sq.x));
    sxy = __fadd_rn(__fmaf_rn(madx, day, sxy), __fmaf_rn(mbdx, dby, sq.y));
    syy = __fadd_rn(__fmaf_rn(mady, day, syy), __fmaf_rn(mbdy, dby, sq.z));
}

// Write node `pidx` over slots [pl, pl + cnt) to the tree arrays: its record,
// its children's parent entries, and the walk groups it ends (a child is a
// maximal subtree of <= gmax bodies when its parent is too big; the whole tree
// is one when n <= gmax).
template <typename K>
__device__ __forceinline__ void emit_node(const BuildArgs<K>& A, uint32_t pidx, uint32_t pl,
                                          uint32_t cnt, uint32_t link, float cx, float cy, float m,
                                          float4 box, float sxx, float sxy, float syy) {
    const uint32_t nm1 = A.n - 1;
    const uint32_t gamma = link_gamma(link);
    const uint32_t li = link_left(link, nm1), ri = link_right(link, nm1);
    if (A.gnode) {
        GNode* const g = &A.gnode[pidx];
        st_half(&g->mom, make_float4(cx, cy, m, sxx),
                make_float4(sxy, syy, __uint_as_float(pl), __uint_as_float(cnt)));
        st_half(&g->box, box,
                make_float4(cx, cy, __uint_as_float(link),
                            __uint_as_float(pack_small(cnt, gamma - pl + 1u))));
    } else {
        // Reference layout (lbvh.wgsl:12-22, split into hot and cold arrays).
        // With the packed records it is derived on request (ref_layout_kernel).
        const float len = fmaxf(__fsub_rn(box.z, box.x), __fsub_rn(box.w, box.y));
        A.node4[pidx] = make_float4(cx, cy, m, len);
        A.aabb[pidx] = box;
        A.children[pidx] = make_uint2(li, ri);
        A.range[pidx] = make_uint2(pl, pl + cnt - 1u);
    }
    A.parent[li] = pidx;
    A.parent[ri] = pidx;
    if (cnt == A.n) A.parent[0] = kSentinel;  // the root (lbvh.wgsl:159-161)
    if (A.groups) {
        if (cnt > A.gmax) {
            const uint32_t lcnt = gamma - pl + 1, rcnt = cnt - lcnt;
            if (lcnt <= A.gmax) A.groups[atomicAdd(A.group_count, 1u)] = make_uint2(pl, lcnt);
            if (rcnt <= A.gmax) A.groups[atomicAdd(A.group_count, 1u)] = make_uint2(gamma + 1, rcnt);
        } else if (cnt == A.n) {
            A.groups[atomicAdd(A.group_count, 1u)] = make_uint2(0u, A.n);
        }
    }
}

__device__ __forceinline__ uint32_t make_link(uint32_t gamma, bool left_leaf, bool right_leaf) {
    return gamma | (left_leaf ? kLinkLeftLeaf : 0u) | (right_leaf ? kLinkRightLeaf : 0u);
}

// The block-local climb of one thread: nodes are made and
// exchanged in shared memory only, so a level costs no global store that the
// fences around the exchange would have to wait for; write_local writes them
// out afterwards.  Returns true when the node in `c` waits for a split outside
// the CTA or has climbed LEVELS levels (0: no limit; a thread goes on with it),
// false when this thread is done.
template <int LEVELS, typename K, int B>
__device__ __forceinline__ bool climb_local(const BuildArgs<K>& A, Climb& c, BuildShared<K, B>& S,
                                            uint32_t B0) {
    const uint32_t n = A.n;
    for (int level = 0; LEVELS == 0 || level < LEVELS; ++level) {
        const bool is_left = c.dr > c.dl;
        // boundary (relative) at which this node meets its sibling
        const int q = (int)((is_left ? c.r : c.l - 1u) - B0) + 1;
        if (q < 1 || q > B - 1 || !S.local[q]) return true;
        __threadfence_block();  // this node's record before the exchange
        const uint32_t other = atomicExch(&S.bound[q], is_left ? c.l : c.r);
        if (other == kSentinel) return false;  // first to arrive: the sibling's thread goes on
        __threadfence_block();
        const uint32_t gamma = B0 + (uint32_t)q - 1u;
        const uint32_t pl = is_left ? c.l : other, pr = is_left ? other : c.r;
        const bool lleaf = pl == gamma, rleaf = pr == gamma + 1u;
        float4 sm, sb, sq = make_float4(0.f, 0.f, 0.f, 0.f);
        const int k = is_left ? q : q - 1;  // the sibling: gamma + 1 or gamma
        if (is_left ? rleaf : lleaf) {
            sm = S.leaf[k];
            sb = make_float4(sm.x, sm.y, sm.x, sm.y);
        } else {
            sm = S.mom[k];
            sb = S.box[k];
            sq = S.quad[k];
        }
        // Parent's boundary deltas; its Karras index is its range end next to
        // the larger one (the root's is 0, its first slot).
        if (is_left) c.dr = S.d[(int)(pr - B0) + 1];
        else c.dl = S.d[(int)(pl - B0)];
        const uint32_t pidx = (c.dr > c.dl) ? pr : pl;
        float tm, ncx, ncy;
        join_centres(c.cm, c.cx, c.cy, sm.z, sm.x, sm.y, tm, ncx, ncy);
        join_moments(c.cm, c.cx, c.cy, sm.z, sm.x, sm.y, ncx, ncy, sq, c.sxx, c.sxy, c.syy);
        c.lox = fminf(c.lox, sb.x);
        c.loy = fminf(c.loy, sb.y);
        c.hix = fmaxf(c.hix, sb.z);
        c.hiy = fmaxf(c.hiy, sb.w);
        c.cm = tm;
        c.cx = ncx;
        c.cy = ncy;
        c.l = pl;
        c.r = pr;
        const int w = (int)(pidx - B0);
        const uint32_t cnt = pr - pl + 1u;
        S.mom[w] = make_float4(ncx, ncy, tm, __uint_as_float(make_link(gamma, lleaf, rleaf)));
        S.box[w] = make_float4(c.lox, c.loy, c.hix, c.hiy);
        S.quad[w] = make_float4(c.sxx, c.sxy, c.syy, __uint_as_float(cnt));
        S.first[w] = (unsigned short)(pl - B0);
        if (cnt == n) return false;  // the root
    }
    return true;
}

// 128-bit relaxed accesses at device scope (single-copy atomic).
__device__ __forceinline__ uint4 exch128(uint4* p, uint4 v) {
    uint4 r;
    asm volatile(
        "{\n .reg .b128 a, b;\n .reg .b64 l, h;\n mov.b64 l, {%5, %6};\n mov.b64 h, {%7, %8};\n"
        " mov.b128 a, {l, h};\n atom.relaxed.gpu.global.exch.b128 b, [%4], a;\n"
        " mov.b128 {l, h}, b;\n mov.b64 {%0, %1}, l;\n mov.b64 {%2, %3}, h;\n}"
        : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
        : "l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
        : "memory");
    return r;
}
__device__ __forceinline__ uint4 ld128(const uint4* p) {
    uint4 r;
    asm volatile(
        "{\n .reg .b128 b;\n .reg .b64 l, h;\n ld.relaxed.gpu.global.b128 b, [%4];\n"
        " mov.b128 {l, h}, b;\n mov.b64 {%0, %1}, l;\n mov.b64 {%2, %3}, h;\n}"
        : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
        : "l"(p)
        : "memory");
    return r;
}
__device__ __forceinline__ void clear128(uint4* p) {
    asm volatile(
        "{\n .reg .b128 a;\n .reg .b64 l;\n mov.b64 l, -1;\n mov.b128 a, {l, l};\n"
        " st.relaxed.gpu.global.b128 [%0], a;\n}" ::"l"(p)
        : "memory");
}

// The sibling's word k of a split: `got` when this thread's exchange returned
// it, else it is on its way (the sibling's exchanges were all issued before
// the one that made this thread the second) and overwrites this thread's own.
// Bounded; false when the wait gives up.
__device__ __forceinline__ bool sibling_word(uint4& got, const uint4* p, uint32_t side) {
    for (uint32_t spins = 0; got.w != side; ++spins) {
        if (spins > kMeetSpins) return false;
        if (spins > 64) __nanosleep(64);
        got = ld128(p);
    }
    return true;
}

// One level of the climb at device scope: returns false when this thread is
// the first to arrive at the split (it stops; the sibling's thread goes on)
// or has created the root, else true with `c` holding the parent.  The two
// children swap their whole records through the split's slot: every word is
// one 128-bit exchange, all of them in flight together, so a level is one
// round trip to the L2 and its arithmetic.  (An acq_rel exchange of the range
// ends, then the sibling's record and the boundary's keys, is three in a row:
// 3,000-3,300 cycles a level, 13 levels at 2k bodies, 27 at 800k, about 1,300
// now.  Tree stage: 2k bodies 32 -> 20 us, 16k 39 -> 25, 100k 48 -> 31, 800k
// 120 -> 93, 16.8M, bound by its local phase, unchanged.)
template <typename K>
__device__ __forceinline__ bool climb_step(const BuildArgs<K>& A, Climb& c) {
    const uint32_t n = A.n;
    const bool is_left = c.dr > c.dl;
    const uint32_t gamma = is_left ? c.r : c.l - 1;
    const uint32_t side = is_left ? 1u : 2u, other_side = 3u - side;
    uint4* const w = A.slots[gamma].w;
    const uint32_t my_cnt = c.r - c.l + 1;
    const bool big = A.fp64 && my_cnt >= kFp64MinBodies;  // carries FP64 sums
    auto bits = [](float v) { return __float_as_uint(v); };
    auto word64 = [&](double v) {
        return make_uint4((uint32_t)__double2loint(v), (uint32_t)__double2hiint(v), 0u, side);
    };
    uint4 o4 = make_uint4(0u, 0u, 0u, 0u), o5 = o4, o6 = o4;
    if (big) {
        o4 = exch128(w + 4, word64(c.dm));
        o5 = exch128(w + 5, word64(c.dmx));
        o6 = exch128(w + 6, word64(c.dmy));
    }
    uint4 o1 = exch128(w + 1, make_uint4(bits(c.lox), bits(c.loy), bits(c.hix), side));
    uint4 o2 = exch128(w + 2, make_uint4(bits(c.hiy), bits(c.sxx), bits(c.sxy), side));
    uint4 o3 = exch128(w + 3, make_uint4(bits(c.syy), (uint32_t)(is_left ? c.dl : c.dr), 0u, side));
    const uint4 o0 = exch128(w, make_uint4(is_left ? c.l : c.r, bits(c.cm), bits(c.cx), bits(c.cy)));
    if (o0.x == kSentinel) return false;  // first to arrive: the sibling finishes the parent
    const uint32_t other = o0.x;
    const uint32_t pl = is_left ? c.l : other;
    const uint32_t pr = is_left ? other : c.r;
    const uint32_t sib_cnt = is_left ? (pr - gamma) : (gamma - pl + 1);
    const bool sib_big = A.fp64 && sib_cnt >= kFp64MinBodies;
    bool ok = sibling_word(o1, w + 1, other_side) && sibling_word(o2, w + 2, other_side) &&
              sibling_word(o3, w + 3, other_side);
    if (sib_big)
        ok = ok && sibling_word(o4, w + 4, other_side) && sibling_word(o5, w + 5, other_side) &&
             sibling_word(o6, w + 6, other_side);
    if (!ok) {
        if (A.err) atomicOr(A.err, kErrTreeSpin);
        return false;
    }
    // The slot is empty again for the next step (both children are done with it).
    clear128(w);
    clear128(w + 1);
    clear128(w + 2);
    clear128(w + 3);
    if (big || sib_big) {
        clear128(w + 4);
        clear128(w + 5);
        clear128(w + 6);
    }
    const float sm = __uint_as_float(o0.y), sx = __uint_as_float(o0.z), sy = __uint_as_float(o0.w);
    c.lox = fminf(c.lox, __uint_as_float(o1.x));
    c.loy = fminf(c.loy, __uint_as_float(o1.y));
    c.hix = fmaxf(c.hix, __uint_as_float(o1.z));
    c.hiy = fmaxf(c.hiy, __uint_as_float(o2.x));
    const float4 sq = make_float4(__uint_as_float(o2.y), __uint_as_float(o2.z), __uint_as_float(o3.x), 0.f);
    const uint32_t cnt = pr - pl + 1;
    // Parent's boundary deltas (the sibling's outer one is the parent's) and
    // its own Karras index.
    if (is_left) c.dr = (int)o3.y;
    else c.dl = (int)o3.y;
    const uint32_t pidx = (cnt == n) ? 0u : ((c.dr > c.dl) ? pr : pl);
    float tm, ncx, ncy;
    if (A.fp64 && cnt >= kFp64MinBodies) {
        auto sum64 = [](const uint4& o) { return __hiloint2double((int)o.y, (int)o.x); };
        if (!big) {
            c.dm = (double)c.cm; c.dmx = (double)c.cm * (double)c.cx; c.dmy = (double)c.cm * (double)c.cy;
        }
        c.dm += sib_big ? sum64(o4) : (double)sm;
        c.dmx += sib_big ? sum64(o5) : (double)sm * (double)sx;
        c.dmy += sib_big ? sum64(o6) : (double)sm * (double)sy;
        tm = (float)c.dm;
        const double inv = c.dm > 0.0 ? 1.0 / c.dm : 0.0;
        ncx = (float)(c.dmx * inv);
        ncy = (float)(c.dmy * inv);
    } else {
        join_centres(c.cm, c.cx, c.cy, sm, sx, sy, tm, ncx, ncy);
    }
    if (A.gnode) join_moments(c.cm, c.cx, c.cy, sm, sx, sy, ncx, ncy, sq, c.sxx, c.sxy, c.syy);
    emit_node(A, pidx, pl, cnt, make_link(gamma, pl == gamma, pr == gamma + 1), ncx, ncy, tm,
              make_float4(c.lox, c.loy, c.hix, c.hiy), c.sxx, c.sxy, c.syy);
    c.cm = tm; c.cx = ncx; c.cy = ncy;
    c.l = pl;
    c.r = pr;
    return cnt != n;
}

// Hierarchy build + fill, one thread per sorted slot.  SPLIT = false: the
// whole climb (fused build, one kernel).  SPLIT = true: only the block-local
// phase; threads that reach a split outside their CTA list their node in the
// frontier and exit, and build_climb_kernel finishes the tree.  A CTA of the
// fused build stays resident while one or two of its threads climb the
// device-scope levels; the split build frees it at the end of its local phase
// and climbs all frontier nodes side by side, which pays off from a few
// million bodies up (fused / split, before the packing: 800k 93 / 105 us, 1.5M
// 154 / 152, 4.2M 404 / 374, 16.8M 1.51 / 1.43 ms).
// (Climbing the local phase in CTA-wide rounds that pack the remaining
// nodes into the lowest warps after every level measured slower than packing
// them once.  Nor do the random leaf gathers set the pace: with the bodies
// uploaded in the previous step's
// sorted order, so the gathers run nearly in sequence, the 16.8M-body build
// took 1.80 against 1.84 ms.)
// PACK: the block's climbers go on in its first warps after kPackAfter levels.
template <typename K, bool SPLIT, bool PACK = SPLIT>
__global__ void __launch_bounds__(build_block<SPLIT>(), build_min_blocks<SPLIT>())
build_fill_kernel(const BuildArgs<K> A) {
    constexpr int B = build_block<SPLIT>();
    // dynamic: sizeof(BuildShared<K, B>) bytes (more than 48 KB for large B)
    extern __shared__ __align__(16) unsigned char build_smem[];
    BuildShared<K, B>& S = *reinterpret_cast<BuildShared<K, B>*>(build_smem);

    wait_previous_kernel();
    const uint32_t n = A.n;
    if (step_failed(A.err)) return;  // uniform over the block
    const int t = (int)threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t B0 = blockIdx.x * (uint32_t)B;
    const uint32_t i = B0 + (uint32_t)t;
    if (n == 1) {
        if (t == 0) {
            const uint32_t body = __ldg(&A.ids[0]);
            const float2 p = __ldg(&A.pos[body]);
            A.node4[0] = make_float4(p.x, p.y, __ldg(&A.mass[body]), 0.0f);  // lbvh.wgsl:179-187
            // The reference's build has no internal node to run for n == 1
            // (lbvh.wgsl:95-97): the only node keeps its buffer's initial 0.
            A.parent[0] = 0u;
            if (A.groups) {
                A.groups[0] = make_uint2(0u, 1u);
                *A.group_count = 1u;
            }
        }
        return;
    }
    const uint32_t nm1 = n - 1;
    // ---- boundary deltas of the CTA's slots and which splits are local ----
    for (int q = t; q < B + 2; q += B) {
        const long long g = (long long)B0 - 1 + q;
        S.key[q] = (g >= 0 && g < (long long)n) ? __ldg(&A.keys[g]) : (K)0;
    }
    for (int q = t; q <= B; q += B) S.bound[q] = kSentinel;
    __syncthreads();
    for (int q = t; q <= B; q += B) {
        const long long g = (long long)B0 - 1 + q;
        S.d[q] = (g < 0 || g >= (long long)nm1)
                     ? -1
                     : delta_keys<K>(S.key[q], S.key[q + 1], (uint32_t)g, (uint32_t)g + 1u);
    }
    __syncthreads();
    {
        const unsigned FULL = 0xFFFFFFFFu;
        // pm = min of d[0..t], sm = min of d[t+1..B]
        int pm = S.d[t], sm = S.d[t + 1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(FULL, pm, o);
            const int c = __shfl_down_sync(FULL, sm, o);
            if (lane >= o) pm = min(pm, a);
            if (lane + o < 32) sm = min(sm, c);
        }
        if (lane == 31) S.wmin[0][warp] = pm;
        if (lane == 0) S.wmin[1][warp] = sm;
        __syncthreads();
        for (int w = 0; w < warp; ++w) pm = min(pm, S.wmin[0][w]);
        for (int w = warp + 1; w < B / 32; ++w) sm = min(sm, S.wmin[1][w]);
        S.suf[t] = sm;
        __syncthreads();
        // Boundary q = t + 1 splits a local node when a smaller delta lies
        // among d[0..q-1] (= pm) and among d[q+1..B] (= suf[q]).
        const int q = t + 1;
        if (q <= B - 1) S.local[q] = (pm < S.d[q] && S.suf[q] < S.d[q]) ? 1 : 0;
        if (t == 0) {
            S.local[0] = 0;
            S.local[B] = 0;
        }
        __syncthreads();
    }
    S.quad[t] = make_float4(0.f, 0.f, 0.f, 0.f);  // no node yet
    const bool active = i < n;
    Climb c;
    if (active) {
        const uint32_t body = __ldg(&A.ids[i]);
        float4 r;
        if (A.xm) {
            r = __ldg(&A.xm[body]);
        } else {
            const float2 p = __ldg(&A.pos[body]);
            r = make_float4(p.x, p.y, __ldg(&A.mass[body]), 0.0f);
        }
        r.w = 0.0f;
        S.leaf[t] = r;
        c.l = i;
        c.r = i;
        // delta at the two boundaries of the current range (-1 outside [0, n-1]);
        // a parent keeps one of them, so each level computes only one new delta.
        c.dl = S.d[t];
        c.dr = S.d[t + 1];
        c.cm = r.z; c.cx = r.x; c.cy = r.y;
        c.lox = r.x; c.loy = r.y; c.hix = r.x; c.hiy = r.y;
        c.sxx = 0.0f; c.sxy = 0.0f; c.syy = 0.0f;
        c.dm = 0.0; c.dmx = 0.0; c.dmy = 0.0;
    }
    if (PACK && t == 0) S.num_open = 0;
    __syncthreads();
    bool on;
    if (PACK) {
        {
            const bool open = active && climb_local<kPackAfter>(A, c, S, B0);
            const unsigned m = __ballot_sync(0xFFFFFFFFu, open);
            uint32_t at = 0;
            if (m != 0u && lane == 0) at = atomicAdd(&S.num_open, (uint32_t)__popc(m));
            at = __shfl_sync(0xFFFFFFFFu, at, 0);
            if (open) {
                const uint32_t w = (c.dr > c.dl ? c.r : c.l) - B0;  // its Karras index
                S.open[at + (uint32_t)__popc(m & ((1u << lane) - 1u))] =
                    (unsigned short)(c.l == c.r ? (uint32_t)B + (c.l - B0) : w);
            }
        }
        __syncthreads();
        on = (uint32_t)t < S.num_open;
        if (on) {
            const uint32_t e = S.open[t];
            const bool is_leaf = e >= (uint32_t)B;
            const uint32_t w = is_leaf ? e - (uint32_t)B : e;
            float4 m, b, q = make_float4(0.f, 0.f, 0.f, 0.f);
            uint32_t first = w, cnt = 1u;
            if (is_leaf) {
                m = S.leaf[w];
                b = make_float4(m.x, m.y, m.x, m.y);
            } else {
                m = S.mom[w];
                b = S.box[w];
                q = S.quad[w];
                first = S.first[w];
                cnt = __float_as_uint(q.w);
            }
            c.l = B0 + first;
            c.r = c.l + cnt - 1u;
            c.dl = S.d[first];
            c.dr = S.d[first + cnt];
            c.cm = m.z; c.cx = m.x; c.cy = m.y;
            c.lox = b.x; c.loy = b.y; c.hix = b.z; c.hiy = b.w;
            c.sxx = q.x; c.sxy = q.y; c.syy = q.z;
            c.dm = 0.0; c.dmx = 0.0; c.dmy = 0.0;
            on = climb_local<0>(A, c, S, B0);
        }
    } else {
        on = active && climb_local<0>(A, c, S, B0);
    }
    __syncthreads();
    // ---- write the CTA's leaves and local nodes, in order ------------------
    if (active) A.node4[nm1 + i] = S.leaf[t];  // leaf (lbvh.wgsl:179-187)
    {
        const float4 quad = S.quad[t];
        const uint32_t cnt = __float_as_uint(quad.w);
        if (cnt != 0u) {
            const float4 mom = S.mom[t];
            emit_node(A, B0 + (uint32_t)t, B0 + (uint32_t)S.first[t], cnt, __float_as_uint(mom.w),
                      mom.x, mom.y, mom.z, S.box[t], quad.x, quad.y, quad.z);
        }
    }
    if (SPLIT) {
        // nodes whose parent split lies outside this CTA: to the climb kernel
        const unsigned m = __ballot_sync(0xFFFFFFFFu, on);
        if (m) {
            uint32_t at = 0;
            if (lane == __ffs(m) - 1) at = atomicAdd(A.frontier_count, (uint32_t)__popc(m));
            at = __shfl_sync(0xFFFFFFFFu, at, __ffs(m) - 1);
            if (on) A.frontier[at + (uint32_t)__popc(m & ((1u << lane) - 1u))] = make_uint2(c.l, c.r);
        }
        return;
    }
    if (on)
        while (climb_step(A, c)) {
        }
}

// Second kernel of the split build: one thread per frontier node (a node
// made in the local phase, or a leaf, whose parent split is outside its
// CTA) continues the climb with the device-scope protocol.  The node's
// record is read back from the tree arrays the first kernel wrote; no
// frontier node is large enough for the FP64 path (local nodes hold fewer
// than kBuildBlockSplit < kFp64MinBodies bodies).  Each climb ends without
// waiting for any other thread, so a thread may take several entries.
template <typename K>
__global__ void __launch_bounds__(kClimbBlock)
build_climb_kernel(const BuildArgs<K> A) {
    wait_previous_kernel();
    if (step_failed(A.err)) return;
    const uint32_t count = *A.frontier_count;
    const uint32_t n = A.n, nm1 = n - 1;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < count; e += gridDim.x * blockDim.x) {
        const uint2 f = A.frontier[e];
        Climb c;
        c.l = f.x;
        c.r = f.y;
        c.dl = (c.l == 0) ? -1 : delta_at(A.keys, c.l - 1, c.l);
        c.dr = (c.r == nm1) ? -1 : delta_at(A.keys, c.r, c.r + 1);
        c.sxx = 0.0f; c.sxy = 0.0f; c.syy = 0.0f;
        c.dm = 0.0; c.dmx = 0.0; c.dmy = 0.0;
        if (c.l == c.r) {
            const float4 leaf = A.node4[nm1 + c.l];
            c.cm = leaf.z; c.cx = leaf.x; c.cy = leaf.y;
            c.lox = leaf.x; c.loy = leaf.y; c.hix = leaf.x; c.hiy = leaf.y;
        } else {
            // Karras index: the range end next to the parent's split.
            const uint32_t idx = (c.dr > c.dl) ? c.r : c.l;
            float4 box, mom;
            if (A.gnode) {
                box = A.gnode[idx].box;
                mom = A.gnode[idx].mom;
                const float4 q = A.gnode[idx].tail;
                c.sxx = mom.w; c.sxy = q.x; c.syy = q.y;
            } else {
                box = A.aabb[idx];
                mom = A.node4[idx];
            }
            c.cm = mom.z; c.cx = mom.x; c.cy = mom.y;
            c.lox = box.x; c.loy = box.y; c.hix = box.z; c.hiy = box.w;
        }
        while (climb_step(A, c)) {
        }
    }
}

}  // namespace bh
