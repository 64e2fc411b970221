// group_walk.cuh -- the Barnes-Hut walk of a warp's 32 nodes together (FP32).
// Included by kernels.cuh, after the per-thread walks.
//
// The 32 nodes of a warp are neighbours in Morton order, and most regions are
// far from, or near to, all of them. The warp keeps a stack of regions, each
// with the mask of the lanes that walk it. A round takes up to 32 regions
// from the stack, one a lane; a lane tests its region against the box of the
// warp's nodes:
//   far from every node   its pull is added by all lanes in a loop over the
//                         round's far regions (broadcast from shared memory);
//   near to every node    its children go on the stack (a region of at most 8
//                         nodes goes on the list of buckets);
//   neither               every lane tests its own node in a loop over the
//                         round's mixed regions; the children go on the stack
//                         with the mask of the lanes that were near.
// The buckets' node pairs are summed at the end (before, if the list fills).
// The top of the tree is tested once for a block: its first warp walks it
// with the box of the block's nodes and leaves the regions far from all of
// them and the regions where the warps' own walks start.
//
// Every lane decides as walk() does, on the same values: the box test uses
// the lanes' own formula, d^2 = fma(dx, dx, dy dy), on the box's smallest and
// largest |dx| and |dy|; rounding is monotonic, so "far from the box" and
// "near to all of the box" hold for every lane's own d^2. The force is summed
// in another order than walk()'s, which differs between warps but is fixed.
//
// What bounds it: instruction issue with the device full, the chain of one
// warp's rounds (each a load, a test and the shared-memory lists) below. A
// node's own walk makes 295 steps of 33 warp instructions and 9 L1 lines each
// at 10^6 nodes (342 M warp instructions, 385 us alone, 418 us after the
// tree build). Together a warp tests 259 regions against its box in 9.8
// rounds, adds 53 far ones, tests 204 lane by lane and sums 134 node pairs,
// without a divergent load: 257 M warp instructions at 70 % issue, 320 us
// after the tree build; 56 against 116 us at 10^5 nodes, 24 against 55 us at
// 10^4. The loops take two regions (nodes) to a packed FP32 instruction
// (f32x2). Blocks of 4 warps at 9 a multiprocessor (56 registers): 8 warps
// 344 us (the top's barrier), 2 warps 339 us (more tops), 48 registers 335
// us, 64 330 us.
#pragma once

namespace fa2cu {

// ---- two floats in one register pair ---------------------------------------
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_make(float a, float b)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_split(f2 v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// 1 / a to 1 ulp, 0 above 2^126 (as the approximate division by a).
__device__ __forceinline__ float rcp_approx(float a)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

// Two regions (or nodes) as the loops take them: a field's two values side by
// side. Coordinates are kept negated, so that a difference is one addition.
struct __align__(16) GroupPair {
    float x[2], y[2], m[2];
    float w[2], floor[2]; // opening distance squared, the floor of its band
    unsigned lanes[2];
};
// Two nodes of the buckets.
struct __align__(16) NodePair {
    float x[2], y[2], m[2];
    unsigned lanes[2];
};

// Shared memory of one warp's group walk.
// The stack: above GW_WIDE waiting regions a round takes two (siblings)
// instead of 32, which walks depth first: 64 more wide, then two a level of a
// tree of at most 59 levels (32 key bits, 27 bits of the index).
constexpr int GW_WIDE = 128;
constexpr int GW_STACK = GW_WIDE + 32 + 2 * 64;
constexpr int GW_BUCKETS = 64; // buckets waiting
constexpr int GW_NODES = 64;   // node places of a flush
struct __align__(16) GroupWalkShared {
    union {
        struct {
            GroupPair entry[17]; // the round's far regions, then the mixed ones
            uint4 vote[17];      // of a pair's: lanes beyond the floor, lanes far
        };
        struct {
            NodePair node[GW_NODES / 2];
            int2 flat[GW_NODES]; // (sorted node, lanes)
            float radius[GW_NODES];
        };
    };
    int2 stack[GW_STACK];    // (region, lanes)
    int2 bucket[GW_BUCKETS]; // (packed range, lanes)
};

// The top of the tree, walked for a whole block.
constexpr int GW_TOP_FAR = 64, GW_TOP_ROOTS = 128;
struct __align__(16) GroupTopShared {
    GroupPair far[GW_TOP_FAR / 2]; // far from all nodes
    int root[GW_TOP_ROOTS];        // where the warps start
    int nfar, nroot;               // nfar: even
    float4 box[32];                // of each warp's nodes
};

// A lane's running force. COMP: Kahan compensation (HUB_MASS); else the terms
// of even and odd places apart, two at a time.
template <bool COMP> struct GroupAcc;
template <> struct GroupAcc<false> {
    f2 ax = 0, ay = 0;
    __device__ __forceinline__ void add2(f2 xd, f2 yd, f2 g)
    {
        ax = f2_fma(xd, g, ax);
        ay = f2_fma(yd, g, ay);
    }
    __device__ __forceinline__ void add(float xd, float yd, float g)
    {
        add2(f2_make(xd, 0.0f), f2_make(yd, 0.0f), f2_make(g, 0.0f));
    }
    __device__ __forceinline__ float2 sum() const
    {
        float a, b, c, d;
        f2_split(ax, a, b);
        f2_split(ay, c, d);
        return make_float2(a + b, c + d);
    }
};
template <> struct GroupAcc<true> {
    float ax = 0.0f, ay = 0.0f, cx = 0.0f, cy = 0.0f;
    __device__ __forceinline__ void add(float xd, float yd, float g)
    {
        acc_add(ax, cx, xd * g);
        acc_add(ay, cy, yd * g);
    }
    __device__ __forceinline__ void add2(f2 xd, f2 yd, f2 g)
    {
        float a, b, c, d, u, v;
        f2_split(xd, a, b);
        f2_split(yd, c, d);
        f2_split(g, u, v);
        add(a, c, u);
        add(b, d, v);
    }
    __device__ __forceinline__ float2 sum() const { return make_float2(ax - cx, ay - cy); }
};

// Shared-memory loads at a 32-bit address plus a constant: two pairs, one
// pair, one float; the store of four words.
template <int OFF> __device__ __forceinline__ void lds_2(unsigned at, f2 &a, f2 &b)
{
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2 + %3];"
                 : "=l"(a), "=l"(b)
                 : "r"(at), "n"(OFF)
                 : "memory");
}
template <int OFF> __device__ __forceinline__ f2 lds_1(unsigned at)
{
    f2 a;
    asm volatile("ld.shared.b64 %0, [%1 + %2];" : "=l"(a) : "r"(at), "n"(OFF) : "memory");
    return a;
}
template <int OFF>
__device__ __forceinline__ void sts_4(unsigned at, unsigned a, unsigned b, unsigned c, unsigned d)
{
    asm volatile("st.shared.v4.b32 [%0 + %1], {%2, %3, %4, %5};" ::"r"(at), "n"(OFF), "r"(a),
                 "r"(b), "r"(c), "r"(d)
                 : "memory");
}

// A lane's own node, in the packed form of the loops.
struct GroupNode {
    f2 x, y;
};

// d^2 of two places, and their differences.
__device__ __forceinline__ f2 dist2(const GroupNode &me, f2 nx, f2 ny, f2 &xd, f2 &yd)
{
    xd = f2_add(me.x, nx);
    yd = f2_add(me.y, ny);
    return f2_fma(xd, xd, f2_mul(yd, yd));
}

// The pulls of two regions at squared distances d2.
__device__ __forceinline__ f2 pull2(f2 m, f2 d2)
{
    float u, v;
    f2_split(d2, u, v);
    return f2_mul(m, f2_make(rcp_approx(u), rcp_approx(v)));
}

// The pulls of `cnt` (even) regions far from every lane, from shared address
// `at` on: every split-th pair from `part`.
template <bool COMP>
__device__ __forceinline__ void group_far(unsigned at, int cnt, int part, int split,
                                          const GroupNode &me, GroupAcc<COMP> &acc)
{
    const unsigned end = at + (unsigned) (sizeof(GroupPair) / 2) * cnt;
    at += (unsigned) sizeof(GroupPair) * part;
#pragma unroll 2
    for (; at < end; at += (unsigned) sizeof(GroupPair) * split) {
        f2 x, y, xd, yd;
        lds_2<0>(at, x, y);
        const f2 m = lds_1<16>(at);
        const f2 d2 = dist2(me, x, y, xd, yd);
        acc.add2(xd, yd, pull2(m, d2));
    }
}

// A region's test by every lane of the warp: `beyond` the lanes of `lanes`
// farther than the band's floor, `far` those farther than w; g stays in the
// far lanes only.
__device__ __forceinline__ void lane_test(unsigned lanes, unsigned bit, float d2, float floor,
                                          float w, float &g, unsigned &beyond, unsigned &far)
{
    asm volatile("{\n .reg .pred a, h, f;\n .reg .b32 t;\n"
                 " and.b32 t, %3, %4;\n setp.ne.b32 a, t, 0;\n"
                 " setp.gt.and.ftz.f32 h, %5, %6, a;\n"
                 " setp.gt.and.ftz.f32 f, %5, %7, h;\n"
                 " vote.sync.ballot.b32 %0, h, 0xffffffff;\n"
                 " vote.sync.ballot.b32 %1, f, 0xffffffff;\n"
                 " selp.f32 %2, %2, 0f00000000, f;\n}"
                 : "=r"(beyond), "=r"(far), "+f"(g)
                 : "r"(lanes), "r"(bit), "f"(d2), "f"(floor), "f"(w));
}

// The node pairs of the listed buckets, eight buckets at a time: their nodes
// in one list with the lanes that need them, fetched a node a lane, then
// summed by every lane two at a time. A pair at distance 0 (a node and
// itself, too) adds nothing.
template <bool ADJUST, bool COMP>
__device__ __forceinline__ void group_pairs(GroupWalkShared &S, int nb, int n, const float4 &own,
                                            const GroupNode &me, const float4 *psort,
                                            GroupAcc<COMP> &acc, int *status)
{
    const int lane = threadIdx.x & 31;
    const unsigned bit = 1u << lane;
    for (int b0 = 0; b0 < nb; b0 += 8) {
        // four lanes a bucket, two nodes each
        const int b = b0 + (lane >> 2);
        int2 q = make_int2(0, 0);
        int first = 0, cnt = 0;
        if (b < nb) {
            q = S.bucket[b];
            first = bucket_first(q.x);
            cnt = bucket_last(q.x) - first + 1;
            if (cnt > 8 || first + cnt > n) { // (never, for a legal tree)
                atomicOr(status + ST_ERROR, ERR_BOUNDS);
                cnt = 0;
            }
        }
        int end = cnt; // inclusive sum over the buckets
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += t;
        }
        const int total = __shfl_sync(0xffffffffu, end, 31), at = end - cnt;
        __syncwarp(); // the round's entries, and the last nodes, are done with
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int s = (lane & 3) + 4 * h;
            if (s < cnt) S.flat[at + s] = make_int2(first + s, q.y);
        }
        __syncwarp();
        for (int i = lane; i < ((total + 1) & ~1); i += 32) {
            float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            unsigned lanes = 0;
            if (i < total) {
                const int2 f = S.flat[i];
                p = psort[f.x];
                lanes = (unsigned) f.y;
            }
            NodePair &t = S.node[i >> 1];
            t.x[i & 1] = -p.x;
            t.y[i & 1] = -p.y;
            t.m[i & 1] = p.z;
            t.lanes[i & 1] = lanes;
            if (ADJUST) S.radius[i] = p.w;
        }
        __syncwarp();
        const unsigned first_node = smem_addr(S.node);
        int i = 0;
#pragma unroll 2
        for (unsigned t = first_node, stop = first_node + (unsigned) (sizeof(NodePair) / 2) * total;
             t < stop; t += sizeof(NodePair), i += 2) {
            f2 x, y, m, k, xd, yd;
            lds_2<0>(t, x, y);
            lds_2<16>(t, m, k);
            float u, v, ku, kv, gu, gv;
            const f2 d2 = dist2(me, x, y, xd, yd);
            f2_split(d2, u, v);
            f2_split(k, ku, kv);
            const bool au = (__float_as_uint(ku) & bit) != 0u, av = (__float_as_uint(kv) & bit) != 0u;
            if (ADJUST) {
                float mu, mv;
                f2_split(m, mu, mv);
                const float du = fsqrt(u) - (own.w + S.radius[i]);
                const float dv = fsqrt(v) - (own.w + S.radius[i + 1]);
                gu = du > 0.0f ? mu * rcp_approx(du * du) : du < 0.0f ? 100.0f * mu : 0.0f;
                gv = dv > 0.0f ? mv * rcp_approx(dv * dv) : dv < 0.0f ? 100.0f * mv : 0.0f;
                acc.add2(xd, yd, f2_make(au ? gu : 0.0f, av ? gv : 0.0f));
            } else {
                f2_split(pull2(m, d2), gu, gv);
                acc.add2(xd, yd, f2_make(au && u > 0.0f ? gu : 0.0f, av && v > 0.0f ? gv : 0.0f));
            }
        }
    }
    __syncwarp();
}

// A region against a box of nodes: 1 far from all, -1 near to all, 0 neither.
__device__ __forceinline__ int box_test(const float4 &box, const float4 &c, float floor)
{
    const float ax = box.x - c.x, bx = c.x - box.z, ay = box.y - c.y, by = c.y - box.w;
    const float nx = fmaxf(fmaxf(ax, bx), 0.0f), ny = fmaxf(fmaxf(ay, by), 0.0f);
    const float fx = fmaxf(fabsf(ax), fabsf(bx)), fy = fmaxf(fabsf(ay), fabsf(by));
    if (fmaf(nx, nx, ny * ny) > c.w) return 1;
    return fmaf(fx, fx, fy * fy) > floor ? 0 : -1;
}

// (min x, min y, max x, max y) over the warp.
__device__ __forceinline__ float4 warp_box(float4 b)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        b.x = fminf(b.x, __shfl_xor_sync(0xffffffffu, b.x, o));
        b.y = fminf(b.y, __shfl_xor_sync(0xffffffffu, b.y, o));
        b.z = fmaxf(b.z, __shfl_xor_sync(0xffffffffu, b.z, o));
        b.w = fmaxf(b.w, __shfl_xor_sync(0xffffffffu, b.w, o));
    }
    return b;
}

// The top of the tree for the box of a block's nodes, by one warp (S: its
// own arrays): the regions far from all nodes and the regions to start from
// (neither far nor near; single nodes and buckets, too). Without room for
// them the warps start at the root.
__device__ __forceinline__ void group_top(GroupTopShared &T, GroupWalkShared &S, int n,
                                          const float4 &box, const float4 *rec_c,
                                          const int2 *rec_t, const int2 *child)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int nl = n - 1;
    int sp = 1, nfar = 0, nroot = 0;
    if (lane == 0) S.stack[0] = make_int2(0, 0);
    __syncwarp();
    for (int budget = n + 64; sp > 0 && budget >= 0; budget--) {
        const int take = min(sp, 32);
        sp -= take;
        const int r = lane < take ? S.stack[sp + lane].x : -1;
        __syncwarp();
        int verdict = 0;
        float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        int2 ch = make_int2(0, 0);
        if ((unsigned) r < (unsigned) nl) {
            c = rec_c[r];
            const int left = rec_t[r].x;
            ch = child[r];
            verdict = box_test(box, c, c.w * DECIDE_LO);
            if (verdict < 0 && left < 0) verdict = 0; // a bucket: left to the warps
        }
        const unsigned fb = __ballot_sync(FULL, verdict > 0);
        const unsigned nb = __ballot_sync(FULL, verdict < 0);
        const unsigned rb = __ballot_sync(FULL, lane < take && verdict == 0);
        int at = nfar + __popc(fb & below);
        if (nfar + __popc(fb) > GW_TOP_FAR || nroot + __popc(rb) > GW_TOP_ROOTS ||
            sp + 2 * __popc(nb) > GW_STACK) { // (uniform) no room
            nfar = 0;
            nroot = -1;
            break;
        }
        if (verdict > 0) {
            GroupPair &p = T.far[at >> 1];
            p.x[at & 1] = -c.x;
            p.y[at & 1] = -c.y;
            p.m[at & 1] = c.z;
        } else if (verdict < 0) {
            at = sp + 2 * __popc(nb & below);
            S.stack[at].x = ch.x;
            S.stack[at + 1].x = ch.y;
        } else if (lane < take) {
            T.root[nroot + __popc(rb & below)] = r;
        }
        nfar += __popc(fb);
        nroot += __popc(rb);
        sp += 2 * __popc(nb);
        __syncwarp();
    }
    if (lane == 0) {
        if (nfar & 1) { // an unused place: no mass, far where the one beside it is
            GroupPair &p = T.far[nfar >> 1];
            p.x[1] = p.x[0];
            p.y[1] = p.y[0];
            p.m[1] = 0.0f;
        }
        T.nfar = (nfar + 1) & ~1;
        T.nroot = nroot;
    }
}

// Part `part` of `split` of the forces (per unit of scaling * m_i) of the
// warp's nodes base .. base + 31 (those below n), each in its lane: every
// split-th of the regions that group_top left. Every lane of the warp calls
// it.
template <bool ADJUST, bool COMP>
__device__ __forceinline__ void group_walk(const GroupTopShared &T, GroupWalkShared &S, int base,
                                           int part, int split, int n, const float4 &own, const float4 &box,
                                           double theta2d, const float4 *psort,
                                           const float4 *rec_c, const int2 *rec_t,
                                           const int2 *child, const Agg<float> *agg,
                                           GroupAcc<COMP> &acc, int *status)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned bit = 1u << lane, below = bit - 1u;
    const int nl = n - 1;
    const unsigned all = __ballot_sync(FULL, base + lane < n);
    GroupNode me;
    me.x = f2_make(own.x, own.x);
    me.y = f2_make(own.y, own.y);
    // the stack holds an even number of places (an unused one: no lanes)
    int sp, nb = 0;
    if (T.nroot < 0) {
        sp = part == 0 ? 2 : 0;
        if (lane < sp) S.stack[lane] = make_int2(0, lane == 0 ? (int) all : 0);
    } else {
        const int mine = (T.nroot - part + split - 1) / split;
        sp = (mine + 1) & ~1;
        for (int q = lane; q < sp; q += 32)
            S.stack[q] = q < mine ? make_int2(T.root[q * split + part], (int) all)
                                  : make_int2(0, 0);
        group_far(smem_addr(T.far), T.nfar, part, split, me, acc);
    }
    __syncwarp();
    // a round takes at least one region, and no region comes twice
    for (int budget = 2 * n + 64; sp > 0; budget--) {
        if (budget < 0) { // (uniform)
            if (lane == 0) atomicOr(status + ST_ERROR, ERR_BOUNDS);
            break;
        }
        const int take = sp > GW_WIDE ? 2 : min(sp, 32);
        sp -= take;
        int2 e = make_int2(0, 0);
        if (lane < take) e = S.stack[sp + lane];
        __syncwarp();
        const unsigned lanes = (unsigned) e.y;
        int2 t = make_int2(0, 0), ch = make_int2(0, 0);
        float4 c;
        int verdict = 2; // 2: nothing; else box_test, and 0 for far from some lanes only
        float floor = 0.0f;
        if (lanes && (unsigned) e.x < (unsigned) nl) {
            c = rec_c[e.x];
            t.x = rec_t[e.x].x;
            ch = child[e.x];
            floor = c.w * DECIDE_LO;
            verdict = box_test(box, c, floor);
            if (verdict > 0 && lanes != all) verdict = 0;
        } else if (lanes) { // a single node
            const int j = e.x - nl;
            if ((unsigned) j < (unsigned) n) {
                t.x = bucket_pack(j, j);
                verdict = -1;
            } else {
                atomicOr(status + ST_ERROR, ERR_BOUNDS);
            }
        }
        // the far regions first, then the mixed ones, each from an even
        // place; the place left over by an odd count has no mass and no lanes,
        // that of the far ones the last one's place (at a distance from all nodes)
        const unsigned wb = __ballot_sync(FULL, verdict == 1), mb = __ballot_sync(FULL, verdict == 0);
        const int nw = __popc(wb), nm = __popc(mb), m0 = (nw + 1) & ~1, end = m0 + nm;
        const int at = verdict == 1 ? __popc(wb & below) : m0 + __popc(mb & below);
        if ((unsigned) verdict < 2u) {
            GroupPair &p = S.entry[at >> 1];
            p.x[at & 1] = -c.x;
            p.y[at & 1] = -c.y;
            p.m[at & 1] = c.z;
            p.w[at & 1] = c.w;
            p.floor[at & 1] = floor;
            p.lanes[at & 1] = lanes;
        }
        if (verdict == 1 && at == nw - 1 && (nw & 1)) {
            GroupPair &p = S.entry[at >> 1];
            p.x[1] = -c.x;
            p.y[1] = -c.y;
            p.m[1] = 0.0f;
        }
        if (lane == 0 && (nm & 1)) {
            GroupPair &p = S.entry[end >> 1];
            p.x[1] = p.y[1] = p.m[1] = 0.0f;
            p.lanes[1] = 0u;
        }
        __syncwarp();
        group_far(smem_addr(S.entry), m0, 0, 1, me, acc);
        const unsigned first = smem_addr(S.entry) + (unsigned) (sizeof(GroupPair) / 2) * m0;
        unsigned vote = smem_addr(S.vote) + 8u * m0;
#pragma unroll 2
        for (unsigned i = first, stop = first + (unsigned) (sizeof(GroupPair) / 2) * nm; i < stop;
             i += sizeof(GroupPair), vote += 16u) {
            f2 x, y, m, w, l, k, xd, yd;
            lds_2<0>(i, x, y);
            lds_2<16>(i, m, w);
            lds_2<32>(i, l, k);
            float u, v, gu, gv, wu, wv, lu, lv, ku, kv;
            const f2 d2 = dist2(me, x, y, xd, yd);
            f2_split(pull2(m, d2), gu, gv);
            f2_split(d2, u, v);
            f2_split(w, wu, wv);
            f2_split(l, lu, lv);
            f2_split(k, ku, kv);
            unsigned h0, f0, h1, f1;
            lane_test(__float_as_uint(ku), bit, u, lu, wu, gu, h0, f0);
            lane_test(__float_as_uint(kv), bit, v, lv, wv, gv, h1, f1);
            sts_4<0>(vote, h0, f0, h1, f1);
            acc.add2(xd, yd, f2_make(gu, gv));
        }
        __syncwarp();
        unsigned open = verdict == -1 ? lanes : 0u;
        uint2 mine = make_uint2(0u, 0u);
        if (verdict == 0) {
            mine = reinterpret_cast<const uint2 *>(S.vote)[at];
            open = lanes & ~mine.y;
        }
        // lanes within the band of a region: decided again in double
        for (unsigned bb = __ballot_sync(FULL, mine.x != mine.y); bb; bb &= bb - 1) {
            const int l = __ffs(bb) - 1;
            const int q = __shfl_sync(FULL, at, l), r = __shfl_sync(FULL, e.x, l);
            const unsigned in = __shfl_sync(FULL, mine.x & ~mine.y, l);
            const bool lf = (in & bit) && far_dd(agg + r, own.x, own.y, theta2d);
            if (lf) {
                const GroupPair &p = S.entry[q >> 1];
                const float xd = own.x + p.x[q & 1], yd = own.y + p.y[q & 1];
                acc.add(xd, yd, p.m[q & 1] * rcp_approx(fmaf(xd, xd, yd * yd)));
            }
            const unsigned more = __ballot_sync(FULL, lf);
            if (lane == l) open &= ~more;
        }
        // what is open: a bucket, or two children
        const bool isb = open && t.x < 0, kids = open && t.x >= 0;
        const unsigned kb = __ballot_sync(FULL, kids), qb = __ballot_sync(FULL, isb);
        const int nk = 2 * __popc(kb), nq = __popc(qb);
        if (sp + nk > GW_STACK) { // (uniform; never, for a legal tree)
            if (lane == 0) atomicOr(status + ST_ERROR, ERR_BOUNDS);
            break;
        }
        if (kids)
            *reinterpret_cast<int4 *>(S.stack + sp + 2 * __popc(kb & below)) =
                make_int4(ch.x, (int) open, ch.y, (int) open);
        sp += nk;
        if (nb + nq > GW_BUCKETS) {
            group_pairs<ADJUST, COMP>(S, nb, n, own, me, psort, acc, status);
            nb = 0;
        }
        if (isb) S.bucket[nb + __popc(qb & below)] = make_int2(t.x, (int) open);
        nb += nq;
        __syncwarp();
    }
    group_pairs<ADJUST, COMP>(S, nb, n, own, me, psort, acc, status);
}

// (The tree is read by plain loads: the batched engine makes it in the same
// launch.)
// The walk of one block's nodes, 32 to each `split` of its warps, which share
// the regions left by group_top: the force of node base0 + 32 (w / split) +
// lane in the lanes of warp w (valid below n and where w % split is 0).
// Without shared_top (split 1) every warp starts at the root, and no barrier is
// met. Every thread of the block calls it. HUBS: the graph has nodes of HUB_MASS
// or more; a warp that holds one adds up with compensation.
template <bool ADJUST, bool HUBS>
__device__ __forceinline__ float2
group_walk_block(GroupTopShared &T, GroupWalkShared *Sw, int base0, int split, bool shared_top,
                 int n,
                 float scaling, double theta2d, const float4 *psort, const float4 *rec_c,
                 const int2 *rec_t, const int2 *child, const Agg<float> *agg, int *status)
{
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int group = w / split, part = w % split;
    const int base = base0 + 32 * group;
    const int k = min(base + lane, n - 1);
    const float4 own = psort[k];
    const float4 box = warp_box(make_float4(own.x, own.y, own.x, own.y));
    GroupWalkShared &S = Sw[w];
    if (shared_top) {
        if (lane == 0) T.box[w] = box;
        __syncthreads();
        if (w == 0) // (a warp past the end holds node n - 1's box)
            group_top(T, S, n, warp_box(T.box[min(lane, warps - 1)]), rec_c, rec_t, child);
        __syncthreads();
    } else {
        if (lane == 0) {
            T.box[w] = box;
            T.nroot = -1; // (the same value from every warp)
        }
        __syncwarp();
    }
    float2 v = make_float2(0.0f, 0.0f);
    if (base < n) {
        if (HUBS && __any_sync(0xffffffffu, own.z >= HUB_MASS)) {
            GroupAcc<true> acc;
            group_walk<ADJUST, true>(T, S, base, part, split, n, own, T.box[w], theta2d, psort,
                                     rec_c, rec_t, child, agg, acc, status);
            v = acc.sum();
        } else {
            GroupAcc<false> acc;
            group_walk<ADJUST, false>(T, S, base, part, split, n, own, T.box[w], theta2d, psort,
                                      rec_c, rec_t, child, agg, acc, status);
            v = acc.sum();
        }
    }
    if (split > 1) { // the parts' sums, in order
        float2 *sum = reinterpret_cast<float2 *>(S.stack);
        sum[lane] = v;
        __syncthreads();
        if (part == 0)
            for (int p = 1; p < split; p++) {
                const float2 o = reinterpret_cast<const float2 *>(Sw[w + p].stack)[lane];
                v.x += o.x;
                v.y += o.y;
            }
    }
    const float smi = scaling * psort[k].z;
    return make_float2(v.x * smi, v.y * smi);
}

} // namespace fa2cu
