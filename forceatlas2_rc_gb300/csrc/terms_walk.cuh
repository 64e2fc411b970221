// terms_walk.cuh -- the FP64 Barnes-Hut walk. Included by kernels.cuh.
#pragma once

namespace fa2cu {

// NODES lanes of a warp walk, each for a node, as walk() does: the same regions
// and nodes in the same order, every force the same operations. Two things are
// done otherwise:
//
// - The opening test is made in float, against bounds on both sides of the
//   region's boundary that hold for every rounding of the float coordinates
//   (TermBounds); between them, in double as stated.
// - What a lane would add is pooled: the lanes list (node, source) pairs, each
//   lane its own in order; a full pool is evaluated 32 pairs at a time,
//   whichever lanes they belong to, and each lane then adds up its own.
//
// Why: an FP64 instruction holds the SM for 16 cycles (two lanes a cycle) and
// its result is 64 cycles away. walk() filled 14 of a warp's 32 lanes in them
// -- lanes that add wait for lanes that test -- and a third of them were
// tests; and 196 blocks of eight warps left most SMs idle while some had two
// (50,021 nodes).
//
// NODES: fewer make more warps and less waiting of one lane for another, and
// more instructions of the walk and of the sums a node. The walk in us, walk()
// and this with 32 / 16 / 8 / 4 nodes a warp: 1,000 nodes - and 145 / 102 / 85 /
// 72; 3,001 447 and 173 / 125 / 104 / 88; 10,007 515 and 207 / 150 / 137 / 135;
// 50,021 1,083 and 322 / 302 / 375 / 424; 300,007 4,548 and 1,827 / 1,791 /
// 2,090 / 2,506. A large layout is bound by the FP64 pipe, a small one by the
// serial chain of a lane's steps.
constexpr int TW_WARPS = 2;      // a block
constexpr int TW_POOL = 128;     // pairs evaluated at a time (64 or 192: within 3 %)
constexpr int TW_ROOM = TW_POOL + 32;

struct TermsShared {
    double4_32a node[32];        // the lanes' nodes
    double term[2][TW_POOL];     // x and y
    int source[TW_ROOM];         // a region, or regions + node
    uint8_t owner[TW_ROOM];      // lane
    uint8_t next[TW_ROOM];       // the lane's next place in the pool
};

// (cx, cy, hi, lo) in float of a region whose record is c: with d2 made in
// float from the float node, the region is far where d2 > hi and near where
// d2 < lo; elsewhere it takes the test in double. w = size^2 / theta^2 times
// 1 .. 1 + 2 DECIDE_BAND.
//
// The float coordinates of a node x and a centre c are off by 2^-24 |x| and
// 2^-24 |c|, and |x| <= |c| + |x - c|: their distance by 2^-23 (|cx| + |cy|)
// and by a relative 2^-22 with its own rounding. D is the distance of the
// boundary; the bounds are D +- 2^-21 (|cx| + |cy|), and 1e-5 of that. Squares
// that could underflow bound nothing, and nothing is near beyond 1e18.
__device__ __forceinline__ float4 term_bounds(double4_32a c, double wscale)
{
    const float x = (float) c.x, y = (float) c.y;
    const float w = (float) (c.w * wscale);
    if (!(w >= 0.0f)) return make_float4(x, y, INFINITY, 0.0f); // theta = 0, size 0
    const float D = sqrtf(w), e = (fabsf(x) + fabsf(y)) * 4.76837158203125e-07f;
    const float up = D + e, down = fminf(D * (1.0f - 2.0f * 1e-4f), 1e18f) - e;
    const float hi = up * up * (1.0f + 1e-5f), lo = down * down * (1.0f - 1e-5f);
    return make_float4(x, y, fmaxf(hi, 1e-30f), down > 0.0f && lo > 1e-30f ? lo : 0.0f);
}

// Evaluates the first `count` pairs of the pool.
template <bool ADJUST>
__device__ __forceinline__ void terms_eval(TermsShared &S, int count, int nl, double scaling,
                                           const double4_32a *__restrict__ psort,
                                           const double4_32a *__restrict__ rec_c)
{
    const int lane = threadIdx.x & 31;
#pragma unroll 2
    for (int t = lane; t < count; t += 32) {
        const int src = S.source[t];
        const bool region = src < nl;
        const double4_32a q = region ? rec_c[src] : psort[src - nl];
        const double4_32a me = S.node[S.owner[t]];
        const double xd = me.x - q.x, yd = me.y - q.y;
        const double d2 = sq_dist(xd, yd), mm = me.z * q.z;
        // (a far region has d2 > 0)
        double g;
        if constexpr (ADJUST) {
            double over = 1.0, den = d2; // over: what is left of the distance between the rims
            if (!region) {
                over = fsqrt(d2) - (me.w + q.w);
                den = over * over;
            }
            g = over > 0.0 ? fdiv(scaling * mm, den) : over < 0.0 ? 100.0 * scaling * mm : 0.0;
        } else {
            g = d2 > 0.0 ? fdiv(scaling * mm, d2) : 0.0;
        }
        S.term[0][t] = xd * g;
        S.term[1][t] = yd * g;
    }
}

template <bool ADJUST, int NODES>
__global__ void __launch_bounds__(32 * TW_WARPS)
k_traverse_terms(int n, double scaling, double theta2, const double4_32a *__restrict__ psort,
                 const double4_32a *__restrict__ rec_c, const float4 *__restrict__ bounds,
                 const int2 *__restrict__ rec_t, const int *__restrict__ rope,
                 const uint32_t *__restrict__ order, double2 *__restrict__ f,
                 int *__restrict__ status)
{
    __shared__ TermsShared shared[TW_WARPS];
    TermsShared &S = shared[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int warp = blockIdx.x * TW_WARPS + (threadIdx.x >> 5);
    const int k = lane < NODES ? warp * NODES + lane : n;
    const int nl = n - 1;
    unsigned below;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(below));
    pdl_wait();
    double mx = 0.0, my = 0.0; // the node
    if (k < n) {
        const double4_32a me = psort[k];
        S.node[lane] = me;
        mx = me.x;
        my = me.y;
    }
    __syncwarp();
    const float fx = (float) mx, fy = (float) my;
    double sum = 0.0; // of the forces' x or y
    // (walk positions and the step limit as in walk())
    const unsigned nend = (unsigned) (nl + n);
    int cur = k < n ? 0 : -1, j = 0, jend = -1;
    const int cap = 3 * n + 64;
    int filled = 0;                       // pairs in the pool
    int mine = 0, head = 0, tail = 0;     // of which this lane's, its first and last
    auto flush = [&](int count) {
        __syncwarp();
        terms_eval<ADJUST>(S, count, nl, scaling, psort, rec_c);
        __syncwarp();
        const bool over = mine > 0 && tail >= count; // one at most, from the last step
        // x by the node's lane, y by the one NODES above
        const int from = lane % NODES;
        int p = __shfl_sync(0xffffffffu, head, from);
        int c = __shfl_sync(0xffffffffu, over ? mine - 1 : mine, from);
        const double *term = S.term[lane / NODES & 1];
        if (lane >= 2 * NODES) c = 0;
        for (; c > 0; c--) {
            sum += term[p];
            p = S.next[p];
        }
        int src = 0;
        if (over) src = S.source[tail];
        __syncwarp();
        mine = 0;
        if (over) {
            head = tail = tail - count;
            S.source[tail] = src;
            S.owner[tail] = (uint8_t) lane;
            mine = 1;
        }
        filled -= count;
    };
    for (int step = 0; __any_sync(0xffffffffu, cur != -1 || j <= jend); step++) {
        int emit = -1;
        if (j <= jend) {
            if (j != k) emit = nl + j;
            j++;
        } else if (cur != -1) {
            if ((unsigned) cur >= nend || step > cap) {
                atomicOr(status + ST_ERROR, ERR_BOUNDS);
                cur = -1;
            } else if (cur >= nl) { // a single node
                if (cur - nl != k) emit = cur;
                cur = rope[cur - nl];
            } else {
                const float4 c = bounds[cur];
                const int2 t = rec_t[cur];
                const float xd = fx - c.x, yd = fy - c.y;
                const float d2 = xd * xd + yd * yd;
                bool far = d2 > c.z;
                if (!far && !(d2 < c.w)) {
                    const double4_32a q = rec_c[cur];
                    const double ex = mx - q.x, ey = my - q.y;
                    far = sq_dist(ex, ey) * theta2 > q.w;
                }
                if (far) {
                    emit = cur;
                    cur = t.y;
                } else if (t.x >= 0) {
                    cur = t.x;
                } else { // at most 8 nodes: node by node
                    j = bucket_first(t.x);
                    jend = bucket_last(t.x);
                    cur = t.y;
                    if (jend >= n) {
                        atomicOr(status + ST_ERROR, ERR_BOUNDS);
                        jend = cur = -1;
                    }
                }
            }
        }
        const unsigned some = __ballot_sync(0xffffffffu, emit >= 0);
        if (!some) continue;
        if (emit >= 0) {
            const int at = filled + __popc(some & below);
            S.source[at] = emit;
            S.owner[at] = (uint8_t) lane;
            if (mine++) S.next[tail] = (uint8_t) at;
            else head = at;
            tail = at;
        }
        filled += __popc(some);
        if (filled >= TW_POOL) flush(TW_POOL);
    }
    if (filled) flush(filled);
    const double other = __shfl_down_sync(0xffffffffu, sum, NODES);
    if (k < n) f[order[k]] = make_double2(sum, other);
}

} // namespace fa2cu
