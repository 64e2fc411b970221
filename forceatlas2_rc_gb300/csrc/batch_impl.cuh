// batch_impl.cuh -- many independent layouts in one persistent launch.
// Included by inst_f32.cu and inst_f64.cu only.
//
// Each graph of a batch is laid out by one thread block from start to end (in
// FP32 one of 1,024 threads, in a launch of its own, if it would outlast the
// others): the block takes the next graph from a work counter (largest first),
// then runs every step of every requested iteration for it:
//   - bounding box;
//   - Morton codes;
//   - a block-level stable radix sort;
//   - the Karras tree;
//   - the bottom-up sums with block-scope arrivals;
//   - the Barnes-Hut walk (or the exact all-pairs sum below the crossover);
//   - gravity and attraction;
//   - the swing/traction totals reduced by the block, the FP64 speed update
//     of that graph;
//   - the displacement.
// No block waits for another while it has work. The blocks of the second launch
// wait at their end for the first launch's (griddepcontrol.wait), which cannot
// depend on them: every block of the first is on an SM before the second starts.
// A graph's result depends on nothing but the graph and the batch's block size,
// and not on which launch had it: it is the same alone or in any mix.
//
// Device arrays are the concatenation of the graphs' arrays (node arrays at
// the graph's first node, its incidences at its first incidence, node indices
// of the incidences local to the graph); the tree arrays of a graph of n
// nodes use n (or 2n for parent) entries from its first node (2x for parent).
#pragma once

#include <algorithm>
#include <cmath>
#include <map>
#include <numeric>
#include <string.h>
#include <vector>

#include "karras.cuh"
#include "kernels.cuh"
#include "layout_impl.cuh" // DevMem
#include "session.h"

namespace fa2cu {

// One graph of a batch, in device memory; the speed state is updated by the
// block that lays the graph out.
struct BatchGraph {
    int n;      // nodes
    int node0;  // first node in the concatenated node arrays
    int exact;  // 1: all-pairs repulsion, 0: Barnes-Hut
    int flags;  // bit 0 strong, 1 linlog, 2 adjust, 3 some node fixed
    double scaling, gravity, theta2d, jitter;
    double speed, efficiency, total_swinging, total_traction;
    int err, pad;
};

// BF_HUBS: a node of mass HUB_MASS or more (FP32: the walk compensates its
// sums)
enum { BF_STRONG = 1, BF_LINLOG = 2, BF_ADJUST = 4, BF_FIXED = 8, BF_HUBS = 16 };

template <class R> struct BatchArrays {
    typedef typename RT<R>::R2 R2;
    typedef typename RT<R>::R4 R4;
    R2 *pos, *f, *fold;
    R *mass, *size, *sw, *tr;
    uint8_t *fixed;
    int *off; // incidence range of node i: off[i] .. off[i+1]-1 (global)
    Inc<R> *inc;
    uint32_t *key, *idx, *key_b, *idx_b;
    R4 *psort;
    int2 *child, *range;
    int *parent, *rope, *visits;
    Agg<R> *agg;
    R4 *rec_c;  // traversal records (common.cuh)
    int2 *rec_t;
    // per block, the cycles spent in each of the 8 phases of an iteration
    // (measurement launches only; nullptr otherwise)
    unsigned long long *prof;
};

// Phases of a batched iteration, as counted in BatchArrays::prof.
enum { BP_CODES, BP_SORT, BP_TREE, BP_SUMS, BP_REPULSION, BP_ATTRACTION, BP_TOTALS, BP_MOVE };

// ---- block-level building blocks ----------------------------------------------

// (block_sort_pairs, the one-block radix sort, is in sort_tree.cuh)

// Sum over the block in a fixed order (H values per thread, of threads t, t + T,
// ...; per warp by shuffles, over the warps by thread 0); the result is valid in
// thread 0.
template <int W, int H> __device__ double block_sum(const double (&v)[H], double *scratch)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
#pragma unroll
    for (int h = 0; h < H; h++) {
        const double x = warp_sum(v[h]);
        if (lane == 0) scratch[h * W + w] = x;
    }
    __syncthreads();
    double s = 0.0, c = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < W * H; k++) neumaier(s, c, scratch[k]);
    return __dadd_rn(s, c);
}

// Two sums over the block of V threads' values each (H a thread): by warp, added
// in pairs, then the V / 32 warps' sums by a warp each, rounded once
// (warp_sum_once). Into a[0] and b[0]. Warps that hold none of the n values have
// 0 and add nothing up (an FP64 instruction of a warp takes the SM 16 cycles).
template <int W, int H>
__device__ void block_sums(int n, const double (&x)[H], const double (&y)[H], double *a, double *b)
{
    static_assert(W * H == 32 && W >= 2, "a lane per warp's sum");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int h = 0; h < H; h++) {
        double u = 0.0, v = 0.0;
        if (32 * (h * W + w) < n) {
            u = warp_sum(x[h]);
            v = warp_sum(y[h]);
        }
        if (lane == 0) {
            a[h * W + w] = u;
            b[h * W + w] = v;
        }
    }
    __syncthreads();
    if (w < 2) {
        double *v = w == 0 ? a : b;
        const double sum = warp_sum_once(v[lane]);
        __syncwarp();
        if (lane == 0) v[0] = sum;
    }
    __syncthreads();
}

// The all-pairs repulsion of an FP32 graph of at most T nodes by its block of T
// threads, into f: two nodes a thread, packed (the terms of k_exact), the sources
// in shared memory and split over the threads, the parts' sums added in order.
//
// Bound by latency: barriers and a chain of n / parts sources. With a thread a
// node (block_exact_tiles) a graph left most threads idle; 10 iterations in ms:
// eight graphs of 60 nodes 0.226 -> 0.099, of 500 0.357 -> 0.262; 2,000 of 100
// nodes 1.82 -> 0.84, of 300 2.47 -> 1.31. Above T nodes these are faster (3,000
// nodes 4.4 against 5.7, 1,100 1.27 against 1.29: as many MUFU operations, and a
// longer record to load for each pair of nodes).
constexpr int BATCH_PARTS = 16; // at most

template <int T> constexpr size_t block_exact_smem()
{
    return T * (sizeof(ExactF32) + 2 * sizeof(float2));
}

template <bool ADJUST, int T>
__device__ __noinline__ void block_exact(int n, float scaling, const float2 *pos,
                                         const float *mass, const float *size, float2 *f,
                                         unsigned char *smem)
{
    ExactF32 *const rec = reinterpret_cast<ExactF32 *>(smem); // T
    float2 *const part = reinterpret_cast<float2 *>(rec + T); // 2 T
    const int tid = threadIdx.x, half = (n + 1) / 2;
    const int parts = min(BATCH_PARTS, T / half); // (2 at least: half <= T / 2)
    const int q = tid / half, slot = tid - q * half;
    if (tid < n) exact_fill(rec + tid, pos[tid], mass[tid], ADJUST ? size[tid] : 0.0f);
    __syncthreads();
    if (q < parts) {
        const ExactF32 a = rec[slot], b = rec[min(slot + half, n - 1)];
        GroupNode me;
        me.x = f2_make(-a.nx[0], -b.nx[0]);
        me.y = f2_make(-a.ny[0], -b.ny[0]);
        const float sa = a.r[0], sb = b.r[0];
        f2 ax = 0, ay = 0;
        const int seg = (n + parts - 1) / parts;
        const int from = min(n, q * seg), to = min(n, from + seg);
        unsigned at = smem_addr(rec + from);
#pragma unroll 4
        for (int j = from; j < to; j++, at += (unsigned) sizeof(ExactF32)) {
            f2 nx, ny, mm, r = 0;
            lds_2<0>(at, nx, ny);
            if (ADJUST)
                lds_2<16>(at, mm, r);
            else
                mm = lds_1<16>(at);
            exact_term<ADJUST>(me, sa, sb, nx, ny, mm, r, ax, ay);
        }
        float xa, xb, ya, yb;
        f2_split(ax, xa, xb);
        f2_split(ay, ya, yb);
        part[q * n + slot] = make_float2(xa, ya);
        if (slot + half < n) part[q * n + slot + half] = make_float2(xb, yb);
    }
    __syncthreads();
    if (tid < n) {
        float2 v = part[tid];
        for (int r = 1; r < parts; r++) {
            const float2 o = part[r * n + tid];
            v.x += o.x;
            v.y += o.y;
        }
        const float m = scaling * rec[tid].m[0];
        f[tid] = make_float2(v.x * m, v.y * m);
    }
}

// The same of a larger graph, or in FP64: every node's sum by a thread, over
// tiles of T records staged in shared memory, in node order. two: the tile shape
// (autotuned), two nodes per thread (i and i + T), each tile record feeding two
// independent sums, or one; every node sums j ascending either way. (Inlined and
// unrolled: eight FP32 graphs of 3,000 nodes, 10 iterations, 4.6 ms; a function
// of its own 5.8, unrolled by four 4.7, not at all 5.4.)
template <class R, bool ADJUST, int T>
__device__ __forceinline__ void block_exact_tiles(int n, bool two, R scaling,
                                               const typename RT<R>::R2 *pos, const R *mass,
                                               const R *size, typename RT<R>::R4 *psort,
                                               typename RT<R>::R2 *f, unsigned char *smem)
{
    typedef typename RT<R>::R2 R2;
    typedef typename RT<R>::R4 R4;
    const int tid = threadIdx.x;
    R4 *const tile = reinterpret_cast<R4 *>(smem);
    for (int i = tid; i < n; i += T) {
        const R2 p = pos[i];
        psort[i] = mk4<R>(p.x, p.y, mass[i], ADJUST ? size[i] : R(0));
    }
    for (int i0 = 0; i0 < n; i0 += two ? 2 * T : T) {
        const int ia = i0 + tid, ib = two ? ia + T : n;
        const R4 zero = mk4<R>(R(0), R(0), R(0), R(0));
        const R4 ma = ia < n ? psort[ia] : zero, mb = ib < n ? psort[ib] : zero;
        R axa = R(0), aya = R(0), axb = R(0), ayb = R(0);
        for (int j0 = 0; j0 < n; j0 += T) {
            __syncthreads();
            if (j0 + tid < n) tile[tid] = psort[j0 + tid];
            __syncthreads();
            const int m = min(T, n - j0);
            // one source on a node (FP32 without radii: d2 carries 1e-30, as in
            // k_exact, and scaling * m_i comes once, at the end)
            auto add = [&](const R4 &me, const R4 &q, R &ax, R &ay) {
                const R xd = me.x - q.x, yd = me.y - q.y;
                if constexpr (sizeof(R) == 4 && !ADJUST) {
                    const float g = q.z * __fdividef(1.0f, fmaf(xd, xd, fmaf(yd, yd, 1e-30f)));
                    ax = fmaf(xd, g, ax);
                    ay = fmaf(yd, g, ay);
                } else {
                    const R g = rep_factor<R, ADJUST>(xd * xd + yd * yd, me.z * q.z,
                                                      ADJUST ? me.w + q.w : R(0), scaling);
                    ax += xd * g;
                    ay += yd * g;
                }
            };
            if (two) {
#pragma unroll 16
                for (int jj = 0; jj < m; jj++) {
                    const R4 q = tile[jj];
                    add(ma, q, axa, aya);
                    add(mb, q, axb, ayb);
                }
            } else {
#pragma unroll 8
                for (int jj = 0; jj < m; jj++) add(ma, tile[jj], axa, aya);
            }
        }
        if (sizeof(R) == 4 && !ADJUST) {
            const R sa = scaling * ma.z, sb = scaling * mb.z;
            axa *= sa;
            aya *= sa;
            axb *= sb;
            ayb *= sb;
        }
        if (ia < n) f[ia] = mk2<R>(axa, aya);
        if (ib < n) f[ib] = mk2<R>(axb, ayb);
    }
}

// ---- the persistent kernel -----------------------------------------------------

// FP32: two blocks of 512 (four of 256) threads per SM, 64 registers a thread,
// which the group walk wants (three blocks at 40 registers: 3.01 against 2.85
// ms an iteration of 1,024 graphs of 50 to 20,000 nodes, which lasted as long as
// its largest graph; the walk's arrays of three, 76 KB each, do not fit an SM).
// FP64 needs more registers: one block of 512 (two of 256).
// FP32 graphs that would outlast the others (wide_graphs) are taken by blocks
// of WIDE threads, which have an SM each. They are launched first, and the
// other blocks when all of them have started (launch_kernel).
constexpr int WIDE = 1024;
constexpr int WIDE_MIN = 1024; // nodes, below which such a block has idle threads

template <class R, int T>
__global__ void __launch_bounds__(T, (sizeof(R) == 8 ? 512 : 1024) / T)
k_batch(int ngraphs, BatchGraph *graphs, const int *queue, int *next, int iterations,
        BatchArrays<R> A, int npt, int *status)
{
    typedef typename RT<R>::R2 R2;
    typedef typename RT<R>::R4 R4;
    constexpr int W = T / 32;
    // the threads that the totals are made for: the same sums whatever T (a
    // graph's layout does not depend on the batch it is in)
    constexpr int V = sizeof(R) == 4 ? WIDE : T, H = V / T;
    // the sort's digit counts; in the same space the exact sum's record tile
    // (T records of at most 32 bytes), and the group walk's arrays
    extern __shared__ __align__(16) unsigned char batch_smem[];
    uint32_t(*cnt)[256] = reinterpret_cast<uint32_t(*)[256]>(batch_smem);
    __shared__ uint32_t dbase[256];
    __shared__ double red[V / 32], red2[V / 32];
    __shared__ R mins[4][W];
    __shared__ __align__(16) double quant[6]; // (as k_bbox makes it)
    __shared__ SpeedTerms terms;
    __shared__ double sh_speed;
    __shared__ int sh_g, sh_stop;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (T == WIDE) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    for (;;) {
        if (tid == 0) sh_g = atomicAdd(next, 1);
        __syncthreads();
        const int qi = sh_g;
        __syncthreads();
        if (qi >= ngraphs) break;
        BatchGraph *G = graphs + queue[qi];
        const int n = G->n, b0 = G->node0;
        const bool exact = G->exact != 0;
        const int flags = G->flags;
        const bool strong = flags & BF_STRONG, linlog = flags & BF_LINLOG;
        const bool adjust = flags & BF_ADJUST, anyfix = flags & BF_FIXED;
        const bool hubs = flags & BF_HUBS;
        const R scaling = (R) G->scaling, gravity = (R) G->gravity;
        const double theta2d = G->theta2d;
        const R theta2 = (R) theta2d;
        // the FP32 records' scale of size^2 (region_far)
        const R wscale = (R) ((1.0 + (double) DECIDE_BAND) / theta2d);
        R2 *pos = A.pos + b0, *f = A.f + b0, *fold = A.fold + b0;
        const R *mass = A.mass + b0;
        const R *size = A.size ? A.size + b0 : nullptr;
        R *sw = A.sw + b0, *tr = A.tr ? A.tr + b0 : nullptr;
        const uint8_t *fixed = anyfix ? A.fixed + b0 : nullptr;
        const int *off = A.off + b0;
        uint32_t *key = A.key + b0, *idx = A.idx + b0, *kb = A.key_b + b0, *vb = A.idx_b + b0;
        R4 *psort = A.psort + b0;
        int2 *child = A.child + b0, *range = A.range + b0;
        int *parent = A.parent + 2 * (size_t) b0, *rope = A.rope + b0, *visits = A.visits + b0;
        Agg<R> *agg = A.agg + b0;
        R4 *rec_c = A.rec_c + b0;
        int2 *rec_t = A.rec_t + b0;
        if (tid == 0) {
            sh_speed = G->speed;
            sh_stop = 0;
            terms = speed_terms(n);
        }
        double speed = G->speed, eff = G->efficiency;

        // phase clock of thread 0, read after each block-wide barrier
        long long tlast = clock64();
        auto phase = [&](int ph) {
            if (A.prof && tid == 0) {
                const long long t = clock64();
                A.prof[(size_t) blockIdx.x * 8 + ph] += (unsigned long long) (t - tlast);
                tlast = t;
            }
        };
        for (int it = 0; it < iterations; it++) {
            __syncthreads();
            phase(BP_MOVE);
            if (sh_stop) break;
            if (exact || n < 2) {
                const bool two = npt == 2 && n > T;
                bool small = false;
                if constexpr (sizeof(R) == 4) {
                    small = n <= T;
                    if (small && adjust)
                        block_exact<true, T>(n, scaling, pos, mass, size, f, batch_smem);
                    else if (small)
                        block_exact<false, T>(n, scaling, pos, mass, size, f, batch_smem);
                }
                if (!small && adjust)
                    block_exact_tiles<R, true, T>(n, two, scaling, pos, mass, size, psort, f,
                                                  batch_smem);
                else if (!small)
                    block_exact_tiles<R, false, T>(n, two, scaling, pos, mass, size, psort, f,
                                                   batch_smem);
            } else {
                // bounding box and the Morton quantisation
                R mnx = pos[0].x, mxx = mnx, mny = pos[0].y, mxy = mny;
                for (int i = tid; i < n; i += T) {
                    const R2 p = pos[i];
                    mnx = cl_min(mnx, p.x);
                    mny = cl_min(mny, p.y);
                    mxx = cl_max(mxx, p.x);
                    mxy = cl_max(mxy, p.y);
                }
                for (int o = 16; o > 0; o >>= 1) {
                    mnx = cl_min(mnx, __shfl_down_sync(0xffffffffu, mnx, o));
                    mny = cl_min(mny, __shfl_down_sync(0xffffffffu, mny, o));
                    mxx = cl_max(mxx, __shfl_down_sync(0xffffffffu, mxx, o));
                    mxy = cl_max(mxy, __shfl_down_sync(0xffffffffu, mxy, o));
                }
                if (lane == 0) {
                    mins[0][w] = mnx;
                    mins[1][w] = mny;
                    mins[2][w] = mxx;
                    mins[3][w] = mxy;
                }
                __syncthreads();
                if (tid == 0) {
                    for (int k = 1; k < W; k++) {
                        mnx = cl_min(mnx, mins[0][k]);
                        mny = cl_min(mny, mins[1][k]);
                        mxx = cl_max(mxx, mins[2][k]);
                        mxy = cl_max(mxy, mins[3][k]);
                    }
                    quant_make<R>(mnx, mny, mxx, mxy, quant);
                }
                __syncthreads();
                const MortonQuant<R> Q(quant);
                for (int i = tid; i < n; i += T) {
                    key[i] = Q.key(pos[i]);
                    idx[i] = (uint32_t) i;
                }
                __syncthreads();
                phase(BP_CODES);
                block_sort_pairs<W>(n, key, idx, kb, vb, cnt, dbase);
                phase(BP_SORT);
                for (int k = tid; k < n; k += T) {
                    const uint32_t i = idx[k];
                    const R2 p = pos[i];
                    psort[k] = mk4<R>(p.x, p.y, mass[i], adjust ? size[i] : R(0));
                }
                for (int i = tid; i < n - 1; i += T)
                    karras_one(i, n, key, child, range, parent, rope, visits);
                __syncthreads();
                phase(BP_TREE);
                // contiguous leaves per thread: a thread's later climbs find
                // the regions of its earlier ones complete
                const int per = (n + T - 1) / T;
                for (int q = 0; q < per; q++) {
                    const int k = tid * per + q;
                    if (k < n)
                        climb<R>(k, n, psort, child, parent, range, rope, visits, agg,
                                       rec_c, rec_t, wscale, status);
                }
                __syncthreads();
                phase(BP_SUMS);
                // FP32: the group walk (the single layout's), compensated for
                // hubs, every warp from the root: a block's shared top is a
                // barrier that few blocks an SM do not hide (3.02 against 2.85
                // ms; with one walk a thread 3.70). FP64: the per-thread walk
                // in the reference's order.
                if constexpr (sizeof(R) == 4) {
                    GroupTopShared &top = *reinterpret_cast<GroupTopShared *>(batch_smem);
                    GroupWalkShared *gw = reinterpret_cast<GroupWalkShared *>(&top + 1);
                    auto go = [&](auto walk_block) {
                        for (int k0 = 0; k0 < n; k0 += T) {
                            const R2 fk = walk_block(k0);
                            if (k0 + tid < n) f[idx[k0 + tid]] = fk;
                        }
                    };
                    if (adjust && hubs)
                        go([&](int k0) {
                            return group_walk_block<true, true>(top, gw, k0, 1, false, n, scaling, theta2d,
                                                                psort, rec_c, rec_t, child, agg,
                                                                status);
                        });
                    else if (adjust)
                        go([&](int k0) {
                            return group_walk_block<true, false>(top, gw, k0, 1, false, n, scaling,
                                                                 theta2d, psort, rec_c, rec_t,
                                                                 child, agg, status);
                        });
                    else if (hubs)
                        go([&](int k0) {
                            return group_walk_block<false, true>(top, gw, k0, 1, false, n, scaling,
                                                                 theta2d, psort, rec_c, rec_t,
                                                                 child, agg, status);
                        });
                    else
                        go([&](int k0) {
                            return group_walk_block<false, false>(top, gw, k0, 1, false, n, scaling,
                                                                  theta2d, psort, rec_c, rec_t,
                                                                  child, agg, status);
                        });
                } else {
                    for (int k = tid; k < n; k += T)
                        f[idx[k]] = adjust ? walk<R, true>(k, n, scaling, theta2, theta2d, psort,
                                                           rec_c, rec_t, agg, rope, status)
                                           : walk<R, false>(k, n, scaling, theta2, theta2d, psort,
                                                            rec_c, rec_t, agg, rope, status);
                }
            }
            __syncthreads();
            phase(BP_REPULSION);
            for (int i = tid; i < n; i += T)
                attract_one<R>(i, gravity, strong, linlog, adjust, pos, mass, size, off, A.inc,
                               f);
            __syncthreads();
            phase(BP_ATTRACTION);
            // swinging and traction; totals in double in a fixed order: in
            // FP64 up to SERIAL_TOTALS_MAX nodes serially in node order (the
            // reference's order, as the single-graph path), else per thread
            // and over the block
            const bool serial = serial_totals<R>(n);
            double ts[H] = {}, tt[H] = {};
            for (int i0 = tid; i0 < n; i0 += V) {
#pragma unroll
                for (int h = 0; h < H; h++) {
                    const int i = i0 + h * T;
                    if (i >= n) break;
                    const R2 a = f[i], b = fold[i];
                    const R sx = b.x - a.x, sy = b.y - a.y;
                    const R tx = b.x + a.x, ty = b.y + a.y;
                    const R m = mass[i];
                    const R s = m * fsqrt(sx * sx + sy * sy);
                    const R t = R(0.5) * m * fsqrt(tx * tx + ty * ty);
                    sw[i] = s;
                    if (serial) tr[i] = t;
                    if (fixed && fixed[i]) continue;
                    ts[h] = __dadd_rn(ts[h], (double) s);
                    tt[h] = __dadd_rn(tt[h], (double) t);
                }
            }
            double tsw, ttr;
            if constexpr (sizeof(R) == 4) {
                // both at once (a serial sum over the warps, compensated, took
                // 100 dependent FP64 operations)
                block_sums<W>(n, ts, tt, red, red2);
                tsw = red[0];
                ttr = red2[0];
            } else {
                tsw = block_sum<W>(ts, red);
                ttr = block_sum<W>(tt, red2);
            }
            if (serial) {
                __syncthreads(); // sw / tr written by every thread
                if (tid < 64) { // a warp each
                    const R *v = tid < 32 ? sw : tr;
                    const double sum = ordered_sum(n, [&](int i) {
                        return fixed && fixed[i] ? 0.0 : (double) v[i];
                    });
                    if ((tid & 31) == 0) red[tid >> 5] = sum;
                }
                __syncthreads();
                tsw = red[0];
                ttr = red[1];
            }
            if (tid == 0) {
                if (!(tsw == tsw) || !(ttr == ttr)) {
                    sh_stop = 1;
                    G->err = ERR_NAN;
                    atomicOr(status + ST_ERROR, ERR_NAN);
                } else {
                    SpeedState s0;
                    s0.speed = speed;
                    s0.efficiency = eff;
                    s0.jitter_tolerance = G->jitter;
                    s0.terms = terms;
                    update_speed(&s0, tsw, ttr);
                    speed = s0.speed;
                    eff = s0.efficiency;
                    sh_speed = speed;
                    G->total_swinging = tsw;
                    G->total_traction = ttr;
                }
            }
            __syncthreads();
            phase(BP_TOTALS);
            if (sh_stop) break;
            const R sp = (R) sh_speed;
            for (int i = tid; i < n; i += T) {
                const R2 a = f[i];
                fold[i] = a;
                if (fixed && fixed[i]) continue;
                R factor;
                if (adjust) {
                    const R df = fsqrt(a.x * a.x + a.y * a.y);
                    factor = fdiv(R(0.1) * sp, R(1) + fsqrt(sp * sw[i]));
                    if (df > R(0)) {
                        if (factor * df > R(10)) factor = fdiv(R(10), df);
                    } else {
                        factor = R(0);
                    }
                } else {
                    factor = fdiv(sp, R(1) + fsqrt(sp * sw[i]));
                }
                R2 p = pos[i];
                p.x += a.x * factor;
                p.y += a.y * factor;
                pos[i] = p;
            }
        }
        __syncthreads();
        if (tid == 0) {
            G->speed = speed;
            G->efficiency = eff;
        }
    }
    // (what follows in the stream waits for this grid: it ends after the wide
    // blocks'; each of those is on an SM already)
    if (T != WIDE) pdl_wait();
}

// Dynamic shared memory of k_batch.
template <class R, int T> constexpr size_t batch_smem_bytes()
{
    const size_t sort = (size_t) (T / 32) * 256 * sizeof(uint32_t);
    const size_t walk =
        sizeof(R) == 4 ? sizeof(GroupTopShared) + (T / 32) * sizeof(GroupWalkShared) : 0;
    static_assert(sizeof(R) == 8 || walk >= block_exact_smem<T>(), "the exact sum's arrays fit");
    return sort > walk ? sort : walk;
}

// ---- host side -------------------------------------------------------------------

template <class R> struct Batch : BatchBase {
    typedef typename RT<R>::R2 R2;
    typedef typename RT<R>::R4 R4;
    int G = 0, N = 0, E = 0, threads = 512, npt = 2;
    cudaStream_t s = nullptr;
    DevMem mem;
    BatchArrays<R> A{};
    BatchGraph *graphs = nullptr;
    int *queue = nullptr, *next = nullptr, *status = nullptr;
    std::vector<int> node0, nsize;
    int blocks = 0;                // of `threads`
    int nwide = 0, wide_blocks = 0; // the first nwide graphs of the queue: blocks of WIDE
    std::map<int, cudaGraphExec_t> execs; // iteration count -> captured launch

    ~Batch() override
    {
        if (s) cudaStreamSynchronize(s);
        drop_graphs();
        mem.release();
        if (s) cudaStreamDestroy(s);
    }

    cudaStream_t stream() override { return s; }
    double bytes() const override { return mem.bytes; }
    int count() const override { return G; }

    int open(const fa2_full_params *ps, int count, const double *const *pos, int exact_below,
             int nthreads, int nodes_per_thread)
    {
        G = count;
        threads = nthreads;
        npt = nodes_per_thread;
        node0.resize(G);
        nsize.resize(G);
        bool any_adjust = false, any_fixed = false;
        std::vector<uint8_t> gfixed(G, 0); // graph g has a fixed node
        long long nn = 0, ee = 0;
        for (int g = 0; g < G; g++) {
            const fa2_full_params &p = ps[g];
            node0[g] = (int) nn;
            nsize[g] = p.n;
            nn += p.n;
            ee += p.inc_off[p.n];
            any_adjust |= p.adjust != 0;
            for (int i = 0; i < p.n && p.fixed && !gfixed[g]; i++) gfixed[g] = p.fixed[i] != 0;
            any_fixed |= gfixed[g] != 0;
        }
        if (nn >= (1LL << 31) / 2 || ee >= (1LL << 31)) {
            set_message("the batch is too large (at most 2^30 nodes and 2^31 incidences)");
            return 1;
        }
        N = (int) nn;
        E = (int) ee;
        FA2_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking),
                "could not create a CUDA stream", 1);
        const size_t n1 = (size_t) N;
        A.pos = mem.get<R2>(n1);
        A.f = mem.get<R2>(n1);
        A.fold = mem.get<R2>(n1);
        A.mass = mem.get<R>(n1);
        A.size = any_adjust ? mem.get<R>(n1) : nullptr;
        A.sw = mem.get<R>(n1);
        A.tr = sizeof(R) == 8 ? mem.get<R>(n1) : nullptr;
        A.fixed = any_fixed ? mem.get<uint8_t>(n1) : nullptr;
        A.off = mem.get<int>(n1 + 1);
        A.inc = mem.get<Inc<R>>((size_t) E);
        A.key = mem.get<uint32_t>(n1);
        A.idx = mem.get<uint32_t>(n1);
        A.key_b = mem.get<uint32_t>(n1);
        A.idx_b = mem.get<uint32_t>(n1);
        A.psort = mem.get<R4>(n1);
        A.child = mem.get<int2>(n1);
        A.range = mem.get<int2>(n1);
        A.parent = mem.get<int>(2 * n1);
        A.rope = mem.get<int>(n1);
        A.visits = mem.get<int>(n1);
        A.agg = mem.get<Agg<R>>(n1);
        A.rec_c = mem.get<R4>(n1);
        A.rec_t = mem.get<int2>(n1);
        graphs = mem.get<BatchGraph>((size_t) G);
        queue = mem.get<int>((size_t) G);
        next = mem.get<int>(2); // of the wide blocks, of the others
        status = mem.get<int>(ST_COUNT);
        if (mem.failed) {
            set_cuda_error("could not allocate memory on the device", mem.err);
            return 1;
        }
        // the graphs, concatenated on the host in the device precision
        std::vector<R2> hp(n1);
        std::vector<R> hm(n1), hs(any_adjust ? n1 : 0);
        std::vector<uint8_t> hf(any_fixed ? n1 : 0);
        std::vector<int> hoff(n1 + 1);
        std::vector<Inc<R>> hinc((size_t) std::max(E, 1));
        std::vector<BatchGraph> hg(G);
        int e0 = 0;
        for (int g = 0; g < G; g++) {
            const fa2_full_params &p = ps[g];
            const int n = p.n, b = node0[g];
            for (int i = 0; i < n; i++) {
                hp[b + i] = mk2h(pos[g][i], pos[g][n + i]);
                hm[b + i] = (R) p.mass[i];
                if (any_adjust) hs[b + i] = p.adjust ? (R) p.size[i] : R(0);
                if (any_fixed) hf[b + i] = gfixed[g] && p.fixed[i] != 0;
                hoff[b + i] = e0 + p.inc_off[i];
            }
            for (int e = 0; e < p.inc_off[n]; e++) {
                hinc[e0 + e].j = p.inc_node[e];
                hinc[e0 + e].coef = (R) p.inc_coef[e];
            }
            e0 += p.inc_off[n];
            BatchGraph &q = hg[g];
            memset(&q, 0, sizeof(q));
            q.n = n;
            q.node0 = b;
            q.exact = n < exact_below ? 1 : 0;
            int fl = 0;
            if (p.strong) fl |= BF_STRONG;
            if (p.linlog) fl |= BF_LINLOG;
            if (p.adjust) fl |= BF_ADJUST;
            if (gfixed[g]) fl |= BF_FIXED;
            for (int i = 0; i < n; i++)
                if ((float) p.mass[i] >= HUB_MASS) {
                    fl |= BF_HUBS;
                    break;
                }
            q.flags = fl;
            q.scaling = p.scaling;
            q.gravity = p.gravity;
            q.theta2d = p.theta * p.theta;
            q.jitter = p.jitter_tolerance;
            q.speed = 1.0;
            q.efficiency = 1.0;
        }
        hoff[n1] = e0;
        // largest work first: a block that takes a graph lays it out to the end
        std::vector<int> hq(G);
        std::iota(hq.begin(), hq.end(), 0);
        auto cost = [&](int g) {
            return hg[g].exact ? (double) hg[g].n * hg[g].n : 300.0 * hg[g].n;
        };
        std::stable_sort(hq.begin(), hq.end(), [&](int a, int b) { return cost(a) > cost(b); });
        int sms = 0, per_sm = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        if constexpr (sizeof(R) == 4) {
            const std::vector<char> wide = wide_graphs(cost, hg.data(), sms);
            nwide = (int) (std::stable_partition(hq.begin(), hq.end(),
                                                 [&](int g) { return wide[g]; }) -
                           hq.begin());
        }
        int rc = 0;
        auto up = [&](void *dst, const void *src, size_t bytes) {
            if (!rc && bytes)
                rc = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s) != cudaSuccess;
        };
        up(A.pos, hp.data(), n1 * sizeof(R2));
        up(A.mass, hm.data(), n1 * sizeof(R));
        if (any_adjust) up(A.size, hs.data(), n1 * sizeof(R));
        if (any_fixed) up(A.fixed, hf.data(), n1);
        up(A.off, hoff.data(), (n1 + 1) * sizeof(int));
        up(A.inc, hinc.data(), (size_t) E * sizeof(Inc<R>));
        up(graphs, hg.data(), (size_t) G * sizeof(BatchGraph));
        up(queue, hq.data(), (size_t) G * sizeof(int));
        if (!rc) rc = cudaMemsetAsync(A.fold, 0, n1 * sizeof(R2), s) != cudaSuccess;
        if (!rc) rc = cudaMemsetAsync(status, 0, ST_COUNT * sizeof(int), s) != cudaSuccess;
        if (!rc) rc = cudaStreamSynchronize(s) != cudaSuccess;
        if (rc) {
            set_cuda_error("could not send the batch to the device", cudaGetLastError());
            return 1;
        }
        auto setup = [&](auto kernel, int th, size_t smem) {
            FA2_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int) smem),
                    "cudaFuncSetAttribute", 1);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, th, smem);
            return 0;
        };
        if constexpr (sizeof(R) == 4) {
            if (nwide && setup(k_batch<R, WIDE>, WIDE, batch_smem_bytes<R, WIDE>())) return 1;
            wide_blocks = std::min(nwide, sms * std::max(per_sm, 1));
        }
        if (threads == 256 ? setup(k_batch<R, 256>, 256, batch_smem_bytes<R, 256>())
                           : setup(k_batch<R, 512>, 512, batch_smem_bytes<R, 512>()))
            return 1;
        blocks = std::min(G - nwide, sms * std::max(per_sm, 1));
        return 0;
    }

    // The graphs that blocks of WIDE threads lay out: those over the tree whose
    // work is more than 0.55 of an SM's share of the whole (if these are more
    // than the SMs: more than the share). A block of 512 on half an SM would
    // still be at work on them when the others are done.
    // 10 iterations in ms, blocks of 512 and with wide ones: 1,024 graphs of 50
    // to 20,000 nodes 29.3 -> 16.0, 300 of 50 to 8,000 10.4 -> 6.2, ten of
    // 20,000 21.6 -> 15.6, 152 of 3,000 3.17 -> 2.40, eight of 2,100 2.26 ->
    // 1.84. 300 of 8,000, all of them wide, 12.0 -> 12.8: two waves of barriers
    // that nothing hides. Exact graphs of 3,000 nodes 4.4 -> 5.2.
    template <class Cost> std::vector<char> wide_graphs(Cost cost, const BatchGraph *g, int sms)
    {
        double share = 0.0;
        for (int q = 0; q < G; q++) share += cost(q) / std::max(sms, 1);
        std::vector<char> wide(G);
        for (double line : {0.55 * share, share}) {
            int count = 0;
            for (int q = 0; q < G; q++) {
                wide[q] = !g[q].exact && g[q].n >= WIDE_MIN && cost(q) > line;
                count += wide[q];
            }
            if (count <= sms) break;
        }
        return wide;
    }

    static R2 mk2h(double x, double y)
    {
        R2 v;
        v.x = (R) x;
        v.y = (R) y;
        return v;
    }

    // The wide blocks, then (a programmatic launch: when every wide block has
    // started) the others, on what is left of the GPU.
    void launch_kernel(int iterations, const BatchArrays<R> &arrays)
    {
        if constexpr (sizeof(R) == 4) {
            if (nwide)
                k_batch<R, WIDE><<<wide_blocks, WIDE, batch_smem_bytes<R, WIDE>(), s>>>(
                    nwide, graphs, queue, next, iterations, arrays, npt, status);
        }
        if (G == nwide) return;
        BatchArrays<R> rest = arrays;
        if (rest.prof) rest.prof += (size_t) wide_blocks * 8;
        auto go = [&](auto kernel, size_t smem) {
            launch_k(nwide > 0, kernel, dim3(blocks), dim3(threads), smem, s, G - nwide, graphs,
                     (const int *) (queue + nwide), next + 1, iterations, rest, npt, status);
        };
        if (threads == 256)
            go(k_batch<R, 256>, batch_smem_bytes<R, 256>());
        else
            go(k_batch<R, 512>, batch_smem_bytes<R, 512>());
    }

    void launch(int iterations)
    {
        cudaMemsetAsync(next, 0, 2 * sizeof(int), s);
        launch_kernel(iterations, A);
    }

    // The work-counter reset and the persistent launch, captured once per
    // iteration count (a few counts kept) and replayed.
    int iterate(int iterations) override
    {
        cudaSetDevice(device);
        auto it = execs.find(iterations);
        if (it == execs.end()) {
            if (execs.size() >= 8) drop_graphs();
            cudaGraph_t g = nullptr;
            cudaGraphExec_t x = nullptr;
            FA2_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal),
                    "could not capture the batched launch", 1);
            launch(iterations);
            cudaError_t e = cudaStreamEndCapture(s, &g);
            if (e == cudaSuccess) e = cudaGraphInstantiate(&x, g, 0);
            if (g) cudaGraphDestroy(g);
            if (e != cudaSuccess) {
                set_cuda_error("could not capture the batched launch", e);
                return 1;
            }
            it = execs.emplace(iterations, x).first;
        }
        FA2_TRY(cudaGraphLaunch(it->second, s), "the computation on the GPU failed", 1);
        return 0;
    }

    void drop_graphs()
    {
        for (auto &kv : execs) cudaGraphExecDestroy(kv.second);
        execs.clear();
    }

    // Cycles of each phase, summed over the blocks, over `iterations`
    // iterations of every graph (an uncaptured, instrumented launch).
    int phase_cycles(int iterations, double out[8]) override
    {
        cudaSetDevice(device);
        DevMem tmp;
        const size_t count = (size_t) (wide_blocks + blocks) * 8;
        unsigned long long *prof = tmp.get<unsigned long long>(count);
        if (tmp.failed) {
            set_cuda_error("could not allocate memory on the device", tmp.err);
            return 1;
        }
        int rc = cudaMemsetAsync(prof, 0, count * sizeof(unsigned long long), s) != cudaSuccess;
        BatchArrays<R> P = A;
        P.prof = prof;
        if (!rc) rc = cudaMemsetAsync(next, 0, 2 * sizeof(int), s) != cudaSuccess;
        if (!rc) launch_kernel(iterations, P);
        std::vector<unsigned long long> h(count);
        if (!rc)
            rc = cudaMemcpyAsync(h.data(), prof, h.size() * sizeof(unsigned long long),
                                 cudaMemcpyDeviceToHost, s) != cudaSuccess;
        if (!rc) rc = cudaStreamSynchronize(s) != cudaSuccess;
        tmp.release();
        if (rc) {
            set_message("the computation on the GPU failed");
            return 1;
        }
        for (int k = 0; k < 8; k++) out[k] = 0.0;
        for (size_t b = 0; b < count; b++) out[b % 8] += (double) h[b];
        return 0;
    }

    int sync() override
    {
        cudaSetDevice(device);
        FA2_TRY(cudaStreamSynchronize(s), "the computation on the GPU failed", 1);
        int h = 0;
        FA2_TRY(cudaMemcpy(&h, status + ST_ERROR, sizeof(int), cudaMemcpyDeviceToHost),
                "the computation on the GPU failed", 1);
        if (h & ERR_NAN) {
            set_message("the computation on the GPU produced invalid numbers");
            return 1;
        }
        if (h) {
            set_message("the computation on the GPU failed (an index left its bounds)");
            return 1;
        }
        return 0;
    }

    int positions(int g, double *out) override
    {
        if (g < 0 || g >= G) {
            set_message("there is no graph %d in this batch", g + 1);
            return 1;
        }
        cudaSetDevice(device);
        const int n = nsize[g];
        std::vector<R2> h((size_t) n);
        FA2_TRY(cudaMemcpyAsync(h.data(), A.pos + node0[g], (size_t) n * sizeof(R2),
                                cudaMemcpyDeviceToHost, s),
                "could not fetch the layout from the device", 1);
        FA2_TRY(cudaStreamSynchronize(s), "could not fetch the layout from the device", 1);
        for (int i = 0; i < n; i++) {
            out[i] = (double) h[i].x;
            out[n + i] = (double) h[i].y;
        }
        return 0;
    }

    // Graph g's forces of the last iteration (at the positions before its
    // displacement): the move keeps them in f.
    int forces(int g, double *out) override
    {
        if (g < 0 || g >= G) {
            set_message("there is no graph %d in this batch", g + 1);
            return 1;
        }
        cudaSetDevice(device);
        const int n = nsize[g];
        std::vector<R2> h((size_t) n);
        FA2_TRY(cudaMemcpyAsync(h.data(), A.f + node0[g], (size_t) n * sizeof(R2),
                                cudaMemcpyDeviceToHost, s),
                "could not fetch the forces from the device", 1);
        FA2_TRY(cudaStreamSynchronize(s), "could not fetch the forces from the device", 1);
        for (int i = 0; i < n; i++) {
            out[i] = (double) h[i].x;
            out[n + i] = (double) h[i].y;
        }
        return 0;
    }
    int speed(int g, double state[4]) override
    {
        if (g < 0 || g >= G) {
            set_message("there is no graph %d in this batch", g + 1);
            return 1;
        }
        BatchGraph h;
        FA2_TRY(cudaMemcpy(&h, graphs + g, sizeof(h), cudaMemcpyDeviceToHost), "cudaMemcpy", 1);
        state[0] = h.speed;
        state[1] = h.efficiency;
        state[2] = h.total_swinging;
        state[3] = h.total_traction;
        return 0;
    }

};

template <class R>
BatchBase *make_batch(const fa2_full_params *ps, int count, const double *const *pos,
                      int exact_below, int threads, int npt)
{
    const int dev = ps[0].device;
    FA2_TRY(cudaSetDevice(dev), "could not use the CUDA device", nullptr);
    Batch<R> *B = new Batch<R>();
    B->device = dev;
    if (B->open(ps, count, pos, exact_below, threads, npt)) {
        delete B;
        return nullptr;
    }
    return B;
}

// ---- autotuner -------------------------------------------------------------------
// The exact-vs-Barnes-Hut crossover, the block size and the exact sum's tile
// shape, measured on the device: Erdos-Renyi graphs (mean degree 8), two per
// SM, laid out for 2 iterations (after 2) in each mode, at 64, 128, .. 16384
// nodes until the tree is faster, then at quarter-octave sizes below that
// one; the crossover is the smallest size measured at which the tree is
// faster. Block sizes 256 and 512 are compared on 2048-node graphs; then 1
// or 2 nodes per thread of the exact sum on graphs of 3/4 of the crossover
// (at least one block of nodes more).

struct TuneGraphs {
    std::vector<std::vector<int>> off, node;
    std::vector<std::vector<double>> coef, mass, size, pos;
    std::vector<fa2_full_params> ps;
    std::vector<const double *> pp;
};

static uint64_t splitmix(uint64_t &x)
{
    uint64_t z = (x += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

static void tune_graphs(TuneGraphs &t, int n, int copies, int device, int use_double)
{
    t.off.resize(copies);
    t.node.resize(copies);
    t.coef.resize(copies);
    t.mass.resize(copies);
    t.size.resize(copies);
    t.pos.resize(copies);
    t.ps.resize(copies);
    t.pp.resize(copies);
    uint64_t seed = 12345 + (uint64_t) n;
    for (int c = 0; c < copies; c++) {
        const int m = 4 * n;
        std::vector<int> a(m), b(m), deg(n, 0);
        for (int e = 0; e < m; e++) {
            a[e] = (int) (splitmix(seed) % (uint64_t) n);
            b[e] = (int) (splitmix(seed) % (uint64_t) n);
            if (a[e] == b[e]) b[e] = (b[e] + 1) % n;
            deg[a[e]]++;
            deg[b[e]]++;
        }
        auto &off = t.off[c];
        off.assign(n + 1, 0);
        for (int i = 0; i < n; i++) off[i + 1] = off[i] + deg[i];
        std::vector<int> at(off.begin(), off.end() - 1);
        t.node[c].resize(2 * m);
        t.coef[c].assign(2 * m, 1.0);
        for (int e = 0; e < m; e++) {
            t.node[c][at[a[e]]++] = b[e];
            t.node[c][at[b[e]]++] = a[e];
        }
        t.mass[c].resize(n);
        t.size[c].assign(n, 1.0);
        for (int i = 0; i < n; i++) t.mass[c][i] = 1.0 + deg[i];
        t.pos[c].resize(2 * n);
        const double r = 10.0 * std::sqrt((double) n);
        for (int i = 0; i < 2 * n; i++)
            t.pos[c][i] = r * (2.0 * (double) (splitmix(seed) >> 11) / 9007199254740992.0 - 1.0);
        fa2_full_params &p = t.ps[c];
        memset(&p, 0, sizeof(p));
        p.n = n;
        p.inc_off = off.data();
        p.inc_node = t.node[c].data();
        p.inc_coef = t.coef[c].data();
        p.mass = t.mass[c].data();
        p.size = t.size[c].data();
        p.scaling = 2.0;
        p.gravity = 1.0;
        p.theta = 1.2;
        p.jitter_tolerance = 1.0;
        p.device = device;
        p.use_double = use_double;
        t.pp[c] = t.pos[c].data();
    }
}

// Milliseconds per graph-iteration of a batch of these graphs (-1 on error).
template <class R>
static double time_batch(TuneGraphs &t, int exact_below, int threads, int npt = 2)
{
    BatchBase *B =
        make_batch<R>(t.ps.data(), (int) t.ps.size(), t.pp.data(), exact_below, threads, npt);
    if (!B) return -1.0;
    double ms = -1.0;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    if (!B->iterate(2)) { // warm-up; also captures the timed launch
        cudaEventRecord(e0, B->stream());
        if (!B->iterate(2)) {
            cudaEventRecord(e1, B->stream());
            if (!B->sync()) {
                float f = 0.f;
                cudaEventElapsedTime(&f, e0, e1);
                ms = f / (2.0 * (double) t.ps.size());
            }
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    delete B;
    return ms;
}

template <class R> int tune_batch(int device, int *exact_below, int *threads, int *npt)
{
    int sms = 0;
    FA2_TRY(cudaSetDevice(device), "could not use the CUDA device", 1);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const int copies = 2 * std::max(sms, 1);
    // 1: tree faster, 0: exact faster, -1: error
    auto tree_wins = [&](int n) {
        TuneGraphs t;
        tune_graphs(t, n, copies, device, sizeof(R) == 8);
        const double te = time_batch<R>(t, 1 << 30, 512);
        const double tb = time_batch<R>(t, 0, 512);
        if (te < 0 || tb < 0) return -1;
        return tb < te ? 1 : 0;
    };
    // the first power of two at which the tree wins, then quarter-octave
    // steps below it
    int hi = 0;
    for (int n = 64; n <= 16384; n *= 2) {
        const int w = tree_wins(n);
        if (w < 0) return 1;
        if (w) {
            hi = n;
            break;
        }
    }
    int cross = hi ? hi : 32768;
    if (hi > 64) {
        for (int q = 1; q < 4; q++) {
            const int n = (int) std::lround((hi / 2) * std::pow(2.0, q / 4.0));
            const int w = tree_wins(n);
            if (w < 0) return 1;
            if (w) {
                cross = n;
                break;
            }
        }
    }
    TuneGraphs t;
    tune_graphs(t, 2048, copies, device, sizeof(R) == 8);
    const double t256 = time_batch<R>(t, 0, 256), t512 = time_batch<R>(t, 0, 512);
    if (t256 < 0 || t512 < 0) return 1;
    const int th = t256 < t512 ? 256 : 512;
    TuneGraphs u;
    tune_graphs(u, std::min(std::max(cross * 3 / 4, th + 1), 4096), copies, device,
                sizeof(R) == 8);
    const double t1 = time_batch<R>(u, 1 << 30, th, 1), t2 = time_batch<R>(u, 1 << 30, th, 2);
    if (t1 < 0 || t2 < 0) return 1;
    *exact_below = cross;
    *threads = th;
    *npt = t1 < t2 ? 1 : 2;
    return 0;
}

} // namespace fa2cu
