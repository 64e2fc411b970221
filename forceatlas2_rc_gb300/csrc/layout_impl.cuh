// layout_impl.cuh -- the device sessions, templated on the real type.
// Included by inst_f32.cu and inst_f64.cu only, so that every kernel they
// launch is compiled with the flags of its precision.
//
// HBM layout of a Layout<R> (n nodes, E incidences; float sizes):
//   pos, f, fold        R2[n]   positions, forces, previous forces
//   mass, size, sw      R[n]    masses, radii (adjust), swinging
//   fixed               u8[n]   (when some node is fixed)
//   inc_off, inc        int[n+1], {int j; R coef}[E]  symmetric CSR
//   key, order (+ ping-pong)  u32[n] x 4, look-back words u32[4 * 256 * n / 2048]
//   psort               R4[n]   (x, y, m, r) in Morton order
//   child, range        int2[n-1], parent int[2n-1], rope int[n],
//   meet                int[n-1], agg Agg<R>[n-1] (double / float-float sums),
//                       rec_c R4[n-1], rec_t int2[n-1] (traversal records),
//                       bounds float4[n-1] (FP64: of the opening tests)
//   piece, pieces       what climbs in the tree's second launch (tree.cuh)
//   bbox, quant         the bounding box and Morton quantisation, computed by
//                       the displacement of the previous iteration
//   packed, exact_part  ExactRec[n], R2[rows n]  (exact repulsion only)
//   st, status          FP64 speed state, status words
#pragma once

#include <stdio.h>
#include <string.h>
#include <time.h>
#include <vector>

#include "devmem.cuh"
#include "kernels.cuh"
#include "prep.cuh"
#include "session.h"
#include "sort_tree.cuh"

namespace fa2cu {

inline double now_s()
{
    struct timespec ts;
    clock_gettime(CLOCK_MONOTONIC, &ts);
    return (double) ts.tv_sec + 1e-9 * (double) ts.tv_nsec;
}

// SMs of the current device (at least 1).
inline int device_sms()
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::max(sms, 1);
}

// FP32 nodes a thread of the all-pairs kernel: six share a source's loads;
// with few nodes two, for more threads and fewer rows to add up (an iteration
// in us with two / six: 4,500 nodes 22.1 / 24.4, 6,007 26.2 / 27.7, 9,000 42.1 /
// 38.7).
inline int exact_ipt(int n) { return n < 7000 ? 2 : 6; }

// The all-pairs repulsion of n records. FP32: `rows` rows of partial sums
// (n entries each; exact_rows) into `partial`, for exact_sum to add up -- or,
// one row, straight into f. FP64: into f.
template <class R>
void launch_exact(cudaStream_t s, bool pdl, int n, bool adjust, R scaling,
                  const typename ExactRec<R>::type *packed, typename RT<R>::R2 *f,
                  typename RT<R>::R2 *partial, int rows, int *status)
{
    if constexpr (sizeof(R) == 8) {
        const int per = exact_ordered_rows(n, device_sms()), grid = ceil_div(n, per);
        if (adjust)
            k_exact_ordered<true><<<grid, EXACT_ORDERED_THREADS, 0, s>>>(n, per, scaling, packed, f);
        else
            k_exact_ordered<false><<<grid, EXACT_ORDERED_THREADS, 0, s>>>(n, per, scaling, packed,
                                                                          f);
    } else {
        const int seg = ceil_div(n, rows), ipt = exact_ipt(n);
        auto go = [&](auto kernel) {
            launch_k(pdl, kernel, dim3(ceil_div(n, EXACT_THREADS * ipt), rows),
                     dim3(EXACT_THREADS), 0, s, n, scaling, packed, rows > 1 ? partial : f, seg,
                     status);
        };
        if (adjust)
            ipt == 2 ? go(k_exact<true, 2>) : go(k_exact<true, 6>);
        else
            ipt == 2 ? go(k_exact<false, 2>) : go(k_exact<false, 6>);
    }
}

template <class R> struct Layout : LayoutBase {
    typedef typename RT<R>::R2 R2;
    typedef typename RT<R>::R4 R4;

    int n = 0, ninc = 0, repulsion = 0, adjust = 0, strong = 0, linlog = 0;
    int any_fixed = 0;
    // FP32: the group walk (group_walk.cuh); FP64: one walk per thread, in
    // the reference's order of the forces
    int walk = sizeof(R) == 4 ? WALK_DEFERRED : WALK_THREAD;
    // Warps that share the group walk of 32 nodes, from the warps the device
    // holds at once (36 an SM, 5472 in all): a layout too small to fill it is
    // bound by the serial chain of one warp's rounds, which more warps
    // shorten; a full device by the instructions, of which each part repeats
    // the first rounds. The repulsion in us with 1 / 2 / 4 warps: 3,001 nodes
    // 31.7 / 25.2 / 22.9; 10,007 35.6 / 27.2 / 24.6; 30,011 (radii) 40.8 /
    // 32.4 / 30.3; 50,007 45.5 / 37.7 / 44.9; 100,000 57.4 / 63.7 / 79.7;
    // 300,007 118 / 158 / 236.
    int walk_split = 1;
    static int pick_split(int n)
    {
        const double x = n / 32.0 / 5472.0; // of the device, with one warp each
        return x < 0.22 ? 4 : x < 0.45 ? 2 : 1;
    }
    bool block_sort = false; // few keys: the one-block sort
    // blocks of the cluster that makes the codes and sorts them in one
    // launch (0: codes and tiled sort), and its kernel's shape
    int cluster = 0, cluster_shape = 0;
    size_t cluster_smem() const { return 2 * sizeof(uint2) * (size_t) ceil_div(n, cluster); }
    // Calls go(kernel, threads) for the shape that holds m pairs a block.
    template <class F> static void with_cluster_kernel(int shape, F go)
    {
        switch (shape) {
        case 0: return go(k_codes_sort<R, 256, 8>, 256);
        case 1: return go(k_codes_sort<R, 512, 8>, 512);
        default: return go(k_codes_sort<R, 512, 16>, 512);
        }
    }
    static constexpr int cluster_pairs[3] = {2048, 4096, 8192};
    // The shape for a cluster of c blocks: the first that holds the nodes.
    bool pick_cluster(int c)
    {
        for (int shape = 0; shape < 3; shape++)
            if (cluster_fits(n, c, shape)) {
                cluster_shape = shape;
                return true;
            }
        return false;
    }
    // Whether a cluster of c blocks of that shape runs on the current device
    // with n nodes.
    static bool cluster_fits(int n, int c, int shape)
    {
        if (c < 1 || c > CS_MAX_BLOCKS || ceil_div(n, c) > cluster_pairs[shape]) return false;
        bool fit = false;
        with_cluster_kernel(shape, [&](auto kernel, int threads) {
            fit = cluster_runs(kernel, c, threads, 2 * sizeof(uint2) * (size_t) ceil_div(n, c),
                               2 * sizeof(uint2) * (size_t) cluster_pairs[shape]);
        });
        return fit;
    }
    // Whether a cluster of c blocks of the kernel runs on the current device
    // with smem bytes of dynamic shared memory a block (at most `most`, which
    // the kernel is allowed).
    template <class K> static bool cluster_runs(K kernel, int c, int threads, size_t smem, size_t most)
    {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned) c);
        cfg.blockDim = dim3((unsigned) threads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned) c;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int fit = 0;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int) most) != cudaSuccess ||
            cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
                cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return fit > 0;
    }

    // The tree's blocks search their edges in a window of 2 W leaves: a wide
    // one shortens the climbs, which bound a small layout; a narrow one fills
    // the blocks, of which a large one has many waves. An iteration in us with
    // W 64 / 32: 10,007 nodes 69.8 / 71.6, 30,011 89.6 / 91.1, 100,000 156.4 /
    // 153.4. The climbs in a launch of their own (32 and 16 then): 300,007 262
    // in one / 264 apart, 10^6 666 / 641.
    int tree_window = 64;
    bool tree_apart = false;
    void pick_tree()
    {
        tree_apart = n >= 400000;
        tree_window = n < 60000 ? 64 : n < 400000 ? 32 : 16;
    }
    // FP32 all-pairs: blocks of the cluster that runs whole iterations
    // (k_small_exact; 0: three launches an iteration)
    int small_blocks = 0;
    // Threads a block of the kernels with a thread a node that end in totals:
    // small blocks spread a small layout over the SMs and have fewer warps to
    // add up. An iteration in us with 256 / 128 / 64: all pairs FP32 1,600
    // nodes 19.5 / 17.4 / 16.4, 6,007 30.4 / 28.5 / 27.7; Barnes-Hut FP32 3,001
    // 57.9 / 56.1 / 55.3, 10,007 66.5 / 64.5 / 64.7, 30,011 84.4 / 82.8 / 85.7;
    // FP64 3,001 155 / 146 / 143, 30,011 305 / 301 / 304.
    int node_threads() const { return n < 20000 ? 64 : n < 200000 ? 128 : 256; }
    bool pick_small(int c)
    {
        if constexpr (sizeof(R) == 4) {
            if (repulsion != FA2CU_REPULSION_EXACT || nheavy > 0 || c < 1 || c > CS_MAX_BLOCKS ||
                ceil_div(n, c) > SE_THREADS || small_exact_smem(n) > SE_SMEM)
                return false;
            auto runs = [&](auto kernel) {
                return cluster_runs(kernel, c, SE_THREADS, small_exact_smem(n), SE_SMEM);
            };
            if (adjust ? runs(k_small_exact<true>) : runs(k_small_exact<false>)) {
                small_blocks = c;
                return true;
            }
        }
        return false;
    }
    R scaling = 0, gravity = 0, theta2 = 0;
    R wscale = 0; // (1 + DECIDE_BAND) / theta^2 (region_far, term_bounds)
    double theta2d = 0.0;
    cudaStream_t s = nullptr;
    DevMem mem;
    R2 *pos = nullptr, *f = nullptr, *fold = nullptr;
    R *mass = nullptr, *size = nullptr, *sw = nullptr, *trac = nullptr;
    uint8_t *fixed = nullptr;
    int *inc_off = nullptr;
    Inc<R> *inc = nullptr;
    // FP32: the nodes of HEAVY_DEGREE incidences or more (heavy_cap of room,
    // then their count), summed by a warp each
    int *heavy = nullptr;
    int heavy_cap = 0, nheavy = 0;
    int launches = 0; // kernels of one captured iteration
    R *bbox = nullptr, *bbox_partial = nullptr;
    double *quant = nullptr; // min x, min y, Morton scale, -, 4 floats (k_bbox)
    int nbbox = 1;
    uint32_t *key = nullptr, *order = nullptr;
    SortScratch ss{};
    R4 *psort = nullptr;
    typename ExactRec<R>::type *packed = nullptr; // exact repulsion: the nodes' records
    R2 *exact_part = nullptr; // exact_rows rows of partial sums (FP32, rows > 1)
    int exact_nrows = 1;
    int2 *child = nullptr, *range = nullptr;
    int *parent = nullptr, *rope = nullptr, *meet = nullptr;
    int2 *piece = nullptr; // what climbs in the tree's second launch (tree.cuh)
    int *pieces = nullptr;
    Agg<R> *agg = nullptr;
    R4 *rec_c = nullptr; // traversal records (common.cuh)
    int2 *rec_t = nullptr;
    float4 *bounds = nullptr; // FP64: bounds of the opening tests (term_bounds)
    double2 *swing_partial = nullptr;
    SpeedState *st = nullptr;
    int *status = nullptr;
    double *xy = nullptr; // 2n doubles of staging
    unsigned long long *counts = nullptr;
    cudaGraphExec_t g1 = nullptr, g8 = nullptr;
    // Iterations to launch kernel by kernel before the graphs are captured: a
    // run of fewer than FEW is shorter with its launches than with a capture of
    // nine iterations (a call of 20 iterations of 3,001 nodes: 2,000 -> 1,769
    // us).
    static constexpr int FEW = 64;
    int direct = 0;
    cudaEvent_t ev[8] = {};
    // FP32 Barnes-Hut: the attraction on a second stream beside the tree
    // build and the walk, into its own buffer fatt, on attract_grid blocks
    // per SM (beside())
    int overlap = sizeof(R) == 4 ? 1 : 0, attract_grid = 1;
    // grid of the join: 4 blocks per SM, grid-stride (0.709-0.712 -> 0.703
    // ms an iteration at 10^6 SBM nodes against one block per 256 nodes,
    // whose last block added 3907 partials)
    int join_blocks = 152 * 4;
    // the iteration's kernels on the main stream launched as programmatic
    // dependents (launch_k; option "pdl"), below 500,000 nodes: ms an
    // iteration without / with, SBM 10^4 0.1435 / 0.1411, BA 10^5 0.2018 /
    // 0.1988, SBM 10^6 0.6799 / 0.6855 (positions identical)
    bool pdl = false;
    cudaStream_t s2 = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    R2 *fatt = nullptr;

    ~Layout() override
    {
        if (s) cudaStreamSynchronize(s);
        if (g1) cudaGraphExecDestroy(g1);
        if (g8) cudaGraphExecDestroy(g8);
        for (auto &e : ev)
            if (e) cudaEventDestroy(e);
        mem.release();
        if (ev_fork) cudaEventDestroy(ev_fork);
        if (ev_join) cudaEventDestroy(ev_join);
        if (s2) cudaStreamDestroy(s2);
        if (s) cudaStreamDestroy(s);
    }

    double bytes() const override { return mem.bytes; }
    cudaStream_t stream() override { return s; }

    int alloc(bool want_tree)
    {
        mem.planned([&] { take_buffers(want_tree); });
        if (mem.failed) {
            set_cuda_error("could not allocate memory on the device", mem.err);
            return 1;
        }
        return 0;
    }
    void take_buffers(bool want_tree)
    {
        const size_t nn = (size_t) n;
        pos = mem.get<R2>(nn);
        f = mem.get<R2>(nn);
        fold = mem.get<R2>(nn);
        mass = mem.get<R>(nn);
        size = adjust ? mem.get<R>(nn) : nullptr;
        sw = mem.get<R>(nn);
        trac = serial_totals<R>(n) ? mem.get<R>(nn) : nullptr;
        fixed = any_fixed ? mem.get<uint8_t>(nn) : nullptr;
        inc_off = mem.get<int>(nn + 1);
        inc = mem.get<Inc<R>>((size_t) ninc);
        if (sizeof(R) == 4) {
            heavy_cap = ninc / HEAVY_DEGREE;
            heavy = mem.get<int>((size_t) heavy_cap + 1);
        }
        swing_partial = mem.get<double2>((size_t) ceil_div(n, node_threads())); // one per block
        st = mem.get<SpeedState>(1);
        status = mem.get<int>(ST_COUNT);
        xy = mem.get<double>(2 * nn);
        counts = mem.get<unsigned long long>(2);
        if (want_tree) {
            nbbox = std::min(ceil_div(n, node_threads()), 152 * 4);
            bbox = mem.get<R>(4);
            quant = mem.get<double>(6);
            bbox_partial = mem.get<R>(4 * (size_t) nbbox);
            key = mem.get<uint32_t>(nn);
            order = mem.get<uint32_t>(nn);
            ss.key_b = mem.get<uint32_t>(nn);
            ss.val_b = mem.get<uint32_t>(nn);
            ss.counts = mem.get<uint32_t>(sort_scratch_counts(n));
            ss.err = status + ST_ERROR;
            ss.digit_total = mem.get<uint32_t>(SORT_AUX);
            psort = mem.get<R4>(nn);
            child = mem.get<int2>(nn - 1);
            range = mem.get<int2>(nn - 1);
            parent = mem.get<int>(2 * nn - 1);
            rope = mem.get<int>(nn);
            meet = mem.get<int>(nn - 1);
            const size_t tree_blocks = (size_t) ceil_div(n, TREE_THREADS - 2 * 64);
            piece = mem.get<int2>(tree_blocks * TREE_PIECES);
            pieces = mem.get<int>(tree_blocks);
            agg = mem.get<Agg<R>>(nn - 1);
            rec_c = mem.get<R4>(nn - 1);
            rec_t = mem.get<int2>(nn - 1);
            if (sizeof(R) == 4) fatt = mem.get<R2>(nn);
            if (sizeof(R) == 8) bounds = mem.get<float4>(nn - 1);
        } else {
            packed = mem.get<typename ExactRec<R>::type>(nn);
            if (exact_nrows > 1) exact_part = mem.get<R2>((size_t) exact_nrows * nn);
        }
    }

    // The graph from its edge list, prepared on the device (prep.cu): the
    // masses, the incidence lists and their coefficients in double, then
    // converted to the layout's precision.
    int prepare_edges(const fa2_full_params *p, const EdgeList &E)
    {
        DevMem tmp;
        tmp.pool = mem.pool;
        tmp.s = s;
        const size_t m1 = (size_t) std::max(E.m, 1);
        int *from = nullptr, *to = nullptr, *dnode = nullptr;
        double *w = nullptr, *dmass = nullptr, *dcoef = nullptr;
        PrepScratch ws;
        tmp.planned([&] {
            from = tmp.get<int>(m1);
            to = tmp.get<int>(m1);
            w = tmp.get<double>(m1);
            dmass = tmp.get<double>((size_t) n);
            dnode = tmp.get<int>(2 * m1);
            dcoef = tmp.get<double>(std::max(2 * m1, (size_t) n));
            prep_scratch(tmp, n, E.m, ws);
        });
        if (tmp.failed) {
            tmp.release();
            set_cuda_error("could not allocate memory on the device", tmp.err);
            return 1;
        }
        int rc = 0;
        auto up = [&](void *dst, const void *src, size_t b) {
            if (!rc && b) rc = cudaMemcpyAsync(dst, src, b, cudaMemcpyHostToDevice, s) != cudaSuccess;
        };
        up(from, E.from, (size_t) E.m * sizeof(int));
        up(to, E.to, (size_t) E.m * sizeof(int));
        up(w, E.w, (size_t) E.m * sizeof(double));
        if (rc) {
            tmp.release();
            set_cuda_error("could not send the graph to the device", cudaGetLastError());
            return 1;
        }
        const long long got =
            prep_graph(s, n, E.m, from, to, w, E.outbound, dmass, inc_off, dnode, dcoef, ws);
        if (got < 0) {
            cudaStreamSynchronize(s);
            tmp.release();
            return 1;
        }
        ninc = (int) got;
        k_real_in<R><<<ceil_div(n, 256), 256, 0, s>>>(n, dmass, mass);
        if (ninc > 0) k_inc_in<R><<<ceil_div(ninc, 256), 256, 0, s>>>(ninc, dnode, dcoef, inc);
        if (adjust) {
            up(dcoef, p->size, (size_t) n * sizeof(double));
            if (!rc) k_real_in<R><<<ceil_div(n, 256), 256, 0, s>>>(n, dcoef, size);
        }
        if (any_fixed) {
            std::vector<uint8_t> f8((size_t) n);
            for (int i = 0; i < n; i++) f8[i] = p->fixed[i] != 0;
            up(fixed, f8.data(), (size_t) n);
        }
        if (!rc) rc = cudaStreamSynchronize(s) != cudaSuccess;
        tmp.release();
        if (rc) {
            set_cuda_error("could not send the graph to the device", cudaGetLastError());
            return 1;
        }
        return 0;
    }

    int open(const fa2_full_params *p, const double *xy0, int rep,
             const LayoutOpts *opts = nullptr, const EdgeList *edges = nullptr)
    {
        n = p->n;
        // from an edge list: at most two incidences per edge until the
        // preparation on the device has counted them
        ninc = edges ? 2 * edges->m : p->inc_off[n];
        repulsion = rep;
        adjust = p->adjust ? 1 : 0;
        strong = p->strong ? 1 : 0;
        linlog = p->linlog ? 1 : 0;
        any_fixed = 0;
        if (p->fixed)
            for (int i = 0; i < n && !any_fixed; i++) any_fixed = p->fixed[i] != 0;
        scaling = (R) p->scaling;
        gravity = (R) p->gravity;
        theta2d = p->theta * p->theta;
        theta2 = (R) theta2d;
        wscale = (R) ((1.0 + (double) DECIDE_BAND) / theta2d);
        if (opts && opts->has_priority)
            FA2_TRY(cudaStreamCreateWithPriority(&s, cudaStreamNonBlocking, opts->priority),
                    "could not create a CUDA stream", 1);
        else
            FA2_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking),
                    "could not create a CUDA stream", 1);
        for (auto &e : ev) FA2_TRY(cudaEventCreate(&e), "could not create a CUDA event", 1);
        if (sizeof(R) == 4 && rep == FA2CU_REPULSION_BH) {
            FA2_TRY(cudaStreamCreateWithFlags(&s2, cudaStreamNonBlocking),
                    "could not create a CUDA stream", 1);
            FA2_TRY(cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming),
                    "could not create a CUDA event", 1);
            FA2_TRY(cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming),
                    "could not create a CUDA event", 1);
        }

        mem.pool = opts ? opts->pool : nullptr;
        mem.s = s;
        if (rep == FA2CU_REPULSION_BH && sort_setup()) return 1;
        if (rep == FA2CU_REPULSION_BH) {
            pick_tree();
            if (n > CS_MAX) attract_grid = 2;
            walk_split = pick_split(n);
            // sort tiles: fewer than ~75 tiles of 8192 keys leave most SMs
            // idle; measured on a GB300 (sort of one iteration, ms, tiles of
            // 256 / 512 / 1024 threads): 1e5 keys 0.050 / 0.051 / 0.060;
            // 3e5 0.054 / 0.054 / 0.066; 1e6 0.092 / 0.077 / 0.070; 3e6
            // 0.178 / 0.164 / 0.163
            ss.tile_threads = n < 600000 ? 512 : 1024;
            pdl = n < 500000;
            ss.pdl = pdl;
            block_sort = n <= SORT_BLOCK_MAX;
            // (an iteration in us with 1 / 4 / 16 blocks: 100 nodes 40.5 / 42.2 /
            // 44.3; 1,000 67.8 / 61.7 / 63.9; 3,001 - / 78.2 / 76.7)
            const int c = n <= 256 ? 1 : n <= 2000 ? 4 : CS_MAX_BLOCKS;
            if (n <= CS_MAX && pick_cluster(c)) cluster = c;
        }
        if (rep == FA2CU_REPULSION_EXACT) {
            int sms = 0;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
            exact_nrows = exact_layout_rows(n, sms);
            pdl = n < 500000;
        }
        if (alloc(rep == FA2CU_REPULSION_BH)) return 1;

        // the graph, once (reference src/gpu_full.c:241-287), or prepared on
        // the device from its edge list
        if (edges) {
            if (prepare_edges(p, *edges)) return 1;
        } else {
            DevMem tmp;
            tmp.pool = mem.pool;
            tmp.s = s;
            double *dd = nullptr;
            int *di = nullptr;
            tmp.planned([&] {
                dd = tmp.get<double>(std::max<size_t>((size_t) n, (size_t) ninc));
                di = tmp.get<int>((size_t) ninc);
            });
            if (tmp.failed) {
                tmp.release();
                set_cuda_error("could not allocate memory on the device", tmp.err);
                return 1;
            }
            int rc = 0;
            auto up = [&](void *dst, const void *src, size_t b) {
                if (!rc && b) rc = cudaMemcpyAsync(dst, src, b, cudaMemcpyHostToDevice, s) != cudaSuccess;
            };
            up(dd, p->mass, (size_t) n * sizeof(double));
            if (!rc) k_real_in<R><<<ceil_div(n, 256), 256, 0, s>>>(n, dd, mass);
            if (adjust) {
                up(dd, p->size, (size_t) n * sizeof(double));
                if (!rc) k_real_in<R><<<ceil_div(n, 256), 256, 0, s>>>(n, dd, size);
            }
            up(inc_off, p->inc_off, ((size_t) n + 1) * sizeof(int));
            if (ninc > 0) {
                up(dd, p->inc_coef, (size_t) ninc * sizeof(double));
                up(di, p->inc_node, (size_t) ninc * sizeof(int));
                if (!rc) k_inc_in<R><<<ceil_div(ninc, 256), 256, 0, s>>>(ninc, di, dd, inc);
            }
            if (any_fixed) {
                std::vector<uint8_t> f8((size_t) n);
                for (int i = 0; i < n; i++) f8[i] = p->fixed[i] != 0;
                up(fixed, f8.data(), (size_t) n);
                if (!rc) rc = cudaStreamSynchronize(s) != cudaSuccess;
            }
            if (!rc) rc = cudaStreamSynchronize(s) != cudaSuccess;
            tmp.release();
            if (rc) {
                set_cuda_error("could not send the graph to the device", cudaGetLastError());
                return 1;
            }
        }
        // the heavy nodes (FP32), listed once
        if (heavy) {
            FA2_TRY(cudaMemsetAsync(heavy + heavy_cap, 0, sizeof(int), s), "cudaMemset", 1);
            if (heavy_cap > 0)
                k_heavy_list<<<ceil_div(n, 256), 256, 0, s>>>(n, inc_off, heavy, heavy_cap);
            FA2_TRY(cudaMemcpyAsync(&nheavy, heavy + heavy_cap, sizeof(int),
                                    cudaMemcpyDeviceToHost, s),
                    "could not prepare the layout", 1);
            FA2_TRY(cudaStreamSynchronize(s), "could not prepare the layout", 1);
            nheavy = std::min(nheavy, heavy_cap);
        }
        // status words (error flags, arrival tickets) and the previous
        // forces start at zero; then the positions (and their bounding box,
        // whose reduction takes a ticket)
        FA2_TRY(cudaMemsetAsync(fold, 0, (size_t) n * sizeof(R2), s), "cudaMemset", 1);
        FA2_TRY(cudaMemsetAsync(status, 0, ST_COUNT * sizeof(int), s), "cudaMemset", 1);
        if (repulsion == FA2CU_REPULSION_BH) {
            sort_prepare(s, ss);
            // nobody has met at any split (each tree leaves them so)
            FA2_TRY(cudaMemsetAsync(meet, 0xff, ((size_t) n - 1) * sizeof(int), s), "cudaMemset",
                    1);
        }
        if (set_positions(xy0)) return 1;
        SpeedState h{};
        h.speed = 1.0;
        h.efficiency = 1.0;
        h.jitter_tolerance = p->jitter_tolerance;
        h.terms = speed_terms(n);
        FA2_TRY(cudaMemcpyAsync(st, &h, sizeof(h), cudaMemcpyHostToDevice, s), "cudaMemcpy", 1);
        FA2_TRY(cudaStreamSynchronize(s), "could not prepare the layout", 1);
        if (n <= SE_MAX) pick_small(n <= 200 ? 1 : CS_MAX_BLOCKS);
        if (p->iterations > 0 && p->iterations < FEW) direct = p->iterations;
        return direct ? 0 : make_graphs();
    }

    static int exact_layout_rows(int n, int sms)
    {
        if (sizeof(R) == 8) return 1;
        const int rows = exact_rows(n, std::max(sms, 1), exact_ipt(n));
        return ceil_div(n, ceil_div(n, rows)); // (no empty row)
    }

    // ---- the steps of one iteration ----
    // The bounding box and Morton quantisation of the current positions (the
    // displacement computes them for the positions it writes; this is for
    // positions set from outside).
    void launch_bbox()
    {
        k_bbox<R><<<nbbox, 256, 0, s>>>(n, pos, bbox_partial, bbox, quant,
                                        (unsigned *) (status + ST_TICKET_BBOX));
    }
    // Morton codes, with the sort's digit histograms in the same launch
    void launch_build()
    {
        if (cluster) return; // with the sort
        const int nb = std::min(ceil_div(n, 256), 152 * 4);
        if (block_sort) { // the one-block sort counts its own digits
            k_morton<R><<<nb, 256, 0, s>>>(n, pos, quant, key, order, nullptr, nullptr, 0);
            return;
        }
        // the histograms, done counter and tickets start at zero: cleared at
        // open, then left at zero by the Morton kernel's last block for the
        // next sort (no memset in the iteration)
        launch_k(pdl, k_morton<R>, dim3(nb), dim3(256), 0, s, n, pos, quant, key, order,
                 ss.digit_total, ss.counts, sort_status_words(n, 4));
    }
    void launch_sort()
    {
        if (cluster)
            with_cluster_kernel(cluster_shape, [&](auto kernel, int threads) {
                launch_cluster(cluster, pdl, kernel, dim3(cluster), dim3(threads), cluster_smem(),
                               s, n, ceil_div(n, cluster), pos, quant, key, order, status);
            });
        else if (block_sort)
            sort_pairs_block(s, n, key, order, ss);
        else
            sort_pairs(s, n, key, order, ss, /*hist_ready=*/true);
    }
    void launch_tree()
    {
        // ranges and parents are made where something reads them
        const bool full = walk == WALK_WARP;
        full ? launch_tree_kernel<true>() : launch_tree_kernel<false>();
    }
    template <bool FULL> void launch_tree_kernel()
    {
        const TreeArrays<R> A{psort, rec_c, child, range, rec_t, parent, rope, meet, agg, bounds,
                              piece, pieces};
        const int blocks = ceil_div(n, TREE_THREADS - 2 * tree_window);
        auto go = [&](auto kernel) {
            launch_k(pdl, kernel, dim3(blocks), dim3(TREE_THREADS), 0, s, n, tree_window, adjust,
                     order, pos, mass, size, key, A, wscale, status);
        };
        if (tree_apart) {
            go(k_tree<R, FULL, true>);
            launch_k(pdl, k_tree_top<R, FULL>, dim3(ceil_div(blocks, TREE_THREADS / 32)),
                     dim3(TREE_THREADS), 0, s, n, blocks, key, A, wscale, status);
        } else {
            go(k_tree<R, FULL, false>);
        }
    }
    // (graphs with hubs: their walks add up with compensation)
    void launch_group_walk()
    {
        auto go = [&](auto kernel) {
            launch_k(pdl, kernel, dim3(ceil_div(n, 32 * GW_WARPS / walk_split)),
                     dim3(32 * GW_WARPS), 0, s, n, walk_split, scaling, theta2d, psort, rec_c, rec_t, child, agg, order, f, status);
        };
        if (adjust)
            nheavy > 0 ? go(k_traverse_group<true, true>) : go(k_traverse_group<true, false>);
        else
            nheavy > 0 ? go(k_traverse_group<false, true>) : go(k_traverse_group<false, false>);
    }
    void launch_repulsion()
    {
        if (repulsion == FA2CU_REPULSION_BH) {
            if (walk == WALK_WARP) {
                if (adjust)
                    k_traverse_warp<R, true><<<ceil_div(n, 256), 256, 0, s>>>(
                        n, scaling, theta2, theta2d, psort, rec_c, rec_t, range, agg, rope, order, f,
                        status);
                else
                    k_traverse_warp<R, false><<<ceil_div(n, 256), 256, 0, s>>>(
                        n, scaling, theta2, theta2d, psort, rec_c, rec_t, range, agg, rope, order, f,
                        status);
            } else if (walk == WALK_THREAD) {
                if constexpr (sizeof(R) == 8) {
                    auto go = [&](auto kernel, int nodes) {
                        launch_k(pdl, kernel, dim3(ceil_div(n, nodes * TW_WARPS)),
                                 dim3(32 * TW_WARPS), 0, s, n, scaling, theta2, psort, rec_c,
                                 bounds, rec_t, rope, order, f, status);
                    };
                    // (four nodes a warp while that does not fill the device)
                    if (n < 12000)
                        adjust ? go(k_traverse_terms<true, 4>, 4) : go(k_traverse_terms<false, 4>, 4);
                    else
                        adjust ? go(k_traverse_terms<true, 16>, 16)
                               : go(k_traverse_terms<false, 16>, 16);
                } else if (adjust) {
                    k_traverse<R, true, 6><<<ceil_div(n, 256), 256, 0, s>>>(
                        n, scaling, theta2, theta2d, psort, rec_c, rec_t, agg, rope, order, f, status);
                } else { // 8 blocks per SM (0.597 against 0.619 ms at 6, 10^6 nodes)
                    k_traverse<R, false, 8><<<ceil_div(n, 256), 256, 0, s>>>(
                        n, scaling, theta2, theta2d, psort, rec_c, rec_t, agg, rope, order, f, status);
                }
            } else if (walk == WALK_DEFERRED) {
                if constexpr (sizeof(R) == 4) {
                    launch_group_walk();
                } else {
                    const int g = ceil_div(n, 256);
                    if (adjust)
                        k_traverse_deferred<R, true, 6><<<g, 256, 0, s>>>(
                            n, scaling, theta2, theta2d, psort, rec_c, rec_t, agg, rope, order,
                            f, status);
                    else
                        k_traverse_deferred<R, false, 6><<<g, 256, 0, s>>>(
                            n, scaling, theta2, theta2d, psort, rec_c, rec_t, agg, rope, order,
                            f, status);
                }
            } else if (walk == WALK_PAIR) {
                const int grid = ceil_div(ceil_div(n, 2), 256);
                if (adjust)
                    k_traverse_multi<R, true, 2><<<grid, 256, 0, s>>>(
                        n, scaling, theta2, theta2d, psort, rec_c, rec_t, agg, rope, order, f, status);
                else
                    k_traverse_multi<R, false, 2><<<grid, 256, 0, s>>>(
                        n, scaling, theta2, theta2d, psort, rec_c, rec_t, agg, rope, order, f, status);
            } else if (walk == WALK_QUAD) {
                const int grid = ceil_div(ceil_div(n, 4), 256);
                if (adjust)
                    k_traverse_multi<R, true, 4><<<grid, 256, 0, s>>>(
                        n, scaling, theta2, theta2d, psort, rec_c, rec_t, agg, rope, order, f, status);
                else
                    k_traverse_multi<R, false, 4><<<grid, 256, 0, s>>>(
                        n, scaling, theta2, theta2d, psort, rec_c, rec_t, agg, rope, order, f, status);
            } else {
                if (adjust)
                    k_traverse<R, true, 1><<<ceil_div(n, 256), 256, 0, s>>>(
                        n, scaling, theta2, theta2d, psort, rec_c, rec_t, agg, rope, order, f, status);
                else
                    k_traverse<R, false, 1><<<ceil_div(n, 256), 256, 0, s>>>(
                        n, scaling, theta2, theta2d, psort, rec_c, rec_t, agg, rope, order, f, status);
            }
        } else {
            launch_exact<R>(s, pdl, n, adjust, scaling, packed, f, exact_part, exact_nrows,
                            status);
        }
    }
    // The all-pairs repulsion into f, where it is still in rows.
    void launch_exact_sum()
    {
        if (repulsion == FA2CU_REPULSION_EXACT && exact_nrows > 1)
            k_exact_sum<R><<<ceil_div(n, 256), 256, 0, s>>>(n, exact_nrows, exact_part, f);
    }
    // The heavy nodes' attraction (FP32), added to their repulsion.
    void launch_heavy()
    {
        if (nheavy > 0)
            k_attract_heavy<R><<<ceil_div(nheavy, 8), 256, 0, s>>>(nheavy, heavy, linlog, adjust,
                                                                  pos, size, inc_off, inc, f);
    }
    // Attraction and gravity only (the forces of fa2cu_layout_forces).
    void launch_attraction()
    {
        launch_exact_sum();
        launch_heavy();
        k_attract<R><<<ceil_div(n, 256), 256, 0, s>>>(n, gravity, strong, linlog, adjust, pos,
                                                      mass, size, inc_off, inc, f);
    }
    // Attraction and gravity, swinging, traction, the totals and the speed
    // update (an iteration's second half before the displacement).
    void launch_attraction_swing()
    {
        // FP64: the warps' terms; serial totals: the last block stages 2n reals
        size_t smem = serial_totals<R>(n) ? 2 * (size_t) n * sizeof(R) : 0;
        if (sizeof(R) == 8)
            smem = std::max(smem, node_threads() / 32 * sizeof(AttractShared));
        // the rows of the all-pairs sum are added up in the same launch,
        // unless a hub's attraction is added to them first
        const bool in_rows =
            repulsion == FA2CU_REPULSION_EXACT && exact_nrows > 1 && nheavy == 0;
        if (!in_rows) launch_exact_sum();
        launch_heavy();
        launch_k(pdl && nheavy == 0, k_attract_swing<R>, dim3(ceil_div(n, node_threads())),
                 dim3(node_threads()), smem, s, n, gravity, strong, linlog, adjust, in_rows ? exact_nrows : 0, exact_part,
                 pos, mass, size, inc_off, inc, f, fold, fixed, sw, trac, swing_partial,
                 (unsigned *) (status + ST_TICKET_SWING), st, status);
    }
    // The displacement, with the next iteration's bounding box.
    void launch_move()
    {
        // with a tree, the bounding box's block count (its partials); else
        // one thread per node
        const int nb = bbox_partial ? nbbox : ceil_div(n, node_threads());
        launch_k(pdl, k_apply<R>, dim3(nb), dim3(node_threads()), 0, s, n, adjust, f, fold, sw,
                 fixed, pos, st, status, bbox_partial, bbox, quant, (unsigned *) (status + ST_TICKET_BBOX),
                 packed);
    }
    void launch_repel()
    {
        if (repulsion == FA2CU_REPULSION_BH) {
            launch_build();
            launch_sort();
            launch_tree();
        }
        launch_repulsion();
    }
    void launch_forces()
    {
        launch_repel();
        if (beside()) { // the iteration's order: repulsion + (gravity + attraction)
            launch_attraction_own(s, true);
            k_add_forces<R><<<ceil_div(n, 256), 256, 0, s>>>(n, fatt, f);
        } else {
            launch_attraction();
        }
    }
    // FP32 Barnes-Hut: gravity and attraction into fatt, on stream s2
    // beside the tree build and the walk, added to the repulsion by the
    // join (overlap 1: forked after the sort, or before the tiled sort's last
    // pass; 2: after the tree; 0: the attraction fused with the totals after
    // the walk). An iteration in us with 0 / 1 at 1 / 2 / 4 blocks an SM:
    // 100,000 SBM nodes 162.5 / 157.6 / 158.9 / 160.7; 300,007 275.2 / 270.5 /
    // 264.3 / 263.0; 10^6 670.7 / 642.9 / 649.6 / 655.0; 2,000,003 1233 / 1369 /
    // 1206 / 1204. Forked at the iteration's start it delays the sort's tiles
    // (10^6: 706 to 754); after the whole sort, the tree's blocks hold the SMs
    // first (703).
    bool beside() const { return overlap && s2 && fatt && !serial_totals<R>(n); }
    // alone: nothing runs beside it (the force query, the phase times), one
    // thread per node; else attract_grid blocks per SM
    void launch_attraction_own(cudaStream_t st, bool alone)
    {
        if constexpr (sizeof(R) == 4) {
            int sms = 0;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
            if (nheavy > 0)
                k_attract_heavy<R, true><<<ceil_div(nheavy, 8), 256, 0, st>>>(
                    nheavy, heavy, linlog, adjust, pos, size, inc_off, inc, fatt);
            const int grid =
                alone ? ceil_div(n, 256)
                      : std::max(1, std::min(std::max(sms, 1) * attract_grid, ceil_div(n, 256)));
            k_attract_own<R><<<grid, 256, 0, st>>>(n, gravity, strong, linlog, adjust, pos, mass,
                                                   size, inc_off, inc, fatt);
        }
    }
    void launch_join_swing()
    {
        const int nb = std::min(ceil_div(n, node_threads()), join_blocks);
        k_join_swing<R><<<nb, node_threads(), 0, s>>>(
            n, fatt, f, fold, mass, fixed, sw, trac, swing_partial,
            (unsigned *) (status + ST_TICKET_SWING), st, status);
    }
    void launch_iteration()
    {
        if (beside()) {
            launch_build();
            // (with the tiled sort, before its last pass: the attraction's
            // blocks are on the SMs before the tree's fill them)
            const bool early = overlap == 1 && !cluster && !block_sort;
            if (early) ss.before_last = ev_fork;
            launch_sort();
            ss.before_last = nullptr;
            if (overlap == 2) launch_tree();
            if (!early) cudaEventRecord(ev_fork, s);
            cudaStreamWaitEvent(s2, ev_fork, 0);
            launch_attraction_own(s2, false);
            cudaEventRecord(ev_join, s2);
            if (overlap != 2) launch_tree();
            launch_repulsion();
            cudaStreamWaitEvent(s, ev_join, 0);
            launch_join_swing();
            launch_move();
            return;
        }
        launch_repel();
        launch_attraction_swing();
        launch_move();
    }

    int capture(cudaGraphExec_t *out, int iters)
    {
        cudaGraph_t g = nullptr;
        FA2_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal),
                "could not capture the iteration", 1);
        for (int k = 0; k < iters; k++) launch_iteration();
        cudaError_t e = cudaStreamEndCapture(s, &g);
        if (e != cudaSuccess) {
            set_cuda_error("could not capture the iteration", e);
            return 1;
        }
        if (iters == 1) { // the kernels of one iteration
            size_t nodes = 0;
            if (cudaGraphGetNodes(g, nullptr, &nodes) == cudaSuccess) {
                std::vector<cudaGraphNode_t> v(nodes);
                launches = 0;
                if (nodes && cudaGraphGetNodes(g, v.data(), &nodes) == cudaSuccess)
                    for (cudaGraphNode_t x : v) {
                        cudaGraphNodeType t;
                        if (cudaGraphNodeGetType(x, &t) == cudaSuccess &&
                            t == cudaGraphNodeTypeKernel)
                            launches++;
                    }
            }
        }
        e = cudaGraphInstantiate(out, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            set_cuda_error("could not instantiate the iteration graph", e);
            return 1;
        }
        return 0;
    }

    int iterate(int iterations) override
    {
        cudaSetDevice(device);
        if constexpr (sizeof(R) == 4) {
            if (small_blocks) return iterate_small(iterations);
        }
        for (; iterations > 0 && direct > 0; iterations--, direct--) launch_iteration();
        if (iterations <= 0) {
            FA2_TRY(cudaGetLastError(), "the computation on the GPU failed", 1);
            return 0;
        }
        if (!g1 && make_graphs()) return 1;
        while (iterations >= 8 && g8) {
            FA2_TRY(cudaGraphLaunch(g8, s), "the computation on the GPU failed", 1);
            iterations -= 8;
        }
        for (; iterations > 0; iterations--)
            FA2_TRY(cudaGraphLaunch(g1, s), "the computation on the GPU failed", 1);
        return 0;
    }

    // (a launch's iterations are bounded: other work may wait for the SMs)
    int iterate_small(int iterations)
    {
        for (; iterations > 0; iterations -= SE_ITERATIONS) {
            auto go = [&](auto kernel) {
                return launch_cluster(small_blocks, pdl, kernel, dim3(small_blocks),
                                      dim3(SE_THREADS), small_exact_smem(n), s, n,
                                      ceil_div(n, small_blocks),
                                      std::min(iterations, SE_ITERATIONS), scaling, gravity,
                                      strong, linlog, mass, size, fixed, inc_off, inc, pos, fold,
                                      sw, trac, packed, st, status);
            };
            FA2_TRY(adjust ? go(k_small_exact<true>) : go(k_small_exact<false>),
                    "the computation on the GPU failed", 1);
        }
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
        if (h & ERR_WAIT) {
            set_message("the computation on the GPU failed (a device wait timed out)");
            return 1;
        }
        if (h & ERR_BOUNDS) {
            set_message("the computation on the GPU failed (an index left its bounds)");
            return 1;
        }
        return 0;
    }

    int positions(double *out) override
    {
        cudaSetDevice(device);
        k_pos_out<R><<<ceil_div(n, 256), 256, 0, s>>>(n, pos, xy);
        FA2_TRY(cudaMemcpyAsync(out, xy, 2 * (size_t) n * sizeof(double),
                                cudaMemcpyDeviceToHost, s),
                "could not fetch the layout from the device", 1);
        FA2_TRY(cudaStreamSynchronize(s), "could not fetch the layout from the device", 1);
        return 0;
    }

    int set_positions(const double *in) override
    {
        cudaSetDevice(device);
        FA2_TRY(cudaMemcpyAsync(xy, in, 2 * (size_t) n * sizeof(double),
                                cudaMemcpyHostToDevice, s),
                "could not send the positions to the device", 1);
        k_pos_in<R><<<ceil_div(n, 256), 256, 0, s>>>(n, xy, pos);
        if (bbox_partial) launch_bbox();
        if (packed) // (the displacement keeps them up to date)
            k_pack<R><<<ceil_div(n, 256), 256, 0, s>>>(n, adjust, pos, mass, size, packed);
        FA2_TRY(cudaStreamSynchronize(s), "could not send the positions to the device", 1);
        return 0;
    }

    int forces(const double *in, double *out) override
    {
        if (set_positions(in)) return 1;
        launch_forces();
        k_forces_out<R><<<ceil_div(n, 256), 256, 0, s>>>(n, f, nullptr, xy, xy + n);
        FA2_TRY(cudaMemcpyAsync(out, xy, 2 * (size_t) n * sizeof(double),
                                cudaMemcpyDeviceToHost, s),
                "could not fetch the forces", 1);
        return sync();
    }

    int speed(double state[4]) override
    {
        cudaSetDevice(device);
        SpeedState h;
        FA2_TRY(cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, s), "cudaMemcpy", 1);
        FA2_TRY(cudaStreamSynchronize(s), "cudaMemcpy", 1);
        state[0] = h.speed;
        state[1] = h.efficiency;
        state[2] = h.total_swinging;
        state[3] = h.total_traction;
        return 0;
    }

    int phase_times(int iterations, double *ms) override
    {
        cudaSetDevice(device);
        for (int it = 0; it < iterations; it++) {
            int e = 0;
            cudaEventRecord(ev[e++], s);
            if (repulsion == FA2CU_REPULSION_BH) {
                launch_build();
                cudaEventRecord(ev[e++], s);
                launch_sort();
                cudaEventRecord(ev[e++], s);
                launch_tree();
                cudaEventRecord(ev[e++], s);
            } else {
                cudaEventRecord(ev[e++], s);
                cudaEventRecord(ev[e++], s);
                cudaEventRecord(ev[e++], s);
            }
            launch_repulsion();
            cudaEventRecord(ev[e++], s);
            if (beside()) { // "attraction": here after the walk, one thread per node, and the join
                launch_attraction_own(s, true);
                launch_join_swing();
            } else {
                launch_attraction_swing(); // with the totals and speed
            }
            cudaEventRecord(ev[e++], s);
            launch_move();
            cudaEventRecord(ev[e++], s);
            FA2_TRY(cudaEventSynchronize(ev[e - 1]), "the computation on the GPU failed", 1);
            double total = 0.0;
            for (int k = 1; k < e; k++) {
                float t = 0.f;
                cudaEventElapsedTime(&t, ev[k - 1], ev[k]);
                ms[k] += t;
                total += t;
            }
            ms[FA2_FULL_T_TOTAL] += total;
        }
        return sync();
    }

    int tree(const double *in, uint32_t *hkey, uint32_t *horder, int *hchild, int *hrange,
             int *hparent, double *hni) override
    {
        if (repulsion != FA2CU_REPULSION_BH) {
            set_message("this layout has no tree (exact repulsion)");
            return 1;
        }
        if (set_positions(in)) return 1;
        launch_build();
        launch_sort();
        launch_tree_kernel<true>();
        std::vector<R4> hc((size_t) n - 1);
        std::vector<Agg<R>> ha(sizeof(R) == 4 ? (size_t) n - 1 : 0);
        const size_t nn = (size_t) n;
        cudaMemcpyAsync(hkey, key, nn * 4, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(horder, order, nn * 4, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(hchild, child, (nn - 1) * sizeof(int2), cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(hrange, range, (nn - 1) * sizeof(int2), cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(hparent, parent, (2 * nn - 1) * sizeof(int), cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(hc.data(), rec_c, (nn - 1) * sizeof(R4), cudaMemcpyDeviceToHost, s);
        if (sizeof(R) == 4)
            cudaMemcpyAsync(ha.data(), agg, (nn - 1) * sizeof(Agg<R>), cudaMemcpyDeviceToHost, s);
        FA2_TRY(cudaStreamSynchronize(s), "could not fetch the tree", 1);
        for (size_t r = 0; r + 1 < nn; r++) {
            hni[4 * r] = (double) hc[r].x;
            hni[4 * r + 1] = (double) hc[r].y;
            hni[4 * r + 2] = (double) hc[r].z;
            if (sizeof(R) == 4) { // the FP32 record holds a scaled size^2 (region_far)
                const float w = (float) (ha[r].maxx - ha[r].minx);
                const float h = (float) (ha[r].maxy - ha[r].miny);
                hni[4 * r + 3] = (double) (2.0f * (w * w + h * h));
            } else {
                hni[4 * r + 3] = (double) hc[r].w;
            }
        }
        return 0;
    }

    // The iteration graphs again, after an option changed the launches.
    int recapture()
    {
        cudaSetDevice(device);
        FA2_TRY(cudaStreamSynchronize(s), "the computation on the GPU failed", 1);
        if (g1) cudaGraphExecDestroy(g1);
        if (g8) cudaGraphExecDestroy(g8);
        g1 = g8 = nullptr;
        return make_graphs();
    }
    int make_graphs()
    {
        if (small_blocks) { // (nothing to capture)
            launches = 1;
            return 0;
        }
        direct = 0;
        if (capture(&g1, 1)) return 1;
        if (n <= (1 << 16) && capture(&g8, 8)) return 1;
        return 0;
    }

    int option(const char *name, double value) override
    {
        if (!strcmp(name, "walk_split") && (value == 1 || value == 2 || value == 4)) {
            walk_split = (int) value;
            return recapture();
        }
        if (!strcmp(name, "sort_cluster") && value >= 0 && value <= CS_MAX_BLOCKS &&
            value == (int) value) {
            const int c = (int) value;
            if (c && !pick_cluster(c)) {
                set_message("a cluster of %d blocks does not hold %d nodes", c, n);
                return 1;
            }
            cluster = c;
            return recapture();
        }
        if (!strcmp(name, "exact_cluster") && value >= 0 && value <= CS_MAX_BLOCKS &&
            value == (int) value) {
            if (value != 0 && !pick_small((int) value)) {
                set_message("a cluster of %d blocks does not run this layout", (int) value);
                return 1;
            }
            small_blocks = (int) value;
            return recapture();
        }
        if (!strcmp(name, "sort_threads") && (value == 256 || value == 512 || value == 1024)) {
            ss.tile_threads = (int) value;
            cluster = 0;
            return recapture();
        }
        if (!strcmp(name, "overlap") && (value == 0 || value == 1 || value == 2)) {
            if (value != 0 && !s2) {
                set_message("the attraction runs beside the walk in FP32 Barnes-Hut layouts only");
                return 1;
            }
            overlap = (int) value;
            return recapture();
        }
        if (!strcmp(name, "pdl") && (value == 0 || value == 1)) {
            pdl = value == 1;
            ss.pdl = pdl;
            return recapture();
        }
        if (!strcmp(name, "join_blocks") && value >= 1 && value <= 1 << 20) {
            join_blocks = (int) value;
            return recapture();
        }
        if (!strcmp(name, "attract_grid") && value >= 1 && value <= 8) {
            attract_grid = (int) value;
            return recapture();
        }
        if (!strcmp(name, "sort_block") && (value == 0 || value == 1)) {
            if (value == 1 && n > SORT_BLOCK_MAX) {
                set_message("the one-block sort handles at most %d keys", SORT_BLOCK_MAX);
                return 1;
            }
            block_sort = value == 1;
            cluster = 0;
            return recapture();
        }
        if (!strcmp(name, "climb") &&
            (value == 1 || value == 2 || value == 4 || value == 8 || value == -2 ||
             value == -4)) {
            tree_apart = value != 1;
            return recapture();
        }
        if (!strcmp(name, "walk") &&
            (value == WALK_WARP || value == WALK_THREAD || value == WALK_THREAD_WIDE ||
             value == WALK_PAIR || value == WALK_QUAD || value == WALK_DEFERRED)) {
            walk = (int) value;
            return recapture();
        }
        if (!strcmp(name, "keep_traction") && value == 1) {
            // per-node traction kept for fa2cu_layout_swing (the FP64 path
            // keeps it anyway up to SERIAL_TOTALS_MAX nodes)
            if (!trac) {
                cudaSetDevice(device);
                FA2_TRY(cudaStreamSynchronize(s), "the computation on the GPU failed", 1);
                trac = mem.get<R>((size_t) n);
                if (!trac) {
                    set_cuda_error("could not allocate memory on the device", mem.err);
                    return 1;
                }
            }
            return recapture();
        }
        set_message("unknown option %s = %g", name, value);
        return 1;
    }

    double info(const char *name) override
    {
        if (!strcmp(name, "launches_per_iteration")) {
            if (!launches && make_graphs()) return -1.0; // (counted there)
            return launches;
        }
        if (!strcmp(name, "heavy_nodes")) return nheavy;
        if (!strcmp(name, "nodes")) return n;
        if (!strcmp(name, "incidences")) return ninc;
        set_message("unknown layout information %s", name);
        return -1.0;
    }

    int swing(double *hsw, double *htr) override
    {
        if (htr && !trac) {
            set_message("the per-node traction is not kept (option keep_traction)");
            return 1;
        }
        cudaSetDevice(device);
        std::vector<R> a((size_t) n), b(htr ? (size_t) n : 0);
        FA2_TRY(cudaMemcpyAsync(a.data(), sw, (size_t) n * sizeof(R), cudaMemcpyDeviceToHost, s),
                "could not fetch the swinging", 1);
        if (htr)
            FA2_TRY(cudaMemcpyAsync(b.data(), trac, (size_t) n * sizeof(R),
                                    cudaMemcpyDeviceToHost, s),
                    "could not fetch the traction", 1);
        FA2_TRY(cudaStreamSynchronize(s), "could not fetch the swinging", 1);
        for (int i = 0; i < n; i++) {
            if (hsw) hsw[i] = (double) a[i];
            if (htr) htr[i] = (double) b[i];
        }
        return 0;
    }

    int traversal_counts(double out[2]) override
    {
        if (repulsion != FA2CU_REPULSION_BH) {
            set_message("this layout has no tree (exact repulsion)");
            return 1;
        }
        cudaSetDevice(device);
        launch_build();
        launch_sort();
        launch_tree();
        cudaMemsetAsync(counts, 0, 2 * sizeof(unsigned long long), s);
        k_traverse_count<R><<<ceil_div(n, 256), 256, 0, s>>>(n, theta2, theta2d, psort, rec_c,
                                                             rec_t, agg, rope, counts);
        unsigned long long h[2] = {0, 0};
        cudaMemcpyAsync(h, counts, sizeof(h), cudaMemcpyDeviceToHost, s);
        FA2_TRY(cudaStreamSynchronize(s), "the computation on the GPU failed", 1);
        out[0] = (double) h[0];
        out[1] = (double) h[1];
        return 0;
    }
};

template <class R>
LayoutBase *make_layout(const fa2_full_params *p, const double *pos, int rep,
                        const LayoutOpts *opts, const EdgeList *edges)
{
    int dev = p->device;
    FA2_TRY(cudaSetDevice(dev), "could not use the CUDA device", nullptr);
    Layout<R> *L = new Layout<R>();
    L->device = dev;
    if (L->open(p, pos, rep, opts, edges)) {
        delete L;
        return nullptr;
    }
    return L;
}

// Device bytes a layout holds (its buffers, counted by the allocation plan
// itself) plus the transient staging of the graph upload at open.
template <class R>
double layout_footprint(int n, int ninc, int adjust, int any_fixed, int rep, int sms)
{
    Layout<R> L;
    L.n = n;
    L.ninc = ninc;
    L.adjust = adjust ? 1 : 0;
    L.any_fixed = any_fixed ? 1 : 0;
    if (rep == FA2CU_REPULSION_EXACT)
        L.exact_nrows = Layout<R>::exact_layout_rows(n, sms);
    L.mem.dry = true;
    L.alloc(rep == FA2CU_REPULSION_BH);
    const double staging = (double) std::max(n, ninc) * sizeof(double) + (double) ninc * sizeof(int);
    return L.mem.bytes + staging;
}

// ---- the repulsion backend of fa2_gpu_open (reference src/gpu.c:357-704) --

template <class R> struct Repulse : RepulseBase {
    typedef typename RT<R>::R2 R2;
    typedef typename RT<R>::R4 R4;
    int n = 0, adjust = 0, barnes_hut = 0;
    cudaStream_t s = nullptr;
    DevMem mem;
    double *in4 = nullptr;   // x, y, mass, size staging (4n)
    double *out2 = nullptr;  // fx, fy (2n)
    double *host2 = nullptr; // pinned copy of out2
    R4 *p = nullptr;                         // Barnes-Hut records, tree order
    typename ExactRec<R>::type *e = nullptr; // all-pairs records
    R2 *f = nullptr;
    R2 *part = nullptr; // partial sums of the split all-pairs kernel
    int nrows = 1;
    int *status = nullptr;
    fa2_region *raw = nullptr;
    QRegion<R> *regs = nullptr;
    int *perm = nullptr;

    ~Repulse() override
    {
        if (s) cudaStreamSynchronize(s);
        mem.release();
        if (host2) cudaFreeHost(host2);
        if (s) cudaStreamDestroy(s);
    }

    int open(int n_, int adjust_, int bh)
    {
        n = n_;
        adjust = adjust_ ? 1 : 0;
        barnes_hut = bh ? 1 : 0;
        const size_t nn = (size_t) n;
        FA2_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking),
                "could not create a CUDA stream", 1);
        in4 = mem.get<double>(4 * nn);
        out2 = mem.get<double>(2 * nn);
        f = mem.get<R2>(nn);
        status = mem.get<int>(ST_COUNT);
        if (!barnes_hut) get_exact();
        if (barnes_hut) {
            p = mem.get<R4>(nn);
            raw = mem.get<fa2_region>(2 * nn);
            regs = mem.get<QRegion<R>>(2 * nn);
            perm = mem.get<int>(nn);
        }
        if (mem.failed) {
            set_cuda_error("could not allocate memory on the device", mem.err);
            return 1;
        }
        FA2_TRY(cudaMallocHost(&host2, 2 * nn * sizeof(double)), "out of memory", 1);
        FA2_TRY(cudaMemsetAsync(status, 0, ST_COUNT * sizeof(int), s), "cudaMemset", 1);
        FA2_TRY(cudaStreamSynchronize(s), "could not prepare the device", 1);
        return 0;
    }

    // The buffers of the all-pairs repulsion (in a Barnes-Hut session, on its
    // first use).
    void get_exact()
    {
        if (e) return;
        e = mem.get<typename ExactRec<R>::type>((size_t) n);
        nrows = Layout<R>::exact_layout_rows(n, device_sms());
        if (nrows > 1) part = mem.get<R2>((size_t) nrows * n);
    }

    int send4(const double *x, const double *y, const double *m, const double *sz, bool all_pairs)
    {
        const size_t b = (size_t) n * sizeof(double);
        FA2_TRY(cudaMemcpyAsync(in4, x, b, cudaMemcpyHostToDevice, s), "the computation on the GPU failed", 1);
        FA2_TRY(cudaMemcpyAsync(in4 + n, y, b, cudaMemcpyHostToDevice, s), "the computation on the GPU failed", 1);
        FA2_TRY(cudaMemcpyAsync(in4 + 2 * (size_t) n, m, b, cudaMemcpyHostToDevice, s), "the computation on the GPU failed", 1);
        const bool with_size = adjust && sz;
        if (with_size)
            FA2_TRY(cudaMemcpyAsync(in4 + 3 * (size_t) n, sz, b, cudaMemcpyHostToDevice, s),
                    "the computation on the GPU failed", 1);
        const double *dsz = with_size ? in4 + 3 * (size_t) n : nullptr;
        if (all_pairs)
            k_pack_exact<R><<<ceil_div(n, 256), 256, 0, s>>>(n, in4, in4 + n,
                                                             in4 + 2 * (size_t) n, dsz, e);
        else
            k_pack_host<R><<<ceil_div(n, 256), 256, 0, s>>>(n, in4, in4 + n,
                                                            in4 + 2 * (size_t) n, dsz, p);
        return 0;
    }

    int fetch_add(const int *dperm, double *dx, double *dy)
    {
        double t0 = now_s();
        k_forces_out<R><<<ceil_div(n, 256), 256, 0, s>>>(n, f, dperm, out2, out2 + n);
        FA2_TRY(cudaMemcpyAsync(host2, out2, 2 * (size_t) n * sizeof(double),
                                cudaMemcpyDeviceToHost, s),
                "the computation on the GPU failed", 1);
        FA2_TRY(cudaStreamSynchronize(s), "the computation on the GPU failed", 1);
        for (int i = 0; i < n; i++) {
            dx[i] += host2[i];
            dy[i] += host2[n + i];
        }
        t_fetch += now_s() - t0;
        return 0;
    }

    int check_status()
    {
        int h = 0;
        FA2_TRY(cudaMemcpy(&h, status + ST_ERROR, sizeof(int), cudaMemcpyDeviceToHost),
                "the computation on the GPU failed", 1);
        if (h) {
            set_message(h & ERR_WAIT ? "the computation on the GPU failed (a device wait timed out)"
                                     : "the computation on the GPU failed (an index left its bounds)");
            return 1;
        }
        return 0;
    }

    int exact(const double *x, const double *y, const double *m, const double *sz,
              double sc, double *dx, double *dy) override
    {
        cudaSetDevice(device);
        get_exact();
        if (mem.failed) {
            set_cuda_error("could not allocate memory on the device", mem.err);
            return 1;
        }
        double t0 = now_s();
        if (send4(x, y, m, sz, true)) return 1;
        FA2_TRY(cudaStreamSynchronize(s), "the computation on the GPU failed", 1);
        double t1 = now_s();
        t_send += t1 - t0;
        launch_exact<R>(s, false, n, adjust, (R) sc, e, f, part, nrows, status);
        if (nrows > 1) k_exact_sum<R><<<ceil_div(n, 256), 256, 0, s>>>(n, nrows, part, f);
        FA2_TRY(cudaGetLastError(), "the computation on the GPU failed", 1);
        FA2_TRY(cudaStreamSynchronize(s), "the computation on the GPU failed", 1);
        if (check_status()) return 1;
        t_compute += now_s() - t1;
        return fetch_add(nullptr, dx, dy);
    }

    int bh(const fa2_tree *t, double sc, double theta, double *dx, double *dy) override
    {
        cudaSetDevice(device);
        if (check_quadtree(n, t)) return 1;
        double t0 = now_s();
        if (send4(t->px, t->py, t->pm, t->ps, false)) return 1;
        FA2_TRY(cudaMemcpyAsync(raw, t->reg, (size_t) t->nreg * sizeof(fa2_region),
                                cudaMemcpyHostToDevice, s),
                "the computation on the GPU failed", 1);
        FA2_TRY(cudaMemcpyAsync(perm, t->perm, (size_t) n * sizeof(int), cudaMemcpyHostToDevice, s),
                "the computation on the GPU failed", 1);
        k_qregions<R><<<ceil_div(t->nreg, 256), 256, 0, s>>>(t->nreg, raw, regs);
        FA2_TRY(cudaStreamSynchronize(s), "the computation on the GPU failed", 1);
        double t1 = now_s();
        t_send += t1 - t0;
        const double theta2d = theta * theta;
        const R theta2 = (R) theta2d;
        const double *px = in4, *py = in4 + n; // the host's doubles, tree order
        if (adjust)
            k_qtraverse<R, true><<<ceil_div(n, 256), 256, 0, s>>>(
                n, (R) sc, theta2, theta2d, p, px, py, regs, raw, t->nreg, f, status);
        else
            k_qtraverse<R, false><<<ceil_div(n, 256), 256, 0, s>>>(
                n, (R) sc, theta2, theta2d, p, px, py, regs, raw, t->nreg, f, status);
        FA2_TRY(cudaGetLastError(), "the computation on the GPU failed", 1);
        FA2_TRY(cudaStreamSynchronize(s), "the computation on the GPU failed", 1);
        if (check_status()) return 1;
        t_compute += now_s() - t1;
        return fetch_add(perm, dx, dy);
    }
};

template <class R> RepulseBase *make_repulse(int device, int n, int adjust, int bh)
{
    FA2_TRY(cudaSetDevice(device), "could not use the CUDA device", nullptr);
    Repulse<R> *g = new Repulse<R>();
    g->device = device;
    if (g->open(n, adjust, bh)) {
        delete g;
        return nullptr;
    }
    return g;
}

} // namespace fa2cu
