// small_exact.cuh -- whole iterations of a small FP32 all-pairs layout in one
// launch. Included by kernels.cuh.
#pragma once

namespace fa2cu {

// One cluster of thread blocks runs `iterations` iterations. Every block holds
// all nodes' records and positions in shared memory and owns the nodes [b m,
// (b + 1) m): their repulsion (two nodes a thread, the sources split over the
// threads, the parts added in order), attraction, swinging and displacement.
// The blocks' totals and new positions go to all blocks through distributed
// shared memory; each block makes the speed update for itself.
//
// Why: three launches an iteration took 15 to 20 us for a few of arithmetic. An
// iteration in us, three launches and this with 1 / 4 / 16 blocks: 50 nodes
// 15.0 and 4.3 / 5.2 / 5.5; 150 14.9 and 5.5 (now 5.1) / 6.2 / 6.3; 300 15.9 and 9.7 /
// 7.6 / 7.3; 1,000 18.2 and - / 20.0 / 11.3; 1,500 19.8 and - / 39.2 / 16.6;
// 2,000 21.1 and - / 59.9 / 22.6. Bound by latency (the block's and cluster's
// barriers, two dependent FP64 divisions of the speed update), from 1,000 nodes
// by the pairs on 16 of the SMs.
constexpr int SE_THREADS = 512;
static_assert(CS_MAX_BLOCKS == 16, "half a warp holds the blocks' sums");
constexpr int SE_MAX = 1500; // nodes up to which it is the faster
constexpr int SE_PARTS = 16; // of the sources, at most
constexpr int SE_ITERATIONS = 256; // a launch, at most
constexpr size_t SE_SMEM = 200 * 1024; // dynamic, at most

inline __host__ __device__ size_t small_exact_smem(int n)
{
    return (size_t) n * (sizeof(ExactF32) + sizeof(float2));
}

__device__ __forceinline__ void cluster_put(uint32_t addr, float4 v)
{
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x),
                 "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}
__device__ __forceinline__ void cluster_put(uint32_t addr, float2 v)
{
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y)
                 : "memory");
}

template <bool ADJUST>
__global__ void __launch_bounds__(SE_THREADS)
k_small_exact(int n, int m, int iterations, float scaling, float gravity, int strong, int linlog,
              const float *__restrict__ mass, const float *__restrict__ size,
              const uint8_t *__restrict__ fixed, const int *__restrict__ off,
              const Inc<float> *__restrict__ inc, float2 *__restrict__ pos,
              float2 *__restrict__ fold, float *__restrict__ sw, float *__restrict__ tr,
              ExactF32 *__restrict__ nodes, SpeedState *__restrict__ st,
              int *__restrict__ status)
{
    constexpr int T = SE_THREADS;
    extern __shared__ __align__(32) unsigned char se_shared[];
    ExactF32 *const rec = reinterpret_cast<ExactF32 *>(se_shared); // n
    float2 *const at = reinterpret_cast<float2 *>(rec + n);        // n positions
    __shared__ float2 part[2 * T]; // a part's sums of the block's nodes
    __shared__ float2 force[T];
    __shared__ float4 warp_sum4[T / 32], block_sum4[CS_MAX_BLOCKS];
    __shared__ SpeedState speed;
    __shared__ int stop;
    __shared__ double traction;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned rank = blockIdx.x, blocks = gridDim.x; // one cluster
    const int base = (int) rank * m, cnt = max(0, min(m, n - base));
    const int half = (cnt + 1) / 2;
    const int parts = half > 0 ? min(SE_PARTS, T / half) : 1;
    const int seg = (n + parts - 1) / parts;
    pdl_wait();
    for (int i = threadIdx.x; i < n; i += T) {
        const float2 p = pos[i];
        at[i] = p;
        exact_fill(rec + i, p, mass[i], ADJUST ? size[i] : 0.0f);
    }
    if (threadIdx.x == 0) {
        speed = *st;
        stop = status[ST_ERROR] != 0;
    }
    const bool own = (int) threadIdx.x < cnt;
    const int k = base + (int) threadIdx.x; // the thread's own node
    const bool held = own && fixed && fixed[k];
    const float mk = own ? mass[k] : 0.0f;
    float2 old = own ? fold[k] : make_float2(0.0f, 0.0f);
    // the thread's two nodes and part of the sources
    const int slot = half > 0 ? (int) threadIdx.x % half : 0;
    const int q = half > 0 ? (int) threadIdx.x / half : parts;
    const int la = slot, lb = min(slot + half, max(cnt - 1, 0));
    const int j0 = min(n, q * seg), j1 = q < parts ? min(n, j0 + seg) : j0;
    __syncthreads();
    cluster_barrier(); // every block has started, and read the speed and status
    float2 f = make_float2(0.0f, 0.0f);
    for (int it = 0; it < iterations; it++) {
        // repulsion: the thread's part (the terms of k_exact)
        if (j0 < j1) {
            const ExactF32 a = rec[base + la], b = rec[base + lb];
            GroupNode me;
            me.x = f2_make(-a.nx[0], -b.nx[0]);
            me.y = f2_make(-a.ny[0], -b.ny[0]);
            f2 ax = 0, ay = 0;
            unsigned s = smem_addr(rec + j0);
#pragma unroll 4
            for (int j = j0; j < j1; j++, s += (unsigned) sizeof(ExactF32)) {
                f2 nx, ny, mm, r = 0;
                lds_2<0>(s, nx, ny);
                if (ADJUST)
                    lds_2<16>(s, mm, r);
                else
                    mm = lds_1<16>(s);
                exact_term<ADJUST>(me, a.r[0], b.r[0], nx, ny, mm, r, ax, ay);
            }
            float xa, xb, ya, yb;
            f2_split(ax, xa, xb);
            f2_split(ay, ya, yb);
            const float ma = scaling * a.m[0], mb = scaling * b.m[0];
            part[q * cnt + la] = make_float2(xa * ma, ya * ma);
            if (slot + half < cnt) part[q * cnt + lb] = make_float2(xb * mb, yb * mb);
        }
        __syncthreads();
        // the parts, attraction and gravity, swinging and traction
        SwingAcc<float> acc;
        if (own) {
            f = part[threadIdx.x];
            for (int r = 1; r < parts && r * seg < n; r++) {
                const float2 v = part[r * cnt + threadIdx.x];
                f.x += v.x;
                f.y += v.y;
            }
            force[threadIdx.x] = f;
            attract_one<float, true>(k, gravity, strong, linlog, ADJUST, at, mass, size, off, inc,
                                     force - base);
            f = force[threadIdx.x];
            swing_node_v<float>(k, f, old, mk, fixed, sw, tr, acc);
        }
        // totals: a warp's, the block's, all blocks'
        for (int o = 16; o > 0; o >>= 1) {
            acc.s = ff_add(acc.s, ff_shfl_down(acc.s, o));
            acc.t = ff_add(acc.t, ff_shfl_down(acc.t, o));
        }
        if (lane == 0) warp_sum4[w] = make_float4(acc.s.hi, acc.s.lo, acc.t.hi, acc.t.lo);
        __syncthreads();
        if (w == 0) {
            const float4 v =
                lane < T / 32 ? warp_sum4[lane] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            ff2 a = ff2{v.x, v.y}, b = ff2{v.z, v.w};
            for (int o = T / 64; o > 0; o >>= 1) {
                a = ff_add(a, ff_shfl_down(a, o));
                b = ff_add(b, ff_shfl_down(b, o));
            }
            const float4 sum = make_float4(__shfl_sync(0xffffffffu, a.hi, 0),
                                           __shfl_sync(0xffffffffu, a.lo, 0),
                                           __shfl_sync(0xffffffffu, b.hi, 0),
                                           __shfl_sync(0xffffffffu, b.lo, 0));
            if (lane < (int) blocks)
                cluster_put(cluster_addr(smem_addr(&block_sum4[rank]), lane), sum);
        }
        if (blocks > 1) cluster_barrier();
        else __syncthreads();
        // the blocks' sums (hi, lo), a lane each, rounded once: the swinging's by
        // the first warp, the traction's by the second
        double a = 0.0;
        if (w < 2 && blocks > 1) {
            const float4 v = (lane & 15) < (int) blocks ? block_sum4[lane & 15]
                                                        : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            a = warp_sum_once((double) (lane < 16 ? w ? v.z : v.x : w ? v.w : v.y));
            if (w == 1 && lane == 0) traction = a;
            asm volatile("bar.sync 1, 64;" ::: "memory");
        }
        if (w == 0) {
            double b = traction;
            if (blocks == 1) {
                const float4 v = block_sum4[0];
                a = (double) v.x + (double) v.y;
                b = (double) v.z + (double) v.w;
            }
            if (lane == 0) {
                if (!(a == a) || !(b == b)) {
                    speed.total_swinging = a;
                    speed.total_traction = b;
                    stop = 1;
                    if (rank == 0) atomicOr(status + ST_ERROR, ERR_NAN);
                } else {
                    update_speed(&speed, a, b);
                }
            }
        }
        __syncthreads();
        if (stop) break; // (the same in every block)
        // displacement, to every block
        if (own) {
            old = f;
            force[threadIdx.x] =
                held ? at[k] : moved<float>(at[k], f, sw[k], (float) speed.speed, ADJUST);
        }
        __syncthreads();
        for (int e = threadIdx.x; e < cnt * (int) blocks; e += T) {
            const int b = e / cnt, i = e - b * cnt;
            const float2 p = force[i];
            cluster_put(cluster_addr(smem_addr(rec + base + i), b),
                        make_float4(-p.x, -p.x, -p.y, -p.y));
            cluster_put(cluster_addr(smem_addr(at + base + i), b), p);
        }
        if (blocks > 1) cluster_barrier();
        else __syncthreads();
    }
    if (own) {
        fold[k] = old;
        pos[k] = at[k];
        exact_move(nodes + k, at[k]);
    }
    if (rank == 0 && threadIdx.x == 0) *st = speed;
}

} // namespace fa2cu
