// tree.cuh -- the nodes in Morton order, the Karras (2012) radix tree over
// their codes and the regions' sums and walk records, in one launch
// (reference inst/opencl/pipeline.cl:195-323). Included by kernels.cuh.
//
// A block takes about 256 consecutive leaves.
//   In the block: a thread per split, round by round; a split's region is made
//   when its two children are, from their sums and ranges in shared memory,
//   until a round makes none -- no search, no counter, no fence.
//   Across blocks: the largest regions (and leaves) inside a block climb. A
//   region [l, r] is the left child of the split after r, or the right child
//   of the split after l - 1, whichever separates less; the two children of a
//   split meet by exchanging their outer ends at the split's slot, and the
//   second to come makes the region, whose range it then knows. No thread
//   waits.
// A region's number is Karras's: the end of its range on its parent's split's
// side, so that the children of split s are s and s + 1 (or leaves). Sums are
// made left child then right child whoever makes them: the tree, its sums and
// records are those of one climbing thread per leaf, bit for bit.
//
// Why: the binary searches over global memory (34 us at 10^6 nodes) and a
// climb whose every level counted its arrivals with a fence and loaded links
// and sums from L2 (83 us; 22 us of latency at 3,001 nodes). Bound: small
// layouts by the climbs' chain (a fence, an exchange and two loads a level of
// the tree's top), large ones by instruction issue. With the gather, phase
// times in us: 3,001 nodes 35 -> 23, 10,007 39 -> 24, 100,000 50 -> 36,
// 300,007 68 -> 58, 10^6 130 -> 119; an iteration 76 -> 66, 84 -> 70, 163 ->
// 153, 290 -> 262, 637 -> 641 (10^6: beside the attraction). Tried: ranges by
// binary search in shared memory and records written in the rounds (10^6:
// tree 164), 512 leaves a block (123), blocks cut at every 256th leaf (10,007:
// tree 42).
#pragma once

namespace fa2cu {

// Length of the common prefix of the codes of sorted leaves i and j, equal
// codes told apart by their places.
__device__ __forceinline__ int code_prefix(uint32_t ki, int i, uint32_t kj, int j)
{
    return ki == kj ? 32 + __clz((unsigned) (i ^ j)) : __clz(ki ^ kj);
}

// The region after the subtree whose last leaf is r: the right child of the
// split after r, a leaf if that is all of it (codes k0, k1, k2 of leaves r, r
// + 1, r + 2, as far as there are any); -1 at the end.
__device__ __forceinline__ int region_after(int r, int n, uint32_t k0, uint32_t k1, uint32_t k2)
{
    const int nl = n - 1;
    if (r >= n - 1) return -1;
    if (r + 2 >= n) return nl + r + 1;
    return code_prefix(k1, r + 1, k2, r + 2) < code_prefix(k0, r, k1, r + 1) ? nl + r + 1 : r + 1;
}

// The tree's arrays in global memory. range and parent only where asked for.
template <class R> struct TreeArrays {
    typename RT<R>::R4 *psort, *rec_c;
    int2 *child, *range, *rec_t;
    int *parent, *rope, *meet;
    Agg<R> *agg;
    float4 *bounds; // of the FP64 walk's opening tests (term_bounds)
    // the regions and leaves that climb (APART): TREE_PIECES places a block,
    // and how many
    int2 *piece;
    int *pieces;
};
// A block's leaves are at most two chains of subtrees, one a level of the tree
// (59 at most).
constexpr int TREE_PIECES = 128;

// The links and record of a finished region: number idx, leaves [l, r], split
// s, sums q, the region after it.
template <class R, bool FULL>
__device__ __forceinline__ void write_region(const TreeArrays<R> &A, int n, int idx, int l, int r,
                                             int s, const Agg<R> &q, int after, R wscale)
{
    const int nl = n - 1;
    const int left = l == s ? nl + s : s, right = r == s + 1 ? nl + s + 1 : s + 1;
    const typename RT<R>::R4 rec = agg_record(q, wscale);
    A.rec_c[idx] = rec;
    if constexpr (sizeof(R) == 8) A.bounds[idx] = term_bounds(rec, wscale);
    // a region of at most 8 nodes is never opened: its left link carries its
    // packed range instead (negative)
    A.rec_t[idx] = make_int2(r - l >= 8 ? left : bucket_pack(l, r), after);
    A.child[idx] = make_int2(left, right);
    if (FULL) {
        A.range[idx] = make_int2(l, r);
        A.parent[left] = idx;
        A.parent[right] = idx;
        if (l == 0 && r == n - 1) A.parent[0] = -1;
    }
}

__device__ __forceinline__ int meet_exchange(int *p, int v)
{
    int prior;
    asm volatile("atom.exch.acq_rel.gpu.b32 %0, [%1], %2;" : "=r"(prior) : "l"(p), "r"(v) : "memory");
    return prior;
}

// The climb of region (or leaf) [l, r], across blocks; `mine` its sums, or
// (LOAD) made in an earlier launch.
template <class R, bool FULL, bool LOAD>
__device__ __forceinline__ void climb_across(int l, int r, Agg<R> mine, int n,
                                             const uint32_t *key, const TreeArrays<R> &A,
                                             R wscale, int *status)
{
    // codes of leaves l - 1, l, r, r + 1
    uint32_t kb = l > 0 ? __ldg(key + l - 1) : 0u, kl = __ldg(key + l);
    uint32_t kr = __ldg(key + r), ka = r < n - 1 ? __ldg(key + r + 1) : 0u;
    // the region made last, whose links are written after the meeting at its
    // parent (whose fence then waits for its sums only)
    int idx = -1, made = 0;
    uint32_t ka2 = 0u;
    for (int depth = 0; depth <= 160; depth++) {
        const int before = l > 0 ? code_prefix(kb, l - 1, kl, l) : -1;
        const int after = r < n - 1 ? code_prefix(kr, r, ka, r + 1) : -1;
        const bool is_left = after > before, root = before < 0 && after < 0;
        const int s = is_left ? r : l - 1; // the parent's split
        if (LOAD && depth == 0)
            mine = l == r ? leaf_agg(A.psort[l]) : load_agg_cg(A.agg + (is_left ? r : l));
        if (made) {
            idx = is_left ? r : l;
            A.agg[idx] = mine;
        }
        const int other = root ? -1 : meet_exchange(A.meet + s, is_left ? l : r);
        if (made)
            write_region<R, FULL>(A, n, idx, l, r, made - 1, mine,
                                  region_after(r, n, kr, ka, ka2), wscale);
        if (other < 0) return; // the root, or the sibling will make the region
        A.meet[s] = -1;        // for the next tree
        if (is_left ? (other <= r || other >= n) : other >= l) {
            atomicOr(status + ST_ERROR, ERR_BOUNDS);
            return;
        }
        Agg<R> sib;
        if (is_left) {
            r = other;
            sib = r == s + 1 ? leaf_agg(ldcg_r4(A.psort + r)) : load_agg_cg(A.agg + s + 1);
            kr = __ldg(key + r);
            ka = r < n - 1 ? __ldg(key + r + 1) : 0u;
        } else {
            l = other;
            sib = l == s ? leaf_agg(ldcg_r4(A.psort + l)) : load_agg_cg(A.agg + s);
            kl = __ldg(key + l);
            kb = l > 0 ? __ldg(key + l - 1) : 0u;
        }
        ka2 = r + 2 < n ? __ldg(key + r + 2) : 0u;
        mine = is_left ? agg_combine(mine, sib) : agg_combine(sib, mine);
        made = s + 1;
    }
    atomicOr(status + ST_ERROR, ERR_BOUNDS);
}

constexpr int TREE_THREADS = 256; // and leaves of a block, at most

// A block's leaves begin and end at the split that separates most (the
// smallest common prefix) among 2 W around every S-th leaf, S = 256 - 2 W: the
// regions that contain a block's edge are then few, the top of the tree, and
// the climbs short. (A split between two random neighbours is at the bottom
// of the tree, and every region above it would be made across blocks.)
// The first leaf of block b; code holds the codes from leaf `from` on.
__device__ __forceinline__ int tree_edge(int b, int n, int W, const uint32_t *code, int from)
{
    const int S = TREE_THREADS - 2 * W;
    if (b == 0) return 0;
    if (b * (long long) S >= n) return n;
    unsigned best = 0xffffffffu; // prefix, place in the window
    for (int q = threadIdx.x & 31; q < 2 * W; q += 32) {
        const int p = b * S - W + q; // the split after leaf p
        if (p + 1 < n)
            best = min(best, (unsigned) code_prefix(code[p - from], p, code[p + 1 - from], p + 1)
                                     << 16 |
                                 (unsigned) q);
    }
    best = __reduce_min_sync(0xffffffffu, best);
    return b * S - W + (int) (best & 0xffffu) + 1;
}

// Blocks of 256 - 2 W leaves, more or less W at either end. APART: what climbs
// is listed for k_tree_top instead.
template <class R, bool FULL, bool APART>
__global__ void __launch_bounds__(TREE_THREADS)
k_tree(int n, int W, int adjust, const uint32_t *__restrict__ order,
       const typename RT<R>::R2 *__restrict__ pos, const R *__restrict__ mass,
       const R *__restrict__ size, const uint32_t *__restrict__ key, TreeArrays<R> A, R wscale,
       int *__restrict__ status)
{
    typedef typename RT<R>::R4 R4;
    constexpr int M = TREE_THREADS;
    __shared__ Agg<R> sums[M];         // of the block's regions, by number
    __shared__ R4 leaf[M];
    __shared__ uint32_t code[M + 4];   // of the leaves the block may have, one before, two after
    __shared__ signed char sep[M + 3]; // the prefixes of the splits, from the one before the block
    __shared__ unsigned char done[M];  // by number: round (+ 1) in which the region was made
    __shared__ unsigned char made[M];  // by split
    __shared__ short other[M];         // by number: the far end of the region's range
    __shared__ int edge[2], listed;
    const int i = threadIdx.x, lane = i & 31;
    const int from = max((int) blockIdx.x * (M - 2 * W) - W - 1, 0);
    if (i == 0) listed = 0;
    done[i] = made[i] = 0;
    pdl_wait();
    // the leaf that a thread may have: its node and place are on their way
    // while the block's edges are found (an iteration of 3,001 nodes 55.3 -> 53.7
    // us, 10,007 65.0 -> 64.3)
    const int place = max((int) blockIdx.x * (M - 2 * W) - W, 0) + i;
    uint32_t node = place < n ? order[place] : 0u;
    for (int j = i; j < M + 4; j += M) code[j] = from + j < n ? key[from + j] : 0u;
    const bool ok = node < (uint32_t) n; // always, for a valid sort
    if (!ok) node = 0u;
    typename RT<R>::R2 p = pos[node];
    R m = mass[node], sz = R(0);
    if (adjust) sz = size[node];
    __syncthreads();
    if (i < 64) {
        const int at = tree_edge(blockIdx.x + (i >> 5), n, W, code, from);
        if (lane == 0) edge[i >> 5] = at;
    }
    __syncthreads();
    const int s0 = edge[0], s1 = edge[1], cnt = s1 - s0;
    const uint32_t *c0 = code + (s0 - from); // c0[i]: leaf s0 + i
    const signed char *d0 = sep + 1;         // d0[i]: the split after leaf s0 + i; -1 past the ends
    if (place >= s0 && place < s1) {
        if (!ok) {
            p = mk2<R>(R(0), R(0));
            m = sz = R(0);
            atomicOr(status + ST_ERROR, ERR_BOUNDS);
        }
        const R4 rec = mk4<R>(p.x, p.y, m, sz);
        leaf[place - s0] = rec;
        A.psort[place] = rec;
    }
    for (int j = i - 1; j < cnt + 1; j += M) {
        const int k = s0 + j;
        sep[j + 1] =
            (signed char) (k >= 0 && k < n - 1 ? code_prefix(c0[j], k, c0[j + 1], k + 1) : -1);
    }
    __syncthreads();
    // A split's left child is leaf s if that shares less with the leaf before
    // it, else the region numbered s, which ends there; its right child leaf
    // s + 1 or the region numbered s + 1, which begins there.
    int lo = 0, hi = 0, num = -1; // the region of the split after leaf i, once made
    bool waits = i + 1 < cnt;
    const bool one_left = waits && d0[i - 1] < d0[i], one_right = waits && d0[i + 1] < d0[i];
    // make the region if its children were made before this round
    auto make = [&](int round) {
        const int da = one_left ? 1 : done[i], db = one_right ? 1 : done[i + 1];
        if (da == 0 || da > round || db == 0 || db > round) return false;
        const Agg<R> x = one_left ? leaf_agg(leaf[i]) : sums[i];
        const Agg<R> y = one_right ? leaf_agg(leaf[i + 1]) : sums[i + 1];
        lo = one_left ? i : other[i];
        hi = one_right ? i + 1 : other[i + 1];
        const bool is_left = d0[hi] > d0[lo - 1]; // of its parent
        num = is_left ? hi : lo;
        sums[num] = agg_combine(x, y);
        other[num] = (short) (is_left ? lo : hi);
        done[num] = (unsigned char) (round + 1);
        made[i] = 1;
        waits = false;
        return true;
    };
    // Each warp makes the regions among its own leaves (a split after its last
    // leaf waits), then the block the others, until a round makes none: what
    // is left contains an edge of the block. (As many rounds as the tree is
    // high, at most 59, and once more.)
    constexpr int HIGH = 100;
    for (int round = 1; round <= HIGH; round++) {
        const bool any = waits && lane != 31 && make(round);
        if (!__any_sync(0xffffffffu, any)) break;
        __syncwarp();
    }
    __syncthreads();
    for (int round = HIGH + 2; round <= 2 * HIGH; round++) {
        const bool any = waits && make(round);
        if (!__syncthreads_or(any)) break;
    }
    // the regions' sums, records and links, all at once (a round's lanes are
    // few), the links of the walk past a single leaf, and the climbs
    auto after = [&](int j) { // region_after of leaf s0 + j
        if (s0 + j >= n - 1) return -1;
        return d0[j + 1] < d0[j] ? n - 1 + s0 + j + 1 : s0 + j + 1;
    };
    if (num >= 0) {
        const Agg<R> z = sums[num];
        A.agg[s0 + num] = z;
        write_region<R, FULL>(A, n, s0 + num, s0 + lo, s0 + hi, s0 + i, z, after(hi), wscale);
    }
    if (i < cnt) A.rope[s0 + i] = after(i);
    // what has no parent in the block climbs: leaves, then regions
#pragma unroll 1
    for (int q = 0; q < 2; q++) {
        int l = i, r = i;
        if (q == 1) {
            if (num < 0) continue;
            l = lo, r = hi;
        } else if (i >= cnt) {
            continue;
        }
        const int up = d0[r] > d0[l - 1] ? r : l - 1; // the parent's split
        if (up >= 0 && up + 1 < cnt && made[up]) continue;
        if (APART) {
            const int at = atomicAdd(&listed, 1);
            if (at < TREE_PIECES)
                A.piece[(size_t) blockIdx.x * TREE_PIECES + at] = make_int2(s0 + l, s0 + r);
            else
                atomicOr(status + ST_ERROR, ERR_BOUNDS); // (never)
        } else {
            climb_across<R, FULL, false>(s0 + l, s0 + r, l == r ? leaf_agg(leaf[i]) : sums[num], n,
                                         key, A, wscale, status);
        }
    }
    if (APART) {
        __syncthreads();
        if (i == 0) A.pieces[blockIdx.x] = min(listed, TREE_PIECES);
    }
}

// The climbs of every block's listed regions and leaves, a warp a block.
template <class R, bool FULL>
__global__ void __launch_bounds__(TREE_THREADS)
k_tree_top(int n, int blocks, const uint32_t *__restrict__ key, TreeArrays<R> A, R wscale,
           int *__restrict__ status)
{
    pdl_wait();
    const int b = (int) ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (b >= blocks) return;
    const int cnt = A.pieces[b];
    for (int q = threadIdx.x & 31; q < cnt; q += 32) {
        const int2 p = A.piece[(size_t) b * TREE_PIECES + q];
        climb_across<R, FULL, true>(p.x, p.y, Agg<R>(), n, key, A, wscale, status);
    }
}

} // namespace fa2cu
