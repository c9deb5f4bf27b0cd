// Adaptive linear octree over Morton-sorted particles: the topology of all levels at once (each
// particle decides from its neighbours' keys which nodes start at it) and a single bottom-up
// moments kernel (last-arriving child computes its parent).
//
// This file is compiled with --fmad=false: the FP64 moment sums must round exactly as written
// (fixed order, no contraction) so that node moments are bit-identical to the oracle's.
//
// Replaces the reference's level loop with a host sync per level
// (engine/physics/octree/cuda/linear/OctBuild.inl:156-199, OctLeafKernels.inl:7-81,
// OctParentKernels.inl:7-103, OctLinkKernels.inl): same idea (node = Morton cell, children
// from the next 3 key bits, FP64 mass/COM), but leaves are adaptive (<= leaf_cap particles),
// children of a node are contiguous (breadth-first layout, no `next` links needed) and the
// moments include the quadrupole.
#include "bz_common.cuh"
#include "bz_kernels.h"

#include <algorithm>

namespace bz {

namespace {

constexpr int kThreads = 256;
constexpr int kLevels = kMaxLevels + 1;  // levels 0 .. kMaxLevels

// ---- topology ---------------------------------------------------------------------------
// A cell of level L is the run of particles whose keys share L octant digits.  It is a node of
// the tree when its parent cell holds more than a leaf (or lies above min_split).  The nodes that
// start at particle i therefore form one chain of levels [b, e]:
//   b = the first level whose cell boundary falls between i - 1 and i;
//   the node (i, b) exists when the cell of level b - 1 around i holds more than leaf_cap
//   particles (a backward search of at most leaf_cap keys finds that cell's start, unless the
//   particle leaf_cap before i still belongs to it);
//   the chain goes on while the cell itself holds more than a leaf: e - 1 = the digits that
//   particle i shares with particle i + leaf_cap.
// So every particle decides alone, and the breadth-first index of a node is its level's offset
// plus the number of that level's starts before i: a count per level and block, one scan of
// each level, and an emission.  A kernel a level (binary searches for the octant boundaries of
// every node, a look-back scan) chained 21 launches of 1 to 38 us.  Topology time, level chain ->
// this: Plummer 65k 163 -> 22 us, isolated TreePM 1M 390 -> 83 us, Hernquist 4M 680 -> 135 us,
// the 256^3 lattice 319 -> 243 us (the tree phase with it 0.73 -> 0.62 ms).  Bound by latency below a
// million particles (four launches), by the issue of the key comparisons above.

// Octant digits two keys share (0 .. kMaxLevels).
__device__ __forceinline__ int common_levels(unsigned long long x, unsigned long long y)
{
    return x == y ? kMaxLevels : (__clzll(static_cast<long long>(x ^ y)) - 1) / 3;
}

// Whether two keys share l octant digits.
__device__ __forceinline__ bool shares(unsigned long long x, unsigned long long y, int l)
{
    return ((x ^ y) >> (3 * (kMaxLevels - l))) == 0ull;
}

// Particles a thread takes, by the system's size: short runs fill the SMs with the smaller
// systems, long ones keep the scan of the block counts short.
constexpr int kTreeSmall = 1 << 20, kTreeMiddle = 1 << 23;
int tree_items(int n) { return n < kTreeSmall ? 2 : (n < kTreeMiddle ? 4 : 16); }
int tree_blocks(int n) { return (n + kThreads * tree_items(n) - 1) / (kThreads * tree_items(n)); }

// The boundary level b and the chain [b, e] of every particle (packed b | e << 8; e < b where no
// node starts) and, per level and block, the nodes.
__global__ void __launch_bounds__(kThreads) k_tree_chains(const unsigned long long* __restrict__ keys, int n,
                                                           int items, int leaf_cap, int min_split,
                                                           unsigned short* __restrict__ chain,
                                                           int* __restrict__ counts)
{
    __shared__ int cnt[kLevels];
    if (threadIdx.x < kLevels)
        cnt[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * kThreads * items;
    const int back = (leaf_cap + 1) / 2, ahead = leaf_cap / 2;
#pragma unroll 4
    for (int it = 0; it < items; ++it) {
        const int i = base + it * kThreads + threadIdx.x;
        if (i >= n)
            break;
        // all the keys that most particles need, loaded side by side
        const unsigned long long key = keys[i], prev = keys[max(i - 1, 0)];
        const unsigned long long kb = keys[max(i - back, 0)], ka = keys[ahead < n - i ? i + ahead : i];
        const unsigned long long kl = keys[max(i - leaf_cap, 0)], kr = keys[leaf_cap < n - i ? i + leaf_cap : i];
        const int b = i > 0 ? common_levels(prev, key) + 1 : 0;
        bool exists = b <= min_split;
        if (!exists && b <= kMaxLevels) {
            // More than leaf_cap particles around i in one cell reach half a leaf to one side of
            // it at least (most particles, inside a leaf, stop here).
            const int l = b - 1;
            if ((i >= back && shares(kb, key, l)) || (ahead < n - i && shares(ka, key, l))) {
                if (i >= leaf_cap && shares(kl, key, l)) {
                    exists = true;
                } else {
                    // the start of the cell of level l around i, less than leaf_cap before it
                    int lo = max(i - leaf_cap + 1, 0), hi = i;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (shares(keys[mid], key, l))
                            hi = mid;
                        else
                            lo = mid + 1;
                    }
                    // (leaf_cap may exceed n: no sum before the comparison)
                    exists = leaf_cap < n - lo && shares(keys[lo + leaf_cap], key, l);
                }
            }
        }
        int packed = b;  // e = 0 < b: no node starts here
        if (exists) {
            int e = max(b, min_split);
            if (leaf_cap < n - i)
                e = max(e, min(common_levels(kr, key) + 1, kMaxLevels));
            packed = b | e << 8;
            for (int l = b; l <= e; ++l)
                atomicAdd(&cnt[l], 1);
        }
        chain[i] = static_cast<unsigned short>(packed);
    }
    __syncthreads();
    if (threadIdx.x < kLevels)
        counts[threadIdx.x * gridDim.x + blockIdx.x] = cnt[threadIdx.x];
}

// Block l: exclusive scan of level l's block counts, its total to lvl_count[l].
__global__ void __launch_bounds__(1024) k_tree_scan(int* __restrict__ counts, int blocks, TreeArrays t)
{
    __shared__ int carry;
    __shared__ int ws[32];
    int* c = counts + static_cast<size_t>(blockIdx.x) * blocks;
    if (threadIdx.x == 0)
        carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int base = 0; base < blocks; base += 1024) {
        const int i = base + threadIdx.x;
        const int v = i < blocks ? c[i] : 0;
        const int x = warp_incl_scan(v);
        if (lane == 31)
            ws[warp] = x;
        __syncthreads();
        if (warp == 0)
            ws[lane] = warp_incl_scan(ws[lane]);
        __syncthreads();
        const int before = (warp > 0 ? ws[warp - 1] : 0) + carry;
        if (i < blocks)
            c[i] = before + x - v;
        __syncthreads();
        if (threadIdx.x == 1023)
            carry = before + x;
        __syncthreads();
    }
    if (threadIdx.x == 0)
        t.lvl_count[blockIdx.x] = carry;
}

// First particle after `from` (which shares l digits with key), at most `limit`, that does not.
__device__ __forceinline__ int cell_end(const unsigned long long* __restrict__ keys, unsigned long long key,
                                        int from, int l, int limit)
{
    int lo = from;
    int step = 32;
    while (step < limit - lo && shares(keys[lo + step], key, l)) {
        lo += step;
        step <<= 1;
    }
    int hi = step < limit - lo ? lo + step : limit;
    ++lo;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (shares(keys[mid], key, l))
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Writes the nodes.  Each warp takes 32 x items consecutive particles, lists those at which nodes
// start, and works on 32 of these at a time (an eighth of a lattice's particles start a node; with
// a lane a particle the kernel took 292 us at 16.7M, 98 so).  Lane l of a warp carries
// the index of level l's next node.  A node ends where the next start with b <= its level lies:
// every cell boundary that ends a node starts another one, a child of their common ancestor.
__global__ void __launch_bounds__(kThreads) k_tree_emit(const unsigned long long* __restrict__ keys, int n, int items,
                                                         const unsigned short* __restrict__ chain,
                                                         const int* __restrict__ counts, TreeArrays t, int* err)
{
    extern __shared__ int s_list[];  // [kThreads * items]: offset | b << 16 | e << 24
    __shared__ int ws[kThreads / 32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = lanemask_lt();
    // level offsets; levels that would pass the node capacity are cut off: the nodes of the last
    // level kept stay leaves, and the overflow is reported
    const int total = lane < kLevels ? t.lvl_count[lane] : 0;
    const long long incl = [&] {
        long long x = total;
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(kFullMask, x, o);
            if (lane >= o)
                x += y;
        }
        return x;
    }();
    const unsigned fits = __ballot_sync(kFullMask, lane < kLevels && incl <= t.cap);
    const int last = 31 - __clz(fits);  // (level 0 holds one node: it always fits)
    const int nodes = static_cast<int>(__shfl_sync(kFullMask, incl, last));
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        t.n_nodes[0] = nodes;
        t.parent[0] = -1;
        if (last < kMaxLevels)
            raise_error(err, kErrTreeCapacity);
    }
    const int base = (blockIdx.x * (kThreads / 32) + warp) * 32 * items;
    int* list = s_list + warp * 32 * items;
    int starts = 0;
    for (int r = 0; r < items; ++r) {
        const int i = base + r * 32 + lane;
        const int c = i < n ? chain[i] : 1;
        const int b = c & 0xff, e = min(c >> 8, last);
        const unsigned m = __ballot_sync(kFullMask, b <= e);
        if (b <= e)
            list[starts + __popc(m & lt)] = (r * 32 + lane) | b << 16 | e << 24;
        starts += __popc(m);
    }
    __syncwarp();
    int mine = 0;
    for (int g = 0; g < starts; g += 32) {
        const int c = g + lane < starts ? list[g + lane] : 1 << 16;
        const int b = c >> 16 & 0xff, e = c >> 24;
        const int lo = __reduce_min_sync(kFullMask, b <= e ? b : kLevels), hi = __reduce_max_sync(kFullMask, b <= e ? e : -1);
        for (int l = lo; l <= hi; ++l) {
            const int k = __popc(__ballot_sync(kFullMask, b <= l && l <= e));
            mine += lane == l ? k : 0;
        }
    }
    ws[warp][lane] = mine;
    __syncthreads();
    int next = static_cast<int>(incl) - total;
    if (lane < kLevels)
        next += counts[static_cast<size_t>(lane) * gridDim.x + blockIdx.x];
    for (int w = 0; w < warp; ++w)
        next += ws[w][lane];
    for (int g = 0; g < starts; g += 32) {
        const bool real = g + lane < starts;
        const int c = real ? list[g + lane] : 1 << 16;
        const int i = base + (c & 0xffff), b = c >> 16 & 0xff, e = c >> 24;
        const int lo = __reduce_min_sync(kFullMask, b <= e ? b : kLevels), hi = __reduce_max_sync(kFullMask, b <= e ? e : -1);
        const int tail = __shfl_sync(kFullMask, i, min(starts - g, 32) - 1);  // the last start here
        const unsigned long long key = real ? keys[i] : 0ull;
        // the node of the level above that starts last before this particle
        int above = lo > 0 ? __shfl_sync(kFullMask, next, lo - 1) - 1 : -1;
        int end = n;
        for (int l = lo; l <= hi; ++l) {
            const bool in = b <= l && l <= e;
            const unsigned m = __ballot_sync(kFullMask, in);
            const unsigned edge = __ballot_sync(kFullMask, real && b <= l) & (0xfffffffeu << lane);
            const int at = __shfl_sync(kFullMask, i, edge != 0u ? __ffs(edge) - 1 : 0);
            const int k = __shfl_sync(kFullMask, next, l) + __popc(m & lt);
            if (in) {
                end = edge != 0u ? at : (l == 0 ? n : cell_end(keys, key, tail, l, end));
                t.start[k] = i;
                t.count[k] = end - i;
                t.parent[k] = above;
                t.level[k] = l;
                t.arrive[k] = 0;
                t.nchild[k] = 0;
                if (l > b)
                    t.child[above] = k;  // the chain's node above starts at this particle too
                if (l == e)
                    t.child[k] = -1;
            }
            above = in ? k : k - 1;
            next += lane == l ? __popc(m) : 0;
        }
    }
}

// The child count of every split node, from the last of its (consecutive) children.  Sorted keys give
// every node but the root a split parent one level up.  After a sort that gave up (the call reports it)
// they need not: a node without such a parent is left out of the tree, so that every link that the moments
// and the walk follow is a node's own.
__global__ void __launch_bounds__(kThreads) k_tree_children(TreeArrays t)
{
    const int nn = t.n_nodes[0];
    for (int k = blockIdx.x * kThreads + threadIdx.x + 1; k < nn; k += gridDim.x * kThreads) {
        const int p = t.parent[k];
        if ((k + 1 == nn || t.parent[k + 1] != p) && p >= 0 && t.child[p] >= 0 && t.level[p] + 1 == t.level[k])
            t.nchild[p] = k - t.child[p] + 1;
    }
}

// QUAD = false (monopole walks): the second moments are left zero, without their pass.
template <bool QUAD>
__device__ void leaf_moments(const float4* __restrict__ pos4, int k, TreeArrays& t)
{
    const int s = t.start[k], e = s + t.count[k];
    float mn[3] = {3.402823466e38f, 3.402823466e38f, 3.402823466e38f};
    float mx[3] = {-3.402823466e38f, -3.402823466e38f, -3.402823466e38f};
    double tm = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
    for (int i = s; i < e; ++i) {
        const float4 p = pos4[i];
        mn[0] = fminf(mn[0], p.x);
        mn[1] = fminf(mn[1], p.y);
        mn[2] = fminf(mn[2], p.z);
        mx[0] = fmaxf(mx[0], p.x);
        mx[1] = fmaxf(mx[1], p.y);
        mx[2] = fmaxf(mx[2], p.z);
        tm += (double)p.w;
        sx += (double)p.w * (double)p.x;
        sy += (double)p.w * (double)p.y;
        sz += (double)p.w * (double)p.z;
    }
    const double cx = tm > 0.0 ? sx / tm : 0.5 * ((double)mn[0] + (double)mx[0]);
    const double cy = tm > 0.0 ? sy / tm : 0.5 * ((double)mn[1] + (double)mx[1]);
    const double cz = tm > 0.0 ? sz / tm : 0.5 * ((double)mn[2] + (double)mx[2]);
    double q[6] = {0, 0, 0, 0, 0, 0};
    for (int i = s; QUAD && i < e; ++i) {
        const float4 p = pos4[i];
        const double dx = (double)p.x - cx, dy = (double)p.y - cy, dz = (double)p.z - cz;
        const double w = (double)p.w;
        q[0] += w * dx * dx;
        q[1] += w * dx * dy;
        q[2] += w * dx * dz;
        q[3] += w * dy * dy;
        q[4] += w * dy * dz;
        q[5] += w * dz * dz;
    }
    t.m64[k] = tm;
    t.s64[3 * k] = sx;
    t.s64[3 * k + 1] = sy;
    t.s64[3 * k + 2] = sz;
    if (QUAD) {  // the FP64 centre and second moments feed only the parents' second moments
        t.c64[3 * k] = cx;
        t.c64[3 * k + 1] = cy;
        t.c64[3 * k + 2] = cz;
        for (int j = 0; j < 6; ++j)
            t.q64[6 * k + j] = q[j];
    }
    t.box0[k] = make_float4(mn[0], mn[1], mn[2], __int_as_float(s));
    t.box1[k] = make_float4(mx[0], mx[1], mx[2], __int_as_float(-(e - s)));
    t.mono[k] = make_float4((float)cx, (float)cy, (float)cz, (float)tm);
    t.quadA[k] = make_float4((float)q[0], (float)q[1], (float)q[2], (float)q[3]);
    t.quadB[k] = make_float2((float)q[4], (float)q[5]);
}

template <bool QUAD>
__device__ void internal_moments(int k, TreeArrays& t)
{
    const int c0 = t.child[k], nc = t.nchild[k];
    // Both passes are unrolled over the (at most 8) children with predication, so the loads of
    // all children issue together and one climb step costs about one memory round trip; the
    // sums still run in octant order.
    float mn[3] = {3.402823466e38f, 3.402823466e38f, 3.402823466e38f};
    float mx[3] = {-3.402823466e38f, -3.402823466e38f, -3.402823466e38f};
    double tm = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (j < nc) {
            const int c = c0 + j;
            const float4 b0 = __ldcg(&t.box0[c]);
            const float4 b1 = __ldcg(&t.box1[c]);
            mn[0] = fminf(mn[0], b0.x);
            mn[1] = fminf(mn[1], b0.y);
            mn[2] = fminf(mn[2], b0.z);
            mx[0] = fmaxf(mx[0], b1.x);
            mx[1] = fmaxf(mx[1], b1.y);
            mx[2] = fmaxf(mx[2], b1.z);
            tm += __ldcg(&t.m64[c]);
            sx += __ldcg(&t.s64[3 * c]);
            sy += __ldcg(&t.s64[3 * c + 1]);
            sz += __ldcg(&t.s64[3 * c + 2]);
        }
    }
    const double cx = tm > 0.0 ? sx / tm : 0.5 * ((double)mn[0] + (double)mx[0]);
    const double cy = tm > 0.0 ? sy / tm : 0.5 * ((double)mn[1] + (double)mx[1]);
    const double cz = tm > 0.0 ? sz / tm : 0.5 * ((double)mn[2] + (double)mx[2]);
    double q[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (QUAD && j < nc) {
            const int c = c0 + j;
            const double dx = __ldcg(&t.c64[3 * c]) - cx;
            const double dy = __ldcg(&t.c64[3 * c + 1]) - cy;
            const double dz = __ldcg(&t.c64[3 * c + 2]) - cz;
            const double w = __ldcg(&t.m64[c]);
            q[0] += __ldcg(&t.q64[6 * c]) + w * dx * dx;
            q[1] += __ldcg(&t.q64[6 * c + 1]) + w * dx * dy;
            q[2] += __ldcg(&t.q64[6 * c + 2]) + w * dx * dz;
            q[3] += __ldcg(&t.q64[6 * c + 3]) + w * dy * dy;
            q[4] += __ldcg(&t.q64[6 * c + 4]) + w * dy * dz;
            q[5] += __ldcg(&t.q64[6 * c + 5]) + w * dz * dz;
        }
    }
    t.m64[k] = tm;
    t.s64[3 * k] = sx;
    t.s64[3 * k + 1] = sy;
    t.s64[3 * k + 2] = sz;
    if (QUAD) {  // the FP64 centre and second moments feed only the parents' second moments
        t.c64[3 * k] = cx;
        t.c64[3 * k + 1] = cy;
        t.c64[3 * k + 2] = cz;
        for (int j = 0; j < 6; ++j)
            t.q64[6 * k + j] = q[j];
    }
    t.box0[k] = make_float4(mn[0], mn[1], mn[2], __int_as_float(c0));
    t.box1[k] = make_float4(mx[0], mx[1], mx[2], __int_as_float(nc));
    t.mono[k] = make_float4((float)cx, (float)cy, (float)cz, (float)tm);
    t.quadA[k] = make_float4((float)q[0], (float)q[1], (float)q[2], (float)q[3]);
    t.quadB[k] = make_float2((float)q[4], (float)q[5]);
}

// One thread per leaf computes its moments, then climbs: the child that arrives last at a
// parent (atomic counter) computes the parent from all children in octant order.
template <bool QUAD>
__global__ void __launch_bounds__(kThreads) k_tree_moments(const float4* __restrict__ pos4,
                                                            TreeArrays t)
{
    const int nn = t.n_nodes[0];
    for (int k = blockIdx.x * kThreads + threadIdx.x; k < nn; k += gridDim.x * kThreads) {
        if (t.nchild[k] != 0)
            continue;
        leaf_moments<QUAD>(pos4, k, t);
        int node = k;
        for (;;) {
            const int p = t.parent[node];
            if (p < 0)
                break;
            // release this node's moments and, for the last child, acquire its siblings'
            int old;
            asm volatile("atom.add.acq_rel.gpu.s32 %0, [%1], 1;" : "=r"(old) : "l"(&t.arrive[p]) : "memory");
            if (old != t.nchild[p] - 1)
                break;
            internal_moments<QUAD>(p, t);
            node = p;
        }
    }
}


// clear_arrive: the arrival counters are not fresh from a build (a refit of an existing tree)
void enqueue_moments(const float4* pos4, TreeArrays& t, int sms, cudaStream_t s, bool quad,
                     bool clear_arrive)
{
    if (clear_arrive)
        cudaMemsetAsync(t.arrive, 0, sizeof(int) * static_cast<size_t>(t.cap), s);
    long long mb = (static_cast<long long>(t.cap) + kThreads - 1) / kThreads;
    if (mb > 16LL * sms)
        mb = 16LL * sms;
    count_launch();
    if (quad)
        k_tree_moments<true><<<static_cast<int>(mb), kThreads, 0, s>>>(pos4, t);
    else
        k_tree_moments<false><<<static_cast<int>(mb), kThreads, 0, s>>>(pos4, t);
}

} // namespace

void launch_tree_refit(const float4* pos4, TreeArrays& t, cudaStream_t s, bool quad)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    enqueue_moments(pos4, t, sms, s, quad, true);
}

size_t tree_count_words(int n)
{
    // the largest of any n' <= n: a workspace serves every smaller system
    const int a = tree_blocks(std::min(n, kTreeSmall - 1)), b = tree_blocks(std::min(n, kTreeMiddle - 1));
    return static_cast<size_t>(std::max(tree_blocks(n), std::max(a, b))) * kLevels;
}

void launch_tree_build(const unsigned long long* sorted_keys, const float4* pos4, int n, int leaf_cap,
                       TreeArrays& t, int* err, cudaStream_t s, int min_split, bool quad)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int items = tree_items(n), blocks = tree_blocks(n);
    count_launch(4);
    k_tree_chains<<<blocks, kThreads, 0, s>>>(sorted_keys, n, items, leaf_cap, min_split, t.chain, t.counts);
    k_tree_scan<<<kLevels, 1024, 0, s>>>(t.counts, blocks, t);
    k_tree_emit<<<blocks, kThreads, sizeof(int) * kThreads * items, s>>>(sorted_keys, n, items, t.chain, t.counts, t, err);
    const int cb = (n + kThreads - 1) / kThreads;
    k_tree_children<<<cb < 8 * sms ? cb : 8 * sms, kThreads, 0, s>>>(t);
    enqueue_moments(pos4, t, sms, s, quad, false);
}

} // namespace bz

// ---- reference-mode topology ------------------------------------------------------------
// The reference's linear octree for its own keys.  Its bit spread keeps 10 bits per axis, so
// keys are < 2^30, while the leaf prefix is key >> 3*(21 - leafDepth) with leafDepth <= 11
// for any n below 16*8^11: every key has prefix 0, the build yields exactly one leaf holding
// all particles in sorted order, the parent loop never runs and that leaf is the root
// (engine/physics/octree/cuda/linear/OctBuild.inl:109-199).  This kernel builds that node as
// buildLinearOctreeLeafNodesKernel does (OctLeafKernels.inl:7-81): FP32 tight box, FP64 mass
// and weighted position sums in sorted order.  The reference is compiled with nvcc's default
// contraction, so its `w += x * m` sums and `0.5f * ext + 1e-6f` execute as fused
// multiply-adds; they are written as explicit fmas here (this file is otherwise compiled
// without contraction).
namespace bz {
namespace {
__global__ void k_reference_leaf(const float* __restrict__ x, const float* __restrict__ y,
                                 const float* __restrict__ z, const float* __restrict__ m,
                                 const uint32_t* __restrict__ sorted_index, int n, float* hot8)
{
    if (blockIdx.x != 0 || threadIdx.x != 0)
        return;
    float mn[3] = {3.402823466e38f, 3.402823466e38f, 3.402823466e38f};
    float mx[3] = {-3.402823466e38f, -3.402823466e38f, -3.402823466e38f};
    double tm = 0.0, wx = 0.0, wy = 0.0, wz = 0.0;
    for (int j = 0; j < n; ++j) {
        const uint32_t p = sorted_index[j];
        const float px = x[p], py = y[p], pz = z[p], pm = m[p];
        mn[0] = fminf(mn[0], px);
        mn[1] = fminf(mn[1], py);
        mn[2] = fminf(mn[2], pz);
        mx[0] = fmaxf(mx[0], px);
        mx[1] = fmaxf(mx[1], py);
        mx[2] = fmaxf(mx[2], pz);
        tm += (double)pm;
        wx = __fma_rn((double)px, (double)pm, wx);
        wy = __fma_rn((double)py, (double)pm, wy);
        wz = __fma_rn((double)pz, (double)pm, wz);
    }
    const float cx = 0.5f * (mn[0] + mx[0]);
    const float cy = 0.5f * (mn[1] + mx[1]);
    const float cz = 0.5f * (mn[2] + mx[2]);
    const float half = __fmaf_rn(0.5f, fmaxf(fmaxf(mx[0] - mn[0], mx[1] - mn[1]), mx[2] - mn[2]), 1.0e-6f);
    hot8[0] = cx;
    hot8[1] = cy;
    hot8[2] = cz;
    hot8[3] = half;
    hot8[4] = (float)tm;
    hot8[5] = tm > 0.0 ? (float)(wx / tm) : cx;
    hot8[6] = tm > 0.0 ? (float)(wy / tm) : cy;
    hot8[7] = tm > 0.0 ? (float)(wz / tm) : cz;
}
} // namespace

void launch_reference_leaf(const float* x, const float* y, const float* z, const float* m,
                           const uint32_t* sorted_index, int n, float* hot8, cudaStream_t s)
{
    count_launch();
    k_reference_leaf<<<1, 32, 0, s>>>(x, y, z, m, sorted_index, n, hot8);
}

} // namespace bz
