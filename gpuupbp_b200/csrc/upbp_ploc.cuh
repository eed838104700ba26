// Beam-map hierarchy by locally-ordered clustering (PLOC: Meister and
// Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume
// Hierarchy Construction", IEEE TVCG 2018).  The chunks are sorted by the
// Morton code of their centres; every cluster then picks, among the
// kPlocRadius clusters on either side in that order, the one whose union
// with it has the smallest surface area, and mutual choices merge into a
// node.  Iterated to one cluster, this yields a tree of surface-area quality
// (the range searches visit fewer nodes than in the Morton-split LBVH).
//
// The passes run in one cooperative launch (k_ploc_cluster): two grid
// barriers a pass, and the last kPlocTail clusters in one block.  As separate
// launches -- nearest neighbours, merge, scan of the tiles, compaction, and
// the places of each pass's nodes, about 35 times each -- a build spent
// nearly all of its time starting and draining kernels of 2-3 us.
//
// The tree is then laid out in the LBVH's node form (Karras 2012): the
// leaves in the tree's left-to-right order, and an internal node covering
// leaf range [a, b] with split g stored at b if it is a left child, at a if
// a right child (the root at 0), so that its children are g and g + 1.  Every
// internal node gets a distinct index that way, and the compressed nodes and
// all walks read the result exactly as an LBVH.  Every node finds its place
// by itself, adding up the left siblings on its way to the root
// (k_ploc_place).  The layout is checked on the device (each index written
// once); the caller replaces the tree by the LBVH when the check fails or
// the passes run out.
#pragma once

#include <cooperative_groups.h>

#include "upbp_build.cuh"

namespace upbp {

constexpr int kPlocRadius = 16;    // clusters searched on each side in Morton order
constexpr int kPlocBlock = 512;    // threads of the clustering's blocks, clusters of a tile
constexpr int kPlocTail = 1024;    // clusters one block finishes
constexpr int kPlocTailIters = 4 * kPlocTail;  // at least one merge per iteration
constexpr int kPlocPasses = 96;    // most passes of the many-cluster phase
constexpr int kPlocMaxDepth = 1 << 14;  // a longer way to the root fails the check

// Outcome words of a build.
enum : int {
    kPcNodes = 0,    // nodes created
    kPcLeft,         // clusters left (1: complete)
    kPcFail,         // layout check failures
    kPcTailIters,    // iterations of the tail
    kPcPasses,       // passes that merged
    kPcWords = 8
};

// A cluster is two float4: (lo, id) and (hi, leaf count), id >= 0 a created
// node, id < 0 the complement of a leaf's Morton position.
struct PlocScratch {
    unsigned capacity = 0;
    float4* cl[2] = {nullptr, nullptr};
    float4* leaf = nullptr;        // leaf boxes in Morton order: (lo, 0), (hi, 0)
    int* act = nullptr;            // per cluster of a pass: its partner if it creates a node, itself, or -1
    uint2* block_sum = nullptr;    // per block of a pass: clusters that stay, nodes created
    float4* node_box = nullptr;    // per created node: (lo, leaf count), (hi, 0)
    int2* node_child = nullptr;
    uint2* node_up = nullptr;      // parent | right child << 31, leaves of the left sibling (right children)
    unsigned* written = nullptr;   // writes per laid-out node index (the check)
    unsigned* order = nullptr;     // laid-out leaf order: chunk per leaf position
    unsigned* count = nullptr;     // kPcWords words
    int grid = 0;                  // blocks of the clustering's launch: what the device holds at once
    unsigned forced = 0;           // UPBP_PLOC_BLOCKS: this many instead (more than fit are refused)
    unsigned blocks = 0;           // of the last build's launch
};

UPBP_D float ploc_area(float3 lo, float3 hi)
{
    const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return dx * dy + dy * dz + dz * dx;
}


// Leaves in Morton order (vals: chunk per Morton position), which is also the
// leaf order of a tree that does not get laid out.
__global__ void k_ploc_init(BoxSource src, const unsigned* vals, unsigned n, float4* cl, float4* leaf, unsigned* order)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float3 lo, hi;
    source_box(src, vals[i], lo, hi);
    cl[2 * i] = make_float4(lo.x, lo.y, lo.z, __int_as_float(~(int)i));
    cl[2 * i + 1] = make_float4(hi.x, hi.y, hi.z, __uint_as_float(1u));
    leaf[2 * i] = make_float4(lo.x, lo.y, lo.z, 0.f);
    leaf[2 * i + 1] = make_float4(hi.x, hi.y, hi.z, 0.f);
    order[i] = vals[i];
}

// Nearest neighbour of cluster ti of s_lo, s_hi among the slots j0..j1 within
// kPlocRadius of it (its own left out), every `step`-th from offset s:
// smallest union area, ties to the lower index (met first).  The slots
// ti - kPlocRadius .. ti + kPlocRadius can all be read, so that the loads of
// several candidates are in flight at once.
template <int step>
UPBP_D int ploc_nearest(const float4* s_lo, const float4* s_hi, int ti, int j0, int j1, int s, float& best)
{
    const float3 lo = xyz(s_lo[ti]), hi = xyz(s_hi[ti]);
    best = INFINITY;
    int bj = -1;
#pragma unroll 8
    for (int d = -kPlocRadius; d < kPlocRadius + step; d += step) {
        const int j = min(ti + d + s, ti + kPlocRadius);
        const float a = ploc_area(min3f(lo, xyz(s_lo[j])), max3f(hi, xyz(s_hi[j])));
        if (d + s <= kPlocRadius && j != ti && j >= j0 && j <= j1 && (a < best || bj < 0)) {
            best = a;
            bj = j;
        }
    }
    return bj;
}

// Block-wide exclusive prefix of one value per thread; returns the prefix,
// *total the sum.
UPBP_D unsigned ploc_block_scan(unsigned v, unsigned* s_warp, unsigned* total)
{
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(~0u, incl, o);
        if (lane >= (unsigned)o) incl += u;
    }
    __syncthreads();
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        unsigned w = lane < nw ? s_warp[lane] : 0u;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(~0u, w, o);
            if (lane >= (unsigned)o) w += u;
        }
        if (lane < nw) s_warp[lane] = w;
    }
    __syncthreads();
    *total = s_warp[nw - 1];
    return incl - v + (wid > 0 ? s_warp[wid - 1] : 0u);
}

// Node k over clusters a and b (each as its two float4); returns the cluster.
UPBP_D void ploc_node(unsigned k, float4& a0, float4& a1, float4 b0, float4 b1, float4* node_box, int2* node_child,
                      uint2* node_up)
{
    const float3 lo = min3f(xyz(a0), xyz(b0)), hi = max3f(xyz(a1), xyz(b1));
    const unsigned left = __float_as_uint(a1.w), cnt = left + __float_as_uint(b1.w);
    const int ca = __float_as_int(a0.w), cb = __float_as_int(b0.w);
    node_box[2 * (size_t)k] = make_float4(lo.x, lo.y, lo.z, __uint_as_float(cnt));
    node_box[2 * (size_t)k + 1] = make_float4(hi.x, hi.y, hi.z, 0.f);
    node_child[k] = make_int2(ca, cb);
    if (ca >= 0) node_up[ca] = make_uint2(k, 0u);
    if (cb >= 0) node_up[cb] = make_uint2(k | 0x80000000u, left);
    a0 = make_float4(lo.x, lo.y, lo.z, __int_as_float((int)k));
    a1 = make_float4(hi.x, hi.y, hi.z, __uint_as_float(cnt));
}

// Shared memory of the clustering: a tile and the 2 kPlocRadius clusters on
// either side of it that its merges can depend on, or the tail.
struct PlocTile {
    float4 lo[kPlocBlock + 4 * kPlocRadius], hi[kPlocBlock + 4 * kPlocRadius];
    int nn[kPlocBlock + 4 * kPlocRadius];
};
struct PlocTailMem {  // kPlocRadius unused slots on either side
    float4 lo[kPlocTail + 2 * kPlocRadius], hi[kPlocTail + 2 * kPlocRadius];
    int nn[kPlocTail + 2 * kPlocRadius];
};
union PlocShared {
    PlocTile tile;
    PlocTailMem tail;
};

// The clustering of n leaves, a cooperative launch of at most ps.grid blocks.
// A pass over m clusters in tiles of kPlocBlock, each block a run of tiles:
// every cluster's nearest neighbour -- of the tile and kPlocRadius clusters
// around it, so that a tile knows both sides of its mutual choices -- and
// the counts of clusters that stay and nodes created; after a grid barrier
// the blocks' counts give every cluster its place in the other buffer and
// every merge its node (the lower index creates it and takes its place);
// another barrier ends the pass.  At kPlocTail clusters block 0 goes on alone.
__global__ void __launch_bounds__(kPlocBlock, 2) k_ploc_cluster(unsigned n, int passes, float4* cl0, float4* cl1,
                                                                int* act, uint2* block_sum, float4* node_box,
                                                                int2* node_child, uint2* node_up, unsigned* count)
{
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    __shared__ PlocShared sh;
    __shared__ unsigned s_warp[kPlocBlock / 32];
    __shared__ unsigned long long s_sum[2][kPlocBlock / 32];
    const int tid = (int)threadIdx.x;
    unsigned m = n, nodes = 0;
    int pass = 0;
    float4* cl = cl0;
    float4* out = cl1;
    while (m > (unsigned)kPlocTail && pass < passes) {
        const unsigned tiles = (m + kPlocBlock - 1) / kPlocBlock;
        const unsigned per = (tiles + gridDim.x - 1) / gridDim.x;
        const unsigned t0 = min(blockIdx.x * per, tiles), t1 = min(t0 + per, tiles);
        unsigned stay = 0, made = 0;  // of this block (the same in every thread)
        for (unsigned t = t0; t < t1; t++) {
            PlocTile& tl = sh.tile;
            const int base = (int)(t * kPlocBlock) - 2 * kPlocRadius;  // cluster of window slot 0
            __syncthreads();
            for (int q = tid; q < kPlocBlock + 4 * kPlocRadius; q += kPlocBlock) {
                const int j = base + q;
                if (j >= 0 && j < (int)m) {
                    tl.lo[q] = cl[2 * (size_t)j];
                    tl.hi[q] = cl[2 * (size_t)j + 1];
                }
            }
            __syncthreads();
            const int lo_slot = max(0, -base), hi_slot = min(kPlocBlock + 4 * kPlocRadius, (int)m - base) - 1;
            for (int q = tid + kPlocRadius; q < kPlocBlock + 3 * kPlocRadius; q += kPlocBlock)
                if (q >= lo_slot && q <= hi_slot) {
                    float best;
                    tl.nn[q] = ploc_nearest<1>(tl.lo, tl.hi, q, lo_slot, hi_slot, 0, best);
                }
            __syncthreads();
            const int q = tid + 2 * kPlocRadius;
            bool keep = false, makes = false;
            if (q <= hi_slot) {
                const int j = tl.nn[q];
                const bool mutual = j >= 0 && tl.nn[j] == q;
                makes = mutual && q < j;
                keep = !mutual || makes;
                act[base + q] = makes ? base + j : keep ? base + q : -1;
            }
            stay += (unsigned)__syncthreads_count(keep);
            made += (unsigned)__syncthreads_count(makes);
        }
        if (tid == 0) block_sum[blockIdx.x] = make_uint2(stay, made);
        grid.sync();
        // clusters that stay and nodes created before this block, and in all
        unsigned before, made_before, total, made_total;
        {
            unsigned long long all = 0, mine = 0;  // nodes created in the high words
            for (unsigned k = tid; k < gridDim.x; k += kPlocBlock) {
                const uint2 v = __ldcg(&block_sum[k]);
                const unsigned long long x = v.x | (unsigned long long)v.y << 32;
                all += x;
                if (k < blockIdx.x) mine += x;
            }
            for (int o = 16; o > 0; o >>= 1) {
                all += __shfl_xor_sync(~0u, all, o);
                mine += __shfl_xor_sync(~0u, mine, o);
            }
            if ((tid & 31) == 0) {
                s_sum[0][tid >> 5] = all;
                s_sum[1][tid >> 5] = mine;
            }
            __syncthreads();
            all = mine = 0;
#pragma unroll
            for (int k = 0; k < kPlocBlock / 32; k++) {
                all += s_sum[0][k];
                mine += s_sum[1][k];
            }
            before = (unsigned)mine;
            made_before = (unsigned)(mine >> 32);
            total = (unsigned)all;
            made_total = (unsigned)(all >> 32);
        }
        for (unsigned t = t0; t < t1; t++) {
            const unsigned i = t * kPlocBlock + tid;
            const int j = i < m ? act[i] : -1;
            const bool keep = j >= 0, makes = keep && j != (int)i;
            unsigned sum;
            const unsigned at = ploc_block_scan((keep ? 1u : 0u) | (makes ? 1u << 16 : 0u), s_warp, &sum);
            if (keep) {
                float4 a0 = cl[2 * (size_t)i], a1 = cl[2 * (size_t)i + 1];
                if (makes)
                    ploc_node(nodes + made_before + (at >> 16), a0, a1, cl[2 * (size_t)j], cl[2 * (size_t)j + 1],
                              node_box, node_child, node_up);
                const size_t o = before + (at & 0xffffu);
                out[2 * o] = a0;
                out[2 * o + 1] = a1;
            }
            before += sum & 0xffffu;
            made_before += sum >> 16;
        }
        grid.sync();
        m = total;
        nodes += made_total;
        pass++;
        float4* swap = cl;
        cl = out;
        out = swap;
    }
    if (blockIdx.x != 0) return;
    if (tid == 0) {
        count[kPcPasses] = (unsigned)pass;
        count[kPcLeft] = m;
    }
    if (m > (unsigned)kPlocTail) return;  // the passes ran out: the caller falls back
    // the rest in this block's shared memory
    PlocTailMem& tl = sh.tail;
    __syncthreads();
    for (unsigned i = tid; i < m; i += kPlocBlock) {
        tl.lo[kPlocRadius + i] = cl[2 * (size_t)i];
        tl.hi[kPlocRadius + i] = cl[2 * (size_t)i + 1];
    }
    __syncthreads();
    int it = 0;
    while (m > 1 && it < kPlocTailIters) {
        const int mm = (int)m, j0 = kPlocRadius, j1 = kPlocRadius + mm - 1;  // slots in use
        if (mm > kPlocBlock / 4) {
            for (int i = tid; i < mm; i += kPlocBlock) {
                float best;
                tl.nn[j0 + i] = ploc_nearest<1>(tl.lo, tl.hi, j0 + i, j0, j1, 0, best);
            }
        } else {
            // few clusters: four threads share one's candidates
            const int i = tid >> 2, s = tid & 3;
            float best = INFINITY;
            int bj = -1;
            if (i < mm) bj = ploc_nearest<4>(tl.lo, tl.hi, j0 + i, j0, j1, s, best);
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                const float ob = __shfl_xor_sync(~0u, best, o);
                const int oj = __shfl_xor_sync(~0u, bj, o);
                if (oj >= 0 && (bj < 0 || ob < best || (ob == best && oj < bj))) {
                    best = ob;
                    bj = oj;
                }
            }
            if (i < mm && s == 0) tl.nn[j0 + i] = bj;
        }
        __syncthreads();
        constexpr int per = kPlocTail / kPlocBlock;
        float4 c0[per], c1[per];
        unsigned keep = 0, makes = 0, v = 0;
        for (int q = 0; q < per; q++) {
            const int i = j0 + tid * per + q;
            if (i > j1) break;
            const int j = tl.nn[i];
            const bool mutual = j >= 0 && tl.nn[j] == i;
            if (!mutual || i < j) {
                keep |= 1u << q;
                v += 1u;
                if (mutual) {
                    makes |= 1u << q;
                    v += 1u << 16;
                }
            }
        }
        unsigned sum;
        unsigned at = ploc_block_scan(v, s_warp, &sum);
        unsigned k = nodes + (at >> 16);
        for (int q = 0; q < per; q++)
            if (keep >> q & 1u) {
                const int i = j0 + tid * per + q;
                c0[q] = tl.lo[i];
                c1[q] = tl.hi[i];
                if (makes >> q & 1u) {
                    const int j = tl.nn[i];
                    ploc_node(k++, c0[q], c1[q], tl.lo[j], tl.hi[j], node_box, node_child, node_up);
                }
            }
        __syncthreads();
        at = j0 + (at & 0xffffu);
        for (int q = 0; q < per; q++)
            if (keep >> q & 1u) {
                tl.lo[at] = c0[q];
                tl.hi[at] = c1[q];
                at++;
            }
        m = sum & 0xffffu;
        nodes += sum >> 16;
        it++;
        __syncthreads();
    }
    if (tid == 0) {
        count[kPcLeft] = m;
        count[kPcTailIters] = (unsigned)it;
        count[kPcNodes] = nodes;
    }
}

// Lays out the tree: node k walks to the root, adding the leaves of the left
// siblings it passes to its first leaf position, and writes the laid-out node
// at its index (children's boxes and links) and the leaf order at its leaf
// children's positions.
__global__ void k_ploc_place(unsigned n, const float4* leaf, const unsigned* vals, const float4* node_box,
                             const int2* node_child, const uint2* node_up, unsigned* written, unsigned* order,
                             BvhNode* nodes, unsigned* count)
{
    const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
    if (count[kPcLeft] != 1u || count[kPcNodes] != n - 1u || k >= n - 1u) return;
    const unsigned root = n - 2u;  // created last
    unsigned first = 0, cur = k;
    int depth = 0;
    while (cur != root && depth < kPlocMaxDepth) {
        const uint2 u = __ldg(&node_up[cur]);
        first += u.y;
        cur = u.x & 0x7fffffffu;
        if (cur >= n - 1u) break;
        depth++;
    }
    const unsigned cnt_k = __float_as_uint(__ldg(&node_box[2 * (size_t)k]).w);
    const unsigned index = k == root ? 0u : __ldg(&node_up[k]).x >> 31 ? first : first + cnt_k - 1u;
    if (cur != root || index >= n - 1u) {
        atomicAdd(&count[kPcFail], 1u);
        return;
    }
    const int2 ch = __ldg(&node_child[k]);
    const int c[2] = {ch.x, ch.y};
    float3 lo[2], hi[2];
    unsigned cnt[2];
    for (int s = 0; s < 2; s++) {
        if (c[s] < 0) {
            lo[s] = xyz(__ldg(&leaf[2 * (size_t)~c[s]]));
            hi[s] = xyz(__ldg(&leaf[2 * (size_t)~c[s] + 1]));
            cnt[s] = 1u;
        } else {
            const float4 b0 = __ldg(&node_box[2 * (size_t)c[s]]), b1 = __ldg(&node_box[2 * (size_t)c[s] + 1]);
            lo[s] = xyz(b0);
            hi[s] = xyz(b1);
            cnt[s] = __float_as_uint(b0.w);
        }
    }
    const int g = (int)(first + cnt[0]) - 1;
    if (g < 0 || g + 1 >= (int)n) {
        atomicAdd(&count[kPcFail], 1u);
        return;
    }
    BvhNode& nd = nodes[index];
    nd.a = make_float4(lo[0].x, lo[0].y, lo[0].z, hi[0].x);
    nd.b = make_float4(hi[0].y, hi[0].z, lo[1].x, lo[1].y);
    nd.c = make_float4(lo[1].z, hi[1].x, hi[1].y, hi[1].z);
    nd.link = make_int4(c[0] < 0 ? ~g : g, c[1] < 0 ? ~(g + 1) : g + 1, (int)cnt[0], (int)cnt[1]);
    atomicAdd(&written[index], 1u);
    if (c[0] < 0) order[g] = vals[~c[0]];
    if (c[1] < 0) order[g + 1] = vals[~c[1]];
}

// The check: every internal index of the laid-out tree written exactly once
// (then each node's children cover disjoint, smaller leaf ranges, and every
// walk ends).
__global__ void k_ploc_check(unsigned n, const unsigned* written, unsigned* count)
{
    unsigned bad = 0;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n - 1u; i += gridDim.x * blockDim.x)
        bad += written[i] != 1u;
    if (bad) atomicAdd(&count[kPcFail], bad);
}

// Builds the n-leaf tree (n >= 2) over the boxes of `src` into `nodes`
// (n - 1 nodes) and its leaf order (*sorted_vals), with at most `passes`
// passes, and copies the outcome into the page-locked words `outcome`
// (kPcWords).  Nothing waits for it: the caller reads the outcome with
// ploc_complete after its next synchronisation with the stream, and until
// then uses the tree for nothing; a tree that is not complete (the passes ran
// out -- boxes so alike that few merge per pass -- or the layout check
// failed) is replaced.  The clustering takes at most max_blocks blocks (0: no
// limit).  When the device refuses its cooperative launch (ploc_refused: too
// many blocks for what it holds at once, or no such launches) there is no tree,
// and the caller builds the LBVH instead.
inline bool ploc_refused(cudaError_t e)
{
    return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported || e == cudaErrorLaunchOutOfResources;
}

inline cudaError_t build_ploc(const BoxSource& src, unsigned n, BvhNode* nodes, BuildScratch& sc, PlocScratch& ps,
                              cudaStream_t st, const unsigned** sorted_vals, unsigned* launches, unsigned* outcome,
                              int passes, unsigned max_blocks)
{
    passes = std::max(1, std::min(passes, kPlocPasses));
    // (leaf links hold kLeafShift bits, and so do the searches' entries)
    if (n < 2 || n > kMaxBvhPrimitives || n > ps.capacity || ps.grid < 1) return cudaErrorInvalidValue;
    // Morton order of the centres
    const unsigned init[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
    cudaError_t e = cudaMemcpyAsync(sc.ord6, init, sizeof(init), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    const unsigned bs = 256;
    const unsigned grid = (n + bs - 1) / bs;
    k_bounds<<<grid < 1184 ? grid : 1184, bs, 0, st>>>(src, n, sc.ord6);
    k_morton<<<grid, bs, 0, st>>>(src, n, sc.ord6, sc.keys, sc.vals);
    cub::DoubleBuffer<unsigned> kb(sc.keys, sc.keys_alt), vb(sc.vals, sc.vals_alt);
    size_t tb = sc.temp_bytes;
    e = cub::DeviceRadixSort::SortPairs(sc.temp, tb, kb, vb, (int)n, 0, 30, st);
    if (e != cudaSuccess) return e;
    const unsigned* vals = vb.Current();
    e = cudaMemsetAsync(ps.count, 0, kPcWords * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(ps.written, 0, (size_t)(n - 1) * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    k_ploc_init<<<grid, bs, 0, st>>>(src, vals, n, ps.cl[0], ps.leaf, ps.order);
    // one block per tile, no more than are resident at once (the grid barriers)
    unsigned blocks = std::min<unsigned>((unsigned)ps.grid, (n + kPlocBlock - 1) / kPlocBlock);
    if (ps.forced) blocks = ps.forced;
    if (max_blocks) blocks = std::min(blocks, max_blocks);
    ps.blocks = blocks;
    void* args[] = {&n, &passes, &ps.cl[0], &ps.cl[1], &ps.act, &ps.block_sum, &ps.node_box, &ps.node_child,
                    &ps.node_up, &ps.count};
    e = cudaLaunchCooperativeKernel((const void*)k_ploc_cluster, dim3(blocks), dim3(kPlocBlock), args, 0, st);
    if (e != cudaSuccess) {
        cudaGetLastError();  // a refused launch is not sticky
        return e;
    }
    k_ploc_place<<<grid, bs, 0, st>>>(n, ps.leaf, vals, ps.node_box, ps.node_child, ps.node_up, ps.written, ps.order,
                                      nodes, ps.count);
    k_ploc_check<<<std::min(grid, 1184u), bs, 0, st>>>(n, ps.written, ps.count);
    *launches += 6;
    e = cudaMemcpyAsync(outcome, ps.count, kPcWords * sizeof(unsigned), cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) return e;
    *sorted_vals = ps.order;
    return cudaGetLastError();
}

// Whether the build whose outcome words these are (n leaves) produced a
// complete, checked tree.
inline bool ploc_complete(const unsigned* outcome, unsigned n)
{
    return outcome[kPcLeft] == 1u && outcome[kPcNodes] == n - 1 && outcome[kPcFail] == 0u;
}

}  // namespace upbp
