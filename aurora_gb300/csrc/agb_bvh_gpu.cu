// GPU binned-SAH BVH2 builder, producing the same 64-byte node layout and leaf encoding as the host
// builder (agb_bvh_build.cpp): over the triangles of a mesh (BLAS, leaves of at most 4 triangles)
// and over instance boxes (TLAS, one instance per leaf).
//
// Top-down, in two parts, split so that the whole chip works on the few large nodes at the top and every
// small subtree is finished by one CTA without going back to the host or to global memory:
//   - nodes of more than kSub primitives, one level per round of four launches whose CTAs each take a
//     chunk of a node's primitives: (1) boxes, (2) bins, both reduced in shared memory and then by
//     atomics on the node's record, (3) the split (every chunk sweeps the node's bins, the node's first
//     chunk writes the node and its children), (4) a stable partition into the other order array;
//   - every node of at most kSub primitives, all in one launch: a CTA holds the node's primitives,
//     order and finished nodes in shared memory and builds the subtree level by level, one warp per node.
// One node, in either part:
//   1. the box and centroid box of its primitives; the box goes into the parent's child slot (the node
//      layout keeps both child boxes in the parent);
//   2. a node of at most leafMax primitives becomes a leaf (ref ~(first << 3 | count - 1));
//   3. otherwise 16 bins per axis over the centroid box collect counts and boxes (atomics on
//      order-preserving integer encodings of the floats); half a warp per axis scans the 15 split planes
//      with the SAH cost area(L) n(L) + area(R) n(R);
//   4. a stable partition, the children, and the node's id (large nodes first, in level order; then each
//      subtree's nodes in one run, in its level order).
// Nodes that could exceed the depth budget (the traversal stack holds 48 entries for TLAS + BLAS)
// split at their index midpoint, which halves every subtree and bounds the depth: the tree is then
// at most maxDepth deep whenever ceil(log2(count / leafMax)) + 2 <= maxDepth.
//
// What bounds it: the top levels by the latency of their four dependent launches (a level of 81,920
// triangles takes 30 us), the subtrees by shared-memory atomics and shuffles of one warp per node.  Device
// time of the kernels for 81,920 triangles and 64 instances: 2.73 ms with one CTA of 128 threads per node
// and a launch and a host round trip per level, 0.41 ms so; agb_geometry_create of 1,310,720 triangles with
// its uploads: 70 and 23 ms.  Subtrees of 512: their top levels keep few warps busy, larger ones would
// leave fewer CTAs (160 for 81,920 triangles) and less of an SM's shared memory to a second one.
#include <algorithm>

#include "agb_kernels.h"

namespace agb
{
namespace
{

constexpr int kBins      = 16;
constexpr int kBlasLeaf  = 4;
// Largest subtree that one CTA builds: its nodes (64 bytes each), boxes, order and task lists and bins are
// 67 KB of shared memory, so three CTAs share an SM.
constexpr int kSub        = 512;
constexpr int kSubThreads = 256;
constexpr int kSubWarps   = kSubThreads / 32;
constexpr int kChunkThreads = 256; // large nodes: threads per chunk
constexpr uint32_t kChunk   = 2048; // and primitives per chunk

struct BuildTask
{
    uint32_t first, count;
    int32_t parent; // node index, -1 for the root
    int32_t side;   // 0 / 1: which child slot of the parent
    int32_t depth;
    uint32_t chunk0; // large nodes: index of the first chunk
    uint32_t buf;    // order array that holds the range (0 / 1)
};

// A large node's record: boxes and bins as order-preserving integers, then the split.
struct BigNode
{
    int32_t box[6], cbox[6]; // lo xyz, hi xyz
    uint32_t cnt[3][kBins];
    int32_t lo[3][kBins][3], hi[3][kBins][3];
    int32_t axis, split; // axis -1: index midpoint
    uint32_t nLeft;
};

enum : int
{
    BC_NEXT = 0, // large nodes of the next level
    BC_CHUNKS,   // and their chunks
    BC_SMALL,    // subtrees for the second part
    BC_NODES,    // nodes numbered so far
    BC_ROOT,     // root ref
    BC_DEPTH,    // deepest node seen
    BC_ERROR,
    BC_COUNT
};

__device__ __forceinline__ int32_t orderedFromFloat(float f)
{
    int32_t i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float floatFromOrdered(int32_t i)
{
    return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF);
}

__device__ __forceinline__ float boxArea(const float* lo, const float* hi)
{
    float d0 = fmaxf(0.f, hi[0] - lo[0]), d1 = fmaxf(0.f, hi[1] - lo[1]), d2 = fmaxf(0.f, hi[2] - lo[2]);
    return 2.f * (d0 * d1 + d1 * d2 + d2 * d0);
}

__device__ __forceinline__ int ceilLog2(uint32_t x)
{
    int r = 0;
    while ((1u << r) < x)
        r++;
    return r;
}

// Min / max over the warp of a box as order-preserving integers (lo xyz, hi xyz).
__device__ __forceinline__ void warpBox(int32_t v[6])
{
#pragma unroll
    for (int k = 0; k < 6; k++)
        v[k] = k < 3 ? __reduce_min_sync(0xffffffffu, v[k]) : __reduce_max_sync(0xffffffffu, v[k]);
}

struct Bounds
{
    int32_t box[6], cbox[6];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int k = 0; k < 6; k++)
            box[k] = cbox[k] = orderedFromFloat(k < 3 ? INFINITY : -INFINITY);
    }
    __device__ __forceinline__ void add(const float* p, int stride)
    {
#pragma unroll
        for (int k = 0; k < 3; k++)
        {
            const float lo = p[k * stride], hi = p[(3 + k) * stride];
            const int32_t c = orderedFromFloat(0.5f * (lo + hi));
            box[k]      = min(box[k], orderedFromFloat(lo));
            box[3 + k]  = max(box[3 + k], orderedFromFloat(hi));
            cbox[k]     = min(cbox[k], c);
            cbox[3 + k] = max(cbox[3 + k], c);
        }
    }
};

__device__ __forceinline__ void writeChildBox(BNode& P, int side, const int32_t box[6])
{
    const float4 xy = make_float4(floatFromOrdered(box[0]), floatFromOrdered(box[3]), floatFromOrdered(box[1]),
        floatFromOrdered(box[4]));
    const float z0 = floatFromOrdered(box[2]), z1 = floatFromOrdered(box[5]);
    if (side == 0)
    {
        P.c0xy = xy;
        P.cz.x = z0;
        P.cz.y = z1;
    }
    else
    {
        P.c1xy = xy;
        P.cz.z = z0;
        P.cz.w = z1;
    }
}
__device__ __forceinline__ void writeChildRef(BNode& P, int side, int32_t ref)
{
    if (side == 0)
        P.ref.x = ref;
    else
        P.ref.y = ref;
}

// Bin of a primitive along axis a of a centroid range.
__device__ __forceinline__ int binOf(float lo, float hi, float c0, float scale)
{
    return min(max(int((0.5f * (lo + hi) - c0) * scale), 0), kBins - 1);
}

// The SAH split of a node from its bins, by one full warp: the axis (-1: none, split at the index
// midpoint), the last bin of the left side and the number of primitives there, the same on every lane.
// Half a warp holds an axis's 16 bins; prefix and suffix boxes by shuffles.  The smallest cost, then the
// lowest axis, then the lowest plane.
__device__ void warpSplit(const uint32_t* cnt, const int32_t* lo, const int32_t* hi, const int32_t cbox[6], int& axis,
    int& split, uint32_t& nLeft)
{
    const int lane = threadIdx.x & 31, k = lane & 15;
    float best    = INFINITY;
    axis          = -1;
    split         = 0;
    nLeft         = 0;
#pragma unroll
    for (int round = 0; round < 2; round++)
    {
        const int a     = min(round * 2 + (lane >> 4), 2); // axes 0, 1, then 2 (twice)
        const float ext = a == 0 ? floatFromOrdered(cbox[3]) - floatFromOrdered(cbox[0])
            : a == 1             ? floatFromOrdered(cbox[4]) - floatFromOrdered(cbox[1])
                                 : floatFromOrdered(cbox[5]) - floatFromOrdered(cbox[2]);
        const int at    = a * kBins + k;
        // L: bins 0 .. k; R: bins k .. 15.
        float L[6], R[6];
#pragma unroll
        for (int q = 0; q < 3; q++)
        {
            L[q] = R[q] = floatFromOrdered(lo[at * 3 + q]);
            L[3 + q] = R[3 + q] = floatFromOrdered(hi[at * 3 + q]);
        }
        uint32_t nl = cnt[at], nr = nl;
#pragma unroll
        for (int off = 1; off < 16; off <<= 1)
        {
#pragma unroll
            for (int q = 0; q < 6; q++)
            {
                const float l = __shfl_up_sync(0xffffffffu, L[q], off, 16), r = __shfl_down_sync(0xffffffffu, R[q], off, 16);
                if (k >= off)
                    L[q] = q < 3 ? fminf(L[q], l) : fmaxf(L[q], l);
                if (k + off < 16)
                    R[q] = q < 3 ? fminf(R[q], r) : fmaxf(R[q], r);
            }
            const uint32_t l = __shfl_up_sync(0xffffffffu, nl, off, 16), r = __shfl_down_sync(0xffffffffu, nr, off, 16);
            nl += k >= off ? l : 0u;
            nr += k + off < 16 ? r : 0u;
        }
        const float areaL  = boxArea(L, L + 3);
        const float areaR  = __shfl_down_sync(0xffffffffu, boxArea(R, R + 3), 1, 16);
        const uint32_t nR1 = __shfl_down_sync(0xffffffffu, nr, 1, 16);
        float cost         = INFINITY;
        if (ext > 0.f && k < kBins - 1 && nl > 0 && nR1 > 0)
            cost = areaL * float(nl) + areaR * float(nR1);
        // Lanes in order are axes in order, planes in order: the first lane with the smallest cost.
        float least = cost;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            least = fminf(least, __shfl_xor_sync(0xffffffffu, least, off));
        if (least < best)
        {
            const int w = __ffs(__ballot_sync(0xffffffffu, cost == least)) - 1;
            best        = least;
            axis        = __shfl_sync(0xffffffffu, a, w);
            split       = w & 15;
            nLeft       = __shfl_sync(0xffffffffu, nl, w);
        }
    }
}

__device__ __forceinline__ bool forceMidpoint(int depth, uint32_t count, uint32_t leafMax, int maxDepth)
{
    return depth + ceilLog2((count + leafMax - 1) / leafMax) + 2 >= maxDepth;
}

__device__ void clearBigNode(BigNode& b, int t, int threads)
{
    const int32_t lo = orderedFromFloat(INFINITY), hi = orderedFromFloat(-INFINITY);
    for (int k = t; k < 6; k += threads)
        b.box[k] = b.cbox[k] = k < 3 ? lo : hi;
    for (int k = t; k < 3 * kBins; k += threads)
        (&b.cnt[0][0])[k] = 0;
    for (int k = t; k < 9 * kBins; k += threads)
    {
        (&b.lo[0][0][0])[k] = lo;
        (&b.hi[0][0][0])[k] = hi;
    }
}

// A new large node (its record, its chunks) or subtree, by one full block.  tasks / chunkTask / big: the
// next level's arrays.
__device__ void createTask(BuildTask t, uint32_t* counters, BuildTask* tasks, uint32_t* chunkTask, BigNode* big,
    BuildTask* small)
{
    __shared__ uint32_t slot, chunk0;
    const bool large      = t.count > uint32_t(kSub);
    const uint32_t chunks = (t.count + kChunk - 1) / kChunk;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        slot = atomicAdd(counters + (large ? BC_NEXT : BC_SMALL), 1u);
        if (large)
        {
            chunk0   = atomicAdd(counters + BC_CHUNKS, chunks);
            t.chunk0 = chunk0;
            tasks[slot] = t;
        }
        else
            small[slot] = t;
    }
    __syncthreads();
    if (!large)
        return;
    clearBigNode(big[slot], threadIdx.x, blockDim.x);
    for (uint32_t k = threadIdx.x; k < chunks; k += blockDim.x)
        chunkTask[chunk0 + k] = slot;
}

// The root's task and the counters.
__global__ void __launch_bounds__(kChunkThreads) k_bvh_begin(uint32_t n, uint32_t* counters, BuildTask* tasks,
    uint32_t* chunkTask, BigNode* big, BuildTask* small)
{
    if (threadIdx.x < BC_COUNT)
        counters[threadIdx.x] = 0;
    createTask(BuildTask{ 0, n, -1, 0, 0, 0, 0 }, counters, tasks, chunkTask, big, small);
}

// A chunk of a large node: its task, and its range of the task's primitives.
struct Chunk
{
    BuildTask task;
    uint32_t index, begin, end; // chunk of the task; positions in the order array
};
__device__ __forceinline__ Chunk chunkOf(const BuildTask* tasks, const uint32_t* chunkTask, uint32_t c)
{
    Chunk q;
    q.task  = tasks[chunkTask[c]];
    q.index = c - q.task.chunk0;
    q.begin = q.task.first + q.index * kChunk;
    q.end   = q.task.first + min(q.task.count, (q.index + 1) * kChunk);
    return q;
}

__global__ void __launch_bounds__(kChunkThreads) k_bvh_bounds(const float* boxes, const uint32_t* order,
    const BuildTask* tasks, const uint32_t* chunkTask, BigNode* big)
{
    const Chunk q = chunkOf(tasks, chunkTask, blockIdx.x);
    BigNode& B    = big[chunkTask[blockIdx.x]];
    Bounds b;
    b.clear();
    for (uint32_t i = q.begin + threadIdx.x; i < q.end; i += kChunkThreads)
        b.add(boxes + 6 * size_t(order[i]), 1);
    warpBox(b.box);
    warpBox(b.cbox);
    __shared__ int32_t part[kChunkThreads / 32][12];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < 6; k++)
        {
            part[warp][k]     = b.box[k];
            part[warp][6 + k] = b.cbox[k];
        }
    __syncthreads();
    if (threadIdx.x < 12)
    {
        const int k  = threadIdx.x % 6;
        int32_t v    = part[0][threadIdx.x];
        for (int w = 1; w < kChunkThreads / 32; w++)
            v = k < 3 ? min(v, part[w][threadIdx.x]) : max(v, part[w][threadIdx.x]);
        int32_t* dst = threadIdx.x < 6 ? B.box + k : B.cbox + k;
        if (k < 3)
            atomicMin(dst, v);
        else
            atomicMax(dst, v);
    }
}

__global__ void __launch_bounds__(kChunkThreads) k_bvh_bins(const float* boxes, const uint32_t* order,
    const BuildTask* tasks, const uint32_t* chunkTask, BigNode* big, int maxDepth, uint32_t leafMax)
{
    const Chunk q = chunkOf(tasks, chunkTask, blockIdx.x);
    BigNode& B    = big[chunkTask[blockIdx.x]];
    if (forceMidpoint(q.task.depth, q.task.count, leafMax, maxDepth))
        return;
    __shared__ BigNode S;
    clearBigNode(S, threadIdx.x, kChunkThreads);
    __syncthreads();
    float c0[3], scale[3];
    bool use[3];
#pragma unroll
    for (int a = 0; a < 3; a++)
    {
        c0[a]           = floatFromOrdered(B.cbox[a]);
        const float ext = floatFromOrdered(B.cbox[3 + a]) - c0[a];
        use[a]          = ext > 0.f;
        scale[a]        = float(kBins) / ext;
    }
    for (uint32_t i = q.begin + threadIdx.x; i < q.end; i += kChunkThreads)
    {
        const float* p = boxes + 6 * size_t(order[i]);
        int32_t e[6];
#pragma unroll
        for (int k = 0; k < 6; k++)
            e[k] = orderedFromFloat(p[k]);
#pragma unroll
        for (int a = 0; a < 3; a++)
        {
            if (!use[a])
                continue;
            const int bin = binOf(p[a], p[3 + a], c0[a], scale[a]);
            atomicAdd(&S.cnt[a][bin], 1u);
#pragma unroll
            for (int k = 0; k < 3; k++)
            {
                atomicMin(&S.lo[a][bin][k], e[k]);
                atomicMax(&S.hi[a][bin][k], e[3 + k]);
            }
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 3 * kBins; k += kChunkThreads)
    {
        const uint32_t c = (&S.cnt[0][0])[k];
        if (c == 0)
            continue;
        atomicAdd(&B.cnt[0][0] + k, c);
#pragma unroll
        for (int j = 0; j < 3; j++)
        {
            atomicMin(&B.lo[0][0][0] + 3 * k + j, (&S.lo[0][0][0])[3 * k + j]);
            atomicMax(&B.hi[0][0][0] + 3 * k + j, (&S.hi[0][0][0])[3 * k + j]);
        }
    }
}

// The split, and the number of left primitives of each chunk; the node's first chunk writes the node
// and its children.
__global__ void __launch_bounds__(kChunkThreads) k_bvh_split(const float* boxes, const uint32_t* order,
    const BuildTask* tasks, const uint32_t* chunkTask, BigNode* big, uint32_t* chunkLeft, BNode* nodes,
    uint32_t nodeCapacity, uint32_t* counters, BuildTask* nextTasks, uint32_t* nextChunkTask, BigNode* nextBig,
    BuildTask* small, int maxDepth, uint32_t leafMax)
{
    const Chunk q = chunkOf(tasks, chunkTask, blockIdx.x);
    BigNode& B    = big[chunkTask[blockIdx.x]];
    __shared__ int axisS, splitS;
    __shared__ uint32_t nLeftS, leftSum;
    __shared__ int32_t nodeId;
    if (threadIdx.x < 32)
    {
        int32_t cbox[6];
#pragma unroll
        for (int k = 0; k < 6; k++)
            cbox[k] = B.cbox[k];
        int axis = -1, split = 0;
        uint32_t nLeft = 0;
        if (!forceMidpoint(q.task.depth, q.task.count, leafMax, maxDepth))
            warpSplit(&B.cnt[0][0], &B.lo[0][0][0], &B.hi[0][0][0], cbox, axis, split, nLeft);
        if (axis < 0)
            nLeft = q.task.count / 2;
        if (threadIdx.x == 0)
        {
            axisS   = axis;
            splitS  = split;
            nLeftS  = nLeft;
            leftSum = 0;
            if (q.index == 0)
            {
                B.axis  = axis;
                B.split = split;
                B.nLeft = nLeft;
            }
        }
    }
    __syncthreads();
    const int a          = axisS;
    const uint32_t nLeft = nLeftS;
    if (a >= 0)
    {
        const float c0 = floatFromOrdered(B.cbox[a]), scale = float(kBins) / (floatFromOrdered(B.cbox[3 + a]) - c0);
        uint32_t mine = 0;
        for (uint32_t i = q.begin + threadIdx.x; i < q.end; i += kChunkThreads)
        {
            const float* p = boxes + 6 * size_t(order[i]);
            mine += binOf(p[a], p[3 + a], c0, scale) <= splitS ? 1u : 0u;
        }
        mine = __reduce_add_sync(0xffffffffu, mine);
        if ((threadIdx.x & 31) == 0)
            atomicAdd(&leftSum, mine);
        __syncthreads();
        if (threadIdx.x == 0)
            chunkLeft[blockIdx.x] = leftSum;
    }
    if (q.index != 0)
        return;
    if (threadIdx.x == 0)
    {
        atomicMax(counters + BC_DEPTH, uint32_t(q.task.depth));
        const uint32_t id = atomicAdd(counters + BC_NODES, 1u);
        nodeId            = id < nodeCapacity ? int32_t(id) : -1;
        if (nodeId < 0)
            atomicExch(counters + BC_ERROR, 1u);
        else
        {
            nodes[id].ref = make_int4(0, 0, 0, 0);
            if (q.task.parent >= 0)
            {
                writeChildBox(nodes[q.task.parent], q.task.side, B.box);
                writeChildRef(nodes[q.task.parent], q.task.side, int32_t(id));
            }
            else
                counters[BC_ROOT] = id;
        }
    }
    __syncthreads();
    if (nodeId < 0)
        return;
    const uint32_t buf = q.task.buf ^ 1u;
    createTask(BuildTask{ q.task.first, nLeft, nodeId, 0, q.task.depth + 1, 0, buf }, counters, nextTasks, nextChunkTask,
        nextBig, small);
    createTask(BuildTask{ q.task.first + nLeft, q.task.count - nLeft, nodeId, 1, q.task.depth + 1, 0, buf }, counters,
        nextTasks, nextChunkTask, nextBig, small);
}

__global__ void __launch_bounds__(kChunkThreads) k_bvh_partition(const float* boxes, const uint32_t* order,
    uint32_t* out, const BuildTask* tasks, const uint32_t* chunkTask, const BigNode* big, const uint32_t* chunkLeft)
{
    const Chunk q    = chunkOf(tasks, chunkTask, blockIdx.x);
    const BigNode& B = big[chunkTask[blockIdx.x]];
    const int a      = B.axis;
    if (a < 0)
    {
        for (uint32_t i = q.begin + threadIdx.x; i < q.end; i += kChunkThreads)
            out[i] = order[i];
        return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ uint32_t beforeS, warpLeft[kChunkThreads / 32];
    if (threadIdx.x == 0)
        beforeS = 0;
    __syncthreads();
    uint32_t mine = 0;
    for (uint32_t k = threadIdx.x; k < q.index; k += kChunkThreads)
        mine += chunkLeft[q.task.chunk0 + k];
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0)
        atomicAdd(&beforeS, mine);
    __syncthreads();
    uint32_t before = beforeS; // left primitives before this slice
    const float c0  = floatFromOrdered(B.cbox[a]), scale = float(kBins) / (floatFromOrdered(B.cbox[3 + a]) - c0);
    const uint32_t rightBase = q.task.first + B.nLeft;
    for (uint32_t base = q.begin; base < q.end; base += kChunkThreads)
    {
        const uint32_t i = base + threadIdx.x;
        const bool valid = i < q.end;
        const uint32_t p = valid ? order[i] : 0;
        bool left        = false;
        if (valid)
        {
            const float* b = boxes + 6 * size_t(p);
            left           = binOf(b[a], b[3 + a], c0, scale) <= B.split;
        }
        const unsigned m = __ballot_sync(0xffffffffu, left);
        __syncthreads();
        if (lane == 0)
            warpLeft[warp] = __popc(m);
        __syncthreads();
        uint32_t rank = before + __popc(m & ((1u << lane) - 1u)), sum = 0;
#pragma unroll
        for (int w = 0; w < kChunkThreads / 32; w++)
        {
            rank += w < warp ? warpLeft[w] : 0u;
            sum += warpLeft[w];
        }
        if (valid)
            out[left ? q.task.first + rank : rightBase + (i - q.task.first - rank)] = p;
        before += sum;
    }
}

// One subtree per CTA.  Shared memory: the finished nodes, the primitives' boxes (six arrays), two order
// arrays (positions in the subtree's range), two task lists, and each warp's bins.
struct SubTask
{
    uint16_t first, count;
    int16_t parent; // local node, -1: the subtree's root
    int16_t side;
};
struct SubShared
{
    BNode nodes[kSub - 1];
    float box[6][kSub];
    uint16_t order[2][kSub];
    uint16_t leafOrder[kSub];
    SubTask tasks[2][kSub];
    uint32_t cnt[kSubWarps][3 * kBins];
    int32_t lo[kSubWarps][9 * kBins], hi[kSubWarps][9 * kBins];
    uint32_t taskCount[2], nodeCount, base;
};

__global__ void __launch_bounds__(kSubThreads) k_bvh_subtree(const float* boxes, uint32_t* orderA,
    const uint32_t* orderB, const BuildTask* tasks, BNode* nodes, uint32_t nodeCapacity, uint32_t* counters,
    int maxDepth, uint32_t leafMax)
{
    extern __shared__ __align__(16) unsigned char raw[];
    SubShared& S      = *reinterpret_cast<SubShared*>(raw);
    const BuildTask T = tasks[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // The range's primitives; the leaves write orderA in place, so they are read here once and for all.
    uint32_t ids[kSub / kSubThreads];
#pragma unroll
    for (int j = 0; j < kSub / kSubThreads; j++)
    {
        const uint32_t i = uint32_t(j * kSubThreads + tid);
        ids[j]           = 0;
        if (i < T.count)
        {
            ids[j]         = (T.buf ? orderB : orderA)[T.first + i];
            const float* p = boxes + 6 * size_t(ids[j]);
#pragma unroll
            for (int k = 0; k < 6; k++)
                S.box[k][i] = p[k];
            S.order[0][i] = uint16_t(i);
        }
    }
    if (tid == 0)
    {
        S.taskCount[0] = 1;
        S.taskCount[1] = 0;
        S.nodeCount    = 0;
        S.tasks[0][0]  = SubTask{ 0, uint16_t(T.count), -1, int16_t(T.side) };
    }
    __syncthreads();
    int level = 0;
    for (; S.taskCount[level & 1] > 0; level++)
    {
        const int cur = level & 1, depth = T.depth + level;
        const uint32_t n = S.taskCount[cur];
        for (uint32_t w = warp; w < n; w += kSubWarps)
        {
            const SubTask t        = S.tasks[cur][w];
            const uint16_t* src    = S.order[cur] + t.first;
            uint16_t* dst          = S.order[cur ^ 1] + t.first;
            const uint32_t count   = t.count;
            BNode* const parent    = t.parent >= 0 ? S.nodes + t.parent : T.parent >= 0 ? nodes + T.parent : nullptr;
            Bounds b;
            b.clear();
            for (uint32_t i = lane; i < count; i += 32)
                b.add(&S.box[0][src[i]], kSub);
            warpBox(b.box);
            warpBox(b.cbox);
            if (lane == 0 && parent)
                writeChildBox(*parent, t.side, b.box);
            if (count <= leafMax)
            {
                for (uint32_t i = lane; i < count; i += 32)
                    S.leafOrder[t.first + i] = src[i];
                if (lane == 0)
                {
                    const int32_t ref = ~int32_t(((T.first + t.first) << 3) | (count - 1));
                    if (parent)
                        writeChildRef(*parent, t.side, ref);
                    else
                        counters[BC_ROOT] = uint32_t(ref);
                }
                continue;
            }
            int axis = -1, split = 0;
            uint32_t nLeft = 0;
            float c0[3], scale[3];
#pragma unroll
            for (int a = 0; a < 3; a++)
            {
                c0[a]    = floatFromOrdered(b.cbox[a]);
                scale[a] = float(kBins) / (floatFromOrdered(b.cbox[3 + a]) - c0[a]);
            }
            if (!forceMidpoint(depth, count, leafMax, maxDepth))
            {
                uint32_t* cnt = S.cnt[warp];
                int32_t *lo = S.lo[warp], *hi = S.hi[warp];
                for (int k = lane; k < 9 * kBins; k += 32)
                {
                    if (k < 3 * kBins)
                        cnt[k] = 0;
                    lo[k] = orderedFromFloat(INFINITY);
                    hi[k] = orderedFromFloat(-INFINITY);
                }
                __syncwarp();
                for (uint32_t i = lane; i < count; i += 32)
                {
                    const uint32_t p = src[i];
                    float v[6];
                    int32_t e[6];
#pragma unroll
                    for (int k = 0; k < 6; k++)
                    {
                        v[k] = S.box[k][p];
                        e[k] = orderedFromFloat(v[k]);
                    }
#pragma unroll
                    for (int a = 0; a < 3; a++)
                    {
                        if (!(floatFromOrdered(b.cbox[3 + a]) - c0[a] > 0.f))
                            continue;
                        const int at = a * kBins + binOf(v[a], v[3 + a], c0[a], scale[a]);
                        atomicAdd(cnt + at, 1u);
#pragma unroll
                        for (int k = 0; k < 3; k++)
                        {
                            atomicMin(lo + 3 * at + k, e[k]);
                            atomicMax(hi + 3 * at + k, e[3 + k]);
                        }
                    }
                }
                __syncwarp();
                warpSplit(cnt, lo, hi, b.cbox, axis, split, nLeft);
            }
            if (axis < 0)
            {
                nLeft = count / 2;
                for (uint32_t i = lane; i < count; i += 32)
                    dst[i] = src[i];
            }
            else
            {
                uint32_t before = 0;
                const float a0 = axis == 0 ? c0[0] : axis == 1 ? c0[1] : c0[2];
                const float as = axis == 0 ? scale[0] : axis == 1 ? scale[1] : scale[2];
                for (uint32_t base = 0; base < count; base += 32)
                {
                    const uint32_t i = base + lane;
                    const bool valid = i < count;
                    const uint32_t p = valid ? src[i] : 0;
                    const bool left  = valid && binOf(S.box[axis][p], S.box[3 + axis][p], a0, as) <= split;
                    const unsigned m = __ballot_sync(0xffffffffu, left);
                    const uint32_t r = before + __popc(m & ((1u << lane) - 1u));
                    if (valid)
                        dst[left ? r : nLeft + (i - r)] = uint16_t(p);
                    before += __popc(m);
                }
            }
            if (lane == 0)
            {
                const uint32_t id = atomicAdd(&S.nodeCount, 1u);
                S.nodes[id].ref   = make_int4(0, 0, 0, 0);
                // Refs are local until the base is known; the subtree root's parent is global.
                if (t.parent >= 0)
                    writeChildRef(*parent, t.side, int32_t(id));
                const uint32_t slot         = atomicAdd(&S.taskCount[cur ^ 1], 2u);
                S.tasks[cur ^ 1][slot]     = SubTask{ t.first, uint16_t(nLeft), int16_t(id), 0 };
                S.tasks[cur ^ 1][slot + 1] = SubTask{ uint16_t(t.first + nLeft), uint16_t(count - nLeft), int16_t(id), 1 };
            }
        }
        __syncthreads();
        if (tid == 0)
            S.taskCount[cur] = 0;
        __syncthreads();
    }
    // The subtree's nodes take one run of ids; the leaves' order goes back through the primitives' ids.
    uint32_t* idOf = reinterpret_cast<uint32_t*>(&S.box[0][0]); // the boxes are no longer needed
#pragma unroll
    for (int j = 0; j < kSub / kSubThreads; j++)
        idOf[j * kSubThreads + tid] = ids[j];
    if (tid == 0)
    {
        S.base = atomicAdd(counters + BC_NODES, S.nodeCount);
        atomicMax(counters + BC_DEPTH, uint32_t(T.depth + level - 1));
    }
    __syncthreads();
    for (uint32_t i = tid; i < T.count; i += kSubThreads)
        orderA[T.first + i] = idOf[S.leafOrder[i]];
    const uint32_t n = S.nodeCount, base = S.base;
    if (n == 0)
        return;
    if (base + n > nodeCapacity)
    {
        if (tid == 0)
            atomicExch(counters + BC_ERROR, 1u);
        return;
    }
    for (uint32_t i = tid; i < n; i += kSubThreads)
    {
        BNode nd = S.nodes[i];
        nd.ref.x += nd.ref.x >= 0 ? int32_t(base) : 0;
        nd.ref.y += nd.ref.y >= 0 ? int32_t(base) : 0;
        nodes[base + i] = nd;
    }
    if (tid == 0)
    {
        if (T.parent >= 0)
            writeChildRef(nodes[T.parent], T.side, int32_t(base));
        else
            counters[BC_ROOT] = base;
    }
}

// See readBvhTop: one warp, a level at a time.
__global__ void __launch_bounds__(32) k_bvh_top(const BNode* nodes, int32_t root, BNode* out)
{
    __shared__ int32_t at[kBvhTopNodes];
    static_assert(kBvhTopNodes < 32, "a lane per node");
    const int t = threadIdx.x;
    if (t < kBvhTopNodes)
        at[t] = t == 0 ? root : -1;
    __syncwarp();
    for (int level = 0; level < kBvhTopLevels; level++)
    {
        if (t < (1 << level))
        {
            const int k = (1 << level) - 1 + t;
            BNode n{};
            if (at[k] >= 0)
            {
                n = nodes[at[k]];
                if (level + 1 < kBvhTopLevels && n.ref.x >= 0)
                {
                    at[2 * k + 1] = n.ref.x;
                    n.ref.x       = 2 * k + 1;
                }
                if (level + 1 < kBvhTopLevels && n.ref.y >= 0)
                {
                    at[2 * k + 2] = n.ref.y;
                    n.ref.y       = 2 * k + 2;
                }
            }
            out[k] = n;
        }
        __syncwarp();
    }
}

__global__ void k_tri_boxes(const float* positions, const uint32_t* indices, uint32_t ntri, float* boxes)
{
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < ntri; t += gridDim.x * blockDim.x)
    {
        float lo[3] = { INFINITY, INFINITY, INFINITY }, hi[3] = { -INFINITY, -INFINITY, -INFINITY };
        for (int v = 0; v < 3; v++)
        {
            const float* p = positions + 3 * size_t(indices[3 * size_t(t) + v]);
            for (int k = 0; k < 3; k++)
            {
                lo[k] = fminf(lo[k], p[k]);
                hi[k] = fmaxf(hi[k], p[k]);
            }
        }
        for (int k = 0; k < 3; k++)
        {
            boxes[6 * size_t(t) + k]     = lo[k];
            boxes[6 * size_t(t) + 3 + k] = hi[k];
        }
    }
}

__global__ void k_iota(uint32_t* order, uint32_t n)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        order[i] = i;
}

// Triangles in leaf order: v0 (w = triangle id bits), v1, v2.
__global__ void k_reorder_tris(const float* positions, const uint32_t* indices, const uint32_t* order,
    uint32_t ntri, float4* tris)
{
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < ntri; s += gridDim.x * blockDim.x)
    {
        uint32_t t = order[s];
        for (int v = 0; v < 3; v++)
        {
            const float* p = positions + 3 * size_t(indices[3 * size_t(t) + v]);
            tris[3 * size_t(s) + v] = make_float4(p[0], p[1], p[2], v == 0 ? __int_as_float(int32_t(t)) : 0.f);
        }
    }
}

// The large nodes' arrays for n primitives, carved out of one allocation (each level's, twice).
struct BigArrays
{
    BuildTask* tasks[2];
    BigNode* nodes[2];
    uint32_t* chunkTask[2];
    uint32_t* chunkLeft;
    size_t bytes;
};
BigArrays carveBig(void* base, size_t n)
{
    // A large node holds more than kSub primitives; each has at most one partly filled chunk.
    const size_t most = n / kSub + 2, chunks = n / kChunk + most + 2;
    size_t at         = 0;
    auto take         = [&](size_t bytes) {
        void* p = static_cast<char*>(base) + at;
        at += (bytes + 255) & ~size_t(255);
        return p;
    };
    BigArrays b;
    for (int k = 0; k < 2; k++)
    {
        b.tasks[k]     = static_cast<BuildTask*>(take(most * sizeof(BuildTask)));
        b.nodes[k]     = static_cast<BigNode*>(take(most * sizeof(BigNode)));
        b.chunkTask[k] = static_cast<uint32_t*>(take(chunks * 4));
    }
    b.chunkLeft = static_cast<uint32_t*>(take(chunks * 4));
    b.bytes     = at;
    return b;
}

// Scratch for n primitives in one allocation: their boxes (written by the caller), order arrays, the large
// nodes' arrays, the subtree list (every split may leave one) and the counters.
cudaError_t reserve(GpuBvhScratch& s, size_t n)
{
    const size_t sizes[6] = { n * 24, n * 4, n * 4, carveBig(nullptr, n).bytes, (n + 2) * sizeof(BuildTask),
        BC_COUNT * sizeof(uint32_t) };
    size_t total = 0;
    for (size_t b : sizes)
        total += (b + 255) & ~size_t(255);
    if (s.arraysBytes < total)
    {
        cudaFree(s.arrays);
        s.arrays      = nullptr;
        s.arraysBytes = 0;
        const cudaError_t e = cudaMalloc(&s.arrays, total);
        if (e != cudaSuccess)
            return e;
        s.arraysBytes = total;
    }
    char* at  = static_cast<char*>(s.arrays);
    auto take = [&](int k) {
        void* p = at;
        at += (sizes[k] + 255) & ~size_t(255);
        return p;
    };
    s.boxes    = static_cast<float*>(take(0));
    s.order    = static_cast<uint32_t*>(take(1));
    s.scratch  = static_cast<uint32_t*>(take(2));
    s.big      = take(3);
    s.subtrees = take(4);
    s.counters = take(5);
    return cudaSuccess;
}

// The build over s.boxes (n primitives); s.order ends in leaf order.
cudaError_t buildLevels(uint32_t n, uint32_t leafMax, int maxDepth, GpuBvhScratch& s, BNode* nodes,
    uint32_t nodeCapacity, int32_t* rootOut, int32_t* depthOut, uint32_t* nodeCountOut, cudaStream_t st)
{
    cudaError_t e;
    static_assert(sizeof(SubShared) <= 227 * 1024, "a subtree's shared memory");
    if ((e = cudaFuncSetAttribute(k_bvh_subtree, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(SubShared)))) !=
        cudaSuccess)
        return e;
    unsigned g = unsigned(std::min<size_t>((size_t(n) + 255) / 256, 4096));
    k_iota<<<g, 256, 0, st>>>(s.order, n);
    uint32_t* cnt   = static_cast<uint32_t*>(s.counters);
    BuildTask* sub  = static_cast<BuildTask*>(s.subtrees);
    BigArrays big   = carveBig(s.big, n);
    k_bvh_begin<<<1, kChunkThreads, 0, st>>>(n, cnt, big.tasks[0], big.chunkTask[0], big.nodes[0], sub);
    const bool large = n > uint32_t(kSub);
    // Large nodes of the level, their chunks, subtrees so far.
    uint32_t h[BC_COUNT] = { large ? 1u : 0u, large ? (n + kChunk - 1) / kChunk : 0u, large ? 0u : 1u };
    for (int level = 0; h[BC_NEXT] > 0; level++)
    {
        if (level > maxDepth + 1)
            return cudaErrorInvalidValue;
        const int c = level & 1, x = c ^ 1;
        uint32_t *in = c ? s.scratch : s.order, *out = c ? s.order : s.scratch;
        if ((e = cudaMemsetAsync(cnt, 0, 2 * sizeof(uint32_t), st)) != cudaSuccess)
            return e;
        const unsigned chunks = h[BC_CHUNKS];
        k_bvh_bounds<<<chunks, kChunkThreads, 0, st>>>(s.boxes, in, big.tasks[c], big.chunkTask[c], big.nodes[c]);
        k_bvh_bins<<<chunks, kChunkThreads, 0, st>>>(s.boxes, in, big.tasks[c], big.chunkTask[c], big.nodes[c], maxDepth,
            leafMax);
        k_bvh_split<<<chunks, kChunkThreads, 0, st>>>(s.boxes, in, big.tasks[c], big.chunkTask[c], big.nodes[c],
            big.chunkLeft, nodes, nodeCapacity, cnt, big.tasks[x], big.chunkTask[x], big.nodes[x], sub, maxDepth, leafMax);
        k_bvh_partition<<<chunks, kChunkThreads, 0, st>>>(s.boxes, in, out, big.tasks[c], big.chunkTask[c], big.nodes[c],
            big.chunkLeft);
        if ((e = cudaGetLastError()) != cudaSuccess ||
            (e = cudaMemcpyAsync(h, cnt, 3 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
            (e = cudaStreamSynchronize(st)) != cudaSuccess)
            return e;
    }
    if (h[BC_SMALL] > 0)
        k_bvh_subtree<<<h[BC_SMALL], kSubThreads, sizeof(SubShared), st>>>(s.boxes, s.order, s.scratch, sub, nodes,
            nodeCapacity, cnt, maxDepth, leafMax);
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = cudaMemcpyAsync(h, cnt, sizeof h, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return e;
    if (h[BC_ERROR])
        return cudaErrorInvalidValue;
    *nodeCountOut = h[BC_NODES];
    *rootOut      = int32_t(h[BC_ROOT]);
    *depthOut     = int32_t(h[BC_DEPTH]);
    return cudaSuccess;
}

} // namespace

cudaError_t buildBlasGpu(const float* positions, const uint32_t* indices, uint32_t ntri, int maxDepth,
    GpuBvhScratch& s, BNode* nodes, uint32_t nodeCapacity, float4* tris, int32_t* rootOut, int32_t* depthOut,
    uint32_t* nodeCountOut, cudaStream_t st)
{
    cudaError_t e = reserve(s, ntri);
    if (e != cudaSuccess)
        return e;
    unsigned g = unsigned(std::min<size_t>((size_t(ntri) + 255) / 256, 4096));
    k_tri_boxes<<<g, 256, 0, st>>>(positions, indices, ntri, s.boxes);
    if ((e = buildLevels(ntri, kBlasLeaf, maxDepth, s, nodes, nodeCapacity, rootOut, depthOut, nodeCountOut,
             st)) != cudaSuccess)
        return e;
    k_reorder_tris<<<g, 256, 0, st>>>(positions, indices, s.order, ntri, tris);
    return cudaGetLastError();
}

cudaError_t buildTlasGpu(const float* boxesHost, uint32_t count, int maxDepth, GpuBvhScratch& s, BNode* nodes,
    uint32_t nodeCapacity, int32_t* orderOut, int32_t* rootOut, int32_t* depthOut, uint32_t* nodeCountOut,
    cudaStream_t st)
{
    cudaError_t e = reserve(s, count);
    if (e != cudaSuccess)
        return e;
    if ((e = cudaMemcpyAsync(s.boxes, boxesHost, size_t(count) * 24, cudaMemcpyHostToDevice, st)) != cudaSuccess)
        return e;
    if ((e = buildLevels(count, 1, maxDepth, s, nodes, nodeCapacity, rootOut, depthOut, nodeCountOut, st)) !=
        cudaSuccess)
        return e;
    return cudaMemcpyAsync(orderOut, s.order, size_t(count) * 4, cudaMemcpyDeviceToDevice, st);
}

cudaError_t readBvhTop(GpuBvhScratch& s, const BNode* nodes, int32_t root, BNode* host, cudaStream_t st)
{
    // The large nodes' arrays, at least two records twice, are free once the tree is built.
    static_assert(sizeof(BigNode) * 4 >= sizeof(BNode) * kBvhTopNodes, "room for the top of the tree");
    BNode* top = static_cast<BNode*>(s.big);
    k_bvh_top<<<1, 32, 0, st>>>(nodes, root, top);
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? e
                            : cudaMemcpyAsync(host, top, sizeof(BNode) * kBvhTopNodes, cudaMemcpyDeviceToHost, st);
}

void freeGpuBvhScratch(GpuBvhScratch& s)
{
    cudaFree(s.nodes);
    cudaFree(s.arrays);
    s = GpuBvhScratch();
}

} // namespace agb
