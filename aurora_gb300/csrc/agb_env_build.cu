// Environment importance-sampling table built on the GPU from FP64 prefix sums.
//
// Replaces the CPU AliasMap::build (AliasMap.cpp:71-166, called from HGI/HGIImage.cpp:45-90
// after a GPU->CPU readback).  Same texel weights (luminance x solid angle of the texel's
// latitude row, luminance weights 0.2125/0.7154/0.0721), same per-texel pdf
// (luminance / integral of luminance over the sphere), and the same entry layout and sampling
// procedure, so Environment.slang:137-186 samples it unchanged.
//
// The table is built in parallel instead of by the reference's sequential sweep.  With the
// normalised weights p_i = N w_i / W, "light" texels (p < 1) and "heavy" texels (p >= 1) in index
// order, deficit prefix sums D (lights, 1 - p) and surplus prefix sums S (heavies, p - 1):
//   light k is aliased to the heavy j whose surplus interval contains D_k (S_j < D_k <= S_{j+1});
//   heavy j is exhausted by the light whose deficit interval crosses S_{j+1}, keeps probability
//   1 + S_{j+1} - D_after and aliases heavy j + 1.
// This is the greedy sweep of Vose's method with the state expressed through prefix sums, so each
// entry is independent: one binary search per texel.  All prefix sums are FP64.
#include <type_traits>

#include "agb_kernels.h"

namespace agb
{

namespace
{

constexpr int kScanThreads = 256;
constexpr int kScanItems   = 4;
constexpr int kScanTile    = kScanThreads * kScanItems;

// Exclusive block scan of one double per thread (fixed summation order); the block total is
// returned through `total`.
__device__ double blockExclusiveScan(double v, double& total)
{
    constexpr int kWarps = kScanThreads / 32;
    __shared__ double warpOffset[kWarps];
    __shared__ double blockTotal;
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1)
    {
        double t = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off)
            incl += t;
    }
    double exw = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0)
        exw = 0.0;
    if (lane == 31)
        warpOffset[warp] = incl;
    __syncthreads();
    if (warp == 0)
    {
        double ws = lane < kWarps ? warpOffset[lane] : 0.0;
        double wi = ws;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1)
        {
            double t = __shfl_up_sync(0xffffffffu, wi, off);
            if (lane >= off)
                wi += t;
        }
        double we = __shfl_up_sync(0xffffffffu, wi, 1);
        if (lane == 0)
            we = 0.0;
        if (lane < kWarps)
            warpOffset[lane] = we;
        if (lane == kWarps - 1)
            blockTotal = wi;
    }
    __syncthreads();
    double excl = warpOffset[warp] + exw;
    total       = blockTotal;
    __syncthreads();
    return excl;
}

// Per texel: luminance (FP32, reference arithmetic) and weight = luminance x solid angle (FP64).
__global__ void k_env_weights(const float4* rgba, uint32_t width, uint32_t height, float* lum,
    double* weight, double* blockSum)
{
    uint32_t n    = width * height;
    uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    double local  = 0.0;
    const double kPiD   = 3.14159265358979323846;
    const double lonInc = 2.0 * kPiD / double(width);
    const double latInc = kPiD / double(height);
    for (int q = 0; q < kScanItems; q++)
    {
        uint32_t i = base + q;
        if (i >= n)
            break;
        float4 c = rgba[i];
        // glm::dot order: (r * 0.2125 + g * 0.7154) + b * 0.0721, no contraction.
        float l = __fadd_rn(__fadd_rn(__fmul_rn(c.x, 0.2125f), __fmul_rn(c.y, 0.7154f)),
            __fmul_rn(c.z, 0.0721f));
        uint32_t y   = i / width;
        double upper = 0.5 * kPiD - double(y) * latInc;
        double sa    = (sin(upper) - sin(upper - latInc)) * lonInc;
        double w     = double(l) * sa;
        lum[i]    = l;
        weight[i] = w;
        local += w;
    }
    double total;
    blockExclusiveScan(local, total);
    if (threadIdx.x == 0)
        blockSum[blockIdx.x] = total;
}

// Single block: exclusive scan over the per-tile values (in place), total to out[count].
__global__ void k_scan_tiles(double* v, uint32_t count, double* totalOut)
{
    double carry = 0.0;
    for (uint32_t b = 0; b < count; b += kScanThreads)
    {
        uint32_t i = b + threadIdx.x;
        double x   = i < count ? v[i] : 0.0;
        double total;
        double e = blockExclusiveScan(x, total);
        if (i < count)
            v[i] = carry + e;
        carry += total;
    }
    if (threadIdx.x == 0 && totalOut)
        *totalOut = carry;
}
__global__ void k_scan_tiles_u32(uint32_t* v, uint32_t count, uint32_t* totalOut)
{
    uint32_t carry = 0;
    for (uint32_t b = 0; b < count; b += kScanThreads)
    {
        uint32_t i = b + threadIdx.x;
        uint32_t x = i < count ? v[i] : 0u;
        double total;
        double e = blockExclusiveScan(double(x), total); // exact: counts are far below 2^53
        if (i < count)
            v[i] = carry + uint32_t(e);
        carry += uint32_t(total);
    }
    if (threadIdx.x == 0 && totalOut)
        *totalOut = carry;
}

// Classifies texels and computes per-tile sums of deficits, surpluses and light counts.
__global__ void k_env_classify(const double* weight, uint32_t n, const double* integral,
    double* p, double* tileDef, double* tileSur, uint32_t* tileLights)
{
    uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    double W      = *integral;
    double def = 0.0, sur = 0.0;
    uint32_t lights = 0;
    for (int q = 0; q < kScanItems; q++)
    {
        uint32_t i = base + q;
        if (i >= n)
            break;
        double pi = W > 0.0 ? weight[i] * double(n) / W : 1.0;
        p[i]      = pi;
        if (pi < 1.0)
        {
            def += 1.0 - pi;
            lights++;
        }
        else
            sur += pi - 1.0;
    }
    double t;
    blockExclusiveScan(def, t);
    if (threadIdx.x == 0)
        tileDef[blockIdx.x] = t;
    blockExclusiveScan(sur, t);
    if (threadIdx.x == 0)
        tileSur[blockIdx.x] = t;
    blockExclusiveScan(double(lights), t);
    if (threadIdx.x == 0)
        tileLights[blockIdx.x] = uint32_t(t);
}

// Element-level exclusive scans with tile offsets; scatters light / heavy prefix arrays.
__global__ void k_env_scatter(const double* p, uint32_t n, const double* tileDef,
    const double* tileSur, const uint32_t* tileLights, uint32_t* rankOut, double* lightIncl,
    double* heavyIncl, uint32_t* heavyIdx)
{
    uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    double pv[kScanItems];
    double def = 0.0, sur = 0.0;
    uint32_t lights = 0;
    for (int q = 0; q < kScanItems; q++)
    {
        uint32_t i = base + q;
        pv[q]      = i < n ? p[i] : 1.0;
        if (i < n)
        {
            if (pv[q] < 1.0)
            {
                def += 1.0 - pv[q];
                lights++;
            }
            else
                sur += pv[q] - 1.0;
        }
    }
    double t;
    double defE = blockExclusiveScan(def, t) + tileDef[blockIdx.x];
    double surE = blockExclusiveScan(sur, t) + tileSur[blockIdx.x];
    uint32_t lightE = uint32_t(blockExclusiveScan(double(lights), t)) + tileLights[blockIdx.x];
    for (int q = 0; q < kScanItems; q++)
    {
        uint32_t i = base + q;
        if (i >= n)
            break;
        if (pv[q] < 1.0)
        {
            defE += 1.0 - pv[q];
            lightIncl[lightE] = defE;
            rankOut[i]        = lightE;
            lightE++;
        }
        else
        {
            uint32_t h = i - lightE;
            surE += pv[q] - 1.0;
            heavyIncl[h] = surE;
            heavyIdx[h]  = i;
            rankOut[i]   = h;
        }
    }
}

// First index in a[0, count) with a[idx] >= x (strict: a[idx] > x), or count.
__device__ uint32_t lowerBound(const double* a, uint32_t count, double x, bool strict)
{
    uint32_t lo = 0, hi = count;
    while (lo < hi)
    {
        uint32_t mid = (lo + hi) >> 1;
        bool go      = strict ? (a[mid] <= x) : (a[mid] < x);
        if (go)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

__global__ void k_env_alias(const double* p, const float* lum, uint32_t n, const double* integral,
    const uint32_t* rank, const double* lightIncl,
    const double* heavyIncl, const uint32_t* heavyIdx, const uint32_t* lightCountPtr,
    agb_alias_entry* out)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    double W        = *integral;
    uint32_t lights = *lightCountPtr;
    uint32_t heavies = n - lights;
    agb_alias_entry e;
    e._padding1 = 0.f;
    e.pdf       = W > 0.0 ? lum[i] / float(W) : 0.f;
    double pi   = p[i];
    if (W <= 0.0 || heavies == 0)
    {
        e.alias = i;
        e.prob  = 1.f;
    }
    else if (pi < 1.0)
    {
        // The deficit consumed before light k is the previous light's inclusive prefix, so light
        // and heavy searches read the same FP64 values.
        uint32_t k = rank[i];
        double Dk  = k == 0 ? 0.0 : lightIncl[k - 1];
        uint32_t j = lowerBound(heavyIncl, heavies, Dk, false);
        j          = j < heavies ? j : heavies - 1;
        e.alias    = heavyIdx[j];
        e.prob     = float(pi);
    }
    else
    {
        uint32_t j = rank[i];
        e.alias    = i;
        e.prob     = 1.f;
        if (j + 1 < heavies)
        {
            double X   = heavyIncl[j];
            uint32_t k = lowerBound(lightIncl, lights, X, true);
            if (k < lights)
            {
                double r = 1.0 + X - lightIncl[k];
                e.prob   = float(r < 0.0 ? 0.0 : r);
                e.alias  = heavyIdx[j + 1];
            }
        }
    }
    out[i] = e;
}

// ---------------------------------------------------------------- reference table layout
// The reference's table (AliasMap.cpp:71-166) rebuilt bit for bit: FP32 luminance x row solid
// angle (row angles from the host, as the reference computes them), FP32 sequential integral, the
// same index map (below-average texels first in index order, the others from the end), and the
// same sequential sweep.

__global__ void k_ref_lum(const float4* rgba, uint32_t width, uint32_t n, const float* rowSA,
    float* lum, float* lumArea)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    float4 c = rgba[i];
    float l  = __fadd_rn(__fadd_rn(__fmul_rn(c.x, 0.2125f), __fmul_rn(c.y, 0.7154f)),
        __fmul_rn(c.z, 0.0721f));
    lum[i]     = l;
    lumArea[i] = __fmul_rn(rowSA[i / width], l);
}

// FP32 sum of v[0, n) in index order, bit for bit as a sequential loop computes it, by one block.
//
// While the running sum stays in one binade its ulp u is fixed and the sum is an integer m of
// [2^23, 2^24) ulps, so adding v = (q + f) u (q whole, 0 <= f < 1) rounds to m + q, to m + q + 1, or,
// at f = 1/2, to the even one of the two: every addend is a map m -> m + a[m & 1], and such maps
// compose into maps of the same kind.  A block scan over kSumPer addends per thread therefore gives
// every thread the sum that the sequential loop would reach before its addends; a chunk is taken as a
// whole while no thread's sum leaves the binade.  The first thread that leaves it (or that holds an
// addend that is negative or not finite) adds its own addends one by one, and the next chunk starts
// behind them in the new binade.  One thread adds one by one, from shared memory, in runs that double
// while that lasts: while the sum is zero, subnormal, infinite or NaN, and after a chunk that such an
// addend stopped early (a chunk takes as long as 1,300 addends of a run).
//
// Bound by the load and scan latency of one block, 3 us per chunk of 8,192 addends and per binade:
// 512 x 256 texels 0.63 ms by the sequential loop (10 cycles an addend), 0.11 ms so.  Where a run is what is left:
// 2048 x 1024 texels of which half, or one in a hundred, are negative 7.7 and 7.6 ms (10.0 by the
// sequential loop; 872 and 68 with every chunk tried), with an infinite one 5.7.  Whole-number
// arithmetic: the same maps from FP64 products took 0.63 ms too (two FP64 lanes' worth per SM).
constexpr int kSumThreads    = 1024;
constexpr int kSumPer        = 8;
constexpr uint32_t kSumFull  = 1u << 24; // one past the binade's last integer
constexpr uint32_t kSumCap   = 1u << 25; // saturation of the maps: any value beyond kSumFull does
constexpr uint32_t kSumRun   = 8192;     // longest one-by-one run
constexpr uint32_t kSumShort = 512;      // a chunk that an addend stops before this many is followed by such a run

struct SumMap
{
    uint32_t a0, a1; // added to an even / odd integer
};
__device__ __forceinline__ SumMap composeSum(SumMap f, SumMap g)
{
    SumMap h;
    h.a0 = min(f.a0 + ((f.a0 & 1u) ? g.a1 : g.a0), kSumCap);
    h.a1 = min(f.a1 + (((f.a1 + 1u) & 1u) ? g.a1 : g.a0), kSumCap);
    return h;
}

__global__ void __launch_bounds__(kSumThreads) k_ref_seq_sum(const float* v, uint32_t n, float* out)
{
    __shared__ SumMap warpMap[kSumThreads / 32];
    __shared__ float run[kSumRun];
    __shared__ float accS;
    __shared__ uint32_t posS;
    __shared__ int firstStop;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    float acc       = 0.f;
    uint32_t pos    = 0;
    uint32_t serial = 64;    // addends of the next one-by-one run
    bool oneByOne   = false; // the last chunk did not get far
    while (pos < n)
    {
        if (oneByOne || !(acc >= 1.17549435e-38f && acc < __int_as_float(0x7f800000)))
        {
            if (acc == 0.f)
            {
                // Zeros leave a zero sum as it is: on to the first addend that is not one (its group of 8).
                uint32_t first = uint32_t(kSumThreads * kSumPer);
#pragma unroll
                for (int k = kSumPer - 1; k >= 0; k--)
                {
                    const uint32_t i = pos + uint32_t(k) * kSumThreads + t;
                    if (i < n && v[i] != 0.f)
                        first = uint32_t(k) * kSumThreads + t;
                }
                if (t == 0)
                    posS = kSumThreads * kSumPer;
                __syncthreads();
                atomicMin(&posS, first);
                __syncthreads();
                pos = min(pos + (posS & ~uint32_t(kSumPer - 1)), n);
                __syncthreads();
                if (pos == n)
                    continue;
            }
            const uint32_t cnt = min(serial, n - pos);
            for (uint32_t k = t; k < cnt; k += kSumThreads)
                run[k] = v[pos + k];
            __syncthreads();
            if (t == 0)
            {
                float s = acc;
#pragma unroll 16
                for (uint32_t k = 0; k < cnt; k++)
                    s = __fadd_rn(s, run[k]);
                accS = s;
            }
            __syncthreads();
            acc = accS;
            pos += cnt;
            serial   = min(serial * 2u, kSumRun);
            oneByOne = false;
            __syncthreads();
            continue;
        }
        const int e        = int(__float_as_uint(acc) >> 23); // biased exponent, 1 .. 254
        const uint32_t m0  = (__float_as_uint(acc) & 0x7fffffu) | 0x800000u;
        const uint32_t at  = pos + uint32_t(t) * kSumPer;
        float x[kSumPer];
        if (at + kSumPer <= n)
        {
            const float4 p = *reinterpret_cast<const float4*>(v + at), q = *reinterpret_cast<const float4*>(v + at + 4);
            x[0] = p.x, x[1] = p.y, x[2] = p.z, x[3] = p.w;
            x[4] = q.x, x[5] = q.y, x[6] = q.z, x[7] = q.w;
        }
        else
#pragma unroll
            for (int k = 0; k < kSumPer; k++)
                x[k] = at + k < n ? v[at + k] : 0.f;
        SumMap mine{ 0u, 0u };
        bool odd = false; // an addend that the maps do not describe
#pragma unroll
        for (int k = 0; k < kSumPer; k++)
        {
            odd             = odd || !(x[k] >= 0.f && x[k] < __int_as_float(0x7f800000));
            // v = M 2^(ev - 150) (M < 2^24) is M / 2^sh ulps of the sum, sh = e - ev.
            const uint32_t bits = __float_as_uint(x[k]);
            const int eb        = int(bits >> 23) & 255;
            const uint32_t M    = (bits & 0x7fffffu) | (eb ? 0x800000u : 0u);
            const int sh        = e - (eb ? eb : 1);
            SumMap g;
            if (sh > 0)
            {
                const int s1        = min(sh, 26); // from 25 on the addend is below half an ulp
                const uint32_t q    = M >> s1;
                const uint32_t rem2 = (M & ((1u << s1) - 1u)) << 1, one = 1u << s1; // 2 f against 1
                g.a0 = q + (rem2 > one ? 1u : (rem2 == one ? (q & 1u) : 0u));
                g.a1 = q + (rem2 > one ? 1u : (rem2 == one ? ((q + 1u) & 1u) : 0u));
            }
            else
                g.a0 = g.a1 = M == 0u ? 0u : (sh < -2 ? kSumCap : min(M << -sh, kSumCap));
            mine = composeSum(mine, g);
        }
        // Inclusive scan of the maps in thread order, then the map before this thread.
        SumMap incl = mine;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1)
        {
            SumMap o{ __shfl_up_sync(0xffffffffu, incl.a0, off), __shfl_up_sync(0xffffffffu, incl.a1, off) };
            if (lane >= off)
                incl = composeSum(o, incl);
        }
        SumMap excl{ __shfl_up_sync(0xffffffffu, incl.a0, 1), __shfl_up_sync(0xffffffffu, incl.a1, 1) };
        if (lane == 0)
            excl = SumMap{ 0u, 0u };
        if (lane == 31)
            warpMap[warp] = incl;
        if (t == 0)
            firstStop = kSumThreads;
        __syncthreads();
        if (warp == 0)
        {
            SumMap w = warpMap[lane];
#pragma unroll
            for (int off = 1; off < 32; off <<= 1)
            {
                SumMap o{ __shfl_up_sync(0xffffffffu, w.a0, off), __shfl_up_sync(0xffffffffu, w.a1, off) };
                if (lane >= off)
                    w = composeSum(o, w);
            }
            SumMap b{ __shfl_up_sync(0xffffffffu, w.a0, 1), __shfl_up_sync(0xffffffffu, w.a1, 1) };
            if (lane == 0)
                b = SumMap{ 0u, 0u };
            warpMap[lane] = b;
        }
        __syncthreads();
        const SumMap before   = composeSum(warpMap[warp], excl);
        const SumMap after    = composeSum(before, mine);
        const uint32_t mStart = m0 + ((m0 & 1u) ? before.a1 : before.a0);
        const uint32_t mEnd   = m0 + ((m0 & 1u) ? after.a1 : after.a0);
        if ((odd || mEnd >= kSumFull) && mStart < kSumFull)
            atomicMin(&firstStop, t);
        __syncthreads();
        // mStart < kSumFull holds for every thread up to the first one that stops.
        const int stop = firstStop;
        if (stop == kSumThreads ? t == kSumThreads - 1 : t == stop)
        {
            const uint32_t m = stop == kSumThreads ? mEnd : mStart;
            float s          = __uint_as_float((uint32_t(e) << 23) | (m & 0x7fffffu));
            if (stop != kSumThreads)
#pragma unroll
                for (int k = 0; k < kSumPer; k++)
                    if (at + k < n)
                        s = __fadd_rn(s, x[k]);
            accS = s;
            // A multiple of 8; bit 0: the chunk stopped at an addend that the maps do not describe.
            posS = pos + uint32_t(stop == kSumThreads ? kSumThreads : stop + 1) * kSumPer + (odd ? 1u : 0u);
        }
        __syncthreads();
        acc               = accS;
        const uint32_t to = posS;
        const bool early  = to - pos < kSumShort;
        oneByOne          = early && (to & 1u);
        serial            = early ? serial : 64;
        pos               = to & ~1u;
        __syncthreads();
    }
    if (t == 0)
        *out = acc;
}

__global__ void k_ref_probs(const float* lum, const float* lumArea, uint32_t n,
    const float* integral, float* prob, float* pdf, uint32_t* tileSmall)
{
    uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    float I       = *integral;
    float average = __fdiv_rn(I, float(n));
    uint32_t smalls = 0;
    for (int q = 0; q < kScanItems; q++)
    {
        uint32_t i = base + q;
        if (i >= n)
            break;
        float pr = __fdiv_rn(lumArea[i], average);
        prob[i]  = pr;
        pdf[i]   = __fdiv_rn(lum[i], I);
        smalls += pr < 1.f ? 1u : 0u;
    }
    double t;
    blockExclusiveScan(double(smalls), t);
    if (threadIdx.x == 0)
        tileSmall[blockIdx.x] = uint32_t(t);
}

// The index map, and in its order the probabilities and (each entry its own) the aliases.
__global__ void k_ref_index(const float* prob, uint32_t n, const uint32_t* tileSmallExcl,
    uint32_t* indexMap, float* posProb, uint32_t* posAlias)
{
    uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t smalls = 0;
    bool isSmall[kScanItems];
    for (int q = 0; q < kScanItems; q++)
    {
        uint32_t i = base + q;
        isSmall[q] = i < n && prob[i] < 1.f;
        smalls += isSmall[q] ? 1u : 0u;
    }
    double t;
    uint32_t before = uint32_t(blockExclusiveScan(double(smalls), t)) + tileSmallExcl[blockIdx.x];
    for (int q = 0; q < kScanItems; q++)
    {
        uint32_t i = base + q;
        if (i >= n)
            break;
        // The k-th large (index order) at position n - 1 - k.
        const uint32_t pos = isSmall[q] ? before++ : n - 1 - (i - before);
        indexMap[pos] = i;
        posProb[pos]  = prob[i];
        posAlias[pos] = pos;
    }
}

// The sweep: for (sml = 0; sml < lrg && lrg < n; sml++) pair indexMap[sml] with indexMap[lrg].
//
// The chain w -= 1 - p is sequential (a large's leftover decides where the next one starts), so its
// latency is the bound: one thread walks it, with everything else taken off its path.  Probabilities
// and aliases are held in position order, so both queues are plain streams: the block stages a window
// of each in shared memory (the smalls as their deficits 1 - p, the larges as their p), the walk only
// subtracts, compares and notes where a large ended and what it was left with, and the block finds each
// small's large from those notes.  w never grows within a large (deficits are >= 0), so the walk tests
// groups of four smalls, or of sixteen while w is far from its end, with one comparison and goes back into
// a group only when the large ends inside it.  Positions in [S, lrg) are larges already exhausted,
// whose probability is final and which follow the smalls as smalls; a window beyond S ends at the lrg it started
// with.
//
// 512 x 256 texels of log-normal(0, 2) radiance with four suns: 16.4 ms with one warp that fetched,
// compared and stored small by small, 2.5 ms with groups of four and a note per small, 0.75 ms so.
__device__ __forceinline__ float subtract4(float w, float4 d)
{
    return __fsub_rn(__fsub_rn(__fsub_rn(__fsub_rn(w, d.x), d.y), d.z), d.w);
}
constexpr int kSweepThreads = 1024;
constexpr int kSweepWin     = 2048; // window of both queues (a multiple of 4)
__global__ void __launch_bounds__(kSweepThreads) k_ref_sweep(float* posProb, uint32_t* posAlias, uint32_t n,
    const uint32_t* smallCount)
{
    __shared__ __align__(16) float def[kSweepWin + 16]; // the walk loads sixteen ahead
    __shared__ float lrgP[kSweepWin + 3]; // the walk reads up to two larges past the window
    __shared__ uint16_t begin[kSweepWin + 1]; // first small of the window that a large takes
    __shared__ uint32_t takenS, endedS;                // smalls consumed, larges ended
    __shared__ float wS;
    const int t      = threadIdx.x;
    const uint32_t S = *smallCount;
    if (S == 0 || S >= n)
        return;
    uint32_t sml = 0, lrg = S;
    float w = posProb[S]; // of the current large
    while (sml < lrg && lrg < n)
    {
        const uint32_t cntS = min(uint32_t(kSweepWin), (sml < S ? S : lrg) - sml);
        const uint32_t cntL = min(uint32_t(kSweepWin), n - lrg);
        for (uint32_t k = t; k < cntS; k += kSweepThreads)
            def[k] = __fsub_rn(1.f, posProb[sml + k]);
        for (uint32_t k = t; k < cntL; k += kSweepThreads)
            lrgP[k] = posProb[lrg + k];
        if (t < 3)
            lrgP[cntL + t] = 0.f;
        __syncthreads();
        if (t == 0)
        {
            uint32_t si = 0, li = 0;
            float next1 = lrgP[1], next2 = lrgP[2];
            auto step = [&](float d, uint32_t at) {
                w                = __fsub_rn(w, d);
                const bool ended = w < 1.f;
                if (ended)
                {
                    lrgP[li]      = w;
                    begin[li + 1] = uint16_t(at + 1);
                }
                w     = ended ? next1 : w;
                next1 = ended ? next2 : next1;
                li += ended ? 1u : 0u;
                if (ended)
                    next2 = lrgP[li + 2];
            };
            while (si + 4 <= cntS && li + 4 <= cntL)
            {
                const float4* dp = reinterpret_cast<const float4*>(def + si);
                // A large with much left takes its smalls sixteen at a time.
                if (w > 18.f && si + 16 <= cntS)
                {
                    float4 d0 = dp[0], d1 = dp[1], d2 = dp[2], d3 = dp[3];
                    const uint32_t from = si;
                    for (;;)
                    {
                        // The next sixteen are loaded while these are subtracted.
                        const float4 n0 = dp[4], n1 = dp[5], n2 = dp[6], n3 = dp[7];
                        const float a = subtract4(subtract4(w, d0), d1);
                        const float b = subtract4(subtract4(a, d2), d3);
                        if (b < 1.f)
                            break;
                        w = b;
                        si += 16;
                        if (!(w > 18.f) || si + 16 > cntS)
                            break;
                        d0 = n0, d1 = n1, d2 = n2, d3 = n3;
                        dp += 4;
                    }
                    if (si != from)
                        continue;
                }
                const float4 d = *dp;
                const float w3 = subtract4(w, d);
                if (!(w3 < 1.f))
                    w = w3;
                else
                {
                    step(d.x, si);
                    step(d.y, si + 1);
                    step(d.z, si + 2);
                    step(d.w, si + 3);
                }
                si += 4;
            }
            while (si < cntS && li < cntL)
            {
                step(def[si], si);
                si++;
            }
            takenS = si;
            endedS = li;
            wS     = w;
        }
        __syncthreads();
        const uint32_t taken = takenS, ended = endedS;
        for (uint32_t k = t; k < taken; k += kSweepThreads)
        {
            // The last large that begins at or before the small.
            uint32_t lo = 0, hi = ended + 1;
            while (hi - lo > 1)
            {
                const uint32_t mid = (lo + hi) >> 1;
                if (begin[mid] <= k)
                    lo = mid;
                else
                    hi = mid;
            }
            posAlias[sml + k] = lrg + lo;
        }
        for (uint32_t k = t; k < ended; k += kSweepThreads)
            posProb[lrg + k] = lrgP[k];
        sml += taken;
        lrg += ended;
        // The large that is current next: carried on, or (the window of larges used up) not yet loaded.
        w = ended < cntL ? wS : (lrg < n ? posProb[lrg] : 0.f);
        __syncthreads();
    }
    if (t == 0 && lrg < n)
        posProb[lrg] = w;
}

__global__ void k_ref_pack(const uint32_t* indexMap, const uint32_t* posAlias, const float* posProb, const float* pdf,
    uint32_t n, agb_alias_entry* out)
{
    uint32_t pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= n)
        return;
    const uint32_t i = indexMap[pos];
    reinterpret_cast<float4*>(out)[i] =
        make_float4(__uint_as_float(indexMap[posAlias[pos]]), posProb[pos], pdf[i], 0.f);
}

} // namespace

void freeEnvScratch(EnvBuildScratch& s)
{
    cudaFree(s.weights); // the first array of the one allocation that holds all
    s = EnvBuildScratch();
}

size_t envScratchTileDoubles(uint32_t texels) { return size_t((texels + kScanTile - 1) / kScanTile) * 3 + 8; }
size_t envScratchTileCounts(uint32_t texels) { return size_t((texels + kScanTile - 1) / kScanTile) + 8; }

cudaError_t buildEnvAlias(const float4* rgba, uint32_t width, uint32_t height, int layout,
    const float* rowSolidAngle, agb_alias_entry* out, double* integralFP64Out,
    float* integralShadingOut, EnvBuildScratch& s, cudaStream_t st)
{
    uint32_t n = width * height;
    if (s.capacity < n || s.rows < height)
    {
        freeEnvScratch(s);
        // One allocation, carved in 256-byte steps; the first array's pointer owns it.
        char* base  = nullptr;
        size_t size = 0;
        EnvBuildScratch t;
        auto take = [&](auto*& p, size_t count) {
            p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + size);
            size += (count * sizeof(*p) + 255) & ~size_t(255);
        };
        auto carve = [&]() {
            size = 0;
            take(t.weights, n);
            take(t.scanA, n);
            take(t.ranks, size_t(n) * 2);
            take(t.heavyIdx, n);
            take(t.heavyIncl, n);
            take(t.lightIncl, n);
            take(t.blockSums, envScratchTileDoubles(n));
            take(t.blockCounts, envScratchTileCounts(n));
            take(t.rowSA, size_t(height) + 4);
        };
        carve();
        const cudaError_t e = cudaMalloc(&base, size);
        if (e != cudaSuccess)
            return e;
        carve();
        t.capacity = n;
        t.rows     = height;
        s          = t;
    }
    return launchEnvAliasBuild(rgba, width, height, layout, rowSolidAngle, out, integralFP64Out,
        integralShadingOut, s, st);
}

cudaError_t launchEnvAliasBuild(const float4* rgba, uint32_t width, uint32_t height, int layout,
    const float* rowSolidAngle, agb_alias_entry* out, double* integralFP64Out,
    float* integralShadingOut, const EnvBuildScratch& s, cudaStream_t st)
{
    uint32_t n       = width * height;
    uint32_t tiles   = (n + kScanTile - 1) / kScanTile;
    float* lum       = reinterpret_cast<float*>(s.ranks + n); // second half of ranks
    double* tileW    = s.blockSums;
    double* tileDef  = s.blockSums + tiles;
    double* tileSur  = s.blockSums + 2 * tiles;
    double* integral = s.blockSums + 3 * tiles;
    uint32_t* lightCount = s.blockCounts + tiles;
    // FP64 luminance integral (always): prefix sums over luminance x solid angle.
    k_env_weights<<<tiles, kScanThreads, 0, st>>>(rgba, width, height, lum, s.weights, tileW);
    k_scan_tiles<<<1, kScanThreads, 0, st>>>(tileW, tiles, integral);
    float* shadingIntegral = reinterpret_cast<float*>(s.blockSums + 3 * tiles + 1);
    if (layout == 1)
    {
        k_env_classify<<<tiles, kScanThreads, 0, st>>>(s.weights, n, integral, s.scanA, tileDef,
            tileSur, s.blockCounts);
        k_scan_tiles<<<1, kScanThreads, 0, st>>>(tileDef, tiles, nullptr);
        k_scan_tiles<<<1, kScanThreads, 0, st>>>(tileSur, tiles, nullptr);
        k_scan_tiles_u32<<<1, kScanThreads, 0, st>>>(s.blockCounts, tiles, lightCount);
        k_env_scatter<<<tiles, kScanThreads, 0, st>>>(s.scanA, n, tileDef, tileSur, s.blockCounts,
            s.ranks, s.lightIncl, s.heavyIncl, s.heavyIdx);
        k_env_alias<<<(n + 255) / 256, 256, 0, st>>>(s.scanA, lum, n, integral, s.ranks,
            s.lightIncl, s.heavyIncl, s.heavyIdx, lightCount, out);
    }
    else
    {
        // Reference layout.  Scratch reuse: lumArea / prob / pdf in the FP64 weight arrays,
        // index map, aliases and position-order probabilities in the FP64 prefix arrays.
        float* lumArea    = reinterpret_cast<float*>(s.scanA);
        float* prob       = reinterpret_cast<float*>(s.scanA) + n;
        float* pdf        = reinterpret_cast<float*>(s.heavyIncl);
        uint32_t* posAlias = reinterpret_cast<uint32_t*>(s.heavyIncl) + n;
        uint32_t* indexMap = reinterpret_cast<uint32_t*>(s.lightIncl);
        float* posProb     = reinterpret_cast<float*>(s.lightIncl) + n;
        uint32_t* smallCount = lightCount;
        if (rowSolidAngle)
        {
            cudaError_t e = cudaMemcpyAsync(s.rowSA, rowSolidAngle, sizeof(float) * height,
                cudaMemcpyHostToDevice, st);
            if (e != cudaSuccess)
                return e;
        }
        k_ref_lum<<<(n + 255) / 256, 256, 0, st>>>(rgba, width, n, s.rowSA, lum, lumArea);
        k_ref_seq_sum<<<1, kSumThreads, 0, st>>>(lumArea, n, shadingIntegral);
        k_ref_probs<<<tiles, kScanThreads, 0, st>>>(lum, lumArea, n, shadingIntegral, prob, pdf,
            s.blockCounts);
        k_scan_tiles_u32<<<1, kScanThreads, 0, st>>>(s.blockCounts, tiles, smallCount);
        k_ref_index<<<tiles, kScanThreads, 0, st>>>(prob, n, s.blockCounts, indexMap, posProb, posAlias);
        k_ref_sweep<<<1, kSweepThreads, 0, st>>>(posProb, posAlias, n, smallCount);
        k_ref_pack<<<(n + 255) / 256, 256, 0, st>>>(indexMap, posAlias, posProb, pdf, n, out);
    }
    cudaError_t e = cudaMemcpyAsync(integralFP64Out, integral, sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess)
        return e;
    if (layout != 1)
    {
        e = cudaMemcpyAsync(integralShadingOut, shadingIntegral, sizeof(float), cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess)
            return e;
    }
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess)
        return e;
    if (layout == 1)
        *integralShadingOut = float(*integralFP64Out);
    return cudaGetLastError();
}

} // namespace agb
