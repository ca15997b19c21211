// The denoiser's 3x3 convolution on the tcgen05 tensor cores: a persistent, warp-specialised
// implicit GEMM fed by TMA tensor copies.
//
// Work unit (tile): R consecutive output rows x 256 consecutive output pixels x N output channels
// of one image, or of several narrow images side by side.  The 256 pixels are split by parity into two MMA tiles of 128 rows: even pixels
// x = 2j and odd pixels x = 2j + 1, j in [j0, j0 + 128).  Every input that a tap of such a tile
// reads is then a run of 128 consecutive entries of a 130-entry "halo row" at offset 0, 1 or 2:
//   - a full-resolution input row is staged as its even-pixel row E and its odd-pixel row O
//     (pairs j0 - 1 .. j0 + 128); taps dx = -1, 0, +1 read O+0, E+1, O+1 for even outputs and
//     E+1, O+1, E+2 for odd outputs;
//   - a nearest-2x-upsampled input (the decoder's in0) is staged at its own half resolution
//     (pixels j0 - 1 .. j0 + 128 of row (y + dy) >> 1), and the same taps read it at offsets
//     0, 1, 1 (even) and 1, 1, 2 (odd): the upsample costs nothing and is never materialised.
// A staged row is one TMA box (16 channels x 130 entries, fewer in a narrow image, 32 bytes per entry) in the K-major
// 32-byte-swizzled layout: the 16-byte halves of entry i sit at 32 i and 32 i + 16, exchanged when
// bit 7 of the address is set.  Both the TMA write and the MMA read apply the swizzle to the shared
// memory address itself, so an A descriptor started 32 bytes per entry of offset later addresses
// the run: every staged byte is a whole 32-byte sector of the source (one request per entry).
//
// Roles (320 threads, one CTA per SM, static round-robin over tiles):
//   warp 0   TMA producer: per 16-channel group, (R + 2) x 2 halo rows (E, O) (or the fewer
//            half-resolution rows of an upsampled input) by cp.async.bulk.tensor
//            with zero fill outside the image, and the group's 9 weight slices (N x 16 each) by
//            one 1D bulk copy, into a ring of `stages` shared-memory stages (full / empty
//            mbarriers);
//   warp 1   MMA issuer: per stage 2 R x 9 tcgen05.mma (M = 128, N, K = 16) into the tile's
//            accumulators in TMEM, double-buffered (2 x 256 columns; four rows of 64 channels take
//            all 512, freed two rows at a time) so that the epilogue of one tile overlaps the MMAs
//            of the next;
//   warps 2-9 epilogue: tcgen05.ld of the accumulators, + bias, optional ReLU, BF16 (and / or FP32)
//            NHWC stores, and optionally the 2x2 average pool of the BF16 outputs (the encoder's
//            downsampling, exactly as a separate pool over the stored values would compute it).
// Every wait is bounded; a wait that runs out sets an error flag and the roles wind down, waiting
// (bounded) for their own copies and MMAs in flight before the TMEM is released.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <mutex>

#include "agb_kernels.h"
#include "agb_tc.cuh"

namespace agb
{

namespace
{

constexpr int kHaloEntries      = 130;               // 128 MMA rows + offsets 0..2
constexpr uint32_t kEntryBytes  = 32;                // 16 channels of one entry
constexpr uint32_t kRowBytes    = 4352;              // a box of 130 entries rounded up to 256 (the swizzle atom)
constexpr int kThreads          = 320; // producer, MMA issuer, 8 epilogue warps
constexpr uint32_t kAccStride   = 256;               // TMEM columns per accumulator buffer
constexpr int kMaxStages        = 4;
constexpr int kMaxGradChannels  = 256;               // channels of a dpre0 output
constexpr size_t kSmemBudget    = 226 * 1024; // of the 227 KB a CTA may have, static shared memory aside

struct ConvTmaArgs
{
    const uint16_t* wpack; // per (channel tile, group): 9 slices (dy, dx) of N x 16, B layout
    const float* bias;     // [Cout] or null
    uint16_t* out;         // [B][H][W][Cout] or null
    float* out32;          // [B][H][W][Cout] or null
    uint16_t* pool;        // [B][H/2][W/2][Cout] or null (2x2 average of the BF16 outputs)
    float4* rad;           // [B][H][W] RGBA radiance or null (the denoiser's output layer)
    const uint16_t* radIn; // [B][H][W][16] features (log1p noisy radiance in channels 0-2)
    int* error;            // set to 1 when a bounded wait runs out
    float* g0;             // data-gradient split (see ConvLaunch)
    float* g1;
    uint16_t* dpre0;
    const uint16_t* act0;
    float* db0;
    int gC0, gUp;
    int B, H, W, Cout, up0, relu;
    int N, nTiles, R, G, G0, stages;
    int tilesX, rowBlocks, numTiles;
    int images, pitch; // images of a tile, staged entries (and MMA rows) from one to the next
    uint32_t stageBytes, aBytes;
};

struct Tile
{
    int nt, j0, y0, b;
};

__device__ __forceinline__ Tile decodeTile(const ConvTmaArgs& a, int t)
{
    Tile q;
    q.nt = t % a.nTiles;
    t /= a.nTiles;
    q.j0 = (t % a.tilesX) * 128;
    t /= a.tilesX;
    q.y0 = (t % a.rowBlocks) * a.R;
    q.b  = t / a.rowBlocks * a.images;
    return q;
}

// Staged half-resolution rows of an upsampled input for output rows y0 .. y0 + R - 1: rows
// (y0 - 1) >> 1 .. (y0 + R) >> 1 (arithmetic shifts: row -1 is outside the image, read as zero).
__device__ __forceinline__ int upRowBase(int y0) { return (y0 - 1) >> 1; }
__device__ __forceinline__ int upRowCount(int y0, int R) { return ((y0 + R) >> 1) - upRowBase(y0) + 1; }

__device__ __forceinline__ bool leaderWait(uint64_t* bar, uint32_t parity, int lane)
{
    int got = 0;
    if (lane == 0)
        got = tc::mbarWait(bar, parity) ? 1 : 0;
    return __shfl_sync(0xffffffffu, got, 0) != 0;
}

// Waits until the grid this one programmatically depends on has completed and its memory is
// visible (returns at once when the launch had no programmatic dependency), then lets the next
// grid in the stream begin its own prologue.
__device__ __forceinline__ void gridDependencyWait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// One 32-byte store (the address 32-byte aligned): a whole sector per lane.
__device__ __forceinline__ void st256(void* p, const uint32_t (&w)[8])
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]),
        "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}

__device__ __forceinline__ float bfv(uint16_t b) { return __uint_as_float(uint32_t(b) << 16); }

// Output rows per tile for N output channels: as many as one TMEM buffer of 256 columns holds
// (2 R N), at most 4 (six rows for 16 channels measured slower: 77 against 66 us for the output
// layer at 1920x1080); see launchConv3x3 for the four-row tiles of 64 channels.
__host__ __device__ constexpr int tileRows(int n) { return n >= 64 ? 2 : 4; }
// Accumulator buffers: two of 256 columns, or one that takes the whole TMEM.
__host__ __device__ constexpr int accBuffers(int n, int r) { return 2 * r * n <= int(kAccStride) ? 2 : 1; }

// The MMAs of one pipeline stage (one 16-channel input group), fully unrolled.  Halo row i (input
// row y0 - 1 + i) feeds output rows r = i - 2 .. i (those inside the tile) through the vertical taps
// dy = i - r; their accumulators are adjacent in TMEM and the weight slices of the three dy are
// stacked (dy = 2, 1, 0), so one MMA per (halo row, parity, dx) covers every output row the halo
// row feeds: N, 2N or 3N accumulator columns at once.  In the first group of a tile an
// accumulator starts its sum (accumulate = 0) with the dx = 0 MMA of halo row r, split off as an
// MMA of its own.  rowsFree(r) is called before the first MMA that writes output rows r and r + 1.
template <int N, int R, bool UP, class RowsFree>
__device__ __forceinline__ void issueStage(uint32_t aAddr, uint32_t bAddr, uint32_t dBase, bool first,
    const RowsFree& rowsFree)
{
    // K-major, 32-byte swizzle: entries of 32 bytes (16 channels), 8-entry atoms 256 bytes apart.
    const uint64_t aDesc0 = tc::smemDescSw32(aAddr, 256);
    const uint64_t bDesc0 = tc::smemDesc(bAddr, tc::kSliceLbo, tc::kSliceSbo);
#pragma unroll
    for (int i = 0; i < R + 2; i++)
    {
        const int rLo   = i - 2 > 0 ? i - 2 : 0;
        const int rHi   = i < R - 1 ? i : R - 1;
        const int count = rHi - rLo + 1;
        if (i % 2 == 0 && i < R)
            rowsFree(i);
#pragma unroll
        for (int par = 0; par < 2; par++)
#pragma unroll
            for (int dx = 0; dx < 3; dx++)
            {
                // Entry offset of the run: 0, 1, 1 (even outputs), 1, 1, 2 (odd outputs).
                const uint32_t shift = par == 0 ? (dx == 0 ? 0u : 1u) : (dx == 2 ? 2u : 1u);
                uint32_t row;
                if (UP)
                    row = uint32_t(((i - 1) >> 1) + 1); // half-resolution row of input row y0 - 1 + i
                else
                {
                    // E for the centre tap of even outputs and the side taps of odd outputs.
                    const int odd = par == 0 ? (dx == 1 ? 0 : 1) : (dx == 1 ? 1 : 0);
                    row           = uint32_t(i * 2 + odd);
                }
                const uint64_t ad = aDesc0 + ((row * kRowBytes + shift * kEntryBytes) >> 4);
                const uint64_t bd =
                    bDesc0 + ((uint32_t(dx) * 3u * N * 32u + uint32_t(2 - (i - rLo)) * N * 32u) >> 4);
                const uint32_t d = dBase + uint32_t((par * R + rLo) * N);
                if (first && dx == 0 && i <= R - 1)
                {
                    if (count > 1)
                        tc::mma(d, ad, bd, tc::idescBf16(128, uint32_t((count - 1) * N)), 1u);
                    tc::mma(d + uint32_t((count - 1) * N), ad, bd + ((uint32_t(count - 1) * N * 32u) >> 4),
                        tc::idescBf16(128, uint32_t(N)), 0u);
                }
                else
                    tc::mma(d, ad, bd, tc::idescBf16(128, uint32_t(count * N)), 1u);
            }
    }
}

// Two 16-byte loads of 16 BF16 values, masked to where they are positive: the ReLU's gradient of f, rounded to
// BF16 pairs.
__device__ __forceinline__ void reluGrad16(const uint16_t* act, const float (&f)[16], uint32_t (&w)[8])
{
    const uint4* ap = reinterpret_cast<const uint4*>(act);
    const uint4 a0 = __ldg(ap), a1 = __ldg(ap + 1);
    const uint32_t y[8] = { a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w };
#pragma unroll
    for (int i = 0; i < 8; i++)
    {
        const float lo = __uint_as_float(y[i] << 16) > 0.f ? f[2 * i] : 0.f;
        const float hi = __uint_as_float(y[i] & 0xFFFF0000u) > 0.f ? f[2 * i + 1] : 0.f;
        const __nv_bfloat162 h2 = __floats2bfloat162_rn(lo, hi);
        w[i]                    = *reinterpret_cast<const uint32_t*>(&h2);
    }
}

__device__ __forceinline__ void addBf16(float (&sum)[16], const uint32_t (&w)[8])
{
#pragma unroll
    for (int i = 0; i < 8; i++)
    {
        sum[2 * i] += __uint_as_float(w[i] << 16);
        sum[2 * i + 1] += __uint_as_float(w[i] & 0xFFFF0000u);
    }
}
__device__ __forceinline__ void stFloat16(float* p, const float (&f)[16])
{
    uint32_t w0[8], w1[8];
#pragma unroll
    for (int i = 0; i < 8; i++)
    {
        w0[i] = __float_as_uint(f[i]);
        w1[i] = __float_as_uint(f[8 + i]);
    }
    st256(p, w0);
    st256(p + 8, w1);
}

// Adds the warp's sums of 16 values per lane to dst[0 .. 16) (shared memory): halves of the values are
// exchanged with the lane across, so 16 shuffles leave every channel's sum in a lane pair.
__device__ __forceinline__ void warpAddChannels(float (&v)[16], float* dst, int lane)
{
#pragma unroll
    for (int n = 8; n >= 1; n >>= 1)
    {
        const int mask  = 2 * n;
        const bool high = (lane & mask) != 0;
#pragma unroll
        for (int k = 0; k < n; k++)
        {
            const float give = high ? v[k] : v[k + n];
            const float keep = high ? v[k + n] : v[k];
            v[k]             = keep + __shfl_xor_sync(0xffffffffu, give, mask);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    if ((lane & 1) == 0)
        atomicAdd(dst + (lane >> 1), v[0]);
}

template <int N, int R, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1) k_conv3x3_tma(const __grid_constant__ CUtensorMap tm0,
    const __grid_constant__ CUtensorMap tm1, const ConvTmaArgs a)
{
    // Two buffers are freed as wholes; one is freed two rows at a time, so that the next tile's MMAs of its
    // first rows overlap the epilogue of the last ones.
    constexpr int kBuffers = accBuffers(N, R);
    constexpr int kFrees   = kBuffers == 2 ? 1 : R / 2; // parts of a buffer that are freed apart
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[kMaxStages], empty[kMaxStages], accFull[kBuffers], accEmpty[kBuffers * kFrees], drain;
    __shared__ uint32_t tmemBase;
    __shared__ float biasGrad[SPLIT ? kMaxGradChannels : 1]; // this CTA's share of db0
    const int tid  = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int S    = a.stages;

    if (SPLIT)
        for (int c = tid; c < kMaxGradChannels; c += kThreads)
            biasGrad[c] = 0.f;
    if (warp == 1)
        tc::tmemAlloc(&tmemBase, 2 * kAccStride);
    if (tid == 0)
    {
        for (int s = 0; s < S; s++)
        {
            tc::mbarInit(&full[s], 1);
            tc::mbarInit(&empty[s], 1);
        }
        for (int i = 0; i < kBuffers; i++)
            tc::mbarInit(&accFull[i], 1);
        for (int i = 0; i < kBuffers * kFrees; i++)
            tc::mbarInit(&accEmpty[i], 8);
        tc::mbarInit(&drain, 1);
        tc::fenceMbarInit();
    }
    tc::fenceBeforeSync();
    __syncthreads();
    tc::fenceAfterSync();
    const uint32_t tmem = tmemBase;
    bool ok             = true;
    // Programmatic dependent launch: the prologue above may overlap the previous kernel's tail;
    // everything below reads or writes memory that kernel may still touch.
    gridDependencyWait();

    if (warp == 0)
    {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0)
        {
            uint32_t it = 0;
            uint32_t lastParity[kMaxStages];
            bool issued[kMaxStages];
            for (int s = 0; s < S; s++)
                issued[s] = false;
            const uint32_t wBytes = 9u * uint32_t(N) * 32u;
            for (int t = blockIdx.x; t < a.numTiles && ok; t += gridDim.x)
            {
                const Tile q = decodeTile(a, t);
                for (int g = 0; g < a.G; g++, it++)
                {
                    const int s        = int(it % uint32_t(S));
                    const uint32_t ph  = (it / uint32_t(S)) & 1u;
                    if (!tc::mbarWait(&empty[s], ph ^ 1u))
                    {
                        ok = false;
                        break;
                    }
                    uint8_t* A      = smem + size_t(s) * a.stageBytes;
                    uint8_t* Bw     = A + a.aBytes;
                    const bool in0  = g < a.G0;
                    const bool up   = in0 && a.up0;
                    const int c     = (in0 ? g : g - a.G0) * 16;
                    const void* map = in0 ? static_cast<const void*>(&tm0) : static_cast<const void*>(&tm1);
                    const int rows  = up ? upRowCount(q.y0, R) : (R + 2) * 2;
                    tc::mbarExpectTx(&full[s], wBytes + uint32_t(rows * a.images * a.pitch) * kEntryBytes);
                    tc::bulkLoad(Bw, a.wpack + (size_t(q.nt) * a.G + g) * 9 * size_t(N) * 16, wBytes, &full[s]);
                    if (up)
                    {
                        const int h0 = upRowBase(q.y0);
                        for (int i = 0; i < rows; i++)
                            tc::tensorLoad4(A + i * kRowBytes, map, c, q.j0 - 1, h0 + i, q.b, &full[s]);
                    }
                    else
                    {
                        for (int i = 0; i < R + 2; i++)
                            for (int p = 0; p < 2; p++)
                                tc::tensorLoad5(A + (i * 2 + p) * kRowBytes, map, c, p,
                                        q.j0 - 1, q.y0 - 1 + i, q.b, &full[s]);
                    }
                    issued[s]     = true;
                    lastParity[s] = ph;
                }
            }
            // Copies still in flight (a consumer that gave up never waited for them) land before
            // the CTA exits.
            for (int s = 0; s < S; s++)
                if (issued[s] && !tc::mbarWait(&full[s], lastParity[s]))
                    ok = false;
        }
        __syncwarp();
    }
    else if (warp == 1)
    {
        // ---------------------------------------------------------------- MMA issuer
        if (lane == 0)
        {
            uint32_t it = 0;
            int k       = 0;
            for (int t = blockIdx.x; t < a.numTiles && ok; t += gridDim.x, k++)
            {
                const int buf      = k % kBuffers;
                const uint32_t aph = uint32_t(k / kBuffers) & 1u;
                if (kFrees == 1)
                {
                    if (!tc::mbarWait(&accEmpty[buf], aph ^ 1u))
                    {
                        ok = false;
                        break;
                    }
                    tc::fenceAfterSync();
                }
                auto rowsFree = [&](int r) {
                    if (!tc::mbarWait(&accEmpty[r / 2], aph ^ 1u))
                        ok = false;
                    tc::fenceAfterSync();
                };
                auto rowsHeld = [](int) {};
                const uint32_t dBase = tmem + uint32_t(buf) * kAccStride;
                for (int g = 0; g < a.G; g++, it++)
                {
                    const int s       = int(it % uint32_t(S));
                    const uint32_t ph = (it / uint32_t(S)) & 1u;
                    if (!tc::mbarWait(&full[s], ph))
                    {
                        ok = false;
                        break;
                    }
                    tc::fenceAfterSync();
                    const uint32_t aAddr = tc::smemAddr(smem + size_t(s) * a.stageBytes);
                    const uint32_t bAddr = aAddr + a.aBytes;
                    if constexpr (kFrees > 1)
                    {
                        if (g == 0)
                        {
                            if (a.up0)
                                issueStage<N, R, true>(aAddr, bAddr, dBase, true, rowsFree);
                            else
                                issueStage<N, R, false>(aAddr, bAddr, dBase, true, rowsFree);
                        }
                        else if (g < a.G0 && a.up0)
                            issueStage<N, R, true>(aAddr, bAddr, dBase, false, rowsHeld);
                        else
                            issueStage<N, R, false>(aAddr, bAddr, dBase, false, rowsHeld);
                    }
                    else if (g < a.G0 && a.up0)
                        issueStage<N, R, true>(aAddr, bAddr, dBase, g == 0, rowsHeld);
                    else
                        issueStage<N, R, false>(aAddr, bAddr, dBase, g == 0, rowsHeld);
                    tc::commit(&empty[s]);
                }
                if (!ok)
                    break;
                tc::commit(&accFull[buf]);
            }
            // Every MMA issued by this thread has completed before the TMEM is released.
            tc::commit(&drain);
            if (!tc::mbarWait(&drain, 0))
                ok = false;
        }
        __syncwarp();
    }
    else
    {
        // ---------------------------------------------------------------- epilogue (warps 2-9)
        // Two warps per TMEM lane quadrant; the tile's work items (a row, or a row pair when
        // pooling, x a 16-channel chunk) alternate between them.
        const int quad     = warp & 3; // TMEM lanes 32 quad .. 32 quad + 31
        const int half     = (warp - 2) >> 2;
        const int m        = quad * 32 + lane;
        const int W2       = a.W >> 1;
        // The data-gradient split is its own instantiation: the forward epilogue keeps its registers.
        constexpr bool split = SPLIT;
        // An item is a row pair x 16 channels: its four accumulators are loaded before one wait,
        // and a pool or an upsample gradient finds its 2x2 blocks in them (R is even).
        constexpr int step = 2;
        const int chunks   = N / 16;
        const int items    = (R / step) * chunks;
        int k              = 0;
        for (int t = blockIdx.x; t < a.numTiles; t += gridDim.x, k++)
        {
            Tile q             = decodeTile(a, t);
            const int buf      = k % kBuffers;
            const uint32_t aph = uint32_t(k / kBuffers) & 1u;
            if (!leaderWait(&accFull[buf], aph, lane))
            {
                ok = false;
                break;
            }
            tc::fenceAfterSync();
            const int j      = q.j0 + m % a.pitch;
            const int image  = m / a.pitch;
            q.b += image;
            const bool colOk     = j < W2 && image < a.images && q.b < a.B;
            const int cb         = q.nt * N;
            const uint32_t tBase = tmem + (uint32_t(quad * 32) << 16) + uint32_t(buf) * kAccStride;
            for (int item = half; item < items; item += 2)
            {
                const int r  = (item / chunks) * step;
                const int c0 = (item % chunks) * 16;
                if (kFrees > 1 && item >= chunks && item - 2 < (item / chunks) * chunks)
                {
                    // This warp's first item of a new row pair: it is done with the one before.
                    tc::fenceBeforeSync();
                    __syncwarp();
                    if (lane == 0)
                        tc::mbarArrive(&accEmpty[item / chunks - 1]);
                }
                // All accumulators of the item (2 or 4) in flight before one wait.
                uint32_t v[4][16];
                // Accumulator (row r, parity p) at columns (p R + r) N.
                tc::tmemLoad16(tBase + uint32_t(r * N + c0), v[0]);
                tc::tmemLoad16(tBase + uint32_t((R + r) * N + c0), v[1]);
                tc::tmemLoad16(tBase + uint32_t((r + 1) * N + c0), v[2]);
                tc::tmemLoad16(tBase + uint32_t((R + r + 1) * N + c0), v[3]);
                tc::tmemWaitLoad();
                float bv[16];
                if (a.bias)
                {
                    const float4* bp = reinterpret_cast<const float4*>(a.bias + cb + c0);
#pragma unroll
                    for (int i = 0; i < 4; i++)
                    {
                        const float4 t4 = __ldg(bp + i);
                        bv[4 * i]       = t4.x;
                        bv[4 * i + 1]   = t4.y;
                        bv[4 * i + 2]   = t4.z;
                        bv[4 * i + 3]   = t4.w;
                    }
                }
                else
                {
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        bv[i] = 0.f;
                }
                float psum[16], gsum[16], bsum[16];
                if (split)
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        bsum[i] = 0.f;
                const int cch   = cb + c0; // output channel of the chunk
                const bool toG0 = split && cch < a.gC0;
#pragma unroll
                for (int acc = 0; acc < 4; acc++)
                {
                    if (acc >= 2 * step)
                        break;
                    const int par = acc & 1;
                    const int y   = q.y0 + r + (acc >> 1);
                    float f[16];
#pragma unroll
                    for (int i = 0; i < 16; i++)
                    {
                        f[i] = __uint_as_float(v[acc][i]) + bv[i];
                        if (a.relu)
                            f[i] = fmaxf(f[i], 0.f);
                    }
                    // BF16 pairs, round to nearest even (low half = the even channel).
                    uint32_t w[8];
#pragma unroll
                    for (int i = 0; i < 8; i++)
                    {
                        const __nv_bfloat162 h2 = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
                        w[i]                    = *reinterpret_cast<const uint32_t*>(&h2);
                    }
                    const bool st   = colOk && y < a.H;
                    const size_t px = (size_t(q.b) * a.H + y) * a.W + 2 * j + par;
                    if (st && a.out)
                        st256(a.out + px * a.Cout + cb + c0, w);
                    if (st && a.out32)
                    {
                        uint32_t w0[8], w1[8];
#pragma unroll
                        for (int i = 0; i < 8; i++)
                        {
                            w0[i] = __float_as_uint(f[i]);
                            w1[i] = __float_as_uint(f[8 + i]);
                        }
                        st256(a.out32 + px * a.Cout + cb + c0, w0);
                        st256(a.out32 + px * a.Cout + cb + c0 + 8, w1);
                    }
                    if (st && a.rad && c0 == 0)
                    {
                        const uint16_t* xin = a.radIn + px * 16;
                        a.rad[px] = make_float4(fmaxf(expm1f(f[0] + bfv(__ldg(xin + 0))), 0.f),
                            fmaxf(expm1f(f[1] + bfv(__ldg(xin + 1))), 0.f), fmaxf(expm1f(f[2] + bfv(__ldg(xin + 2))), 0.f),
                            1.f);
                    }
                    if (split)
                    {
                        if (toG0 && a.gUp)
                        {
                            // 2x2 block sum ((x00 + x01) + x10) + x11, stored below.
#pragma unroll
                            for (int i = 0; i < 16; i++)
                                gsum[i] = acc == 0 ? f[i] : gsum[i] + f[i];
                        }
                        else if (st && toG0 && a.dpre0)
                        {
                            reluGrad16(a.act0 + px * a.gC0 + cch, f, w);
                            st256(a.dpre0 + px * a.gC0 + cch, w);
                            addBf16(bsum, w);
                        }
                        else if (st)
                        {
                            float* g = toG0 ? a.g0 + px * a.gC0 + cch : a.g1 + px * (a.Cout - a.gC0) + (cch - a.gC0);
                            stFloat16(g, f);
                        }
                    }
                    if (a.pool)
                    {
                        // ((x00 + x01) + x10) + x11 over the stored BF16 values.
#pragma unroll
                        for (int i = 0; i < 8; i++)
                        {
                            const float lo = __uint_as_float(w[i] << 16), hi = __uint_as_float(w[i] & 0xFFFF0000u);
                            psum[2 * i]     = acc == 0 ? lo : psum[2 * i] + lo;
                            psum[2 * i + 1] = acc == 0 ? hi : psum[2 * i + 1] + hi;
                        }
                    }
                }
                if (split && toG0 && a.gUp && colOk && q.y0 + r + 1 < a.H)
                {
                    const size_t at = ((size_t(q.b) * (a.H >> 1) + ((q.y0 + r) >> 1)) * W2 + j) * a.gC0 + cch;
                    if (a.dpre0)
                    {
                        uint32_t w[8];
                        reluGrad16(a.act0 + at, gsum, w);
                        st256(a.dpre0 + at, w);
                        addBf16(bsum, w);
                    }
                    else
                        stFloat16(a.g0 + at, gsum);
                }
                if (split && toG0 && a.dpre0)
                    warpAddChannels(bsum, biasGrad + cch, lane);
                if (a.pool && colOk && q.y0 + r + 1 < a.H)
                {
                    uint32_t w[8];
#pragma unroll
                    for (int i = 0; i < 8; i++)
                    {
                        const __nv_bfloat162 h2 = __floats2bfloat162_rn(psum[2 * i] * 0.25f, psum[2 * i + 1] * 0.25f);
                        w[i]                    = *reinterpret_cast<const uint32_t*>(&h2);
                    }
                    const size_t pp = (size_t(q.b) * (a.H >> 1) + ((q.y0 + r) >> 1)) * W2 + j;
                    st256(a.pool + pp * a.Cout + cb + c0, w);
                }
            }
            tc::fenceBeforeSync();
            __syncwarp();
            if (lane == 0)
                tc::mbarArrive(&accEmpty[buf * kFrees + kFrees - 1]);
        }
    }
    tc::fenceBeforeSync();
    __syncthreads();
    tc::fenceAfterSync();
    if (SPLIT && a.dpre0)
        for (int c = tid; c < a.gC0; c += kThreads)
            atomicAdd(a.db0 + c, biasGrad[c]);
    if (warp == 1)
        tc::tmemDealloc(tmem, 2 * kAccStride);
    if (!ok)
        atomicExch(a.error, 1);
}

// ----------------------------------------------------------------------------- weight gradient
// dW[tap][ci][co] += sum over pixels p of X[p + d(tap)][ci] dY[p][co], X = concat(up?(in0), in1):
// a tcgen05 GEMM with M = input channels, N = output channels and K = pixels, both operands
// MN-major (NHWC keeps a pixel's channels contiguous).  A unit of K is 128 output pixels of one
// row (64 pairs), or up to four rows of a narrow image, split by parity as in the forward pass: dY is
// staged as its even and odd entries (64 each), X as even and odd halo rows with two entries more a
// row, so that the horizontal taps are K offsets of 0, 1 or 2 entries into the same staged rows (an
// upsampled source is staged at half resolution, the same row in both slots).  The vertical taps: when
// 3 x Cin <= 128 the M rows are (dy, ci) - the three halo rows' channel groups are stacked at a uniform
// stride, so one MMA covers all nine taps' rows for its horizontal tap - otherwise a work item takes one
// dy and 128 input channels.  Accumulators: the three horizontal taps x N columns in TMEM, one set of
// them or (N <= 80) two, one for each half of the item's rows; their sums go through shared memory and
// are added to dW by bulk reductions of whole rows of N floats.
constexpr uint32_t kWgSlotA    = 2304; // 72 entries of 32 bytes: 1 x 66, 2 x 34 or 4 x 18 (64 pairs, offsets 0..2)
constexpr uint32_t kWgSlotB    = 2048; // 64 entries
constexpr int kWgThreads       = 192;  // producer, MMA issuer, 4 epilogue warps
constexpr int kWgMaxStages     = 6;

struct WgradTmaArgs
{
    float* dw;
    int B, H, W, Cin, Cout, C0, up0;
    int T;               // vertical taps per item: 3 (M = (dy, ci)) or 1 (M = ci)
    int Gci;             // 16-channel groups of X per tap in an item
    int ciTiles, coTiles, N, splits;
    int unitsX, numUnits, unitsPerItem, numItems;
    int rows, rowBlocks; // image rows of a unit, units down an image
    int steps;           // K steps (of 16 pairs) of a unit's row
    int entriesA;        // of a staged row of X: 16 steps + 2
    uint32_t stageBytes, aBytes;
    int stages;
    int* error;
};

// Shared memory of one accumulator row of the epilogue: 16 bytes of padding keep its stores free of conflicts.
template <int N>
constexpr uint32_t kWgRowBytes = uint32_t(N) * 4u + 16u;

// kHalves: the halves of an item may meet inside a unit (of several rows).  A variant of its own: the selects cost the
// other units' issue of short MMAs 1.2 us of 28 (32 to 32 channels at 4 x 256 x 256).
template <int N, bool kHalves>
__global__ void __launch_bounds__(kWgThreads, 1) k_conv_wgrad_tma(const __grid_constant__ CUtensorMap tm0,
    const __grid_constant__ CUtensorMap tm1, const __grid_constant__ CUtensorMap tmDy, const WgradTmaArgs a)
{
    // Where the TMEM holds two sets of the accumulators, an item sums the halves of its rows apart and adds
    // them at the end: the tensor core's FP32 accumulation loses a little with every step, so a sum is
    // kept no longer than half of what one item per SM has to cover.
    constexpr bool kTwoSets = 6 * N <= 512;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[kWgMaxStages], empty[kWgMaxStages], accFull;
    __shared__ uint32_t tmemBase;
    const int tid  = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int S    = a.stages;
    // Item: (dy or all three, ci tile, co tile, unit range).
    int item      = blockIdx.x;
    const int sp  = item % a.splits;
    item /= a.splits;
    const int coT = item % a.coTiles;
    item /= a.coTiles;
    const int ciT  = item % a.ciTiles;
    const int dyIt = item / a.ciTiles; // the item's dy when T == 1
    const int u0   = sp * a.unitsPerItem;
    const int u1   = min(a.numUnits, u0 + a.unitsPerItem);
    // Image rows of a unit (its other rows lie below the image); rows (or whole units) of the item, and how many of
    // them, the first half, go to the first set.
    auto rowsIn         = [&](int u) { return min(a.rows, a.H - (u / a.unitsX) % a.rowBlocks * a.rows); };
    const int itemRows  = !kHalves ? u1 - u0 : u1 - u0 == 1 ? rowsIn(u0) : (u1 - u0) * a.rows;
    const int firstRows = kTwoSets ? (itemRows + 1) / 2 : itemRows;

    if (warp == 1)
        tc::tmemAlloc(&tmemBase, 512);
    if (tid == 0)
    {
        for (int s = 0; s < S; s++)
        {
            tc::mbarInit(&full[s], 1);
            tc::mbarInit(&empty[s], 1);
        }
        tc::mbarInit(&accFull, 1);
        tc::fenceMbarInit();
    }
    tc::fenceBeforeSync();
    __syncthreads();
    tc::fenceAfterSync();
    const uint32_t tmem = tmemBase;
    bool ok             = true;
    // Programmatic dependent launch: the prologue above may overlap the previous kernel's tail;
    // everything below reads or writes memory that kernel may still touch.
    gridDependencyWait();

    if (warp == 0)
    {
        if (lane == 0)
        {
            uint32_t lastParity[kWgMaxStages];
            bool issued[kWgMaxStages];
            for (int s = 0; s < S; s++)
                issued[s] = false;
            const uint32_t bytesA = uint32_t(a.T * a.Gci) * 2u * uint32_t(a.rows * a.entriesA) * 32u;
            const uint32_t bytesB = uint32_t(N / 16) * 2u * uint32_t(a.rows * a.steps) * 16u * 32u;
            uint32_t it = 0;
            for (int u = u0; u < u1; u++, it++)
            {
                const int s       = int(it % uint32_t(S));
                const uint32_t ph = (it / uint32_t(S)) & 1u;
                if (!tc::mbarWait(&empty[s], ph ^ 1u))
                {
                    ok = false;
                    break;
                }
                const int xs = u % a.unitsX;
                const int r  = u / a.unitsX;
                const int y  = (r % a.rowBlocks) * a.rows;
                const int b  = r / a.rowBlocks;
                const int j0 = xs * 64;
                uint8_t* A   = smem + size_t(s) * a.stageBytes;
                uint8_t* Bm  = A + a.aBytes;
                tc::mbarExpectTx(&full[s], bytesA + bytesB);
                // X: slot (parity p, tap row t, group g) at ((p * 8) + t * Gci + g) * kWgSlotA.
                for (int t = 0; t < a.T; t++)
                {
                    const int dy = a.T == 3 ? t : dyIt;
                    const int yi = y + dy - 1;
                    for (int g = 0; g < a.Gci; g++)
                    {
                        const int c = (a.T == 3 ? 0 : ciT * 128) + g * 16;
                        for (int p = 0; p < 2; p++)
                        {
                            uint8_t* dst = A + (p * 8 + t * a.Gci + g) * kWgSlotA;
                            if (c < a.C0 && a.up0)
                                tc::tensorLoad4(dst, &tm0, c, j0 - 1, yi >> 1, b, &full[s]);
                            else if (c < a.C0)
                                tc::tensorLoad5(dst, &tm0, c, p, j0 - 1, yi, b, &full[s]);
                            else
                                tc::tensorLoad5(dst, &tm1, c - a.C0, p, j0 - 1, yi, b, &full[s]);
                        }
                    }
                }
                // dY: slot (parity p, group g) at (p * N / 16 + g) * kWgSlotB.
                for (int g = 0; g < N / 16; g++)
                    for (int p = 0; p < 2; p++)
                        tc::tensorLoad5(Bm + (p * (N / 16) + g) * kWgSlotB, &tmDy, coT * N + g * 16, p, j0, y, b,
                            &full[s]);
                issued[s]     = true;
                lastParity[s] = ph;
            }
            for (int s = 0; s < S; s++)
                if (issued[s] && !tc::mbarWait(&full[s], lastParity[s]))
                    ok = false;
        }
        __syncwarp();
    }
    else if (warp == 1)
    {
        if (lane == 0)
        {
            // MN-major A and B (bits 15, 16), M = 128, N.
            const uint32_t idesc = tc::idescBf16(128, N) | (1u << 15) | (1u << 16);
            // K step k of a unit: its row's staged entries, 16 pairs on (in 16-byte units).
            uint32_t stepA[4];
#pragma unroll
            for (int k = 0; k < 4; k++)
                stepA[k] = uint32_t((k / a.steps) * a.entriesA + (k % a.steps) * 16) * 2u;
            uint32_t it = 0;
            bool second = false;
            for (int u = u0; u < u1; u++, it++)
            {
                // Steps within the image: pairs and rows beyond it are staged as zeros.
                const int pairs  = a.W / 2 - (u % a.unitsX) * 64;
                const int across = min(a.steps, (pairs + 15) / 16);
                const int steps  = across * rowsIn(u);
                // Steps from `turn` on go to the second set.
                const int turn = kHalves ? max(0, firstRows - (u - u0) * a.rows) * a.steps
                    : u - u0 < firstRows ? 4 : 0;
                const int s       = int(it % uint32_t(S));
                const uint32_t ph = (it / uint32_t(S)) & 1u;
                if (!tc::mbarWait(&full[s], ph))
                {
                    ok = false;
                    break;
                }
                tc::fenceAfterSync();
                const uint32_t aAddr  = tc::smemAddr(smem + size_t(s) * a.stageBytes);
                const uint32_t bAddr  = aAddr + a.aBytes;
                // MN-major, 32-byte swizzle: 16-channel atoms a slot apart (leading byte offset), 8-entry
                // atoms 256 bytes apart (stride byte offset).
                const uint64_t aDesc0 = tc::smemDesc(aAddr, kWgSlotA, 256) | (uint64_t(6) << 61);
                const uint64_t bDesc0 = tc::smemDesc(bAddr, kWgSlotB, 256) | (uint64_t(6) << 61);
                // A pair of parities and a horizontal tap: the staged entries that they read.
                auto shiftOf = [](int par, int dx) { return par == 0 ? (dx == 0 ? 0u : 1u) : (dx == 2 ? 2u : 1u); };
                auto oddOf   = [](int par, int dx) { return par == 0 ? (dx == 1 ? 0u : 1u) : (dx == 1 ? 1u : 0u); };
                if (kHalves && turn > 0 && turn < steps)
                {
                    // The halves meet inside the unit.
#pragma unroll 1
                    for (int i = 0; i < 6 * steps; i++)
                    {
                        const int ks = i % steps, dx = i / steps % 3, par = i / steps / 3;
                        tc::mma(tmem + uint32_t(dx * N) + (ks < turn ? 0u : 3u * N),
                            aDesc0 + ((oddOf(par, dx) * 8u * kWgSlotA + shiftOf(par, dx) * 32u) >> 4) +
                                uint32_t((ks / a.steps) * a.entriesA + (ks % a.steps) * 16) * 2u,
                            bDesc0 + ((uint32_t(par) * (N / 16) * kWgSlotB) >> 4) + uint32_t(ks * 32), idesc,
                            par == 0 && (ks == turn || (u == u0 && ks == 0)) ? 0u : 1u);
                    }
                    second = true;
                }
                else
                {
                    const uint32_t acc = tmem + (turn == 0 ? 3u * N : 0u);
                    const bool first   = turn == 0 ? !second : u == u0;
                    second             = turn == 0;
#pragma unroll
                    for (int par = 0; par < 2; par++)
#pragma unroll
                        for (int dx = 0; dx < 3; dx++)
                        {
                            const uint64_t ad = aDesc0 + ((oddOf(par, dx) * 8u * kWgSlotA + shiftOf(par, dx) * 32u) >> 4);
                            const uint64_t bd = bDesc0 + ((uint32_t(par) * (N / 16) * kWgSlotB) >> 4);
#pragma unroll
                            for (int ks = 0; ks < 4; ks++)
                                if (ks < steps)
                                    tc::mma(acc + uint32_t(dx * N), ad + stepA[ks],
                                        bd + ((uint32_t(ks) * 16u * 32u) >> 4), idesc,
                                        (first && par == 0 && ks == 0) ? 0u : 1u);
                        }
                }
                tc::commit(&empty[s]);
            }
            tc::commit(&accFull);
            if (!tc::mbarWait(&accFull, 0))
                ok = false;
        }
        __syncwarp();
    }
    else
    {
        // Epilogue (warps 2-5): TMEM lane m = the M row of this thread.
        const int quad = warp & 3;
        const int m    = quad * 32 + lane;
        if (!leaderWait(&accFull, 0, lane))
            ok = false;
        else if (u1 > u0)
        {
            tc::fenceAfterSync();
            const int rowsPerTap = a.Gci * 16;
            const int t          = m / rowsPerTap;
            const int dy         = a.T == 3 ? t : dyIt;
            const int ci         = (a.T == 3 ? 0 : ciT * 128) + m % rowsPerTap;
            const bool valid     = t < a.T && ci < a.Cin;
            // Each thread's rows (one per horizontal tap) go through shared memory - the stages are free once
            // the MMAs are done - and are added to dW by one bulk reduction each: whole rows of N floats
            // instead of N / 4 16-byte reductions that each touch half a sector.
            uint8_t* const rows = smem + size_t(m) * kWgRowBytes<N>;
            for (int dx = 0; dx < 3; dx++)
            {
                uint8_t* const row = rows + size_t(dx) * 128 * kWgRowBytes<N>;
                for (int c0 = 0; c0 < N; c0 += 16)
                {
                    uint32_t v[16], v2[16];
                    const uint32_t col = tmem + (uint32_t(quad * 32) << 16) + uint32_t(dx * N + c0);
                    tc::tmemLoad16(col, v);
                    if (firstRows < itemRows)
                        tc::tmemLoad16(col + 3u * N, v2);
                    tc::tmemWaitLoad();
                    if (firstRows < itemRows)
#pragma unroll
                        for (int q = 0; q < 16; q++)
                            v[q] = __float_as_uint(__uint_as_float(v[q]) + __uint_as_float(v2[q]));
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        reinterpret_cast<uint4*>(row)[c0 / 4 + q] =
                            make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                }
                tc::fenceProxyAsync();
                if (valid)
                    tc::bulkReduceAdd(a.dw + (size_t(dy * 3 + dx) * a.Cin + ci) * a.Cout + coT * N, row, uint32_t(N) * 4u);
            }
            tc::bulkCommitWait();
        }
    }
    tc::fenceBeforeSync();
    __syncthreads();
    tc::fenceAfterSync();
    if (warp == 1)
        tc::tmemDealloc(tmem, 512);
    if (!ok)
        atomicExch(a.error, 1);
}

// ----------------------------------------------------------------------------- host side

PFN_cuTensorMapEncodeTiled_v12000 encodeTiled()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// Even / odd view of a full-resolution NHWC BF16 tensor: (C, parity, W / 2, H, B), box 16 x 1 x
// entries x rows x images, 32-byte swizzle.
cudaError_t mapPairs(CUtensorMap* m, const uint16_t* base, int B, int H, int W, int C, int entries,
    int rows, int images = 1)
{
    auto enc = encodeTiled();
    if (!enc)
        return cudaErrorNotSupported;
    cuuint64_t dims[5]    = { cuuint64_t(C), 2, cuuint64_t(W / 2), cuuint64_t(H), cuuint64_t(B) };
    cuuint64_t strides[4] = { cuuint64_t(C) * 2, cuuint64_t(C) * 4, cuuint64_t(W) * C * 2, cuuint64_t(H) * W * C * 2 };
    cuuint32_t box[5]     = { 16, 1, cuuint32_t(entries), cuuint32_t(rows), cuuint32_t(images) };
    cuuint32_t es[5]      = { 1, 1, 1, 1, 1 };
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<uint16_t*>(base), dims, strides, box, es,
        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Plain view of a half-resolution NHWC BF16 tensor: (C, W0, H0, B), box 16 x entries x
// images, 32-byte swizzle.
cudaError_t mapRows(CUtensorMap* m, const uint16_t* base, int B, int H0, int W0, int C, int entries,
    int images = 1)
{
    auto enc = encodeTiled();
    if (!enc)
        return cudaErrorNotSupported;
    cuuint64_t dims[4]    = { cuuint64_t(C), cuuint64_t(W0), cuuint64_t(H0), cuuint64_t(B) };
    cuuint64_t strides[3] = { cuuint64_t(C) * 2, cuuint64_t(W0) * C * 2, cuuint64_t(H0) * W0 * C * 2 };
    cuuint32_t box[4]     = { 16, cuuint32_t(entries), 1, cuuint32_t(images) };
    cuuint32_t es[4]      = { 1, 1, 1, 1 };
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<uint16_t*>(base), dims, strides, box, es,
        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Launch with programmatic stream serialisation: the kernel may start while the previous kernel
// in the stream finishes (its prologue overlaps that kernel's last wave).
template <typename... Args, typename... Params>
cudaError_t launchOverlapped(void (*kern)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
    Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim            = dim3(grid);
    cfg.blockDim           = dim3(block);
    cfg.dynamicSmemBytes   = smem;
    cfg.stream             = st;
    cudaLaunchAttribute attr[1];
    attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs                                          = attr;
    cfg.numAttrs                                       = 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

int smCountOf(int dev)
{
    static int counts[64] = {};
    if (dev < 0 || dev >= 64)
        return 148;
    if (counts[dev] == 0)
    {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
            n = 148;
        counts[dev] = n;
    }
    return counts[dev];
}

} // namespace

// Output channels per tile: 64, 32 or 16, the widest that divides cout.  Narrow tiles keep two or
// more output rows per tile (the halo rows are shared between them, the 2x2 pool needs both rows
// of a pair) and move fewer weight bytes per MMA than 128-channel tiles would.
__host__ __device__ int convTileChannels(int cout) { return cout % 64 == 0 ? 64 : cout % 32 == 0 ? 32 : 16; }

cudaError_t launchConv3x3(const ConvLaunch& c, cudaStream_t st)
{
    if (c.W % 2 || (c.up0 && c.H % 2) || (c.pool && c.H % 2))
        return cudaErrorInvalidValue;
    // Outputs are written in 32-byte pieces, the bias read in 16-byte ones.
    if (((reinterpret_cast<uintptr_t>(c.out) | reinterpret_cast<uintptr_t>(c.out32) | reinterpret_cast<uintptr_t>(c.pool)) &
            31u) ||
        (reinterpret_cast<uintptr_t>(c.bias) & 15u))
        return cudaErrorInvalidValue;
    ConvTmaArgs a{};
    a.wpack = c.wpack;
    a.bias  = c.bias;
    a.out   = c.out;
    a.out32 = c.out32;
    a.pool  = c.pool;
    a.rad   = reinterpret_cast<float4*>(c.radiance);
    a.radIn = c.radianceInput;
    a.g0    = c.grad0;
    a.g1    = c.grad1;
    a.gC0   = c.gradC0;
    a.gUp   = c.gradUp;
    a.dpre0 = c.dpre0;
    a.act0  = c.act0;
    a.db0   = c.db0;
    const bool split = c.grad0 || c.grad1 || c.dpre0;
    if (split &&
        (c.gradC0 % 16 || (c.gradUp && c.H % 2) || (c.gradC0 > 0 && !c.grad0 && !c.dpre0) ||
            (c.gradC0 < c.Cout && !c.grad1) || (c.dpre0 && (!c.act0 || !c.db0 || c.gradC0 > kMaxGradChannels)) ||
            ((reinterpret_cast<uintptr_t>(c.grad0) | reinterpret_cast<uintptr_t>(c.grad1) |
                 reinterpret_cast<uintptr_t>(c.dpre0)) & 31u) ||
            (reinterpret_cast<uintptr_t>(c.act0) & 15u)))
        return cudaErrorInvalidValue;
    a.B = c.B, a.H = c.H, a.W = c.W, a.Cout = c.Cout, a.up0 = c.up0, a.relu = c.relu;
    a.N      = convTileChannels(c.Cout);
    a.nTiles = c.Cout / a.N;
    a.G         = (c.C0 + c.C1) / 16;
    a.G0        = c.C0 / 16;
    a.tilesX    = (c.W / 2 + 127) / 128;
    // Images of at most 63 pairs a row share a tile's 128 MMA rows, each with its halo of two entries (rows
    // that start on a halo entry are computed and dropped): four of 16 pairs are 70 rows of one tile where they
    // would be 16 of each of four.  256 to 256 channels at 4 x 32 x 32 are 64 tiles of two rows so, 22 us, and with a
    // tile an image (by the rule below) 128 of four rows, 33 us; the training step on four 256x256 crops 1228 and 1364.
    a.pitch  = std::min(c.W / 2 + 2, kHaloEntries);
    a.images = a.tilesX > 1 ? 1 : std::min(c.B, (128 - c.W / 2) / a.pitch + 1);
    const int groups = (c.B + a.images - 1) / a.images;
    int dev     = 0;
    if (cudaError_t ed = cudaGetDevice(&dev); ed != cudaSuccess)
        return ed;
    const int sms    = smCountOf(dev);
    auto tilesOf     = [&](int rows) { return long(groups) * ((c.H + rows - 1) / rows) * a.tilesX * a.nTiles; };
    a.R              = tileRows(a.N);
    // Four rows of 64 channels take the whole TMEM, so a tile's epilogue holds up the next tile's MMAs in part;
    // but halo rows, weights and MMA operands are read for twice the outputs (414 cycles of MMAs for a 16-channel
    // group instead of 2 x 222).  Worth it from 128 input channels on: 960x540, 128 up + 64 to 64 channels
    // 111.4 us with two rows, 98.7 with four; 1920x1080 inference 948 us with two rows everywhere, 910 with
    // four from 128 input channels, 923 with four from 64.
    if (a.N == 64 && a.G >= 8 && (tilesOf(4) + sms - 1) / sms * 414 <= (tilesOf(2) + sms - 1) / sms * 222)
        a.R = 4;
    a.rowBlocks = (c.H + a.R - 1) / a.R;
    long tiles  = tilesOf(a.R);
    if (tiles >= (1L << 31))
        return cudaErrorInvalidValue;
    a.numTiles   = int(tiles);
    a.aBytes     = uint32_t(a.R + 2) * 2 * kRowBytes;
    a.stageBytes = (a.aBytes + 9u * uint32_t(a.N) * 32u + 1023u) & ~1023u;
    a.stages     = int(std::min<size_t>(kMaxStages, kSmemBudget / a.stageBytes));
    if (a.stages < 2)
        return cudaErrorInvalidValue;
    cudaError_t e0 = tcErrorFlag(&a.error);
    if (e0 != cudaSuccess)
        return e0;
    CUtensorMap m0, m1;
    cudaError_t e = c.up0 ? mapRows(&m0, c.in0, c.B, c.H / 2, c.W / 2, c.C0, a.pitch, a.images)
                           : mapPairs(&m0, c.in0, c.B, c.H, c.W, c.C0, a.pitch, 1, a.images);
    if (e != cudaSuccess)
        return e;
    if (c.C1 > 0)
    {
        if ((e = mapPairs(&m1, c.in1, c.B, c.H, c.W, c.C1, a.pitch, 1, a.images)) != cudaSuccess)
            return e;
    }
    else
        m1 = m0;
    // At least half of the SM's shared memory, so that one CTA (with all 512 TMEM columns) runs
    // per SM.
    const size_t smem = std::max<size_t>(size_t(a.stages) * a.stageBytes, 120 * 1024);
    auto kern = split ? (a.N == 64 ? (a.R == 4 ? k_conv3x3_tma<64, 4, true> : k_conv3x3_tma<64, 2, true>)
                            : a.N == 32 ? k_conv3x3_tma<32, 4, true> : k_conv3x3_tma<16, 4, true>)
                      : (a.N == 64 ? (a.R == 4 ? k_conv3x3_tma<64, 4, false> : k_conv3x3_tma<64, 2, false>)
                            : a.N == 32 ? k_conv3x3_tma<32, 4, false> : k_conv3x3_tma<16, 4, false>);
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem))) != cudaSuccess)
        return e;
    const int grid = int(std::min<long>(tiles, sms));
    return launchOverlapped(kern, unsigned(grid), kThreads, smem, st, m0, m1, a);
}

cudaError_t launchConvWgrad(const ConvLaunch& c, const uint16_t* dy, float* dw, int smCount, cudaStream_t st)
{
    if (c.W % 2 || (c.up0 && c.H % 2) || (reinterpret_cast<uintptr_t>(dw) & 15u))
        return cudaErrorInvalidValue;
    WgradTmaArgs a{};
    a.dw = dw;
    a.B = c.B, a.H = c.H, a.W = c.W, a.Cin = c.C0 + c.C1, a.Cout = c.Cout, a.C0 = c.C0, a.up0 = c.up0;
    a.T       = 3 * a.Cin <= 128 ? 3 : 1;
    a.Gci     = a.T == 3 ? a.Cin / 16 : std::min(8, a.Cin / 16);
    a.ciTiles = a.T == 3 ? 1 : (a.Cin + 127) / 128;
    a.N       = c.Cout <= 128 ? c.Cout : (c.Cout % 128 == 0 ? 128 : 64);
    if (c.Cout % a.N || (a.N != 16 && a.N != 32 && a.N != 48 && a.N != 64 && a.N != 96 && a.N != 128))
        return cudaErrorInvalidValue;
    a.coTiles  = c.Cout / a.N;
    a.unitsX   = (c.W / 2 + 63) / 64;
    a.steps              = std::min(4, (c.W / 2 + 15) / 16);
    const int fixedItems = (a.T == 3 ? 1 : 3) * a.ciTiles * a.coTiles;
    const int sms        = smCount > 0 ? smCount : 148;
    const bool twoSets   = 6 * a.N <= 512;
    // Narrow images: a unit is as many rows as make 64 pairs, and its steps end with its rows (whole units of one row
    // left up to three quarters of the loads and MMAs to padding).  No sum takes more rows than two items per SM
    // of single rows would: the tensor core's FP32 accumulation loses a little with every step.  Longer sums
    // raised the error against 64 bits: 256 to 256 channels at 4 x 32 x 32, one set of accumulators, 1.7e-7 to
    // 2.3e-7; 64 to 64 channels at 1 x 32 x 32, two sets, 1.12e-7 to 1.28e-7 (0.91e-7 so).  An upsampled source,
    // whose staged rows repeat, goes row by row.  Training step on four 256x256 crops 1251 us with single rows
    // where one set is kept, 1232 so.
    const int lines    = c.B * c.H * a.unitsX; // units of one row
    const int twoItems = std::max(1, std::min(lines, (2 * sms + fixedItems - 1) / fixedItems));
    const int each     = (lines + twoItems - 1) / twoItems; // rows of the longest sum
    a.entriesA         = 16 * a.steps + 2;
    auto setRows       = [&](int rows) {
        a.rows      = rows;
        a.rowBlocks = (c.H + rows - 1) / rows;
        a.numUnits  = c.B * a.rowBlocks * a.unitsX;
    };
    // A CTA takes a whole SM.  Two items per SM; where the kernel sums two halves of an item apart, two at most
    // (306 items on 152 SMs take three rounds), or one, if the item is short and its halves are no longer than
    // that: every item pays a prologue, a pipeline fill and its reductions into dW (64 to 64 channels at
    // 4 x 128 x 128, 11 units an item: 20 us against 26), which long items hide.  One sum over a whole
    // item would double the error against 64 bits.
    auto splitsFor = [&](int items) { return std::max(1, std::min(a.numUnits, items / fixedItems)); };
    auto dealt     = [&](int n) { return (a.numUnits + n - 1) / n; }; // the units dealt out in n parts, or in parts of n
    auto onePerSm  = [&]() {
        const int units = dealt(splitsFor(sms));
        return (units * a.rows + 1) / 2 <= each && units <= 32;
    };
    const int maxRows = c.up0 ? 1 : std::min(4 / a.steps, twoSets ? 2 * each : each);
    setRows(maxRows);
    if (twoSets)
    {
        while (!onePerSm() && a.rows > 1)
            setRows(a.rows - 1);
        if (onePerSm())
            a.splits = splitsFor(sms);
        else
        {
            setRows(maxRows);
            a.splits = std::max(splitsFor(2 * sms), dealt(2 * each / a.rows));
        }
    }
    else
        a.splits = dealt(each / a.rows);
    a.unitsPerItem = (a.numUnits + a.splits - 1) / a.splits;
    a.splits       = (a.numUnits + a.unitsPerItem - 1) / a.unitsPerItem;
    a.numItems     = fixedItems * a.splits;
    a.aBytes       = 2u * 8u * kWgSlotA; // all eight M atoms of both parities (unloaded ones unused)
    a.stageBytes   = (a.aBytes + 2u * uint32_t(a.N / 16) * kWgSlotB + 1023u) & ~1023u;
    a.stages       = int(std::min<size_t>(kWgMaxStages, kSmemBudget / a.stageBytes));
    cudaError_t e  = tcErrorFlag(&a.error);
    if (e != cudaSuccess)
        return e;
    CUtensorMap m0, m1, md;
    e = c.up0 ? mapRows(&m0, c.in0, c.B, c.H / 2, c.W / 2, c.C0, a.entriesA)
              : mapPairs(&m0, c.in0, c.B, c.H, c.W, c.C0, a.entriesA, a.rows);
    if (e != cudaSuccess)
        return e;
    if (c.C1 > 0)
    {
        if ((e = mapPairs(&m1, c.in1, c.B, c.H, c.W, c.C1, a.entriesA, a.rows)) != cudaSuccess)
            return e;
    }
    else
        m1 = m0;
    if ((e = mapPairs(&md, dy, c.B, c.H, c.W, c.Cout, 16 * a.steps, a.rows)) != cudaSuccess)
        return e;
    // The stages, or the epilogue's rows (three times 128) in their place.
    const size_t smem = std::max<size_t>(std::max<size_t>(size_t(a.stages) * a.stageBytes, 120 * 1024),
        size_t(3) * 128 * (size_t(a.N) * 4 + 16));
    const bool halves = twoSets && a.rows > 1;
    auto kern = a.N == 128 ? k_conv_wgrad_tma<128, false>
        : a.N == 96        ? k_conv_wgrad_tma<96, false>
        : a.N == 64        ? (halves ? k_conv_wgrad_tma<64, true> : k_conv_wgrad_tma<64, false>)
        : a.N == 48        ? (halves ? k_conv_wgrad_tma<48, true> : k_conv_wgrad_tma<48, false>)
        : a.N == 32        ? (halves ? k_conv_wgrad_tma<32, true> : k_conv_wgrad_tma<32, false>)
                           : (halves ? k_conv_wgrad_tma<16, true> : k_conv_wgrad_tma<16, false>);
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem))) != cudaSuccess)
        return e;
    return launchOverlapped(kern, unsigned(a.numItems), kWgThreads, smem, st, m0, m1, md, a);
}

// Packs FP32 weights w[tap][ci][co] (9 x Cin x Cout) into the conv kernel's B layout (BF16): per
// channel tile and 16-channel input group, for dx = 0, 1, 2 a stack of the three vertical taps'
// slices (dy = 2, 1, 0; N x 16 each) in the K-major core-matrix layout, so that any run of them is
// one B operand.  flip: pack the data-gradient weights instead, w'[tap'][co][ci] =
// w[8 - tap'][ci][co], so that the convolution over dY computes dX (its Cin is then the layer's
// Cout and vice versa).
__global__ void k_pack_conv_weights(const float* w, int Cin, int Cout, int flip, int nt, uint16_t* out)
{
    const int kCin = flip ? Cout : Cin, kCout = flip ? Cin : Cout;
    const long total = 9L * kCin * kCout;
    for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < total; i += long(gridDim.x) * blockDim.x)
    {
        const int n   = int(i % kCout); // kernel output channel
        const long kk = i / kCout;      // tap * kCin + c
        const int tap = int(kk / kCin), c = int(kk % kCin);
        const float v = flip ? w[(size_t(8 - tap) * Cin + n) * Cout + c] : w[(size_t(tap) * Cin + c) * Cout + n];
        const int G = kCin / 16, tile = n / nt, nn = n % nt;
        const int dy = tap / 3, dx = tap % 3;
        const size_t stack = (size_t(tile) * G + c / 16) * 3 + dx;
        const uint32_t row = uint32_t((2 - dy) * nt + nn);
        const size_t off   = stack * 3 * nt * 16 + tc::sliceOffset(row, uint32_t(c % 16)) / 2;
        out[off]           = __bfloat16_as_ushort(__float2bfloat16_rn(v));
    }
}

struct PackJobs
{
    PackJob job[kMaxPackJobs];
    long first[kMaxPackJobs + 1]; // offsets of the jobs' weights, in runs of eight
    int bias[kMaxPackJobs + 1];   // of their biases, which follow all the weights
    int count;
    AdamStep step;
};

// Position of element (tap, c, n) of a kCin x kCout layer in the packed B layout (tiles of nt).
__device__ __forceinline__ size_t packedOffset(int kCin, int nt, int tap, int c, int n)
{
    const int G = kCin / 16, tile = n / nt, nn = n % nt;
    const int dy = tap / 3, dx = tap % 3;
    const size_t stack = (size_t(tile) * G + c / 16) * 3 + dx;
    const uint32_t row = uint32_t((2 - dy) * nt + nn);
    return stack * 3 * nt * 16 + tc::sliceOffset(row, uint32_t(c % 16)) / 2;
}

// Eight floats, 16-byte aligned.
__device__ __forceinline__ void load8(const float* p, float (&f)[8])
{
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w;
    f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
}
__device__ __forceinline__ void store8(float* p, const float (&f)[8])
{
    reinterpret_cast<float4*>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
}
__device__ __forceinline__ void adam8(float* w, const AdamStep& s, float (&f)[8])
{
    const size_t k = size_t(w - s.params);
    float g[8], m[8], v[8];
    load8(s.g + k, g);
    load8(s.m + k, m);
    load8(s.v + k, v);
#pragma unroll
    for (int i = 0; i < 8; i++)
    {
        m[i] = s.b1 * m[i] + (1.f - s.b1) * g[i];
        v[i] = s.b2 * v[i] + (1.f - s.b2) * g[i] * g[i];
        f[i] -= s.lr * (m[i] / s.c1) / (sqrtf(v[i] / s.c2) + s.eps);
    }
    store8(s.m + k, m);
    store8(s.v + k, v);
    store8(w, f);
}
__device__ __forceinline__ uint4 bf16x8(const float (&f)[8])
{
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
    {
        const __nv_bfloat162 h2 = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
        w[i]                    = *reinterpret_cast<const uint32_t*>(&h2);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// A thread takes eight output channels of one (tap, input channel), eight lanes in a row eight input channels:
// a core matrix (8 x 8 values, 128 bytes) of either packed layout.  The data gradient's is the lanes' own
// values; the forward one's is their transpose.  The parameters' update shares the pass over them: an update
// by single floats and a packing by single values were 19.6 and 21.2 us of a training step, this is 23.4 (bound by
// the memory's 60 MB of parameters, gradients and moments, most of them not in the L2 by then).
__global__ void __launch_bounds__(256) k_pack_conv_weights_many(const PackJobs jobs)
{
    const long weights = jobs.first[jobs.count]; // a multiple of 32
    const long i       = blockIdx.x * long(blockDim.x) + threadIdx.x;
    const bool step    = jobs.step.g != nullptr;
    if (i >= weights)
    {
        const long e = i - weights;
        if (!step || e >= jobs.bias[jobs.count])
            return;
        int k = 0;
        while (e >= jobs.bias[k + 1])
            k++;
        const PackJob& J = jobs.job[k];
        float* b         = J.w + 9L * J.cin * J.cout + 8 * (e - jobs.bias[k]);
        float f[8];
        load8(b, f);
        adam8(b, jobs.step, f);
        return;
    }
    int k = 0;
    while (i >= jobs.first[k + 1])
        k++;
    const PackJob& J = jobs.job[k];
    const int lane8  = threadIdx.x & 7;
    const long block = (i - jobs.first[k]) >> 3; // (tap, ci / 8, co / 8)
    const int co     = int(block % (J.cout / 8)) * 8;
    const long kk    = block / (J.cout / 8);
    const int tap = int(kk / (J.cin / 8)), ci = int(kk % (J.cin / 8)) * 8 + lane8;
    float* const w   = J.w + (size_t(tap) * J.cin + ci) * J.cout + co;
    float f[8];
    load8(w, f);
    if (step)
        adam8(w, jobs.step, f);
    if (J.outFlip)
        *reinterpret_cast<uint4*>(J.outFlip + packedOffset(J.cout, convTileChannels(J.cin), 8 - tap, co, ci)) = bf16x8(f);
    // Lane r of the eight: value r of every lane.
#pragma unroll
    for (int n = 4; n >= 1; n >>= 1)
    {
        const bool high = (lane8 & n) != 0;
#pragma unroll
        for (int q = 0; q < 8; q++)
            if ((q & n) == 0)
            {
                const float got = __shfl_xor_sync(0xffffffffu, high ? f[q] : f[q + n], n);
                if (high)
                    f[q] = got;
                else
                    f[q + n] = got;
            }
    }
    if (J.out)
        *reinterpret_cast<uint4*>(
            J.out + packedOffset(J.cin, convTileChannels(J.cout), tap, ci - lane8, co + lane8)) = bf16x8(f);
}

cudaError_t launchPackConvWeightsMany(const PackJob* jobs, int count, const AdamStep& step, cudaStream_t st)
{
    if (count < 0 || count > kMaxPackJobs)
        return cudaErrorInvalidValue;
    PackJobs p{};
    p.count = count;
    p.step  = step;
    for (int k = 0; k < count; k++)
    {
        // Channels in sixteens, so that the runs of a layer fill whole warps.
        if (jobs[k].cin % 16 || jobs[k].cout % 16 || (reinterpret_cast<uintptr_t>(jobs[k].w) & 15u))
            return cudaErrorInvalidValue;
        p.job[k]       = jobs[k];
        p.first[k + 1] = p.first[k] + 9L * jobs[k].cin * jobs[k].cout / 8;
        p.bias[k + 1]  = p.bias[k] + jobs[k].cout / 8;
    }
    const long total = p.first[count] + (step.g ? p.bias[count] : 0);
    if (total == 0)
        return cudaSuccess;
    k_pack_conv_weights_many<<<unsigned((total + 255) / 256), 256, 0, st>>>(p);
    return cudaGetLastError();
}

cudaError_t launchPackConvWeights(const float* w, int Cin, int Cout, int flip, uint16_t* out, cudaStream_t st)
{
    k_pack_conv_weights<<<256, 256, 0, st>>>(w, Cin, Cout, flip, convTileChannels(flip ? Cin : Cout), out);
    return cudaGetLastError();
}


} // namespace agb
