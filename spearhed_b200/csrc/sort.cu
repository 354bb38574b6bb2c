// Device radix sort of (cell key, particle index) pairs and an exclusive scan.
//
// Replaces the reference's region bookkeeping (region AABB update, region-pair
// overlap search with a host-side inclusive scan in the middle of every step:
// spmacc/particles/regions/NeighbourRegions.hpp:140-222, RegionBoundsUpdate.hpp:39-215):
// particles are re-binned every step by a stable LSD radix sort on their cell
// key, with no host round trip.
//
// Layout: one pass per 8-bit digit, tiles of 256 x rounds keys.  A pass is (1) a
// per-tile digit histogram, (2) the tiles' exclusive prefix per digit, (3) a
// stable scatter: every tile ranks its keys per digit in input order (warp
// __match_any_sync ranks, then a per-digit prefix over the warps of the block)
// and writes them at the digit's base plus its tile's prefix.  Keys are read
// coalesced, once per kernel.
//
// A pass is bound by latency and launches, not by its bytes (8 B in, 8 B out per
// key): tiles of a fixed 4096 keys gave 18 k keys 5 blocks (10 us a histogram,
// 12 us a scatter).  rounds follows the key count, rounded down: up to kFewKeys
// keys the key count over 128 tiles (128 to 256 tiles come of it, fewer below 32 k
// keys), above that over four tiles per SM (513 to 1184 tiles until 16 rounds, the
// most a tile takes).  Up to kFewTiles tiles (to 49,152 keys, and from 65,536 to
// kFewKeys) the scatter adds the tiles' counts itself and step (2) needs no launch.
#include "sph_launch.hpp"

namespace sph
{
    namespace
    {
        constexpr int kThreads = 256;
        constexpr uint32_t kMaxRounds = 16;
        constexpr uint32_t kFewTiles = 192;
        constexpr uint32_t kFewKeys = 1u << 17;

        uint32_t tileRounds(uint32_t n)
        {
            uint32_t const tiles = n <= kFewKeys ? 128u : 4u * 148u;
            uint32_t const r = n / (tiles * kThreads);
            return r < 1u ? 1u : (r > kMaxRounds ? kMaxRounds : r);
        }
        uint32_t tileCount(uint32_t n)
        {
            uint32_t const tile = kThreads * tileRounds(n);
            return (n + tile - 1) / tile;
        }

        constexpr int kScanItems = 8;
        constexpr int kScanTile = kThreads * kScanItems;

        //! Digit counts of each tile, at tileHist[digit * ntile + tile], or with few
        //! tiles at tileHist[tile * 256 + digit].  Keys come nearly sorted (the
        //! order of the last step), so a warp's equal digits are counted once.
        __global__ void __launch_bounds__(kThreads) kRadixHist(
            uint32_t const* __restrict__ keys,
            uint32_t n,
            int shift,
            uint32_t rounds,
            uint32_t* __restrict__ tileHist,
            uint32_t ntile,
            bool few)
        {
            __shared__ uint32_t h[256];
            h[threadIdx.x] = 0;
            __syncthreads();
            int const lane = threadIdx.x & 31;
            uint32_t const base = blockIdx.x * uint32_t(kThreads) * rounds;
#pragma unroll 4
            for(uint32_t r = 0; r < rounds; ++r)
            {
                uint32_t const i = base + r * kThreads + threadIdx.x;
                bool const valid = i < n;
                uint32_t const digit = valid ? (keys[i] >> shift) & 255u : 0x100u;
                uint32_t const peers = __match_any_sync(0xffffffffu, digit);
                if(valid && (peers & ((1u << lane) - 1u)) == 0u)
                    atomicAdd(&h[digit], uint32_t(__popc(peers)));
            }
            __syncthreads();
            tileHist[few ? blockIdx.x * 256u + threadIdx.x : threadIdx.x * ntile + blockIdx.x] = h[threadIdx.x];
        }

        //! Exclusive prefix over the tiles of digit blockIdx.x, in place, and the
        //! digit's total.
        __global__ void __launch_bounds__(kThreads)
            kRadixRows(uint32_t* __restrict__ tileHist, uint32_t ntile, uint32_t* __restrict__ totals)
        {
            __shared__ uint32_t warpTot[kThreads / 32];
            int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            uint32_t* const row = tileHist + size_t(blockIdx.x) * ntile;
            uint32_t carry = 0;
            for(uint32_t t0 = 0; t0 < ntile; t0 += kThreads)
            {
                uint32_t const t = t0 + threadIdx.x;
                uint32_t const v = t < ntile ? row[t] : 0u;
                uint32_t incl = v;
#pragma unroll
                for(int d = 1; d < 32; d <<= 1)
                {
                    uint32_t const o = __shfl_up_sync(0xffffffffu, incl, d);
                    if(lane >= d)
                        incl += o;
                }
                if(lane == 31)
                    warpTot[warp] = incl;
                __syncthreads();
                uint32_t before = carry;
#pragma unroll
                for(int w = 0; w < kThreads / 32; ++w)
                {
                    if(w < warp)
                        before += warpTot[w];
                    carry += warpTot[w];
                }
                if(t < ntile)
                    row[t] = before + incl - v;
                __syncthreads();
            }
            if(threadIdx.x == 0)
                totals[blockIdx.x] = carry;
        }

        __global__ void __launch_bounds__(kThreads) kRadixScatter(
            uint32_t const* __restrict__ keysIn,
            uint32_t const* __restrict__ valsIn,
            uint32_t* __restrict__ keysOut,
            uint32_t* __restrict__ valsOut,
            uint32_t n,
            int shift,
            uint32_t rounds,
            uint32_t const* __restrict__ tileHist,
            uint32_t const* __restrict__ totals,
            uint32_t ntile,
            bool few)
        {
            __shared__ uint32_t running[256];
            __shared__ uint32_t warpCnt[kThreads / 32][256];
            int const tid = threadIdx.x;
            int const warp = tid >> 5;
            int const lane = tid & 31;
            {
                // digit tid: the tiles before this one, and all keys of the digit
                uint32_t before = 0, total = 0;
                if(few)
                {
#pragma unroll 8
                    for(uint32_t t = 0; t < ntile; ++t)
                    {
                        uint32_t const v = tileHist[t * 256u + uint32_t(tid)];
                        before += t < blockIdx.x ? v : 0u;
                        total += v;
                    }
                }
                else
                {
                    before = tileHist[size_t(tid) * ntile + blockIdx.x];
                    total = totals[tid];
                }
                uint32_t incl = total;
#pragma unroll
                for(int d = 1; d < 32; d <<= 1)
                {
                    uint32_t const o = __shfl_up_sync(0xffffffffu, incl, d);
                    if(lane >= d)
                        incl += o;
                }
                if(lane == 31)
                    warpCnt[0][warp] = incl;
                __syncthreads();
                uint32_t base = 0;
                for(int w = 0; w < warp; ++w)
                    base += warpCnt[0][w];
                running[tid] = base + incl - total + before;
                __syncthreads();
            }
            uint32_t const lanesBelow = (1u << lane) - 1u;
            uint32_t const base = blockIdx.x * uint32_t(kThreads) * rounds;
            for(uint32_t r = 0; r < rounds; ++r)
            {
                for(int w = 0; w < kThreads / 32; ++w)
                    warpCnt[w][tid] = 0;
                __syncthreads();
                uint32_t const i = base + r * kThreads + uint32_t(tid);
                bool const valid = i < n;
                uint32_t key = 0, val = 0;
                if(valid)
                {
                    key = keysIn[i];
                    val = valsIn[i];
                }
                uint32_t const digit = (key >> shift) & 255u;
                // Invalid lanes get a value no valid lane can have, so they rank alone.
                uint32_t const peers = __match_any_sync(0xffffffffu, valid ? digit : 0x100u + uint32_t(lane));
                uint32_t const rank = __popc(peers & lanesBelow);
                bool const leader = (peers & lanesBelow) == 0u;
                if(valid && leader)
                    warpCnt[warp][digit] = __popc(peers);
                __syncthreads();
                {
                    uint32_t run = running[tid];
#pragma unroll
                    for(int w = 0; w < kThreads / 32; ++w)
                    {
                        uint32_t const c = warpCnt[w][tid];
                        warpCnt[w][tid] = run;
                        run += c;
                    }
                    running[tid] = run;
                }
                __syncthreads();
                if(valid)
                {
                    uint32_t const dst = warpCnt[warp][digit] + rank;
                    keysOut[dst] = key;
                    valsOut[dst] = val;
                }
                __syncthreads();
            }
        }

        //! Block-level exclusive scan of kScanTile items; writes each tile's total.
        __global__ void __launch_bounds__(kThreads) kScanTiles(
            uint32_t const* __restrict__ in,
            uint32_t* __restrict__ out,
            uint32_t m,
            uint32_t* __restrict__ tileSums)
        {
            __shared__ uint32_t warpTot[kThreads / 32];
            int const tid = threadIdx.x;
            int const lane = tid & 31;
            int const warp = tid >> 5;
            uint32_t const base = blockIdx.x * uint32_t(kScanTile) + uint32_t(tid) * kScanItems;
            uint32_t v[kScanItems];
            uint32_t sum = 0;
#pragma unroll
            for(int k = 0; k < kScanItems; ++k)
            {
                uint32_t const i = base + k;
                v[k] = i < m ? in[i] : 0u;
                sum += v[k];
            }
            uint32_t incl = sum;
#pragma unroll
            for(int d = 1; d < 32; d <<= 1)
            {
                uint32_t const o = __shfl_up_sync(0xffffffffu, incl, d);
                if(lane >= d)
                    incl += o;
            }
            if(lane == 31)
                warpTot[warp] = incl;
            __syncthreads();
            uint32_t warpBase = 0, blockTot = 0;
#pragma unroll
            for(int w = 0; w < kThreads / 32; ++w)
            {
                uint32_t const t = warpTot[w];
                if(w < warp)
                    warpBase += t;
                blockTot += t;
            }
            uint32_t run = warpBase + incl - sum;
#pragma unroll
            for(int k = 0; k < kScanItems; ++k)
            {
                uint32_t const i = base + k;
                if(i < m)
                    out[i] = run;
                run += v[k];
            }
            if(tid == 0 && tileSums)
                tileSums[blockIdx.x] = blockTot;
        }

        __global__ void kAddTileBase(uint32_t* __restrict__ out, uint32_t m, uint32_t const* __restrict__ tileBase)
        {
            uint32_t const i = blockIdx.x * blockDim.x + threadIdx.x;
            if(i < m)
                out[i] += tileBase[i / kScanTile];
        }
    } // namespace

    size_t scanScratchWords(uint32_t m)
    {
        size_t words = 0;
        while(m > uint32_t(kScanTile))
        {
            m = (m + kScanTile - 1) / kScanTile;
            words += 2 * size_t(m);
        }
        return words + 2;
    }

    void exclusiveScan(uint32_t const* in, uint32_t* out, uint32_t m, uint32_t* scratch, cudaStream_t s)
    {
        if(m == 0)
            return;
        uint32_t const ntile = (m + kScanTile - 1) / kScanTile;
        if(ntile == 1)
        {
            kScanTiles<<<1, kThreads, 0, s>>>(in, out, m, nullptr);
            countLaunches(1);
            return;
        }
        uint32_t* sums = scratch;
        uint32_t* sumsScanned = scratch + ntile;
        kScanTiles<<<ntile, kThreads, 0, s>>>(in, out, m, sums);
        countLaunches(1);
        exclusiveScan(sums, sumsScanned, ntile, scratch + 2 * size_t(ntile), s);
        kAddTileBase<<<(m + 255) / 256, 256, 0, s>>>(out, m, sumsScanned);
        countLaunches(1);
    }

    size_t radixScratchWords(uint32_t n)
    {
        return size_t(256) * tileCount(n) + 256;
    }

    bool radixSortPairs(
        uint32_t* keysA,
        uint32_t* valsA,
        uint32_t* keysB,
        uint32_t* valsB,
        uint32_t n,
        int bits,
        uint32_t* scratch,
        cudaStream_t s)
    {
        bool inB = false;
        if(n == 0)
            return inB;
        uint32_t const rounds = tileRounds(n), ntile = tileCount(n);
        bool const few = ntile <= kFewTiles;
        uint32_t* tileHist = scratch;
        uint32_t* totals = scratch + size_t(256) * ntile;
        for(int shift = 0; shift < bits; shift += 8)
        {
            uint32_t const* kin = inB ? keysB : keysA;
            uint32_t const* vin = inB ? valsB : valsA;
            uint32_t* kout = inB ? keysA : keysB;
            uint32_t* vout = inB ? valsA : valsB;
            kRadixHist<<<ntile, kThreads, 0, s>>>(kin, n, shift, rounds, tileHist, ntile, few);
            countLaunches(1);
            if(!few)
            {
                kRadixRows<<<256, kThreads, 0, s>>>(tileHist, ntile, totals);
                countLaunches(1);
            }
            kRadixScatter<<<ntile, kThreads, 0, s>>>(
                kin, vin, kout, vout, n, shift, rounds, tileHist, totals, ntile, few);
            countLaunches(1);
            inB = !inB;
        }
        return inB;
    }
} // namespace sph
