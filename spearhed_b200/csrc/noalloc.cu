// sph_density_noalloc: density summation on caller-owned device arrays, with no
// device allocation at all.
//
// Who needs it: code that must not call cudaMalloc/cudaFree while it runs — a
// host framework that owns every byte of device memory through its own pool
// (and would see foreign allocations as leaks or fragmentation), a solver that
// calls in from a phase where allocation would synchronise the device, or a
// plugin inside another program that forbids the CUDA allocator.  The regular
// entry points allocate their buffers inside the context (sph_create /
// sph_set_species / first compute call); this one uses a fixed scratch area
// instead.
//
// Scratch: one file-scope device array of kScratchBytes (32 MiB), present on
// every GPU that loads this library for as long as the process lives.  It holds
// the cell keys and particle indices of the radix sort (two copies each), the
// sort's tile histograms, the cell ranges and the packed positions of the
// sorted particles.  Limits: at most kMaxParticles particles and kMaxCells cells,
// and the layout must fit the array; larger calls return SPH_ERR_INVALID.
//
// Every call shares the one array, and it keeps the previous call's contents:
// everything that must start at zero (the cell ranges) is cleared by each call.
// Calls whose device work overlaps (two host threads, or two streams, without
// ordering between them) race on the array and give wrong results.
//
// Set-up: the first call on each device looks up the array's device address
// with cudaGetSymbolAddress while that device is current; that first call
// should be made before any stream capture begins.  The address is kept for
// the life of the process, so the entry point must not be called on a device
// after cudaDeviceReset() on it (the reset unloads the module that holds the
// array; a later call would write through the stale address).
//
// Inputs are checked on the device as in sph_set_species: a non-finite
// position, or a mass or h that is not finite and positive, returns
// SPH_ERR_NONFINITE; a finite position outside the box returns SPH_ERR_OUTSIDE.
// Those inputs are found by the same launch sequence that computes rho, so
// on either return rho holds values that must not be used.  Every call waits
// for its own work on `stream` before it returns.
#include "pair_common.cuh"

#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>

namespace sph
{
    int recordError(int code, std::string msg); // context.cu: sets sph_last_error_string()
}

namespace
{
    constexpr size_t kScratchBytes = size_t(32) << 20;
    constexpr uint32_t kMaxParticles = 1u << 18;
    constexpr uint32_t kMaxCells = 1u << 18;
    constexpr int kMaxDevices = 64;
    constexpr int kStatus = sph::kStatWords; //!< status words of a call; the bounds checks set kStatCheck

    static __device__ __align__(256) unsigned char g_noallocScratch[kScratchBytes];

    std::mutex g_addrLock;
    void* g_scratchAddr[kMaxDevices] = {};

    int failNoAlloc(int code, std::string msg)
    {
        return sph::recordError(code, std::move(msg));
    }

    //! Device address of the scratch array on the current device (looked up once per device).
    int scratchAddress(int device, void** out)
    {
        std::lock_guard<std::mutex> g(g_addrLock);
        if(!g_scratchAddr[device])
        {
            void* p = nullptr;
            cudaError_t const e = cudaGetSymbolAddress(&p, g_noallocScratch);
            if(e != cudaSuccess || !p)
                return failNoAlloc(SPH_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
            g_scratchAddr[device] = p;
        }
        *out = g_scratchAddr[device];
        return SPH_OK;
    }

    //! Bump allocator over the scratch array (256-byte aligned slices).
    struct Carve
    {
        unsigned char* base;
        size_t used = 0;
        template<typename T>
        T* take(size_t count)
        {
            used = (used + 255) & ~size_t(255);
            T* p = reinterpret_cast<T*>(base + used);
            used += count * sizeof(T);
            return p;
        }
    };

    constexpr int kThreads = 256;
    constexpr int kWarps = 4;

    //! Cell key of every particle (input order); one box, every particle a target.
    //! status[0] counts finite positions outside the box (on every axis,
    //! periodic ones included), status[1] non-finite positions and masses or
    //! smoothing lengths that are not finite and positive.
    __global__ void kKeysInput(
        sph::BoxDev const B,
        uint32_t n,
        double const* __restrict__ x,
        double const* __restrict__ y,
        double const* __restrict__ z,
        double const* __restrict__ m,
        double const* __restrict__ h,
        uint32_t* __restrict__ keys,
        uint32_t* __restrict__ vals,
        uint32_t* __restrict__ status)
    {
        uint32_t const p = blockIdx.x * blockDim.x + threadIdx.x;
        if(p >= n)
            return;
        double const pos[3] = {x[p], y[p], z[p]};
        double const mp = m[p], hp = h[p];
        bool nonfinite = !(isfinite(mp) && mp > 0.0) || !(isfinite(hp) && hp > 0.0);
        bool outside = false;
        for(int a = 0; a < 3; ++a)
        {
            nonfinite = nonfinite || !isfinite(pos[a]);
            outside = outside || pos[a] < B.lo[a] || pos[a] > B.lo[a] + B.L[a];
        }
        if(nonfinite)
            atomicAdd(&status[1], 1u);
        else if(outside)
            atomicAdd(&status[0], 1u);
        int const cx = sph::cellCoord(B, 0, isfinite(pos[0]) ? pos[0] : B.lo[0]);
        int const cy = sph::cellCoord(B, 1, isfinite(pos[1]) ? pos[1] : B.lo[1]);
        int const cz = sph::cellCoord(B, 2, isfinite(pos[2]) ? pos[2] : B.lo[2]);
        keys[p] = 2u * ((uint32_t(cz) * uint32_t(B.n[1]) + uint32_t(cy)) * uint32_t(B.n[0]) + uint32_t(cx));
        vals[p] = p;
    }

    template<typename V4, typename T>
    __global__ void kPackSorted(
        sph::BoxDev const B,
        uint32_t n,
        uint32_t* status,
        uint32_t const* __restrict__ perm,
        double const* __restrict__ x,
        double const* __restrict__ y,
        double const* __restrict__ z,
        double const* __restrict__ m,
        double const* __restrict__ h,
        V4* __restrict__ pm,
        T* __restrict__ hc)
    {
        uint32_t const p = blockIdx.x * blockDim.x + threadIdx.x;
        if(p >= n)
            return;
        uint32_t const q = perm[p];
        if(!sph::checkIndex(q < n, status, sph::kChkPermute))
            return;
        double const pos[3] = {x[q], y[q], z[q]};
        double rel[3];
        for(int a = 0; a < 3; ++a)
        {
            int const ca = sph::cellCoord(B, a, pos[a]);
            rel[a] = __dsub_rn(pos[a], cellOrigin(B, a, ca));
        }
        pm[p] = sph::mk4<V4>(rel[0], rel[1], rel[2], m[q]);
        hc[p] = T(h[q]);
    }

    //! Density with the accumulation inside the cull (no neighbour list): a warp
    //! takes a group of up to kGroup targets of one cell (few particles: smaller
    //! groups, so that more warps share a cell), stages the candidates of the
    //! 27-cell stencil that come within the cull radius of the group's bounding
    //! box into shared memory, shift applied, and each target sums them with
    //! 32 / kGroup or more lanes.  Every staged candidate is evaluated: about one
    //! in three is accepted, and a divergent walk over the accepted ones would cost
    //! more than the rejected evaluations.  A thread per target reading the
    //! stencil from global memory waited for one dependent 16-byte load per
    //! candidate with a third of its lanes.  Whole calls, 40 neighbours each, thread
    //! per target -> staged: 250 k FP32 cubic 490 -> 222 us, FP64 625 -> 304; 6 k
    //! FP32 150 -> 67, FP64 168 -> 73 (the cell sort's share of that included).
    //!
    //! The acceptance rule is the list-based path's (unfused r^2 in x, y, z order
    //! against R^2); the target itself is its candidate at r = 0, which gives the
    //! self term (added by hand where R^2 underflows to zero).  FP32 lanes fold
    //! blocks of 8 candidates by TwoSum; lane sums are added in FP64.  rho is
    //! written in input order.
    constexpr int kWindow = 128; //!< staged candidates per warp

    template<typename T>
    __device__ __forceinline__ T boxDistance(T lo, T hi, T negX)
    {
        return fmax(fmax(sph::addRn(lo, negX), -sph::addRn(hi, negX)), T(0));
    }

    //! r from r^2: correctly rounded in FP32 (this path has no later pass to match).
    __device__ __forceinline__ float distance(float r2)
    {
        return __fsqrt_rn(r2);
    }
    __device__ __forceinline__ double distance(double r2)
    {
        return r2 * sph::invDistance(r2);
    }

    template<int K, typename V4, typename T>
    __global__ void __launch_bounds__(kWarps * 32) kDensityStaged(
        sph::BoxDev const box,
        uint32_t n,
        uint32_t* status,
        sph::Cells cells,
        uint32_t const* __restrict__ perm,
        V4 const* __restrict__ pm,
        T const* __restrict__ hc,
        T R2g,
        uint32_t group,
        int partShift,
        double* __restrict__ rhoOut)
    {
        __shared__ V4 staged[kWarps][kWindow];
        int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        V4* const win = staged[warp];
        uint32_t const items = cells.ncells << partShift;
        for(uint32_t q = blockIdx.x * kWarps + uint32_t(warp); q < items; q += gridDim.x * kWarps)
        {
            uint32_t const cell = q >> partShift;
            uint32_t const tBeg = cells.start[cell] + (q & ((1u << partShift) - 1u)) * group, tEnd = cells.mid[cell];
            if(tBeg >= tEnd || !sph::checkIndex(tEnd <= n, status, sph::kChkTargets))
                continue;
            // lane d < 27: the source range and image shift of stencil slot d
            uint32_t sBeg = 0, cnt = 0;
            T sh[3] = {T(0), T(0), T(0)};
            if(lane < 27)
            {
                uint32_t const n0 = uint32_t(box.n[0]), n1 = uint32_t(box.n[1]);
                int const cc[3] = {int(cell % n0), int((cell / n0) % n1), int(cell / (n0 * n1))};
                int nc[3];
                bool ok = true;
#pragma unroll
                for(int a = 0; a < 3; ++a)
                {
                    int const o = sph::stencilOff(lane, a);
                    nc[a] = cc[a] + o;
                    if(nc[a] < 0 || nc[a] >= box.n[a])
                    {
                        if(box.periodic[a])
                            nc[a] = (nc[a] + box.n[a]) % box.n[a];
                        else
                            ok = false;
                    }
                    sh[a] = T(o) * sph::edgeOf<T>(box, a);
                }
                if(ok)
                {
                    uint32_t const ncell = (uint32_t(nc[2]) * n1 + uint32_t(nc[1])) * n0 + uint32_t(nc[0]);
                    if(sph::checkIndex(ncell < cells.ncells, status, sph::kChkCell))
                    {
                        sBeg = cells.start[ncell];
                        cnt = cells.end[ncell] - sBeg;
                    }
                    if(!sph::checkIndex(sBeg <= n && cnt <= n - sBeg, status, sph::kChkRange))
                        cnt = 0;
                }
            }
            uint32_t pre = cnt;
#pragma unroll
            for(int d = 1; d < 32; d <<= 1)
            {
                uint32_t const o = __shfl_up_sync(0xffffffffu, pre, d);
                if(lane >= d)
                    pre += o;
            }
            uint32_t const total = __shfl_sync(0xffffffffu, pre, 31);
            pre -= cnt;
            for(uint32_t tc = tBeg; tc < tEnd; tc += group << partShift)
            {
                uint32_t const nt = min(group, tEnd - tc);
                int S = 1; // lanes per target
                while(nt * uint32_t(2 * S) <= 32u)
                    S *= 2;
                uint32_t const t = tc + uint32_t(lane) / uint32_t(S);
                int const sub = lane & (S - 1);
                bool const act = t < tc + nt;
                V4 own{};
                T hi = T(1);
                if(act)
                {
                    own = sph::ld4(pm + t);
                    hi = hc[t];
                }
                T bLo[3], bHi[3];
                T const x[3] = {own.x, own.y, own.z};
#pragma unroll
                for(int a = 0; a < 3; ++a)
                {
                    bLo[a] = sph::warpMinT(act ? x[a] : T(1e30f));
                    bHi[a] = sph::warpMaxT(act ? x[a] : T(-1e30f));
                }
                // rounding is monotone, so with the radius widened by 2^-10 the box
                // test passes every candidate that the exact test accepts; the added
                // smallest normal number keeps that so where R^2 is denormal and the
                // factor rounds away
                constexpr T tiny = sizeof(T) == 4 ? T(FLT_MIN) : T(DBL_MIN);
                T const reach = R2g * (T(1) + T(1.0 / 1024.0)) + tiny;
                sph::HConst<T> const hk = sph::hconst<K, T>(hi);
                sph::Acc<T> rho;
                // R^2 rounds to zero: no pair is in reach, and the target's own
                // candidate (r^2 = 0) is not below it either
                if(R2g == T(0) && act && sub == 0)
                    rho.add(own.w * sph::kernelW<K, T>(T(0), hk));
                uint32_t next = 0; // stencil position to stage
                while(next < total)
                {
                    uint32_t m = 0;
                    __syncwarp();
                    while(next < total && m + 32u <= uint32_t(kWindow))
                    {
                        uint32_t const p = next + uint32_t(lane);
                        // the last slot whose prefix is <= p
                        int d = 0;
#pragma unroll
                        for(int step = 16; step >= 1; step >>= 1)
                            if(__shfl_sync(0xffffffffu, pre, d + step) <= p)
                                d += step;
                        uint32_t const j = __shfl_sync(0xffffffffu, sBeg, d) + p - __shfl_sync(0xffffffffu, pre, d);
                        T const sx = __shfl_sync(0xffffffffu, sh[0], d), sy = __shfl_sync(0xffffffffu, sh[1], d),
                                sz = __shfl_sync(0xffffffffu, sh[2], d);
                        bool pass = false;
                        V4 c{};
                        if(p < total && sph::checkIndex(j < n, status, sph::kChkStaged))
                        {
                            c = sph::ld4(pm + j);
                            c.x = -sph::addRn(c.x, sx);
                            c.y = -sph::addRn(c.y, sy);
                            c.z = -sph::addRn(c.z, sz);
                            T const dx = boxDistance(bLo[0], bHi[0], c.x), dy = boxDistance(bLo[1], bHi[1], c.y),
                                    dz = boxDistance(bLo[2], bHi[2], c.z);
                            pass = dx * dx + dy * dy + dz * dz < reach;
                        }
                        uint32_t const passed = __ballot_sync(0xffffffffu, pass);
                        uint32_t const w = m + uint32_t(__popc(passed & ((1u << lane) - 1u)));
                        if(pass && sph::checkIndex(w < uint32_t(kWindow), status, sph::kChkWindow))
                            win[w] = c;
                        m += uint32_t(__popc(passed));
                        next += 32;
                    }
                    __syncwarp();
                    uint32_t k = uint32_t(sub);
                    while(k < m)
                    {
                        for(int b = 0; b < sph::kBlock && k < m; ++b, k += uint32_t(S))
                        {
                            V4 const c = win[k];
                            T const dx = sph::addRn(own.x, c.x), dy = sph::addRn(own.y, c.y), dz = sph::addRn(own.z, c.z);
                            T const r2 = sph::addRn(
                                sph::addRn(sph::mulRn(dx, dx), sph::mulRn(dy, dy)), sph::mulRn(dz, dz));
                            T const w = c.w * sph::kernelW<K, T>(distance(r2), hk);
                            rho.add(r2 < R2g ? w : T(0));
                        }
                        rho.fold();
                    }
                }
                double v = rho.value();
                for(int o = 1; o < S; o <<= 1)
                    v += __shfl_xor_sync(0xffffffffu, v, o);
                if(act && sub == 0)
                {
                    uint32_t const q = perm[t];
                    if(sph::checkIndex(q < n, status, sph::kChkPermute))
                        rhoOut[q] = v;
                }
            }
        }
    }

    template<int K, typename V4, typename T>
    void launchStaged(
        sph::BoxDev const& box,
        uint32_t n,
        uint32_t* status,
        sph::Cells const& cells,
        uint32_t const* perm,
        V4 const* pm,
        T const* hc,
        SphParams const& p,
        double* rho,
        cudaStream_t s)
    {
        // Targets per warp: a cell's, at most 32, halved while the groups would
        // not give each of 16 warps per SM one.
        uint32_t group = 32;
        int partShift = 0;
        while(group > 4 && uint64_t(n) < uint64_t(group) * 148u * 16u)
        {
            group /= 2;
            ++partShift;
        }
        uint32_t blocks = ((cells.ncells << partShift) + kWarps - 1) / kWarps;
        blocks = blocks > 148u * 32u ? 148u * 32u : blocks;
        // the global cull radius only: pair-max calls are refused before any launch
        T const Rg = T(sph::Kern<K>::support) * T(p.h0);
        kDensityStaged<K, V4, T>
            <<<blocks, kWarps * 32, 0, s>>>(box, n, status, cells, perm, pm, hc, T(Rg * Rg), group, partShift, rho);
        sph::countLaunches(1);
    }

    template<typename V4, typename T>
    void launchStagedK(
        sph::BoxDev const& box,
        uint32_t n,
        uint32_t* status,
        sph::Cells const& cells,
        uint32_t const* perm,
        V4 const* pm,
        T const* hc,
        SphParams const& p,
        double* rho,
        cudaStream_t s)
    {
        if(p.kernel == SPH_KERNEL_QUINTIC)
            launchStaged<SPH_KERNEL_QUINTIC>(box, n, status, cells, perm, pm, hc, p, rho, s);
        else if(p.kernel == SPH_KERNEL_WENDLAND_C2)
            launchStaged<SPH_KERNEL_WENDLAND_C2>(box, n, status, cells, perm, pm, hc, p, rho, s);
        else
            launchStaged<SPH_KERNEL_CUBIC>(box, n, status, cells, perm, pm, hc, p, rho, s);
    }
} // namespace

extern "C" {

int sph_density_noalloc(
    SphParams const* params,
    SphBox const* box,
    int64_t n,
    double const* x,
    double const* y,
    double const* z,
    double const* mass,
    double const* h,
    double* rho,
    void* stream)
{
    if(!params || !box || n < 0 || (n > 0 && (!x || !y || !z || !mass || !h || !rho)))
        return failNoAlloc(SPH_ERR_INVALID, "sph_density_noalloc: null argument");
    SphParams const& p = *params;
    if(p.kernel < SPH_KERNEL_CUBIC || p.kernel > SPH_KERNEL_WENDLAND_C2 || !(p.h0 > 0.0)
       || (p.precision != SPH_PREC_FP64 && p.precision != SPH_PREC_FP32_COMP)
       || (p.cull != SPH_CULL_GLOBAL && p.cull != SPH_CULL_PAIR_MAX))
        return failNoAlloc(SPH_ERR_INVALID, "sph_density_noalloc: bad params");
    if(n == 0)
        return SPH_OK;
    if(uint64_t(n) > kMaxParticles)
        return failNoAlloc(
            SPH_ERR_INVALID,
            "sph_density_noalloc: " + std::to_string(n) + " particles exceed the fixed scratch limit of "
                + std::to_string(kMaxParticles));
    if(p.cull == SPH_CULL_PAIR_MAX)
        return failNoAlloc(
            SPH_ERR_UNSUPPORTED,
            "sph_density_noalloc: the global cull radius (SPH_CULL_GLOBAL) is required: the cell size cannot "
            "be derived from device-resident smoothing lengths without a host round trip");
    int device = 0;
    if(cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices)
        return failNoAlloc(SPH_ERR_CUDA, "sph_density_noalloc: no current CUDA device");
    // Cell grid of the box (same rule as the context path: edge >= support * h0).
    int const sup = p.kernel == SPH_KERNEL_QUINTIC ? 3 : 2;
    double const r64 = double(sup) * p.h0, r32 = double(float(sup) * float(p.h0));
    double const rc = (r64 > r32 ? r64 : r32) * (1.0 + 1.0 / 1048576.0);
    sph::BoxDev bd{};
    uint64_t ncells = 1;
    for(int a = 0; a < 3; ++a)
    {
        bd.lo[a] = box->lo[a];
        bd.L[a] = box->hi[a] - box->lo[a];
        if(!(bd.L[a] > 0.0) || !std::isfinite(bd.L[a]))
            return failNoAlloc(SPH_ERR_INVALID, "sph_density_noalloc: empty or non-finite box");
        bd.periodic[a] = box->periodic[a] ? 1 : 0;
        double const nd = std::floor(bd.L[a] / rc);
        bd.n[a] = nd < 1.0 ? 1 : (nd > 1.0e6 ? 1000000 : int32_t(nd));
        bd.edge[a] = bd.L[a] / bd.n[a];
        bd.edgef[a] = float(bd.edge[a]);
        if(bd.periodic[a] && bd.L[a] < rc)
            return failNoAlloc(SPH_ERR_UNSUPPORTED, "sph_density_noalloc: periodic box thinner than the radius");
        ncells *= uint64_t(bd.n[a]);
    }
    if(ncells > kMaxCells)
        return failNoAlloc(
            SPH_ERR_INVALID,
            "sph_density_noalloc: " + std::to_string(ncells) + " cells exceed the fixed scratch limit of "
                + std::to_string(kMaxCells));
    bd.cellBase = 0;
    bd.ncells = uint32_t(ncells);
    void* base = nullptr;
    int st = scratchAddress(device, &base);
    if(st)
        return st;
    uint32_t const nn = uint32_t(n);
    bool const fp64 = p.precision == SPH_PREC_FP64;
    Carve cv{static_cast<unsigned char*>(base)};
    uint32_t* status = cv.take<uint32_t>(kStatus);
    uint32_t* keysA = cv.take<uint32_t>(nn);
    uint32_t* valsA = cv.take<uint32_t>(nn);
    uint32_t* keysB = cv.take<uint32_t>(nn);
    uint32_t* valsB = cv.take<uint32_t>(nn);
    uint32_t* sortScr = cv.take<uint32_t>(sph::radixScratchWords(nn));
    sph::Cells cells{};
    cells.ncells = uint32_t(ncells);
    cells.start = cv.take<uint32_t>(3 * ncells); // one array, see Cells
    cells.mid = cells.start + ncells;
    cells.end = cells.mid + ncells;
    sph::D4* pm64 = nullptr;
    double* hc64 = nullptr;
    float4* pm32 = nullptr;
    float* hc32 = nullptr;
    if(fp64)
    {
        pm64 = cv.take<sph::D4>(nn);
        hc64 = cv.take<double>(nn);
    }
    else
    {
        pm32 = cv.take<float4>(nn);
        hc32 = cv.take<float>(nn);
    }
    if(cv.used > kScratchBytes)
        return failNoAlloc(
            SPH_ERR_INVALID,
            "sph_density_noalloc: needs " + std::to_string(cv.used) + " bytes of scratch, the fixed array holds "
                + std::to_string(kScratchBytes));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // A launch error left pending by earlier, unrelated work on this thread
    // would otherwise be reported as this call's failure: clear it first.
    (void)cudaGetLastError();
    // Everything below is stream-ordered; nothing that must start at zero is
    // assumed to be zero from an earlier call.
    if(cudaMemsetAsync(status, 0, kStatus * sizeof(uint32_t), s) != cudaSuccess)
        return failNoAlloc(SPH_ERR_CUDA, "sph_density_noalloc: stream operation failed");
    auto launched = [](char const* what) -> int
    {
        // launch configuration errors and failed memsets of the launchers
        cudaError_t const e = cudaGetLastError();
        if(e == cudaSuccess)
            return SPH_OK;
        return failNoAlloc(SPH_ERR_CUDA, std::string("sph_density_noalloc: ") + what + ": " + cudaGetErrorString(e));
    };
    unsigned const g = (nn + kThreads - 1) / kThreads;
    kKeysInput<<<g, kThreads, 0, s>>>(bd, nn, x, y, z, mass, h, keysA, valsA, status);
    sph::countLaunches(1);
    if((st = launched("cell keys")))
        return st;
    int bits = 1;
    while((uint64_t(1) << bits) <= ncells * 2)
        ++bits;
    bool const inB = sph::radixSortPairs(keysA, valsA, keysB, valsB, nn, bits, sortScr, s);
    if((st = launched("radix sort")))
        return st;
    uint32_t const* keys = inB ? keysB : keysA;
    uint32_t const* perm = inB ? valsB : valsA;
    sph::DevCtx dc{};
    dc.n = nn;
    dc.cells = cells;
    sph::launchCellRanges(dc, keys, s); // clears start/mid/end, then fills them
    if((st = launched("cell ranges")))
        return st;
    if(fp64)
    {
        kPackSorted<sph::D4, double><<<g, kThreads, 0, s>>>(bd, nn, status, perm, x, y, z, mass, h, pm64, hc64);
        sph::countLaunches(1);
        if((st = launched("packing")))
            return st;
        launchStagedK<sph::D4, double>(bd, nn, status, cells, perm, pm64, hc64, p, rho, s);
    }
    else
    {
        kPackSorted<float4, float><<<g, kThreads, 0, s>>>(bd, nn, status, perm, x, y, z, mass, h, pm32, hc32);
        sph::countLaunches(1);
        if((st = launched("packing")))
            return st;
        launchStagedK<float4, float>(bd, nn, status, cells, perm, pm32, hc32, p, rho, s);
    }
    if((st = launched("density")))
        return st;
    // Bad inputs are only known after the work ran, so the density kernel is
    // told nothing; rho is written but must not be used on an error return.
    uint32_t bad[kStatus] = {};
    cudaError_t e = cudaMemcpyAsync(bad, status, sizeof(bad), cudaMemcpyDeviceToHost, s);
    if(e == cudaSuccess)
        e = cudaStreamSynchronize(s);
    if(e != cudaSuccess)
        return failNoAlloc(SPH_ERR_CUDA, std::string("sph_density_noalloc: ") + cudaGetErrorString(e));
    if(bad[1])
        return failNoAlloc(
            SPH_ERR_NONFINITE,
            "sph_density_noalloc: " + std::to_string(bad[1])
                + " particles with a non-finite position or a mass or h that is not finite and positive");
    if(bad[0])
        return failNoAlloc(
            SPH_ERR_OUTSIDE, "sph_density_noalloc: " + std::to_string(bad[0]) + " particles outside the box");
    if(bad[sph::kStatCheck])
        return failNoAlloc(
            SPH_ERR_STATE,
            "sph_density_noalloc: a device bounds check failed (sites " + std::to_string(bad[sph::kStatCheck])
                + "; the access was skipped and rho is not valid)");
    return SPH_OK;
}
}
