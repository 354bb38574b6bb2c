// Neighbour build: the sorted cells' accepted pairs as list rows.
//
// Replaces the search half of the reference's pair engine (interact() ->
// FrameInteractionKernel, spmacc/particles/algorithms/InteractParticles.hpp:140-199,
// ParticleParticleInteraction.hpp:219-612): candidate staging, the r^2 < R^2
// test and the hand-over of accepted pairs.  The functors it drove run over the
// rows written here (pair_kernels.cu).
//
// One warp per target cell (cell edge >= cull radius).  The warp stages the
// 27-cell stencil's sources into shared memory with the stencil shift already
// added (the reference's origin-shifted staging,
// ParticleParticleInteraction.hpp:241-265); each lane owns one target and
// sweeps the staged candidates with broadcast reads, culling with r^2
// evaluated unfused in x, y, z order exactly as the reference's CPU path does.
// The acceptance masks are then written out one target at a time by the whole
// warp: lane l holds candidate l of a 32-candidate slab and stores its entry
// when the target's mask has bit l, at the row position the bits below it give.
#include "pair_common.cuh"

namespace sph
{
    namespace
    {
        constexpr int kWarps = 4;

        //! Lanes per target for a chunk of nt targets (power of two, nt * S <= 32):
        //! a full chunk gives every lane its own target; a short chunk spreads each
        //! target over S lanes that take consecutive blocks of four candidates.
        __device__ __forceinline__ int subLanes(uint32_t nt)
        {
            return nt > 16 ? 1 : (nt > 8 ? 2 : (nt > 4 ? 4 : (nt > 2 ? 8 : (nt > 1 ? 16 : 32))));
        }

        //! Far coordinate written into the staged tail past the last candidate:
        //! its r^2 overflows (FP32) or dwarfs any cull radius (FP64).
        constexpr float kFar = 1e30f;

        //! Acceptance mask of 32 staged candidates X/Y/Z[0..31] (negated, shifted
        //! source positions) for one target: bit 31-u set when candidate u has
        //! r^2 < R^2.  r^2 is the unfused x, y, z sum of the reference's CPU path;
        //! the test reads the sign of the exactly rounded r^2 - R^2, which is
        //! negative exactly when r^2 < R^2, and funnels it into the mask.
        //! FP32: two candidates per instruction with the paired f32x2 arithmetic
        //! of sm_100 (round-to-nearest per element, the scalar rounding).
        //! UNR: how many of the eight 4-candidate groups the compiler unrolls
        //! (8 = all; 2 keeps the hot code small where warps run several phases
        //! at once and the instruction caches become the bound).
        template<bool PAIRMAX, int UNR>
        __device__ __forceinline__ uint32_t cullMask32(
            float px,
            float py,
            float pz,
            float nRi2,
            float const* X,
            float const* Y,
            float const* Z,
            float const* H,
            float supT,
            float R2g)
        {
            float2 const ox = make_float2(px, px);
            float2 const oy = make_float2(py, py);
            float2 const oz = make_float2(pz, pz);
            float2 const nR2 = make_float2(-R2g, -R2g);
            float2 const zero = opaqueZero2(supT);
            uint32_t mask = 0;
#pragma unroll UNR
            for(int q = 0; q < 32; q += 4)
            {
                float4 const xv = *reinterpret_cast<float4 const*>(X + q);
                float4 const yv = *reinterpret_cast<float4 const*>(Y + q);
                float4 const zv = *reinterpret_cast<float4 const*>(Z + q);
                float4 hv{};
                if constexpr(PAIRMAX)
                    hv = *reinterpret_cast<float4 const*>(H + q);
#pragma unroll
                for(int p = 0; p < 2; ++p)
                {
                    float2 const dx = add2Rn(ox, p ? make_float2(xv.z, xv.w) : make_float2(xv.x, xv.y));
                    float2 const dy = add2Rn(oy, p ? make_float2(yv.z, yv.w) : make_float2(yv.x, yv.y));
                    float2 const dz = add2Rn(oz, p ? make_float2(zv.z, zv.w) : make_float2(zv.x, zv.y));
                    float2 const r2 = add2Rn(add2Rn(sq2Rn(dx, zero), sq2Rn(dy, zero)), sq2Rn(dz, zero));
                    float2 nr = nR2;
                    if constexpr(PAIRMAX)
                    {
                        // -(supT max(h_i, h_j))^2 = min(-(supT h_i)^2, -(supT h_j)^2):
                        // the rounded product and square are monotone in h
                        float const n0 = p ? hv.z : hv.x, n1 = p ? hv.w : hv.y;
                        nr = make_float2(fminf(nRi2, n0), fminf(nRi2, n1));
                    }
                    float2 const d = add2Rn(r2, nr);
                    mask = __funnelshift_l(__float_as_uint(d.x), mask, 1);
                    mask = __funnelshift_l(__float_as_uint(d.y), mask, 1);
                }
            }
            return mask;
        }

        template<bool PAIRMAX, int UNR>
        __device__ __forceinline__ uint32_t cullMask32(
            double px,
            double py,
            double pz,
            double nRi2,
            double const* X,
            double const* Y,
            double const* Z,
            double const* H,
            double supT,
            double R2g)
        {
            uint32_t mask = 0;
#pragma unroll 4
            for(int q = 0; q < 32; q += 2)
            {
                double2 const xv = *reinterpret_cast<double2 const*>(X + q);
                double2 const yv = *reinterpret_cast<double2 const*>(Y + q);
                double2 const zv = *reinterpret_cast<double2 const*>(Z + q);
#pragma unroll
                for(int p = 0; p < 2; ++p)
                {
                    double const dx = __dadd_rn(px, p ? xv.y : xv.x);
                    double const dy = __dadd_rn(py, p ? yv.y : yv.x);
                    double const dz = __dadd_rn(pz, p ? zv.y : zv.x);
                    double const r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
                    double nR2 = -R2g;
                    if constexpr(PAIRMAX)
                        nR2 = fmin(nRi2, H[q + p]);
                    double const d = __dadd_rn(r2, nR2);
                    mask = __funnelshift_l(uint32_t(__double2hiint(d)), mask, 1);
                }
            }
            return mask;
        }

        //! Staged columns are laid out in 32-candidate slabs, each followed by 16
        //! bytes of padding: the sub-lanes of a short chunk read the same offset
        //! of different slabs at once, and the skew puts up to eight such slabs
        //! on different shared-memory banks.  skewed(q) is the column index of
        //! window position q; a slab's 32 candidates stay contiguous.
        __device__ __forceinline__ uint32_t skewed(uint32_t q)
        {
            return q + ((q >> 5) << 2);
        }
        template<int CAP>
        constexpr int colLen()
        {
            return CAP + CAP / 8;
        }

        //! Per-lane state of one chunk of up to 32 targets of a cell.
        template<typename T>
        struct TargetChunk
        {
            T x, y, z;
            T nR2;         //!< -(supT h_i)^2, the target's side of the pair-max cull radius
            uint32_t t;    //!< sorted target index
            uint32_t nl;   //!< entries accepted by this lane
            uint32_t fill; //!< entries in the target's row so far (same on every lane of the target)
            int S, sub;
            bool act;
        };

        template<typename V4, typename T>
        __device__ __forceinline__ void initChunk(
            TargetChunk<T>& ch,
            Records<V4, T> const& rec,
            uint32_t tc,
            uint32_t nt,
            int lane,
            T supT)
        {
            ch.S = subLanes(nt == 0 ? 32u : nt);
            ch.sub = lane & (ch.S - 1);
            uint32_t const tt = uint32_t(lane) / uint32_t(ch.S);
            ch.act = tt < nt;
            ch.t = tc + tt;
            ch.nl = 0;
            ch.fill = 0;
            V4 own{};
            T hi = T(1);
            if(ch.act)
            {
                own = ld4(rec.pm + ch.t);
                hi = rec.hc[ch.t];
            }
            ch.x = own.x;
            ch.y = own.y;
            ch.z = own.z;
            T const Ri = mulRn(supT, hi);
            ch.nR2 = -mulRn(Ri, Ri);
        }

        //! One target's share of a slab during the write-out: x its mask, bit l for
        //! lane l's candidate; then, FP32 (interleaved rows): y one before the slab's
        //! first place in the row, z the row's start; FP64: y the two added up.
        template<typename T>
        struct RowRef;
        template<>
        struct RowRef<float>
        {
            using Type = uint4;
            static __device__ __forceinline__ uint4 make(uint32_t bits, uint32_t row, uint32_t k)
            {
                return make_uint4(bits, k - 1u, row, 0u);
            }
            static __device__ __forceinline__ uint32_t place(uint4 r, uint32_t below)
            {
                return r.z + rowPlace<float>(r.y + below);
            }
        };
        template<>
        struct RowRef<double>
        {
            using Type = uint2;
            static __device__ __forceinline__ uint2 make(uint32_t bits, uint32_t row, uint32_t k)
            {
                return make_uint2(bits, row + k - 1u);
            }
            static __device__ __forceinline__ uint32_t place(uint2 r, uint32_t below)
            {
                return r.y + below;
            }
        };

        //! Stores a candidate's entry into one target's row when the target
        //! accepts it; up = 31 - lane.  The mask's bits up to the lane's own are
        //! moved to the top: the sign is its own bit, the population its place.
        //! The store is predicated (a branch around it would add the warp's
        //! divergence bookkeeping to every target).  room: words of the lists from
        //! rows on (bounds-checked builds).
        template<typename T>
        __device__ __forceinline__ void storeEntry(
            typename RowRef<T>::Type r,
            uint32_t up,
            uint32_t* rows,
            uint32_t ent,
            size_t room,
            uint32_t* status)
        {
            uint32_t const b = r.x << up;
            uint32_t const place = RowRef<T>::place(r, uint32_t(__popc(b)));
            if(!checkIndex(int32_t(b) >= 0 || place < room, status, kChkRowStore))
                return;
            asm volatile("{ .reg .pred q; setp.lt.s32 q, %0, 0; @q st.global.u32 [%1], %2; }"
                         :
                         : "r"(b), "l"(rows + place), "r"(ent)
                         : "memory");
        }

        //! Culls the staged candidates [0, m) against one target chunk (nt targets
        //! from tc) and appends the accepted entries, in candidate order, to each
        //! target's row.  The staging holds negated shifted positions, so
        //! dx = x_i + (-x_j) is the reference's x_i - x_j, rounding included; the
        //! window is far-padded to whole 32-candidate slabs.
        //!
        //! A target has S lanes (S = 1 for a full chunk); in round r sub-lane s
        //! builds the acceptance mask of slab r S + s and clears the bit of the
        //! target's own entry (its window position, recorded at staging).
        //!
        //! Write-out: a lane that walks its own mask runs as long as the busiest
        //! lane of each slab (25 trips for 8 entries on the Orszag-Tang lattice)
        //! and scatters 4-byte stores over 32 rows.  Here the slab's 32 entries
        //! stay in one register per lane and the warp visits the targets in turn,
        //! so a target costs the same few instructions however many entries it
        //! accepts and its entries leave in one contiguous store.
        template<typename T, bool PAIRMAX, int UNR>
        __device__ __forceinline__ void cullChunk(
            TargetChunk<T>& ch,
            T const* sNX,
            T const* sNY,
            T const* sNZ,
            T const* sH,
            uint32_t const* sEnt,
            uint32_t const* sSelf,
            typename RowRef<T>::Type* sRow,
            uint32_t tc,
            uint32_t nt,
            uint32_t m,
            T supT,
            T R2g,
            uint32_t* rows,
            size_t room,
            uint32_t* status,
            uint32_t cap,
            int lane,
            bool countOnly)
        {
            int const S = ch.S;
            uint32_t const selfq = ch.act ? sSelf[ch.t - tc] : ~0u;
            uint32_t const nSlab = (m + 31u) >> 5;
            uint32_t const rowOff = rowStart<T>(ch.t, cap) - rowStart<T>(tc & ~3u, cap);
            uint32_t const up = 31u - uint32_t(lane);
            for(uint32_t g0 = 0; g0 < nSlab; g0 += uint32_t(S))
            {
                uint32_t const g = g0 + uint32_t(ch.sub);
                uint32_t const q0 = g << 5;
                uint32_t mask = 0;
                if(g < nSlab)
                {
                    uint32_t const c0 = skewed(q0);
                    mask = cullMask32<PAIRMAX, UNR>(
                        ch.x, ch.y, ch.z, ch.nR2, sNX + c0, sNY + c0, sNZ + c0, sH + c0, supT, R2g);
                    if(!ch.act)
                        mask = 0;
                    if(selfq - q0 < 32u)
                        mask &= ~(0x80000000u >> (selfq - q0));
                }
                uint32_t const cnt = uint32_t(__popc(mask));
                ch.nl += cnt;
                if(countOnly)
                    continue;
                // row position of this lane's slab: an exclusive scan of the
                // accepted counts over the target's S lanes (candidate order)
                uint32_t incl = cnt;
                for(int d = 1; d < S; d <<= 1)
                {
                    uint32_t const o = __shfl_up_sync(0xffffffffu, incl, d, S);
                    if(ch.sub >= d)
                        incl += o;
                }
                uint32_t const k = ch.fill + incl - cnt;
                ch.fill += S == 1 ? cnt : __shfl_sync(0xffffffffu, incl, S - 1, S);
                // entries past the row's end are dropped (the counts report the overflow)
                if(k + cnt > cap)
                    for(uint32_t over = min(cnt, k + cnt - cap); over > 0; --over)
                        mask &= mask - 1u;
                __syncwarp();
                sRow[lane] = RowRef<T>::make(__brev(mask), rowOff, k);
                __syncwarp();
                if(S == 1)
                {
                    // full chunk: eight targets' stores at a time (lanes past the
                    // last target hold no bits)
                    uint32_t const ent = sEnt[(g0 << 5) + uint32_t(lane)];
                    for(uint32_t i = 0; i < nt; i += 8)
#pragma unroll
                        for(uint32_t u = 0; u < 8; ++u)
                            storeEntry<T>(sRow[i + u], up, rows, ent, room, status);
                    continue;
                }
                int const nS = int(min(uint32_t(S), nSlab - g0));
                for(int s = 0; s < nS; ++s)
                {
                    uint32_t const ent = sEnt[((g0 + uint32_t(s)) << 5) + uint32_t(lane)];
#pragma unroll 4
                    for(uint32_t i = 0; i < nt; ++i)
                        storeEntry<T>(sRow[i * uint32_t(S) + uint32_t(s)], up, rows, ent, room, status);
                }
            }
        }

        //! Warps per cell, as a power of two: a cell's targets are dealt to 2^shift
        //! warps in groups of 64 >> shift.  A group shares its staged windows, so
        //! large groups cost least work, but few particles in groups of 64 leave
        //! most warps idle behind the cells with the longest stencils: the group
        //! halves until n / group fills the resident warps 1.25 times (FP32: 64 from
        //! 284,160 particles on, 32 from 142,080 and so on; FP64: 189,440, 94,720, ...).
        //! Neighbour build and density sum at groups of 64 / 32 / 16 / 8 / 4, ms, * the
        //! one this line picks:
        //!   FP32 Sod         2.3 k  0.085 / 0.057 / 0.049 / 0.045 / 0.049*
        //!        Sod          18 k  0.109 / 0.082 / 0.086 / 0.086 / 0.084*
        //!        Orszag-Tang  50 k  0.093 / 0.104 / 0.100 / 0.096* / 0.113
        //!        Orszag-Tang 100 k  0.144 / 0.134 / 0.132* / 0.143 / 0.177
        //!        Orszag-Tang 201 k  0.191 / 0.199* / 0.216 / 0.250 / 0.321
        //!        Orszag-Tang 300 k  0.235* / 0.261 / 0.290 / 0.346 / 0.457
        //!        Brio-Wu      60 k  0.137 / 0.105 / 0.108 / 0.118* / 0.149
        //!        Brio-Wu      82 k  0.158 / 0.117 / 0.124* / 0.131 / 0.186
        //!        Brio-Wu     224 k  0.230 / 0.199* / 0.222 / 0.287 / 0.446
        //!        Brio-Wu     581 k  0.433* / 0.417 / 0.481 / 0.634 / 1.043
        //!        Brio-Wu       2 M  1.212* / 1.233 / 1.478 / 2.096 / 3.695
        //!   FP64 Sod         2.3 k  0.137 / 0.081 / 0.069 / 0.061 / 0.062*
        //!        Orszag-Tang 100 k  0.186 / 0.179* / 0.189 / 0.219 / 0.287
        //!        Orszag-Tang 151 k  0.204 / 0.227* / 0.245 / 0.294 / 0.400
        //!        Orszag-Tang 180 k  0.249 / 0.264* / 0.289 / 0.349 / 0.475
        //!        Orszag-Tang 201 k  0.264* / 0.285 / 0.312 / 0.382 / 0.521
        //!        Brio-Wu     109 k  0.260 / 0.198* / 0.201 / 0.241 / 0.356
        //!        Brio-Wu     176 k  0.316 / 0.246* / 0.266 / 0.361 / 0.550
        //!        Brio-Wu     224 k  0.364* / 0.296 / 0.346 / 0.465 / 0.729
        //!        Brio-Wu     263 k  0.399* / 0.343 / 0.390 / 0.510 / 0.811
        //! The particle count alone is a compromise: one-level slabs want 64 from
        //! somewhere below 150 k (FP64) or 200 k (FP32) particles on, two-level tubes 32
        //! up to 263 k and more (FP64) or 581 k (FP32).  At the points above the line
        //! costs up to 11% on the slabs' side and 23% on the tubes'.
        //! Grids with many more cells than particles are not split (each part asks for
        //! the cell's range).  The rows are the same for every group: a target's
        //! entries keep their candidate order.
        constexpr int kMaxPartShift = 4;
        __device__ __forceinline__ int partsShift(uint32_t n, uint32_t cells, uint32_t warps)
        {
            int s = 0;
            while(s < kMaxPartShift && uint64_t(n) * 4u < uint64_t(warps) * 5u * (64u >> s))
                ++s;
            while(s > 0 && (uint64_t(cells) << s) > 16ull * n)
                --s;
            return s;
        }

        //! Tunable launch shapes (picked per context by sph_autotune): CAP is the
        //! staging depth (candidates per shared-memory window), MINB the blocks
        //! per SM the register allocation must admit, CU the unroll depth of the
        //! FP32 mask cull (8 or 2; the FP64 cull ignores it).
        template<typename T, bool PAIRMAX, int CAP, int MINB, int CU>
        __global__ void __launch_bounds__(kWarps * 32, MINB) kNeighbours(DevCtx c, double h0, bool countOnly)
        {
            using V4 = typename PairCfg<T>::V4;
            extern __shared__ __align__(32) unsigned char smem[];
            int const warp = threadIdx.x >> 5;
            int const lane = threadIdx.x & 31;
            // per warp: negated shifted x, y, z, (pair-max cull) smoothing length, list entry
            constexpr int kCols = PAIRMAX ? 4 : 3;
            // (columns in skewed slabs, see skewed())
            constexpr int kCol = colLen<CAP>();
            T* const sNX = reinterpret_cast<T*>(smem) + warp * kCol;
            T* const sNY = sNX + kWarps * kCol;
            T* const sNZ = sNY + kWarps * kCol;
            T* const sH = sNZ + kWarps * kCol; // only with PAIRMAX: -(supT h_j)^2
            uint32_t* const sEnt = reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(smem) + kCols * kWarps * kCol)
                                   + warp * CAP;
            // per warp: window position of each target's own entry (up to 64
            // targets of the chunk pair; ~0 = not in this window)
            uint32_t* const sSelf = reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(smem) + kCols * kWarps * kCol)
                                    + kWarps * CAP + warp * 64;
            // per warp: each lane's slab mask and row position during the write-out
            using Row = typename RowRef<T>::Type;
            Row* const sRow = reinterpret_cast<Row*>(sSelf - warp * 64 + kWarps * 64) + warp * 32;
            Records<V4, T> const rec = records<T>(c);
            T const supT = T(c.support);
            T const Rg = mulRn(supT, T(h0));
            T const R2g = mulRn(Rg, Rg);
            uint32_t const cap = c.lists.cap;
            uint32_t maxCount = 0;
            unsigned long long pairs = 0;
            unsigned long long cand = 0; // warp-uniform: staged sources x targets culled

            // Work queue over the cells of the boxes' current grids: each warp
            // takes its next item from a counter; the fetch for the next item is
            // issued first and read at the loop's end.  Item q is cell
            // q - activeBase of the box whose range holds it.
            int const partShift = partsShift(c.n, *c.activeTotal, 148u * uint32_t(MINB) * kWarps);
            uint32_t const group = 64u >> partShift;
            uint32_t const parts = 1u << partShift;
            uint32_t const nWork = *c.activeTotal << partShift;
            uint32_t pending = 0;
            int box = 0; // items come in ascending order, so the box only moves up
            if(lane == 0)
                pending = atomicAdd(c.work, 1u);
            for(uint32_t q = __shfl_sync(0xffffffffu, pending, 0); q < nWork; q = __shfl_sync(0xffffffffu, pending, 0))
            {
                if(lane == 0)
                    pending = atomicAdd(c.work, 1u);
                uint32_t const item = q >> partShift;
                if(item - c.boxes[box].activeBase >= c.boxes[box].nItems)
                    box = boxOfWork(c.boxes, c.nbox, item);
                // item -> cell: the box's level-0 cells first, then its level-1 cells
                uint32_t const l = item - c.boxes[box].activeBase;
                uint32_t const nc0 = c.boxes[box].ncells;
                uint32_t const cell = c.boxes[box].cellBase + (l < nc0 ? l : c.boxes[box].ncellsMax + (l - nc0));
                if(!checkIndex(cell < c.cells.ncells, c.status, kChkCell))
                    continue;
                uint32_t const tBeg = c.cells.start[cell];
                uint32_t const tEnd = c.cells.mid[cell];
                // this part's first targets; the parts of a cell take groups in turn
                uint32_t const tFirst = tBeg + (q & (parts - 1u)) * group;
                if(tFirst >= tEnd || !checkIndex(tEnd <= c.n, c.status, kChkTargets))
                    continue;
                BoxDev const& B = c.boxes[box];
                // Target cell: level 0 (the grid) or level 1 (one of the m0 x m1 x m2
                // sub-cells of a level-0 cell, numbered parent-major), its level-0
                // parent c0 and, for level 1, its coordinates ct on the fine grid
                // (m_a n_a cells per axis).
                int const lt = l < B.ncells ? 0 : 1;
                int ct[3], c0[3];
                {
                    uint32_t const li = lt ? l - B.ncells : l;
                    uint32_t const par = lt ? li >> __popc(B.msub - 1u) : li; // msub is 2, 4 or 8
                    uint32_t const n0 = uint32_t(B.n[0]), n1 = uint32_t(B.n[1]);
                    uint32_t const row = par / n0, plane = row / n1;
                    c0[0] = int(par - row * n0);
                    c0[1] = int(row - plane * n1);
                    c0[2] = int(plane);
                    uint32_t sub = lt ? li & (B.msub - 1u) : 0u;
#pragma unroll
                    for(int a = 0; a < 3; ++a)
                    {
                        uint32_t const sh = uint32_t(B.m[a] - 1); // splits are 1 or 2
                        ct[a] = (c0[a] << sh) + int(sub & sh);
                        sub >>= sh;
                    }
                }
                // Candidate descriptors: the 27 level-0 cells around the parent, then
                // with two levels either the 27 level-1 cells around a level-1 target
                // or, for a level-0 target, the level-1 block (all sub-cells) of each
                // of those 27 cells.  Each carries its source range and the level-0
                // stencil slot of its image.
                //
                // Order: a periodic axis of one or two cells shows the same cell through
                // two or three images.  Such axes run fastest, equal cells adjacent (-1,
                // +1, 0), so a row lists a cell's images one after another and the lanes
                // of a pair pass, which stand at different images, stay on the same
                // lines of records: 16.8 -> 12.0 distinct lines a request on the
                // Orszag-Tang slab (one cell thick; simulated), force pass 0.643 -> 0.600
                // ms when it was made.
                int const nDesc = 27 + (B.levels == 2 ? 27 : 0);
                auto describe = [&](int d, uint32_t& sBeg, uint32_t& sCnt, uint32_t& slot, T sh[3])
                {
                    sBeg = 0;
                    sCnt = 0;
                    slot = 0;
                    sh[0] = sh[1] = sh[2] = T(0);
                    if(d >= nDesc)
                        return;
                    int o[3], f[3];
                    bool ok = true;
                    bool const fine = d >= 27;
                    int const k = fine ? d - 27 : d;
                    bool const fineCell = fine && lt; // a level-1 neighbour of a level-1 target
                    bool thin[3];
                    int nThin = 0, before = 0, off[3];
#pragma unroll
                    for(int a = 0; a < 3; ++a)
                    {
                        thin[a] = B.periodic[a] && (fineCell ? B.n[a] << (B.m[a] - 1) : B.n[a]) <= 2;
                        nThin += thin[a] ? 1 : 0;
                    }
#pragma unroll
                    for(int a = 0; a < 3; ++a)
                    {
                        int const place = thin[a] ? before : nThin + a - before;
                        before += thin[a] ? 1 : 0;
                        int const digit = stencilOff(k, place) + 1;
                        off[a] = !thin[a] ? digit - 1 : (digit == 2 ? 0 : 2 * digit - 1);
                    }
#pragma unroll
                    for(int a = 0; a < 3; ++a)
                    {
                        int const n0 = B.n[a];
                        if(fineCell)
                        {
                            // fine-grid neighbour; its level-0 parent (image-aware) gives o
                            int const sh = B.m[a] - 1; // splits are 1 or 2
                            int const n1 = n0 << sh;
                            int const fa = ct[a] + off[a];
                            o[a] = (fa >> sh) - c0[a];
                            f[a] = fa < 0 ? fa + n1 : (fa >= n1 ? fa - n1 : fa);
                            ok = ok && (f[a] == fa || B.periodic[a]);
                        }
                        else
                        {
                            o[a] = off[a];
                            int const ca = c0[a] + o[a];
                            f[a] = ca < 0 ? ca + n0 : (ca >= n0 ? ca - n0 : ca);
                            ok = ok && (f[a] == ca || B.periodic[a]);
                        }
                    }
                    slot = uint32_t((o[0] + 1) + 3 * (o[1] + 1) + 9 * (o[2] + 1));
#pragma unroll
                    for(int a = 0; a < 3; ++a)
                        sh[a] = T(o[a]) * edgeOf<T>(B, a);
                    if(!ok)
                        return;
                    if(fineCell)
                    {
                        int p[3];
                        uint32_t subc = 0, stride = 1;
#pragma unroll
                        for(int a = 0; a < 3; ++a)
                        {
                            int const sh = B.m[a] - 1;
                            p[a] = f[a] >> sh;
                            subc += uint32_t(f[a] & sh) * stride;
                            stride <<= sh;
                        }
                        uint32_t const par = (uint32_t(p[2]) * uint32_t(B.n[1]) + uint32_t(p[1])) * uint32_t(B.n[0])
                                             + uint32_t(p[0]);
                        uint32_t const cellId = B.cellBase + B.ncellsMax + par * B.msub + subc;
                        if(!checkIndex(cellId < c.cells.ncells, c.status, kChkCell))
                            return;
                        sBeg = c.cells.start[cellId];
                        sCnt = c.cells.end[cellId] - sBeg;
                        if(!checkIndex(sBeg <= c.n && sCnt <= c.n - sBeg, c.status, kChkRange))
                            sCnt = 0;
                        return;
                    }
                    uint32_t const cellId
                        = B.cellBase + (uint32_t(f[2]) * uint32_t(B.n[1]) + uint32_t(f[1])) * uint32_t(B.n[0]) + uint32_t(f[0]);
                    if(!checkIndex(cellId < c.cells.ncells, c.status, kChkCell))
                        return;
                    if(fine)
                    {
                        // all level-1 sub-cells of a level-0 neighbour, as one range
                        sBeg = c.cells.bstart[cellId];
                        sCnt = c.cells.bend[cellId] - sBeg;
                    }
                    else
                    {
                        sBeg = c.cells.start[cellId];
                        sCnt = c.cells.end[cellId] - sBeg;
                    }
                    if(!checkIndex(sBeg <= c.n && sCnt <= c.n - sBeg, c.status, kChkRange))
                        sCnt = 0;
                };

                // exclusive prefix of the page's source counts and the page total
                auto scan = [&](uint32_t cnt, uint32_t& pre, uint32_t& total)
                {
                    uint32_t incl = cnt;
#pragma unroll
                    for(int d = 1; d < 32; d <<= 1)
                    {
                        uint32_t const o = __shfl_up_sync(0xffffffffu, incl, d);
                        if(lane >= d)
                            incl += o;
                    }
                    pre = incl - cnt;
                    total = __shfl_sync(0xffffffffu, incl, 31);
                };
                // Page 0 (all of a single-level box's 27 slots) is described once per
                // cell; later pages once per target chunk.
                uint32_t sBeg0, sCnt0, slot0, pre0, total0;
                T sh0[3];
                describe(lane, sBeg0, sCnt0, slot0, sh0);
                scan(sCnt0, pre0, total0);

                // Two target chunks (a group of up to 64 targets) share every staged window.
                for(uint32_t tc = tFirst; tc < tEnd; tc += group << partShift)
                {
                    TargetChunk<T> A, Bc;
                    uint32_t const nTargets = min(group, tEnd - tc);
                    uint32_t const ntA = min(32u, nTargets);
                    uint32_t const ntB = nTargets - ntA;
                    initChunk(A, rec, tc, ntA, lane, supT);
                    initChunk(Bc, rec, tc + 32, ntB, lane, supT);
                    // Bounding box of the two chunks' targets and their largest cull
                    // radius: staging keeps only candidates within that radius of the
                    // box.  For a target x_i in [lo, hi] and a staged -x_j, rounding
                    // is monotone, so |x_i - x_j| (rounded) >= max(lo - x_j, x_j - hi,
                    // 0) (rounded) on each axis; with the radius widened by 2^-10 the
                    // box test passes every candidate the exact cull accepts.
                    T bLo[3], bHi[3];
                    {
                        T const inf = T(kFar);
                        T const ax[3] = {A.x, A.y, A.z}, bx[3] = {Bc.x, Bc.y, Bc.z};
#pragma unroll
                        for(int a = 0; a < 3; ++a)
                        {
                            T const l0 = A.act ? ax[a] : inf, l1 = Bc.act ? bx[a] : inf;
                            T const h0 = A.act ? ax[a] : -inf, h1 = Bc.act ? bx[a] : -inf;
                            bLo[a] = warpMinT(l0 < l1 ? l0 : l1);
                            bHi[a] = warpMaxT(h0 > h1 ? h0 : h1);
                        }
                    }
                    T const widen = T(1) + T(1.0 / 1024.0);
                    // PAIRMAX: the pair radius is max(R_i, R_j); nRt = -(max_i R_i)^2
                    T nRt = -R2g;
                    if constexpr(PAIRMAX)
                    {
                        T const nA = A.act ? A.nR2 : T(0), nB = Bc.act ? Bc.nR2 : T(0);
                        nRt = warpMinT(nA < nB ? nA : nB);
                    }
                    // The page of 32 descriptors being staged; page 0 (all of a
                    // single-level box's 27 slots) was described for the cell.
                    uint32_t sBeg = sBeg0, pre = pre0, total = total0;
                    T sh[3] = {sh0[0], sh0[1], sh0[2]};
                    // entry of staged position q: eBase of q's descriptor + (q << 5)
                    // (j = sBeg + q - pre, packed as (j << 5) | slot)
                    uint32_t eBase = ((sBeg - pre) << 5) | slot0;
                    uint32_t cb = 0; // next position of the page
                    int page = 0;
                    for(bool more = true; more;)
                    {
                        // Fill a window.  Flat staging: lane l reads positions l, l + 32,
                        // ...; the descriptor of position q is the last one whose prefix
                        // is <= q (a shuffle binary search over the page's prefixes; empty
                        // descriptors share the next one's prefix and are passed over).
                        // kStageBatch positions' records are in flight at once.  The
                        // candidates that pass the box test are staged in order at
                        // 0 .. m-1, until the window may not hold another batch: the box
                        // test passes about 4 in 10, and windows that ended with a
                        // fixed count of positions were culled as 16 part-filled slabs
                        // where 12 full ones do (jittered Orszag-Tang slab).
                        constexpr int KB = PairCfg<T>::kStageBatch;
                        uint32_t mW = 0; // staged so far (warp-uniform)
                        __syncwarp();
                        sSelf[lane] = ~0u;
                        sSelf[lane + 32] = ~0u;
                        // another lane may write the same word while staging; the
                        // shuffles and ballots in between do not order memory
                        __syncwarp();
                        while(mW + 32u * KB <= uint32_t(CAP))
                        {
                            if(cb >= total)
                            {
                                ++page;
                                more = page * 32 < nDesc;
                                if(!more)
                                    break;
                                uint32_t sCnt, slotD;
                                describe(page * 32 + lane, sBeg, sCnt, slotD, sh);
                                scan(sCnt, pre, total);
                                eBase = ((sBeg - pre) << 5) | slotD;
                                cb = 0;
                                continue;
                            }
                            uint32_t ent[KB];
                            int dsc[KB];
                            V4 pj[KB];
                            T hj[KB];
#pragma unroll
                            for(int k = 0; k < KB; ++k)
                            {
                                uint32_t const q = cb + uint32_t(lane) + 32u * uint32_t(k);
                                int sd = 0;
#pragma unroll
                                for(int step = 16; step >= 1; step >>= 1)
                                {
                                    uint32_t const v = __shfl_sync(0xffffffffu, pre, sd + step);
                                    if(v <= q)
                                        sd += step;
                                }
                                dsc[k] = sd;
                                ent[k] = __shfl_sync(0xffffffffu, eBase, sd) + (q << 5);
                                if(q < total && checkIndex((ent[k] >> 5) < c.n, c.status, kChkStaged))
                                {
                                    pj[k] = ld4(rec.pm + (ent[k] >> 5));
                                    if constexpr(PAIRMAX)
                                        hj[k] = rec.hc[ent[k] >> 5];
                                }
                            }
#pragma unroll
                            for(int k = 0; k < KB; ++k)
                            {
                                bool const in = cb + uint32_t(lane) + 32u * uint32_t(k) < total;
                                T const sx = __shfl_sync(0xffffffffu, sh[0], dsc[k]);
                                T const sy = __shfl_sync(0xffffffffu, sh[1], dsc[k]);
                                T const sz = __shfl_sync(0xffffffffu, sh[2], dsc[k]);
                                T const nx = in ? -addRn(pj[k].x, sx) : T(kFar);
                                T const ny = in ? -addRn(pj[k].y, sy) : T(kFar);
                                T const nz = in ? -addRn(pj[k].z, sz) : T(kFar);
                                T nRj = T(0);
                                if constexpr(PAIRMAX)
                                {
                                    T const Rj = mulRn(supT, in ? hj[k] : T(0));
                                    nRj = -mulRn(Rj, Rj);
                                }
                                T const dx = fmax(fmax(addRn(bLo[0], nx), -addRn(bHi[0], nx)), T(0));
                                T const dy = fmax(fmax(addRn(bLo[1], ny), -addRn(bHi[1], ny)), T(0));
                                T const dz = fmax(fmax(addRn(bLo[2], nz), -addRn(bHi[2], nz)), T(0));
                                T const nR = (nRj < nRt ? nRj : nRt) * widen;
                                bool const pass = in && dx * dx + dy * dy + dz * dz + nR < T(0);
                                uint32_t const passMask = __ballot_sync(0xffffffffu, pass);
                                if(pass)
                                {
                                    uint32_t const w = mW + uint32_t(__popc(passMask & ((1u << lane) - 1u)));
                                    uint32_t const ws = skewed(w);
                                    sNX[ws] = nx;
                                    sNY[ws] = ny;
                                    sNZ[ws] = nz;
                                    sEnt[w] = ent[k];
                                    if constexpr(PAIRMAX)
                                        sH[ws] = nRj;
                                    // a target's own entry: centre slot, index among the pair's targets
                                    uint32_t const jr = (ent[k] >> 5) - tc;
                                    if((ent[k] & 31u) == kCentreSlot && jr < nTargets)
                                        sSelf[jr] = w;
                                }
                                mW += uint32_t(__popc(passMask));
                            }
                            cb += 32u * KB;
                        }
                        uint32_t const m = mW;
                        // far candidates up to the next multiple of 32
                        for(uint32_t q = m + uint32_t(lane); q < ((m + 31u) & ~31u); q += 32)
                        {
                            uint32_t const qs = skewed(q);
                            sNX[qs] = T(kFar);
                            sNY[qs] = T(kFar);
                            sNZ[qs] = T(kFar);
                            if constexpr(PAIRMAX)
                                sH[qs] = T(0);
                        }
                        __syncwarp();
                        // One copy of the cull serves both chunks (a loop that is not
                        // unrolled): the kernel's hot code stays small enough for the
                        // instruction caches when warps run different phases at once.
#pragma unroll 1
                        for(int w = 0; w < (ntB ? 2 : 1); ++w)
                        {
                            TargetChunk<T> ch = w ? Bc : A;
                            uint32_t const first = tc + 32u * uint32_t(w);
                            size_t const row0 = rowStart<T>(size_t(first & ~3u), size_t(cap));
                            cullChunk<T, PAIRMAX, CU>(
                                ch, sNX, sNY, sNZ, sH, sEnt, sSelf + 32 * w, sRow, first, w ? ntB : ntA, m, supT, R2g,
                                c.lists.list + row0, listWords(c.n, cap) - row0, c.status, cap, lane, countOnly);
                            if(w)
                                Bc = ch;
                            else
                                A = ch;
                        }
                        cand += uint64_t(m) * nTargets;
                    }
#pragma unroll 1
                    for(int w = 0; w < (ntB ? 2 : 1); ++w)
                    {
                        TargetChunk<T> const ch = w ? Bc : A;
                        uint32_t nl = ch.nl;
                        for(int d = 1; d < ch.S; d <<= 1)
                            nl += __shfl_xor_sync(0xffffffffu, nl, d);
                        if(ch.act && ch.sub == 0)
                        {
                            maxCount = max(maxCount, nl);
                            pairs += nl;
                            if(!countOnly)
                            {
                                c.lists.count[ch.t] = nl;
                                c.lists.rowLen[ch.t] = min(ch.fill, cap);
                            }
                        }
                    }
                }
            }
            maxCount = warpMaxU(maxCount);
            pairs = warpSumU64(pairs);
            if(lane == 0)
            {
                if(maxCount > cap)
                    atomicMax(&c.status[kStatOverflow], maxCount);
                atomicMax(&c.status[kStatMaxCount], maxCount);
                atomicAdd(&c.scal->pairs, pairs);
                atomicAdd(&c.scal->candidates, cand);
            }
        }

        template<typename T, bool PM, int CAP>
        constexpr size_t neighbourSmem()
        {
            return size_t(kWarps)
                   * (colLen<CAP>() * (PM ? 4 : 3) * sizeof(T) + (CAP + 64) * sizeof(uint32_t) + 32 * sizeof(typename RowRef<T>::Type));
        }

        // ---- launch-shape variants -------------------------------------------
        // FP32: (CAP, blocks/SM) = (256, 6), (256, 5), (128, 6), (128, 5), each with
        // the mask cull fully unrolled and unrolled twice; FP64: (256, 4), (128, 4).
        // Variant 0 is the default.
        constexpr int kVariants32 = 8, kVariants64 = 2;
        constexpr int kCap32[kVariants32] = {256, 256, 128, 128, 256, 256, 128, 128};
        constexpr int kBlk32[kVariants32] = {6, 5, 6, 5, 6, 5, 6, 5};
        constexpr int kUnr32[kVariants32] = {8, 8, 8, 8, 2, 2, 2, 2};
        constexpr int kCap64[kVariants64] = {256, 128};
        constexpr int kBlk64 = 4;

        //! Shared-memory carve-out (percent of the maximum) that fits `blocks`
        //! blocks of `smem` bytes; the rest of the unified array stays L1 for
        //! the staging loads.
        int carveout(size_t smem, int blocks)
        {
            size_t const need = size_t(blocks) * (smem + 1024);
            size_t const maxSmem = 228 * 1024;
            int pct = int((need * 100 + maxSmem - 1) / maxSmem);
            return pct > 100 ? 100 : pct;
        }

        template<typename T, bool PM, int CAP, int MINB, int CU = 8>
        void configureOne()
        {
            auto f = kNeighbours<T, PM, CAP, MINB, CU>;
            size_t const smem = neighbourSmem<T, PM, CAP>();
            cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
            cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, carveout(smem, MINB));
        }

        template<typename T, bool PM, int CAP, int MINB, int CU = 8>
        void launchOne(DevCtx const& c, PhysArgs const& pa, bool countOnly, cudaStream_t s)
        {
            size_t const smem = neighbourSmem<T, PM, CAP>();
            // persistent grid: enough resident blocks to fill every SM; cells come
            // from the work queue
            uint32_t const resident = 148u * uint32_t(MINB);
            uint64_t const items = (uint64_t(c.cells.ncells) << kMaxPartShift) / kWarps + 1;
            uint32_t const blocks = items > resident ? resident : uint32_t(items);
            if(blocks)
            {
                kNeighbours<T, PM, CAP, MINB, CU><<<blocks, kWarps * 32, smem, s>>>(c, pa.h0, countOnly);
                countLaunches(1);
            }
        }

        template<bool PM>
        void launch32(DevCtx const& c, PhysArgs const& pa, bool countOnly, int variant, cudaStream_t s)
        {
            switch(variant)
            {
#define SPH_NB32(v) launchOne<float, PM, kCap32[v], kBlk32[v], kUnr32[v]>(c, pa, countOnly, s)
            case 1: SPH_NB32(1); break;
            case 2: SPH_NB32(2); break;
            case 3: SPH_NB32(3); break;
            case 4: SPH_NB32(4); break;
            case 5: SPH_NB32(5); break;
            case 6: SPH_NB32(6); break;
            case 7: SPH_NB32(7); break;
            default: SPH_NB32(0); break;
#undef SPH_NB32
            }
        }

        template<bool PM>
        void launch64(DevCtx const& c, PhysArgs const& pa, bool countOnly, int variant, cudaStream_t s)
        {
            if(variant == 1)
                launchOne<double, PM, kCap64[1], kBlk64>(c, pa, countOnly, s);
            else
                launchOne<double, PM, kCap64[0], kBlk64>(c, pa, countOnly, s);
        }

        template<bool PM>
        void configurePM()
        {
#define SPH_CONF32(v) configureOne<float, PM, kCap32[v], kBlk32[v], kUnr32[v]>()
            SPH_CONF32(0);
            SPH_CONF32(1);
            SPH_CONF32(2);
            SPH_CONF32(3);
            SPH_CONF32(4);
            SPH_CONF32(5);
            SPH_CONF32(6);
            SPH_CONF32(7);
#undef SPH_CONF32
            configureOne<double, PM, kCap64[0], kBlk64>();
            configureOne<double, PM, kCap64[1], kBlk64>();
        }
    } // namespace

    void configureNeighbourKernels()
    {
        configurePM<true>();
        configurePM<false>();
    }

    int densityVariants(int precision)
    {
        return precision == SPH_PREC_FP64 ? kVariants64 : kVariants32;
    }

    void densityShape(int precision, int variant, int* stagingDepth, int* blocksPerSm, int* cullUnroll)
    {
        bool const f64 = precision == SPH_PREC_FP64;
        int const v = variant < 0 || variant >= densityVariants(precision) ? 0 : variant;
        *stagingDepth = f64 ? kCap64[v] : kCap32[v];
        *blocksPerSm = f64 ? kBlk64 : kBlk32[v];
        *cullUnroll = f64 ? 0 : kUnr32[v];
    }

    void launchNeighbours(DevCtx const& c, PhysArgs const& pa, int precision, bool countOnly, int variant, cudaStream_t s)
    {
        bool const pm = pa.cull == SPH_CULL_PAIR_MAX;
        if(precision == SPH_PREC_FP64)
            pm ? launch64<true>(c, pa, countOnly, variant, s) : launch64<false>(c, pa, countOnly, variant, s);
        else
            pm ? launch32<true>(c, pa, countOnly, variant, s) : launch32<false>(c, pa, countOnly, variant, s);
    }
} // namespace sph
