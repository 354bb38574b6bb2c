// Pair passes: density summation and the force pass, over the list rows of the
// neighbour build (neighbours.cu).
//
// Replaces the functors the reference's pair engine drives (AccumulateDensity,
// DensitySummation.hpp:50-74; HydroInteraction, HydroForces.hpp:86-176), plus
// the viscosity, SPMHD and Dedner terms the reference lacks.  The density pass
// writes rho (FP64) and the target's derived record for the force pass.
//
// What bounds both passes is the gather of the sources' 16-byte records: a warp
// request costs the L1 about one wavefront per 128-byte line it touches, and 32
// lanes stand at 32 places of their rows (9.6 wavefronts a gather on the jittered
// Orszag-Tang slab).  S lanes can share a target and read S consecutive entries,
// which mostly lie in one cell and touch fewer lines.  Against that stand S times
// the per-target work (records, reductions, FP64 epilogue).  S = 1 / 2, ms:
//   FP32 force  1 M slab 0.579 / 0.697, 1.35 M Kelvin-Helmholtz 0.821 / 0.960,
//               2 M Brio-Wu particles 0.759 / 0.917
//   FP32 build and density sum, the same three: 0.692 / 0.739, 1.072 / 1.136,
//               1.212 / 1.292
//   FP64 force  206 k slab 0.329 / 0.314, 176 k Brio-Wu particles 0.195 / 0.191
//   FP64 build and density sum, the same two: 0.315 / 0.297, 0.281 / 0.270
// So one lane in FP32, two in FP64 (twice the bytes per record and fewer resident
// warps).
//
// Precision: an FP32 lane sums its entries in blocks of 8 folded by TwoSum
// (CompAcc); FP64 lanes sum plainly.  Lane sums are added in FP64.
#include "pair_common.cuh"

namespace sph
{
    namespace
    {
        constexpr int kThreads = 128;
        //! Lanes that share a target's row.
        template<typename T>
        constexpr int kLanes = sizeof(T) == 4 ? 1 : 2;

        //! Exchange over the S lanes (1 or 2) of a target: lane s comes in with
        //! words 4 s .. 4 s + 3 of 4 S and leaves with words s, s + S, ..., s + 3 S.
        template<int S>
        __device__ __forceinline__ uint4 spread(uint4 v, uint32_t sub, uint32_t lanes)
        {
            if constexpr(S == 1)
                return v;
            else
            {
                static_assert(S == 2);
                uint32_t const a = __shfl_xor_sync(lanes, sub ? v.x : v.y, 1), b = __shfl_xor_sync(lanes, sub ? v.z : v.w, 1);
                return sub ? make_uint4(a, b, v.y, v.w) : make_uint4(v.x, v.z, a, b);
            }
        }

        //! Walks a lane's share of a row, entries sub, sub + S, ...: fetch(e)
        //! starts loading the records of entry e, term(next) uses the fetched ones
        //! and fetches `next`; fold() closes each block of 8 terms.  The S lanes
        //! load 4 S entries as one 16-byte word each and exchange them (a 4-byte
        //! load per entry would cost a wavefront per target and entry).  `any` is
        //! a valid entry, fetched past the row's end.
        template<typename T, int S, typename F, typename M, typename D>
        __device__ __forceinline__ void walkRow(
            uint32_t const* row,
            uint32_t n,
            uint32_t sub,
            uint32_t any,
            F&& fetch,
            M&& term,
            D&& fold)
        {
            if(n == 0)
                return;
            uint32_t const lanes = ((1u << S) - 1u) << (threadIdx.x & (32u - S));
            auto quad = [&](uint32_t k) // entries k .. k + 3, k a multiple of 4
            { return *reinterpret_cast<uint4 const*>(row + rowPlace<T>(k)); };
            uint4 e = spread<S>(quad(4 * sub), sub, lanes);
            fetch(sub < n ? e.x : any);
            for(uint32_t k = sub;; k += 4 * S)
            {
                // all lanes of the target agree: a group that is not the last is full
                bool const more = k - sub + 4 * S < n;
                uint4 next = e;
                if(more)
                    next = quad(k - sub + 4 * (S + sub));
                if(k >= n)
                    break;
                term(k + S < n ? e.y : any);
                if(k + S >= n)
                    break;
                term(k + 2 * S < n ? e.z : any);
                if(k + 2 * S >= n)
                    break;
                term(k + 3 * S < n ? e.w : any);
                if(k + 3 * S >= n)
                    break;
                if(more)
                    next = spread<S>(next, sub, lanes);
                term(k + 4 * S < n ? next.x : any);
                if((k & (4u * S)) != 0)
                    fold();
                if(!more)
                    break;
                e = next;
            }
            fold();
        }

        //! Lanes per target of the FP32 passes on small systems: each takes blocks of
        //! 8 consecutive entries, and the blocks' partial sums are folded in row
        //! order by every lane (foldBlocks), so the sums, to the bit, are those of one
        //! lane walking the whole row.
        constexpr int kWide = 8;

        //! Folds the lanes' block partials, in block order, into each lane's sum.
        __device__ __forceinline__ void foldBlocks(Acc<float>& a, int blocks, uint32_t lanes)
        {
            for(int s = 0; s < blocks; ++s)
                a.c.fold(__shfl_sync(lanes, a.part, s, kWide));
            a.part = 0.f;
        }

        //! Walks a row with kWide lanes: lane s takes the blocks s, s + 8, ... of 8
        //! entries; foldAll(blocks, lanes) closes each round of up to 8 blocks.
        template<typename F, typename M, typename D>
        __device__ __forceinline__ void walkRowWide(
            uint32_t const* row,
            uint32_t n,
            uint32_t sub,
            uint32_t any,
            F&& fetch,
            M&& term,
            D&& foldAll)
        {
            uint32_t const lanes = 0xffu << (threadIdx.x & 24u);
            for(uint32_t base = 0; base < n; base += 8 * kWide)
            {
                uint32_t const k = base + 8 * sub;
                if(k < n)
                {
                    uint4 const* const q = reinterpret_cast<uint4 const*>(row + rowPlace<float>(k));
                    uint4 const a = q[0], b = q[1];
                    uint32_t const m = n - k;
                    fetch(a.x);
                    term(m > 1 ? a.y : any);
                    if(m > 1)
                        term(m > 2 ? a.z : any);
                    if(m > 2)
                        term(m > 3 ? a.w : any);
                    if(m > 3)
                        term(m > 4 ? b.x : any);
                    if(m > 4)
                        term(m > 5 ? b.y : any);
                    if(m > 5)
                        term(m > 6 ? b.z : any);
                    if(m > 6)
                        term(m > 7 ? b.w : any);
                    if(m > 7)
                        term(any);
                }
                __syncwarp(lanes);
                uint32_t const left = (n - base + 7) / 8;
                foldAll(int(left < kWide ? left : kWide), lanes);
            }
        }

        //! A source's position with its stencil image's shift added.
        //!
        //! FP32: the slot's offsets o in {-1, 0, 1} are worked out in floats (slot s =
        //! (o0 + 1) + 3 (o1 + 1) + 9 (o2 + 1), so o2 = round((s - 13)/9) and so on; no
        //! quotient comes within 0.05 of a half) and the shift o e is an exact
        //! product, so the fused add rounds like the sum with the shift table's
        //! entry.  Reading the table per entry went through the gathers' own
        //! bottleneck: 6 of 18 (density) and 47 (force) L1 wavefronts per entry, for
        //! 6 instructions saved; offsets read from constant memory were slower still
        //! (density pass 0.51 ms against 0.23: divergent constant reads serialise).
        //! FP64, not bound by the L1, reads the table.
        template<typename T>
        struct ImageShift;
        template<>
        struct ImageShift<float>
        {
            float e0, e1, e2;
            __device__ __forceinline__ ImageShift(DevCtx const& c, int box)
                : e0(c.boxes[box].edgef[0])
                , e1(c.boxes[box].edgef[1])
                , e2(c.boxes[box].edgef[2])
            {
            }
            __device__ __forceinline__ float4 at(float4 p, uint32_t entry) const
            {
                constexpr float kRound = 12582912.f; // 1.5 2^23: adding it rounds to an integer
                float const s = __uint_as_float((entry & 31u) | 0x4b000000u) - (8388608.f + float(kCentreSlot));
                float const oz = __fmaf_rn(s, 1.f / 9.f, kRound) - kRound;
                float const r = __fmaf_rn(oz, -9.f, s);
                float const oy = __fmaf_rn(r, 1.f / 3.f, kRound) - kRound;
                float const ox = __fmaf_rn(oy, -3.f, r);
                return make_float4(__fmaf_rn(ox, e0, p.x), __fmaf_rn(oy, e1, p.y), __fmaf_rn(oz, e2, p.z), p.w);
            }
        };
        template<>
        struct ImageShift<double>
        {
            D4 const* table;
            __device__ __forceinline__ ImageShift(DevCtx const& c, int box) : table(c.shift64 + size_t(box) * 32)
            {
            }
            __device__ __forceinline__ D4 at(D4 p, uint32_t entry) const
            {
                D4 const o = ld4(table + (entry & 31u));
                return D4{p.x + o.x, p.y + o.y, p.z + o.z, p.w};
            }
        };

        //! Sum over the lanes of a target (every lane gets it).
        template<int S>
        __device__ __forceinline__ double laneSum(double v)
        {
#pragma unroll
            for(int o = 1; o < S; o <<= 1)
                v += __shfl_xor_sync(0xffffffffu, v, o);
            return v;
        }

        //! Largest / smallest value per box over the calling threads: one atomic
        //! per warp when its active threads are in one box.
        __device__ __forceinline__ void boxMax(unsigned long long* bits, int box, bool act, double v)
        {
            int const box0 = __reduce_max_sync(0xffffffffu, act ? box : -1);
            if(box0 < 0)
                return;
            if(__all_sync(0xffffffffu, box == box0 || !act))
            {
                v = warpMaxD(act ? v : 0.0);
                if((threadIdx.x & 31) == 0)
                    atomicMax(&bits[box0], orderedBits(v));
            }
            else if(act)
                atomicMax(&bits[box], orderedBits(v));
        }
        __device__ __forceinline__ void boxMin(unsigned long long* bits, int box, bool act, double v)
        {
            int const box0 = __reduce_max_sync(0xffffffffu, act ? box : -1);
            if(box0 < 0)
                return;
            if(__all_sync(0xffffffffu, box == box0 || !act))
            {
                v = warpMinD(act ? v : 1e300);
                if((threadIdx.x & 31) == 0 && v < 1e300)
                    atomicMin(&bits[box0], orderedBits(v));
            }
            else if(act && v < 1e300)
                atomicMin(&bits[box], orderedBits(v));
        }

        //! Density sum of every target over its row: rho, the force pass's
        //! records and the box's largest signal speed (Dedner's c_h).  A kernel of
        //! its own, beside the neighbour build: its lanes all have work (the
        //! build's warps hold one cell each), and neither kernel carries the
        //! other's registers and instructions.
        template<int K, typename T, bool kSmall>
        __global__ void __launch_bounds__(kThreads) kDensity(DevCtx c, PhysArgs pa)
        {
            using V4 = typename PairCfg<T>::V4;
            Records<V4, T> const rec = records<T>(c);
            constexpr int S = kSmall ? kWide : kLanes<T>;
            uint32_t const sub = threadIdx.x & uint32_t(S - 1);
            uint32_t const t = (blockIdx.x * kThreads + threadIdx.x) / S;
            if(blockIdx.x == 0 && threadIdx.x == 0)
                *c.work = 0; // the neighbour build's queue, should it run again on these cells
            bool const act = t < c.n && isTarget(c.cur.role[t]);
            int const myBox = act ? c.cur.box[t] : -1;
            Acc<T> rho;
            if(act)
            {
                V4 const own = ld4(rec.pm + t);
                HConst<T> const hk = hconst<K, T>(rec.hc[t]);
                ImageShift<T> const shift(c, myBox);
                if(sub == 0)
                    rho.add(own.w * kernelW<K, T>(T(0), hk));
                V4 npm{};
                uint32_t entry = 0; // the fetched one
                auto fetch = [&](uint32_t e)
                {
                    if(!checkIndex((e >> 5) < c.n, c.status, kChkRowEntry))
                        e = 0;
                    entry = e;
                    npm = ld4(rec.pm + (e >> 5));
                };
                auto term = [&](uint32_t next)
                {
                    V4 const pj = shift.at(npm, entry);
                    fetch(next);
                    T const dx = own.x - pj.x;
                    T const dy = own.y - pj.y;
                    T const dz = own.z - pj.z;
                    T const r2 = dot3(dx, dy, dz, dx, dy, dz);
                    rho.addProduct(pj.w, kernelW<K, T>(r2 * invDistance(r2), hk));
                };
                uint32_t const n = min(c.lists.rowLen[t], c.lists.cap);
                uint32_t const* const row = c.lists.list + rowStart<T>(size_t(t), size_t(c.lists.cap));
                uint32_t const any = packEntry(t, kCentreSlot);
                if constexpr(kSmall)
                {
                    walkRowWide(
                        row, n, sub, any, fetch, term,
                        [&](int blocks, uint32_t lanes) { foldBlocks(rho, blocks, lanes); });
                    if(n == 0)
                        foldBlocks(rho, 1, 0xffu << (threadIdx.x & 24u)); // the self term alone
                }
                else
                {
                    walkRow<T, S>(row, n, sub, any, fetch, term, [&]() { rho.fold(); });
                    rho.fold();
                }
            }
            double const rhoD = kSmall ? rho.value() : laneSum<S>(rho.value());
            double ch = 0.0;
            if(act && sub == 0)
            {
                c.cur.rho[t] = rhoD;
                double Bv[3] = {c.cur.B[0][t], c.cur.B[1][t], c.cur.B[2][t]};
                double ft[4], fb[4];
                derivedRecord(rhoD, c.cur.u[t], Bv, c.cur.psi[t], pa, ft, fb);
                rec.ft[t] = mk4<V4>(ft[0], ft[1], ft[2], ft[3]);
                rec.fb[t] = mk4<V4>(fb[0], fb[1], fb[2], fb[3]);
                ch = ft[2];
            }
            boxMax(c.bs.chBits, myBox, act && sub == 0, ch);
        }

        //! Physics variants compiled separately: 0 = the reference's inviscid
        //! hydro, 1 = hydro + viscosity, 2 = SPMHD with viscosity, Dedner and the
        //! tensile correction switched at run time, 3 = SPMHD with all three on.
        //!
        //! Accumulators (compensated in FP32): a (pressure, viscosity and magnetic
        //! force together), D = sum m_j s_i v_ij.r (P dV work and div v), the viscous
        //! heating, T = sum m_j s_i ((B_i.r) v_ij - B_i (v_ij.r)) + rho_i^2 (Dedner
        //! gradient term) for the induction, and the div B sum.
        //! With the tensile correction the Maxwell-stress force and the Borve term
        //! combine to sum m_j s_j (B_j.r)/(mu0 rho_j^2) (B_j - B_i).
        template<typename T>
        struct ForceAcc
        {
            Acc<T> ax, ay, az, D, duav, tx, ty, tz, divb;
            T vsig;
        };

        //! Target-side data of the force pass.  hh, hc: half of h and of the signal
        //! speed (the pair means h_ij, c_ij are sums of halves).
        template<typename V4, typename T>
        struct OwnTarget
        {
            V4 pi, vi, ti, bi;
            HConst<T> hk;
            T hh, hc, alpha, beta, eps, rho2i;
            bool av, dedner, tensile;
        };

        template<int K, typename T, int PH, typename V4>
        __device__ __forceinline__ OwnTarget<V4, T> loadOwn(
            Records<V4, T> const& rec,
            PhysArgs const& pa,
            uint32_t t)
        {
            OwnTarget<V4, T> o;
            o.av = (PH == 1) || (PH == 3) || (PH == 2 && (pa.physics & SPH_PHYS_AV));
            o.dedner = (PH == 3) || (PH == 2 && (pa.physics & SPH_PHYS_DEDNER));
            o.tensile = (PH == 3) || (PH == 2 && (pa.physics & SPH_PHYS_TENSILE));
            o.pi = ld4(rec.pm + t);
            o.vi = ld4(rec.fv + t);
            o.ti = ld4(rec.ft + t);
            o.bi = V4{};
            if constexpr(PH >= 2)
                o.bi = ld4(rec.fb + t);
            o.hk = hconst<K, T>(o.vi.w);
            o.hh = T(0.5) * o.vi.w;
            o.hc = T(0.5) * o.ti.z;
            o.alpha = T(pa.alpha);
            o.beta = T(pa.beta);
            o.eps = T(pa.avEps);
            o.rho2i = o.ti.x * o.ti.x;
            return o;
        }

        //! One pair term of the force pass: source records pj (shifted to its
        //! image), vj, tj, bj.
        template<int K, typename T, int PH, typename V4>
        __device__ __forceinline__ void pairTerm(
            OwnTarget<V4, T> const& ow,
            ForceAcc<T>& A,
            V4 const& pj,
            V4 const& vj,
            V4 const& tj,
            V4 const& bj)
        {
            V4 const& pi = ow.pi;
            V4 const& vi = ow.vi;
            V4 const& ti = ow.ti;
            V4 const& bi = ow.bi;
            T const rx = pi.x - pj.x;
            T const ry = pi.y - pj.y;
            T const rz = pi.z - pj.z;
            T const r2 = dot3(rx, ry, rz, rx, ry, rz);
            T const invR = invDistance(r2);
            T const r = r2 * invR;
            T const si = slopeOverR<K>(r, invR, ow.hk);
            T sj = si; // equal smoothing lengths give the same factor
            if(vj.w != vi.w)
                sj = slopeOverR<K>(r, invR, hconstFromInv<K, T>(rcpT(vj.w)));
            T const mj = pj.w;
            T const vx = vi.x - vj.x, vy = vi.y - vj.y, vz = vi.z - vj.z;
            T const vr = dot3(vx, vy, vz, rx, ry, rz);
            T const msi = mj * si;
            // Isotropic pressure gradient (HydroForces.hpp:155-166).
            T fs = fmaT(ti.y, si, tj.y * sj);
            T const cb = ow.hc + T(0.5) * tj.z; // mean signal speed
            if(ow.av)
            {
                // branch-free: mu = 0 (no viscosity) for receding pairs
                T const vn = vr < T(0) ? vr : T(0);
                T const hb = ow.hh + T(0.5) * vj.w;
                T const mu = hb * vn * rcpT(fmaT(ow.eps * hb, hb, r2));
                // Pi_ij (s_i + s_j)/2: the halves of the means 1/rho_ij and s_ij cancel
                T const Pi = mu * fmaT(ow.beta, mu, -ow.alpha * cb) * rcpT(ti.x + tj.x);
                T const g = mulRn(Pi, addRn(si, sj));
                fs += g;
                A.duav.addProduct(mj * g, vr); // twice the heating
            }
            T const f = -mj * fs;
            A.D.addProduct(msi, vr);
            T const w = vr * invR;
            T const vs = fmaT(-ow.beta, w < T(0) ? w : T(0), T(2) * cb);
            A.vsig = vs > A.vsig ? vs : A.vsig;
            if constexpr(PH >= 2)
            {
                T const dBx = bj.x - bi.x, dBy = bj.y - bi.y, dBz = bj.z - bi.z;
                T const Bir = dot3(bi.x, bi.y, bi.z, rx, ry, rz);
                T const dBr = dot3(dBx, dBy, dBz, rx, ry, rz);
                T const cj = mj * tj.w * sj * (Bir + dBr);
                T fx = f * rx, fy = f * ry, fz = f * rz;
                if(ow.tensile)
                {
                    // stress + Borve: c_i B_i + c_j B_j - B_i (c_i + c_j) = c_j (B_j - B_i)
                    fx = fmaT(cj, dBx, fx);
                    fy = fmaT(cj, dBy, fy);
                    fz = fmaT(cj, dBz, fz);
                }
                else
                {
                    T const ci = msi * Bir * ti.w;
                    fx = fmaT(cj, bj.x, fmaT(ci, bi.x, fx));
                    fy = fmaT(cj, bj.y, fmaT(ci, bi.y, fy));
                    fz = fmaT(cj, bj.z, fmaT(ci, bi.z, fz));
                }
                A.ax.add(fx);
                A.ay.add(fy);
                A.az.add(fz);
                // the large parts of (B_i.r) v_ij and B_i (v_ij.r) cancel here, pair by
                // pair, before any sum rounds them
                A.tx.addProduct(msi, fmaT(Bir, vx, -(vr * bi.x)));
                A.ty.addProduct(msi, fmaT(Bir, vy, -(vr * bi.y)));
                A.tz.addProduct(msi, fmaT(Bir, vz, -(vr * bi.z)));
                if(ow.dedner)
                {
                    // rho_i^2 * m_j (psi_i/rho_i^2 s_i + psi_j/rho_j^2 s_j) r
                    T const g = ow.rho2i * mj * fmaT(bi.w, si, bj.w * sj);
                    A.tx.addProduct(g, rx);
                    A.ty.addProduct(g, ry);
                    A.tz.addProduct(g, rz);
                }
                A.divb.addProduct(msi, dBr); // minus m_j s_i (B_i - B_j).r
            }
            else
            {
                A.ax.addProduct(f, rx);
                A.ay.addProduct(f, ry);
                A.az.addProduct(f, rz);
            }
        }

        //! The sums of one target, in FP64.
        struct ForceSums
        {
            double a[3], D, duav, t[3], divb, vsig;
        };

        //! FP64 epilogue of one target: derivatives and its CFL time step.  Roundings are
        //! spelled out (see fmaT): the one-lane and the eight-lane kernel each hold a copy.
        template<int PH>
        __device__ __forceinline__ double forceEpilogue(
            DevCtx const& c,
            PhysArgs const& pa,
            uint32_t t,
            int box,
            ForceSums const& A,
            bool dedner)
        {
            double const rho = c.cur.rho[t];
            double const h = c.cur.h[t];
            double const pr2 = (pa.gamma - 1.0) * c.cur.u[t] / rho; // P_i / rho_i^2
            double const* const a = A.a;
            double const Dv = A.D;
            c.d.dudt[t] = fmaT(pr2, Dv, A.duav);
            if constexpr(PH >= 2)
            {
                double const psi = c.cur.psi[t];
                double const* const tv = A.t;
                double const invRho = 1.0 / rho;
                double const divB = -invRho * A.divb;
                double const divv = -invRho * Dv;
                double const ch = __longlong_as_double(static_cast<long long>(c.bs.chBits[box]));
                // dB/dt = -(1/rho) T_induction - rho grad(psi); T carries rho^2 grad(psi)/rho.
#pragma unroll
                for(int q = 0; q < 3; ++q)
                    c.d.dBdt[q][t] = -invRho * tv[q];
                c.d.divB[t] = divB;
                double const decay = psi * pa.sigma * ch / h;
                c.d.dpsidt[t] = dedner ? fmaT(-0.5 * psi, divv, fmaT(-ch * ch, divB, -decay)) : 0.0;
            }
#pragma unroll
            for(int q = 0; q < 3; ++q)
                c.d.dvdt[q][t] = a[q];
            double dt = pa.cfl * h / A.vsig;
            double const amag = sqrt(dot3(a[0], a[1], a[2], a[0], a[1], a[2]));
            if(amag > 0.0 && pa.cflForce > 0.0)
                dt = fmin(dt, pa.cflForce * sqrt(h / amag));
            return dt;
        }

        //! Force pass; the records of the next entry are in flight while the
        //! current one is used.
        template<int K, typename T, int PH, int MINB, bool kSmall = false>
        __global__ void __launch_bounds__(kThreads, MINB) kForce(DevCtx c, PhysArgs pa)
        {
            using V4 = typename PairCfg<T>::V4;
            constexpr bool kMhd = PH >= 2;
            Records<V4, T> const rec = records<T>(c);
            constexpr int S = kSmall ? kWide : kLanes<T>;
            uint32_t const sub = threadIdx.x & uint32_t(S - 1);
            uint32_t const t = (blockIdx.x * kThreads + threadIdx.x) / S;
            bool const act = t < c.n && isTarget(c.cur.role[t]);
            int const myBox = act ? c.cur.box[t] : -1;
            bool const av = (PH == 1) || (PH == 3) || (PH == 2 && (pa.physics & SPH_PHYS_AV));
            bool const dedner = (PH == 3) || (PH == 2 && (pa.physics & SPH_PHYS_DEDNER));
            ForceAcc<T> A;
            A.vsig = T(0);
            if(act)
            {
                OwnTarget<V4, T> const own = loadOwn<K, T, PH>(rec, pa, t);
                ImageShift<T> const shift(c, myBox);
                A.vsig = own.ti.z;
                V4 npm{}, nfv{}, nft{}, nfb{};
                uint32_t entry = 0; // the fetched one
                auto fetch = [&](uint32_t e)
                {
                    if(!checkIndex((e >> 5) < c.n, c.status, kChkRowEntry))
                        e = 0;
                    uint32_t const j = e >> 5;
                    entry = e;
                    npm = ld4(rec.pm + j);
                    nfv = ld4(rec.fv + j);
                    nft = ld4(rec.ft + j);
                    if constexpr(kMhd)
                        nfb = ld4(rec.fb + j);
                };
                auto term = [&](uint32_t next)
                {
                    V4 const pj = shift.at(npm, entry), vj = nfv, tj = nft, bj = nfb;
                    fetch(next);
                    pairTerm<K, T, PH>(own, A, pj, vj, tj, bj);
                };
                auto fold = [&]()
                {
                    A.ax.fold();
                    A.ay.fold();
                    A.az.fold();
                    A.D.fold();
                    if(av)
                        A.duav.fold();
                    if constexpr(kMhd)
                    {
                        A.tx.fold();
                        A.ty.fold();
                        A.tz.fold();
                        A.divb.fold();
                    }
                };
                uint32_t const n = min(c.lists.rowLen[t], c.lists.cap);
                uint32_t const* const row = c.lists.list + rowStart<T>(size_t(t), size_t(c.lists.cap));
                uint32_t const any = packEntry(t, kCentreSlot);
                if constexpr(kSmall)
                    walkRowWide(
                        row, n, sub, any, fetch, term,
                        [&](int blocks, uint32_t lanes)
                        {
                            foldBlocks(A.ax, blocks, lanes);
                            foldBlocks(A.ay, blocks, lanes);
                            foldBlocks(A.az, blocks, lanes);
                            foldBlocks(A.D, blocks, lanes);
                            if(av)
                                foldBlocks(A.duav, blocks, lanes);
                            if constexpr(kMhd)
                            {
                                foldBlocks(A.tx, blocks, lanes);
                                foldBlocks(A.ty, blocks, lanes);
                                foldBlocks(A.tz, blocks, lanes);
                                foldBlocks(A.divb, blocks, lanes);
                            }
                        });
                else
                    walkRow<T, S>(row, n, sub, any, fetch, term, fold);
            }
            // kSmall: every lane holds the folded sums already
            constexpr int kSum = kSmall ? 1 : S;
            ForceSums s{};
            s.a[0] = laneSum<kSum>(A.ax.value());
            s.a[1] = laneSum<kSum>(A.ay.value());
            s.a[2] = laneSum<kSum>(A.az.value());
            s.D = laneSum<kSum>(A.D.value());
            if(av)
                s.duav = 0.5 * laneSum<kSum>(A.duav.value());
            if constexpr(kMhd)
            {
                s.t[0] = laneSum<kSum>(A.tx.value());
                s.t[1] = laneSum<kSum>(A.ty.value());
                s.t[2] = laneSum<kSum>(A.tz.value());
                s.divb = -laneSum<kSum>(A.divb.value());
            }
#pragma unroll
            for(int o = 1; o < S; o <<= 1)
            {
                T const v = __shfl_xor_sync(0xffffffffu, A.vsig, o);
                A.vsig = v > A.vsig ? v : A.vsig;
            }
            s.vsig = double(A.vsig);
            double dtLocal = 1e300;
            if(act && sub == 0)
                dtLocal = forceEpilogue<PH>(c, pa, t, myBox, s, dedner);
            boxMin(c.bs.dtBits, myBox, act && sub == 0, dtLocal);
        }

        // ---- launch-shape variants -------------------------------------------
        // force FP32: 4 or 5 blocks/SM (SPMHD default 4, hydro default 5); force
        // FP64: 3.  Variant 0 is the default.
        constexpr int kForceVariants32 = 2, kForceVariants64 = 1;

        //! Blocks of a pass with this many lanes per target.
        unsigned rowBlocks(DevCtx const& c, int lanes)
        {
            return unsigned((uint64_t(c.n) * uint64_t(lanes) + kThreads - 1) / kThreads);
        }

        //! Particle counts up to which the FP32 passes use kWide lanes per target:
        //! below them one lane per target leaves most warp slots empty and the pass
        //! waits for its longest row.  The fold of every block by every lane costs
        //! 8 x 8 instructions per sum and round, so the line lies lower the more sums
        //! a pass has.  One lane -> eight, ms:
        //!   density (with the neighbour build)  Sod 2.3 k 0.051 -> 0.043, 18 k 0.093 ->
        //!     0.084, 36 k 0.090 -> 0.087; Orszag-Tang 26 k 0.083 -> 0.075, 37 k 0.085 ->
        //!     0.081, 45 k 0.092 -> 0.092, 54 k 0.102 -> 0.104, 66 k 0.112 -> 0.117
        //!   hydro force  Sod 2.3 k 0.023 -> 0.012, 18 k 0.027 -> 0.024, 22 k 0.028 ->
        //!     0.025, 26 k 0.029 -> 0.031, 31 k 0.029 -> 0.033, 36 k 0.029 -> 0.037
        //!   SPMHD force  Orszag-Tang 4 k 0.032 -> 0.020, 8.1 k 0.032 -> 0.024, 9.2 k
        //!     0.032 -> 0.024, 10 k 0.031 -> 0.032, 12 k 0.032 -> 0.035, 16 k 0.031 -> 0.038
        //! Each line (256, 128 and 64 targets for each of the 148 SMs) lies on the gaining
        //! side of its change of sign: 45 k, 22 to 26 k and 9.2 to 10 k.
        constexpr uint32_t kWideDensity = 148 * 256, kWideHydro = 148 * 128, kWideMhd = 148 * 64;

        template<int K, typename T, int PH>
        void forceLaunch(DevCtx const& c, PhysArgs const& pa, int variant, cudaStream_t s)
        {
            if(!c.n)
                return;
            if constexpr(sizeof(T) == 4)
            {
                // variant 0: SPMHD 4 blocks/SM (128 registers), hydro 5; variant 1 the other
                constexpr int a = PH >= 2 ? 4 : 5, b = PH >= 2 ? 5 : 4;
                unsigned const wide = rowBlocks(c, kWide), narrow = rowBlocks(c, kLanes<T>);
                bool const small = c.n <= (PH >= 2 ? kWideMhd : kWideHydro);
                if(small && variant == 1)
                    kForce<K, T, PH, b, true><<<wide, kThreads, 0, s>>>(c, pa);
                else if(small)
                    kForce<K, T, PH, a, true><<<wide, kThreads, 0, s>>>(c, pa);
                else if(variant == 1)
                    kForce<K, T, PH, b><<<narrow, kThreads, 0, s>>>(c, pa);
                else
                    kForce<K, T, PH, a><<<narrow, kThreads, 0, s>>>(c, pa);
            }
            else
                kForce<K, T, PH, 3><<<rowBlocks(c, kLanes<T>), kThreads, 0, s>>>(c, pa);
            countLaunches(1);
        }

        template<int K, typename T>
        void forceOne(DevCtx const& c, PhysArgs const& pa, int variant, cudaStream_t s)
        {
            uint32_t const full = SPH_PHYS_MHD | SPH_PHYS_AV | SPH_PHYS_DEDNER | SPH_PHYS_TENSILE;
            if((pa.physics & full) == full)
                forceLaunch<K, T, 3>(c, pa, variant, s);
            else if(pa.physics & SPH_PHYS_MHD)
                forceLaunch<K, T, 2>(c, pa, variant, s);
            else if(pa.physics & SPH_PHYS_AV)
                forceLaunch<K, T, 1>(c, pa, variant, s);
            else
                forceLaunch<K, T, 0>(c, pa, variant, s);
        }

        template<int K, typename T>
        void densityOne(DevCtx const& c, PhysArgs const& pa, cudaStream_t s)
        {
            if(!c.n)
                return;
            if(sizeof(T) == 4 && c.n <= kWideDensity)
                kDensity<K, float, true><<<rowBlocks(c, kWide), kThreads, 0, s>>>(c, pa);
            else
                kDensity<K, T, false><<<rowBlocks(c, kLanes<T>), kThreads, 0, s>>>(c, pa);
            countLaunches(1);
        }

        template<typename T>
        void densityK(DevCtx const& c, PhysArgs const& pa, int kernel, cudaStream_t s)
        {
            if(kernel == SPH_KERNEL_QUINTIC)
                densityOne<SPH_KERNEL_QUINTIC, T>(c, pa, s);
            else if(kernel == SPH_KERNEL_WENDLAND_C2)
                densityOne<SPH_KERNEL_WENDLAND_C2, T>(c, pa, s);
            else
                densityOne<SPH_KERNEL_CUBIC, T>(c, pa, s);
        }

        template<typename T>
        void forceK(DevCtx const& c, PhysArgs const& pa, int kernel, int variant, cudaStream_t s)
        {
            if(kernel == SPH_KERNEL_QUINTIC)
                forceOne<SPH_KERNEL_QUINTIC, T>(c, pa, variant, s);
            else if(kernel == SPH_KERNEL_WENDLAND_C2)
                forceOne<SPH_KERNEL_WENDLAND_C2, T>(c, pa, variant, s);
            else
                forceOne<SPH_KERNEL_CUBIC, T>(c, pa, variant, s);
        }

        //! The gathers want the whole unified array as L1.
        template<typename F>
        void preferL1(F* f)
        {
            cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, 0);
        }

        template<int K, int PH>
        void configureForceK()
        {
            preferL1(kForce<K, float, PH, 4, true>);
            preferL1(kForce<K, float, PH, 5, true>);
            preferL1(kForce<K, float, PH, 4>);
            preferL1(kForce<K, float, PH, 5>);
            preferL1(kForce<K, double, PH, 3>);
        }

        template<int K>
        void configureK()
        {
            preferL1(kDensity<K, float, false>);
            preferL1(kDensity<K, float, true>);
            preferL1(kDensity<K, double, false>);
            configureForceK<K, 0>();
            configureForceK<K, 1>();
            configureForceK<K, 2>();
            configureForceK<K, 3>();
        }
    } // namespace

    void configurePairKernels()
    {
        static bool done = false;
        if(done)
            return;
        configureNeighbourKernels();
        configureK<SPH_KERNEL_CUBIC>();
        configureK<SPH_KERNEL_QUINTIC>();
        configureK<SPH_KERNEL_WENDLAND_C2>();
        done = true;
    }

    int forceVariants(int precision)
    {
        return precision == SPH_PREC_FP64 ? kForceVariants64 : kForceVariants32;
    }

    int forceBlocksPerSm(int precision, int physics, int variant)
    {
        if(precision == SPH_PREC_FP64)
            return 3;
        bool const mhd = physics & SPH_PHYS_MHD;
        return (variant == 1) == mhd ? 5 : 4;
    }

    void launchDensity(DevCtx const& c, PhysArgs const& pa, int kernel, int precision, cudaStream_t s)
    {
        if(precision == SPH_PREC_FP64)
            densityK<double>(c, pa, kernel, s);
        else
            densityK<float>(c, pa, kernel, s);
    }

    void launchForce(DevCtx const& c, PhysArgs const& pa, int kernel, int precision, int variant, cudaStream_t s)
    {
        if(precision == SPH_PREC_FP64)
            forceK<double>(c, pa, kernel, variant, s);
        else
            forceK<float>(c, pa, kernel, variant, s);
    }
} // namespace sph
