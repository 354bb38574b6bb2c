// Shared by the neighbour build and the pair passes: record access, unfused
// and paired arithmetic, accumulators, warp reductions.
#pragma once

#include "sph_launch.hpp"

namespace sph
{
    constexpr int kBlock = 8; //!< terms per summation block of a row

    template<typename T>
    struct PairCfg;
    template<>
    struct PairCfg<float>
    {
        using V4 = float4;
        static constexpr int kStageBatch = 2; //!< staged positions per lane with loads in flight
    };
    template<>
    struct PairCfg<double>
    {
        using V4 = D4;
        static constexpr int kStageBatch = 2;
    };

    template<typename T>
    __device__ __forceinline__ Records<typename PairCfg<T>::V4, T> records(DevCtx const& c);
    template<>
    __device__ __forceinline__ Records<float4, float> records<float>(DevCtx const& c)
    {
        return c.r32;
    }
    template<>
    __device__ __forceinline__ Records<D4, double> records<double>(DevCtx const& c)
    {
        return c.r64;
    }

    //! Paired FP32 arithmetic (sm_100 f32x2) that rounds like the reference's
    //! unfused scalar x, y, z sum.  A paired multiply feeding a paired add is
    //! contracted into a fused multiply-add even when both are written in
    //! PTX with an explicit .rn (measured on sm_100a: r^2 then differs from
    //! the scalar __fmul_rn/__fadd_rn sum by one ulp, which moves pairs at
    //! r^2 = R^2 across the cull).  Squares are therefore formed as
    //! fma.rn(a, a, zero) with a zero the compiler cannot see (one computed
    //! from a kernel argument): that is round(a^2) exactly, and an add of
    //! two fused results has nothing left to contract.
    __device__ __forceinline__ float2 add2Rn(float2 a, float2 b)
    {
        unsigned long long r;
        asm("add.rn.f32x2 %0, %1, %2;"
            : "=l"(r)
            : "l"(*reinterpret_cast<unsigned long long const*>(&a)),
              "l"(*reinterpret_cast<unsigned long long const*>(&b)));
        return *reinterpret_cast<float2 const*>(&r);
    }
    __device__ __forceinline__ float2 sq2Rn(float2 a, float2 zero)
    {
        unsigned long long r;
        asm("fma.rn.f32x2 %0, %1, %1, %2;"
            : "=l"(r)
            : "l"(*reinterpret_cast<unsigned long long const*>(&a)),
              "l"(*reinterpret_cast<unsigned long long const*>(&zero)));
        return *reinterpret_cast<float2 const*>(&r);
    }
    //! The hardware's approximate reciprocal and reciprocal square root, without
    //! the rescaling of denormal arguments that __fdividef and rsqrtf add: the
    //! callers' arguments are normal.
    __device__ __forceinline__ float rcpApprox(float a)
    {
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
        return r;
    }
    __device__ __forceinline__ float rsqrtApprox(float a)
    {
        float r;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
        return r;
    }
    //! A run-time zero: R * 0 with R a finite kernel argument.  IEEE
    //! arithmetic does not let the compiler fold it (R could be NaN or
    //! infinite), so it stays opaque to contraction.
    __device__ __forceinline__ float2 opaqueZero2(float R)
    {
        float const z = __fmul_rn(R, 0.0f);
        return make_float2(z, z);
    }

    //! 1/r from r^2.  At r = 0: FP64 zero; FP32 large and finite, where the
    //! callers' products (r = r^2/r, the kernel slope at r = 0) are zero.
    __device__ __forceinline__ float invDistance(float r2)
    {
        return rsqrtApprox(fmaxf(r2, 1e-37f));
    }
    __device__ __forceinline__ double invDistance(double r2)
    {
        return r2 > 0.0 ? rsqrt(r2) : 0.0;
    }
    //! Reciprocal in the pair precision: approximate in FP32 (the pair terms
    //! carry no tighter requirement), IEEE in FP64.
    __device__ __forceinline__ float rcpT(float x)
    {
        return rcpApprox(x);
    }
    __device__ __forceinline__ double rcpT(double x)
    {
        return 1.0 / x;
    }

    //! dW/dr(r, h) / r: gradWScalar, with the FP32 kernels' zero beyond the
    //! support (and at r = 0) coming from the clamped shapes themselves.
    template<int K>
    __device__ __forceinline__ float slopeOverR(float r, float invR, HConst<float> const& c)
    {
        float const x = mulRn(r, c.invh);
        if constexpr(K == SPH_KERNEL_WENDLAND_C2)
        {
            float const t = fmaxf(fmaT(-0.5f, x, 1.f), 0.f);
            return c.dwnorm * (-5.f * x * t) * (t * t) * invR;
        }
        else if constexpr(K == SPH_KERNEL_CUBIC)
        {
            float const t = fmaxf(2.f - x, 0.f);
            return c.dwnorm * (x < 1.f ? fmaT(2.25f, x, -3.f) * x : -0.75f * t * t) * invR;
        }
        else
            return gradWScalar<K, float>(r, invR, c);
    }
    template<int K>
    __device__ __forceinline__ double slopeOverR(double r, double invR, HConst<double> const& c)
    {
        return gradWScalar<K, double>(r, invR, c);
    }

    template<typename T>
    __device__ __forceinline__ T edgeOf(BoxDev const& B, int a);
    template<>
    __device__ __forceinline__ float edgeOf<float>(BoxDev const& B, int a)
    {
        return B.edgef[a];
    }
    template<>
    __device__ __forceinline__ double edgeOf<double>(BoxDev const& B, int a)
    {
        return B.edge[a];
    }

    //! Accumulator: FP32 compensated (CompAcc + block partial) or FP64 plain.
    template<typename T>
    struct Acc;
    template<>
    struct Acc<float>
    {
        CompAcc c;
        float part = 0.f;
        __device__ __forceinline__ void add(float x)
        {
            part += x;
        }
        __device__ __forceinline__ void addProduct(float a, float b)
        {
            part = fmaT(a, b, part);
        }
        __device__ __forceinline__ void fold()
        {
            c.fold(part);
            part = 0.f;
        }
        __device__ __forceinline__ double value() const
        {
            return c.value();
        }
    };
    template<>
    struct Acc<double>
    {
        double s = 0.0;
        __device__ __forceinline__ void add(double x)
        {
            s += x;
        }
        __device__ __forceinline__ void addProduct(double a, double b)
        {
            s = fmaT(a, b, s);
        }
        __device__ __forceinline__ void fold()
        {
        }
        __device__ __forceinline__ double value() const
        {
            return s;
        }
    };

    __device__ __forceinline__ uint32_t warpMaxU(uint32_t v)
    {
#pragma unroll
        for(int o = 16; o > 0; o >>= 1)
            v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    }
    __device__ __forceinline__ unsigned long long warpSumU64(unsigned long long v)
    {
#pragma unroll
        for(int o = 16; o > 0; o >>= 1)
            v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    }
    __device__ __forceinline__ double warpMaxD(double v)
    {
#pragma unroll
        for(int o = 16; o > 0; o >>= 1)
            v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    }
    __device__ __forceinline__ double warpMinD(double v)
    {
#pragma unroll
        for(int o = 16; o > 0; o >>= 1)
            v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    }

    //! Minimum and maximum over the warp (FP32: one sm_100 reduction instruction
    //! instead of five shuffles and compares).
    __device__ __forceinline__ float warpMinT(float v)
    {
        float r;
        asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
        return r;
    }
    __device__ __forceinline__ float warpMaxT(float v)
    {
        float r;
        asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
        return r;
    }
    __device__ __forceinline__ double warpMinT(double v)
    {
        return warpMinD(v);
    }
    __device__ __forceinline__ double warpMaxT(double v)
    {
        return warpMaxD(v);
    }
} // namespace sph
