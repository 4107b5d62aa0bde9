/*
 * tg_f32x2.cuh -- two binary32 values in one 64-bit register pair.
 *
 * sm_100 executes one add, multiply or fused multiply-add on both values per
 * instruction (add/mul/fma.rn.f32x2).  Each half is the IEEE operation, so
 * results are those of two scalar instructions; what it saves is issue slots,
 * which bound the tracking step: measured on one B200, a stream of these runs
 * at 124 fused multiply-adds per clock and SM, the rate of the scalar form,
 * from half the instructions.  Taking a pair apart is free (its halves are
 * registers); putting one together is free where the producers can write
 * neighbouring registers.
 */
#ifndef TG_F32X2_CUH
#define TG_F32X2_CUH

namespace tg {

struct F2 {
    unsigned long long v;
};

__device__ __forceinline__ F2 f2(float lo, float hi)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}

__device__ __forceinline__ F2 f2(float both) { return f2(both, both); }

__device__ __forceinline__ float lo(F2 a)
{
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return x;
}

__device__ __forceinline__ float hi(F2 a)
{
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return y;
}

__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

__device__ __forceinline__ F2 mul2(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

}  // namespace tg

#endif  // TG_F32X2_CUH
