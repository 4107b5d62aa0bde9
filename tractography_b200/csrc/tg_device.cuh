/*
 * tg_device.cuh -- per-step device arithmetic of the streamline tracker.
 *
 * Implements, for sm_100a, the reference tracking kernel's per-step work
 * (tractography/tracking.py:121-147): image-domain test (domain.py:358-382),
 * nearest-voxel field gather (field.py:88-114), local models
 * (local.py:91-120 spherical harmonics, local.py:212-230 tensor),
 * orientation updates (algorithm.py:83-112 Transport, 198-228 Diffusion),
 * the spherical exponential map (core.cl:101-109) and the random streams
 * (core.cl:180-245 MWC64X, plus a counter-based Philox4x32-10 mode).
 *
 * Every floating-point operation is an IEEE binary32 operation in a fixed
 * order with explicit fmaf; the translation unit is compiled with
 * -fmad=false so nothing is contracted behind our back.  This is the same
 * sequence the CPU oracle performs, which makes GPU and CPU results equal
 * bit for bit (the Transport update amplifies last-bit differences into
 * whole voxels, so tolerance-level agreement would not be reproducible).
 */
#ifndef TG_DEVICE_CUH
#define TG_DEVICE_CUH

#include <cstdint>

#include "tg_f32x2.cuh"
#include "tg_fmath.h"

namespace tg {

constexpr float kSoftmaxScale = 100.0f;   // local.py:17
constexpr float kSoftmaxInvScale = 0x1.47ae14p-7f;   // 1/100 rounded

template <int LMAX>
__device__ __forceinline__ void sh_eval(const float* c, float ct, float st, float cp, float sp,
                                        float* val, float* dth, float* dph);
template <int LMAX>
__device__ __forceinline__ void sh_basis(float ct, float st, float cp, float sp, float* Y);
template <int LMAX>
__device__ __forceinline__ void sh_fold(const float* c, float* a);
template <int LMAX>
__device__ __forceinline__ void sh_eval_folded(const float* a, float ct, float st, float cp, float sp,
                                               float* val, float* dth, float* dph);

}  // namespace tg

#include "tg_sh_eval.cuh"
#include "tg_sh_folded.cuh"

namespace tg {

enum { kModelSH = 0, kModelDTI = 1 };
enum { kTransport = 0, kDiffusion = 1 };
enum { kRngMWC64X = 0, kRngPhilox = 1 };

__host__ __device__ constexpr int n_coef_full(int lmax) { return (lmax + 1) * (lmax + 2) / 2; }

// OpenCL float max(): y if x < y else x.
__device__ __forceinline__ float cl_max(float x, float y) { return (x < y) ? y : x; }

// ---------------------------------------------------------------- RNG

struct Mwc {
    uint32_t x, c;
};

__device__ __forceinline__ uint32_t mwc64x(Mwc& s)
{
    constexpr uint32_t A = 4294883355u;
    const uint32_t res = s.x ^ s.c;
    const uint64_t next = (uint64_t)s.x * A + s.c;     // at most (2^32 - 1) A + 2^32 - 1 < 2^64
    s.x = (uint32_t)next;
    s.c = (uint32_t)(next >> 32);
    return res;
}

__device__ __forceinline__ uint32_t rng_mix32(uint32_t v)
{
    v ^= v >> 16;
    v *= 0x7feb352du;
    v ^= v >> 15;
    v *= 0x846ca68bu;
    v ^= v >> 16;
    return v;
}

__device__ __forceinline__ Mwc rng_init(uint32_t seed, uint32_t id)
{
    Mwc s;
    uint32_t x = rng_mix32(seed ^ (id + 0x9e3779b9u));
    s.x = x < 1u ? 1u : x;
    s.c = rng_mix32(seed + id * 0x85ebca6bu) % 4294883355u;
    return s;
}

__device__ __forceinline__ float randu(Mwc& s)
{
    return (float)(mwc64x(s) >> 8) * 0x1p-24f;
}

__device__ __forceinline__ uint32_t randi(Mwc& s, uint32_t max)
{
    return (uint32_t)(randu(s) * (float)max);
}

__device__ __forceinline__ float randn(Mwc& s)
{
    float n = randu(s);
    while (n <= 0.0f) n = randu(s);   // terminates: 2^-24 resolution, MWC64X period ~2^63
    const float radius = sqrtf(-2.0f * tgm_log_pos(n));
    // cos(2 pi randu): the same draw, as its 24-bit integer
    return radius * tgm_cos2pi_u24(mwc64x(s) >> 8);
}

// tgm_log_pos of both halves.
__device__ __forceinline__ F2 log_pos2(F2 x)
{
    const uint32_t xa = __float_as_uint(lo(x)), xb = __float_as_uint(hi(x));
    const int ea = (int)(xa - 0x3f3504f3u) >> 23, eb = (int)(xb - 0x3f3504f3u) >> 23;
    const F2 m = f2(__uint_as_float(xa - ((uint32_t)ea << 23)), __uint_as_float(xb - ((uint32_t)eb << 23)));
    const F2 f = add2(m, f2(-1.0f));
    F2 q = f2(-0x1.38b4ccp-4f);
    q = fma2(q, f, f2(0x1.055b46p-3f));
    q = fma2(q, f, f2(-0x1.0d8552p-3f));
    q = fma2(q, f, f2(0x1.22da22p-3f));
    q = fma2(q, f, f2(-0x1.547244p-3f));
    q = fma2(q, f, f2(0x1.99a008p-3f));
    q = fma2(q, f, f2(-0x1.000228p-2f));
    q = fma2(q, f, f2(0x1.555554p-2f));
    const F2 t = fma2(f, q, f2(-0.5f));
    const F2 logm = fma2(mul2(f, f), t, f);
    const F2 ef = f2((float)ea, (float)eb);
    return fma2(ef, f2(TGM_LN2_HI), fma2(ef, f2(TGM_LN2_LO), logm));
}

// tgm_cos2pi_u24 of the upper 24 bits of two draws.  With v = w + 2^29 the
// quarter turns are q = v >> 30 (mod 4) and the remainder is the low 30 bits of
// w, sign-extended; q's bit 0 is v's bit 30, and the sign, bit 1 of q + 1, is
// bit 31 of v + 2^30.
__device__ __forceinline__ F2 cos2pi_2(uint32_t wa, uint32_t wb)
{
    const int ra = (int)(wa << 2) >> 10, rb = (int)(wb << 2) >> 10;
    const F2 t = mul2(f2((float)ra, (float)rb), f2(TGM_TWO_PI_2M24));
    const F2 t2 = mul2(t, t);
    F2 ps = f2(-0x1.9943e0p-13f);
    ps = fma2(ps, t2, f2(0x1.11073ap-7f));
    ps = fma2(ps, t2, f2(-0x1.555546p-3f));
    const F2 st = fma2(mul2(t, t2), ps, t);
    F2 pc = f2(0x1.9916a0p-16f);
    pc = fma2(pc, t2, f2(-0x1.6c07f2p-10f));
    pc = fma2(pc, t2, f2(0x1.55553cp-5f));
    pc = fma2(pc, t2, f2(-0.5f));
    const F2 ct = fma2(t2, pc, f2(1.0f));
    const uint32_t va = wa + 0x20000000u, vb = wb + 0x20000000u;
    const float ca = (va & 0x40000000u) ? lo(st) : lo(ct), cb = (vb & 0x40000000u) ? hi(st) : hi(ct);
    return f2(__uint_as_float(__float_as_uint(ca) ^ ((va + 0x40000000u) & 0x80000000u)),
              __uint_as_float(__float_as_uint(cb) ^ ((vb + 0x40000000u) & 0x80000000u)));
}

// Square roots of both halves, correctly rounded, for values in [2^-24, 64]
// (-2 log u of Box-Muller's uniforms): one Newton step with a fused residual
// from the hardware's approximate reciprocal root (Markstein 1990, as in
// tgm_rcp).  Equal to sqrtf on all 2^24 - 1 such values and on all mantissas of
// two neighbouring exponents (checked exhaustively on B200): 6 instructions for
// both instead of 20.
__device__ __forceinline__ F2 sqrt_pos2(F2 x)
{
    float ya, yb;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(ya) : "f"(lo(x)));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yb) : "f"(hi(x)));
    const F2 y = f2(ya, yb);
    const F2 g = mul2(x, y), h = mul2(y, f2(0.5f));
    const F2 r = fma2(f2(-lo(g), -hi(g)), g, x);
    return fma2(r, h, g);
}

// The same for one value, or a zero (u = 1, which the counter-based draws
// reach), which is its own root.
__device__ __forceinline__ float sqrt_pos(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    const float g = x * y;
    const float root = fmaf(fmaf(-g, g, x), 0.5f * y, g);
    return x > 0.0f ? root : x;
}

// Two draws of randn, evaluated together: one pass of pairwise arithmetic
// instead of two, and one test for randn's rejection of u <= 0, which happens
// once in 2^23 pairs (the draws then move up and the next ones follow).
// 90 instructions measured alone, against 141 for two calls of randn (100k SDE
// seeds: tracking kernel 558 ms, 576 ms with the same code one value at a time).
__device__ __forceinline__ void randn2(Mwc& s, float* n1, float* n2)
{
    uint32_t ua = mwc64x(s), wa = mwc64x(s), ub = mwc64x(s), wb = mwc64x(s);
    if (min(ua, ub) < 256u) {
        while (ua < 256u) {
            ua = wa;
            wa = ub;
            ub = wb;
            wb = mwc64x(s);
        }
        while (ub < 256u) {
            ub = wb;
            wb = mwc64x(s);
        }
    }
    const F2 u = mul2(f2((float)(ua >> 8), (float)(ub >> 8)), f2(0x1p-24f));
    const F2 n = mul2(sqrt_pos2(mul2(f2(-2.0f), log_pos2(u))), cos2pi_2(wa, wb));
    *n1 = lo(n);
    *n2 = hi(n);
}

__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k)
{
#pragma unroll
    for (int round = 0; round < 10; ++round) {
        const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
        k.x += 0x9E3779B9u;
        k.y += 0xBB67AE85u;
    }
    return c;
}

__device__ __forceinline__ void philox_normal2(uint64_t key, uint64_t index, uint32_t step,
                                               float* n1, float* n2)
{
    const uint4 w = philox4x32_10(make_uint4((uint32_t)index, (uint32_t)(index >> 32), step, 0x5eedu),
                                  make_uint2((uint32_t)key, (uint32_t)(key >> 32)));
    const float u1 = (float)((w.x >> 8) + 1u) * 0x1p-24f;
    const float u2 = (float)(w.y >> 8) * 0x1p-24f;
    // sqrtf's bits (sqrt_pos) without its branch, which kept the draw from
    // overlapping the model's evaluation: 2000 seeds at lmax 8 in the
    // dense tracker 1.69 -> 1.60 ms.
    const float radius = sqrt_pos(-2.0f * tgm_log_pos(u1));
    float s, c;
    tgm_sincosf(TGM_TWO_PI * u2, &s, &c);
    *n1 = radius * c;
    *n2 = radius * s;
}

// ----------------------------------------------------------- geometry

struct Frame {
    float ct, st, cp, sp;
};

// cart2sph (core.cl:142-153) as direction cosines of colatitude/azimuth:
// ct = z/r, st = rho/r, cp = x/rho, sp = y/rho.  Orientations leave the
// exponential map with |o|^2 = 1 within a few ulp; for |r^2 - 1| < 2^-14,
// 1/r = 1.5 - r^2/2 to within 1.4e-9 relative (its expansion about 1), far
// inside binary32 rounding, and 1/rho comes from tgm_rsqrt_pos (rho^2 at
// least 2^-100; nearer the axis from a square root and a division).
// Otherwise both reciprocals come from one division, 1/r = rho q and
// 1/rho = r q with q = 1/(r rho); on the axis (r rho rounds to 0) phi is
// taken as 0.
__device__ __forceinline__ Frame frame_of(float x, float y, float z)
{
    Frame f;
    const float rho2 = fmaf(y, y, x * x);
    const float r2 = fmaf(z, z, rho2);
    if (fabsf(r2 - 1.0f) < 0x1p-14f) {
        const float ir = fmaf(-0.5f, r2, 1.5f);
        f.ct = fminf(fmaxf(z * ir, -1.0f), 1.0f);
        if (rho2 >= 0x1p-100f) {
            // 1/rho without a square root or a division; rho = rho2 / rho
            const float irho = tgm_rsqrt_pos(rho2);
            f.st = fminf((rho2 * irho) * ir, 1.0f);
            f.cp = x * irho;
            f.sp = y * irho;
            return f;
        }
        const float rho = sqrtf(rho2);
        f.st = fminf(rho * ir, 1.0f);
        if (rho > 0.0f) {
            const float irho = 1.0f / rho;
            f.cp = x * irho;
            f.sp = y * irho;
        } else {
            f.cp = 1.0f;
            f.sp = 0.0f;
        }
        return f;
    }
    const float r = sqrtf(r2);
    if (r <= 0.0f) {
        f.ct = 1.0f; f.st = 0.0f; f.cp = 1.0f; f.sp = 0.0f;
        return f;
    }
    const float rho = sqrtf(rho2);
    const float rr = r * rho;
    if (rr > 0.0f) {
        const float q = 1.0f / rr;
        const float ir = rho * q, irho = r * q;
        f.ct = fminf(fmaxf(z * ir, -1.0f), 1.0f);
        f.st = fminf(rho * ir, 1.0f);
        f.cp = x * irho;
        f.sp = y * irho;
    } else {
        f.ct = fminf(fmaxf(z / r, -1.0f), 1.0f);
        f.st = 0.0f;
        f.cp = 1.0f;
        f.sp = 0.0f;
    }
    return f;
}

__device__ __forceinline__ float dot4(float4 a, float x, float y, float z, float w)
{
    return fmaf(a.w, w, fmaf(a.z, z, fmaf(a.y, y, a.x * x)));
}

// ------------------------------------------------------------- models

struct ModelValue {
    float value, dtheta, dphi;
    float inv;   // 1 / max(value, 1e-6), the drift's divisor (algorithm.py:98, :216)
};

// core.cl:111-115, log(1 + e^{kx}) / k below kx = 30, else x: the seeding kernel's
// model value (tracking uses tgm_softplus).  tgm_expf, tgm_logf and the two
// divisions in their operations, for the arguments that occur here: 1 + e is
// in [1, 1 + e^30] (and 1 wherever the exponential is below 2^-24, so its
// argument may be capped), and both quotients are one Newton step with a fused
// residual from the reciprocal (Markstein 1990, as in tgm_rcp).  Equal to
// tgm_logf(1 + tgm_expf(kx)) / k on all 2^32 floats (checked exhaustively on B200)
// in half its instructions.
__device__ __forceinline__ float softmax(float x)
{
    const float kx = x * kSoftmaxScale;
    const float y = fminf(fmaxf(kx, -87.0f), 30.0f);
    const float shifted = y * TGM_LOG2E + 0x1.8p+23f;
    const float k = shifted - 0x1.8p+23f;
    float r = fmaf(-k, TGM_LN2_HI, y);
    r = fmaf(-k, TGM_LN2_LO, r);
    float p = 0x1.a01a02p-13f;
    p = fmaf(p, r, 0x1.6c16c2p-10f);
    p = fmaf(p, r, 0x1.111112p-7f);
    p = fmaf(p, r, 0x1.555556p-5f);
    p = fmaf(p, r, 0x1.555556p-3f);
    p = fmaf(p, r, 0.5f);
    p = fmaf(p, r, 1.0f);
    p = fmaf(p, r, 1.0f);
    const float w = 1.0f + p * __uint_as_float((__float_as_uint(shifted) << 23) + 0x3f800000u);
    // m in (sqrt(1/2), sqrt(2)]: the exponent is one more above sqrt(2)
    const uint32_t bits = __float_as_uint(w);
    const uint32_t e = (bits + (0x00800000u - 0x003504f4u)) >> 23;
    const float f = __uint_as_float(bits - (e << 23) + 0x3f800000u) - 1.0f;
    const float d = 2.0f + f;
    const float inv = tgm_rcp(d);
    const float q = f * inv;
    const float s = fmaf(fmaf(-q, d, f), inv, q);
    const float z = s * s;
    float t = 0x1.c71c72p-4f;
    t = fmaf(t, z, 0x1.24924ap-3f);
    t = fmaf(t, z, 0x1.99999ap-3f);
    t = fmaf(t, z, 0x1.555556p-2f);
    const float two_s = s + s;
    const float logm = fmaf(two_s * z, t, two_s);
    const float ef = (float)((int)e - 127);
    const float lg = fmaf(ef, TGM_LN2_HI, fmaf(ef, TGM_LN2_LO, logm));
    const float h = lg * kSoftmaxInvScale;
    return kx < 30.0f ? fmaf(fmaf(-h, kSoftmaxScale, lg), kSoftmaxInvScale, h) : x;
}

// softmax of both halves.
__device__ __forceinline__ F2 softmax2(F2 x)
{
    const F2 kx = mul2(x, f2(kSoftmaxScale));
    const F2 y = f2(fminf(fmaxf(lo(kx), -87.0f), 30.0f), fminf(fmaxf(hi(kx), -87.0f), 30.0f));
    const F2 shifted = add2(mul2(y, f2(TGM_LOG2E)), f2(0x1.8p+23f));
    const F2 nk = mul2(add2(shifted, f2(-0x1.8p+23f)), f2(-1.0f));
    const F2 r = fma2(nk, f2(TGM_LN2_LO), fma2(nk, f2(TGM_LN2_HI), y));
    F2 p = f2(0x1.a01a02p-13f);
    p = fma2(p, r, f2(0x1.6c16c2p-10f));
    p = fma2(p, r, f2(0x1.111112p-7f));
    p = fma2(p, r, f2(0x1.555556p-5f));
    p = fma2(p, r, f2(0x1.555556p-3f));
    p = fma2(p, r, f2(0.5f));
    p = fma2(p, r, f2(1.0f));
    p = fma2(p, r, f2(1.0f));
    const F2 scale = f2(__uint_as_float((__float_as_uint(lo(shifted)) << 23) + 0x3f800000u),
                        __uint_as_float((__float_as_uint(hi(shifted)) << 23) + 0x3f800000u));
    const F2 w = add2(f2(1.0f), mul2(p, scale));
    const uint32_t wa = __float_as_uint(lo(w)), wb = __float_as_uint(hi(w));
    const uint32_t ea = (wa + (0x00800000u - 0x003504f4u)) >> 23, eb = (wb + (0x00800000u - 0x003504f4u)) >> 23;
    const F2 f = add2(f2(__uint_as_float(wa - (ea << 23) + 0x3f800000u), __uint_as_float(wb - (eb << 23) + 0x3f800000u)),
                      f2(-1.0f));
    const F2 d = add2(f2(2.0f), f);
    const F2 inv = f2(tgm_rcp(lo(d)), tgm_rcp(hi(d)));
    const F2 q = mul2(f, inv);
    const F2 s = fma2(fma2(f2(-lo(q), -hi(q)), d, f), inv, q);
    const F2 z = mul2(s, s);
    F2 t = f2(0x1.c71c72p-4f);
    t = fma2(t, z, f2(0x1.24924ap-3f));
    t = fma2(t, z, f2(0x1.99999ap-3f));
    t = fma2(t, z, f2(0x1.555556p-2f));
    const F2 two_s = add2(s, s);
    const F2 logm = fma2(mul2(two_s, z), t, two_s);
    const F2 ef = f2((float)((int)ea - 127), (float)((int)eb - 127));
    const F2 lg = fma2(ef, f2(TGM_LN2_HI), fma2(ef, f2(TGM_LN2_LO), logm));
    const F2 h = mul2(lg, f2(kSoftmaxInvScale));
    const F2 v = fma2(fma2(f2(-lo(h), -hi(h)), f2(kSoftmaxScale), lg), f2(kSoftmaxInvScale), h);
    return f2(lo(kx) < 30.0f ? lo(v) : lo(x), hi(kx) < 30.0f ? hi(v) : hi(x));
}

// local.py:91-120 from folded coefficients (sh_fold): the field the
// trackers read is folded once per voxel when it is created.
template <int LMAX>
__device__ __forceinline__ ModelValue sh_model(const float* folded, const Frame& f)
{
    ModelValue r;
    float raw, d;
    sh_eval_folded<LMAX>(folded, f.ct, f.st, f.cp, f.sp, &raw, &r.dtheta, &r.dphi);
    // local.py:106-118: softplus of the value, derivatives times its slope
    tgm_softplus(raw, kSoftmaxScale, kSoftmaxInvScale, &r.value, &d, &r.inv);
    r.dtheta = r.dtheta * d;
    r.dphi = r.dphi * d;
    return r;
}

__device__ __forceinline__ ModelValue dti_model(const float* m, float x, float y, float z, const Frame& f)
{
    const float dux = fmaf(m[4], z, fmaf(m[3], y, m[0] * x));
    const float duy = fmaf(m[5], z, fmaf(m[1], y, m[3] * x));
    const float duz = fmaf(m[2], z, fmaf(m[5], y, m[4] * x));
    ModelValue r;
    r.value = fmaf(z, duz, fmaf(y, duy, x * dux));
    const float etx = f.ct * f.cp, ety = f.ct * f.sp, etz = -f.st;
    r.dtheta = 2.0f * fmaf(duz, etz, fmaf(duy, ety, dux * etx));
    r.dphi = 2.0f * fmaf(duy, f.cp, dux * (-f.sp));
    r.inv = tgm_rcp(cl_max(r.value, 1e-6f));
    return r;
}

template <int MODEL, int LMAX>
__device__ __forceinline__ ModelValue model_eval(const float* c, float x, float y, float z, const Frame& f)
{
    if constexpr (MODEL == kModelDTI) {
        return dti_model(c, x, y, z, f);
    } else {
        return sh_model<LMAX>(c, f);
    }
}

// --------------------------------------------------------- algorithms

struct AlgoParams {
    float step_size;
    float gamma;
    float noise_variance;
    float scale_drift;   // gamma * step_size
    float scale_noise;   // sqrt(noise_variance * gamma * step_size)
    int32_t rng_mode;
    uint64_t philox_key;
};

// A streamline's random stream: the MWC64X state, or in the counter-based
// mode its index (low word in mwc.x, high word in mwc.c).
struct RngState {
    Mwc mwc;
};

__device__ __forceinline__ RngState rng_state(const AlgoParams& a, Mwc mwc, uint64_t index)
{
    RngState r;
    r.mwc = mwc;
    if (a.rng_mode != kRngMWC64X) {
        r.mwc.x = (uint32_t)index;
        r.mwc.c = (uint32_t)(index >> 32);
    }
    return r;
}

__device__ __forceinline__ void exps2(float& ox, float& oy, float& oz, float tx, float ty, float tz)
{
    const float n2 = fmaf(tz, tz, fmaf(ty, ty, tx * tx));
    if (n2 <= 0.0f) return;
    float c, k;
    if (n2 < 1.0f) {
        // tgm_exps2_factors' two polynomials side by side
        const F2 nn = f2(n2);
        F2 q = f2(0x1.94a4c6p-16f, 0x1.69b0f6p-19f);
        q = fma2(q, nn, f2(-0x1.6beef6p-10f, -0x1.9ffe56p-13f));
        q = fma2(q, nn, f2(0x1.5554e6p-5f, 0x1.1110ecp-7f));
        q = fma2(q, nn, f2(-0x1.fffffep-2f, -0x1.555556p-3f));
        q = fma2(q, nn, f2(1.0f));
        c = lo(q);
        k = hi(q);
    } else {
        tgm_exps2_factors(n2, &c, &k);
    }
    ox = fmaf(tx, k, c * ox);
    oy = fmaf(ty, k, c * oy);
    oz = fmaf(tz, k, c * oz);
}

// f: the frame of (ox, oy, oz); step: updates made before this one (the
// counter-based stream's counter).
template <int MODEL, int LMAX, int ALGO>
__device__ __forceinline__ void update_orientation(const AlgoParams& a, const float* c, const Frame& f,
                                                   float& ox, float& oy, float& oz, RngState& rng, uint32_t step)
{
    const ModelValue mv = model_eval<MODEL, LMAX>(c, ox, oy, oz, f);
    const float etx = f.ct * f.cp, ety = f.ct * f.sp, etz = -f.st;
    const float epx = -f.sp, epy = f.cp;
    const float inv = mv.inv;
    const float gx = fmaf(mv.dphi, epx, mv.dtheta * etx);
    const float gy = fmaf(mv.dphi, epy, mv.dtheta * ety);
    const float gz = mv.dtheta * etz;
    const float dx = gx * inv, dy = gy * inv, dz = gz * inv;
    float tx, ty, tz;
    if constexpr (ALGO == kTransport) {
        tx = a.scale_drift * dx;
        ty = a.scale_drift * dy;
        tz = a.scale_drift * dz;
    } else {
        float nx = 0.0f, ny = 0.0f, nz = 0.0f;
        if (a.noise_variance > 0.0f) {
            float n1, n2;
            if (a.rng_mode == kRngMWC64X) {
                randn2(rng.mwc, &n1, &n2);
            } else {
                philox_normal2(a.philox_key, (uint64_t)rng.mwc.c << 32 | rng.mwc.x, step, &n1, &n2);
            }
            nx = fmaf(n2, epx, n1 * etx);
            ny = fmaf(n2, epy, n1 * ety);
            nz = n1 * etz;
        }
        tx = fmaf(a.scale_noise, nx, a.scale_drift * dx);
        ty = fmaf(a.scale_noise, ny, a.scale_drift * dy);
        tz = fmaf(a.scale_noise, nz, a.scale_drift * dz);
    }
    exps2(ox, oy, oz, tx, ty, tz);
}

template <int MODEL, int LMAX, int ALGO>
__device__ __forceinline__ void update_orientation(const AlgoParams& a, const float* c,
                                                   float& ox, float& oy, float& oz, RngState& rng, uint32_t step)
{
    update_orientation<MODEL, LMAX, ALGO>(a, c, frame_of(ox, oy, oz), ox, oy, oz, rng, step);
}

// tracking.py:343: a track stops on a non-finite orientation or one
// shorter than 0.5.  sqrt is correctly rounded and monotonic, so len < 0.5 is
// len^2 < 0.25, and a finite len^2 has finite components.
__device__ __forceinline__ bool degenerate(float x, float y, float z)
{
    const float len2 = x * x + y * y + z * z;
    if (len2 >= 0.25f && len2 < __int_as_float(0x7f800000)) return false;
    return !(isfinite(x) && isfinite(y) && isfinite(z)) || len2 < 0.25f;
}

// ----------------------------------------------------- domain / field

struct Grid {
    float4 row0, row1, row2;   // inverse affine rows 0..2
    uint32_t nx, ny, nz;
};

// domain.py:358-382: voxel = floor(v + 0.5), half-open cells; -1 outside.
__device__ __forceinline__ int64_t voxel_floor_half(const Grid& g, float x, float y, float z)
{
    const float vx = floorf(dot4(g.row0, x, y, z, 1.0f) + 0.5f);
    const float vy = floorf(dot4(g.row1, x, y, z, 1.0f) + 0.5f);
    const float vz = floorf(dot4(g.row2, x, y, z, 1.0f) + 0.5f);
    if (!(vx >= 0.0f && vx < (float)g.nx && vy >= 0.0f && vy < (float)g.ny && vz >= 0.0f && vz < (float)g.nz))
        return -1;
    return ((int64_t)(int32_t)vx * g.ny + (int32_t)vy) * g.nz + (int32_t)vz;
}

// field.py:88-114: voxel = rint(v) (ties to even); -1 outside.
__device__ __forceinline__ int64_t voxel_rint(const Grid& g, float x, float y, float z)
{
    const float vx = rintf(dot4(g.row0, x, y, z, 1.0f));
    const float vy = rintf(dot4(g.row1, x, y, z, 1.0f));
    const float vz = rintf(dot4(g.row2, x, y, z, 1.0f));
    if (!(vx >= 0.0f && vx < (float)g.nx && vy >= 0.0f && vy < (float)g.ny && vz >= 0.0f && vz < (float)g.nz))
        return -1;
    return ((int64_t)(int32_t)vx * g.ny + (int32_t)vy) * g.nz + (int32_t)vz;
}

}  // namespace tg

#endif  // TG_DEVICE_CUH
