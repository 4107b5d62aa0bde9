/*
 * math_check.cu -- the device's shorter forms against the operations they stand for.
 *
 * A test program, not part of the library.  The step and the FOD sampler write
 * reciprocals, square roots, the logarithm of a sum and pairs of normals in
 * forms of their own (tg_fmath.h, tg_device.cuh, tg_bvh.cuh) that give the bits of
 * the IEEE operation or of the shared math layer.  Each line printed is a form,
 * the arguments tried and how many of them differ: every argument that the
 * form's caller can pass, where it says so in the table in main().
 */
#include <cuda_runtime.h>

#include <cstdio>

#include "tg_bvh.cuh"
#include "tg_step.cuh"

using namespace tg;

namespace {

__device__ __forceinline__ bool differs(float a, float b)
{
    return __float_as_uint(a) != __float_as_uint(b) && !(isnan(a) && isnan(b));
}

// Form F's check of argument i: true when it differs.
struct Reciprocal {          // i: the bits of x in [2^-125, 2^125)
    static __device__ bool bad(uint64_t i)
    {
        const float x = __uint_as_float((uint32_t)i);
        return differs(tgm_rcp(x), 1.0f / x);
    }
};

struct ReciprocalSigned {    // i: the bits of any float
    static __device__ bool bad(uint64_t i)
    {
        const float x = __uint_as_float((uint32_t)i);
        return differs(rcp_signed(x), 1.0f / x);
    }
};

struct RootOfDraw {          // i = 1 .. 2^24 - 1: Box-Muller's uniform in 2^-24
    static __device__ bool bad(uint64_t i)
    {
        const float x = -2.0f * tgm_log_pos((float)i * 0x1p-24f);
        const float y = -2.0f * tgm_log_pos((float)(0x1000000u - i) * 0x1p-24f);
        const F2 r = sqrt_pos2(f2(x, y));
        return differs(lo(r), sqrtf(x)) || differs(hi(r), sqrtf(y));
    }
};

struct RootOfCounterDraw {   // i = 1 .. 2^24: the counter-based draw's uniform in 2^-24
    static __device__ bool bad(uint64_t i)
    {
        const float x = -2.0f * tgm_log_pos((float)i * 0x1p-24f);
        return differs(sqrt_pos(x), sqrtf(x));
    }
};

struct RootOfMantissa {      // i: the bits of x in [1, 4)
    static __device__ bool bad(uint64_t i)
    {
        const float x = __uint_as_float((uint32_t)i);
        const F2 r = sqrt_pos2(f2(x, x));
        return differs(lo(r), sqrtf(x)) || differs(hi(r), sqrtf(x));
    }
};

struct LogOfDraw {           // i = 1 .. 2^24 - 1
    static __device__ bool bad(uint64_t i)
    {
        const float u = (float)i * 0x1p-24f, v = (float)(0x1000000u - i) * 0x1p-24f;
        const F2 r = log_pos2(f2(u, v));
        return differs(lo(r), tgm_log_pos(u)) || differs(hi(r), tgm_log_pos(v));
    }
};

struct CosineOfDraw {        // i: all 32 bits of a draw
    static __device__ bool bad(uint64_t i)
    {
        const uint32_t w = (uint32_t)i;
        const F2 r = cos2pi_2(w, ~w);
        return differs(lo(r), tgm_cos2pi_u24(w >> 8)) || differs(hi(r), tgm_cos2pi_u24(~w >> 8));
    }
};

struct Exponential {         // i: the bits of a tangent's length in [0, 1]
    static __device__ bool bad(uint64_t i)
    {
        const float t = __uint_as_float((uint32_t)i);
        if (t * t <= 0.0f) return false;
        float ox = 1.0f, oy = 0.0f, oz = 0.0f, c, k;
        exps2(ox, oy, oz, 0.0f, t, 0.0f);
        tgm_exps2_factors(t * t, &c, &k);
        return differs(ox, c) || differs(oy, t * k);
    }
};

struct Softplus {            // i: the bits of any float
    static __device__ bool bad(uint64_t i)
    {
        const float x = __uint_as_float((uint32_t)i), kx = x * kSoftmaxScale;
        const float want = kx < 30.0f ? tgm_logf(1.0f + tgm_expf(kSoftmaxScale * x)) / kSoftmaxScale : x;
        const float y = __uint_as_float(~(uint32_t)i);
        const F2 pair = softmax2(f2(x, y));
        return differs(softmax(x), want) || differs(lo(pair), want) || differs(hi(pair), softmax(y));
    }
};

template <typename F>
__global__ void __launch_bounds__(256) check(uint64_t first, uint64_t end, unsigned long long* bad)
{
    unsigned long long mine = 0;
    for (uint64_t i = first + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < end;
         i += (uint64_t)gridDim.x * blockDim.x)
        mine += F::bad(i) ? 1u : 0u;
    if (mine != 0) atomicAdd(bad, mine);
}

template <typename F>
bool run(const char* name, uint64_t first, uint64_t end, unsigned long long* d_bad)
{
    unsigned long long bad = 0;
    if (cudaMemset(d_bad, 0, sizeof bad) != cudaSuccess) return false;
    check<F><<<148 * 8, 256>>>(first, end, d_bad);
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpy(&bad, d_bad, sizeof bad, cudaMemcpyDeviceToHost) != cudaSuccess)
        return false;
    std::printf("%s %llu %llu\n", name, (unsigned long long)(end - first), bad);
    return true;
}

}  // namespace

int main()
{
    unsigned long long* d_bad = nullptr;
    if (cudaMalloc(reinterpret_cast<void**>(&d_bad), sizeof *d_bad) != cudaSuccess) {
        std::fprintf(stderr, "math_check: device allocation failed\n");
        return 1;
    }
    const uint64_t all = 1ull << 32;
    const bool ok = run<Reciprocal>("tgm_rcp", 0x01000000u, 0x7e000000u, d_bad) &&           // 2^-125 .. 2^125
                    run<ReciprocalSigned>("rcp_signed", 0, all, d_bad) &&
                    run<RootOfDraw>("sqrt_pos2_draws", 1, 1u << 24, d_bad) &&
                    run<RootOfCounterDraw>("sqrt_pos", 1, (1u << 24) + 1, d_bad) &&
                    run<RootOfMantissa>("sqrt_pos2_mantissas", 0x3f800000u, 0x40800000u, d_bad) &&
                    run<LogOfDraw>("log_pos2", 1, 1u << 24, d_bad) &&
                    run<CosineOfDraw>("cos2pi_2", 0, all, d_bad) &&
                    run<Exponential>("exps2", 0, 0x3f800001u, d_bad) && run<Softplus>("softmax", 0, all, d_bad);
    cudaFree(d_bad);
    if (!ok) std::fprintf(stderr, "math_check: %s\n", cudaGetErrorString(cudaGetLastError()));
    return ok ? 0 : 1;
}
