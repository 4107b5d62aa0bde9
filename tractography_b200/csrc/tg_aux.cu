/*
 * tg_aux.cu -- FOD seeding and the per-element kernels behind the
 * reference's standalone entry points:
 *
 *   seeds_from_fod_kernel    seeds.cl:99-118 (tg.seeds.from_fod, OpenCL path)
 *   contains_kernel          domain.py:456-469 (tg.domain.contains)
 *   field_evaluate_kernel    field.py:158-175 (tg.field.evaluate)
 *   local_evaluate_kernel    local.py:316-335 (tg.local.evaluate)
 *   update_orientation_kernel algorithm.py:738-759 (tg.algorithm.update_orientation)
 *   rng_stream_kernel        core.cl:218-238 (randus / randis test streams)
 */
#include <cuda_pipeline.h>
#include <cuda_runtime.h>

#include "tg_internal.h"
#include "tg_step.cuh"

namespace tg {

constexpr int kDirections = 1000;   // seeds.cl:10

// ------------------------------------------------------------ seeding

// seeds.cl:12-25: n-th of n_points Fibonacci-lattice directions.
__device__ __forceinline__ float3 fibonacci(uint32_t n, uint32_t n_points)
{
    const float phi = (sqrtf(5.0f) + 1.0f) * 0.5f;
    const float golden_angle = TGM_TWO_PI / phi;
    const float theta = (float)n * golden_angle;
    const float z = 1.0f - (2.0f * (float)n / (float)(n_points - 1));
    const float radius = sqrtf(fmaf(-z, z, 1.0f));
    float s, c;
    tgm_sincosf(theta, &s, &c);
    return make_float3(radius * c, radius * s, z);
}

// The 1000 directions (w = 0) and the basis values Y_i at each, rows of CPAD
// floats per band limit.  In module memory: allocating them on each call took
// longer than the kernels (the stream-ordered pool gives its memory back at
// every synchronisation).  Every call writes its band's table again, always with
// the same bits, so calls on several streams do not disturb one another.
__device__ float4 g_fod_dirs[kDirections];

__host__ __device__ constexpr int fod_row(int lmax) { return (n_coef_full(lmax) + 3) / 4; }     // float4s
__host__ __device__ constexpr int fod_table_at(int lmax)
{
    return lmax == 0 ? 0 : fod_table_at(lmax - 2) + kDirections * fod_row(lmax - 2);
}
__device__ float4 g_fod_tables[fod_table_at(8) + kDirections * fod_row(8)];

template <int MODEL, int LMAX>
__global__ void fod_table_kernel()
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kDirections) return;
    const float3 d = fibonacci((uint32_t)i, kDirections);
    g_fod_dirs[i] = make_float4(d.x, d.y, d.z, 0.0f);
    if constexpr (MODEL == kModelSH) {
        constexpr int N = n_coef_full(LMAX), ROW = fod_row(LMAX);
        float row[4 * ROW];
        const Frame f = frame_of(d.x, d.y, d.z);
        sh_basis<LMAX>(f.ct, f.st, f.cp, f.sp, row);
#pragma unroll
        for (int j = N; j < 4 * ROW; ++j) row[j] = 0.0f;
#pragma unroll
        for (int k = 0; k < ROW; ++k)
            g_fod_tables[fod_table_at(LMAX) + i * ROW + k] =
                make_float4(row[4 * k], row[4 * k + 1], row[4 * k + 2], row[4 * k + 3]);
    }
}

// The model's values of S seeds at one direction, floored at 0; row: the
// direction's basis values, or the direction itself for tensors.
template <int MODEL, int LMAX, int CPAD, int S>
__device__ __forceinline__ void fod_values(const float (&c)[S][CPAD], const float4* row, float (&value)[S])
{
    if constexpr (MODEL == kModelDTI) {
        const float4 d = row[0];
        const Frame f = frame_of(d.x, d.y, d.z);
#pragma unroll
        for (int s = 0; s < S; ++s) value[s] = dti_model(c[s], d.x, d.y, d.z, f).value;
    } else {
        float raw[S];
#pragma unroll
        for (int s = 0; s < S; ++s) raw[s] = 0.0f;
#pragma unroll
        for (int k = 0; k < CPAD / 4; ++k) {
            const float4 y = row[k];
#pragma unroll
            for (int s = 0; s < S; ++s) {
                raw[s] = fmaf(c[s][4 * k], y.x, raw[s]);
                if (4 * k + 1 < n_coef_full(LMAX)) raw[s] = fmaf(c[s][4 * k + 1], y.y, raw[s]);
                if (4 * k + 2 < n_coef_full(LMAX)) raw[s] = fmaf(c[s][4 * k + 2], y.z, raw[s]);
                if (4 * k + 3 < n_coef_full(LMAX)) raw[s] = fmaf(c[s][4 * k + 3], y.w, raw[s]);
            }
        }
        if constexpr (S == 2) {
            const F2 v = softmax2(f2(raw[0], raw[1]));
            value[0] = lo(v);
            value[1] = hi(v);
        } else {
#pragma unroll
            for (int s = 0; s < S; ++s) value[s] = softmax(raw[s]);
        }
    }
#pragma unroll
    for (int s = 0; s < S; ++s) value[s] = cl_max(value[s], 0.0f);
}

// S seeds per thread.  The cumulative sum over the directions is kept every
// kCheck of them, so that the search for the first one above the threshold
// evaluates kCheck directions again instead of all 1000.  The basis goes through
// shared memory kCheck directions at a time, the next ones copied meanwhile.
// Bound by what it takes to hand a basis row to a warp (12 16-byte loads, four
// cycles each, at lmax 8) and by instruction issue (45 multiply-adds and a
// softplus per direction and seed); two seeds per thread share a row's loads
// and a softplus's instructions.  1M seeds at lmax 8: 15.6 ms as two passes over
// a table in global memory, 4.2 ms so; 1000 seeds 1.5 and 0.25 ms.
constexpr int kCheck = 16;
constexpr int kChecks = (kDirections + kCheck - 1) / kCheck;
constexpr int kFodThreads = 128;

template <int MODEL, int LMAX>
struct FodShape {
    static constexpr int CPAD = MODEL == kModelDTI ? 8 : ModelShape<kModelSH, LMAX>::CPAD;
    static constexpr int ROW = MODEL == kModelDTI ? 1 : CPAD / 4;       // float4s per direction
};

template <int MODEL, int LMAX, int S>
constexpr size_t fod_shared_bytes()
{
    return 2 * kCheck * FodShape<MODEL, LMAX>::ROW * sizeof(float4) + (size_t)kChecks * kFodThreads * S * sizeof(float);
}

template <int MODEL, int LMAX, int S>
__global__ void __launch_bounds__(kFodThreads) seeds_from_fod_kernel(
    const float* __restrict__ fod, uint32_t C, const float4* __restrict__ voxels, uint32_t nnz,
    const float* __restrict__ affine, const uint2* __restrict__ states, uint32_t n_seeds, float4* __restrict__ seeds)
{
    constexpr int CPAD = FodShape<MODEL, LMAX>::CPAD, ROW = FodShape<MODEL, LMAX>::ROW;
    constexpr int kTile = kCheck * ROW;                    // float4s
    const float4* const table = MODEL == kModelDTI ? g_fod_dirs : g_fod_tables + fod_table_at(LMAX);
    extern __shared__ float4 fod_shared[];
    float4* const tile = fod_shared;
    float* const check = reinterpret_cast<float*>(fod_shared + 2 * kTile);
    const uint32_t tid = threadIdx.x;
    float c[S][CPAD];
    Mwc state[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const uint32_t gid = (blockIdx.x * S + s) * kFodThreads + tid;
        const uint32_t seed = gid < n_seeds ? gid : n_seeds - 1;   // past the end: the last one again, not written
        const uint2 st = states[seed];
        Mwc r;
        r.x = st.x;
        r.c = st.y;
        uint32_t vi = randi(r, nnz);                      // seeds.cl:89
        if (vi >= nnz) vi = nnz - 1;
        const float4 v = voxels[vi];
        float vx = v.x, vy = v.y, vz = v.z;
        vx = vx + (randu(r) - 0.5f);                      // seeds.cl:94 (x, y, z order)
        vy = vy + (randu(r) - 0.5f);
        vz = vz + (randu(r) - 0.5f);
        state[s] = r;
#pragma unroll
        for (int k = 0; k < CPAD; ++k) c[s][k] = (uint32_t)k < C ? fod[(size_t)vi * C + k] : 0.0f;
        if (gid < n_seeds) {
            float4 loc;
            const float4 r0 = make_float4(affine[0], affine[1], affine[2], affine[3]);
            const float4 r1 = make_float4(affine[4], affine[5], affine[6], affine[7]);
            const float4 r2 = make_float4(affine[8], affine[9], affine[10], affine[11]);
            const float4 r3 = make_float4(affine[12], affine[13], affine[14], affine[15]);
            loc.x = dot4(r0, vx, vy, vz, v.w);
            loc.y = dot4(r1, vx, vy, vz, v.w);
            loc.z = dot4(r2, vx, vy, vz, v.w);
            loc.w = dot4(r3, vx, vy, vz, v.w);
            seeds[2 * (size_t)gid] = loc;
        }
    }

    auto copy_tile = [&](int b) {                          // directions b kCheck .. of the table
        for (int q = (int)tid; q < kTile && b * kTile + q < kDirections * ROW; q += kFodThreads)
            __pipeline_memcpy_async(tile + (b & 1) * kTile + q, table + b * kTile + q, sizeof(float4));
        __pipeline_commit();
    };
    float sum[S], value[S];                               // seeds.cl:29-35
#pragma unroll
    for (int s = 0; s < S; ++s) sum[s] = 0.0f;
    copy_tile(0);
    for (int b = 0; b < kChecks; ++b) {
        __pipeline_wait_prior(0);
        __syncthreads();                                  // tile b is there, tile b - 1 read
        if (b + 1 < kChecks) copy_tile(b + 1);
        const float4* rows = tile + (b & 1) * kTile;
        const int n = min(kCheck, kDirections - b * kCheck);
#pragma unroll 2
        for (int i = 0; i < n; ++i) {
            fod_values<MODEL, LMAX, CPAD, S>(c, rows + i * ROW, value);
#pragma unroll
            for (int s = 0; s < S; ++s) sum[s] = sum[s] + value[s];
        }
#pragma unroll
        for (int s = 0; s < S; ++s) check[(b * S + s) * kFodThreads + tid] = sum[s];
    }

    float threshold[S], cs[S];                            // seeds.cl:38
    int from[S], selected[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        threshold[s] = randu(state[s]) * sum[s];
        // first kept sum above the threshold (they never fall; none is above a NaN)
        int low = 0, high = kChecks;
        while (low < high) {
            const int mid = (low + high) / 2;
            if (check[(mid * S + s) * kFodThreads + tid] > threshold[s]) high = mid;
            else low = mid + 1;
        }
        from[s] = low;
        cs[s] = low > 0 && low < kChecks ? check[((low - 1) * S + s) * kFodThreads + tid] : 0.0f;
        selected[s] = kDirections;
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
        if (from[s] == kChecks) continue;
        float one[1][CPAD], v[1];
#pragma unroll
        for (int k = 0; k < CPAD; ++k) one[0][k] = c[s][k];
        const int end = min((from[s] + 1) * kCheck, kDirections);
        for (int i = from[s] * kCheck; i < end; ++i) {
            fod_values<MODEL, LMAX, CPAD, 1>(one, table + i * ROW, v);
            cs[s] = cs[s] + v[0];
            if (cs[s] > threshold[s]) {
                selected[s] = i;
                break;
            }
        }
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const uint32_t gid = (blockIdx.x * S + s) * kFodThreads + tid;
        if (gid < n_seeds)
            seeds[2 * (size_t)gid + 1] = selected[s] < kDirections ? g_fod_dirs[selected[s]] : make_float4(0.0f, 0.0f, 1.0f, 0.0f);
    }
}

template <int MODEL, int LMAX, int S>
cudaError_t run_seeds_from_fod(const float* fod, uint32_t C, const float4* voxels, uint32_t nnz, const float* affine,
                               const uint2* states, uint32_t n_seeds, float4* seeds, cudaStream_t stream)
{
    constexpr size_t bytes = fod_shared_bytes<MODEL, LMAX, S>();
    cudaError_t e = cudaFuncSetAttribute(seeds_from_fod_kernel<MODEL, LMAX, S>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    fod_table_kernel<MODEL, LMAX><<<(kDirections + 31) / 32, 32, 0, stream>>>();
    seeds_from_fod_kernel<MODEL, LMAX, S><<<(n_seeds - 1) / (kFodThreads * S) + 1, kFodThreads, bytes, stream>>>(
        fod, C, voxels, nnz, affine, states, n_seeds, seeds);
    return cudaGetLastError();
}

// Two seeds per thread where one per thread would be more than two warps per
// scheduler: fewer loads and instructions per seed, but half as many warps to
// hide their latency.  lmax 8, one and two seeds per thread: 30k seeds 0.281 and
// 0.334 ms, 100k 0.627 and 0.522 ms, 1M 4.46 and 4.25 ms.  A tensor's row is one
// load, so two seeds save nothing there (1M: 0.68 and 0.75 ms).
template <int MODEL, int LMAX, typename... Args>
cudaError_t seeds_from_fod(uint32_t n_seeds, int sms, Args... args)
{
    if constexpr (MODEL == kModelSH) {
        if (n_seeds > (uint32_t)sms * kFodThreads * 2) return run_seeds_from_fod<MODEL, LMAX, 2>(args...);
    }
    return run_seeds_from_fod<MODEL, LMAX, 1>(args...);
}

cudaError_t launch_seeds_from_fod(int model, uint32_t C, const float* fod, const float4* voxels, uint32_t nnz,
                                  const float* affine, const uint2* states, uint32_t n_seeds, float4* seeds,
                                  cudaStream_t stream)
{
    if (n_seeds == 0) return cudaSuccess;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
#define TG_FOD(M, L) seeds_from_fod<M, L>(n_seeds, sms, fod, C, voxels, nnz, affine, states, n_seeds, seeds, stream)
    if (model == kModelDTI) return TG_FOD(kModelDTI, 0);
    switch (lmax_for(C)) {
    case 0: return TG_FOD(kModelSH, 0);
    case 2: return TG_FOD(kModelSH, 2);
    case 4: return TG_FOD(kModelSH, 4);
    case 6: return TG_FOD(kModelSH, 6);
    default: return TG_FOD(kModelSH, 8);
    }
#undef TG_FOD
}

// ------------------------------------------------------------ unit hooks

__global__ void contains_kernel(Grid g, const uint8_t* __restrict__ mask, const float4* __restrict__ pts,
                                uint32_t n, uint8_t* __restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pts[i];
    const int64_t k = voxel_floor_half(g, p.x, p.y, p.z);
    out[i] = (k >= 0 && mask[k] != 0) ? 1 : 0;
}

__global__ void field_evaluate_kernel(Grid g, const float* __restrict__ field, uint32_t C, uint32_t cpad,
                                      const float4* __restrict__ pts, uint32_t n, float* __restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pts[i];
    const int64_t k = voxel_rint(g, p.x, p.y, p.z);
    for (uint32_t j = 0; j < C; ++j) out[(size_t)i * C + j] = k >= 0 ? field[k * cpad + j] : 0.0f;
}

// The coefficients model_eval takes: SH coefficients folded (sh_fold),
// tensor coefficients as they are.
template <int MODEL, int LMAX, int CP>
__device__ __forceinline__ void model_coefficients(const float (&raw)[CP], float (&c)[CP])
{
    if constexpr (MODEL == kModelDTI) {
#pragma unroll
        for (int k = 0; k < CP; ++k) c[k] = raw[k];
    } else {
        sh_fold<LMAX>(raw, c);
    }
}

// Folds a field's SH coefficients per voxel (CPAD floats each, zero beyond
// the band) for the tracking kernels.  Bound by memory (8 CPAD bytes per
// voxel); the fold is straight-line code on registers.
template <int LMAX>
__global__ void __launch_bounds__(128) fold_field_kernel(const float4* __restrict__ raw, float4* __restrict__ folded,
                                                         uint64_t n_voxels)
{
    constexpr int N = n_coef_full(LMAX), CPAD = ModelShape<kModelSH, LMAX>::CPAD;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n_voxels;
         v += (uint64_t)gridDim.x * blockDim.x) {
        float c[CPAD], a[CPAD];
#pragma unroll
        for (int k = 0; k < CPAD / 4; ++k) {
            const float4 q = __ldg(raw + v * (CPAD / 4) + k);
            c[4 * k] = q.x;
            c[4 * k + 1] = q.y;
            c[4 * k + 2] = q.z;
            c[4 * k + 3] = q.w;
        }
        sh_fold<LMAX>(c, a);
#pragma unroll
        for (int k = N; k < CPAD; ++k) a[k] = 0.0f;
#pragma unroll
        for (int k = 0; k < CPAD / 4; ++k)
            folded[v * (CPAD / 4) + k] = make_float4(a[4 * k], a[4 * k + 1], a[4 * k + 2], a[4 * k + 3]);
    }
}

__global__ void __launch_bounds__(256) pad_field_kernel(const float* __restrict__ packed, float4* __restrict__ padded,
                                                        uint64_t n_quads, uint32_t n_params, uint32_t quads)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n_quads;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t v = i / quads;
        const uint32_t k = (uint32_t)(i - v * quads) * 4;
        const float* row = packed + v * n_params;
        padded[i] = make_float4(k < n_params ? row[k] : 0.0f, k + 1 < n_params ? row[k + 1] : 0.0f,
                                k + 2 < n_params ? row[k + 2] : 0.0f, k + 3 < n_params ? row[k + 3] : 0.0f);
    }
}

cudaError_t launch_pad_field(const float* packed, float* padded, uint64_t n_voxels, uint32_t n_params, uint32_t cpad,
                             cudaStream_t stream)
{
    if (n_voxels == 0) return cudaSuccess;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint64_t quads = n_voxels * (cpad / 4);
    const uint64_t want = (quads + 255) / 256, full = (uint64_t)sms * 32;
    pad_field_kernel<<<(int)(want < full ? want : full), 256, 0, stream>>>(packed, reinterpret_cast<float4*>(padded), quads,
                                                                          n_params, cpad / 4);
    return cudaGetLastError();
}

cudaError_t launch_fold_field(const float* raw, float* folded, uint64_t n_voxels, int lmax, cudaStream_t stream)
{
    if (n_voxels == 0) return cudaSuccess;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int block = 128;
    uint64_t grid = (n_voxels + block - 1) / block;
    if (grid > (uint64_t)sms * 32) grid = (uint64_t)sms * 32;
    const float4* src = reinterpret_cast<const float4*>(raw);
    float4* dst = reinterpret_cast<float4*>(folded);
    switch (lmax) {
    case 0: fold_field_kernel<0><<<(int)grid, block, 0, stream>>>(src, dst, n_voxels); break;
    case 2: fold_field_kernel<2><<<(int)grid, block, 0, stream>>>(src, dst, n_voxels); break;
    case 4: fold_field_kernel<4><<<(int)grid, block, 0, stream>>>(src, dst, n_voxels); break;
    case 6: fold_field_kernel<6><<<(int)grid, block, 0, stream>>>(src, dst, n_voxels); break;
    case 8: fold_field_kernel<8><<<(int)grid, block, 0, stream>>>(src, dst, n_voxels); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// A thread's row of n_params floats (zero beyond them).  Rows of more than six
// floats (kStagedRows) go through dynamic shared memory of blockDim.x rows: they
// are one piece of global memory, but a thread's own row is 180 bytes from its
// neighbour's.  A row of up to 24 bytes shares its sectors with its neighbours',
// and staging it cost more than it gave (4M rows, read directly / staged: tensor
// values 35.6 / 41.9 us, tensor updates 38.1 / 51.6 us, lmax 2 values 38.9 / 50.2 us).
template <int CP>
constexpr bool kStagedRows = CP > 6;

template <int MODEL, int LMAX>
size_t row_bytes(int block, uint32_t n_params)      // load_row's shared memory: at most 23 KB
{
    constexpr int CP = MODEL == kModelDTI ? 6 : n_coef_full(LMAX);
    return kStagedRows<CP> ? (size_t)block * n_params * sizeof(float) : 0;
}

// Row i, the thread's; false past the end.  Called by the whole block.
template <int CP>
__device__ __forceinline__ bool load_row(const float* __restrict__ params, uint32_t n_params, uint32_t n, uint32_t i,
                                         float (&raw)[CP])
{
    if constexpr (kStagedRows<CP>) {
        extern __shared__ float staged_rows[];
        const size_t first = (size_t)blockIdx.x * blockDim.x;
        const uint32_t rows = n - first < blockDim.x ? (uint32_t)(n - first) : blockDim.x;
        for (uint32_t q = threadIdx.x; q < rows * n_params; q += blockDim.x)     // all copies in flight at once
            __pipeline_memcpy_async(staged_rows + q, params + first * n_params + q, sizeof(float));
        __pipeline_commit();
        __pipeline_wait_prior(0);
        __syncthreads();
        if (i >= n) return false;
#pragma unroll
        for (int k = 0; k < CP; ++k) raw[k] = (uint32_t)k < n_params ? staged_rows[threadIdx.x * n_params + k] : 0.0f;
    } else {
        if (i >= n) return false;
#pragma unroll
        for (int k = 0; k < CP; ++k) raw[k] = (uint32_t)k < n_params ? params[(size_t)i * n_params + k] : 0.0f;
    }
    return true;
}

template <int MODEL, int LMAX>
__global__ void local_evaluate_kernel(const float* __restrict__ params, uint32_t n_params,
                                      const float4* __restrict__ o, uint32_t n, float* __restrict__ out)
{
    constexpr int CP = MODEL == kModelDTI ? 6 : n_coef_full(LMAX);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    float raw[CP], c[CP];
    if (!load_row<CP>(params, n_params, n, i, raw)) return;
    model_coefficients<MODEL, LMAX, CP>(raw, c);
    const float4 v = o[i];
    const Frame f = frame_of(v.x, v.y, v.z);
    const ModelValue r = model_eval<MODEL, LMAX>(c, v.x, v.y, v.z, f);
    out[3 * (size_t)i] = r.value;
    out[3 * (size_t)i + 1] = r.dtheta;
    out[3 * (size_t)i + 2] = r.dphi;
}

template <int MODEL, int LMAX, int ALGO>
__global__ void update_orientation_kernel(AlgoParams a, uint32_t rng_seed, uint64_t seed_offset,
                                          const float* __restrict__ params, uint32_t n_params,
                                          const float4* __restrict__ o, uint32_t n, float4* __restrict__ out)
{
    constexpr int CP = MODEL == kModelDTI ? 6 : n_coef_full(LMAX);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    float raw[CP], c[CP];
    if (!load_row<CP>(params, n_params, n, i, raw)) return;
    model_coefficients<MODEL, LMAX, CP>(raw, c);
    RngState rng = rng_state(a, rng_init(rng_seed, i), seed_offset + i);
    float4 v = o[i];
    update_orientation<MODEL, LMAX, ALGO>(a, c, v.x, v.y, v.z, rng, 0u);
    out[i] = make_float4(v.x, v.y, v.z, 0.0f);
}

__global__ void rng_stream_kernel(int which, uint32_t s0, uint32_t s1, uint32_t n, uint32_t max, void* out)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    Mwc s;
    s.x = s0;
    s.c = s1;
    for (uint32_t i = 0; i < n; ++i) {
        if (which == 0) reinterpret_cast<float*>(out)[i] = randu(s);
        else if (which == 1) reinterpret_cast<float*>(out)[i] = randn(s);
        else reinterpret_cast<uint32_t*>(out)[i] = randi(s, max);
    }
}

static Grid grid_of(const float* inv, uint32_t nx, uint32_t ny, uint32_t nz)
{
    Grid g;
    g.row0 = make_float4(inv[0], inv[1], inv[2], inv[3]);
    g.row1 = make_float4(inv[4], inv[5], inv[6], inv[7]);
    g.row2 = make_float4(inv[8], inv[9], inv[10], inv[11]);
    g.nx = nx;
    g.ny = ny;
    g.nz = nz;
    return g;
}

cudaError_t launch_contains(const DomainDev& d, const float4* points, uint32_t n, uint8_t* out, cudaStream_t stream)
{
    if (n == 0) return cudaSuccess;
    const int block = 256;
    contains_kernel<<<(n + block - 1) / block, block, 0, stream>>>(grid_of(d.inv_affine, d.nx, d.ny, d.nz), d.mask,
                                                                   points, n, out);
    return cudaGetLastError();
}

cudaError_t launch_field_evaluate(const FieldDev& f, const float4* points, uint32_t n, float* out,
                                  cudaStream_t stream)
{
    if (n == 0) return cudaSuccess;
    const int block = 256;
    field_evaluate_kernel<<<(n + block - 1) / block, block, 0, stream>>>(grid_of(f.inv_affine, f.nx, f.ny, f.nz),
                                                                         f.data, f.n_params, f.cpad, points, n, out);
    return cudaGetLastError();
}

cudaError_t launch_local_evaluate(int model, uint32_t n_params, const float* params, const float4* o, uint32_t n,
                                  float* out, cudaStream_t stream)
{
    if (n == 0) return cudaSuccess;
    const int block = 128, grid = (int)((n - 1) / block + 1);
    if (model == kModelDTI) {
        local_evaluate_kernel<kModelDTI, 0><<<grid, block, 0, stream>>>(params, n_params, o, n, out);
    } else {
#define TG_EVALUATE(L)                                                                                              \
    case L:                                                                                                        \
        local_evaluate_kernel<kModelSH, L><<<grid, block, row_bytes<kModelSH, L>(block, n_params), stream>>>(       \
            params, n_params, o, n, out);                                                                          \
        break;
        switch (lmax_for(n_params)) {
            TG_EVALUATE(0)
            TG_EVALUATE(2)
            TG_EVALUATE(4)
            TG_EVALUATE(6)
            TG_EVALUATE(8)
        default: return cudaErrorInvalidValue;
        }
#undef TG_EVALUATE
    }
    return cudaGetLastError();
}

template <int M, int L>
static void launch_uo(int algorithm, int grid, int block, cudaStream_t stream, const AlgoParams& a, uint32_t rng_seed,
                      uint64_t seed_offset, const float* params, uint32_t n_params, const float4* o, uint32_t n,
                      float4* out)
{
    const size_t shared = row_bytes<M, L>(block, n_params);
    if (algorithm == kTransport)
        update_orientation_kernel<M, L, kTransport><<<grid, block, shared, stream>>>(a, rng_seed, seed_offset, params,
                                                                                n_params, o, n, out);
    else
        update_orientation_kernel<M, L, kDiffusion><<<grid, block, shared, stream>>>(a, rng_seed, seed_offset, params,
                                                                                n_params, o, n, out);
}

cudaError_t launch_update_orientation(int model, uint32_t n_params, int algorithm, const AlgoParams& a,
                                      uint32_t rng_seed, uint64_t seed_offset, const float* params, const float4* o,
                                      uint32_t n, float4* out, cudaStream_t stream)
{
    if (n == 0) return cudaSuccess;
    const int block = 128, grid = (int)((n + block - 1) / block);
    if (model == kModelDTI) {
        launch_uo<kModelDTI, 0>(algorithm, grid, block, stream, a, rng_seed, seed_offset, params, n_params, o, n, out);
    } else {
        switch (lmax_for(n_params)) {
        case 0: launch_uo<kModelSH, 0>(algorithm, grid, block, stream, a, rng_seed, seed_offset, params, n_params, o, n, out); break;
        case 2: launch_uo<kModelSH, 2>(algorithm, grid, block, stream, a, rng_seed, seed_offset, params, n_params, o, n, out); break;
        case 4: launch_uo<kModelSH, 4>(algorithm, grid, block, stream, a, rng_seed, seed_offset, params, n_params, o, n, out); break;
        case 6: launch_uo<kModelSH, 6>(algorithm, grid, block, stream, a, rng_seed, seed_offset, params, n_params, o, n, out); break;
        case 8: launch_uo<kModelSH, 8>(algorithm, grid, block, stream, a, rng_seed, seed_offset, params, n_params, o, n, out); break;
        default: return cudaErrorInvalidValue;
        }
    }
    return cudaGetLastError();
}

// domain.py:95-120 domain_sample_boundary + :520-545 per seed: triangle by
// the normalised cumulative areas, uniform point in it, inward normal, point
// moved 1e-4 inward.  Vector operations in the reference's order (OpenCL
// float3 arithmetic component by component, normalize = v / length(v)).
__global__ void __launch_bounds__(128) boundary_seeds_kernel(const float4* __restrict__ vertices,
                                                             const uint4* __restrict__ triangles,
                                                             const float* __restrict__ cumulative,
                                                             uint32_t n_triangles, uint32_t rng_seed, uint32_t n,
                                                             float4* __restrict__ out)
{
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= n) return;
    Mwc st = rng_init(rng_seed, gid);
    float px, py, pz, ox, oy, oz;
    sample_boundary(vertices, triangles, cumulative, n_triangles, st, px, py, pz, ox, oy, oz);
    out[2 * (size_t)gid] = make_float4(px, py, pz, 1.0f);
    out[2 * (size_t)gid + 1] = make_float4(ox, oy, oz, 0.0f);
}

cudaError_t launch_boundary_seeds(const float4* vertices, const uint4* triangles, const float* cumulative,
                                  uint32_t n_triangles, uint32_t rng_seed, uint32_t n, float4* out,
                                  cudaStream_t stream)
{
    if (n == 0) return cudaSuccess;
    boundary_seeds_kernel<<<(n + 127) / 128, 128, 0, stream>>>(vertices, triangles, cumulative, n_triangles,
                                                              rng_seed, n, out);
    return cudaGetLastError();
}

cudaError_t launch_rng_streams(int which, uint32_t s0, uint32_t s1, uint32_t n, uint32_t max, void* out,
                               cudaStream_t stream)
{
    if (n == 0) return cudaSuccess;
    rng_stream_kernel<<<1, 1, 0, stream>>>(which, s0, s1, n, max, out);
    return cudaGetLastError();
}

}  // namespace tg
