/* Generated by gen_sh_tables.py -- do not edit. */
/* The fold of a voxel's SH coefficients (tgsh_fold's sums), and the value,
 * d/dtheta and (d/dphi)/sin(theta) of the real symmetric SH model from it: per
 * order m and part, S(u) and S'(u) by one Horner pass, then A = x^p S and dA/dx.
 * Written for scalar instructions: with cosine and sine part of an order in
 * register pairs (tg_f32x2.cuh) it took 147 instructions instead of 182 but, at
 * 96 registers, 40 to 150 bytes of spills, and the paired multiply-adds hold the
 * arithmetic pipe for two cycles each: 593 ms against 558 ms for 100k SDE seeds.
 * Each order's trigonometric factors and powers stand right before their block:
 * all of them up front took 570 ms where this order takes 540 ms. */
#ifndef TG_SH_FOLDED_CUH
#define TG_SH_FOLDED_CUH

namespace tg {

template <> __device__ __forceinline__ void sh_fold<0>(const float* c, float* a)
{
    a[0] = (float)(0.0 + (double)c[0] * 0x1.20dd750429b6dp-2);
}

template <> __device__ __forceinline__ void sh_eval_folded<0>(
    const float* a, float ct, float st, float cp, float sp,
    float* val_out, float* dth_out, float* dph_out)
{
    const float u = ct * ct;
    const float x2 = ct + ct;
    const float u2 = u + u;
    const float tc = cp + cp;
    (void)x2; (void)u2; (void)tc; (void)sp;
    const float cm0 = 1.0f, sm0 = 0.0f;
    (void)cm0; (void)sm0;
    const float stp0 = 1.0f;
    (void)stp0;
    float val = 0.0f, dth = 0.0f, dph = 0.0f;
    const float stp1 = stp0 * st;
    {
        const float SA = a[0];
        const float A = SA;
        val = val + A;
    }
    *val_out = val;
    *dth_out = dth;
    *dph_out = dph;
}

template <> __device__ __forceinline__ void sh_fold<2>(const float* c, float* a)
{
    a[0] = (float)(0.0 + (double)c[3] * 0x1.e471027d29b68p-1);
    a[1] = (float)((0.0 + (double)c[0] * 0x1.20dd750429b6dp-2) + (double)c[3] * -0x1.42f601a8c679bp-2);
    a[2] = (float)(0.0 + (double)c[4] * -0x1.17b14102b0694p+0);
    a[3] = (float)(0.0 + (double)c[2] * -0x1.17b14102b0694p+0);
    a[4] = (float)(0.0 + (double)c[5] * 0x1.17b14102b0694p-1);
    a[5] = (float)(0.0 + (double)c[1] * 0x1.17b14102b0694p-1);
}

template <> __device__ __forceinline__ void sh_eval_folded<2>(
    const float* a, float ct, float st, float cp, float sp,
    float* val_out, float* dth_out, float* dph_out)
{
    const float u = ct * ct;
    const float x2 = ct + ct;
    const float u2 = u + u;
    const float tc = cp + cp;
    (void)x2; (void)u2; (void)tc; (void)sp;
    const float cm0 = 1.0f, sm0 = 0.0f;
    (void)cm0; (void)sm0;
    const float cm1 = cp, sm1 = sp;
    const float stp0 = 1.0f;
    (void)stp0;
    float val = 0.0f, dth = 0.0f, dph = 0.0f;
    const float stp1 = stp0 * st;
    {
        float DA = a[0];
        float SA = fmaf(a[0], u, a[1]);
        const float A = SA;
        const float Ap = x2 * DA;
        val = val + A;
        dth = fmaf(-stp1, Ap, dth);
    }
    const float stp2 = stp1 * st;
    {
        const float SA = a[2];
        const float A = SA * ct;
        const float Ap = SA;
        const float SB = a[3];
        const float B = SB * ct;
        const float Bp = SB;
        const float F = fmaf(B, sm1, A * cm1);
        const float Fp = fmaf(Bp, sm1, Ap * cm1);
        const float G = fmaf(-A, sm1, B * cm1);
        val = fmaf(stp1, F, val);
        const float mw = 1.0f * stp0;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp2, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm2 = fmaf(tc, cm1, -cm0);
    const float sm2 = fmaf(tc, sm1, -sm0);
    const float stp3 = stp2 * st;
    {
        const float SA = a[4];
        const float A = SA;
        const float SB = a[5];
        const float B = SB;
        const float F = fmaf(B, sm2, A * cm2);
        const float G = fmaf(-A, sm2, B * cm2);
        val = fmaf(stp2, F, val);
        const float mw = 2.0f * stp1;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dph = fmaf(mw, G, dph);
    }
    *val_out = val;
    *dth_out = dth;
    *dph_out = dph;
}

template <> __device__ __forceinline__ void sh_fold<4>(const float* c, float* a)
{
    a[0] = (float)(0.0 + (double)c[10] * 0x1.d9eb53fad46ffp+1);
    a[1] = (float)((0.0 + (double)c[3] * 0x1.e471027d29b68p-1) + (double)c[10] * -0x1.96376c8ddaa92p+1);
    a[2] = (float)(((0.0 + (double)c[0] * 0x1.20dd750429b6dp-2) + (double)c[3] * -0x1.42f601a8c679bp-2) + (double)c[10] * 0x1.44f923a4aeedbp-2);
    a[3] = (float)(0.0 + (double)c[11] * -0x1.2bbb9c2824049p+2);
    a[4] = (float)((0.0 + (double)c[4] * -0x1.17b14102b0694p+0) + (double)c[11] * 0x1.00e9f3901edf5p+1);
    a[5] = (float)(0.0 + (double)c[9] * -0x1.2bbb9c2824049p+2);
    a[6] = (float)((0.0 + (double)c[2] * -0x1.17b14102b0694p+0) + (double)c[9] * 0x1.00e9f3901edf5p+1);
    a[7] = (float)(0.0 + (double)c[12] * 0x1.a7e2e22d847fap+1);
    a[8] = (float)((0.0 + (double)c[5] * 0x1.17b14102b0694p-1) + (double)c[12] * -0x1.e471027d29b67p-2);
    a[9] = (float)(0.0 + (double)c[8] * 0x1.a7e2e22d847fap+1);
    a[10] = (float)((0.0 + (double)c[1] * 0x1.17b14102b0694p-1) + (double)c[8] * -0x1.e471027d29b67p-2);
    a[11] = (float)(0.0 + (double)c[13] * -0x1.c5274a45d91d9p+0);
    a[12] = (float)(0.0 + (double)c[7] * -0x1.c5274a45d91d9p+0);
    a[13] = (float)(0.0 + (double)c[14] * 0x1.406d8aa0d83a5p-1);
    a[14] = (float)(0.0 + (double)c[6] * 0x1.406d8aa0d83a5p-1);
}

template <> __device__ __forceinline__ void sh_eval_folded<4>(
    const float* a, float ct, float st, float cp, float sp,
    float* val_out, float* dth_out, float* dph_out)
{
    const float u = ct * ct;
    const float x2 = ct + ct;
    const float u2 = u + u;
    const float tc = cp + cp;
    (void)x2; (void)u2; (void)tc; (void)sp;
    const float cm0 = 1.0f, sm0 = 0.0f;
    (void)cm0; (void)sm0;
    const float cm1 = cp, sm1 = sp;
    const float stp0 = 1.0f;
    (void)stp0;
    float val = 0.0f, dth = 0.0f, dph = 0.0f;
    const float stp1 = stp0 * st;
    {
        float DA = a[0];
        float SA = fmaf(a[0], u, a[1]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[2]);
        const float A = SA;
        const float Ap = x2 * DA;
        val = val + A;
        dth = fmaf(-stp1, Ap, dth);
    }
    const float stp2 = stp1 * st;
    {
        float DA = a[3];
        float SA = fmaf(a[3], u, a[4]);
        const float A = SA * ct;
        const float Ap = fmaf(u2, DA, SA);
        float DB = a[5];
        float SB = fmaf(a[5], u, a[6]);
        const float B = SB * ct;
        const float Bp = fmaf(u2, DB, SB);
        const float F = fmaf(B, sm1, A * cm1);
        const float Fp = fmaf(Bp, sm1, Ap * cm1);
        const float G = fmaf(-A, sm1, B * cm1);
        val = fmaf(stp1, F, val);
        const float mw = 1.0f * stp0;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp2, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm2 = fmaf(tc, cm1, -cm0);
    const float sm2 = fmaf(tc, sm1, -sm0);
    const float stp3 = stp2 * st;
    {
        float DA = a[7];
        float SA = fmaf(a[7], u, a[8]);
        const float A = SA;
        const float Ap = x2 * DA;
        float DB = a[9];
        float SB = fmaf(a[9], u, a[10]);
        const float B = SB;
        const float Bp = x2 * DB;
        const float F = fmaf(B, sm2, A * cm2);
        const float Fp = fmaf(Bp, sm2, Ap * cm2);
        const float G = fmaf(-A, sm2, B * cm2);
        val = fmaf(stp2, F, val);
        const float mw = 2.0f * stp1;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp3, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm3 = fmaf(tc, cm2, -cm1);
    const float sm3 = fmaf(tc, sm2, -sm1);
    const float stp4 = stp3 * st;
    {
        const float SA = a[11];
        const float A = SA * ct;
        const float Ap = SA;
        const float SB = a[12];
        const float B = SB * ct;
        const float Bp = SB;
        const float F = fmaf(B, sm3, A * cm3);
        const float Fp = fmaf(Bp, sm3, Ap * cm3);
        const float G = fmaf(-A, sm3, B * cm3);
        val = fmaf(stp3, F, val);
        const float mw = 3.0f * stp2;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp4, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm4 = fmaf(tc, cm3, -cm2);
    const float sm4 = fmaf(tc, sm3, -sm2);
    const float stp5 = stp4 * st;
    {
        const float SA = a[13];
        const float A = SA;
        const float SB = a[14];
        const float B = SB;
        const float F = fmaf(B, sm4, A * cm4);
        const float G = fmaf(-A, sm4, B * cm4);
        val = fmaf(stp4, F, val);
        const float mw = 4.0f * stp3;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dph = fmaf(mw, G, dph);
    }
    *val_out = val;
    *dth_out = dth;
    *dph_out = dph;
}

template <> __device__ __forceinline__ void sh_fold<6>(const float* c, float* a)
{
    a[0] = (float)(0.0 + (double)c[21] * 0x1.d5e74e9acca49p+3);
    a[1] = (float)((0.0 + (double)c[10] * 0x1.d9eb53fad46ffp+1) + (double)c[21] * -0x1.4063870c7441bp+4);
    a[2] = (float)(((0.0 + (double)c[3] * 0x1.e471027d29b68p-1) + (double)c[10] * -0x1.96376c8ddaa92p+1) + (double)c[21] * 0x1.ab2f5ebb45acep+2);
    a[3] = (float)((((0.0 + (double)c[0] * 0x1.20dd750429b6dp-2) + (double)c[3] * -0x1.42f601a8c679bp-2) + (double)c[10] * 0x1.44f923a4aeedbp-2) + (double)c[21] * -0x1.45796cbf7209dp-2);
    a[4] = (float)(0.0 + (double)c[22] * -0x1.339fc3ab0f95dp+4);
    a[5] = (float)((0.0 + (double)c[11] * -0x1.2bbb9c2824049p+2) + (double)c[22] * 0x1.17a88355b113ep+4);
    a[6] = (float)(((0.0 + (double)c[4] * -0x1.17b14102b0694p+0) + (double)c[11] * 0x1.00e9f3901edf5p+1) + (double)c[22] * -0x1.74e0af1cec1a8p+1);
    a[7] = (float)(0.0 + (double)c[20] * -0x1.339fc3ab0f95dp+4);
    a[8] = (float)((0.0 + (double)c[9] * -0x1.2bbb9c2824049p+2) + (double)c[20] * 0x1.17a88355b113ep+4);
    a[9] = (float)(((0.0 + (double)c[2] * -0x1.17b14102b0694p+0) + (double)c[9] * 0x1.00e9f3901edf5p+1) + (double)c[20] * -0x1.74e0af1cec1a8p+1);
    a[10] = (float)(0.0 + (double)c[23] * 0x1.e66578f6f272ep+3);
    a[11] = (float)((0.0 + (double)c[12] * 0x1.a7e2e22d847fap+1) + (double)c[23] * -0x1.094e9f1255b30p+3);
    a[12] = (float)(((0.0 + (double)c[5] * 0x1.17b14102b0694p-1) + (double)c[12] * -0x1.e471027d29b67p-2) + (double)c[23] * 0x1.d7a8373d0a21dp-2);
    a[13] = (float)(0.0 + (double)c[19] * 0x1.e66578f6f272ep+3);
    a[14] = (float)((0.0 + (double)c[8] * 0x1.a7e2e22d847fap+1) + (double)c[19] * -0x1.094e9f1255b30p+3);
    a[15] = (float)(((0.0 + (double)c[1] * 0x1.17b14102b0694p-1) + (double)c[8] * -0x1.e471027d29b67p-2) + (double)c[19] * 0x1.d7a8373d0a21dp-2);
    a[16] = (float)(0.0 + (double)c[24] * -0x1.4443a5f9f6f74p+3);
    a[17] = (float)((0.0 + (double)c[13] * -0x1.c5274a45d91d9p+0) + (double)c[24] * 0x1.61be296dc7996p+1);
    a[18] = (float)(0.0 + (double)c[18] * -0x1.4443a5f9f6f74p+3);
    a[19] = (float)((0.0 + (double)c[7] * -0x1.c5274a45d91d9p+0) + (double)c[18] * 0x1.61be296dc7996p+1);
    a[20] = (float)(0.0 + (double)c[25] * 0x1.6336b4652ee84p+2);
    a[21] = (float)((0.0 + (double)c[14] * 0x1.406d8aa0d83a5p-1) + (double)c[25] * -0x1.025654a6adc03p-1);
    a[22] = (float)(0.0 + (double)c[17] * 0x1.6336b4652ee84p+2);
    a[23] = (float)((0.0 + (double)c[6] * 0x1.406d8aa0d83a5p-1) + (double)c[17] * -0x1.025654a6adc03p-1);
    a[24] = (float)(0.0 + (double)c[26] * -0x1.2eed606fefa75p+1);
    a[25] = (float)(0.0 + (double)c[16] * -0x1.2eed606fefa75p+1);
    a[26] = (float)(0.0 + (double)c[27] * 0x1.5dca4e99e480ep-1);
    a[27] = (float)(0.0 + (double)c[15] * 0x1.5dca4e99e480ep-1);
}

template <> __device__ __forceinline__ void sh_eval_folded<6>(
    const float* a, float ct, float st, float cp, float sp,
    float* val_out, float* dth_out, float* dph_out)
{
    const float u = ct * ct;
    const float x2 = ct + ct;
    const float u2 = u + u;
    const float tc = cp + cp;
    (void)x2; (void)u2; (void)tc; (void)sp;
    const float cm0 = 1.0f, sm0 = 0.0f;
    (void)cm0; (void)sm0;
    const float cm1 = cp, sm1 = sp;
    const float stp0 = 1.0f;
    (void)stp0;
    float val = 0.0f, dth = 0.0f, dph = 0.0f;
    const float stp1 = stp0 * st;
    {
        float DA = a[0];
        float SA = fmaf(a[0], u, a[1]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[2]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[3]);
        const float A = SA;
        const float Ap = x2 * DA;
        val = val + A;
        dth = fmaf(-stp1, Ap, dth);
    }
    const float stp2 = stp1 * st;
    {
        float DA = a[4];
        float SA = fmaf(a[4], u, a[5]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[6]);
        const float A = SA * ct;
        const float Ap = fmaf(u2, DA, SA);
        float DB = a[7];
        float SB = fmaf(a[7], u, a[8]);
        DB = fmaf(DB, u, SB);
        SB = fmaf(SB, u, a[9]);
        const float B = SB * ct;
        const float Bp = fmaf(u2, DB, SB);
        const float F = fmaf(B, sm1, A * cm1);
        const float Fp = fmaf(Bp, sm1, Ap * cm1);
        const float G = fmaf(-A, sm1, B * cm1);
        val = fmaf(stp1, F, val);
        const float mw = 1.0f * stp0;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp2, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm2 = fmaf(tc, cm1, -cm0);
    const float sm2 = fmaf(tc, sm1, -sm0);
    const float stp3 = stp2 * st;
    {
        float DA = a[10];
        float SA = fmaf(a[10], u, a[11]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[12]);
        const float A = SA;
        const float Ap = x2 * DA;
        float DB = a[13];
        float SB = fmaf(a[13], u, a[14]);
        DB = fmaf(DB, u, SB);
        SB = fmaf(SB, u, a[15]);
        const float B = SB;
        const float Bp = x2 * DB;
        const float F = fmaf(B, sm2, A * cm2);
        const float Fp = fmaf(Bp, sm2, Ap * cm2);
        const float G = fmaf(-A, sm2, B * cm2);
        val = fmaf(stp2, F, val);
        const float mw = 2.0f * stp1;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp3, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm3 = fmaf(tc, cm2, -cm1);
    const float sm3 = fmaf(tc, sm2, -sm1);
    const float stp4 = stp3 * st;
    {
        float DA = a[16];
        float SA = fmaf(a[16], u, a[17]);
        const float A = SA * ct;
        const float Ap = fmaf(u2, DA, SA);
        float DB = a[18];
        float SB = fmaf(a[18], u, a[19]);
        const float B = SB * ct;
        const float Bp = fmaf(u2, DB, SB);
        const float F = fmaf(B, sm3, A * cm3);
        const float Fp = fmaf(Bp, sm3, Ap * cm3);
        const float G = fmaf(-A, sm3, B * cm3);
        val = fmaf(stp3, F, val);
        const float mw = 3.0f * stp2;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp4, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm4 = fmaf(tc, cm3, -cm2);
    const float sm4 = fmaf(tc, sm3, -sm2);
    const float stp5 = stp4 * st;
    {
        float DA = a[20];
        float SA = fmaf(a[20], u, a[21]);
        const float A = SA;
        const float Ap = x2 * DA;
        float DB = a[22];
        float SB = fmaf(a[22], u, a[23]);
        const float B = SB;
        const float Bp = x2 * DB;
        const float F = fmaf(B, sm4, A * cm4);
        const float Fp = fmaf(Bp, sm4, Ap * cm4);
        const float G = fmaf(-A, sm4, B * cm4);
        val = fmaf(stp4, F, val);
        const float mw = 4.0f * stp3;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp5, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm5 = fmaf(tc, cm4, -cm3);
    const float sm5 = fmaf(tc, sm4, -sm3);
    const float stp6 = stp5 * st;
    {
        const float SA = a[24];
        const float A = SA * ct;
        const float Ap = SA;
        const float SB = a[25];
        const float B = SB * ct;
        const float Bp = SB;
        const float F = fmaf(B, sm5, A * cm5);
        const float Fp = fmaf(Bp, sm5, Ap * cm5);
        const float G = fmaf(-A, sm5, B * cm5);
        val = fmaf(stp5, F, val);
        const float mw = 5.0f * stp4;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp6, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm6 = fmaf(tc, cm5, -cm4);
    const float sm6 = fmaf(tc, sm5, -sm4);
    const float stp7 = stp6 * st;
    {
        const float SA = a[26];
        const float A = SA;
        const float SB = a[27];
        const float B = SB;
        const float F = fmaf(B, sm6, A * cm6);
        const float G = fmaf(-A, sm6, B * cm6);
        val = fmaf(stp6, F, val);
        const float mw = 6.0f * stp5;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dph = fmaf(mw, G, dph);
    }
    *val_out = val;
    *dth_out = dth;
    *dph_out = dph;
}

template <> __device__ __forceinline__ void sh_fold<8>(const float* c, float* a)
{
    a[0] = (float)(0.0 + (double)c[36] * 0x1.d3c97538aa04dp+5);
    a[1] = (float)((0.0 + (double)c[21] * 0x1.d5e74e9acca49p+3) + (double)c[36] * -0x1.b499e4df8d9e1p+6);
    a[2] = (float)(((0.0 + (double)c[10] * 0x1.d9eb53fad46ffp+1) + (double)c[21] * -0x1.4063870c7441bp+4) + (double)c[36] * 0x1.f7c5432954a2cp+5);
    a[3] = (float)((((0.0 + (double)c[3] * 0x1.e471027d29b68p-1) + (double)c[10] * -0x1.96376c8ddaa92p+1) + (double)c[21] * 0x1.ab2f5ebb45acep+2) + (double)c[36] * -0x1.6e60eb06c9308p+3);
    a[4] = (float)(((((0.0 + (double)c[0] * 0x1.20dd750429b6dp-2) + (double)c[3] * -0x1.42f601a8c679bp-2) + (double)c[10] * 0x1.44f923a4aeedbp-2) + (double)c[21] * -0x1.45796cbf7209dp-2) + (double)c[36] * 0x1.45ab7b94410ebp-2);
    a[5] = (float)(0.0 + (double)c[37] * -0x1.37dba37b1c035p+6);
    a[6] = (float)((0.0 + (double)c[22] * -0x1.339fc3ab0f95dp+4) + (double)c[37] * 0x1.b499e4df8d9e3p+6);
    a[7] = (float)(((0.0 + (double)c[11] * -0x1.2bbb9c2824049p+2) + (double)c[22] * 0x1.17a88355b113ep+4) + (double)c[37] * -0x1.4fd8d770e3174p+5);
    a[8] = (float)((((0.0 + (double)c[4] * -0x1.17b14102b0694p+0) + (double)c[11] * 0x1.00e9f3901edf5p+1) + (double)c[22] * -0x1.74e0af1cec1a8p+1) + (double)c[37] * 0x1.e881395e61963p+1);
    a[9] = (float)(0.0 + (double)c[35] * -0x1.37dba37b1c035p+6);
    a[10] = (float)((0.0 + (double)c[20] * -0x1.339fc3ab0f95dp+4) + (double)c[35] * 0x1.b499e4df8d9e3p+6);
    a[11] = (float)(((0.0 + (double)c[9] * -0x1.2bbb9c2824049p+2) + (double)c[20] * 0x1.17a88355b113ep+4) + (double)c[35] * -0x1.4fd8d770e3174p+5);
    a[12] = (float)((((0.0 + (double)c[2] * -0x1.17b14102b0694p+0) + (double)c[9] * 0x1.00e9f3901edf5p+1) + (double)c[20] * -0x1.74e0af1cec1a8p+1) + (double)c[35] * 0x1.e881395e61963p+1);
    a[13] = (float)(0.0 + (double)c[38] * 0x1.04eb499a11669p+6);
    a[14] = (float)((0.0 + (double)c[23] * 0x1.e66578f6f272ep+3) + (double)c[38] * -0x1.04eb499a11669p+6);
    a[15] = (float)(((0.0 + (double)c[12] * 0x1.a7e2e22d847fap+1) + (double)c[23] * -0x1.094e9f1255b30p+3) + (double)c[38] * 0x1.e1b2607ee50c1p+3);
    a[16] = (float)((((0.0 + (double)c[5] * 0x1.17b14102b0694p-1) + (double)c[12] * -0x1.e471027d29b67p-2) + (double)c[23] * 0x1.d7a8373d0a21dp-2) + (double)c[38] * -0x1.d31993dfe5dd3p-2);
    a[17] = (float)(0.0 + (double)c[34] * 0x1.04eb499a11669p+6);
    a[18] = (float)((0.0 + (double)c[19] * 0x1.e66578f6f272ep+3) + (double)c[34] * -0x1.04eb499a11669p+6);
    a[19] = (float)(((0.0 + (double)c[8] * 0x1.a7e2e22d847fap+1) + (double)c[19] * -0x1.094e9f1255b30p+3) + (double)c[34] * 0x1.e1b2607ee50c1p+3);
    a[20] = (float)((((0.0 + (double)c[1] * 0x1.17b14102b0694p-1) + (double)c[8] * -0x1.e471027d29b67p-2) + (double)c[19] * 0x1.d7a8373d0a21dp-2) + (double)c[34] * -0x1.d31993dfe5dd3p-2);
    a[21] = (float)(0.0 + (double)c[39] * -0x1.81672da8b934bp+5);
    a[22] = (float)((0.0 + (double)c[24] * -0x1.4443a5f9f6f74p+3) + (double)c[39] * 0x1.00ef73c5d0cddp+5);
    a[23] = (float)(((0.0 + (double)c[13] * -0x1.c5274a45d91d9p+0) + (double)c[24] * 0x1.61be296dc7996p+1) + (double)c[39] * -0x1.da579aa846684p+1);
    a[24] = (float)(0.0 + (double)c[33] * -0x1.81672da8b934bp+5);
    a[25] = (float)((0.0 + (double)c[18] * -0x1.4443a5f9f6f74p+3) + (double)c[33] * 0x1.00ef73c5d0cddp+5);
    a[26] = (float)(((0.0 + (double)c[7] * -0x1.c5274a45d91d9p+0) + (double)c[18] * 0x1.61be296dc7996p+1) + (double)c[33] * -0x1.da579aa846684p+1);
    a[27] = (float)(0.0 + (double)c[40] * 0x1.f18d9d94cf977p+4);
    a[28] = (float)((0.0 + (double)c[25] * 0x1.6336b4652ee84p+2) + (double)c[40] * -0x1.8e0ae4770c793p+3);
    a[29] = (float)(((0.0 + (double)c[14] * 0x1.406d8aa0d83a5p-1) + (double)c[25] * -0x1.025654a6adc03p-1) + (double)c[40] * 0x1.e9e6057ed4466p-2);
    a[30] = (float)(0.0 + (double)c[32] * 0x1.f18d9d94cf977p+4);
    a[31] = (float)((0.0 + (double)c[17] * 0x1.6336b4652ee84p+2) + (double)c[32] * -0x1.8e0ae4770c793p+3);
    a[32] = (float)(((0.0 + (double)c[6] * 0x1.406d8aa0d83a5p-1) + (double)c[17] * -0x1.025654a6adc03p-1) + (double)c[32] * 0x1.e9e6057ed4466p-2);
    a[33] = (float)(0.0 + (double)c[41] * -0x1.13fe2b6702c05p+4);
    a[34] = (float)((0.0 + (double)c[26] * -0x1.2eed606fefa75p+1) + (double)c[41] * 0x1.b996abd80466ep+1);
    a[35] = (float)(0.0 + (double)c[31] * -0x1.13fe2b6702c05p+4);
    a[36] = (float)((0.0 + (double)c[16] * -0x1.2eed606fefa75p+1) + (double)c[31] * 0x1.b996abd80466ep+1);
    a[37] = (float)(0.0 + (double)c[42] * 0x1.ff0a19c00e5b2p+2);
    a[38] = (float)((0.0 + (double)c[27] * 0x1.5dca4e99e480ep-1) + (double)c[42] * -0x1.108deb99a141bp-1);
    a[39] = (float)(0.0 + (double)c[30] * 0x1.ff0a19c00e5b2p+2);
    a[40] = (float)((0.0 + (double)c[15] * 0x1.5dca4e99e480ep-1) + (double)c[30] * -0x1.108deb99a141bp-1);
    a[41] = (float)(0.0 + (double)c[43] * -0x1.7535e00d444d1p+1);
    a[42] = (float)(0.0 + (double)c[29] * -0x1.7535e00d444d1p+1);
    a[43] = (float)(0.0 + (double)c[44] * 0x1.7535e00d444d1p-1);
    a[44] = (float)(0.0 + (double)c[28] * 0x1.7535e00d444d1p-1);
}

template <> __device__ __forceinline__ void sh_eval_folded<8>(
    const float* a, float ct, float st, float cp, float sp,
    float* val_out, float* dth_out, float* dph_out)
{
    const float u = ct * ct;
    const float x2 = ct + ct;
    const float u2 = u + u;
    const float tc = cp + cp;
    (void)x2; (void)u2; (void)tc; (void)sp;
    const float cm0 = 1.0f, sm0 = 0.0f;
    (void)cm0; (void)sm0;
    const float cm1 = cp, sm1 = sp;
    const float stp0 = 1.0f;
    (void)stp0;
    float val = 0.0f, dth = 0.0f, dph = 0.0f;
    const float stp1 = stp0 * st;
    {
        float DA = a[0];
        float SA = fmaf(a[0], u, a[1]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[2]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[3]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[4]);
        const float A = SA;
        const float Ap = x2 * DA;
        val = val + A;
        dth = fmaf(-stp1, Ap, dth);
    }
    const float stp2 = stp1 * st;
    {
        float DA = a[5];
        float SA = fmaf(a[5], u, a[6]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[7]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[8]);
        const float A = SA * ct;
        const float Ap = fmaf(u2, DA, SA);
        float DB = a[9];
        float SB = fmaf(a[9], u, a[10]);
        DB = fmaf(DB, u, SB);
        SB = fmaf(SB, u, a[11]);
        DB = fmaf(DB, u, SB);
        SB = fmaf(SB, u, a[12]);
        const float B = SB * ct;
        const float Bp = fmaf(u2, DB, SB);
        const float F = fmaf(B, sm1, A * cm1);
        const float Fp = fmaf(Bp, sm1, Ap * cm1);
        const float G = fmaf(-A, sm1, B * cm1);
        val = fmaf(stp1, F, val);
        const float mw = 1.0f * stp0;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp2, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm2 = fmaf(tc, cm1, -cm0);
    const float sm2 = fmaf(tc, sm1, -sm0);
    const float stp3 = stp2 * st;
    {
        float DA = a[13];
        float SA = fmaf(a[13], u, a[14]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[15]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[16]);
        const float A = SA;
        const float Ap = x2 * DA;
        float DB = a[17];
        float SB = fmaf(a[17], u, a[18]);
        DB = fmaf(DB, u, SB);
        SB = fmaf(SB, u, a[19]);
        DB = fmaf(DB, u, SB);
        SB = fmaf(SB, u, a[20]);
        const float B = SB;
        const float Bp = x2 * DB;
        const float F = fmaf(B, sm2, A * cm2);
        const float Fp = fmaf(Bp, sm2, Ap * cm2);
        const float G = fmaf(-A, sm2, B * cm2);
        val = fmaf(stp2, F, val);
        const float mw = 2.0f * stp1;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp3, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm3 = fmaf(tc, cm2, -cm1);
    const float sm3 = fmaf(tc, sm2, -sm1);
    const float stp4 = stp3 * st;
    {
        float DA = a[21];
        float SA = fmaf(a[21], u, a[22]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[23]);
        const float A = SA * ct;
        const float Ap = fmaf(u2, DA, SA);
        float DB = a[24];
        float SB = fmaf(a[24], u, a[25]);
        DB = fmaf(DB, u, SB);
        SB = fmaf(SB, u, a[26]);
        const float B = SB * ct;
        const float Bp = fmaf(u2, DB, SB);
        const float F = fmaf(B, sm3, A * cm3);
        const float Fp = fmaf(Bp, sm3, Ap * cm3);
        const float G = fmaf(-A, sm3, B * cm3);
        val = fmaf(stp3, F, val);
        const float mw = 3.0f * stp2;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp4, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm4 = fmaf(tc, cm3, -cm2);
    const float sm4 = fmaf(tc, sm3, -sm2);
    const float stp5 = stp4 * st;
    {
        float DA = a[27];
        float SA = fmaf(a[27], u, a[28]);
        DA = fmaf(DA, u, SA);
        SA = fmaf(SA, u, a[29]);
        const float A = SA;
        const float Ap = x2 * DA;
        float DB = a[30];
        float SB = fmaf(a[30], u, a[31]);
        DB = fmaf(DB, u, SB);
        SB = fmaf(SB, u, a[32]);
        const float B = SB;
        const float Bp = x2 * DB;
        const float F = fmaf(B, sm4, A * cm4);
        const float Fp = fmaf(Bp, sm4, Ap * cm4);
        const float G = fmaf(-A, sm4, B * cm4);
        val = fmaf(stp4, F, val);
        const float mw = 4.0f * stp3;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp5, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm5 = fmaf(tc, cm4, -cm3);
    const float sm5 = fmaf(tc, sm4, -sm3);
    const float stp6 = stp5 * st;
    {
        float DA = a[33];
        float SA = fmaf(a[33], u, a[34]);
        const float A = SA * ct;
        const float Ap = fmaf(u2, DA, SA);
        float DB = a[35];
        float SB = fmaf(a[35], u, a[36]);
        const float B = SB * ct;
        const float Bp = fmaf(u2, DB, SB);
        const float F = fmaf(B, sm5, A * cm5);
        const float Fp = fmaf(Bp, sm5, Ap * cm5);
        const float G = fmaf(-A, sm5, B * cm5);
        val = fmaf(stp5, F, val);
        const float mw = 5.0f * stp4;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp6, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm6 = fmaf(tc, cm5, -cm4);
    const float sm6 = fmaf(tc, sm5, -sm4);
    const float stp7 = stp6 * st;
    {
        float DA = a[37];
        float SA = fmaf(a[37], u, a[38]);
        const float A = SA;
        const float Ap = x2 * DA;
        float DB = a[39];
        float SB = fmaf(a[39], u, a[40]);
        const float B = SB;
        const float Bp = x2 * DB;
        const float F = fmaf(B, sm6, A * cm6);
        const float Fp = fmaf(Bp, sm6, Ap * cm6);
        const float G = fmaf(-A, sm6, B * cm6);
        val = fmaf(stp6, F, val);
        const float mw = 6.0f * stp5;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp7, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm7 = fmaf(tc, cm6, -cm5);
    const float sm7 = fmaf(tc, sm6, -sm5);
    const float stp8 = stp7 * st;
    {
        const float SA = a[41];
        const float A = SA * ct;
        const float Ap = SA;
        const float SB = a[42];
        const float B = SB * ct;
        const float Bp = SB;
        const float F = fmaf(B, sm7, A * cm7);
        const float Fp = fmaf(Bp, sm7, Ap * cm7);
        const float G = fmaf(-A, sm7, B * cm7);
        val = fmaf(stp7, F, val);
        const float mw = 7.0f * stp6;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp8, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    const float cm8 = fmaf(tc, cm7, -cm6);
    const float sm8 = fmaf(tc, sm7, -sm6);
    const float stp9 = stp8 * st;
    {
        const float SA = a[43];
        const float A = SA;
        const float SB = a[44];
        const float B = SB;
        const float F = fmaf(B, sm8, A * cm8);
        const float G = fmaf(-A, sm8, B * cm8);
        val = fmaf(stp8, F, val);
        const float mw = 8.0f * stp7;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dph = fmaf(mw, G, dph);
    }
    *val_out = val;
    *dth_out = dth;
    *dph_out = dph;
}

}  // namespace tg

#endif
