/* Generated by gen_sh_tables.py -- do not edit. */
/* Straight-line evaluation of the real symmetric SH model value, d/dtheta and
 * (d/dphi)/sin(theta) at one orientation.  Operation order equals the
 * table-driven evaluation described in gen_sh_tables.py. */
#ifndef TG_SH_EVAL_CUH
#define TG_SH_EVAL_CUH

namespace tg {

template <> __device__ __forceinline__ void sh_eval<0>(
    const float* c, float ct, float st, float cp, float sp,
    float* val_out, float* dth_out, float* dph_out)
{
    const float u = ct * ct;
    const float tc = cp + cp;
    (void)u; (void)tc;
    const float cm0 = 1.0f, sm0 = 0.0f;
    (void)cm0; (void)sm0;
    float stp0 = 1.0f;
    const float stp1 = stp0 * st;
    (void)stp0;
    float val = 0.0f, dth = 0.0f, dph = 0.0f;
    {
        float A = 0.0f, Ap = 0.0f;
        {
        float R = 0x1.20dd76p-2f;
        A = fmaf(c[0], R, A);
        }
        val = val + A;
        dth = fmaf(-stp1, Ap, dth);
    }
    *val_out = val;
    *dth_out = dth;
    *dph_out = dph;
}

template <> __device__ __forceinline__ void sh_eval<2>(
    const float* c, float ct, float st, float cp, float sp,
    float* val_out, float* dth_out, float* dph_out)
{
    const float u = ct * ct;
    const float tc = cp + cp;
    (void)u; (void)tc;
    const float cm0 = 1.0f, sm0 = 0.0f;
    float cm1 = cp, sm1 = sp;
    const float cm2 = fmaf(tc, cm1, -cm0);
    const float sm2 = fmaf(tc, sm1, -sm0);
    (void)cm0; (void)sm0;
    float stp0 = 1.0f;
    const float stp1 = stp0 * st;
    const float stp2 = stp1 * st;
    const float stp3 = stp2 * st;
    (void)stp0;
    float val = 0.0f, dth = 0.0f, dph = 0.0f;
    {
        float A = 0.0f, Ap = 0.0f;
        {
        float R = 0x1.20dd76p-2f;
        A = fmaf(c[0], R, A);
        }
        {
        float R = 0x1.e47102p-1f;
        R = fmaf(R, u, -0x1.42f602p-2f);
        A = fmaf(c[3], R, A);
        float Rp = 0x1.e47102p+0f;
        Rp = Rp * ct;
        Ap = fmaf(c[3], Rp, Ap);
        }
        val = val + A;
        dth = fmaf(-stp1, Ap, dth);
    }
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = -0x1.17b142p+0f;
        R = R * ct;
        A = fmaf(c[4], R, A);
        B = fmaf(c[2], R, B);
        float Rp = -0x1.17b142p+0f;
        Ap = fmaf(c[4], Rp, Ap);
        Bp = fmaf(c[2], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = 0x1.17b142p-1f;
        A = fmaf(c[5], R, A);
        B = fmaf(c[1], R, B);
        }
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
    *val_out = val;
    *dth_out = dth;
    *dph_out = dph;
}

template <> __device__ __forceinline__ void sh_eval<4>(
    const float* c, float ct, float st, float cp, float sp,
    float* val_out, float* dth_out, float* dph_out)
{
    const float u = ct * ct;
    const float tc = cp + cp;
    (void)u; (void)tc;
    const float cm0 = 1.0f, sm0 = 0.0f;
    float cm1 = cp, sm1 = sp;
    const float cm2 = fmaf(tc, cm1, -cm0);
    const float sm2 = fmaf(tc, sm1, -sm0);
    const float cm3 = fmaf(tc, cm2, -cm1);
    const float sm3 = fmaf(tc, sm2, -sm1);
    const float cm4 = fmaf(tc, cm3, -cm2);
    const float sm4 = fmaf(tc, sm3, -sm2);
    (void)cm0; (void)sm0;
    float stp0 = 1.0f;
    const float stp1 = stp0 * st;
    const float stp2 = stp1 * st;
    const float stp3 = stp2 * st;
    const float stp4 = stp3 * st;
    const float stp5 = stp4 * st;
    (void)stp0;
    float val = 0.0f, dth = 0.0f, dph = 0.0f;
    {
        float A = 0.0f, Ap = 0.0f;
        {
        float R = 0x1.20dd76p-2f;
        A = fmaf(c[0], R, A);
        }
        {
        float R = 0x1.e47102p-1f;
        R = fmaf(R, u, -0x1.42f602p-2f);
        A = fmaf(c[3], R, A);
        float Rp = 0x1.e47102p+0f;
        Rp = Rp * ct;
        Ap = fmaf(c[3], Rp, Ap);
        }
        {
        float R = 0x1.d9eb54p+1f;
        R = fmaf(R, u, -0x1.96376cp+1f);
        R = fmaf(R, u, 0x1.44f924p-2f);
        A = fmaf(c[10], R, A);
        float Rp = 0x1.d9eb54p+3f;
        Rp = fmaf(Rp, u, -0x1.96376cp+2f);
        Rp = Rp * ct;
        Ap = fmaf(c[10], Rp, Ap);
        }
        val = val + A;
        dth = fmaf(-stp1, Ap, dth);
    }
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = -0x1.17b142p+0f;
        R = R * ct;
        A = fmaf(c[4], R, A);
        B = fmaf(c[2], R, B);
        float Rp = -0x1.17b142p+0f;
        Ap = fmaf(c[4], Rp, Ap);
        Bp = fmaf(c[2], Rp, Bp);
        }
        {
        float R = -0x1.2bbb9cp+2f;
        R = fmaf(R, u, 0x1.00e9f4p+1f);
        R = R * ct;
        A = fmaf(c[11], R, A);
        B = fmaf(c[9], R, B);
        float Rp = -0x1.c1996ap+3f;
        Rp = fmaf(Rp, u, 0x1.00e9f4p+1f);
        Ap = fmaf(c[11], Rp, Ap);
        Bp = fmaf(c[9], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = 0x1.17b142p-1f;
        A = fmaf(c[5], R, A);
        B = fmaf(c[1], R, B);
        }
        {
        float R = 0x1.a7e2e2p+1f;
        R = fmaf(R, u, -0x1.e47102p-2f);
        A = fmaf(c[12], R, A);
        B = fmaf(c[8], R, B);
        float Rp = 0x1.a7e2e2p+2f;
        Rp = Rp * ct;
        Ap = fmaf(c[12], Rp, Ap);
        Bp = fmaf(c[8], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = -0x1.c5274ap+0f;
        R = R * ct;
        A = fmaf(c[13], R, A);
        B = fmaf(c[7], R, B);
        float Rp = -0x1.c5274ap+0f;
        Ap = fmaf(c[13], Rp, Ap);
        Bp = fmaf(c[7], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = 0x1.406d8ap-1f;
        A = fmaf(c[14], R, A);
        B = fmaf(c[6], R, B);
        }
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
    *val_out = val;
    *dth_out = dth;
    *dph_out = dph;
}

template <> __device__ __forceinline__ void sh_eval<6>(
    const float* c, float ct, float st, float cp, float sp,
    float* val_out, float* dth_out, float* dph_out)
{
    const float u = ct * ct;
    const float tc = cp + cp;
    (void)u; (void)tc;
    const float cm0 = 1.0f, sm0 = 0.0f;
    float cm1 = cp, sm1 = sp;
    const float cm2 = fmaf(tc, cm1, -cm0);
    const float sm2 = fmaf(tc, sm1, -sm0);
    const float cm3 = fmaf(tc, cm2, -cm1);
    const float sm3 = fmaf(tc, sm2, -sm1);
    const float cm4 = fmaf(tc, cm3, -cm2);
    const float sm4 = fmaf(tc, sm3, -sm2);
    const float cm5 = fmaf(tc, cm4, -cm3);
    const float sm5 = fmaf(tc, sm4, -sm3);
    const float cm6 = fmaf(tc, cm5, -cm4);
    const float sm6 = fmaf(tc, sm5, -sm4);
    (void)cm0; (void)sm0;
    float stp0 = 1.0f;
    const float stp1 = stp0 * st;
    const float stp2 = stp1 * st;
    const float stp3 = stp2 * st;
    const float stp4 = stp3 * st;
    const float stp5 = stp4 * st;
    const float stp6 = stp5 * st;
    const float stp7 = stp6 * st;
    (void)stp0;
    float val = 0.0f, dth = 0.0f, dph = 0.0f;
    {
        float A = 0.0f, Ap = 0.0f;
        {
        float R = 0x1.20dd76p-2f;
        A = fmaf(c[0], R, A);
        }
        {
        float R = 0x1.e47102p-1f;
        R = fmaf(R, u, -0x1.42f602p-2f);
        A = fmaf(c[3], R, A);
        float Rp = 0x1.e47102p+0f;
        Rp = Rp * ct;
        Ap = fmaf(c[3], Rp, Ap);
        }
        {
        float R = 0x1.d9eb54p+1f;
        R = fmaf(R, u, -0x1.96376cp+1f);
        R = fmaf(R, u, 0x1.44f924p-2f);
        A = fmaf(c[10], R, A);
        float Rp = 0x1.d9eb54p+3f;
        Rp = fmaf(Rp, u, -0x1.96376cp+2f);
        Rp = Rp * ct;
        Ap = fmaf(c[10], Rp, Ap);
        }
        {
        float R = 0x1.d5e74ep+3f;
        R = fmaf(R, u, -0x1.406388p+4f);
        R = fmaf(R, u, 0x1.ab2f5ep+2f);
        R = fmaf(R, u, -0x1.45796cp-2f);
        A = fmaf(c[21], R, A);
        float Rp = 0x1.606d7ap+6f;
        Rp = fmaf(Rp, u, -0x1.406388p+6f);
        Rp = fmaf(Rp, u, 0x1.ab2f5ep+3f);
        Rp = Rp * ct;
        Ap = fmaf(c[21], Rp, Ap);
        }
        val = val + A;
        dth = fmaf(-stp1, Ap, dth);
    }
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = -0x1.17b142p+0f;
        R = R * ct;
        A = fmaf(c[4], R, A);
        B = fmaf(c[2], R, B);
        float Rp = -0x1.17b142p+0f;
        Ap = fmaf(c[4], Rp, Ap);
        Bp = fmaf(c[2], Rp, Bp);
        }
        {
        float R = -0x1.2bbb9cp+2f;
        R = fmaf(R, u, 0x1.00e9f4p+1f);
        R = R * ct;
        A = fmaf(c[11], R, A);
        B = fmaf(c[9], R, B);
        float Rp = -0x1.c1996ap+3f;
        Rp = fmaf(Rp, u, 0x1.00e9f4p+1f);
        Ap = fmaf(c[11], Rp, Ap);
        Bp = fmaf(c[9], Rp, Bp);
        }
        {
        float R = -0x1.339fc4p+4f;
        R = fmaf(R, u, 0x1.17a884p+4f);
        R = fmaf(R, u, -0x1.74e0b0p+1f);
        R = R * ct;
        A = fmaf(c[22], R, A);
        B = fmaf(c[20], R, B);
        float Rp = -0x1.8087b4p+6f;
        Rp = fmaf(Rp, u, 0x1.a37cc6p+5f);
        Rp = fmaf(Rp, u, -0x1.74e0b0p+1f);
        Ap = fmaf(c[22], Rp, Ap);
        Bp = fmaf(c[20], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = 0x1.17b142p-1f;
        A = fmaf(c[5], R, A);
        B = fmaf(c[1], R, B);
        }
        {
        float R = 0x1.a7e2e2p+1f;
        R = fmaf(R, u, -0x1.e47102p-2f);
        A = fmaf(c[12], R, A);
        B = fmaf(c[8], R, B);
        float Rp = 0x1.a7e2e2p+2f;
        Rp = Rp * ct;
        Ap = fmaf(c[12], Rp, Ap);
        Bp = fmaf(c[8], Rp, Bp);
        }
        {
        float R = 0x1.e66578p+3f;
        R = fmaf(R, u, -0x1.094ea0p+3f);
        R = fmaf(R, u, 0x1.d7a838p-2f);
        A = fmaf(c[23], R, A);
        B = fmaf(c[19], R, B);
        float Rp = 0x1.e66578p+5f;
        Rp = fmaf(Rp, u, -0x1.094ea0p+4f);
        Rp = Rp * ct;
        Ap = fmaf(c[23], Rp, Ap);
        Bp = fmaf(c[19], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = -0x1.c5274ap+0f;
        R = R * ct;
        A = fmaf(c[13], R, A);
        B = fmaf(c[7], R, B);
        float Rp = -0x1.c5274ap+0f;
        Ap = fmaf(c[13], Rp, Ap);
        Bp = fmaf(c[7], Rp, Bp);
        }
        {
        float R = -0x1.4443a6p+3f;
        R = fmaf(R, u, 0x1.61be2ap+1f);
        R = R * ct;
        A = fmaf(c[24], R, A);
        B = fmaf(c[18], R, B);
        float Rp = -0x1.e66578p+4f;
        Rp = fmaf(Rp, u, 0x1.61be2ap+1f);
        Ap = fmaf(c[24], Rp, Ap);
        Bp = fmaf(c[18], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = 0x1.406d8ap-1f;
        A = fmaf(c[14], R, A);
        B = fmaf(c[6], R, B);
        }
        {
        float R = 0x1.6336b4p+2f;
        R = fmaf(R, u, -0x1.025654p-1f);
        A = fmaf(c[25], R, A);
        B = fmaf(c[17], R, B);
        float Rp = 0x1.6336b4p+3f;
        Rp = Rp * ct;
        Ap = fmaf(c[25], Rp, Ap);
        Bp = fmaf(c[17], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = -0x1.2eed60p+1f;
        R = R * ct;
        A = fmaf(c[26], R, A);
        B = fmaf(c[16], R, B);
        float Rp = -0x1.2eed60p+1f;
        Ap = fmaf(c[26], Rp, Ap);
        Bp = fmaf(c[16], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = 0x1.5dca4ep-1f;
        A = fmaf(c[27], R, A);
        B = fmaf(c[15], R, B);
        }
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
    *val_out = val;
    *dth_out = dth;
    *dph_out = dph;
}

template <> __device__ __forceinline__ void sh_eval<8>(
    const float* c, float ct, float st, float cp, float sp,
    float* val_out, float* dth_out, float* dph_out)
{
    const float u = ct * ct;
    const float tc = cp + cp;
    (void)u; (void)tc;
    const float cm0 = 1.0f, sm0 = 0.0f;
    float cm1 = cp, sm1 = sp;
    const float cm2 = fmaf(tc, cm1, -cm0);
    const float sm2 = fmaf(tc, sm1, -sm0);
    const float cm3 = fmaf(tc, cm2, -cm1);
    const float sm3 = fmaf(tc, sm2, -sm1);
    const float cm4 = fmaf(tc, cm3, -cm2);
    const float sm4 = fmaf(tc, sm3, -sm2);
    const float cm5 = fmaf(tc, cm4, -cm3);
    const float sm5 = fmaf(tc, sm4, -sm3);
    const float cm6 = fmaf(tc, cm5, -cm4);
    const float sm6 = fmaf(tc, sm5, -sm4);
    const float cm7 = fmaf(tc, cm6, -cm5);
    const float sm7 = fmaf(tc, sm6, -sm5);
    const float cm8 = fmaf(tc, cm7, -cm6);
    const float sm8 = fmaf(tc, sm7, -sm6);
    (void)cm0; (void)sm0;
    float stp0 = 1.0f;
    const float stp1 = stp0 * st;
    const float stp2 = stp1 * st;
    const float stp3 = stp2 * st;
    const float stp4 = stp3 * st;
    const float stp5 = stp4 * st;
    const float stp6 = stp5 * st;
    const float stp7 = stp6 * st;
    const float stp8 = stp7 * st;
    const float stp9 = stp8 * st;
    (void)stp0;
    float val = 0.0f, dth = 0.0f, dph = 0.0f;
    {
        float A = 0.0f, Ap = 0.0f;
        {
        float R = 0x1.20dd76p-2f;
        A = fmaf(c[0], R, A);
        }
        {
        float R = 0x1.e47102p-1f;
        R = fmaf(R, u, -0x1.42f602p-2f);
        A = fmaf(c[3], R, A);
        float Rp = 0x1.e47102p+0f;
        Rp = Rp * ct;
        Ap = fmaf(c[3], Rp, Ap);
        }
        {
        float R = 0x1.d9eb54p+1f;
        R = fmaf(R, u, -0x1.96376cp+1f);
        R = fmaf(R, u, 0x1.44f924p-2f);
        A = fmaf(c[10], R, A);
        float Rp = 0x1.d9eb54p+3f;
        Rp = fmaf(Rp, u, -0x1.96376cp+2f);
        Rp = Rp * ct;
        Ap = fmaf(c[10], Rp, Ap);
        }
        {
        float R = 0x1.d5e74ep+3f;
        R = fmaf(R, u, -0x1.406388p+4f);
        R = fmaf(R, u, 0x1.ab2f5ep+2f);
        R = fmaf(R, u, -0x1.45796cp-2f);
        A = fmaf(c[21], R, A);
        float Rp = 0x1.606d7ap+6f;
        Rp = fmaf(Rp, u, -0x1.406388p+6f);
        Rp = fmaf(Rp, u, 0x1.ab2f5ep+3f);
        Rp = Rp * ct;
        Ap = fmaf(c[21], Rp, Ap);
        }
        {
        float R = 0x1.d3c976p+5f;
        R = fmaf(R, u, -0x1.b499e4p+6f);
        R = fmaf(R, u, 0x1.f7c544p+5f);
        R = fmaf(R, u, -0x1.6e60ecp+3f);
        R = fmaf(R, u, 0x1.45ab7cp-2f);
        A = fmaf(c[36], R, A);
        float Rp = 0x1.d3c976p+8f;
        Rp = fmaf(Rp, u, -0x1.47736cp+9f);
        Rp = fmaf(Rp, u, 0x1.f7c544p+7f);
        Rp = fmaf(Rp, u, -0x1.6e60ecp+4f);
        Rp = Rp * ct;
        Ap = fmaf(c[36], Rp, Ap);
        }
        val = val + A;
        dth = fmaf(-stp1, Ap, dth);
    }
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = -0x1.17b142p+0f;
        R = R * ct;
        A = fmaf(c[4], R, A);
        B = fmaf(c[2], R, B);
        float Rp = -0x1.17b142p+0f;
        Ap = fmaf(c[4], Rp, Ap);
        Bp = fmaf(c[2], Rp, Bp);
        }
        {
        float R = -0x1.2bbb9cp+2f;
        R = fmaf(R, u, 0x1.00e9f4p+1f);
        R = R * ct;
        A = fmaf(c[11], R, A);
        B = fmaf(c[9], R, B);
        float Rp = -0x1.c1996ap+3f;
        Rp = fmaf(Rp, u, 0x1.00e9f4p+1f);
        Ap = fmaf(c[11], Rp, Ap);
        Bp = fmaf(c[9], Rp, Bp);
        }
        {
        float R = -0x1.339fc4p+4f;
        R = fmaf(R, u, 0x1.17a884p+4f);
        R = fmaf(R, u, -0x1.74e0b0p+1f);
        R = R * ct;
        A = fmaf(c[22], R, A);
        B = fmaf(c[20], R, B);
        float Rp = -0x1.8087b4p+6f;
        Rp = fmaf(Rp, u, 0x1.a37cc6p+5f);
        Rp = fmaf(Rp, u, -0x1.74e0b0p+1f);
        Ap = fmaf(c[22], Rp, Ap);
        Bp = fmaf(c[20], Rp, Bp);
        }
        {
        float R = -0x1.37dba4p+6f;
        R = fmaf(R, u, 0x1.b499e4p+6f);
        R = fmaf(R, u, -0x1.4fd8d8p+5f);
        R = fmaf(R, u, 0x1.e8813ap+1f);
        R = R * ct;
        A = fmaf(c[37], R, A);
        B = fmaf(c[35], R, B);
        float Rp = -0x1.10e030p+9f;
        Rp = fmaf(Rp, u, 0x1.10e030p+9f);
        Rp = fmaf(Rp, u, -0x1.f7c544p+6f);
        Rp = fmaf(Rp, u, 0x1.e8813ap+1f);
        Ap = fmaf(c[37], Rp, Ap);
        Bp = fmaf(c[35], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = 0x1.17b142p-1f;
        A = fmaf(c[5], R, A);
        B = fmaf(c[1], R, B);
        }
        {
        float R = 0x1.a7e2e2p+1f;
        R = fmaf(R, u, -0x1.e47102p-2f);
        A = fmaf(c[12], R, A);
        B = fmaf(c[8], R, B);
        float Rp = 0x1.a7e2e2p+2f;
        Rp = Rp * ct;
        Ap = fmaf(c[12], Rp, Ap);
        Bp = fmaf(c[8], Rp, Bp);
        }
        {
        float R = 0x1.e66578p+3f;
        R = fmaf(R, u, -0x1.094ea0p+3f);
        R = fmaf(R, u, 0x1.d7a838p-2f);
        A = fmaf(c[23], R, A);
        B = fmaf(c[19], R, B);
        float Rp = 0x1.e66578p+5f;
        Rp = fmaf(Rp, u, -0x1.094ea0p+4f);
        Rp = Rp * ct;
        Ap = fmaf(c[23], Rp, Ap);
        Bp = fmaf(c[19], Rp, Bp);
        }
        {
        float R = 0x1.04eb4ap+6f;
        R = fmaf(R, u, -0x1.04eb4ap+6f);
        R = fmaf(R, u, 0x1.e1b260p+3f);
        R = fmaf(R, u, -0x1.d31994p-2f);
        A = fmaf(c[38], R, A);
        B = fmaf(c[34], R, B);
        float Rp = 0x1.8760eep+8f;
        Rp = fmaf(Rp, u, -0x1.04eb4ap+8f);
        Rp = fmaf(Rp, u, 0x1.e1b260p+4f);
        Rp = Rp * ct;
        Ap = fmaf(c[38], Rp, Ap);
        Bp = fmaf(c[34], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = -0x1.c5274ap+0f;
        R = R * ct;
        A = fmaf(c[13], R, A);
        B = fmaf(c[7], R, B);
        float Rp = -0x1.c5274ap+0f;
        Ap = fmaf(c[13], Rp, Ap);
        Bp = fmaf(c[7], Rp, Bp);
        }
        {
        float R = -0x1.4443a6p+3f;
        R = fmaf(R, u, 0x1.61be2ap+1f);
        R = R * ct;
        A = fmaf(c[24], R, A);
        B = fmaf(c[18], R, B);
        float Rp = -0x1.e66578p+4f;
        Rp = fmaf(Rp, u, 0x1.61be2ap+1f);
        Ap = fmaf(c[24], Rp, Ap);
        Bp = fmaf(c[18], Rp, Bp);
        }
        {
        float R = -0x1.81672ep+5f;
        R = fmaf(R, u, 0x1.00ef74p+5f);
        R = fmaf(R, u, -0x1.da579ap+1f);
        R = R * ct;
        A = fmaf(c[39], R, A);
        B = fmaf(c[33], R, B);
        float Rp = -0x1.e1c0fap+7f;
        Rp = fmaf(Rp, u, 0x1.81672ep+6f);
        Rp = fmaf(Rp, u, -0x1.da579ap+1f);
        Ap = fmaf(c[39], Rp, Ap);
        Bp = fmaf(c[33], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = 0x1.406d8ap-1f;
        A = fmaf(c[14], R, A);
        B = fmaf(c[6], R, B);
        }
        {
        float R = 0x1.6336b4p+2f;
        R = fmaf(R, u, -0x1.025654p-1f);
        A = fmaf(c[25], R, A);
        B = fmaf(c[17], R, B);
        float Rp = 0x1.6336b4p+3f;
        Rp = Rp * ct;
        Ap = fmaf(c[25], Rp, Ap);
        Bp = fmaf(c[17], Rp, Bp);
        }
        {
        float R = 0x1.f18d9ep+4f;
        R = fmaf(R, u, -0x1.8e0ae4p+3f);
        R = fmaf(R, u, 0x1.e9e606p-2f);
        A = fmaf(c[40], R, A);
        B = fmaf(c[32], R, B);
        float Rp = 0x1.f18d9ep+6f;
        Rp = fmaf(Rp, u, -0x1.8e0ae4p+4f);
        Rp = Rp * ct;
        Ap = fmaf(c[40], Rp, Ap);
        Bp = fmaf(c[32], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = -0x1.2eed60p+1f;
        R = R * ct;
        A = fmaf(c[26], R, A);
        B = fmaf(c[16], R, B);
        float Rp = -0x1.2eed60p+1f;
        Ap = fmaf(c[26], Rp, Ap);
        Bp = fmaf(c[16], Rp, Bp);
        }
        {
        float R = -0x1.13fe2cp+4f;
        R = fmaf(R, u, 0x1.b996acp+1f);
        R = R * ct;
        A = fmaf(c[41], R, A);
        B = fmaf(c[31], R, B);
        float Rp = -0x1.9dfd42p+5f;
        Rp = fmaf(Rp, u, 0x1.b996acp+1f);
        Ap = fmaf(c[41], Rp, Ap);
        Bp = fmaf(c[31], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = 0x1.5dca4ep-1f;
        A = fmaf(c[27], R, A);
        B = fmaf(c[15], R, B);
        }
        {
        float R = 0x1.ff0a1ap+2f;
        R = fmaf(R, u, -0x1.108decp-1f);
        A = fmaf(c[42], R, A);
        B = fmaf(c[30], R, B);
        float Rp = 0x1.ff0a1ap+3f;
        Rp = Rp * ct;
        Ap = fmaf(c[42], Rp, Ap);
        Bp = fmaf(c[30], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = -0x1.7535e0p+1f;
        R = R * ct;
        A = fmaf(c[43], R, A);
        B = fmaf(c[29], R, B);
        float Rp = -0x1.7535e0p+1f;
        Ap = fmaf(c[43], Rp, Ap);
        Bp = fmaf(c[29], Rp, Bp);
        }
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
    {
        float A = 0.0f, Ap = 0.0f;
        float B = 0.0f, Bp = 0.0f;
        {
        float R = 0x1.7535e0p-1f;
        A = fmaf(c[44], R, A);
        B = fmaf(c[28], R, B);
        }
        const float F = fmaf(B, sm8, A * cm8);
        const float Fp = fmaf(Bp, sm8, Ap * cm8);
        const float G = fmaf(-A, sm8, B * cm8);
        val = fmaf(stp8, F, val);
        const float mw = 8.0f * stp7;
        const float wct = mw * ct;
        dth = fmaf(wct, F, dth);
        dth = fmaf(-stp9, Fp, dth);
        dph = fmaf(mw, G, dph);
    }
    *val_out = val;
    *dth_out = dth;
    *dph_out = dph;
}

template <> __device__ __forceinline__ void sh_basis<0>(
    float ct, float st, float cp, float sp, float* Y)
{
    const float u = ct * ct;
    const float tc = cp + cp;
    (void)u;
    (void)tc; (void)st; (void)sp;
    {
        float R = 0x1.20dd76p-2f;
        Y[0] = R;
    }
}

template <> __device__ __forceinline__ void sh_basis<2>(
    float ct, float st, float cp, float sp, float* Y)
{
    const float u = ct * ct;
    const float tc = cp + cp;
    (void)u;
    const float cm0 = 1.0f, sm0 = 0.0f; (void)cm0; (void)sm0;
    float cm1 = cp, sm1 = sp;
    float stp0 = 1.0f; (void)stp0;
    {
        float R = 0x1.20dd76p-2f;
        Y[0] = R;
    }
    {
        float R = 0x1.e47102p-1f;
        R = fmaf(R, u, -0x1.42f602p-2f);
        Y[3] = R;
    }
    const float stp1 = stp0 * st;
    {
        float R = -0x1.17b142p+0f;
        R = R * ct;
        const float P = R * stp1;
        Y[4] = P * cm1;
        Y[2] = P * sm1;
    }
    const float cm2 = fmaf(tc, cm1, -cm0);
    const float sm2 = fmaf(tc, sm1, -sm0);
    const float stp2 = stp1 * st;
    {
        float R = 0x1.17b142p-1f;
        const float P = R * stp2;
        Y[5] = P * cm2;
        Y[1] = P * sm2;
    }
}

template <> __device__ __forceinline__ void sh_basis<4>(
    float ct, float st, float cp, float sp, float* Y)
{
    const float u = ct * ct;
    const float tc = cp + cp;
    (void)u;
    const float cm0 = 1.0f, sm0 = 0.0f; (void)cm0; (void)sm0;
    float cm1 = cp, sm1 = sp;
    float stp0 = 1.0f; (void)stp0;
    {
        float R = 0x1.20dd76p-2f;
        Y[0] = R;
    }
    {
        float R = 0x1.e47102p-1f;
        R = fmaf(R, u, -0x1.42f602p-2f);
        Y[3] = R;
    }
    {
        float R = 0x1.d9eb54p+1f;
        R = fmaf(R, u, -0x1.96376cp+1f);
        R = fmaf(R, u, 0x1.44f924p-2f);
        Y[10] = R;
    }
    const float stp1 = stp0 * st;
    {
        float R = -0x1.17b142p+0f;
        R = R * ct;
        const float P = R * stp1;
        Y[4] = P * cm1;
        Y[2] = P * sm1;
    }
    {
        float R = -0x1.2bbb9cp+2f;
        R = fmaf(R, u, 0x1.00e9f4p+1f);
        R = R * ct;
        const float P = R * stp1;
        Y[11] = P * cm1;
        Y[9] = P * sm1;
    }
    const float cm2 = fmaf(tc, cm1, -cm0);
    const float sm2 = fmaf(tc, sm1, -sm0);
    const float stp2 = stp1 * st;
    {
        float R = 0x1.17b142p-1f;
        const float P = R * stp2;
        Y[5] = P * cm2;
        Y[1] = P * sm2;
    }
    {
        float R = 0x1.a7e2e2p+1f;
        R = fmaf(R, u, -0x1.e47102p-2f);
        const float P = R * stp2;
        Y[12] = P * cm2;
        Y[8] = P * sm2;
    }
    const float cm3 = fmaf(tc, cm2, -cm1);
    const float sm3 = fmaf(tc, sm2, -sm1);
    const float stp3 = stp2 * st;
    {
        float R = -0x1.c5274ap+0f;
        R = R * ct;
        const float P = R * stp3;
        Y[13] = P * cm3;
        Y[7] = P * sm3;
    }
    const float cm4 = fmaf(tc, cm3, -cm2);
    const float sm4 = fmaf(tc, sm3, -sm2);
    const float stp4 = stp3 * st;
    {
        float R = 0x1.406d8ap-1f;
        const float P = R * stp4;
        Y[14] = P * cm4;
        Y[6] = P * sm4;
    }
}

template <> __device__ __forceinline__ void sh_basis<6>(
    float ct, float st, float cp, float sp, float* Y)
{
    const float u = ct * ct;
    const float tc = cp + cp;
    (void)u;
    const float cm0 = 1.0f, sm0 = 0.0f; (void)cm0; (void)sm0;
    float cm1 = cp, sm1 = sp;
    float stp0 = 1.0f; (void)stp0;
    {
        float R = 0x1.20dd76p-2f;
        Y[0] = R;
    }
    {
        float R = 0x1.e47102p-1f;
        R = fmaf(R, u, -0x1.42f602p-2f);
        Y[3] = R;
    }
    {
        float R = 0x1.d9eb54p+1f;
        R = fmaf(R, u, -0x1.96376cp+1f);
        R = fmaf(R, u, 0x1.44f924p-2f);
        Y[10] = R;
    }
    {
        float R = 0x1.d5e74ep+3f;
        R = fmaf(R, u, -0x1.406388p+4f);
        R = fmaf(R, u, 0x1.ab2f5ep+2f);
        R = fmaf(R, u, -0x1.45796cp-2f);
        Y[21] = R;
    }
    const float stp1 = stp0 * st;
    {
        float R = -0x1.17b142p+0f;
        R = R * ct;
        const float P = R * stp1;
        Y[4] = P * cm1;
        Y[2] = P * sm1;
    }
    {
        float R = -0x1.2bbb9cp+2f;
        R = fmaf(R, u, 0x1.00e9f4p+1f);
        R = R * ct;
        const float P = R * stp1;
        Y[11] = P * cm1;
        Y[9] = P * sm1;
    }
    {
        float R = -0x1.339fc4p+4f;
        R = fmaf(R, u, 0x1.17a884p+4f);
        R = fmaf(R, u, -0x1.74e0b0p+1f);
        R = R * ct;
        const float P = R * stp1;
        Y[22] = P * cm1;
        Y[20] = P * sm1;
    }
    const float cm2 = fmaf(tc, cm1, -cm0);
    const float sm2 = fmaf(tc, sm1, -sm0);
    const float stp2 = stp1 * st;
    {
        float R = 0x1.17b142p-1f;
        const float P = R * stp2;
        Y[5] = P * cm2;
        Y[1] = P * sm2;
    }
    {
        float R = 0x1.a7e2e2p+1f;
        R = fmaf(R, u, -0x1.e47102p-2f);
        const float P = R * stp2;
        Y[12] = P * cm2;
        Y[8] = P * sm2;
    }
    {
        float R = 0x1.e66578p+3f;
        R = fmaf(R, u, -0x1.094ea0p+3f);
        R = fmaf(R, u, 0x1.d7a838p-2f);
        const float P = R * stp2;
        Y[23] = P * cm2;
        Y[19] = P * sm2;
    }
    const float cm3 = fmaf(tc, cm2, -cm1);
    const float sm3 = fmaf(tc, sm2, -sm1);
    const float stp3 = stp2 * st;
    {
        float R = -0x1.c5274ap+0f;
        R = R * ct;
        const float P = R * stp3;
        Y[13] = P * cm3;
        Y[7] = P * sm3;
    }
    {
        float R = -0x1.4443a6p+3f;
        R = fmaf(R, u, 0x1.61be2ap+1f);
        R = R * ct;
        const float P = R * stp3;
        Y[24] = P * cm3;
        Y[18] = P * sm3;
    }
    const float cm4 = fmaf(tc, cm3, -cm2);
    const float sm4 = fmaf(tc, sm3, -sm2);
    const float stp4 = stp3 * st;
    {
        float R = 0x1.406d8ap-1f;
        const float P = R * stp4;
        Y[14] = P * cm4;
        Y[6] = P * sm4;
    }
    {
        float R = 0x1.6336b4p+2f;
        R = fmaf(R, u, -0x1.025654p-1f);
        const float P = R * stp4;
        Y[25] = P * cm4;
        Y[17] = P * sm4;
    }
    const float cm5 = fmaf(tc, cm4, -cm3);
    const float sm5 = fmaf(tc, sm4, -sm3);
    const float stp5 = stp4 * st;
    {
        float R = -0x1.2eed60p+1f;
        R = R * ct;
        const float P = R * stp5;
        Y[26] = P * cm5;
        Y[16] = P * sm5;
    }
    const float cm6 = fmaf(tc, cm5, -cm4);
    const float sm6 = fmaf(tc, sm5, -sm4);
    const float stp6 = stp5 * st;
    {
        float R = 0x1.5dca4ep-1f;
        const float P = R * stp6;
        Y[27] = P * cm6;
        Y[15] = P * sm6;
    }
}

template <> __device__ __forceinline__ void sh_basis<8>(
    float ct, float st, float cp, float sp, float* Y)
{
    const float u = ct * ct;
    const float tc = cp + cp;
    (void)u;
    const float cm0 = 1.0f, sm0 = 0.0f; (void)cm0; (void)sm0;
    float cm1 = cp, sm1 = sp;
    float stp0 = 1.0f; (void)stp0;
    {
        float R = 0x1.20dd76p-2f;
        Y[0] = R;
    }
    {
        float R = 0x1.e47102p-1f;
        R = fmaf(R, u, -0x1.42f602p-2f);
        Y[3] = R;
    }
    {
        float R = 0x1.d9eb54p+1f;
        R = fmaf(R, u, -0x1.96376cp+1f);
        R = fmaf(R, u, 0x1.44f924p-2f);
        Y[10] = R;
    }
    {
        float R = 0x1.d5e74ep+3f;
        R = fmaf(R, u, -0x1.406388p+4f);
        R = fmaf(R, u, 0x1.ab2f5ep+2f);
        R = fmaf(R, u, -0x1.45796cp-2f);
        Y[21] = R;
    }
    {
        float R = 0x1.d3c976p+5f;
        R = fmaf(R, u, -0x1.b499e4p+6f);
        R = fmaf(R, u, 0x1.f7c544p+5f);
        R = fmaf(R, u, -0x1.6e60ecp+3f);
        R = fmaf(R, u, 0x1.45ab7cp-2f);
        Y[36] = R;
    }
    const float stp1 = stp0 * st;
    {
        float R = -0x1.17b142p+0f;
        R = R * ct;
        const float P = R * stp1;
        Y[4] = P * cm1;
        Y[2] = P * sm1;
    }
    {
        float R = -0x1.2bbb9cp+2f;
        R = fmaf(R, u, 0x1.00e9f4p+1f);
        R = R * ct;
        const float P = R * stp1;
        Y[11] = P * cm1;
        Y[9] = P * sm1;
    }
    {
        float R = -0x1.339fc4p+4f;
        R = fmaf(R, u, 0x1.17a884p+4f);
        R = fmaf(R, u, -0x1.74e0b0p+1f);
        R = R * ct;
        const float P = R * stp1;
        Y[22] = P * cm1;
        Y[20] = P * sm1;
    }
    {
        float R = -0x1.37dba4p+6f;
        R = fmaf(R, u, 0x1.b499e4p+6f);
        R = fmaf(R, u, -0x1.4fd8d8p+5f);
        R = fmaf(R, u, 0x1.e8813ap+1f);
        R = R * ct;
        const float P = R * stp1;
        Y[37] = P * cm1;
        Y[35] = P * sm1;
    }
    const float cm2 = fmaf(tc, cm1, -cm0);
    const float sm2 = fmaf(tc, sm1, -sm0);
    const float stp2 = stp1 * st;
    {
        float R = 0x1.17b142p-1f;
        const float P = R * stp2;
        Y[5] = P * cm2;
        Y[1] = P * sm2;
    }
    {
        float R = 0x1.a7e2e2p+1f;
        R = fmaf(R, u, -0x1.e47102p-2f);
        const float P = R * stp2;
        Y[12] = P * cm2;
        Y[8] = P * sm2;
    }
    {
        float R = 0x1.e66578p+3f;
        R = fmaf(R, u, -0x1.094ea0p+3f);
        R = fmaf(R, u, 0x1.d7a838p-2f);
        const float P = R * stp2;
        Y[23] = P * cm2;
        Y[19] = P * sm2;
    }
    {
        float R = 0x1.04eb4ap+6f;
        R = fmaf(R, u, -0x1.04eb4ap+6f);
        R = fmaf(R, u, 0x1.e1b260p+3f);
        R = fmaf(R, u, -0x1.d31994p-2f);
        const float P = R * stp2;
        Y[38] = P * cm2;
        Y[34] = P * sm2;
    }
    const float cm3 = fmaf(tc, cm2, -cm1);
    const float sm3 = fmaf(tc, sm2, -sm1);
    const float stp3 = stp2 * st;
    {
        float R = -0x1.c5274ap+0f;
        R = R * ct;
        const float P = R * stp3;
        Y[13] = P * cm3;
        Y[7] = P * sm3;
    }
    {
        float R = -0x1.4443a6p+3f;
        R = fmaf(R, u, 0x1.61be2ap+1f);
        R = R * ct;
        const float P = R * stp3;
        Y[24] = P * cm3;
        Y[18] = P * sm3;
    }
    {
        float R = -0x1.81672ep+5f;
        R = fmaf(R, u, 0x1.00ef74p+5f);
        R = fmaf(R, u, -0x1.da579ap+1f);
        R = R * ct;
        const float P = R * stp3;
        Y[39] = P * cm3;
        Y[33] = P * sm3;
    }
    const float cm4 = fmaf(tc, cm3, -cm2);
    const float sm4 = fmaf(tc, sm3, -sm2);
    const float stp4 = stp3 * st;
    {
        float R = 0x1.406d8ap-1f;
        const float P = R * stp4;
        Y[14] = P * cm4;
        Y[6] = P * sm4;
    }
    {
        float R = 0x1.6336b4p+2f;
        R = fmaf(R, u, -0x1.025654p-1f);
        const float P = R * stp4;
        Y[25] = P * cm4;
        Y[17] = P * sm4;
    }
    {
        float R = 0x1.f18d9ep+4f;
        R = fmaf(R, u, -0x1.8e0ae4p+3f);
        R = fmaf(R, u, 0x1.e9e606p-2f);
        const float P = R * stp4;
        Y[40] = P * cm4;
        Y[32] = P * sm4;
    }
    const float cm5 = fmaf(tc, cm4, -cm3);
    const float sm5 = fmaf(tc, sm4, -sm3);
    const float stp5 = stp4 * st;
    {
        float R = -0x1.2eed60p+1f;
        R = R * ct;
        const float P = R * stp5;
        Y[26] = P * cm5;
        Y[16] = P * sm5;
    }
    {
        float R = -0x1.13fe2cp+4f;
        R = fmaf(R, u, 0x1.b996acp+1f);
        R = R * ct;
        const float P = R * stp5;
        Y[41] = P * cm5;
        Y[31] = P * sm5;
    }
    const float cm6 = fmaf(tc, cm5, -cm4);
    const float sm6 = fmaf(tc, sm5, -sm4);
    const float stp6 = stp5 * st;
    {
        float R = 0x1.5dca4ep-1f;
        const float P = R * stp6;
        Y[27] = P * cm6;
        Y[15] = P * sm6;
    }
    {
        float R = 0x1.ff0a1ap+2f;
        R = fmaf(R, u, -0x1.108decp-1f);
        const float P = R * stp6;
        Y[42] = P * cm6;
        Y[30] = P * sm6;
    }
    const float cm7 = fmaf(tc, cm6, -cm5);
    const float sm7 = fmaf(tc, sm6, -sm5);
    const float stp7 = stp6 * st;
    {
        float R = -0x1.7535e0p+1f;
        R = R * ct;
        const float P = R * stp7;
        Y[43] = P * cm7;
        Y[29] = P * sm7;
    }
    const float cm8 = fmaf(tc, cm7, -cm6);
    const float sm8 = fmaf(tc, sm7, -sm6);
    const float stp8 = stp7 * st;
    {
        float R = 0x1.7535e0p-1f;
        const float P = R * stp8;
        Y[44] = P * cm8;
        Y[28] = P * sm8;
    }
}

}  // namespace tg

#endif
