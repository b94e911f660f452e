// tpord_f32.cuh -- one TPORd step in the mixed form: FP32 gates, currents and
// fluxes, the eight concentrations as compensated FP32 pairs (tpord.cuh).
//
// What bounds it.  The step is about 90 exponentials and 100 divisions in
// SingleCell/TPORd.cc:379-1021.  Written term by term they are 214
// special-function (MUFU) instructions, 8 issue slots of that pipe each, and
// 1853 instructions in all per warp: issue and MUFU are about equally full.
// Both are cut here without changing the model:
//   * exp((v + a) / k) is one FFMA (constants folded at compile time) and one
//     ex2; subnormal results are flushed (every use adds them to a normal
//     number or multiplies a rate by the step), which drops the range scaling
//     around each MUFU instruction;
//   * exponentials of multiples of v/20, v/7 come from one another
//     (exp(v/10) = exp(v/20)^2, exp(-(v+60)/5) = const * exp(-v/20)^4);
//   * tau = A + 1/s enters as the rate s/(A s + 1), products of 1/(1 + x) as
//     one reciprocal, and neighbouring reciprocals as 1/a = b * (1/ab);
//   * x/(e^x - 1) of the GHK terms from one exponential (a Taylor polynomial
//     below |x| = 0.5, where e^x - 1 would cancel).
// Where a factor could overflow at extreme V and meet a zero, it is bounded
// at a value (1e12 .. 1e18) whose effect is below FP32 resolution; the product
// of a calcium concentration under a shared reciprocal is kept off zero by the
// smallest normal number (kTiny, in the product's FMA), so that empty stores and
// clefts (cajsr, cass = 0) step as in the reference's formulas.
//
// Measured (GB300): 20,011 cells x 1000 updates 2.62 -> 1.84 ms, 320 x 320 x
// 420 ventricle with the surrogate, 50 steps, 11.40 -> 10.36 ms, mixed shell of
// 1.11 M voxels, 50 steps, 5.65 -> 5.22 ms; errors against 64 bits unchanged
// (7.6e-7 of the state after 1000 updates in both writings).  Single
// exponentials are not all as close as term by term: exp((v + a) / k) is one FMA
// with a / k rounded to FP32, so near v = -a its argument is off by up to half a
// unit of a number of 2..17 (1e-6 of the result at the most), as much as half a
// unit of v itself is worth; and e^x - 1 of the GHK terms beyond |x| = 0.5 is a
// difference of the hardware's ex2 (a few 2^-23).
// The batch kernel (k_batch.cu) keeps the term-by-term writing of tpord.cuh.  A
// last-bit change of V moves a few activation times, which are multiples of the
// step, by one step, and their bits are kept.  It is no nearer to 64 bits: of
// 36,132 activations of a sweep of strands 14 differ from the FP64 form's, 15
// with the writing here.
#pragma once
#include <cuda_runtime.h>

namespace lqt {

__device__ __forceinline__ float ex2f_(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float lg2f_(float x)
{
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcpf_(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

constexpr double kLog2e = 1.4426950408889634;
constexpr float kTiny = 1.17549435e-38f;

// A product that enters a sum, rounded by itself: with every other sum of
// products written as an FMA the step has one rounding whatever kernel it is
// inlined into (left to the compiler, which of two products is fused changes
// from kernel to kernel, and with it last bits).
__device__ __forceinline__ float mulp(float a, float b) { return __fmul_rn(a, b); }

// exp((v + a) / k): the offset is formed from the rounded slope, so that the
// slope's rounding acts on v + a and not on v.
__device__ __forceinline__ float exva(float v, double a, double k)
{
    const float c = (float)(kLog2e / k);
    const float d = (float)((double)c * a);
    return ex2f_(fmaf(v, c, d));
}
// 1 / (1 + exp((v + a) / k))
__device__ __forceinline__ float sigva(float v, double a, double k) { return rcpf_(1.0f + exva(v, a, k)); }

// x -> inf - (inf - x) exp(-rate dt), ndtl = -dt log2(e)
__device__ __forceinline__ float relaxf(float x, float inf, float rate, float ndtl)
{
    return fmaf(x - inf, ex2f_(ndtl * rate), inf);
}

__device__ __forceinline__ void tpord_step_f32(CellState<float> &c, int ctype, const ModelT<float> &m,
                                               const StepT<float> &k, float Ist, float dVgap_dt, StepOut<float> *out)
{
    const bool epi = (ctype == 2);
    const bool mid = (ctype == 4);
    const float dt = k.dt;
    const float ndtl = dt * (float)-kLog2e;
    const float v = c.v;

    // constants, TPORd.cc:382-421
    constexpr double nao = 140.0, cao = 1.8, ko = 5.4;
    constexpr double R_ = 8314.0, T_ = 310.0, F_ = 96485.0;
    constexpr double L_ = 0.01, rad = 0.0011;
    constexpr double vcell = 1000 * 3.14 * rad * rad * L_;
    constexpr double Ageo = 2 * 3.14 * rad * rad + 2 * 3.14 * rad * L_;
    constexpr double Acap = 2 * Ageo;
    constexpr double vmyo = 0.68 * vcell, vnsr = 0.0552 * vcell, vjsr = 0.0048 * vcell, vss = 0.02 * vcell;
    constexpr double RTF = R_ * T_ / F_;
    constexpr double FRT = F_ / (R_ * T_);
    constexpr double kLn2 = 0.6931471805599453;

    const float nai = c.nai.x, nass = c.nass.x, ki = c.ki.x, kss = c.kss.x;
    const float cai = c.cai.x, cass = c.cass.x, cajsr = c.cajsr.x, cansr = c.cansr.x;

    // reversal potentials, TPORd.cc:425-427 (log2 of the outside terms folded)
    constexpr double lg_nao = 7.129283016944966, lg_ko = 2.432959407276106, lg_eks = 2.9938917005640255;
    const float ENa = (float)(RTF * kLn2) * ((float)lg_nao - lg2f_(nai));
    const float EK = (float)(RTF * kLn2) * ((float)lg_ko - lg2f_(ki));
    const float EKs = (float)(RTF * kLn2) * ((float)lg_eks - lg2f_(fmaf(0.01833f, nai, ki)));

    // CaMK, TPORd.cc:430-433; 1/cass and 1/(cass + KmCaM) from one reciprocal
    const float cq = cass + 0.0015f;
    const float r_cc = rcpf_(fmaf(cass, cq, kTiny));
    const float rcass = r_cc * cq;
    const float CaMKb = 0.05f * (1.0f - c.CaMKt) * (r_cc * cass) * cass;
    const float CaMKa = CaMKb + c.CaMKt;
    const float fP = CaMKa * rcpf_(CaMKa + 0.15f);   // phosphorylated fraction (fINaLp, fItop, ...)
    const float vfrt = v * (float)FRT;

    // exp(+-v/20) and its powers; exp(+-v/7)
    const float E20 = ex2f_(v * (float)(kLog2e / 20.0)), I20 = ex2f_(v * (float)(-kLog2e / 20.0));
    const float E10 = E20 * E20, I10 = I20 * I20;
    const float E5 = E10 * E10, I5 = I10 * I10;

    // TP06 fast INa, TPORd.cc:465-504
    {
        // 1/(AM BM), AM = 1/(1+a), BM = 0.1/(1+b) + 0.1/(1+e); a b = exp(-5)
        const float a = mulp(6.14421235332821e-6f, I5);               // exp((-60 - v)/5)
        const float b = fminf(1096.6331584284585f * E5, 1e18f);  // exp((v + 35)/5)
        const float e = exva(v, -50, 200);
        const float rate_m = 10.0f * ((1.0067379469990854f + a) + b) * (1.0f + e) * rcpf_((2.0f + b) + e);
        const float em = 1.0f + exva(v, 56.86, -9.03);
        const float M_INF = rcpf_(em * em);
        float rate_h, rate_j;   // 1/tau
        if (v >= -40.0f) {
            const float x = 1.0f + exva(v, 10.66, -11.1);
            const float y = fmaf(0.04076220397836621f, I10, 1.0f);   // 1 + exp(-0.1 (v + 32))
            const float r = rcpf_(x * y);
            rate_h = (float)(0.77 / 0.13) * (y * r);
            rate_j = 0.6f * ex2f_(v * (float)(0.057 * kLog2e)) * (x * r);
        } else {
            rate_h = fmaf(0.057f, exva(v, 80, -6.8), fmaf(2.7f, ex2f_(v * (float)(0.079 * kLog2e)),
                                                          3.1e5f * ex2f_(v * (float)(0.3485 * kLog2e))));
            const float n1 = fmaf(-2.5428e4f, ex2f_(v * (float)(0.2444 * kLog2e)),
                                  -6.948e-6f * ex2f_(v * (float)(-0.04391 * kLog2e))) * (v + 37.78f);
            const float n2 = 0.02424f * ex2f_(v * (float)(-0.01052 * kLog2e));
            const float x = 1.0f + exva(v, 79.23, 1.0 / 0.311);
            const float y = 1.0f + fminf(exva(v, 40.14, -1.0 / 0.1378), 1e18f);
            rate_j = fmaf(n1, y, n2 * x) * rcpf_(x * y);
        }
        const float eh = 1.0f + exva(v, 71.55, 7.43);
        const float H_INF = rcpf_(eh * eh);
        c.sm = relaxf(c.sm, M_INF, rate_m, ndtl);
        c.sh = relaxf(c.sh, H_INF, rate_h, ndtl);
        c.sj = relaxf(c.sj, H_INF, rate_j, ndtl);
    }
    const float INa = mulp(14.838f * c.sm * c.sm * c.sm * c.sh * c.sj, v - ENa);

    // INaL, TPORd.cc:509-528
    const float mLss = sigva(v, 42.85, -5.264);
    const float rate_mL = fmaf(6.765f, exva(v, 11.64, 34.77), 8.552f * exva(v, 77.42, -5.955));
    c.mL = relaxf(c.mL, mLss, rate_mL, ndtl);
    {
        const float x = fminf(exva(v, 87.61, 7.488), 1e18f);
        const float p = 1.0f + x, q = fmaf(2.288717124596482f, x, 1.0f);   // exp((v + 93.81)/7.488)
        const float r = rcpf_(p * q);
        const float hLss = mulp(q, r), hLssp = mulp(p, r);
        c.hL = fmaf(c.hL - hLss, k.e_hl, hLss);
        c.hLp = fmaf(c.hLp - hLssp, k.e_hlp, hLssp);
    }
    const float GNaL = epi ? (float)(0.0075 * 0.6) : 0.0075f;
    const float INaL = mulp(GNaL * (v - ENa) * c.mL, fmaf(1.0f - fP, c.hL, fP * c.hLp));

    // Ito, TPORd.cc:530-571
    {
        const float x = exva(v, -14.34, -14.82);
        const float p = 1.0f + x, q = fmaf(1.9635691902911017f, x, 1.0f);   // exp(-(v - 24.34)/14.82)
        const float r = rcpf_(p * q);
        const float ass = mulp(q, r), assp = mulp(p, r);
        // 1/ta from its two terms over one denominator
        const float y = 1.0f + exva(v, -18.4099, -29.3814), z = 1.0f + exva(v, 100, 29.3814);
        const float rate_a = fmaf((float)(1.0 / (1.2089 * 1.0515)), z, (float)(3.5 / 1.0515) * y) * rcpf_(y * z);
        const float e_ta = ex2f_(ndtl * rate_a);
        c.a = fmaf(c.a - ass, e_ta, ass);
        c.ap = fmaf(c.ap - assp, e_ta, assp);
    }
    const float iss = sigva(v, 43.94, 5.711);
    {
        // tiF = (4.562 + 1/sF) delta, tiS = (23.62 + 1/sS) delta
        const float sF = fminf(fmaf(0.3933f, exva(v, 100, -100), 0.08004f * exva(v, 50, 16.59)), 1e12f);
        const float sS = fminf(fmaf(0.001416f, exva(v, 96.52, -59.05), 1.780e-8f * exva(v, 114.1, 8.079)), 1e12f);
        const float dF = fmaf(4.562f, sF, 1.0f), dS = fmaf(23.62f, sS, 1.0f);
        // delta = 1 - 0.95/(1 + z) in the epicardium, else 1
        const float z = fminf(1202604.2841647768f * E5, 1e10f);   // exp((v + 70)/5)
        const float dn = epi ? 1.0f + z : 1.0f, dd = epi ? 0.05f + z : 1.0f;
        const float r = rcpf_(dF * dS * dd) * dn;
        const float rF = sF * dS * r, rS = sS * dF * r;
        // 1/(dti_develop dti_recover)
        const float t = fminf(exva(v, -167.4, 15.89) + exva(v, -12.23, -0.2154), 1e15f);
        const float w = fminf(33.11545195869231f * E20, 1e15f);   // exp((v + 70)/20)
        const float f = t * (1.0f + w) * rcpf_(fmaf(1.354f, t, 1.0e-4f) * (0.5f + w));
        c.iF = relaxf(c.iF, iss, rF, ndtl);
        c.iS = relaxf(c.iS, iss, rS, ndtl);
        c.iFp = relaxf(c.iFp, iss, rF * f, ndtl);
        c.iSp = relaxf(c.iSp, iss, rS * f, ndtl);
    }
    const float AiF = sigva(v, -213.6, 151.2);
    const float ii = fmaf(AiF, c.iF, (1.0f - AiF) * c.iS);
    const float ip = fmaf(AiF, c.iFp, (1.0f - AiF) * c.iSp);
    const float Gto = (epi || mid) ? (float)(0.02 * 4.0) : 0.02f;
    const float Ito = mulp(Gto * (v - EK), fmaf((1.0f - fP) * c.a, ii, fP * c.ap * ip));

    // ICaL, ICaNa, ICaK, TPORd.cc:573-652
    {
        const float dss = rcpf_(1.0f + ex2f_((v + (3.940f + m.dss_shift)) * (float)(-kLog2e / 4.230)));
        const float s = fminf(fmaf(0.7408182206817179f, I20, exva(v, 14, 1.0 / 0.09)), 1e12f);   // exp(-0.05 (v + 6))
        c.d = relaxf(c.d, dss, s * rcpf_(fmaf(0.6f, s, 1.0f)), ndtl);
    }
    const float fss = rcpf_(1.0f + ex2f_((v + (19.58f + m.fss_shift)) * (float)(kLog2e / 3.696)));   // = fcass
    const float E7 = ex2f_(v * (float)(kLog2e / 7.0)), I7 = ex2f_(v * (float)(-kLog2e / 7.0));
    {
        // tff = 7 + 1/sf, tfs = 1000 + 1/ss
        const float sf = fminf(fmaf((float)(0.0045 * 0.1353352832366127), I10, (float)(0.0045 * 7.38905609893065) * E10), 1e12f);
        const float ss = fminf(0.000035f * (exva(v, 5, -4) + exva(v, 5, 6)), 1e12f);
        const float df = fmaf(7.0f, sf, 1.0f), ds = fmaf(1000.0f, ss, 1.0f);
        const float r = rcpf_(df * ds);
        const float rf = sf * ds * r;
        c.ff = relaxf(c.ff, fss, rf, ndtl);
        c.ffp = relaxf(c.ffp, fss, 0.4f * rf, ndtl);
        c.fs = relaxf(c.fs, fss, ss * df * r, ndtl);
    }
    {
        // tfcaf = 7 + 1/sf, tfcas = 100 + 1/ss
        const float sf = fminf(fmaf((float)(0.04 * 1.770794952435155), I7, (float)(0.04 * 0.5647181220077593) * E7), 1e12f);
        const float ss = fminf(0.00012f * (ex2f_(v * (float)(-kLog2e / 3.0)) + E7), 1e12f);
        const float df = fmaf(7.0f, sf, 1.0f), ds = fmaf(100.0f, ss, 1.0f);
        const float r = rcpf_(df * ds);
        const float rf = sf * ds * r;
        c.fcaf = relaxf(c.fcaf, fss, rf, ndtl);
        c.fcafp = relaxf(c.fcafp, fss, 0.4f * rf, ndtl);
        c.fcas = relaxf(c.fcas, fss, ss * df * r, ndtl);
    }
    const float Afcaf = fmaf(0.6f, rcpf_(fmaf(0.36787944117144233f, E10, 1.0f)), 0.3f);   // exp((v - 10)/10)
    const float Afcas = 1.0f - Afcaf;
    c.jca = fmaf(c.jca - fss, k.e_jca, fss);
    {
        const float q = fmaf(0.002f, rcass, 1.0f), q2 = q * q;
        const float nss = rcpf_(fmaf(1.0e-3f * c.jca, q2 * q2, 1.0f));   // anca k2n / km2n
        c.nca = relaxf(c.nca, nss, c.jca, ndtl);
    }
    const float fs4 = mulp(0.4f, c.fs), fcs = mulp(Afcas, c.fcas);
    const float f = fmaf(0.6f, c.ff, fs4), fp = fmaf(0.6f, c.ffp, fs4);
    const float fca = fmaf(Afcaf, c.fcaf, fcs), fcap = fmaf(Afcaf, c.fcafp, fcs);
    float PhiCaL, PhiCaNa, PhiCaK, INab_phi, ICab_phi;
    {
        // em1 = e^x - 1, x = v F / RT
        const float x = vfrt;
        float p = fmaf(x, 1.0f / 40320.0f, 1.0f / 5040.0f);
        p = fmaf(x, p, 1.0f / 720.0f);
        p = fmaf(x, p, 1.0f / 120.0f);
        p = fmaf(x, p, 1.0f / 24.0f);
        p = fmaf(x, p, 1.0f / 6.0f);
        p = fmaf(x, p, 0.5f);
        p = fmaf(x * x, p, x);
        const float em1 = fabsf(x) < 0.5f ? p : ex2f_(x * (float)kLog2e) - 1.0f;
        const float e1 = em1 + 1.0f, e1p = e1 + 1.0f;
        const float e2m1 = mulp(em1, e1p), e2 = e2m1 + 1.0f;
        // vffrt/(e1 - 1) = F x/(e^x - 1) and vffrt/(e2 - 1), 1 - x/2 near 0
        const float r = rcpf_(e2m1) * x;
        const bool tiny = fabsf(x) < 1e-4f;
        const float g1 = (float)F_ * (tiny ? fmaf(-0.5f, x, 1.0f) : r * e1p);
        const float g2 = (float)F_ * (tiny ? fmaf(-0.5f, x, 0.5f) : r);
        PhiCaL = 4.0f * g2 * fmaf(cass, e2, (float)(-0.341 * cao));
        PhiCaNa = g1 * fmaf(0.75f * nass, e1, (float)(-0.75 * nao));
        PhiCaK = g1 * fmaf(0.75f * kss, e1, (float)(-0.75 * ko));
        INab_phi = g1 * fmaf(nai, e1, (float)-nao);
        ICab_phi = 4.0f * g2 * fmaf(cai, e2, (float)(-0.341 * cao));
    }
    const float PCa = epi ? m.pca[1] : (mid ? m.pca[2] : m.pca[0]);
    const float jn = c.jca * c.nca;
    const float gate_np = c.d * fmaf(f, 1.0f - c.nca, fca * jn);
    const float gate_p = c.d * fmaf(fp, 1.0f - c.nca, fcap * jn);
    // (1 - fP) PCa gate_np + fP (1.1 PCa) gate_p, shared by the three fluxes
    const float G = PCa * fmaf(1.0f - fP, gate_np, 1.1f * fP * gate_p);
    const float ICaL = mulp(G, PhiCaL);
    const float ICaNa = mulp(0.00125f * G, PhiCaNa);
    const float ICaK = mulp(3.574e-4f * G, PhiCaK);

    // IKr, TPORd.cc:654-678 (sqrt(ko/5.4) = 1)
    const float xrss = sigva(v, 8.337, -6.789);
    {
        const float sf = fminf(fmaf(0.3652f, exva(v, -31.66, 3.869), 4.123e-5f * exva(v, -47.78, -20.38)), 1e12f);
        const float ss = fminf(fmaf(0.06629f, exva(v, -34.70, 7.355), 1.128e-5f * exva(v, -29.74, -25.94)), 1e12f);
        const float df = fmaf(12.98f, sf, 1.0f), ds = fmaf(1.865f, ss, 1.0f);
        const float r = rcpf_(df * ds);
        c.xrf = relaxf(c.xrf, xrss, sf * ds * r, ndtl);
        c.xrs = relaxf(c.xrs, xrss, ss * df * r, ndtl);
    }
    float IKr;
    {
        const float p = 1.0f + exva(v, 54.81, 38.21);
        const float q = (1.0f + exva(v, 55, 75)) * (1.0f + exva(v, -10, 30));
        const float r = rcpf_(p * q);
        const float Axrf = mulp(q, r), rkr = p * r;
        const float xr = fmaf(Axrf, c.xrf, (1.0f - Axrf) * c.xrs);
        const float GKr = epi ? (float)(0.046 * 1.3) : (mid ? (float)(0.046 * 0.8) : 0.046f);
        IKr = mulp(GKr * xr * rkr, v - EK);
    }

    // IKs, TPORd.cc:680-735
    const float xs1ss = sigva(v, 11.60, -8.932);
    {
        const float s = fminf(fmaf(2.326e-4f, exva(v, 48.28, 17.80), 0.001292f * exva(v, 210, -230)), 1e12f);
        c.xs1 = relaxf(c.xs1, xs1ss, s * rcpf_(fmaf(817.3f, s, 1.0f)), ndtl);
        const float rate2 = fmaf((float)(0.01 * 0.0820849986238988), E20, 0.0193f * exva(v, 66.54, -31));
        c.xs2 = relaxf(c.xs2, xs1ss, rate2, ndtl);
    }
    // 1 + 0.6/(1 + (3.8e-5/cai)^1.4)
    constexpr double lg_ks = -14.683641055880589;   // log2(3.8e-5)
    const float KsCa = fmaf(0.6f, rcpf_(1.0f + ex2f_(1.4f * ((float)lg_ks - lg2f_(cai)))), 1.0f);
    const float GKs = epi ? m.gks[1] : (mid ? m.gks[2] : m.gks[0]);
    const float IKs = mulp(GKs * KsCa * c.xs1 * c.xs2, v - EKs);

    // IK1, TPORd.cc:738-751 (sqrt(ko) constant)
    float rk1;
    {
        const float x = 1.0f + exva(v, 2.5538 * ko + 144.59, -(1.5692 * ko + 3.8115));
        const float y = 1.0f + fminf(exva(v, 105.8 - 2.6 * ko, 9.493), 1e18f);
        const float r = rcpf_(x * y);
        rk1 = x * r;
        const float rate = (float)(1.0 / 122.2) * (exva(v, 127.2, -20.36) + exva(v, 236.8, 69.33));
        c.xk1 = relaxf(c.xk1, mulp(y, r), rate, ndtl);
    }
    const float GK1 = epi ? (float)(0.1908 * 1.2) : (mid ? (float)(0.1908 * 1.3) : 0.1908f);
    const float IK1 = mulp(GK1 * 2.32379000772445f /* sqrt(ko) */ * rk1 * c.xk1, v - EK);

    // INaCa_i and INaCa_ss, TPORd.cc:753-852
    constexpr double kna1 = 15.0, kna2 = 5.0, kna3 = 88.12, kasymm = 12.5;
    constexpr double wna = 6.0e4, wca = 6.0e4, wnaca = 5.0e3, kcaon = 1.5e6;
    constexpr double h10 = kasymm + 1.0 + nao / kna1 * (1.0 + nao / kna2);
    constexpr double h11 = nao * nao / (h10 * kna1 * kna2);
    constexpr double k1 = cao * kcaon / h10;
    constexpr float k2 = 5.0e3f;   // kcaoff; k5 = k2
    const float ihca = ex2f_(v * (float)(-0.1670 * FRT * kLog2e));
    const float hna = ex2f_(v * (float)(0.5224 * FRT * kLog2e));
    // h8 = nao/(kna3 hna h7), h9 = 1/h7 with h7 = 1 + nao/kna3 (1 + 1/hna)
    const float r7 = rcpf_(fmaf(hna, (float)(kna3 + nao), (float)nao));
    const float h8 = (float)nao * r7;
    const float k3pp = mulp(h8, (float)wnaca);
    const float k3 = fmaf((float)(kna3 * wca) * hna, r7, k3pp);
    const float k8 = mulp(h8, (float)(h11 * wna));
    const float Gncx = epi ? (float)(0.0008 * 1.1) : (mid ? (float)(0.0008 * 1.4) : 0.0008f);
    const float hna1 = (1.0f + hna) * (float)(1.0 / kna3);
    float INaCa_i, INaCa_ss;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
        const float na = pass == 0 ? nai : nass;
        const float ca = pass == 0 ? cai : cass;
        const float h1 = fmaf(na, hna1, 1.0f);
        const float h4 = fmaf(na * (float)(1.0 / kna1), fmaf(na, (float)(1.0 / kna2), 1.0f), 1.0f);
        const float r14 = rcpf_(h1 * h4);
        const float h3 = h4 * r14, h6 = h1 * r14;      // 1/h1, 1/h4
        const float h2 = na * hna * (float)(1.0 / kna3) * h3;
        const float h5 = na * na * (float)(1.0 / (kna1 * kna2)) * h6;
        const float k4pp = mulp(h2, (float)wnaca);
        const float k4 = fmaf(h3 * (float)wca, ihca, k4pp);
        const float k6 = mulp(h6 * ca, (float)kcaon);
        const float k7 = mulp(h5 * h2, (float)wna);
        const float k67 = k6 + k7, k23 = k2 + k3, k45 = k4 + k2, k18 = (float)k1 + k8;
        const float x1 = mulp(k2, fmaf(k4, k67, k7 * k23));
        const float x2 = fmaf((float)k1 * k7, k45, k4 * k6 * k18);
        const float x3 = fmaf((float)k1 * k3, k67, k8 * k6 * k23);
        const float x4 = mulp(k2, fmaf(k8, k45, k3 * k18));
        const float xs = (x1 + x2) + (x3 + x4);
        // J = (3 (x4 k7 - x1 k8) + x3 k4pp - x2 k3pp + 2 (x2 k2 - x1 k1)) / xs; allo = ca^2/(ca^2 + KmCaAct^2)
        const float a = fmaf(x4, k7, -mulp(x1, k8)), b = fmaf(x2, k2, -mulp(x1, (float)k1));
        const float num = fmaf(2.0f, b, fmaf(3.0f, a, fmaf(x3, k4pp, -mulp(x2, k3pp))));
        const float ca2 = mulp(ca, ca);
        const float val = Gncx * num * ca2 * rcpf_(xs * (ca2 + (float)(150.0e-6 * 150.0e-6)));
        if (pass == 0) INaCa_i = mulp(0.8f, val);
        else INaCa_ss = mulp(0.2f, val);
    }
    const float INaCa = INaCa_i + INaCa_ss;

    // INaK, TPORd.cc:854-906
    float INaK;
    {
        constexpr double k1p = 949.5, k1m = 182.4, k2p = 687.2, k2m = 39.4;
        constexpr double k3p_ = 1899.0, k3m = 79300.0, k4p_ = 639.0, k4m = 40.0;
        constexpr double Knai0 = 9.073, Knao0 = 27.78, delta = -0.1550;
        constexpr double Kki = 0.5, Kko = 0.3582, MgADP = 0.05, MgATP = 9.8, Kmgatp = 1.698e-7;
        constexpr double H = 1.0e-7, eP = 4.2, Khp = 1.698e-7, Knap = 224.0, Kxkur = 292.0;
        constexpr double rko = ko / Kko;
        const float rnai = mulp(nai * (float)(1.0 / Knai0), ex2f_(v * (float)(-delta / 3.0 * FRT * kLog2e)));
        const float rnao = mulp((float)(nao / Knao0), ex2f_(v * (float)(-(1.0 - delta) / 3.0 * FRT * kLog2e)));
        const float rki = mulp(ki, (float)(1.0 / Kki));
        const float pP = fmaf(ki, (float)(1.0 / Kxkur), fmaf(nai, (float)(1.0 / Knap), (float)(1.0 + H / Khp)));   // eP/P
        const float pnai = 1.0f + rnai, pnao = 1.0f + rnao, pki = 1.0f + rki;
        const float den_i = fmaf(pnai * pnai, pnai, fmaf(pki, pki, -1.0f));
        const float den_o = fmaf(pnao * pnao, pnao, (float)((1.0 + rko) * (1.0 + rko) - 1.0));
        const float rio = rcpf_(den_i * den_o);
        const float ri = den_o * rio, ro = den_i * rio;
        const float a1 = mulp((float)k1p * (rnai * rnai * rnai), ri);
        const float b4 = mulp((float)k4m * (rki * rki), ri);
        const float b2 = mulp((float)k2m * (rnao * rnao * rnao), ro);
        const float a3 = mulp((float)(k3p_ * rko * rko), ro);
        const float b3 = mulp((float)(k3m * H / (1.0 + MgATP / Kmgatp) * eP), rcpf_(pP));
        constexpr float b1 = (float)(k1m * MgADP), a2 = (float)k2p;
        constexpr float a4 = (float)((k4p_ * MgATP / Kmgatp) / (1.0 + MgATP / Kmgatp));
        const float b43 = mulp(b4, b3), b23 = mulp(b2, b3);
        const float y1 = fmaf(a2, fmaf(a1, a4 + b3, b43), b2 * b43);
        const float y2 = fmaf(b1 * b4, b2 + a3, a2 * a3 * (a1 + b4));
        const float y3 = fmaf(a3 * a4, a2 + b1, b1 * b2 * (b3 + a4));
        const float y4 = fmaf(b23, b4 + a1, a4 * a1 * (a3 + b2));
        const float J = fmaf(3.0f, fmaf(y1, a3, -mulp(y2, b3)), 2.0f * fmaf(y4, b1, -mulp(y3, a1)));
        const float Pnak = epi ? (float)(30 * 0.9) : (mid ? (float)(30 * 0.7) : 30.0f);
        INaK = mulp(Pnak * J, rcpf_((y1 + y2) + (y3 + y4)));
    }

    // background currents and pump, TPORd.cc:908-923
    const float GKb = epi ? (float)(0.003 * 0.6) : 0.003f;
    const float IKb = mulp(GKb * sigva(v, -14.48, -18.34), v - EK);
    const float INab = mulp(3.75e-10f, INab_phi);
    const float ICab = mulp(2.5e-8f, ICab_phi);
    // cytosolic buffer and pump: Bcai = 1/(1 + cm/qc^2 + ct/qt^2), IpCa = 0.0005 cai/qt (qt = 0.0005 + cai)
    constexpr double cmdnmax = 0.05, kmcmdn = 0.00238, trpnmax = 0.07, kmtrpn = 0.0005;
    float IpCa, Bcai;
    {
        const float qc = (float)kmcmdn + cai, qt = (float)kmtrpn + cai;
        const float qc2 = mulp(qc, qc), qt2 = mulp(qt, qt), qq = mulp(qc2, qt2);
        const float cm = epi ? (float)(1.3 * cmdnmax * kmcmdn) : (float)(cmdnmax * kmcmdn);
        const float D = fmaf((float)(trpnmax * kmtrpn), qc2, fmaf(cm, qt2, qq));
        const float r = rcpf_(D * qt);
        Bcai = qq * (r * qt);
        IpCa = mulp(0.0005f * cai, r * D);
    }

    // membrane potential, TPORd.cc:927-935
    const float Iion = INa + INaL + Ito + ICaL + ICaNa + ICaK + IKr + IKs + IK1 + INaCa + INaK + INab + IKb + IpCa + ICab;
    const float dV_dt = -(Iion + Ist);
    c.v = fmaf(dV_dt + dVgap_dt, dt, v);
    if (out) {
        out->dvdt = dV_dt;
        out->ical = ICaL;
        out->iks = IKs;
        out->ina = INa;
        out->ikr = IKr;
        out->ik1 = IK1;
    }

    // CaMK and fluxes, TPORd.cc:939-995
    c.CaMKt = fmaf(dt, fmaf(0.05f * CaMKb, CaMKa, -mulp(0.00068f, c.CaMKt)), c.CaMKt);
    // concentration differences from the full-precision values (file comment of tpord.cuh)
    const float JdiffNa = mulp(cdiff(c.nass, c.nai), 0.5f);
    const float JdiffK = mulp(cdiff(c.kss, c.ki), 0.5f);
    const float Jdiff = mulp(cdiff(c.cass, c.cai), 5.0f);
    const float Jtr = mulp(cdiff(c.cansr, c.cajsr), 0.01f);
    {
        // 1/(1 + (1.5/cajsr)^8) and 1/cajsr from one reciprocal
        // (bounded: beyond 200 mM the first is 1, and j8 itself would overflow from 65,000 on)
        const float j2 = cajsr * cajsr, j4 = j2 * j2, j8 = fminf(mulp(j4, j4), 1e18f);
        const float dj = j8 + 25.62890625f;
        const float r = rcpf_(fmaf(dj, cajsr, kTiny));
        const float rel = (mid ? 1.7f : 1.0f) * -ICaL * j8 * (r * cajsr);
        // 1/tau_rel; tau_rel below 0.005, negative ones too (cajsr < 0), is 0.005: the
        // sign bit makes a negative rate the larger unsigned number
        const float rate = fmaf((float)(0.0123 / 4.75), r * dj, (float)(1.0 / 4.75));
        auto bound = [](float x) { return __float_as_uint(x) < 0x43480000u ? x : 200.0f; };
        const float Jrel_inf = mulp((float)(0.5 * 4.75), rel), Jrel_infp = mulp((float)(0.5 * 1.25 * 4.75), rel);
        c.Jrelnp = relaxf(c.Jrelnp, Jrel_inf, bound(rate), ndtl);
        c.Jrelp = relaxf(c.Jrelp, Jrel_infp, bound(0.8f * rate), ndtl);
    }
    const float Jrel = fmaf(1.0f - fP, c.Jrelnp, fP * c.Jrelp);
    float Jup;
    {
        const float p = cai + 0.00092f, q = cai + (float)(0.00092 - 0.00017);
        const float s = (epi ? 1.3f : 1.0f) * cai * rcpf_(p * q);
        const float u = fmaf((1.0f - fP) * 0.004375f, q, fP * (float)(2.75 * 0.004375) * p);
        Jup = fmaf(s, u, -mulp((float)(0.0039375 / 15.0), cansr));
    }

    // concentrations, forward Euler, TPORd.cc:997-1020
    constexpr float cm = (float)(Acap / (F_ * vmyo)), cs = (float)(Acap / (F_ * vss));
    const float dnai = fmaf(-fmaf(3.0f, INaCa_i + INaK, INa + INaL + INab), cm, JdiffNa * (float)(vss / vmyo));
    const float dnass = fmaf(-fmaf(3.0f, INaCa_ss, ICaNa), cs, -JdiffNa);
    const float dki = fmaf(-fmaf(-2.0f, INaK, Ito + IKr + IKs + IK1 + IKb + Ist), cm, JdiffK * (float)(vss / vmyo));
    const float dkss = fmaf(-ICaK, cs, -JdiffK);
    const float dcai = Bcai * fmaf(-fmaf(-2.0f, INaCa_i, IpCa + ICab), 0.5f * cm,
                                   fmaf(-Jup, (float)(vnsr / vmyo), Jdiff * (float)(vss / vmyo)));
    // Bcass and Bcajsr from one reciprocal
    constexpr double BSRmax = 0.047, KmBSR = 0.00087, BSLmax = 1.124, KmBSL = 0.0087;
    constexpr double csqnmax = 10.0, kmcsqn = 0.8;
    const float qsr = (float)KmBSR + cass, qsl = (float)KmBSL + cass, qj = (float)kmcsqn + cajsr;
    const float qsr2 = mulp(qsr, qsr), qsl2 = mulp(qsl, qsl), qs = mulp(qsr2, qsl2), qj2 = mulp(qj, qj);
    const float Ds = fmaf((float)(BSLmax * KmBSL), qsr2, fmaf((float)(BSRmax * KmBSR), qsl2, qs));
    const float Dj = qj2 + (float)(csqnmax * kmcsqn);
    const float rsj = rcpf_(Ds * Dj);
    const float Bcass = qs * (Dj * rsj), Bcajsr = qj2 * (Ds * rsj);
    const float dcass = Bcass * fmaf(-fmaf(-2.0f, INaCa_ss, ICaL), 0.5f * cs, fmaf(Jrel, (float)(vjsr / vss), -Jdiff));
    const float dcansr = fmaf(-Jtr, (float)(vjsr / vnsr), Jup);
    const float dcajsr = Bcajsr * (Jtr - Jrel);
    cadd(c.nai, dt * dnai);
    cadd(c.nass, dt * dnass);
    cadd(c.ki, dt * dki);
    cadd(c.kss, dt * dkss);
    cadd(c.cai, dt * dcai);
    cadd(c.cass, dt * dcass);
    cadd(c.cansr, dt * dcansr);
    cadd(c.cajsr, dt * dcajsr);
}

// The step of the cell, grid and surrogate kernels in each form.
__device__ __forceinline__ void tpord_update(CellState<float> &c, int ctype, const ModelT<float> &m,
                                             const StepT<float> &k, float Ist, float dVgap_dt, StepOut<float> *out)
{
    tpord_step_f32(c, ctype, m, k, Ist, dVgap_dt, out);
}

}  // namespace lqt
