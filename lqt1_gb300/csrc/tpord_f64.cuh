// tpord_f64.cuh -- one TPORd step in the FP64 form.
//
// What bounds it.  GB300 issues FP64 at 1/64 of its FP32 rate, so the step's
// time is its count of FP64 instructions (the FP64 pipe 86% busy).  Written
// expression by expression (SingleCell/TPORd.cc:379-1021) with the library's
// exp, log and division it is 3624 of them per cell; here less than half:
//   * an exponential is 9 with its argument: reduction by 2^(j/256) from a table
//     of 256 correctly rounded powers (the table is read and the exponent added
//     by the load and integer pipes), a fourth-degree polynomial on
//     |x| <= 1/512 (truncation 2^-58.5); two units of 2^-53 in all;
//   * a reciprocal is 3: the hardware's approximation (2^-20 or better) and one
//     third-order correction r (1 + e + e^2), e = 1 - d r;
//   * a logarithm is 9, from an FP32 estimate, the table and ln(1 + x);
//   * the terms are arranged as in tpord_f32.cuh (rates for time constants,
//     shared reciprocals and exponentials), without its bounds: exponentials
//     saturate at 2^+-100, far outside their effect on any term, and products
//     of several stay finite; a shared reciprocal's product of a calcium
//     concentration is kept off zero by 1e-60 (kTinyD).
// Each of these is within a few units of 2^-53; the argument (v + a) / k of an
// exponential is one FMA with a / k rounded, so near v = -a, where the sum
// cancels, it is up to 25 such units off and not a fraction of one.  After one
// step of 20,000 cells (-120 to 80 mV) the state values agree with the oracle to
// 6e-12 of their size at the worst and 99.9% of them to 3e-14, V to 3e-16.
// Measured (GB300): shell of 78k voxels 684 -> 297 us a step.
#pragma once
#include <cuda_runtime.h>

namespace lqt {

// 2^(j/256), correctly rounded
static __device__ const double kEx2Table[256] = {
    0x1.0000000000000p+0, 0x1.00b1afa5abcbfp+0, 0x1.0163da9fb3335p+0, 0x1.02168143b0281p+0,
    0x1.02c9a3e778061p+0, 0x1.037d42e11bbccp+0, 0x1.04315e86e7f85p+0, 0x1.04e5f72f654b1p+0,
    0x1.059b0d3158574p+0, 0x1.0650a0e3c1f89p+0, 0x1.0706b29ddf6dep+0, 0x1.07bd42b72a836p+0,
    0x1.0874518759bc8p+0, 0x1.092bdf66607e0p+0, 0x1.09e3ecac6f383p+0, 0x1.0a9c79b1f3919p+0,
    0x1.0b5586cf9890fp+0, 0x1.0c0f145e46c85p+0, 0x1.0cc922b7247f7p+0, 0x1.0d83b23395decp+0,
    0x1.0e3ec32d3d1a2p+0, 0x1.0efa55fdfa9c5p+0, 0x1.0fb66affed31bp+0, 0x1.1073028d7233ep+0,
    0x1.11301d0125b51p+0, 0x1.11edbab5e2ab6p+0, 0x1.12abdc06c31ccp+0, 0x1.136a814f204abp+0,
    0x1.1429aaea92de0p+0, 0x1.14e95934f312ep+0, 0x1.15a98c8a58e51p+0, 0x1.166a45471c3c2p+0,
    0x1.172b83c7d517bp+0, 0x1.17ed48695bbc0p+0, 0x1.18af9388c8deap+0, 0x1.1972658375d2fp+0,
    0x1.1a35beb6fcb75p+0, 0x1.1af99f8138a1cp+0, 0x1.1bbe084045cd4p+0, 0x1.1c82f95281c6bp+0,
    0x1.1d4873168b9aap+0, 0x1.1e0e75eb44027p+0, 0x1.1ed5022fcd91dp+0, 0x1.1f9c18438ce4dp+0,
    0x1.2063b88628cd6p+0, 0x1.212be3578a819p+0, 0x1.21f49917ddc96p+0, 0x1.22bdda27912d1p+0,
    0x1.2387a6e756238p+0, 0x1.2451ffb82140ap+0, 0x1.251ce4fb2a63fp+0, 0x1.25e85711ece75p+0,
    0x1.26b4565e27cddp+0, 0x1.2780e341ddf29p+0, 0x1.284dfe1f56381p+0, 0x1.291ba7591bb70p+0,
    0x1.29e9df51fdee1p+0, 0x1.2ab8a66d10f13p+0, 0x1.2b87fd0dad990p+0, 0x1.2c57e39771b2fp+0,
    0x1.2d285a6e4030bp+0, 0x1.2df961f641589p+0, 0x1.2ecafa93e2f56p+0, 0x1.2f9d24abd886bp+0,
    0x1.306fe0a31b715p+0, 0x1.31432edeeb2fdp+0, 0x1.32170fc4cd831p+0, 0x1.32eb83ba8ea32p+0,
    0x1.33c08b26416ffp+0, 0x1.3496266e3fa2dp+0, 0x1.356c55f929ff1p+0, 0x1.36431a2de883bp+0,
    0x1.371a7373aa9cbp+0, 0x1.37f26231e754ap+0, 0x1.38cae6d05d866p+0, 0x1.39a401b7140efp+0,
    0x1.3a7db34e59ff7p+0, 0x1.3b57fbfec6cf4p+0, 0x1.3c32dc313a8e5p+0, 0x1.3d0e544ede173p+0,
    0x1.3dea64c123422p+0, 0x1.3ec70df1c5175p+0, 0x1.3fa4504ac801cp+0, 0x1.40822c367a024p+0,
    0x1.4160a21f72e2ap+0, 0x1.423fb2709468ap+0, 0x1.431f5d950a897p+0, 0x1.43ffa3f84b9d4p+0,
    0x1.44e086061892dp+0, 0x1.45c2042a7d232p+0, 0x1.46a41ed1d0057p+0, 0x1.4786d668b3237p+0,
    0x1.486a2b5c13cd0p+0, 0x1.494e1e192aed2p+0, 0x1.4a32af0d7d3dep+0, 0x1.4b17dea6db7d7p+0,
    0x1.4bfdad5362a27p+0, 0x1.4ce41b817c114p+0, 0x1.4dcb299fddd0dp+0, 0x1.4eb2d81d8abffp+0,
    0x1.4f9b2769d2ca7p+0, 0x1.508417f4531eep+0, 0x1.516daa2cf6642p+0, 0x1.5257de83f4eefp+0,
    0x1.5342b569d4f82p+0, 0x1.542e2f4f6ad27p+0, 0x1.551a4ca5d920fp+0, 0x1.56070dde910d2p+0,
    0x1.56f4736b527dap+0, 0x1.57e27dbe2c4cfp+0, 0x1.58d12d497c7fdp+0, 0x1.59c0827ff07ccp+0,
    0x1.5ab07dd485429p+0, 0x1.5ba11fba87a03p+0, 0x1.5c9268a5946b7p+0, 0x1.5d84590998b93p+0,
    0x1.5e76f15ad2148p+0, 0x1.5f6a320dceb71p+0, 0x1.605e1b976dc09p+0, 0x1.6152ae6cdf6f4p+0,
    0x1.6247eb03a5585p+0, 0x1.633dd1d1929fdp+0, 0x1.6434634ccc320p+0, 0x1.652b9febc8fb7p+0,
    0x1.6623882552225p+0, 0x1.671c1c70833f6p+0, 0x1.68155d44ca973p+0, 0x1.690f4b19e9538p+0,
    0x1.6a09e667f3bcdp+0, 0x1.6b052fa75173ep+0, 0x1.6c012750bdabfp+0, 0x1.6cfdcddd47645p+0,
    0x1.6dfb23c651a2fp+0, 0x1.6ef9298593ae5p+0, 0x1.6ff7df9519484p+0, 0x1.70f7466f42e87p+0,
    0x1.71f75e8ec5f74p+0, 0x1.72f8286ead08ap+0, 0x1.73f9a48a58174p+0, 0x1.74fbd35d7cbfdp+0,
    0x1.75feb564267c9p+0, 0x1.77024b1ab6e09p+0, 0x1.780694fde5d3fp+0, 0x1.790b938ac1cf6p+0,
    0x1.7a11473eb0187p+0, 0x1.7b17b0976cfdbp+0, 0x1.7c1ed0130c132p+0, 0x1.7d26a62ff86f0p+0,
    0x1.7e2f336cf4e62p+0, 0x1.7f3878491c491p+0, 0x1.80427543e1a12p+0, 0x1.814d2add106d9p+0,
    0x1.82589994cce13p+0, 0x1.8364c1eb941f7p+0, 0x1.8471a4623c7adp+0, 0x1.857f4179f5b21p+0,
    0x1.868d99b4492edp+0, 0x1.879cad931a436p+0, 0x1.88ac7d98a6699p+0, 0x1.89bd0a478580fp+0,
    0x1.8ace5422aa0dbp+0, 0x1.8be05bad61778p+0, 0x1.8cf3216b5448cp+0, 0x1.8e06a5e0866d9p+0,
    0x1.8f1ae99157736p+0, 0x1.902fed0282c8ap+0, 0x1.9145b0b91ffc6p+0, 0x1.925c353aa2fe2p+0,
    0x1.93737b0cdc5e5p+0, 0x1.948b82b5f98e5p+0, 0x1.95a44cbc8520fp+0, 0x1.96bdd9a7670b3p+0,
    0x1.97d829fde4e50p+0, 0x1.98f33e47a22a2p+0, 0x1.9a0f170ca07bap+0, 0x1.9b2bb4d53fe0dp+0,
    0x1.9c49182a3f090p+0, 0x1.9d674194bb8d5p+0, 0x1.9e86319e32323p+0, 0x1.9fa5e8d07f29ep+0,
    0x1.a0c667b5de565p+0, 0x1.a1e7aed8eb8bbp+0, 0x1.a309bec4a2d33p+0, 0x1.a42c980460ad8p+0,
    0x1.a5503b23e255dp+0, 0x1.a674a8af46052p+0, 0x1.a799e1330b358p+0, 0x1.a8bfe53c12e59p+0,
    0x1.a9e6b5579fdbfp+0, 0x1.ab0e521356ebap+0, 0x1.ac36bbfd3f37ap+0, 0x1.ad5ff3a3c2774p+0,
    0x1.ae89f995ad3adp+0, 0x1.afb4ce622f2ffp+0, 0x1.b0e07298db666p+0, 0x1.b20ce6c9a8952p+0,
    0x1.b33a2b84f15fbp+0, 0x1.b468415b749b1p+0, 0x1.b59728de5593ap+0, 0x1.b6c6e29f1c52ap+0,
    0x1.b7f76f2fb5e47p+0, 0x1.b928cf22749e4p+0, 0x1.ba5b030a1064ap+0, 0x1.bb8e0b79a6f1fp+0,
    0x1.bcc1e904bc1d2p+0, 0x1.bdf69c3f3a207p+0, 0x1.bf2c25bd71e09p+0, 0x1.c06286141b33dp+0,
    0x1.c199bdd85529cp+0, 0x1.c2d1cd9fa652cp+0, 0x1.c40ab5fffd07ap+0, 0x1.c544778fafb22p+0,
    0x1.c67f12e57d14bp+0, 0x1.c7ba88988c933p+0, 0x1.c8f6d9406e7b5p+0, 0x1.ca3405751c4dbp+0,
    0x1.cb720dcef9069p+0, 0x1.ccb0f2e6d1675p+0, 0x1.cdf0b555dc3fap+0, 0x1.cf3155b5bab74p+0,
    0x1.d072d4a07897cp+0, 0x1.d1b532b08c968p+0, 0x1.d2f87080d89f2p+0, 0x1.d43c8eacaa1d6p+0,
    0x1.d5818dcfba487p+0, 0x1.d6c76e862e6d3p+0, 0x1.d80e316c98398p+0, 0x1.d955d71ff6075p+0,
    0x1.da9e603db3285p+0, 0x1.dbe7cd63a8315p+0, 0x1.dd321f301b460p+0, 0x1.de7d5641c0658p+0,
    0x1.dfc97337b9b5fp+0, 0x1.e11676b197d17p+0, 0x1.e264614f5a129p+0, 0x1.e3b333b16ee12p+0,
    0x1.e502ee78b3ff6p+0, 0x1.e653924676d76p+0, 0x1.e7a51fbc74c83p+0, 0x1.e8f7977cdb740p+0,
    0x1.ea4afa2a490dap+0, 0x1.eb9f4867cca6ep+0, 0x1.ecf482d8e67f1p+0, 0x1.ee4aaa2188510p+0,
    0x1.efa1bee615a27p+0, 0x1.f0f9c1cb6412ap+0, 0x1.f252b376bba97p+0, 0x1.f3ac948dd7274p+0,
    0x1.f50765b6e4540p+0, 0x1.f6632798844f8p+0, 0x1.f7bfdad9cbe14p+0, 0x1.f91d802243c89p+0,
    0x1.fa7c1819e90d8p+0, 0x1.fbdba3692d514p+0, 0x1.fd3c22b8f71f1p+0, 0x1.fe9d96b2a23d9p+0
};

constexpr double kTinyD = 1e-60;

// 2^x, saturating at 2^+-100, at infinities too (NaN stays NaN: x comes from
// arithmetic, so a NaN's high word is above infinity's).  |x| is first held at
// 1000, by its high word, so that 256 x fits the sum's low word.
__device__ __forceinline__ double ex2d(double x)
{
    constexpr double shift = 26388279066624.0;   // 1.5 * 2^44: the sum's low word is round(256 x)
    constexpr int top = 0x408F4000;              // high word of 1000.0
    const int hx = __double2hiint(x), ha = hx & 0x7fffffff;
    const bool far = (unsigned)(ha - top) <= (unsigned)(0x7ff00000 - top);
    x = __hiloint2double(far ? (hx & (int)0x80000000) | top : hx, far ? 0 : __double2loint(x));
    const double t = x + shift;
    const double r = x - (t - shift);
    const int k = min(max(__double2loint(t), -25600), 25600);
    const double T0 = __ldg(kEx2Table + (k & 255));
    const double T = __hiloint2double(__double2hiint(T0) + ((k >> 8) << 20), __double2loint(T0));
    // (2^r - 1) / r on |r| <= 1/512: ln2^i / i! with the fifth power's part spread
    // over the first and third (r^5 - T5(512 r) / (16 512^5)), which leaves a sixteenth of it
    const double p =
        fma(fma(fma(0.009618129107628477, r, 0.05550411502275755), r, 0.24022650695910072), r, 0.6931471805599393);
    return fma(T, p * r, T);
}

// 1 / x, x finite and not zero
__device__ __forceinline__ double rcpd(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// log2(x): an FP32 estimate from x's high word, rounded to k/256;
// x 2^(-k/256) = 1 + d with |d| < 1.4e-3.  -infinity at zero (and subnormal x),
// infinity at infinity, NaN for the others that are not normal and positive.
__device__ __forceinline__ double lg2d(double x)
{
    const int hi = __double2hiint(x);
    const int ex = (hi >> 20) - 1023;
    float m;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(m) : "f"(__int_as_float(0x3f800000 | ((hi & 0xfffff) << 3))));
    const int k = (ex << 8) + __float2int_rn(m * 256.0f);
    const double T0 = __ldg(kEx2Table + (-k & 255));
    const double T = __hiloint2double(__double2hiint(T0) + ((-k >> 8) << 20), __double2loint(T0));
    const double d = fma(x, T, -1.0);
    const double p = fma(fma(fma(fma(0.2, d, -0.25), d, 1.0 / 3.0), d, -0.5), d, 1.0);
    // k/256 exactly, by the sum that ex2d takes apart
    const double kd = __hiloint2double(0x42B80000 + (k >> 31), k) - 26388279066624.0;
    const int end = (hi & 0x7fffffff) < 0x00100000 ? (int)0xfff00000 : (hi == 0x7ff00000 ? hi : 0x7ff80000);
    return (unsigned)(hi - 0x00100000) < 0x7fe00000u ? fma(p * d, 1.4426950408889634, kd) : __hiloint2double(end, 0);
}

// exp((v + a) / k)
__device__ __forceinline__ double exvad(double v, double a, double k)
{
    const double c = kLog2e / k;
    return ex2d(fma(v, c, c * a));
}
// 1 / (1 + exp((v + a) / k))
__device__ __forceinline__ double sigvad(double v, double a, double k) { return rcpd(1.0 + exvad(v, a, k)); }

// x -> inf - (inf - x) exp(-rate dt), ndtl = -dt log2(e)
__device__ __forceinline__ double relaxd(double x, double inf, double rate, double ndtl)
{
    return fma(x - inf, ex2d(ndtl * rate), inf);
}

__device__ __forceinline__ void tpord_step_f64(CellState<double> &c, int ctype, const ModelT<double> &m,
                                               const StepT<double> &k, double Ist, double dVgap_dt, StepOut<double> *out)
{
    const bool epi = (ctype == 2);
    const bool mid = (ctype == 4);
    const double dt = k.dt;
    const double ndtl = dt * -kLog2e;
    const double v = c.v;

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

    const double nai = c.nai, nass = c.nass, ki = c.ki, kss = c.kss;
    const double cai = c.cai, cass = c.cass, cajsr = c.cajsr, cansr = c.cansr;

    // reversal potentials, TPORd.cc:425-427 (log2 of the outside terms folded)
    constexpr double lg_nao = 7.129283016944966, lg_ko = 2.432959407276106, lg_eks = 2.9938917005640255;
    const double ENa = (RTF * kLn2) * (lg_nao - lg2d(nai));
    const double EK = (RTF * kLn2) * (lg_ko - lg2d(ki));
    const double EKs = (RTF * kLn2) * (lg_eks - lg2d(fma(0.01833, nai, ki)));

    // CaMK, TPORd.cc:430-433; 1/cass and 1/(cass + KmCaM) from one reciprocal
    const double cq = cass + 0.0015;
    const double r_cc = rcpd(fma(cass, cq, kTinyD));
    const double rcass = r_cc * cq;
    const double CaMKb = 0.05 * (1.0 - c.CaMKt) * (r_cc * cass) * cass;
    const double CaMKa = CaMKb + c.CaMKt;
    const double fP = CaMKa * rcpd(CaMKa + 0.15);   // phosphorylated fraction (fINaLp, fItop, ...)
    const double vfrt = v * FRT;

    // exp(+-v/20) and its powers; exp(+-v/7)
    const double E20 = ex2d(v * (kLog2e / 20.0)), I20 = ex2d(v * (-kLog2e / 20.0));
    const double E10 = E20 * E20, I10 = I20 * I20;
    const double E5 = E10 * E10, I5 = I10 * I10;

    // TP06 fast INa, TPORd.cc:465-504
    {
        // 1/(AM BM), AM = 1/(1+a), BM = 0.1/(1+b) + 0.1/(1+e); a b = exp(-5)
        const double a = (6.14421235332821e-06 * I5);               // exp((-60 - v)/5)
        const double b = 1096.6331584284585 * E5;  // exp((v + 35)/5)
        const double e = exvad(v, -50, 200);
        const double rate_m = 10.0 * ((1.0067379469990854 + a) + b) * (1.0 + e) * rcpd((2.0 + b) + e);
        const double em = 1.0 + exvad(v, 56.86, -9.03);
        const double M_INF = rcpd(em * em);
        double rate_h, rate_j;   // 1/tau
        if (v >= -40.0) {
            const double x = 1.0 + exvad(v, 10.66, -11.1);
            const double y = fma(0.04076220397836621, I10, 1.0);   // 1 + exp(-0.1 (v + 32))
            const double r = rcpd(x * y);
            rate_h = (0.77 / 0.13) * (y * r);
            rate_j = 0.6 * ex2d(v * (0.057 * kLog2e)) * (x * r);
        } else {
            rate_h = fma(0.057, exvad(v, 80, -6.8), fma(2.7, ex2d(v * (0.079 * kLog2e)),
                                                          3.1e5 * ex2d(v * (0.3485 * kLog2e))));
            const double n1 = fma(-2.5428e4, ex2d(v * (0.2444 * kLog2e)),
                                  -6.948e-6 * ex2d(v * (-0.04391 * kLog2e))) * (v + 37.78);
            const double n2 = 0.02424 * ex2d(v * (-0.01052 * kLog2e));
            const double x = 1.0 + exvad(v, 79.23, 1.0 / 0.311);
            const double y = 1.0 + exvad(v, 40.14, -1.0 / 0.1378);
            rate_j = fma(n1, y, n2 * x) * rcpd(x * y);
        }
        const double eh = 1.0 + exvad(v, 71.55, 7.43);
        const double H_INF = rcpd(eh * eh);
        c.sm = relaxd(c.sm, M_INF, rate_m, ndtl);
        c.sh = relaxd(c.sh, H_INF, rate_h, ndtl);
        c.sj = relaxd(c.sj, H_INF, rate_j, ndtl);
    }
    const double INa = (14.838 * c.sm * c.sm * c.sm * c.sh * c.sj * (v - ENa));

    // INaL, TPORd.cc:509-528
    const double mLss = sigvad(v, 42.85, -5.264);
    const double rate_mL = fma(6.765, exvad(v, 11.64, 34.77), 8.552 * exvad(v, 77.42, -5.955));
    c.mL = relaxd(c.mL, mLss, rate_mL, ndtl);
    {
        const double x = exvad(v, 87.61, 7.488);
        const double p = 1.0 + x, q = fma(2.288717124596482, x, 1.0);   // exp((v + 93.81)/7.488)
        const double r = rcpd(p * q);
        const double hLss = (q * r), hLssp = (p * r);
        c.hL = fma(c.hL - hLss, k.e_hl, hLss);
        c.hLp = fma(c.hLp - hLssp, k.e_hlp, hLssp);
    }
    const double GNaL = epi ? (0.0075 * 0.6) : 0.0075;
    const double INaL = (GNaL * (v - ENa) * c.mL * fma(1.0 - fP, c.hL, fP * c.hLp));

    // Ito, TPORd.cc:530-571
    {
        const double x = exvad(v, -14.34, -14.82);
        const double p = 1.0 + x, q = fma(1.9635691902911017, x, 1.0);   // exp(-(v - 24.34)/14.82)
        const double r = rcpd(p * q);
        const double ass = (q * r), assp = (p * r);
        // 1/ta from its two terms over one denominator
        const double y = 1.0 + exvad(v, -18.4099, -29.3814), z = 1.0 + exvad(v, 100, 29.3814);
        const double rate_a = fma((1.0 / (1.2089 * 1.0515)), z, (3.5 / 1.0515) * y) * rcpd(y * z);
        const double e_ta = ex2d(ndtl * rate_a);
        c.a = fma(c.a - ass, e_ta, ass);
        c.ap = fma(c.ap - assp, e_ta, assp);
    }
    const double iss = sigvad(v, 43.94, 5.711);
    {
        // tiF = (4.562 + 1/sF) delta, tiS = (23.62 + 1/sS) delta
        const double sF = fma(0.3933, exvad(v, 100, -100), 0.08004 * exvad(v, 50, 16.59));
        const double sS = fma(0.001416, exvad(v, 96.52, -59.05), 1.780e-8 * exvad(v, 114.1, 8.079));
        const double dF = fma(4.562, sF, 1.0), dS = fma(23.62, sS, 1.0);
        // delta = 1 - 0.95/(1 + z) in the epicardium, else 1
        const double z = 1202604.2841647768 * E5;   // exp((v + 70)/5)
        const double dn = epi ? 1.0 + z : 1.0, dd = epi ? 0.05 + z : 1.0;
        const double r = rcpd(dF * dS * dd) * dn;
        const double rF = sF * dS * r, rS = sS * dF * r;
        // 1/(dti_develop dti_recover)
        const double t = exvad(v, -167.4, 15.89) + exvad(v, -12.23, -0.2154);
        const double w = 33.11545195869231 * E20;   // exp((v + 70)/20)
        const double f = t * (1.0 + w) * rcpd(fma(1.354, t, 1.0e-4) * (0.5 + w));
        c.iF = relaxd(c.iF, iss, rF, ndtl);
        c.iS = relaxd(c.iS, iss, rS, ndtl);
        c.iFp = relaxd(c.iFp, iss, rF * f, ndtl);
        c.iSp = relaxd(c.iSp, iss, rS * f, ndtl);
    }
    const double AiF = sigvad(v, -213.6, 151.2);
    const double ii = fma(AiF, c.iF, (1.0 - AiF) * c.iS);
    const double ip = fma(AiF, c.iFp, (1.0 - AiF) * c.iSp);
    const double Gto = (epi || mid) ? (0.02 * 4.0) : 0.02;
    const double Ito = (Gto * (v - EK) * fma((1.0 - fP) * c.a, ii, fP * c.ap * ip));

    // ICaL, ICaNa, ICaK, TPORd.cc:573-652
    {
        const double dss = rcpd(1.0 + ex2d((v + (3.940 + m.dss_shift)) * (-kLog2e / 4.230)));
        const double s = fma(0.7408182206817179, I20, exvad(v, 14, 1.0 / 0.09));   // exp(-0.05 (v + 6))
        c.d = relaxd(c.d, dss, s * rcpd(fma(0.6, s, 1.0)), ndtl);
    }
    const double fss = rcpd(1.0 + ex2d((v + (19.58 + m.fss_shift)) * (kLog2e / 3.696)));   // = fcass
    const double E7 = ex2d(v * (kLog2e / 7.0)), I7 = ex2d(v * (-kLog2e / 7.0));
    {
        // tff = 7 + 1/sf, tfs = 1000 + 1/ss
        const double sf = fma((0.0045 * 0.1353352832366127), I10, (0.0045 * 7.38905609893065) * E10);
        const double ss = 0.000035 * (exvad(v, 5, -4) + exvad(v, 5, 6));
        const double df = fma(7.0, sf, 1.0), ds = fma(1000.0, ss, 1.0);
        const double r = rcpd(df * ds);
        const double rf = sf * ds * r;
        c.ff = relaxd(c.ff, fss, rf, ndtl);
        c.ffp = relaxd(c.ffp, fss, 0.4 * rf, ndtl);
        c.fs = relaxd(c.fs, fss, ss * df * r, ndtl);
    }
    {
        // tfcaf = 7 + 1/sf, tfcas = 100 + 1/ss
        const double sf = fma((0.04 * 1.770794952435155), I7, (0.04 * 0.5647181220077592) * E7);
        const double ss = 0.00012 * (ex2d(v * (-kLog2e / 3.0)) + E7);
        const double df = fma(7.0, sf, 1.0), ds = fma(100.0, ss, 1.0);
        const double r = rcpd(df * ds);
        const double rf = sf * ds * r;
        c.fcaf = relaxd(c.fcaf, fss, rf, ndtl);
        c.fcafp = relaxd(c.fcafp, fss, 0.4 * rf, ndtl);
        c.fcas = relaxd(c.fcas, fss, ss * df * r, ndtl);
    }
    const double Afcaf = fma(0.6, rcpd(fma(0.36787944117144233, E10, 1.0)), 0.3);   // exp((v - 10)/10)
    const double Afcas = 1.0 - Afcaf;
    c.jca = fma(c.jca - fss, k.e_jca, fss);
    {
        const double q = fma(0.002, rcass, 1.0), q2 = q * q;
        const double nss = rcpd(fma(1.0e-3 * c.jca, q2 * q2, 1.0));   // anca k2n / km2n
        c.nca = relaxd(c.nca, nss, c.jca, ndtl);
    }
    const double fs4 = (0.4 * c.fs), fcs = (Afcas * c.fcas);
    const double f = fma(0.6, c.ff, fs4), fp = fma(0.6, c.ffp, fs4);
    const double fca = fma(Afcaf, c.fcaf, fcs), fcap = fma(Afcaf, c.fcafp, fcs);
    double PhiCaL, PhiCaNa, PhiCaK, INab_phi, ICab_phi;
    {
        // as the reference: e^x - 1 by subtraction, 0/0 at V = 0
        const double x = vfrt, em1 = ex2d(x * kLog2e) - 1.0;
        const double e1 = em1 + 1.0, e1p = e1 + 1.0;
        const double e2m1 = (em1 * e1p), e2 = e2m1 + 1.0;
        // vffrt/(e1 - 1) = F x/(e^x - 1) and vffrt/(e2 - 1)
        const double r = rcpd(e2m1) * x;
        const double g1 = F_ * (r * e1p), g2 = F_ * r;
        PhiCaL = 4.0 * g2 * fma(cass, e2, (-0.341 * cao));
        PhiCaNa = g1 * fma(0.75 * nass, e1, (-0.75 * nao));
        PhiCaK = g1 * fma(0.75 * kss, e1, (-0.75 * ko));
        INab_phi = g1 * fma(nai, e1, -nao);
        ICab_phi = 4.0 * g2 * fma(cai, e2, (-0.341 * cao));
    }
    const double PCa = epi ? m.pca[1] : (mid ? m.pca[2] : m.pca[0]);
    const double jn = c.jca * c.nca;
    const double gate_np = c.d * fma(f, 1.0 - c.nca, fca * jn);
    const double gate_p = c.d * fma(fp, 1.0 - c.nca, fcap * jn);
    // (1 - fP) PCa gate_np + fP (1.1 PCa) gate_p, shared by the three fluxes
    const double G = PCa * fma(1.0 - fP, gate_np, 1.1 * fP * gate_p);
    const double ICaL = (G * PhiCaL);
    const double ICaNa = (0.00125 * G * PhiCaNa);
    const double ICaK = (3.574e-4 * G * PhiCaK);

    // IKr, TPORd.cc:654-678 (sqrt(ko/5.4) = 1)
    const double xrss = sigvad(v, 8.337, -6.789);
    {
        const double sf = fma(0.3652, exvad(v, -31.66, 3.869), 4.123e-5 * exvad(v, -47.78, -20.38));
        const double ss = fma(0.06629, exvad(v, -34.70, 7.355), 1.128e-5 * exvad(v, -29.74, -25.94));
        const double df = fma(12.98, sf, 1.0), ds = fma(1.865, ss, 1.0);
        const double r = rcpd(df * ds);
        c.xrf = relaxd(c.xrf, xrss, sf * ds * r, ndtl);
        c.xrs = relaxd(c.xrs, xrss, ss * df * r, ndtl);
    }
    double IKr;
    {
        const double p = 1.0 + exvad(v, 54.81, 38.21);
        const double q = (1.0 + exvad(v, 55, 75)) * (1.0 + exvad(v, -10, 30));
        const double r = rcpd(p * q);
        const double Axrf = (q * r), rkr = p * r;
        const double xr = fma(Axrf, c.xrf, (1.0 - Axrf) * c.xrs);
        const double GKr = epi ? (0.046 * 1.3) : (mid ? (0.046 * 0.8) : 0.046);
        IKr = (GKr * xr * rkr * (v - EK));
    }

    // IKs, TPORd.cc:680-735
    const double xs1ss = sigvad(v, 11.60, -8.932);
    {
        const double s = fma(2.326e-4, exvad(v, 48.28, 17.80), 0.001292 * exvad(v, 210, -230));
        c.xs1 = relaxd(c.xs1, xs1ss, s * rcpd(fma(817.3, s, 1.0)), ndtl);
        const double rate2 = fma((0.01 * 0.0820849986238988), E20, 0.0193 * exvad(v, 66.54, -31));
        c.xs2 = relaxd(c.xs2, xs1ss, rate2, ndtl);
    }
    // 1 + 0.6/(1 + (3.8e-5/cai)^1.4)
    constexpr double lg_ks = -14.683641055880589;   // log2(3.8e-5)
    const double KsCa = fma(0.6, rcpd(1.0 + ex2d(1.4 * (lg_ks - lg2d(cai)))), 1.0);
    const double GKs = epi ? m.gks[1] : (mid ? m.gks[2] : m.gks[0]);
    const double IKs = (GKs * KsCa * c.xs1 * c.xs2 * (v - EKs));

    // IK1, TPORd.cc:738-751 (sqrt(ko) constant)
    double rk1;
    {
        const double x = 1.0 + exvad(v, 2.5538 * ko + 144.59, -(1.5692 * ko + 3.8115));
        const double y = 1.0 + exvad(v, 105.8 - 2.6 * ko, 9.493);
        const double r = rcpd(x * y);
        rk1 = x * r;
        const double rate = (1.0 / 122.2) * (exvad(v, 127.2, -20.36) + exvad(v, 236.8, 69.33));
        c.xk1 = relaxd(c.xk1, (y * r), rate, ndtl);
    }
    const double GK1 = epi ? (0.1908 * 1.2) : (mid ? (0.1908 * 1.3) : 0.1908);
    const double IK1 = (GK1 * 2.32379000772445 /* sqrt(ko) */ * rk1 * c.xk1 * (v - EK));

    // INaCa_i and INaCa_ss, TPORd.cc:753-852
    constexpr double kna1 = 15.0, kna2 = 5.0, kna3 = 88.12, kasymm = 12.5;
    constexpr double wna = 6.0e4, wca = 6.0e4, wnaca = 5.0e3, kcaon = 1.5e6;
    constexpr double h10 = kasymm + 1.0 + nao / kna1 * (1.0 + nao / kna2);
    constexpr double h11 = nao * nao / (h10 * kna1 * kna2);
    constexpr double k1 = cao * kcaon / h10;
    constexpr double k2 = 5.0e3;   // kcaoff; k5 = k2
    const double ihca = ex2d(v * (-0.1670 * FRT * kLog2e));
    const double hna = ex2d(v * (0.5224 * FRT * kLog2e));
    // h8 = nao/(kna3 hna h7), h9 = 1/h7 with h7 = 1 + nao/kna3 (1 + 1/hna)
    const double r7 = rcpd(fma(hna, (kna3 + nao), nao));
    const double h8 = nao * r7;
    const double k3pp = (h8 * wnaca);
    const double k3 = fma((kna3 * wca) * hna, r7, k3pp);
    const double k8 = (h8 * (h11 * wna));
    const double Gncx = epi ? (0.0008 * 1.1) : (mid ? (0.0008 * 1.4) : 0.0008);
    const double hna1 = (1.0 + hna) * (1.0 / kna3);
    double INaCa_i, INaCa_ss;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
        const double na = pass == 0 ? nai : nass;
        const double ca = pass == 0 ? cai : cass;
        const double h1 = fma(na, hna1, 1.0);
        const double h4 = fma(na * (1.0 / kna1), fma(na, (1.0 / kna2), 1.0), 1.0);
        const double r14 = rcpd(h1 * h4);
        const double h3 = h4 * r14, h6 = h1 * r14;      // 1/h1, 1/h4
        const double h2 = na * hna * (1.0 / kna3) * h3;
        const double h5 = na * na * (1.0 / (kna1 * kna2)) * h6;
        const double k4pp = (h2 * wnaca);
        const double k4 = fma(h3 * wca, ihca, k4pp);
        const double k6 = (h6 * ca * kcaon);
        const double k7 = (h5 * h2 * wna);
        const double k67 = k6 + k7, k23 = k2 + k3, k45 = k4 + k2, k18 = k1 + k8;
        const double x1 = (k2 * fma(k4, k67, k7 * k23));
        const double x2 = fma(k1 * k7, k45, k4 * k6 * k18);
        const double x3 = fma(k1 * k3, k67, k8 * k6 * k23);
        const double x4 = (k2 * fma(k8, k45, k3 * k18));
        const double xs = (x1 + x2) + (x3 + x4);
        // J = (3 (x4 k7 - x1 k8) + x3 k4pp - x2 k3pp + 2 (x2 k2 - x1 k1)) / xs; allo = ca^2/(ca^2 + KmCaAct^2)
        const double a = fma(x4, k7, -(x1 * k8)), b = fma(x2, k2, -(x1 * k1));
        const double num = fma(2.0, b, fma(3.0, a, fma(x3, k4pp, -(x2 * k3pp))));
        const double ca2 = (ca * ca);
        const double val = Gncx * num * ca2 * rcpd(xs * (ca2 + (150.0e-6 * 150.0e-6)));
        if (pass == 0) INaCa_i = (0.8 * val);
        else INaCa_ss = (0.2 * val);
    }
    const double INaCa = INaCa_i + INaCa_ss;

    // INaK, TPORd.cc:854-906
    double INaK;
    {
        constexpr double k1p = 949.5, k1m = 182.4, k2p = 687.2, k2m = 39.4;
        constexpr double k3p_ = 1899.0, k3m = 79300.0, k4p_ = 639.0, k4m = 40.0;
        constexpr double Knai0 = 9.073, Knao0 = 27.78, delta = -0.1550;
        constexpr double Kki = 0.5, Kko = 0.3582, MgADP = 0.05, MgATP = 9.8, Kmgatp = 1.698e-7;
        constexpr double H = 1.0e-7, eP = 4.2, Khp = 1.698e-7, Knap = 224.0, Kxkur = 292.0;
        constexpr double rko = ko / Kko;
        const double rnai = (nai * (1.0 / Knai0) * ex2d(v * (-delta / 3.0 * FRT * kLog2e)));
        const double rnao = ((nao / Knao0) * ex2d(v * (-(1.0 - delta) / 3.0 * FRT * kLog2e)));
        const double rki = (ki * (1.0 / Kki));
        const double pP = fma(ki, (1.0 / Kxkur), fma(nai, (1.0 / Knap), (1.0 + H / Khp)));   // eP/P
        const double pnai = 1.0 + rnai, pnao = 1.0 + rnao, pki = 1.0 + rki;
        const double den_i = fma(pnai * pnai, pnai, fma(pki, pki, -1.0));
        const double den_o = fma(pnao * pnao, pnao, ((1.0 + rko) * (1.0 + rko) - 1.0));
        const double rio = rcpd(den_i * den_o);
        const double ri = den_o * rio, ro = den_i * rio;
        const double a1 = (k1p * (rnai * rnai * rnai) * ri);
        const double b4 = (k4m * (rki * rki) * ri);
        const double b2 = (k2m * (rnao * rnao * rnao) * ro);
        const double a3 = ((k3p_ * rko * rko) * ro);
        const double b3 = ((k3m * H / (1.0 + MgATP / Kmgatp) * eP) * rcpd(pP));
        constexpr double b1 = (k1m * MgADP), a2 = k2p;
        constexpr double a4 = ((k4p_ * MgATP / Kmgatp) / (1.0 + MgATP / Kmgatp));
        const double b43 = (b4 * b3), b23 = (b2 * b3);
        const double y1 = fma(a2, fma(a1, a4 + b3, b43), b2 * b43);
        const double y2 = fma(b1 * b4, b2 + a3, a2 * a3 * (a1 + b4));
        const double y3 = fma(a3 * a4, a2 + b1, b1 * b2 * (b3 + a4));
        const double y4 = fma(b23, b4 + a1, a4 * a1 * (a3 + b2));
        const double J = fma(3.0, fma(y1, a3, -(y2 * b3)), 2.0 * fma(y4, b1, -(y3 * a1)));
        const double Pnak = epi ? (30 * 0.9) : (mid ? (30 * 0.7) : 30.0);
        INaK = (Pnak * J * rcpd((y1 + y2) + (y3 + y4)));
    }

    // background currents and pump, TPORd.cc:908-923
    const double GKb = epi ? (0.003 * 0.6) : 0.003;
    const double IKb = (GKb * sigvad(v, -14.48, -18.34) * (v - EK));
    const double INab = (3.75e-10 * INab_phi);
    const double ICab = (2.5e-8 * ICab_phi);
    // cytosolic buffer and pump: Bcai = 1/(1 + cm/qc^2 + ct/qt^2), IpCa = 0.0005 cai/qt (qt = 0.0005 + cai)
    constexpr double cmdnmax = 0.05, kmcmdn = 0.00238, trpnmax = 0.07, kmtrpn = 0.0005;
    double IpCa, Bcai;
    {
        const double qc = kmcmdn + cai, qt = kmtrpn + cai;
        const double qc2 = (qc * qc), qt2 = (qt * qt), qq = (qc2 * qt2);
        const double cm = epi ? (1.3 * cmdnmax * kmcmdn) : (cmdnmax * kmcmdn);
        const double D = fma((trpnmax * kmtrpn), qc2, fma(cm, qt2, qq));
        const double r = rcpd(D * qt);
        Bcai = qq * (r * qt);
        IpCa = (0.0005 * cai * r * D);
    }

    // membrane potential, TPORd.cc:927-935
    const double Iion = INa + INaL + Ito + ICaL + ICaNa + ICaK + IKr + IKs + IK1 + INaCa + INaK + INab + IKb + IpCa + ICab;
    const double dV_dt = -(Iion + Ist);
    c.v = fma(dV_dt + dVgap_dt, dt, v);
    if (out) {
        out->dvdt = dV_dt;
        out->ical = ICaL;
        out->iks = IKs;
        out->ina = INa;
        out->ikr = IKr;
        out->ik1 = IK1;
    }

    // CaMK and fluxes, TPORd.cc:939-995
    c.CaMKt = fma(dt, fma(0.05 * CaMKb, CaMKa, -(0.00068 * c.CaMKt)), c.CaMKt);
    // concentration differences from the full-precision values (file comment of tpord.cuh)
    const double JdiffNa = (cdiff(c.nass, c.nai) * 0.5);
    const double JdiffK = (cdiff(c.kss, c.ki) * 0.5);
    const double Jdiff = (cdiff(c.cass, c.cai) * 5.0);
    const double Jtr = (cdiff(c.cansr, c.cajsr) * 0.01);
    {
        // 1/(1 + (1.5/cajsr)^8) and 1/cajsr from one reciprocal
        const double j2 = cajsr * cajsr, j4 = j2 * j2, j8 = (j4 * j4);
        const double dj = j8 + 25.62890625;
        const double r = rcpd(fma(dj, cajsr, kTinyD));
        const double rel = (mid ? 1.7 : 1.0) * -ICaL * j8 * (r * cajsr);
        // 1/tau_rel; tau_rel below 0.005, negative ones too (cajsr < 0), is 0.005: the
        // sign bit makes a negative rate's high word the larger unsigned number
        const double rate = fma(0.0123 / 4.75, r * dj, 1.0 / 4.75);
        auto bound = [](double x) { return (unsigned)__double2hiint(x) < 0x40690000u ? x : 200.0; };
        const double Jrel_inf = ((0.5 * 4.75) * rel), Jrel_infp = ((0.5 * 1.25 * 4.75) * rel);
        c.Jrelnp = relaxd(c.Jrelnp, Jrel_inf, bound(rate), ndtl);
        c.Jrelp = relaxd(c.Jrelp, Jrel_infp, bound(0.8 * rate), ndtl);
    }
    const double Jrel = fma(1.0 - fP, c.Jrelnp, fP * c.Jrelp);
    double Jup;
    {
        const double p = cai + 0.00092, q = cai + (0.00092 - 0.00017);
        const double s = (epi ? 1.3 : 1.0) * cai * rcpd(p * q);
        const double u = fma((1.0 - fP) * 0.004375, q, fP * (2.75 * 0.004375) * p);
        Jup = fma(s, u, -((0.0039375 / 15.0) * cansr));
    }

    // concentrations, forward Euler, TPORd.cc:997-1020
    constexpr double cm = (Acap / (F_ * vmyo)), cs = (Acap / (F_ * vss));
    const double dnai = fma(-fma(3.0, INaCa_i + INaK, INa + INaL + INab), cm, JdiffNa * (vss / vmyo));
    const double dnass = fma(-fma(3.0, INaCa_ss, ICaNa), cs, -JdiffNa);
    const double dki = fma(-fma(-2.0, INaK, Ito + IKr + IKs + IK1 + IKb + Ist), cm, JdiffK * (vss / vmyo));
    const double dkss = fma(-ICaK, cs, -JdiffK);
    const double dcai = Bcai * fma(-fma(-2.0, INaCa_i, IpCa + ICab), 0.5 * cm,
                                   fma(-Jup, (vnsr / vmyo), Jdiff * (vss / vmyo)));
    // Bcass and Bcajsr from one reciprocal
    constexpr double BSRmax = 0.047, KmBSR = 0.00087, BSLmax = 1.124, KmBSL = 0.0087;
    constexpr double csqnmax = 10.0, kmcsqn = 0.8;
    const double qsr = KmBSR + cass, qsl = KmBSL + cass, qj = kmcsqn + cajsr;
    const double qsr2 = (qsr * qsr), qsl2 = (qsl * qsl), qs = (qsr2 * qsl2), qj2 = (qj * qj);
    const double Ds = fma((BSLmax * KmBSL), qsr2, fma((BSRmax * KmBSR), qsl2, qs));
    const double Dj = qj2 + (csqnmax * kmcsqn);
    const double rsj = rcpd(Ds * Dj);
    const double Bcass = qs * (Dj * rsj), Bcajsr = qj2 * (Ds * rsj);
    const double dcass = Bcass * fma(-fma(-2.0, INaCa_ss, ICaL), 0.5 * cs, fma(Jrel, (vjsr / vss), -Jdiff));
    const double dcansr = fma(-Jtr, (vjsr / vnsr), Jup);
    const double dcajsr = Bcajsr * (Jtr - Jrel);
    cadd(c.nai, dt * dnai);
    cadd(c.nass, dt * dnass);
    cadd(c.ki, dt * dki);
    cadd(c.kss, dt * dkss);
    cadd(c.cai, dt * dcai);
    cadd(c.cass, dt * dcass);
    cadd(c.cansr, dt * dcansr);
    cadd(c.cajsr, dt * dcajsr);
}

// The step of every kernel in the FP64 form, and the batch kernel's in the mixed form.
__device__ __forceinline__ void tpord_update(CellState<double> &c, int ctype, const ModelT<double> &m,
                                             const StepT<double> &k, double Ist, double dVgap_dt, StepOut<double> *out)
{
    tpord_step_f64(c, ctype, m, k, Ist, dVgap_dt, out);
}
__device__ __forceinline__ void tpord_batch_update(CellState<double> &c, int ctype, const ModelT<double> &m,
                                                   const StepT<double> &k, double Ist, double dVgap_dt,
                                                   StepOut<double> *out)
{
    tpord_step_f64(c, ctype, m, k, Ist, dVgap_dt, out);
}
__device__ __forceinline__ void tpord_batch_update(CellState<float> &c, int ctype, const ModelT<float> &m,
                                                   const StepT<float> &k, float Ist, float dVgap_dt, StepOut<float> *out)
{
    tpord_step_terms(c, ctype, m, k, Ist, dVgap_dt, out);
}

}  // namespace lqt
