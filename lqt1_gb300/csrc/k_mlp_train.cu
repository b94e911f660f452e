// k_mlp_train.cu -- one training step of the learned surrogate's network
// (48 -> 128 -> 128 -> 48, SiLU, BF16 operands, FP32 accumulation) in two
// kernels.
//
// k_mlp_grad: forward, loss gradient, backward and weight gradients of up to
// 128 batch rows per CTA without leaving the SM.  The weights (56 KB), the row
// tile's inputs, both hidden tiles and the three gradient tiles live in shared
// memory (208 KB), the accumulators in TMEM (480 of 512 columns).  Every tile
// is stored once, as 8 x 8 core matrices of 8 rows x 16 bytes: read K-major it
// is the operand of a forward or data-gradient GEMM, read MN-major (the
// descriptor's strides exchanged, the transpose bits of the instruction set)
// the same bytes are the transposed operand of a weight gradient, and W2 and
// W3 those of a data gradient.  Each CTA writes one slice of the weight gradients
// (to which its later tiles, in batches above 16384 rows, are added) and its
// rows' output and pre-activation gradients.
// k_mlp_update: adds the slices in a fixed order (the same bits on every run),
// the bias gradients by rows, and applies Adam to the FP32 master weights and
// their BF16 copy.
//
// Sixteen steps amplify the last bit of a sum through the weights' BF16
// rounding, so the sums have one order that does not depend on how the work is
// laid out: a weight's by at most 128 slices of whole half tiles, a bias's by
// row mod 256 and a tree.
//
// What bounds it: one tile's serial chain of five GEMMs and their epilogues
// (a batch of 8192 is 128 half tiles on 152 SMs); tensor time and traffic are
// below 3 us.  As 17 launches that passed every tile through L2 a batch took
// 253 us with its input preparation (16 batches of 8192); this form takes 43.
#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mlp.h"
#include "tc.cuh"

namespace lqt {

namespace {

constexpr int kTM = 128;                   // batch rows per tile (TMEM lanes)
constexpr int kThreads = 512;              // four warps per 32 rows: 32 columns each
constexpr uint32_t kWaitLimit = 1u << 24;  // bounded mbarrier polls

// shared-memory plan (bytes): core-matrix tiles
constexpr uint32_t kT128 = kTM * kMlpHid * 2, kT48 = kTM * kMlpIn * 2;
constexpr uint32_t kOffW1 = 0;                                  // [128][48]
constexpr uint32_t kOffW2 = kOffW1 + kMlpHid * kMlpIn * 2;      // [128][128]
constexpr uint32_t kOffW3 = kOffW2 + kMlpHid * kMlpHid * 2;     // [48][128]
constexpr uint32_t kOffX = kOffW3 + kMlpOut * kMlpHid * 2;      // [128][48] inputs
constexpr uint32_t kOffH1 = kOffX + kT48;                       // [128][128] hidden
constexpr uint32_t kOffH2 = kOffH1 + kT128;
constexpr uint32_t kOffDY = kOffH2 + kT128;                     // [128][48] output gradient
constexpr uint32_t kOffDZ2 = kOffDY + kT48;                     // [128][128] pre-activation gradients
constexpr uint32_t kOffDZ1 = kOffDZ2 + kT128;
constexpr uint32_t kOffBias = kOffDZ1 + kT128;                  // b1[128], b2[128], b3[48]
constexpr uint32_t kNBias = 2 * kMlpHid + kMlpOut;
constexpr uint32_t kOffBar = kOffBias + kNBias * 4;
constexpr uint32_t kSmemBytes = kOffBar + 32;
static_assert(kMlpIn == kMlpOut, "one 48-column tile type");
static_assert(kOffBias % 16 == 0 && kOffBar % 8 == 0 && kSmemBytes <= 227 * 1024, "shared memory");

// TMEM columns: the pre-activations; the outputs, then the two data gradients
// (work); the weight gradients (W2's over pre-activation 2, whose last use is
// the gradient that W2's is formed from)
constexpr uint32_t kColZ1 = 0, kColZ2 = 128, kColWork = 256, kColG2 = kColZ2, kColG3 = 384, kColG1 = 432, kTmemCols = 512;

// Slice layout (floats): the parameter block's order W1 b1 W2 b2 W3 b3
constexpr int kOW1 = 0, kOB1 = kOW1 + kMlpHid * kMlpIn, kOW2 = kOB1 + kMlpHid, kOB2 = kOW2 + kMlpHid * kMlpHid,
              kOW3 = kOB2 + kMlpHid, kOB3 = kOW3 + kMlpOut * kMlpHid, kNP = kOB3 + kMlpOut;
static_assert(kNP == kMlpNParam32, "parameter block");

// 1 / (1 + exp(-z)): the hardware reciprocal with one Newton step on its exact
// residual (an FMA), which is the correctly rounded quotient but for about one
// argument in a million.  exp(-z) is held at the largest finite value, whose
// reciprocal is flushed to 0 (as from z = -87 on), so that z * sigm(z) is 0 for
// any z below.
__device__ __forceinline__ float sigm(float z)
{
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z * -1.4426950408889634f));
    const float d = 1.0f + fminf(e, 3.402823466e38f);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fmaf(fmaf(-d, r, 1.0f), r, r);
}

// Copy `rows` valid rows of a row-major [R][K] BF16 matrix into core matrices, zeros below them.
__device__ __forceinline__ void stage_tile(uint8_t *dst, const __nv_bfloat16 *src, int R, int K, int rows)
{
    for (int c = threadIdx.x; c < R * (K / 8); c += kThreads) {
        const int r = c / (K / 8), kg = c % (K / 8);
        *reinterpret_cast<uint4 *>(dst + tc::kmaj_off(r, kg * 8, K)) =
            r < rows ? *reinterpret_cast<const uint4 *>(src + (int64_t)r * K + kg * 8) : make_uint4(0, 0, 0, 0);
    }
}

// An operand tile of F features: read K-major (rows = M or N, features = K)
// or MN-major (features = M or N, rows = K).  Per MMA K advances by 16.
struct Operand {
    uint32_t addr, lbo, sbo, step;
};
__device__ __forceinline__ Operand kmajor(const uint8_t *p, int F)
{
    return Operand{tc::smem_u32(p), 128u, (uint32_t)(F / 8) * 128u, 256u};
}
__device__ __forceinline__ Operand mnmajor(const uint8_t *p, int F)
{
    const uint32_t row8 = (uint32_t)(F / 8) * 128u;     // next 8 rows
    return Operand{tc::smem_u32(p), row8, 128u, 2u * row8};
}
// D[128 x N] (+)= A B^T over K; at, bt = operand MN-major.
__device__ __forceinline__ void mma_all(uint32_t d, const Operand &a, bool at, const Operand &b, bool bt, int N, int K,
                                        bool accum)
{
    const uint32_t id = tc::idesc_bf16_f32(128, N) | (at ? 1u << 15 : 0u) | (bt ? 1u << 16 : 0u);
    for (int k = 0; k < K / 16; ++k)
        tc::mma_bf16(d, tc::smem_desc(a.addr + k * a.step, a.lbo, a.sbo), tc::smem_desc(b.addr + k * b.step, b.lbo, b.sbo),
                     id, (accum || k > 0) ? 1u : 0u);
}

__device__ __forceinline__ uint32_t pack2(float a, float b)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

}  // namespace

// CTA b takes rows [b chunk, (b + 1) chunk) of the batch.  part: its slice of
// the weight gradients; lossp: its sum of squared errors over the valid
// outputs; grow: per row the output and pre-activation gradients (dY, dZ2,
// dZ1), whose column sums are the bias gradients.  dY = 2 (Y - T) / (B nvalid).
__global__ void __launch_bounds__(kThreads, 1) k_mlp_grad(const __nv_bfloat16 *__restrict__ X,
                                                          const float *__restrict__ T, int64_t B, int nvalid,
                                                          MlpDev w, float *__restrict__ part,
                                                          double *__restrict__ lossp,
                                                          __nv_bfloat16 *__restrict__ grow, int chunk, int *err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ double lred[kThreads / 32];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + kOffBar);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + kOffBar + 8);
    float *bias = reinterpret_cast<float *>(smem + kOffBias);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quarter = warp >> 2;                     // columns [32 quarter, + 32) of the hidden tiles
    const int row = (warp & 3) * 32 + lane;            // row of the tile = TMEM lane
    const int c0 = quarter * 32, o0 = quarter * 16;    // and [16 quarter, + 16) of the outputs, for three of them

    stage_tile(smem + kOffW1, w.w1t, kMlpHid, kMlpIn, kMlpHid);
    stage_tile(smem + kOffW2, w.w2t, kMlpHid, kMlpHid, kMlpHid);
    stage_tile(smem + kOffW3, w.w3t, kMlpOut, kMlpHid, kMlpOut);
    for (int i = tid; i < (int)kNBias; i += kThreads)
        bias[i] = i < kMlpHid ? w.b1[i] : (i < 2 * kMlpHid ? w.b2[i - kMlpHid] : w.b3[i - 2 * kMlpHid]);
    if (tid == 0) {
        tc::mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tc::tmem_alloc(tslot, kTmemCols);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tm = *tslot;
    const uint32_t tl = tm + ((uint32_t)((warp & 3) * 32) << 16);   // this warp's TMEM lanes
    const float scale = 2.0f / (float)(B * nvalid);
    const bool wide = (reinterpret_cast<uintptr_t>(T) & 15) == 0;   // target rows readable 16 bytes at a time
    uint32_t phase = 0;
    bool ok = true, first = true;
    float lhi = 0.f, llo = 0.f;                        // this thread's squared errors, a compensated pair
    float *const out = part + (int64_t)blockIdx.x * kNP;

    // writes before it are visible to the MMAs, TMEM reads before it are done
    auto publish = [&]() {
        tc::fence_proxy_async();
        tc::fence_before();
        __syncthreads();
    };
    // the MMAs committed so far are complete; the CTA takes one decision
    auto arrived = [&]() -> bool {
        const bool w_ok = tc::mbar_wait(bar, phase, kWaitLimit);
        if (!__syncthreads_and(w_ok ? 1 : 0)) {
            if (!w_ok) tc::mbar_wait(bar, phase, kWaitLimit);       // let the MMAs in flight land before TMEM is freed
            if (tid == 0 && err) atomicExch(err, 2);
            return false;
        }
        phase ^= 1;
        tc::fence_after();
        return true;
    };
    // pre-activation (TMEM + bias) of this thread's 32 columns
    auto load_z = [&](uint32_t col, const float *b, float *z) {
        tc::tmem_ld32(tl + col + c0, z);
#pragma unroll
        for (int i = 0; i < 32; ++i) z[i] += b[c0 + i];
    };
    // hidden layer: SiLU to the operand tile
    auto hidden = [&](uint32_t col, const float *b, uint8_t *dst) {
        float z[32];
        load_z(col, b, z);
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
            uint32_t p[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float x = z[i + 2 * j], y = z[i + 2 * j + 1];
                p[j] = pack2(x * sigm(x), y * sigm(y));
            }
            *reinterpret_cast<uint4 *>(dst + tc::kmaj_off(row, c0 + i, kMlpHid)) = make_uint4(p[0], p[1], p[2], p[3]);
        }
    };
    // pre-activation gradient: the work columns times SiLU'(z)
    auto dact = [&](uint32_t col, const float *b, uint8_t *dst, __nv_bfloat16 *keep) {
        float z[32], v[32];
        load_z(col, b, z);
        tc::tmem_ld32(tl + kColWork + c0, v);
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
            uint32_t p[4];
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                float d[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float zz = z[i + j + u], sz = sigm(zz);
                    d[u] = v[i + j + u] * (sz + zz * sz * (1.0f - sz));
                }
                p[j / 2] = pack2(d[0], d[1]);
            }
            const uint4 q = make_uint4(p[0], p[1], p[2], p[3]);
            *reinterpret_cast<uint4 *>(dst + tc::kmaj_off(row, c0 + i, kMlpHid)) = q;
            if (keep) *reinterpret_cast<uint4 *>(keep + c0 + i) = q;
        }
    };
    // a slice element: the first tile's value, later tiles added to it
    auto put = [&](int i, float x) { out[i] = first ? x : out[i] + x; };

    const int64_t mend = (int64_t)(blockIdx.x + 1) * chunk < B ? (int64_t)(blockIdx.x + 1) * chunk : B;
    for (int64_t m0 = (int64_t)blockIdx.x * chunk; m0 < mend && ok; m0 += kTM) {
        const int rows = (int)(mend - m0 < kTM ? mend - m0 : kTM);
        const bool live = row < rows;
        __nv_bfloat16 *keep = live ? grow + (m0 + row) * kNBias : nullptr;
        stage_tile(smem + kOffX, X + m0 * kMlpIn, kTM, kMlpIn, rows);
        // this thread's targets
        float tg[16];
        const float *trow = T + (m0 + row) * kMlpOut + o0;
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live && quarter < 3)
                q = wide ? __ldg(reinterpret_cast<const float4 *>(trow + j)) : make_float4(trow[j], trow[j + 1], trow[j + 2], trow[j + 3]);
            tg[j] = q.x;
            tg[j + 1] = q.y;
            tg[j + 2] = q.z;
            tg[j + 3] = q.w;
        }
        publish();
        if (tid == 0) {
            tc::fence_after();
            mma_all(tm + kColZ1, kmajor(smem + kOffX, kMlpIn), false, kmajor(smem + kOffW1, kMlpIn), false, kMlpHid, kMlpIn, false);
            tc::mma_commit(bar);
        }
        if (!(ok = arrived())) break;
        hidden(kColZ1, bias, smem + kOffH1);
        publish();
        if (tid == 0) {
            tc::fence_after();
            mma_all(tm + kColZ2, kmajor(smem + kOffH1, kMlpHid), false, kmajor(smem + kOffW2, kMlpHid), false, kMlpHid, kMlpHid, false);
            tc::mma_commit(bar);
        }
        if (!(ok = arrived())) break;
        hidden(kColZ2, bias + kMlpHid, smem + kOffH2);
        publish();
        if (tid == 0) {
            tc::fence_after();
            mma_all(tm + kColWork, kmajor(smem + kOffH2, kMlpHid), false, kmajor(smem + kOffW3, kMlpHid), false, kMlpOut, kMlpHid, false);
            tc::mma_commit(bar);
        }
        if (!(ok = arrived())) break;
        // outputs: loss and its gradient
        if (quarter < 3) {
            float y[16];
            tc::tmem_ld16(tl + kColWork + o0, y);
#pragma unroll
            for (int i = 0; i < 16; i += 8) {
                uint32_t p[4];
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    float g[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int c = o0 + i + j + u;
                        float d = (y[i + j + u] + bias[2 * kMlpHid + c]) - tg[i + j + u];
                        if (c >= nvalid || !live) d = 0.f;
                        g[u] = scale * d;
                        // (lhi, llo) += d^2: the square's rounding error by an FMA, the sum's by TwoSum
                        const float sq = __fmul_rn(d, d), se = fmaf(d, d, -sq);
                        const float s = __fadd_rn(lhi, sq), bb = __fsub_rn(s, lhi);
                        llo += __fadd_rn(__fsub_rn(lhi, __fsub_rn(s, bb)), __fsub_rn(sq, bb)) + se;
                        lhi = s;
                    }
                    p[j / 2] = pack2(g[0], g[1]);
                }
                const uint4 q = make_uint4(p[0], p[1], p[2], p[3]);
                *reinterpret_cast<uint4 *>(smem + kOffDY + tc::kmaj_off(row, o0 + i, kMlpOut)) = q;
                if (keep) *reinterpret_cast<uint4 *>(keep + o0 + i) = q;
            }
        }
        publish();
        if (tid == 0) {
            tc::fence_after();
            mma_all(tm + kColWork, kmajor(smem + kOffDY, kMlpOut), false, mnmajor(smem + kOffW3, kMlpHid), true, kMlpHid, kMlpOut, false);
            tc::mma_commit(bar);
            // W3 gradient, transposed: [hidden][output]
            mma_all(tm + kColG3, mnmajor(smem + kOffH2, kMlpHid), true, mnmajor(smem + kOffDY, kMlpOut), true, kMlpOut, kTM, false);
        }
        if (!(ok = arrived())) break;
        dact(kColZ2, bias + kMlpHid, smem + kOffDZ2, keep ? keep + kMlpOut : nullptr);
        publish();
        if (tid == 0) {
            tc::fence_after();
            mma_all(tm + kColWork, kmajor(smem + kOffDZ2, kMlpHid), false, mnmajor(smem + kOffW2, kMlpHid), true, kMlpHid, kMlpHid, false);
            tc::mma_commit(bar);
            // W2 gradient, transposed: [in][out]
            mma_all(tm + kColG2, mnmajor(smem + kOffH1, kMlpHid), true, mnmajor(smem + kOffDZ2, kMlpHid), true, kMlpHid, kTM, false);
        }
        if (!(ok = arrived())) break;
        dact(kColZ1, bias, smem + kOffDZ1, keep ? keep + kMlpOut + kMlpHid : nullptr);
        publish();
        if (tid == 0) {
            tc::fence_after();
            // W1 gradient: [out][in]
            mma_all(tm + kColG1, mnmajor(smem + kOffDZ1, kMlpHid), true, mnmajor(smem + kOffX, kMlpIn), true, kMlpIn, kTM, false);
            tc::mma_commit(bar);
        }
        if (!(ok = arrived())) break;               // and with it every earlier MMA: the tiles may be overwritten
        // the slice; [in][out] accumulators: a warp writes 32 neighbouring inputs of one output
        {
            float v[32];
            tc::tmem_ld32(tl + kColG2 + c0, v);
#pragma unroll
            for (int i = 0; i < 32; ++i) put(kOW2 + (c0 + i) * kMlpHid + row, v[i]);
            if (quarter < 3) {
                tc::tmem_ld16(tl + kColG3 + o0, v);
                tc::tmem_ld16(tl + kColG1 + o0, v + 16);
#pragma unroll
                for (int i = 0; i < 16; ++i) put(kOW3 + (o0 + i) * kMlpHid + row, v[i]);
#pragma unroll
                for (int i = 0; i < 16; ++i) put(kOW1 + row * kMlpIn + o0 + i, v[16 + i]);
            }
        }
        tc::fence_before();
        __syncthreads();                             // before the next tile's inputs and MMAs
        first = false;
    }
    if (ok) {
        double l = (double)lhi + (double)llo;
        for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
        if (lane == 0) lred[warp] = l;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int q = 0; q < kThreads / 32; ++q) s += lred[q];
            lossp[blockIdx.x] = s;
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tm, kTmemCols);
}

constexpr int kUpThreads = 256;
constexpr int kUpWeights = (kNP + kUpThreads - 1) / kUpThreads, kUpColumns = kNBias / 8;
static_assert(kNBias % 8 == 0, "columns in groups of 8");

struct AdamArgs {
    float *g, *p, *m, *v;
    __nv_bfloat16 *pb;
    float lr, b1, b2, eps, c1, c2;
};

// G = the slices of a weight added in slice order, or the row gradients of a
// bias added by rows (row mod 256, then a tree: independent of the slices);
// with lr > 0 one Adam step with bias correction c1, c2 on the FP32 master
// parameters and their BF16 copy.  loss = sum of lossp.  Bound by latency: a
// thread's loads are all under way before it adds the first.
__global__ void __launch_bounds__(kUpThreads) k_mlp_update(const float *__restrict__ part,
                                                           const double *__restrict__ lossp, int slices,
                                                           const __nv_bfloat16 *__restrict__ grow, int64_t B,
                                                           double *__restrict__ loss, AdamArgs a)
{
    __shared__ float red[8][kUpThreads];
    __shared__ double sl[kUpThreads];
    const int t = threadIdx.x;
    auto finish = [&](int i, float gi, float p0, float m0, float v0) {
        a.g[i] = gi;
        if (a.lr > 0.f) {
            const float mi = fmaf(1.f - a.b1, gi, __fmul_rn(a.b1, m0));
            const float vi = fmaf(__fmul_rn(1.f - a.b2, gi), gi, __fmul_rn(a.b2, v0));
            a.m[i] = mi;
            a.v[i] = vi;
            const float pn = p0 - __fmul_rn(a.lr, mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
            a.p[i] = pn;
            a.pb[i] = __float2bfloat16(pn);
        }
    };
    if ((int)blockIdx.x < kUpWeights) {
        constexpr int kAhead = 64;
        const int i = blockIdx.x * kUpThreads + t;
        const bool bias = (i >= kOB1 && i < kOW2) || (i >= kOB2 && i < kOW3) || i >= kOB3;
        if (bias) return;
        const float p0 = a.p[i], m0 = a.m[i], v0 = a.v[i];
        float gi = 0.f;
        for (int s = 0; s < slices; s += kAhead) {
            float x[kAhead];
#pragma unroll
            for (int j = 0; j < kAhead; ++j)
                if (s + j < slices) x[j] = part[(int64_t)(s + j) * kNP + i];
#pragma unroll
            for (int j = 0; j < kAhead; ++j)
                if (s + j < slices) gi += x[j];
        }
        finish(i, gi, p0, m0, v0);
    } else if ((int)blockIdx.x < kUpWeights + kUpColumns) {
        const int c0 = ((int)blockIdx.x - kUpWeights) * 8;
        float acc[8] = {};
        constexpr int kAhead = 16;
        for (int64_t r = t; r < B; r += kAhead * kUpThreads) {
            uint4 q[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                q[u] = r + u * kUpThreads < B ? *reinterpret_cast<const uint4 *>(grow + (r + u * kUpThreads) * kNBias + c0)
                                              : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&q[u]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 f = __bfloat1622float2(h[j]);
                    acc[2 * j] += f.x;
                    acc[2 * j + 1] += f.y;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) red[j][t] = acc[j];
        __syncthreads();
        for (int w = kUpThreads / 2; w > 0; w >>= 1) {
            if (t < w) {
#pragma unroll
                for (int j = 0; j < 8; ++j) red[j][t] += red[j][t + w];
            }
            __syncthreads();
        }
        if (t < 8) {
            const int c = c0 + t;
            const int i = c < kMlpOut ? kOB3 + c : (c < kMlpOut + kMlpHid ? kOB2 + c - kMlpOut : kOB1 + c - kMlpOut - kMlpHid);
            finish(i, red[t][0], a.p[i], a.m[i], a.v[i]);
        }
    } else {
        double s = 0.0;
        for (int k = 0; k < slices; k += kUpThreads) {
            if (k + t < slices) sl[t] = lossp[k + t];
            __syncthreads();
            if (t == 0)
                for (int j = 0; j < kUpThreads && k + j < slices; ++j) s += sl[j];
            __syncthreads();
        }
        if (t == 0) *loss = s;
    }
}

// Rows per slice, a multiple of half a tile: at most 128 slices, each a CTA of
// its own; up to 16384 rows a slice is one tile (half of one up to 8192: then
// twice as many SMs work, each for the time of a tile).
int mlp_grad_chunk(int64_t B)
{
    const int64_t want = std::min<int64_t>(128, std::max<int64_t>(1, B / 64));
    return (int)(((B + want - 1) / want + 63) / 64 * 64);
}
int mlp_grad_slices(int64_t B)
{
    const int64_t chunk = mlp_grad_chunk(B);
    return (int)((B + chunk - 1) / chunk);
}

cudaError_t launch_mlp_grad(const __nv_bfloat16 *X, const float *T, int64_t B, int nvalid, const MlpDev &w, float *part,
                            double *lossp, __nv_bfloat16 *grow, int *err, cudaStream_t st)
{
    if (B <= 0) return cudaSuccess;
    static std::atomic<uint64_t> attr_done{0};
    cudaError_t e = tc::smem_attr_once(k_mlp_grad, kSmemBytes, attr_done);
    if (e != cudaSuccess) return e;
    k_mlp_grad<<<(unsigned)mlp_grad_slices(B), kThreads, kSmemBytes, st>>>(X, T, B, nvalid, w, part, lossp, grow,
                                                                           mlp_grad_chunk(B), err);
    return cudaGetLastError();
}

cudaError_t launch_mlp_update(const float *part, const double *lossp, int slices, const __nv_bfloat16 *grow, int64_t B,
                              float *g, double *loss, float *p, float *m, float *v, __nv_bfloat16 *pb, float lr, float b1,
                              float b2, float eps, float c1, float c2, cudaStream_t st)
{
    const AdamArgs a{g, p, m, v, pb, lr, b1, b2, eps, c1, c2};
    k_mlp_update<<<kUpWeights + kUpColumns + 1, kUpThreads, 0, st>>>(part, lossp, slices, grow, B, loss, a);
    return cudaGetLastError();
}

}  // namespace lqt
