// k_mlp_tc.cu -- BF16 MLP inference on the 5th-generation tensor cores.
//
// Network of the learned surrogate: 48 -> 128 -> 128 -> 48, SiLU between
// layers, BF16 weights and activations, FP32 accumulation.  One persistent CTA
// per SM of four warpgroups; the three weight matrices (56 KB) are staged once
// per CTA.  Each warpgroup walks its own tiles of 128 rows with its own operand
// buffer (the input tile, then the hidden tile, then the output rows, in the
// same 32 KB) and 128 TMEM columns: per layer one elected thread issues
// tcgen05.mma (M = 128, K = 16 per instruction) into the accumulator and
// commits to the group's mbarrier; the four warps read their 32 TMEM lanes
// back with tcgen05.ld, add the bias, apply SiLU and write the next layer's
// BF16 operand into shared memory.
//
// What bounds it: the 256 SiLUs per row.  Each needs an exponential and a
// division; as ex2 + one reciprocal for two of them (1.5 MUFU, about 8 issue
// slots in all, the FP32 arithmetic two
// values per instruction) a row costs the MUFU pipe about 80 us per million rows, against
// 42 us of memory traffic and 30 us of tensor time, so four groups per SM keep
// that pipe fed while the others' MMAs, loads and stores run.  The quotient is
// corrected by its exact remainder, so the BF16 activations are those of the
// IEEE division (which rows with a pre-activation beyond +-43 take).  Rows leave
// through a padded slab per warp: 16-byte shared-memory stores without bank
// conflicts, then 512-byte global stores.
// Measured (GB300, the call with its status read-back): 1,000,003 rows 988 ->
// 157 us, 20,590 rows 60 -> 30 us against one group of one tile per CTA, two
// CTAs per SM; the outputs are the same bits.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mlp.h"
#include "tc.cuh"

namespace lqt {

namespace {

constexpr int kTile = 128;
constexpr int kGroups = 4;                  // warpgroups (tiles in flight) per CTA
constexpr uint32_t kColsPerGroup = 128;     // hidden accumulator; the 48 output columns reuse it
constexpr uint32_t kTmemCols = kColsPerGroup * kGroups;
constexpr uint32_t kWaitLimit = 1u << 24;   // bounded mbarrier polls
constexpr uint32_t kSlabPitch = kMlpOut + 4;   // floats per row of a warp's output slab: no bank conflicts

// shared-memory plan (bytes)
constexpr uint32_t kOffW1 = 0;                                      // 128 x 48
constexpr uint32_t kOffW2 = kOffW1 + kMlpHid * kMlpIn * 2;          // 128 x 128
constexpr uint32_t kOffW3 = kOffW2 + kMlpHid * kMlpHid * 2;         // 48 x 128
constexpr uint32_t kOffXH = kOffW3 + kMlpOut * kMlpHid * 2;         // per group: inputs, hidden, output slabs
constexpr uint32_t kXHBytes = kTile * kMlpHid * 2;
constexpr uint32_t kOffBias = kOffXH + kGroups * kXHBytes;          // b1[128], b2[128], b3[48]
constexpr uint32_t kOffBar = kOffBias + (2 * kMlpHid + kMlpOut) * 4;
constexpr uint32_t kSmemBytes = kOffBar + 8 * kGroups + 16;         // mbarriers, TMEM slot
static_assert(kOffXH % 1024 == 0 && kXHBytes % 1024 == 0, "operand tiles 1 KB aligned");
static_assert(4 * 32 * kSlabPitch * 4 <= kXHBytes, "output slabs fit the operand buffer");
static_assert(kOffBar % 8 == 0 && kSmemBytes <= 227 * 1024, "shared memory");

// Copy a row-major [R][K] BF16 matrix from global into the K-major core layout.
__device__ void stage_kmajor(uint8_t *dst, const __nv_bfloat16 *src, int R, int K)
{
    const int chunks = R * (K / 8);
    for (int c = threadIdx.x; c < chunks; c += blockDim.x) {
        const int r = c / (K / 8), kg = c % (K / 8);
        const uint4 v = *reinterpret_cast<const uint4 *>(src + (int64_t)r * K + kg * 8);
        *reinterpret_cast<uint4 *>(dst + tc::kmaj_off(r, kg * 8, K)) = v;
    }
}

__device__ __forceinline__ float mlp_ex2(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float mlp_rcp(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// SiLU of two values, x / (1 + exp(-x)), as a BF16 pair.  One reciprocal of
// the product of the two denominators serves both; each quotient is corrected
// once by its remainder, which an FMA gives exactly (Markstein's correction),
// so it is within 2^-40 or so of the division before it is rounded.  (The
// reciprocals and quotients are carried negated: the remainder is then one
// FMA.)  That holds for |x| up to 43, where the product of two denominators,
// at most e^86, and its reciprocal are normal numbers; top keeps the largest
// |x| (a NaN stays), for silu_plain to see what is beyond.
__device__ __forceinline__ uint32_t silu2_bf16(uint64_t x, float &top)
{
    float x0, x1, a0, a1, d0, d1, q0, q1;
    tc::split2(x, x0, x1);
    asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(top) : "f"(fabsf(x0)), "f"(fabsf(x1)));
    tc::split2(tc::mul2(x, tc::pair2(-1.4426950408889634f, -1.4426950408889634f)), a0, a1);
    const uint64_t d = tc::add2(tc::pair2(mlp_ex2(a0), mlp_ex2(a1)), tc::pair2(1.0f, 1.0f));
    tc::split2(d, d0, d1);
    const float r = mlp_rcp(d0 * -d1);
    const uint64_t nr = tc::pair2(r * d1, r * d0);
    uint64_t nq = tc::mul2(x, nr);
    nq = tc::fma2(tc::fma2(nq, d, x), nr, nq);
    tc::split2(nq, q0, q1);
    const __nv_bfloat162 h = __floats2bfloat162_rn(-q0, -q1);
    return *reinterpret_cast<const uint32_t *>(&h);
}

// Whether the values behind top are all in silu2_bf16's range.  (One maximum of
// three operands a pair costs what bounding the two exponentials did, 155 us for
// a million rows; the extremes of the exponentials or of x with its sign, which
// would let large positive x pass, take 163.)
__device__ __forceinline__ bool silu_plain(float top) { return top <= 43.f; }

// The division itself, for the others: 0 for large negative x, x for large
// positive, infinities and NaN as the formula gives them.
__device__ __forceinline__ uint32_t silu2_div(float x0, float x1)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(x0 / (1.0f + __expf(-x0)), x1 / (1.0f + __expf(-x1)));
    return *reinterpret_cast<const uint32_t *>(&h);
}

// Named barrier of one warpgroup (ids 1..4; 0 is __syncthreads), and the same
// with the AND of a flag.
__device__ __forceinline__ void wg_sync(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }
__device__ __forceinline__ int wg_and(int id, int v)
{
    int r;
    asm volatile(
        "{\n.reg .pred p, q;\nsetp.ne.s32 p, %1, 0;\nbar.red.and.pred q, %2, 128, p;\nselp.s32 %0, 1, 0, q;\n}\n"
        : "=r"(r)
        : "r"(v), "r"(id)
        : "memory");
    return r;
}

// GEMM D[128 x N] = A[128 x K] * B[N x K]^T from shared memory into TMEM.
__device__ __forceinline__ void gemm(uint32_t tmem_d, const uint8_t *A, const uint8_t *B, int K, int N, bool swap)
{
    const uint32_t lbo = 128, sbo = (uint32_t)(K / 8) * 128;
    const uint32_t l = swap ? sbo : lbo, s = swap ? lbo : sbo;
    const uint32_t id = tc::idesc_bf16_f32(128, N);
    const uint32_t a0 = tc::smem_u32(A), b0 = tc::smem_u32(B);
    for (int kk = 0; kk < K / 16; ++kk) {
        const uint32_t step = (uint32_t)kk * 256;     // two core matrices along K
        tc::mma_bf16(tmem_d, tc::smem_desc(a0 + step, l, s), tc::smem_desc(b0 + step, l, s), id, kk > 0);
    }
}

}  // namespace

// X: [n][48] BF16 (normalised inputs), Y: [n][48] FP32 outputs.
__global__ void __launch_bounds__(128 * kGroups, 1) k_mlp_infer_tc(const __nv_bfloat16 *__restrict__ X,
                                                                   float *__restrict__ Y, MlpDev w, int64_t n,
                                                                   int *err, int swap)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int grp = tid >> 7, t = tid & 127;          // warpgroup, row within its tile
    const int bar_id = 1 + grp;
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + kOffBar) + grp;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + kOffBar + 8 * kGroups);
    float *bias = reinterpret_cast<float *>(smem + kOffBias);
    uint8_t *xh = smem + kOffXH + grp * kXHBytes;
    float *slab = reinterpret_cast<float *>(xh) + (warp & 3) * (32 * kSlabPitch);

    stage_kmajor(smem + kOffW1, w.w1t, kMlpHid, kMlpIn);
    stage_kmajor(smem + kOffW2, w.w2t, kMlpHid, kMlpHid);
    stage_kmajor(smem + kOffW3, w.w3t, kMlpOut, kMlpHid);
    for (int i = tid; i < 2 * kMlpHid + kMlpOut; i += blockDim.x)
        bias[i] = i < kMlpHid ? w.b1[i] : (i < 2 * kMlpHid ? w.b2[i - kMlpHid] : w.b3[i - 2 * kMlpHid]);
    if (t == 0) {
        tc::mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tc::tmem_alloc(tslot, kTmemCols);
    tc::fence_proxy_async();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t t_mma = *tslot + grp * kColsPerGroup;
    // warp w of the CTA may access TMEM lanes 32 * (w % 4) .. + 31
    const uint32_t t_acc = t_mma + ((uint32_t)((warp & 3) * 32) << 16);
    uint32_t phase = 0;
    const int64_t ntiles = (n + kTile - 1) / kTile;
    const bool wide = (reinterpret_cast<uintptr_t>(Y) & 15) == 0;

    // tiles are dealt to the CTAs first and then to their groups, so that few
    // tiles spread over the SMs
    const int64_t tstride = (int64_t)gridDim.x * kGroups;
    int64_t tile = blockIdx.x + (int64_t)gridDim.x * grp;
    uint4 xin[kMlpIn / 8];
    auto load_x = [&](int64_t tl) {
        const int64_t row = tl * kTile + t;
#pragma unroll
        for (int j = 0; j < kMlpIn / 8; ++j)
            xin[j] = row < n ? __ldcs(reinterpret_cast<const uint4 *>(X + row * kMlpIn) + j) : make_uint4(0, 0, 0, 0);
    };
    if (tile < ntiles) load_x(tile);
    for (; tile < ntiles; tile += tstride) {
#pragma unroll
        for (int j = 0; j < kMlpIn / 8; ++j) *reinterpret_cast<uint4 *>(xh + tc::kmaj_off(t, j * 8, kMlpIn)) = xin[j];
        tc::fence_proxy_async();
        tc::fence_before();       // the previous tile's tcgen05.ld before this barrier
        wg_sync(bar_id);
        if (tile + tstride < ntiles) load_x(tile + tstride);   // in flight during this tile's layers
        bool ok = true;
        for (int layer = 0; layer < 3; ++layer) {
            if (t == 0) {
                tc::fence_after();
                if (layer == 0) gemm(t_mma, xh, smem + kOffW1, kMlpIn, kMlpHid, swap);
                else if (layer == 1) gemm(t_mma, xh, smem + kOffW2, kMlpHid, kMlpHid, swap);
                else gemm(t_mma, xh, smem + kOffW3, kMlpHid, kMlpOut, swap);
                tc::mma_commit(bar);
            }
            // the group takes one decision: a wait that ran out ends its work,
            // after one more bounded wait for the MMA in flight (TMEM is freed
            // at the end)
            const bool w_ok = tc::mbar_wait(bar, phase, kWaitLimit);
            if (!wg_and(bar_id, w_ok ? 1 : 0)) {
                if (!w_ok) tc::mbar_wait(bar, phase, kWaitLimit);
                if (t == 0) atomicExch(err, 1);
                ok = false;
                break;
            }
            phase ^= 1;
            tc::fence_after();
            if (layer == 2) break;
            // hidden layer: TMEM -> bias, SiLU -> BF16 operand (over the bytes
            // of the operand that the finished MMA no longer needs)
            const float4 *bs = reinterpret_cast<const float4 *>(bias + layer * kMlpHid);
            float top = 0.f;
#pragma unroll 1
            for (int c = 0; c < kMlpHid; c += 32) {
                float v[32];
                tc::tmem_ld32(t_acc + c, v);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t p[4];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float4 b = bs[(c >> 2) + q * 2 + i];
                        const float *u = v + q * 8 + 4 * i;
                        p[2 * i] = silu2_bf16(tc::add2(tc::pair2(u[0], u[1]), tc::pair2(b.x, b.y)), top);
                        p[2 * i + 1] = silu2_bf16(tc::add2(tc::pair2(u[2], u[3]), tc::pair2(b.z, b.w)), top);
                    }
                    *reinterpret_cast<uint4 *>(xh + tc::kmaj_off(t, c + q * 8, kMlpHid)) = make_uint4(p[0], p[1], p[2], p[3]);
                }
            }
            // (a warp whose rows hold a value out of range: its columns again)
            if (__any_sync(0xffffffffu, !silu_plain(top))) {
#pragma unroll 1
                for (int c = 0; c < kMlpHid; c += 16) {
                    float v[16];
                    tc::tmem_ld16(t_acc + c, v);
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const float4 b = bs[(c >> 2) + q * 2], e = bs[(c >> 2) + q * 2 + 1];
                        const float *u = v + q * 8;
                        *reinterpret_cast<uint4 *>(xh + tc::kmaj_off(t, c + q * 8, kMlpHid)) =
                            make_uint4(silu2_div(u[0] + b.x, u[1] + b.y), silu2_div(u[2] + b.z, u[3] + b.w),
                                       silu2_div(u[4] + e.x, u[5] + e.y), silu2_div(u[6] + e.z, u[7] + e.w));
                    }
                }
            }
            tc::fence_before();
            tc::fence_proxy_async();
            wg_sync(bar_id);
        }
        if (!ok) break;
        // output rows: TMEM -> bias -> this warp's slab -> whole row segments
        const float4 *b3 = reinterpret_cast<const float4 *>(bias + 2 * kMlpHid);
#pragma unroll
        for (int c = 0; c < kMlpOut; c += 16) {
            float v[16];
            tc::tmem_ld16(t_acc + c, v);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 b = b3[(c >> 2) + q];
                *reinterpret_cast<float4 *>(slab + lane * kSlabPitch + c + 4 * q) =
                    make_float4(v[4 * q] + b.x, v[4 * q + 1] + b.y, v[4 * q + 2] + b.z, v[4 * q + 3] + b.w);
            }
        }
        __syncwarp();
        const int64_t row0 = tile * kTile + (warp & 3) * 32;
        float *out = Y + row0 * kMlpOut;
        const int rows = (int)(n - row0 < 32 ? (n - row0 > 0 ? n - row0 : 0) : 32);
        if (wide) {
#pragma unroll
            for (int j = 0; j < kMlpOut / 4; ++j) {
                const int e = j * 32 + lane, r = e / (kMlpOut / 4), c4 = e - r * (kMlpOut / 4);
                const float4 v = *reinterpret_cast<const float4 *>(slab + r * kSlabPitch + 4 * c4);
                if (r < rows) __stcs(reinterpret_cast<float4 *>(out) + e, v);
            }
        } else {
            for (int e = lane; e < rows * kMlpOut; e += 32) out[e] = slab[(e / kMlpOut) * kSlabPitch + e % kMlpOut];
        }
        wg_sync(bar_id);          // every slab is read before the next inputs overwrite it
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(*tslot, kTmemCols);
}

cudaError_t launch_mlp_infer_tc(const __nv_bfloat16 *X, float *Y, const MlpDev &w, int64_t n, int *err, int swap,
                                cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    static std::atomic<uint64_t> attr_done{0};
    cudaError_t e = tc::smem_attr_once(k_mlp_infer_tc, kSmemBytes, attr_done);
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int64_t ntiles = (n + kTile - 1) / kTile;
    // one CTA per SM: its 512 TMEM columns are the SM's whole TMEM and the
    // shared memory admits one, so tcgen05.alloc never waits
    const int64_t grid = ntiles < nsm ? ntiles : nsm;
    k_mlp_infer_tc<<<(unsigned)grid, 128 * kGroups, kSmemBytes, st>>>(X, Y, w, n, err, swap);
    return cudaGetLastError();
}

}  // namespace lqt
