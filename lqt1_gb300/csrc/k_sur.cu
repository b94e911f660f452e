// k_sur.cu -- the learned surrogate around the plain integrator:
//   * training pairs generated by the plain mixed-form TPORd step,
//   * feature normalisation into the network's BF16 inputs.
// A surrogate macro step advances a cell by nsub plain steps (nsub = 5: 0.1 ms
// at dt = 0.02 ms) with no diffusion and no stimulus: one coarse TPORd step of
// the macro length plus the network's correction of the 38 evolving states.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "mlp.h"
#include "sur.h"
#include "sur_dev.cuh"

namespace lqt {

__device__ __forceinline__ void sur_init_cell(CellState<float> &c)
{
    c.v = -87.5f;
    c.nai = make_float2(7.f, 0.f); c.nass = make_float2(7.f, 0.f);
    c.ki = make_float2(145.f, 0.f); c.kss = make_float2(145.f, 0.f);
    c.cai = make_float2(1.0e-4f, 0.f); c.cass = make_float2(1.0e-4f, 0.f);
    c.cansr = make_float2(1.2f, 0.f); c.cajsr = make_float2(1.2f, 0.f);
    c.sm = 0.f; c.sh = 1.f; c.sj = 1.f; c.mL = 0.f; c.hL = 1.f; c.hLp = 1.f; c.a = 0.f; c.iF = 1.f; c.iS = 1.f;
    c.ap = 0.f; c.iFp = 1.f; c.iSp = 1.f; c.d = 0.f; c.ff = 1.f; c.fs = 1.f; c.fcaf = 1.f; c.fcas = 1.f;
    c.jca = 1.f; c.nca = 0.f; c.ffp = 1.f; c.fcafp = 1.f; c.xrf = 0.f; c.xrs = 0.f; c.xs1 = 0.f; c.xs2 = 0.f;
    c.xk1 = 1.f; c.Jrelnp = 0.f; c.Jrelp = 0.f; c.CaMKt = 0.f;
}

// One thread per cell: pace with the plain mixed step, and at macro-step
// boundaries in the surrogate's regime (|dV/dt| <= dvdt_max, no stimulus in
// the coming macro step, past the warm-up) record, with probability `prob`,
// the inputs and the correction: state after nsub plain steps minus the
// state after one coarse step of the macro length from the same start.
// Macro steps that are not recorded carry a constant current uniform in
// +-jitter (a stand-in for the electrotonic load of tissue).
// Two passes make the pair set and its order independent of thread timing:
// with counts != NULL the kernel only counts each cell's recorded macro steps;
// with offsets != NULL the j-th pair of cell i goes to row offsets[i] + j
// (rows at or past cap are dropped, so a truncated set keeps the first cells
// in cell order).  A cell's trajectory is the same in both passes: a macro
// step chosen for recording carries no jitter current whether or not its row
// is kept.
__global__ void __launch_bounds__(128) k_sur_datagen(const SurCell *__restrict__ cells, int64_t ncells,
                                                     const ModelK *__restrict__ models, StepT<float> k,
                                                     StepT<float> kmac, float *__restrict__ X,
                                                     float *__restrict__ D, int64_t *__restrict__ counts,
                                                     const int64_t *__restrict__ offsets, int64_t cap, uint64_t seed,
                                                     float dvdt_max, float prob, float jitter, int nsub)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= ncells) return;
    const SurCell sc = cells[i];
    const ModelT<float> m = model_as<float>(models[sc.model]);
    CellState<float> c;
    sur_init_cell(c);
    const int ct = sc.ctype;
    const int cls = sur_class(ct);
    StepOut<float> o{};
    int64_t slot = -1, nrec = 0;
    float xc[kMlpNState] = {};   // coarse end state (hi parts) of the pending sample
    float loc[8] = {};           // and its concentration lo parts
    float ipert = 0.f;
    // completes the pending sample at the end of its macro step: fine minus coarse
    auto finish = [&]() {
        if (slot < 0) return;
        float x1[kMlpNState];
        state38(c, x1);
        float2 *cp[8];
        conc_ptrs(c, cp);
        float *d = D + slot * kMlpNState;
        d[0] = x1[0] - xc[0];
#pragma unroll
        for (int j = 0; j < 8; ++j) d[1 + j] = (cp[j]->x - xc[1 + j]) + (cp[j]->y - loc[j]);
#pragma unroll
        for (int j = 9; j < kMlpNState; ++j) d[j] = x1[j] - xc[j];
        slot = -1;
    };
    for (int64_t st = 0; st < sc.nsteps; ++st) {
        const int64_t ph = st % sc.bcl_steps;
        if (st % nsub == 0) {
            finish();
            const bool stim_ahead = ph + nsub > sc.stim_on && ph < sc.stim_off;
            ipert = 0.f;
            if (st >= sc.warm_steps && !stim_ahead && fabsf(o.dvdt) <= dvdt_max && st + nsub <= sc.nsteps &&
                (sur_hash(seed, (uint64_t)i, (uint64_t)st) & 0xFFFFFF) < (uint32_t)(prob * 16777216.f)) {
                const int64_t s = counts ? -1 : offsets[i] + nrec;
                ++nrec;
                if (s >= 0 && s < cap) {
                    slot = s;
                    float x0[kMlpNState];
                    state38(c, x0);
                    float *xr = X + slot * kSurFeat;
#pragma unroll
                    for (int j = 0; j < kMlpNState; ++j) xr[j] = x0[j];
                    xr[38] = sc.gks_scale;
                    xr[39] = sc.pca_scale;
                    xr[40] = sc.iso_scale;
                    xr[41] = cls == 0;
                    xr[42] = cls == 1;
                    xr[43] = cls == 2;
                    CellState<float> cc = c;
                    StepOut<float> oc;
                    tpord_update(cc, ct, m, kmac, 0.f, 0.f, &oc);
                    state38(cc, xc);
                    float2 *cp[8];
                    conc_ptrs(cc, cp);
#pragma unroll
                    for (int j = 0; j < 8; ++j) loc[j] = cp[j]->y;
                }
            } else if (jitter > 0.f && !stim_ahead) {
                const uint32_t h = sur_hash(seed ^ 0x5bd1e995ull, (uint64_t)i, (uint64_t)st);
                ipert = jitter * ((float)(h >> 8) * (2.0f / 16777216.0f) - 1.0f);
            }
        }
        const float ist = (ph >= sc.stim_on && ph < sc.stim_off) ? sc.stim : (slot >= 0 ? 0.f : ipert);
        tpord_update(c, ct, m, k, ist, 0.f, &o);
    }
    finish();   // a sample of the cell's very last macro step
    if (counts) counts[i] = nrec;
}

// Raw features (kSurFeat floats per row) -> normalised BF16 network inputs
// (48 per row, zero padded); optional raw changes -> normalised FP32 targets.
// The rows are gathered, so what counts is that a row is read and written in
// whole sectors: a thread takes four neighbouring features of a row (12
// threads per row, its normalisation held in registers), with 16- and 8-byte
// accesses where the four buffers are aligned for them (WIDE).  One thread per
// row walking its 48 features took 31 us for 8192 rows, waiting on loads 32
// rows apart; this form takes 6 us.
constexpr int kPrepChunks = kMlpIn / 4;            // threads per row
constexpr int kPrepRows = 16;                      // rows per block
template <bool WIDE>
__global__ void __launch_bounds__(kPrepChunks * kPrepRows)
    k_sur_prepare(const float *__restrict__ X, const float *__restrict__ D, const int64_t *__restrict__ idx, int64_t n,
                  const float *__restrict__ norm, __nv_bfloat16 *__restrict__ xb, float *__restrict__ t)
{
    const int c = threadIdx.x % kPrepChunks, j0 = 4 * c;
    float mu[4], sc[4], os[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        mu[i] = norm[j0 + i];
        sc[i] = norm[kMlpIn + j0 + i];
        os[i] = norm[2 * kMlpIn + j0 + i];
    }
    for (int64_t r = blockIdx.x * (int64_t)kPrepRows + threadIdx.x / kPrepChunks; r < n; r += (int64_t)gridDim.x * kPrepRows) {
        const int64_t s = idx ? idx[r] : r;
        float x[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {0.f, 0.f, 0.f, 0.f};
        const float *xr = X + s * kSurFeat + j0;
        if (j0 < kSurFeat) {
            if (WIDE) {
                const float4 q = __ldg(reinterpret_cast<const float4 *>(xr));
                x[0] = q.x; x[1] = q.y; x[2] = q.z; x[3] = q.w;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = xr[i];
            }
        }
        if (t) {
            const float *dr = D + s * kMlpNState + j0;
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
                if (j0 + i < kMlpNState) {
                    if (WIDE) {
                        const float2 q = __ldg(reinterpret_cast<const float2 *>(dr + i));
                        d[i] = q.x; d[i + 1] = q.y;
                    } else {
                        d[i] = dr[i]; d[i + 1] = dr[i + 1];
                    }
                }
            }
        }
        __align__(8) __nv_bfloat16 h[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __float2bfloat16(j0 + i < kSurFeat ? (x[i] - mu[i]) * sc[i] : 0.f);
        __nv_bfloat16 *xo = xb + r * kMlpIn + j0;
        if (WIDE) {
            *reinterpret_cast<uint2 *>(xo) = *reinterpret_cast<const uint2 *>(h);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) xo[i] = h[i];
        }
        if (t) {
            float *to = t + r * kMlpOut + j0;
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = j0 + i < kMlpNState ? d[i] / os[i] : 0.f;
            if (WIDE) {
                *reinterpret_cast<float4 *>(to) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) to[i] = v[i];
            }
        }
    }
}
static_assert(kMlpIn == kMlpOut && kSurFeat % 4 == 0 && kMlpNState % 2 == 0, "four features per thread");

cudaError_t launch_sur_datagen(const SurCell *cells, int64_t ncells, const ModelK *models, const StepK &k,
                               const StepK &kmac, float *X, float *D, int64_t *counts, const int64_t *offsets,
                               int64_t cap, uint64_t seed, float dvdt_max, float prob, float jitter, int nsub,
                               cudaStream_t st)
{
    if (ncells <= 0) return cudaSuccess;
    k_sur_datagen<<<(unsigned)((ncells + 127) / 128), 128, 0, st>>>(cells, ncells, models, step_as<float>(k),
                                                                    step_as<float>(kmac), X, D, counts, offsets, cap,
                                                                    seed, dvdt_max, prob, jitter, nsub);
    return cudaGetLastError();
}

cudaError_t launch_sur_prepare(const float *X, const float *D, const int64_t *idx, int64_t n, const float *norm,
                               __nv_bfloat16 *xb, float *t, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    int64_t nb = (n + kPrepRows - 1) / kPrepRows;
    if (nb > 152 * 64) nb = 152 * 64;
    // rows are 176 (X), 152 (D), 96 (xb) and 192 (t) bytes: aligned buffers have aligned four-feature groups
    auto off = [](const void *p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) != 0; };
    const bool wide = !(off(X, 16) || off(D, 8) || off(xb, 8) || off(t, 16));
    if (wide) k_sur_prepare<true><<<(unsigned)nb, kPrepChunks * kPrepRows, 0, st>>>(X, D, idx, n, norm, xb, t);
    else k_sur_prepare<false><<<(unsigned)nb, kPrepChunks * kPrepRows, 0, st>>>(X, D, idx, n, norm, xb, t);
    return cudaGetLastError();
}

}  // namespace lqt
