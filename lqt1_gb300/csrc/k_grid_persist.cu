// k_grid_persist.cu -- many plain steps of a small grid in one launch (mixed
// form, 1D/2D/3D).
//
// On a small grid a step is a chain: read the state, the cell update, write
// the state and V, end the launch, start the next one.  Here the grid is
// resident: one thread per voxel keeps its state in registers for the whole
// launch, and blocks exchange V through the two dense grids, which the L2
// holds.  97 x 64 voxels take 2.7 us a step instead of 5.5; what remains is
// one warp's chain through the update and the exchange.
//
// A voxel's ionic update needs only its own V, so a step is: the ionic update;
// then wait until the blocks around have published their V of this step (they
// did so before their own ionic update, so the wait is short); the stencil; V
// and its mirror voxels; publish.  A block's fifth warp waits, publishes and
// keeps the clock, so that no voxel does.  The wait also guards the other
// grid: a block that has published step s has read everything of step s - 1,
// whose grid the next V goes to, and the relation is symmetric.  Blocks that
// exchange no V, directly or through others, are not ordered by it.
//
// The launch is cooperative: every block is resident, so every wait ends.  It
// is bounded all the same; one that runs out sets *err, the blocks leave, and
// the run is reported as failed.  It also sets the word behind the flags, by
// which launches that are queued already leave at once instead of waiting in
// their turn.
#include <cuda_runtime.h>
#include <stdint.h>

#include "k_grid.cuh"

namespace lqt {

namespace {

constexpr uint32_t kPersistPolls = 1u << 23;     // a second or more

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(uint32_t *p, uint32_t v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void ran_out(const PersistArgs &a)
{
    atomicExch(a.err, 1);
    atomicExch(a.flags + gridDim.x, 1u);
}

// What a voxel's diffusion needs besides V, for the whole launch.
template <int DIM> struct Diffusion {
    float D[6], B[3];
};

// grid_du with V from the L2 (other blocks write it during this launch).
template <int DIM>
__device__ __forceinline__ float persist_du(const GridDev<float> &gd, const float *V, int64_t g, float vc,
                                            const Diffusion<DIM> &d)
{
    if constexpr (DIM == 1) {
        const int64_t n = gd.ntissue;
        float fo, so;
        if (n == 1) return 0.f;
        if (g == 0) {
            const float vp = __ldcg(V + g + 1);
            fo = (vp - vc) * gd.inv_dx;
            so = (vp + vc - 2.f * vc) * gd.inv_dx2;
        } else if (g == n - 1) {
            const float vm = __ldcg(V + g - 1);
            fo = (vc - vm) * gd.inv_dx;
            so = (vc + vm - 2.f * vc) * gd.inv_dx2;
        } else {
            const float vp = __ldcg(V + g + 1), vm = __ldcg(V + g - 1);
            fo = (vp - vm) * gd.inv_2dx;
            so = (vp + vm - 2.f * vc) * gd.inv_dx2;
        }
        return du_fma(d.B[0], fo, du_mul(d.D[0], so));
    } else {
        const int64_t sx = gd.sx, sy = gd.sy;
        auto at = [&](int i, int j, int l) { return __ldcg(V + (g + i * sx + j * sy + l)); };
        if (gd.d6) return sub_du_of<DIM>(gd, at, vc, d.D, d.B);
        const float c2 = gd.inv_dx2;
        const float lxx = du_mul(at(1, 0, 0) + at(-1, 0, 0) - 2.f * vc, c2);
        const float lyy = du_mul(at(0, 1, 0) + at(0, -1, 0) - 2.f * vc, c2);
        float lzz = 0.f;
        if constexpr (DIM == 3) lzz = du_mul(at(0, 0, 1) + at(0, 0, -1) - 2.f * vc, c2);
        return gd.diso * (lxx + lyy + lzz);
    }
}

}  // namespace

// (Three blocks fit on an SM: several simulations run side by side.  Eight of
// 120 x 120 voxels take 1.5 us a step and simulation so, 2.5 with the registers
// of two blocks, 1.7 with a launch per step of each.)
template <int DIM>
__global__ void __launch_bounds__(kPersistBlock + 32, 3)
    k_grid_persist(GridDev<float> gd, StepT<float> kst, int cur, PersistArgs a)
{
    // three clocks: the detector of step s runs beside the making of s + 2's
    __shared__ Clock clk[3];
    __shared__ int go;
    __shared__ uint32_t base, dead;       // steps published, or a wait run out, when the launch begins
    const int t = threadIdx.x, b = blockIdx.x;
    const uint32_t limit = gd.sub_wait_limit ? gd.sub_wait_limit : kPersistPolls;
    if (t == kPersistBlock) {
        // (three loads in flight together)
        const uint32_t f = ld_relaxed(a.flags + b), out = ld_relaxed(a.flags + gridDim.x);
        const Clock c0 = gd.clk[cur];
        clk[0] = c0;
        base = f;
        dead = out;
    }
    __syncthreads();
    if (t >= kPersistBlock) {
        const int lane = t - kPersistBlock;
        const int2 dep = a.dep[b];
        const uint32_t base0 = base;
        bool ok = dead == 0;
        for (int s = 0; s < a.nsteps; ++s) {
            if (lane == 0) clk[(s + 1) % 3] = next_clock(gd, clk[s % 3]);
            if (s > 0) {
                for (int i = dep.x + lane; i <= dep.y; i += 32) {
                    uint32_t polls = 0;
                    while ((int32_t)(ld_acquire(a.flags + i) - (base0 + s)) < 0 && polls < limit) ++polls;
                    ok = ok && polls < limit;
                }
            }
            ok = __all_sync(0xffffffffu, ok);
            if (lane == 0) {
                go = ok;
                if (!ok) ran_out(a);
            }
            __syncthreads();
            if (!ok) break;
            __syncthreads();
            // (a failure-path test keeps block 0 from publishing)
            if (lane == 0 && !(b == 0 && gd.sub_skip_copy)) {
                __threadfence();
                st_release(a.flags + b, base0 + s + 1);
            }
        }
        // Block 0 leaves the clock of the launch's end, once every block has read
        // the one of its beginning (the voxels' threads look, below).
        if (b == 0 && __syncthreads_and(ok) && lane == 0) gd.clk[(cur + a.nsteps) & 1] = clk[a.nsteps % 3];
        return;
    }

    const int64_t k = (int64_t)b * kPersistBlock + t;
    const bool on = k < gd.ntissue;
    CellState<float> c{};
    Diffusion<DIM> d{};
    int64_t g = 0;
    uint8_t ctl = 0;
    int32_t gref = 0;
    if (on) {
        g = DIM == 1 ? k : (int64_t)gd.gidx[k];
        ctl = gd.ctl[k];
        gref = ghost_ref(gd, k, ctl);
        load_cell(c, gd.s, k);
        c.v = gd.vg[cur][g];
        if constexpr (DIM == 1) {
            d.D[0] = gd.coeff[k];
            d.B[0] = gd.dcoeff[k];
        } else if (gd.d6) {
#pragma unroll
            for (int i = 0; i < 6; ++i) d.D[i] = gd.d6[6 * k + i];
#pragma unroll
            for (int i = 0; i < 3; ++i) d.B[i] = gd.b3[3 * k + i];
        }
    }
    bool ran = true;
    for (int s = 0; s < a.nsteps; ++s) {
        const Clock &ck = clk[s % 3];
        const float vc = c.v;
        StepOut<float> o{};
        float4 det{};
        if (on) {
            if (gd.det) det = gd.det[k];
            tpord_update(c, ctl & kCtlType, gd.model, kst, grid_stim(gd, ck, ctl, k), 0.f, &o);
        }
        __syncthreads();
        if (!go) {
            ran = false;
            break;
        }
        if (on) {
            const float du = persist_du<DIM>(gd, gd.vg[(cur + s) & 1], g, vc, d);
            c.v = fmaf(o.dvdt + du, kst.dt, vc);
            put_v(gd, gd.vg[(cur + s + 1) & 1], g, ctl, gref, c.v);
        }
        __syncthreads();
        if (on) {
            if (gd.det) grid_detect_rec(gd, ck, k, det, vc, c.v, o.dvdt);
            grid_count_bad(gd, c.v);
        }
    }
    if (on) store_cell(c, gd.s, k);
    if (b == 0) {
        // After an even number of steps the slot of the end is the one that every
        // block starts from.  Blocks that exchange no V with this one are not
        // ordered with it, so all must have published their first step, which
        // they do after reading the clock.
        bool begun = ran;
        if (ran && (a.nsteps & 1) == 0) {
            const uint32_t first = base + 1;
            begun = false;
            for (uint32_t polls = 0; !begun && polls < limit; ++polls) {
                begun = true;
                for (int i = t; i < (int)gridDim.x; i += kPersistBlock)
                    begun = begun && (int32_t)(ld_relaxed(a.flags + i) - first) >= 0;
            }
            __threadfence();
            if (!begun) ran_out(a);
        }
        __syncthreads_and(begun);
    }
}

int grid_persist_capacity(int dim)
{
    int dev = 0, nsm = 0, per = 0, coop = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    const int bs = kPersistBlock + 32;
    cudaError_t e = dim == 1   ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_grid_persist<1>, bs, 0)
                    : dim == 2 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_grid_persist<2>, bs, 0)
                               : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_grid_persist<3>, bs, 0);
    if (e != cudaSuccess || !coop) return 0;
    return nsm * (per < kPersistPerSM ? per : kPersistPerSM);
}

cudaError_t launch_grid_persist(const GridDev<float> &gd, const StepK &k, int cur, int dim, const PersistArgs &a,
                                cudaStream_t st)
{
    GridDev<float> g = gd;
    StepT<float> kk = step_as<float>(k);
    PersistArgs pa = a;
    void *args[] = {&g, &kk, &cur, &pa};
    const void *f = dim == 1   ? (const void *)k_grid_persist<1>
                    : dim == 2 ? (const void *)k_grid_persist<2>
                               : (const void *)k_grid_persist<3>;
    const unsigned nb = (unsigned)((gd.ntissue + kPersistBlock - 1) / kPersistBlock);
    return cudaLaunchCooperativeKernel(f, dim3(nb), dim3(kPersistBlock + 32), args, 0, st);
}

}  // namespace lqt
