// k_sur_sub.cu -- the V-only step of the voxels inside a surrogate macro step,
// mixed form, 1D/2D/3D: k_sur_substep (k_grid.cuh, one thread per voxel,
// direct loads) and, below, persistent kernels whose streamed rows are staged
// in shared memory: k_sur_substep_tile, k_sur_substep_vbox (with the V halo),
// k_sur_substep_pair and k_sur_substep_warp (two voxels per thread).
#include <atomic>
#include <cstddef>

#include "k_grid.cuh"
#include "tc.cuh"

namespace lqt {

namespace {

constexpr uint32_t kSubWaitLimit = 1u << 22;   // bounded mbarrier polls per tile

// One tile's rows, in the order of the copies: the macro step's ionic rate,
// the dense index, the FP16 tensor row (3 half2 per voxel: the scaled fibre
// direction and the divergence, GridDev::t3h), the control byte and the
// detector flag.
struct __align__(16) SubStage {
    float rate[kSubTile];
    int32_t gidx[kSubTile];
    __half2 t3[kSubTile * 3];
    uint8_t ctl[kSubTile];
    uint8_t flag[kSubTile];
};
static_assert(sizeof(SubStage) % 16 == 0 && offsetof(SubStage, gidx) % 16 == 0 && offsetof(SubStage, t3) % 16 == 0 &&
                  offsetof(SubStage, ctl) % 16 == 0 && offsetof(SubStage, flag) % 16 == 0,
              "bulk copies need 16-byte aligned destinations");

// Thread 0: the copies of tile k0 / kSubTile into one stage, completing on bar.
// Every array holds whole tiles (pad_tiles), so each copy is in bounds, and
// k0 is a multiple of kSubTile, so every source is 16-byte aligned.
__device__ __forceinline__ void sub_issue(SubStage &sg, uint64_t *bar, const GridDev<float> &gd, int64_t k0, bool det)
{
    constexpr uint32_t n = kSubTile;
    tc::mbar_expect_tx(bar, n * (4 + 4 + 12 + 1) + (det ? n : 0));
    tc::bulk_g2s(sg.rate, gd.srate + k0, n * 4, bar);
    tc::bulk_g2s(sg.gidx, gd.gidx + k0, n * 4, bar);
    tc::bulk_g2s(sg.t3, gd.t3h + 3 * k0, n * 12, bar);
    tc::bulk_g2s(sg.ctl, gd.ctl + k0, n, bar);
    if (det) tc::bulk_g2s(sg.flag, gd.sdflag + k0, n, bar);
}

}  // namespace

// Persistent: CTA b takes tiles b, b + gridDim.x, ...  Two stages: while the
// threads step the voxels of one tile (V stencil from the dense grid, through
// L1/L2), the copy engine brings the next tile's rows, so the streamed bytes
// stay in flight without a per-thread load chain in front of the stencil.
// Arithmetic identical to k_sur_substep.  A copy wait that runs out sets bit 1
// of *serr; the CTA waits (bounded) for its copies still in flight and leaves
// its remaining tiles unstepped.  gd.sub_skip_copy / gd.sub_wait_limit drive
// that path in a test: the first tile's copies are left out and the wait
// bound shortened, so the wait runs out on a phase nothing completes.
template <int DIM, int MINB>
__global__ void __launch_bounds__(kSubTile, MINB) k_sur_substep_tile(GridDev<float> gd, float dt, int cur)
{
    __shared__ SubStage stg[2];
    __shared__ __align__(8) uint64_t bar[2];
    const int t = threadIdx.x;
    const int64_t ntiles = (gd.ntissue + kSubTile - 1) / kSubTile;
    const int64_t stride = gridDim.x;
    int64_t tile = blockIdx.x;
    if (tile >= ntiles) return;
    const bool det = gd.det != nullptr;
    const uint32_t lim = gd.sub_wait_limit ? gd.sub_wait_limit : kSubWaitLimit;
    if (t == 0) {
        tc::mbar_init(&bar[0], 1);
        tc::mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // (a failure-path test leaves the first tile's copies out: nothing
        // completes that phase and its wait runs out)
        if (!gd.sub_skip_copy) sub_issue(stg[0], &bar[0], gd, tile * kSubTile, det);
        if (tile + stride < ntiles) sub_issue(stg[1], &bar[1], gd, (tile + stride) * kSubTile, det);
    }
    __syncthreads();
    const Clock ck = gd.clk[cur];
    const float *__restrict__ V = gd.vg[cur];
    float *__restrict__ Vn = gd.vg[cur ^ 1];
    for (uint32_t it = 0; tile < ntiles; tile += stride, ++it) {
        const int s = it & 1;
        const bool ok = tc::mbar_wait(&bar[s], (it >> 1) & 1, lim);
        if (!__syncthreads_and(ok ? 1 : 0)) {
            if (t == 0) {
                atomicOr(gd.serr, 2);
                // let this CTA's copies in flight land before it leaves
                // (the full bound: these are real copies; a first tile left
                // out by the failure-path test has none)
                if (it > 0 || !gd.sub_skip_copy) tc::mbar_wait(&bar[s], (it >> 1) & 1, kSubWaitLimit);
                if (tile + stride < ntiles) tc::mbar_wait(&bar[s ^ 1], ((it + 1) >> 1) & 1, kSubWaitLimit);
            }
            return;
        }
        const SubStage &sg = stg[s];
        const int64_t k = tile * kSubTile + t;
        const float r = sg.rate[t];
        if (k < gd.ntissue && r == r) {
            const int64_t g = sg.gidx[t];
            float2 q[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) q[i] = __half22float2(sg.t3[3 * t + i]);
            float Dt[6], Bt[3];
            sub_tensor_unpack<DIM>(q, gd.sub_dtr, gd.sub_dsg, Dt, Bt);
            const float vc = V[g];
            const float du = sub_du<DIM>(gd, V, g, k, vc, Dt, Bt);
            const float ist = grid_stim(gd, ck, sg.ctl[t], k);
            const float dvdt = r - ist;
            const float vn = fmaf(dvdt + du, dt, vc);
            Vn[g] = vn;
            if (det && sg.flag[t]) grid_detect(gd, ck, k, vc, vn, dvdt);
            const bool bad = !(vn == vn) || vn < gd.vmin_ok || vn > gd.vmax_ok;
            if (bad) atomicAdd(gd.nbad, 1ull);
        }
        __syncthreads();   // every thread is done with stage s
        if (t == 0 && tile + 2 * stride < ntiles) {
            tc::fence_proxy_async();
            sub_issue(stg[s], &bar[s], gd, (tile + 2 * stride) * kSubTile, det);
        }
    }
}

namespace {

// One stage of the V-halo kernel: the tile's streamed rows, each voxel's index
// in the tile's V box, the box itself and the tile's box header.
struct __align__(16) VStage {
    SubStage rows;
    int32_t li[kSubTile];
    float vb[kVBoxFloats];
    int32_t hdr[8];
};
static_assert(offsetof(VStage, li) % 16 == 0 && offsetof(VStage, vb) % 16 == 0 && sizeof(VStage) % 16 == 0,
              "bulk copies need 16-byte aligned destinations");
// The rows-only stage of the same pipeline (no V box).
struct __align__(16) RStage {
    SubStage rows;
    int32_t hdr[8];
};
template <bool BOX> struct StageOf { using T = VStage; };
template <> struct StageOf<false> { using T = RStage; };

struct VHdr {
    int32_t ok, zlo, xlo, ylo, bx, by, bz;
};

__device__ __forceinline__ VHdr vhdr_load(const int32_t *h)
{
    const int4 a = __ldg(reinterpret_cast<const int4 *>(h)), b = __ldg(reinterpret_cast<const int4 *>(h) + 1);
    return VHdr{a.x, a.y, a.z, a.w, b.x, b.y, b.z};
}

// The producer warp's share of the copies of tile k0 / kSubTile into one
// stage: lane 0 first writes the header and arms the stage's mbarrier with
// the byte count, then the lanes issue the copies in parallel -- the 6 row
// copies (rate, index, tensor row, control, detector flag, box index; 5
// without the box) and, when the box fits, one per box column.  A box column is the
// z-segment [zlo, zlo + bz) of grid column (xlo + i, ylo + j), copied whole:
// nz, zlo and bz are multiples of 4, so every source and destination is
// 16-byte aligned and every size a multiple of 16 bytes; the host builder
// keeps every segment inside its column and every column inside the grid.
template <bool BOX>
__device__ __forceinline__ void vbox_issue(typename StageOf<BOX>::T &st, uint64_t *bar, const GridDev<float> &gd,
                                           const float *V, int64_t k0, bool det, const VHdr &h, int lane, int64_t ny,
                                           int64_t nz)
{
    constexpr uint32_t n = kSubTile;
    const int ncol = (BOX && h.ok) ? h.bx * h.by : 0;
    if (lane == 0) {
        st.hdr[0] = BOX ? h.ok : 0;
        st.hdr[1] = h.by * h.bz;
        st.hdr[2] = h.bz;
        const uint32_t box = (uint32_t)ncol * (uint32_t)h.bz * 4u;
        tc::mbar_expect_tx(bar, n * (4 + 4 + 12 + 1) + (det ? n : 0) + (BOX ? n * 4 : 0) + box);
    }
    __syncwarp();
    for (int c = lane; c < (BOX ? 6 : 5) + ncol; c += 32) {
        switch (c) {
        case 0: tc::bulk_g2s(st.rows.rate, gd.srate + k0, n * 4, bar); break;
        case 1: tc::bulk_g2s(st.rows.gidx, gd.gidx + k0, n * 4, bar); break;
        case 2: tc::bulk_g2s(st.rows.t3, gd.t3h + 3 * k0, n * 12, bar); break;
        case 3: tc::bulk_g2s(st.rows.ctl, gd.ctl + k0, n, bar); break;
        case 4: if (det) tc::bulk_g2s(st.rows.flag, gd.sdflag + k0, n, bar); break;
        default:
            if constexpr (BOX) {
                if (c == 5) {
                    tc::bulk_g2s(st.li, gd.vli + k0, n * 4, bar);
                } else {
                    const int col = c - 6, i = col / h.by, j = col - i * h.by;
                    tc::bulk_g2s(st.vb + col * h.bz, V + ((int64_t)(h.xlo + i) * ny + (h.ylo + j)) * nz + h.zlo,
                                 (uint32_t)h.bz * 4u, bar);
                }
            }
        }
    }
}

// The producer warp: fills a stage as soon as the consumer warps have released
// it (mbarrier `empty`) and arms `full` with the stage's byte count.  A wait
// that runs out stops the issuing; before it returns, the copies it issued
// have landed (bounded).
template <bool BOX>
__device__ __forceinline__ void sub_produce(typename StageOf<BOX>::T *stg, uint64_t *full, uint64_t *empty,
                                            const GridDev<float> &gd, const float *V, int64_t ntiles, uint32_t lim, int lane)
{
    const bool det = gd.det != nullptr;
    const int64_t ny = BOX ? gd.sx / gd.sy : 0, nz = BOX ? gd.sy : 0;
    const bool skip0 = gd.sub_skip_copy != 0;   // failure-path test: tile 0's stage is never filled
    uint32_t issued = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++issued) {
        const int s = issued & 1;
        // the whole warp takes one decision (vbox_issue synchronises the warp)
        const bool free = issued < 2 || tc::mbar_wait(&empty[s], ((issued - 2) >> 1) & 1, lim);
        if (!__all_sync(0xffffffffu, free)) {
            if (lane == 0) atomicOr(gd.serr, 2);
            break;
        }
        if (issued == 0 && skip0) continue;
        tc::fence_proxy_async();
        const VHdr h = BOX ? vhdr_load(gd.vbox_hdr + 8 * tile) : VHdr{};
        vbox_issue<BOX>(stg[s], &full[s], gd, V, tile * kSubTile, det, h, lane, ny, nz);
    }
    // the copies of the last two stages have landed before the CTA ends
    for (uint32_t j = issued > 2 ? issued - 2 : 0; j < issued; ++j)
        if (j > 0 || !skip0) tc::mbar_wait(&full[j & 1], (j >> 1) & 1, kSubWaitLimit);
}

// Barriers of a CTA's two stages, for `warps` consumer warps.
__device__ __forceinline__ void sub_barriers(uint64_t *full, uint64_t *empty, int warps)
{
    if (threadIdx.x == 0) {
        tc::mbar_init(&full[0], 1);
        tc::mbar_init(&full[1], 1);
        tc::mbar_init(&empty[0], warps);
        tc::mbar_init(&empty[1], warps);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}

// The rest of a voxel's substep where a stimulus can act or the detector runs.
__device__ __forceinline__ float sub_special(const GridDev<float> &gd, const Clock &ck, uint32_t k, uint32_t ctl,
                                             uint32_t fl, float r, float du, float vc, float kdt)
{
    const float dvdt = r - grid_stim(gd, ck, (uint8_t)ctl, (int64_t)k);
    const float vn = fmaf(dvdt + du, kdt, vc);
    if (fl) grid_detect(gd, ck, (int64_t)k, vc, vn, dvdt);
    return vn;
}

}  // namespace

// 3D V-only substep with the V halo staged.  Persistent CTAs of 8 consumer
// warps (one voxel per thread of a 256-voxel tile) and one producer warp, two
// stages: each stage holds a tile's streamed rows and the box of the dense V
// grid its stencils reach.  The consumers wait on `full`, read the 19-point
// stencil from shared memory and release the stage -- no CTA-wide barrier per
// tile.  A tile whose box exceeds the stage reads V from the grid.  Arithmetic
// identical to k_sur_substep.  Every wait is bounded: a consumer warp whose
// wait runs out sets bit 1 of *serr and ends its loop.
template <int MINB>
__global__ void __launch_bounds__(kSubTile + 32, MINB) k_sur_substep_vbox(GridDev<float> gd, float kdt, int cur)
{
    extern __shared__ __align__(128) uint8_t vsm[];
    VStage *stg = reinterpret_cast<VStage *>(vsm);
    __shared__ __align__(8) uint64_t full[2], empty[2];
    const int t = threadIdx.x;
    const int64_t ntiles = (gd.ntissue + kSubTile - 1) / kSubTile;
    if (blockIdx.x >= ntiles) return;
    const uint32_t lim = gd.sub_wait_limit ? gd.sub_wait_limit : kSubWaitLimit;
    const float *__restrict__ V = gd.vg[cur];
    sub_barriers(full, empty, kSubTile / 32);
    if (t >= kSubTile) {
        sub_produce<true>(stg, full, empty, gd, V, ntiles, lim, t - kSubTile);
        return;
    }
    float *__restrict__ Vn = gd.vg[cur ^ 1];
    const Clock ck = gd.clk[cur];
    const uint32_t smask = stim_mask(gd, ck), dmask = gd.det ? 0xffu : 0u;
    const uint32_t sx4 = (uint32_t)gd.sx * 4u, sy4 = (uint32_t)gd.sy * 4u, n = (uint32_t)gd.ntissue;
    uint32_t it = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
        const int s = it & 1;
        const bool ok = tc::mbar_wait(&full[s], (it >> 1) & 1, lim);
        if (!__all_sync(0xffffffffu, ok)) {
            if ((t & 31) == 0) atomicOr(gd.serr, 2);
            break;
        }
        const VStage &st = stg[s];
        const SubStage &sg = st.rows;
        const uint32_t k = (uint32_t)tile * kSubTile + t;
        const float r = sg.rate[t];
        if (k < n && r == r) {
            const uint32_t o = (uint32_t)sg.gidx[t] * 4u;       // byte offset in the grid
            float2 q[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) q[i] = __half22float2(sg.t3[3 * t + i]);
            float Dt[6], Bt[3];
            sub_tensor_unpack<3>(q, gd.sub_dtr, gd.sub_dsg, Dt, Bt);
            float vc, du;
            if (st.hdr[0]) {
                const int64_t li = st.li[t];
                vc = st.vb[li];
                du = sub_du_at<3>(gd, st.vb, li, st.hdr[1], st.hdr[2], vc, Dt, Bt);
            } else {
                vc = *reinterpret_cast<const float *>(reinterpret_cast<const char *>(V) + o);
                du = sub_du_32<3>(gd, V, o, sx4, sy4, vc, Dt, Bt);
            }
            const uint32_t ctl = sg.ctl[t], fl = sg.flag[t] & dmask;
            float vn = fmaf(r + du, kdt, vc);
            if ((ctl & smask) | fl) vn = sub_special(gd, ck, k, ctl, fl, r, du, vc, kdt);
            *reinterpret_cast<float *>(reinterpret_cast<char *>(Vn) + o) = vn;
            if (!(vn >= gd.vmin_ok && vn <= gd.vmax_ok)) atomicAdd(gd.nbad, 1ull);
        }
        __syncwarp();
        if ((t & 31) == 0) tc::mbar_arrive(&empty[s]);   // this warp is done with stage s
    }
}

// What a pair kernel's thread keeps across its voxels.
struct PairConst {
    Clock ck;
    uint32_t smask, dmask, sx4, sy4, n;
    float kdt;
};
__device__ __forceinline__ PairConst pair_const(const GridDev<float> &gd, float kdt, int cur)
{
    PairConst p;
    p.ck = gd.clk[cur];
    p.smask = stim_mask(gd, p.ck);
    p.dmask = gd.det ? 0xffu : 0u;
    p.sx4 = (uint32_t)gd.sx * 4u;
    p.sy4 = (uint32_t)gd.sy * 4u;
    p.n = (uint32_t)gd.ntissue;
    p.kdt = kdt;
    return p;
}

// The substep of two voxels (ka, kb; rows ta, tb of staged arrays) in packed
// FP32 arithmetic: a pair shares every FP32 instruction, the waits and the
// loop (one voxel per thread took 234 instructions a warp of voxels, which was
// what bounded it; this takes 171).  Each value is rounded as in k_sur_substep.
// 7.5 million voxels 73 -> 66 us, 1.1 million 15.1 -> 12.7 us.  What bounds it
// now: the V gather, whose 25 bytes a voxel come through the L2 (L1 hit rate
// 75%), beside 22 bytes of rows; 226 MB from HBM would take 34 us.  More rows
// in flight (3 and 4 stages) and V prefetched into the L2 changed nothing.
template <int DIM>
__device__ __forceinline__ void sub_pair(const GridDev<float> &gd, const PairConst &pc, int cur, uint32_t ka, uint32_t kb,
                                         int ta, int tb, const float *rate, const int32_t *gidx, const __half2 *t3,
                                         const uint8_t *ctl, const uint8_t *flag)
{
    const float ra = rate[ta], rb = rate[tb];
    const bool ona = ka < pc.n && ra == ra, onb = kb < pc.n && rb == rb;
    if (!(ona || onb)) return;
    const char *__restrict__ Vb = reinterpret_cast<const char *>(gd.vg[cur]);
    char *__restrict__ Vn = reinterpret_cast<char *>(gd.vg[cur ^ 1]);
    const uint32_t sx4 = pc.sx4, sy4 = pc.sy4, smask = pc.smask, dmask = pc.dmask;
    const float kdt = pc.kdt;
    auto dup = [](float x) { return tc::pair2(x, x); };
    const uint64_t m1 = dup(-1.f), m2 = dup(-2.f), c2 = dup(gd.inv_dx2), c4 = dup(gd.inv_4dx2), c1 = dup(gd.inv_2dx);
    const uint64_t dtr = dup(gd.sub_dtr), dsg = dup(gd.sub_dsg), kdt2 = dup(kdt);
    // a voxel that takes no part reads the other one's neighbours
    const uint32_t ga = (uint32_t)gidx[ona ? ta : tb] * 4u, gb = (uint32_t)gidx[onb ? tb : ta] * 4u;
    uint64_t q[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float2 a = __half22float2(t3[3 * ta + i]), b = __half22float2(t3[3 * tb + i]);
        q[2 * i] = tc::pair2(a.x, b.x);
        q[2 * i + 1] = tc::pair2(a.y, b.y);
    }
    // V of both voxels' neighbour i, j, l
    auto at = [&](int i, int j, int l) {
        const uint32_t d = (uint32_t)i * sx4 + (uint32_t)j * sy4;
        return tc::pair2(*reinterpret_cast<const float *>(Vb + (ga + d) + 4 * l),
                         *reinterpret_cast<const float *>(Vb + (gb + d) + 4 * l));
    };
    auto sub2 = [&](uint64_t x, uint64_t y) { return tc::fma2(m1, y, x); };
    // (xp + xm - 2 vc) / dx^2 and (pp + mm - mp - pm) / 4 dx^2
    const uint64_t vc = at(0, 0, 0);
    auto second = [&](uint64_t xp, uint64_t xm) { return tc::mul2(tc::fma2(m2, vc, tc::add2(xp, xm)), c2); };
    auto mixed = [&](uint64_t pp, uint64_t mm, uint64_t mp, uint64_t pm) {
        return tc::mul2(sub2(sub2(tc::add2(pp, mm), mp), pm), c4);
    };
    const uint64_t vxp = at(1, 0, 0), vxm = at(-1, 0, 0), vyp = at(0, 1, 0), vym = at(0, -1, 0);
    const uint64_t lxx = second(vxp, vxm), lyy = second(vyp, vym);
    const uint64_t lxy = mixed(at(1, 1, 0), at(-1, -1, 0), at(-1, 1, 0), at(1, -1, 0));
    const uint64_t s0 = tc::mul2(dsg, q[0]), s1 = tc::mul2(dsg, q[1]);
    const uint64_t D0 = tc::fma2(s0, q[0], dtr), D1 = tc::fma2(s1, q[1], dtr), D3 = tc::mul2(s0, q[1]);
    uint64_t du = tc::fma2(D0, lxx, tc::fma2(D1, lyy, tc::mul2(tc::add2(D3, D3), lxy)));
    du = tc::fma2(q[3], tc::mul2(sub2(vxp, vxm), c1), tc::fma2(q[4], tc::mul2(sub2(vyp, vym), c1), du));
    if constexpr (DIM == 3) {
        const uint64_t s2 = tc::mul2(dsg, q[2]);
        const uint64_t D2 = tc::fma2(s2, q[2], dtr), D4 = tc::mul2(s0, q[2]), D5 = tc::mul2(s1, q[2]);
        const uint64_t vzp = at(0, 0, 1), vzm = at(0, 0, -1);
        const uint64_t lzz = second(vzp, vzm);
        const uint64_t lxz = mixed(at(1, 0, 1), at(-1, 0, -1), at(-1, 0, 1), at(1, 0, -1));
        const uint64_t lyz = mixed(at(0, 1, 1), at(0, -1, -1), at(0, -1, 1), at(0, 1, -1));
        const uint64_t dz = tc::fma2(q[5], tc::mul2(sub2(vzp, vzm), c1), du);
        const uint64_t m = tc::fma2(D4, lxz, tc::mul2(D5, lyz));
        du = tc::fma2(D2, lzz, tc::fma2(dup(2.f), m, dz));
    }
    float va, vb;
    tc::split2(tc::fma2(tc::add2(tc::pair2(ra, rb), du), kdt2, vc), va, vb);
    const uint32_t ca = ctl[ta], cb = ctl[tb], fa = flag[ta] & dmask, fb = flag[tb] & dmask;
    if (((ca | cb) & smask) | fa | fb) {
        float dua, dub, vca, vcb;
        tc::split2(du, dua, dub);
        tc::split2(vc, vca, vcb);
        if (ona && ((ca & smask) | fa)) va = sub_special(gd, pc.ck, ka, ca, fa, ra, dua, vca, kdt);
        if (onb && ((cb & smask) | fb)) vb = sub_special(gd, pc.ck, kb, cb, fb, rb, dub, vcb, kdt);
    }
    if (ona) {
        *reinterpret_cast<float *>(Vn + ga) = va;
        if (!(va >= gd.vmin_ok && va <= gd.vmax_ok)) atomicAdd(gd.nbad, 1ull);
    }
    if (onb) {
        *reinterpret_cast<float *>(Vn + gb) = vb;
        if (!(vb >= gd.vmin_ok && vb <= gd.vmax_ok)) atomicAdd(gd.nbad, 1ull);
    }
}

// The rows-only pipeline of a producer warp with V from the grid (2D and 3D),
// two voxels per thread (rows t and t + 128 of a tile).
constexpr int kPairThreads = kSubTile / 2;
template <int DIM, int MINB>
__global__ void __launch_bounds__(kPairThreads + 32, MINB) k_sur_substep_pair(GridDev<float> gd, float kdt, int cur)
{
    __shared__ RStage stg[2];
    __shared__ __align__(8) uint64_t full[2], empty[2];
    const int t = threadIdx.x;
    const int64_t ntiles = (gd.ntissue + kSubTile - 1) / kSubTile;
    if (blockIdx.x >= ntiles) return;
    const uint32_t lim = gd.sub_wait_limit ? gd.sub_wait_limit : kSubWaitLimit;
    sub_barriers(full, empty, kPairThreads / 32);
    if (t >= kPairThreads) {
        sub_produce<false>(stg, full, empty, gd, gd.vg[cur], ntiles, lim, t - kPairThreads);
        return;
    }
    const PairConst pc = pair_const(gd, kdt, cur);
    uint32_t it = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
        const int s = it & 1;
        const bool ok = tc::mbar_wait(&full[s], (it >> 1) & 1, lim);
        if (!__all_sync(0xffffffffu, ok)) {
            if ((t & 31) == 0) atomicOr(gd.serr, 2);
            break;
        }
        const SubStage &sg = stg[s].rows;
        const uint32_t k = (uint32_t)tile * kSubTile + t;
        sub_pair<DIM>(gd, pc, cur, k, k + kPairThreads, t, t + kPairThreads, sg.rate, sg.gidx, sg.t3, sg.ctl, sg.flag);
        __syncwarp();
        if ((t & 31) == 0) tc::mbar_arrive(&empty[s]);   // this warp is done with stage s
    }
}

// Every warp on its own: units of 64 voxels (lane and lane + 32), rows copied
// one unit ahead by the warp itself (16 bytes a lane and copy), no barrier, no
// producer warp whose registers would cost a fifth of the consumers.  Faster
// while the grid lives in the L2 (1.1 million voxels 12.7 us against 14.7 for
// k_sur_substep_pair), slower beyond it (7.5 million: 70 against 66).
constexpr int kUnit = 64;
struct __align__(16) WStage {
    float rate[kUnit];
    int32_t gidx[kUnit];
    __half2 t3[kUnit * 3];
    uint8_t ctl[kUnit];
    uint8_t flag[kUnit];
};
static_assert(offsetof(WStage, gidx) == 256 && offsetof(WStage, t3) == 512 && offsetof(WStage, ctl) == 1280 &&
                  offsetof(WStage, flag) == 1344 && sizeof(WStage) == 1408,
              "the copies below address the stage in 16-byte chunks");
template <int DIM, int MINB>
__global__ void __launch_bounds__(128, MINB) k_sur_substep_warp(GridDev<float> gd, float kdt, int cur)
{
    __shared__ WStage stg[4][2];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t units = (uint32_t)((gd.ntissue + kUnit - 1) / kUnit), stride = gridDim.x * 4;
    uint32_t u = blockIdx.x * 4 + w;
    if (u >= units) return;
    const PairConst pc = pair_const(gd, kdt, cur);
    // chunk sources of this lane: rate | index; tensor; tensor, control, flag
    const char *p0 = lane < 16 ? reinterpret_cast<const char *>(gd.srate) + 16 * lane
                               : reinterpret_cast<const char *>(gd.gidx) + 16 * (lane - 16);
    const char *p1 = reinterpret_cast<const char *>(gd.t3h) + 16 * lane;
    const char *p2 = lane < 16 ? p1 + 512
                   : lane < 20 ? reinterpret_cast<const char *>(gd.ctl) + 16 * (lane - 16)
                               : reinterpret_cast<const char *>(gd.sdflag) + 16 * (lane - 20);
    const uint32_t m2 = lane < 16 ? 12u * kUnit : (uint32_t)kUnit;
    const bool has2 = lane < 20 || (lane < 24 && gd.det);
    auto fetch = [&](int s, uint32_t unit) {
        const uint32_t d = (uint32_t)__cvta_generic_to_shared(&stg[w][s]) + 16u * lane;
        auto cp = [](uint32_t dst, const char *src) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
        };
        cp(d, p0 + (uint64_t)unit * (4u * kUnit));
        cp(d + 512, p1 + (uint64_t)unit * (12u * kUnit));
        if (has2) cp(d + 1024, p2 + (uint64_t)unit * m2);
    };
    fetch(0, u);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int s = 0; u < units; u += stride, s ^= 1) {
        if (u + stride < units) fetch(s ^ 1, u + stride);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const WStage &sg = stg[w][s];
        const uint32_t k = u * kUnit + lane;
        sub_pair<DIM>(gd, pc, cur, k, k + 32, lane, lane + 32, sg.rate, sg.gidx, sg.t3, sg.ctl, sg.flag);
        __syncwarp();                      // the stage is read before the next copies into it
    }
}

// What follows the substep in a step inside a macro step, in one launch: the
// plain step of the listed voxels, which write their mirror voxels themselves
// (the first nlist blocks), and the mirror voxels of all other sources and the
// clock (the rest).  For grids whose mirror voxels are one wave of blocks
// (kMergeBndPerSM): there the two launches, whose blocks mostly find little to
// do, took as long as the substep.
template <int DIM> __global__ void __launch_bounds__(256, 2) k_list_ghost(GridDev<float> gd, StepT<float> kst, int cur, int nlist)
{
    if ((int)blockIdx.x < nlist) {
        const int64_t n = *gd.plist_n;
        int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
        if (i >= n) return;
        const Clock ck = gd.clk[cur];
        for (; i < n; i += (int64_t)nlist * blockDim.x)
            grid_step_voxel_call<float, DIM, true>(gd, kst, cur, gd.plist[i], ck);
        return;
    }
    const int64_t j = ((int64_t)blockIdx.x - nlist) * blockDim.x + threadIdx.x;
    if (j == 0) advance_clock(gd, cur);
    float *V = gd.vg[cur ^ 1];
    // four entries a thread, their loads in flight together
    int32_t src[4], dst[4], k[4];
    if (4 * j + 3 < gd.nbnd) {
        *reinterpret_cast<int4 *>(src) = reinterpret_cast<const int4 *>(gd.bnd_src)[j];
        *reinterpret_cast<int4 *>(dst) = reinterpret_cast<const int4 *>(gd.bnd_dst)[j];
        *reinterpret_cast<int4 *>(k) = reinterpret_cast<const int4 *>(gd.bnd_k)[j];
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool on = 4 * j + i < gd.nbnd;
            src[i] = on ? gd.bnd_src[4 * j + i] : 0;
            dst[i] = on ? gd.bnd_dst[4 * j + i] : 0;
            k[i] = on ? gd.bnd_k[4 * j + i] : -1;
        }
    }
    // (k < 0: no entry, or one without a tissue source, which has nothing to copy)
    float r[4], v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        r[i] = k[i] >= 0 ? gd.srate[k[i]] : __int_as_float(0x7fc00000);
        v[i] = k[i] >= 0 ? V[src[i]] : 0.f;        // (not used where the list steps the source)
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (r[i] == r[i]) V[dst[i]] = v[i];
}

cudaError_t launch_list_ghost(const GridDev<float> &gd, const StepK &k, int cur, int dim, cudaStream_t st)
{
    const unsigned nl = grid_list_blocks(gd.ntissue), ng = (unsigned)((gd.nbnd + 1023) / 1024 + (gd.nbnd == 0));
    const StepT<float> kk = step_as<float>(k);
    if (dim == 1) k_list_ghost<1><<<nl + ng, 256, 0, st>>>(gd, kk, cur, (int)nl);
    else if (dim == 2) k_list_ghost<2><<<nl + ng, 256, 0, st>>>(gd, kk, cur, (int)nl);
    else k_list_ghost<3><<<nl + ng, 256, 0, st>>>(gd, kk, cur, (int)nl);
    return cudaGetLastError();
}

// A whole step inside a surrogate macro step on a small grid, in one launch:
// the V-only step of the surrogate voxels, the plain step of the others, the
// mirror voxels and (block 0) the clock.  There the time of a step is its
// launches: with three of them 20 steps of a 200 x 200 sheet, V read back after
// each, took 0.46 ms, with one 0.37 ms.
template <int DIM> __global__ void __launch_bounds__(64, 4) k_sur_step_small(GridDev<float> gd, StepT<float> kst, int cur)
{
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) advance_clock(gd, cur);
        return;
    }
    const int64_t k = (blockIdx.x - 1) * (int64_t)blockDim.x + threadIdx.x;
    if (k >= gd.ntissue) return;
    const float r = gd.srate[k];
    if (!(r == r)) {
        grid_step_voxel<float, DIM, true>(gd, kst, cur, k, gd.clk[cur]);
        return;
    }
    const int64_t g = DIM == 1 ? k : (int64_t)gd.gidx[k];
    const uint8_t ctl = gd.ctl[k], fl = gd.det ? gd.sdflag[k] : 0;
    float Dt[6] = {}, Bt[3] = {};
    if (DIM > 1 && gd.d6 && gd.t3h) {
        float2 q[3];
        sub_tensor_f16(gd.t3h + 3 * k, q);
        sub_tensor_unpack<DIM>(q, gd.sub_dtr, gd.sub_dsg, Dt, Bt);
    }
    const Clock ck = gd.clk[cur];
    const float *__restrict__ V = gd.vg[cur];
    const float vc = V[g];
    const int32_t gref = ghost_ref(gd, k, ctl);
    const float du = sub_du<DIM>(gd, V, g, k, vc, Dt, Bt);
    const float ist = grid_stim(gd, ck, ctl, k);
    const float dvdt = r - ist;
    const float vn = fmaf(dvdt + du, kst.dt, vc);
    put_v(gd, gd.vg[cur ^ 1], g, ctl, gref, vn);
    if (fl) grid_detect(gd, ck, k, vc, vn, dvdt);
    if (!(vn == vn) || vn < gd.vmin_ok || vn > gd.vmax_ok) atomicAdd(gd.nbad, 1ull);
}

cudaError_t launch_sur_step_small(const GridDev<float> &gd, const StepK &k, int cur, int dim, cudaStream_t st)
{
    if (dim >= 2 && gd.d6 && !gd.t3h) return cudaErrorInvalidValue;   // FP16 tensor rows missing
    const unsigned nb = (unsigned)((gd.ntissue + 63) / 64 + 1);
    const StepT<float> kk = step_as<float>(k);
    if (dim == 1) k_sur_step_small<1><<<nb, 64, 0, st>>>(gd, kk, cur);
    else if (dim == 2) k_sur_step_small<2><<<nb, 64, 0, st>>>(gd, kk, cur);
    else k_sur_step_small<3><<<nb, 64, 0, st>>>(gd, kk, cur);
    return cudaGetLastError();
}

namespace {

template <int MINB> void launch_minb(const GridDev<float> &gd, double dt, int cur, int dim, unsigned nb, cudaStream_t st)
{
    if (dim == 1) k_sur_substep<1, MINB><<<nb, 256, 0, st>>>(gd, (float)dt, cur);
    else if (dim == 2) k_sur_substep<2, MINB><<<nb, 256, 0, st>>>(gd, (float)dt, cur);
    else k_sur_substep<3, MINB><<<nb, 256, 0, st>>>(gd, (float)dt, cur);
}

// The kernel's shared-memory carve-out at its maximum, once per device, so
// that MINB CTAs of two stages each fit on an SM.
template <typename K> cudaError_t carveout_once(K kernel, std::atomic<uint64_t> &done)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? (1ull << dev) : 0;
    if (bit && (done.load() & bit)) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e == cudaSuccess && bit) done.fetch_or(bit);
    return e;
}

template <int DIM, int MINB> cudaError_t launch_tile(const GridDev<float> &gd, double dt, int cur, cudaStream_t st)
{
    static std::atomic<uint64_t> done{0};
    cudaError_t e = carveout_once(k_sur_substep_tile<DIM, MINB>, done);
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int64_t ntiles = (gd.ntissue + kSubTile - 1) / kSubTile;
    const int64_t grid = ntiles < (int64_t)nsm * MINB ? ntiles : (int64_t)nsm * MINB;
    k_sur_substep_tile<DIM, MINB><<<(unsigned)grid, kSubTile, 0, st>>>(gd, (float)dt, cur);
    return cudaGetLastError();
}

int num_sms()
{
    int dev = 0, nsm = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}

template <int MINB> cudaError_t launch_vbox(const GridDev<float> &gd, double dt, int cur, cudaStream_t st)
{
    static std::atomic<uint64_t> done{0}, carve{0};
    const uint32_t bytes = 2 * sizeof(VStage);
    cudaError_t e = tc::smem_attr_once(k_sur_substep_vbox<MINB>, bytes, done);
    if (e == cudaSuccess) e = carveout_once(k_sur_substep_vbox<MINB>, carve);
    if (e != cudaSuccess) return e;
    const int64_t ntiles = (gd.ntissue + kSubTile - 1) / kSubTile, cap = (int64_t)num_sms() * MINB;
    k_sur_substep_vbox<MINB><<<(unsigned)(ntiles < cap ? ntiles : cap), kSubTile + 32, bytes, st>>>(gd, (float)dt, cur);
    return cudaGetLastError();
}

template <int DIM, int MINB> cudaError_t launch_pair(const GridDev<float> &gd, double dt, int cur, cudaStream_t st)
{
    static std::atomic<uint64_t> carve{0};
    cudaError_t e = carveout_once(k_sur_substep_pair<DIM, MINB>, carve);
    if (e != cudaSuccess) return e;
    const int64_t ntiles = (gd.ntissue + kSubTile - 1) / kSubTile, cap = (int64_t)num_sms() * MINB;
    k_sur_substep_pair<DIM, MINB><<<(unsigned)(ntiles < cap ? ntiles : cap), kPairThreads + 32, 0, st>>>(gd, (float)dt, cur);
    return cudaGetLastError();
}

template <int DIM, int MINB> cudaError_t launch_warp(const GridDev<float> &gd, double dt, int cur, cudaStream_t st)
{
    static std::atomic<uint64_t> carve{0};
    cudaError_t e = carveout_once(k_sur_substep_warp<DIM, MINB>, carve);
    if (e != cudaSuccess) return e;
    const int64_t need = (gd.ntissue + 4 * kUnit - 1) / (4 * kUnit), cap = (int64_t)num_sms() * MINB;
    k_sur_substep_warp<DIM, MINB><<<(unsigned)(need < cap ? need : cap), 128, 0, st>>>(gd, (float)dt, cur);
    return cudaGetLastError();
}

bool al16(const void *p) { return p && ((uintptr_t)p & 15u) == 0; }

}  // namespace

cudaError_t launch_sur_substep(const GridDev<float> &gd, double dt, int cur, int dim, int variant, cudaStream_t st)
{
    if (gd.ntissue <= 0) return cudaSuccess;
    const bool rows_ok = dim >= 2 && gd.d6 && al16(gd.t3h) && al16(gd.srate) && al16(gd.gidx) &&
                         al16(gd.ctl) && gd.serr && (!gd.det || al16(gd.sdflag));
    // (those two families address the grid in 32-bit bytes)
    const bool bytes32 = gd.ngrid < (int64_t)1 << 30;
    if (variant >= 200 && !bytes32) variant = 105;
    if (variant >= 300) {
        // rows staged by a producer warp, V from the grid, two voxels a thread (2D/3D)
        if (rows_ok) {
            if (dim == 2) {
                if (variant == 306) return launch_warp<2, 10>(gd, dt, cur, st);
                if (variant == 305) return launch_warp<2, 8>(gd, dt, cur, st);
                return launch_pair<2, 6>(gd, dt, cur, st);
            }
            if (variant == 306) return launch_warp<3, 8>(gd, dt, cur, st);
            if (variant == 305) return launch_warp<3, 6>(gd, dt, cur, st);
            return launch_pair<3, 5>(gd, dt, cur, st);
        }
        variant = 105;
    } else if (variant >= 200) {
        if (dim == 3 && rows_ok && gd.vbox_hdr && gd.vli && al16(gd.vli) && al16(gd.vg[0]) && al16(gd.vg[1]))
            return variant == 203 ? launch_vbox<3>(gd, dt, cur, st) : launch_vbox<4>(gd, dt, cur, st);
        variant = 105;
    }
    const bool tile = variant >= 100;
    const int minb = tile ? variant - 100 : variant;
    if (dim >= 2 && gd.d6 && !gd.t3h) return cudaErrorInvalidValue;   // FP16 tensor rows missing
    if (tile && dim >= 2 && gd.d6 && al16(gd.t3h) && al16(gd.srate) && al16(gd.gidx) &&
        al16(gd.ctl) && gd.serr && (!gd.det || al16(gd.sdflag))) {
        if (dim == 2) {
            if (minb == 8) return launch_tile<2, 8>(gd, dt, cur, st);
            if (minb == 6) return launch_tile<2, 6>(gd, dt, cur, st);
            return launch_tile<2, 5>(gd, dt, cur, st);
        }
        if (minb == 8) return launch_tile<3, 8>(gd, dt, cur, st);
        if (minb == 6) return launch_tile<3, 6>(gd, dt, cur, st);
        return launch_tile<3, 5>(gd, dt, cur, st);
    }
    const unsigned nb = (unsigned)((gd.ntissue + 256 * kSubU - 1) / (256 * kSubU));
    if (minb == 8) launch_minb<8>(gd, dt, cur, dim, nb, st);
    else if (minb == 6) launch_minb<6>(gd, dt, cur, dim, nb, st);
    else launch_minb<5>(gd, dt, cur, dim, nb, st);
    return cudaGetLastError();
}

}  // namespace lqt
