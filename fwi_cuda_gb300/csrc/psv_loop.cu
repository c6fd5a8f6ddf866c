// psv_loop.cu -- many time steps of the FP32 time loop in one launch.
//
// The two-launch families move v and sigma through HBM twice per step and
// pay a kernel boundary per half-step.  Here a launch runs up to hundreds of
// steps.  The work is a list of items, one per (step, half-step, tile of 64
// columns x TZ rows, shot), and a CTA claims the next item of the list with
// an atomic counter.  An item waits until its own tile and the four beside it
// have finished the half-step before (one progress word per tile), which is
// all a staggered stencil needs, in place: the neighbours have then read what
// the item overwrites and written what it reads.  There is no grid barrier
// and no assumption about which CTAs are resident: an item depends on earlier
// items of the list only, these are held by running CTAs, and a CTA works its
// items in order, so the earliest unfinished item can always run.
//
// Order of the list (List): shots fastest, then columns, then bands of tiles;
// velocity tiles follow the stress tiles a few bands behind, so they find v
// and sigma in L2 and the wavefields cross HBM once per step instead of twice.
//
// A CTA is warp-specialised:
//   claimer (1 warp): claims items ahead and works out what they need.
//   keepers (1 warp per stage of the shared-memory ring): wait for the item's
//           progress words and fill the stage by TMA; once it is computed,
//           inject the tile's sources and record its receivers in the stage,
//           store the tile by TMA, start the next item's loads and publish
//           the tile's progress.  The next item's words are polled and the
//           fences paid while the current one is loaded and computed.
//           Adjacent planes go in one 3-D box (v: 2, sigma: 3): a box costs
//           its issuing thread about 150 ns whatever its size, measured.
//   team    (TZ / 2 warps): computes the stages in turn, four columns of one
//           row per thread with 128-bit shared-memory accesses; new values
//           overwrite the old ones in the stage.
// Nobody meets at a block barrier inside the loop.
//
// Memory order: a tile's values are written by the async proxy (TMA store)
// and read by it (TMA load): the keeper publishes after the store's completion,
// with release at gpu scope, and fences between its acquire and its loads, for
// the scope and for the proxy.  What the team writes directly
// (CPML memories, snapshots, shot gradients) belongs to one tile and reaches
// its next visitor through the same release / acquire chain; these are read
// past L1 (ld.global.cg).
//
// What bounds it: on grids beyond L2, DRAM and the shared-memory pipe (1001 x
// 2001, order 8, eight shots: 48 B a point and step cross DRAM in modelling, 66
// in storing passes, 104 in the adjoint, against 61, 76 and 99 for two launches;
// DRAM 55, 63 and 75 % busy, the pipe 58, 50 and 38 %); below, the latency from
// claim to publication against the items a half-step has.  us a step, forward /
// adjoint, two launches before -> loop (TZ = 16):
//   1001 x 2001 x 8, order 8   251 / 310 -> 214 / 284
//   1001 x 2001 x 3, order 8   modelling 145 (direct) -> 64
//   601 x 1203 x 4, order 8    61 / 68 (direct, two chains) -> 36 / 50
//   301 x 601 x 8, order 4     23.3 / 24.4 (direct, two chains) -> 17.8 / 22.5
// Tried and slower: one row of warps per stage doing the keeper's work; two
// rows per thread (20 % less shared-memory traffic, 3 x the time of a tile:
// longer code run by fewer warps); two teams a CTA; four CTAs per SM at 64
// registers; every plane of a tile by TMA (two stages instead of three);
// claiming further ahead on grids inside L2 (18.7 -> 17.5 us a step without).
//
// Every wait is bounded: after two seconds it records error code 1 in
// StepParams::err and the CTA winds down; the host turns that into
// PSV_ERR_CUDA.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "psv_kernels_impl.cuh"
#include "psv_plan.cuh"
#include "psv_quads.cuh"
#include "psv_tma.cuh"

namespace psv {

namespace {

constexpr int TW = 64;           // tile columns
constexpr int SW = TW + 2 * HX;  // staged row length (floats)
constexpr unsigned ALL = 0xffffffffu;
// Words between two tiles' progress words: a 32-byte sector each.  Packed, the
// polls of a thousand waiting warps met on a dozen L2 lines: the one-shot
// 301 x 601 step took 16.6 us instead of 11.0, the eight-shot one 18.7 instead
// of 17.5.
constexpr int FLAG_STRIDE = 8;

__host__ __device__ constexpr int pad32(int n) { return (n + 31) / 32 * 32; }
template <int NS, int TZ> struct Geo {
    static constexpr int HR = TZ + 2 * NS;  // staged halo rows
    static constexpr int HP = HR * SW;      // floats of a halo plane
    static constexpr int OP = TW * TZ;      // floats of an own plane
};
// Floats of a stage.  Stress: v halo (2), sigma own (3).  Velocity: sigma halo
// (3), v own (2).  Coefficients, We and u, which no neighbour reads, go from
// global memory to registers and back: they would take 6 of 16 planes of an
// adjoint stage, and stages are what limits the loads in flight.
template <int NS, int TZ> __host__ __device__ constexpr int stage_floats()
{
    using G = Geo<NS, TZ>;
    constexpr int s = pad32(2 * G::HP) + 3 * G::OP, v = pad32(3 * G::HP) + 2 * G::OP;
    return s > v ? s : v;
}
// CTAs per SM the register budget is set for, and stages that then fit in
// 227 KB of shared memory per SM (1 KB per CTA reserved by the system).
template <int TZ> __host__ __device__ constexpr int ctas_per_sm() { return TZ == 8 ? 3 : 2; }
template <int NS, int TZ> __host__ __device__ constexpr int stages()
{
    constexpr int budget = 227 * 1024 / ctas_per_sm<TZ>() - 2048;
    constexpr int n = budget / (stage_floats<NS, TZ>() * 4);
    return n < 2 ? 2 : n > 3 ? 3 : n;
}
// Warps of a CTA: the team (16 quads x TZ rows), a storer per stage, the loader.
template <int TZ> __host__ __device__ constexpr int team_warps() { return TZ / 2; }
template <int NS, int TZ> __host__ __device__ constexpr int loop_threads()
{
    return 32 * (team_warps<TZ>() + stages<NS, TZ>() + 1);
}

// An item, written by the claimer (two per stage: the one in work, the next).
struct Rec {
    int kind;  // 0 stress, 1 velocity, -1 no more items
    int bz, z0, x0;
    int plain, it, slot, need;  // need: progress the item waits for (it publishes need + 1)
    int flag[5];                // progress words: the tile, above, below, left, right
    int keep;                   // keeps what its sums round off (keep_sum)
    int pad[2];
    TileSR sr;
};
static_assert(sizeof(Rec) == 80, "record size");

// n / d and n % d for 0 <= n < 2^31 by multiplication (Granlund and Montgomery,
// Division by invariant integers using multiplication, 1994).
struct FastDiv {
    unsigned m, s, d;
    __device__ void set(unsigned div)
    {
        d = div;
        if (div == 1) { m = 0; s = 0; return; }
        const int l = 32 - __clz(div - 1);  // ceil(log2 div)
        s = l - 1;
        m = (unsigned)(((1ull << (31 + l)) + div - 1) / div);
    }
    __device__ int div(int n) const { return d == 1 ? n : (int)(__umulhi((unsigned)n, m) >> s); }
};

// The item list of a launch, a stream over the bands of all its steps: stress
// band x (band x mod ntz of step x div ntz), then velocity band x - lag.  A
// velocity band comes lag - 1 pairs of bands after the last stress band it
// waits for, and a stress band ntz - 1 - lag pairs after the last velocity
// band of the step before.  Few steps' worth of L2 and, on small grids, the
// same distance both ways: lag is two more bands than the items in flight
// cover, at most half the grid.  Fewer than three bands: half-step by half-step.
struct List {
    FastDiv band, band2, shots, depth;
    int W, NB, S1, S2, ntx, ntz, nsh, total;
    __device__ void init(const StepParams<float> &p, int nsteps, int tz, int window)
    {
        nsh = p.ctl[1];
        ntx = (p.nx + TW - 1) / TW;
        ntz = (p.nz + tz - 1) / tz;
        W = ntx * nsh;
        NB = ntz * nsteps;
        total = 2 * NB * W;
        const int lag = W ? min(ntz / 2, window / (2 * W) + 2) : 0;
        S1 = lag * W;
        S2 = (2 * NB - lag) * W;
        band.set(max(W, 1));
        band2.set(max(2 * W, 1));
        shots.set(max(nsh, 1));
        depth.set(ntz);
    }
    // Item n: step index k, half (0 stress, 1 velocity), band, column, shot.
    __device__ void item(int n, int &k, int &half, int &b, int &c, int &s) const
    {
        int B, w;
        if (ntz < 3) {
            const int g = band.div(n), h = depth.div(g);  // band of the launch, half-step
            w = n - g * W;
            half = h & 1;
            k = h >> 1;
            b = g - h * ntz;
        } else {
            int t;
            if (n < S1) {
                half = 0;
                t = n;
            } else if (n < S2) {
                const int q = n - S1, pair = band2.div(q), r = q - pair * 2 * W;
                half = r >= W;
                t = half ? pair * W + r - W : S1 + pair * W + r;
            } else {
                half = 1;
                t = NB * W - S1 + n - S2;
            }
            B = band.div(t);
            w = t - B * W;
            k = depth.div(B);
            b = B - k * ntz;
        }
        c = shots.div(w);
        s = w - c * nsh;
    }
};

// Relaxed, so that several are in flight; acquire_fence() after the last.
__device__ __forceinline__ int ld_relaxed(const int *a)
{
    int v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
    return v;
}
__device__ __forceinline__ void acquire_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
// Whether barrier `bar` has completed phase `parity`, without waiting.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ void st_release(int *a, int v)
{
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_proxy_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// One box from shared memory to a 3-D tensor; rows, columns and planes
// outside the tensor are not written.
__device__ __forceinline__ void tma_store(const CUtensorMap *map, int x, int y, int z, uint32_t src)
{
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(z), "r"(src)
                 : "memory");
}
// A box on its way into L2.
__device__ __forceinline__ void tma_prefetch(const CUtensorMap *map, int x, int y, int z)
{
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(z)
                 : "memory");
}
__device__ __forceinline__ void store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void store_read_done() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void store_done() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ------------------------------------------------------------------ stress
// vdiff2 + pml_diff2 + update_s2 + surf_mirror (src/cpu/n_kernel_lib_PSV.cpp:
// 100-205, 272-395) of the thread's quads of a staged tile.  A top free
// surface and the rows it mirrors lie in the first band of tiles
// (loop_supported): the mirrored cells are in the same stage.
template <int NS, int TZ>
__device__ __forceinline__ void stress_team(const StepParams<float> &p, float *st, const Rec &T, int t)
{
    using G = Geo<NS, TZ>;
    const int q = 4 * (t & 15), lr = t >> 4;  // the thread's quad and tile row
    const int ix = T.x0 + q, iz = T.z0 + lr;
    float *own = st + pad32(2 * G::HP), *o = own + lr * TW + q;
    unsigned mask = 0xf;
    if (!T.plain) {
        mask = inner_mask(p, ix);
        if (!mask || iz < p.nz1 || iz >= p.nz2) return;
    }
    const int i = iz * p.pitch + ix;
    const Q4 cl = ldro4(p.c_lam + i), c2 = ldro4(p.c_l2m + i), cm = ldro4(p.c_muzx + i);
    const float *hz = st + lr * SW + HX + q, *hx = hz + G::HP;  // staged row lr = tile row lr - NS
    Q4 zz, xx, zx, xz;  // vz_z, vx_x, vz_x, vx_z
    float h[12];
    {
        Q4 w[2 * NS];
#pragma unroll
        for (int j = 0; j < 2 * NS; j++) w[j] = lds4(hz + j * SW);
        row12(hz + NS * SW, w[NS], h);
        zz = dvert<NS>(w, p.cz);
        zx = dhorz<NS, 1>(h, p.cx);
    }
    {
        Q4 w[2 * NS];
#pragma unroll
        for (int j = 0; j < 2 * NS; j++) w[j] = lds4(hx + (j + 1) * SW);
        row12(hx + NS * SW, w[NS - 1], h);
        xz = dvert<NS>(w, p.cz);
        xx = dhorz<NS, 0>(h, p.cx);
    }
    if (!T.plain)
        cpml_quads(p, T.bz, iz, ix, mask, MZ_VZ, MZ_VX, zz, xz, MX_VX, MX_VZ, xx, zx);
    // (A mirrored row's szz and szx are another thread's to write: it reads v in
    // their place.  With the row's flags in a struct instead, the adjoint took 27.3 us
    // a step on 4000 x 48, 4 shots, for 22.1.)
    const float *mine = T.plain || surface_own(iz, p.st) ? o : st;
    Q4 szz = lds4(mine), szx = lds4(mine + G::OP), sxx = lds4(o + 2 * G::OP);
    bool wz = true;      // szz, szx are this row's own (not mirrored into it)
    int mirror = -1;     // row of the stage this row is mirrored into
    bool image = false;  // the free-surface row itself
    if (!T.plain && p.st) {
        image = surface_image(iz, p.st);
        wz = surface_own(iz, p.st);
        if (surface_mirrors(iz, p.st, p.nz1)) mirror = 2 * p.st - iz - T.z0;
    }
    if (T.keep) {
        float *f = p.fld + (long long)T.bz * p.shot_stride + (long long)(F_SZZ + p.pp_planes) * p.plane + i;
        Q4 rzz = ldg4(f), rzx = ldg4(f + p.plane), rxx = ldg4(f + 2 * p.plane);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (!(mask >> j & 1)) continue;
            keep_sum(szz.v[j], rzz.v[j], fmaf(c2.v[j], zz.v[j], fmaf(cl.v[j], xx.v[j], rzz.v[j])));
            keep_sum(sxx.v[j], rxx.v[j], fmaf(c2.v[j], xx.v[j], fmaf(cl.v[j], zz.v[j], rxx.v[j])));
            keep_sum(szx.v[j], rzx.v[j], fmaf(cm.v[j], zx.v[j] + xz.v[j], rzx.v[j]));
            if (image) rzz.v[j] = rzx.v[j] = rxx.v[j] = 0.f;
        }
        st4(f, rzz);
        st4(f + p.plane, rzx);
        st4(f + 2 * p.plane, rxx);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (!(mask >> j & 1)) continue;
        if (!T.keep) {
            szz.v[j] += fmaf(c2.v[j], zz.v[j], cl.v[j] * xx.v[j]);
            sxx.v[j] += fmaf(c2.v[j], xx.v[j], cl.v[j] * zz.v[j]);
            szx.v[j] = fmaf(cm.v[j], zx.v[j] + xz.v[j], szx.v[j]);
        }
        if (image) {
            szz.v[j] = szx.v[j] = 0.f;
            sxx.v[j] = p.fs_top[ix + j] * xx.v[j];
        }
    }
    if (wz) {
        st4(o, szz);
        st4(o + G::OP, szx);
    }
    st4(o + 2 * G::OP, sxx);
    if (mirror >= 0) {
        float *d = own + mirror * TW + q;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (mask >> j & 1) {
                d[j] = -szz.v[j];
                d[G::OP + j] = -szx.v[j];
            }
    }
}

// ---------------------------------------------------------------- velocity
// sdiff2 + pml_diff2 + update_v2, snapshot store / imaging
// (src/cpu/n_kernel_lib_PSV.cpp:207-270, 398-484) of the thread's quads.
// Cells outside the interior only take part in the snapshot / imaging work.
template <int NS, int TZ, int MODE>
__device__ __forceinline__ void velocity_team(const StepParams<float> &p, float *st, const Rec &T, int t)
{
    using G = Geo<NS, TZ>;
    constexpr bool U = has_u<MODE>(), WE = has_we<MODE>();
    const int q = 4 * (t & 15), lr = t >> 4;
    const int ix = T.x0 + q, iz = T.z0 + lr;
    float *o = st + pad32(3 * G::HP) + lr * TW + q;
    unsigned mask = 0xf;
    if (!T.plain) {
        if (ix >= p.nx || iz >= p.nz) return;
        mask = iz >= p.nz1 && iz < p.nz2 ? inner_mask(p, ix) : 0;
        if (!mask && T.slot < 0) return;
    }
    const float *azz = st + lr * SW + HX + q, *azx = azz + G::HP, *axx = azx + G::HP;
    const int i = iz * p.pitch + ix;
    float *f = p.fld + (long long)T.bz * p.shot_stride + i;
    float *fw = f + (MODE == MODE_ADJ ? F_WEA : F_WE) * p.plane;
    float *fuz = f + F_UZ * p.plane, *fux = f + F_UX * p.plane;
    Q4 uz = all4(0.f), ux = all4(0.f), we = all4(0.f);
    if constexpr (U) {
        uz = ldg4(fuz);
        ux = ldg4(fux);
    }
    if constexpr (WE) we = ldg4(fw);
    const Q4 crz = ldro4(p.c_rz + i), crx = ldro4(p.c_rx + i);
    Q4 vz = lds4(o), vx = lds4(o + G::OP);
    if (mask) {
        Q4 zz_z, zx_z, zx_x, xx_x;
        float h[12];
        {
            Q4 w[2 * NS];
#pragma unroll
            for (int j = 0; j < 2 * NS; j++) w[j] = lds4(azz + (j + 1) * SW);
            zz_z = dvert<NS>(w, p.cz);
        }
        {
            Q4 w[2 * NS];
#pragma unroll
            for (int j = 0; j < 2 * NS; j++) w[j] = lds4(azx + j * SW);
            row12(azx + NS * SW, w[NS], h);
            zx_z = dvert<NS>(w, p.cz);
            zx_x = dhorz<NS, 0>(h, p.cx);
        }
        row12(axx + NS * SW, lds4(axx + NS * SW), h);
        xx_x = dhorz<NS, 1>(h, p.cx);
        if (!T.plain)
            cpml_quads(p, T.bz, iz, ix, mask, MZ_SZZ, MZ_SZX, zz_z, zx_z, MX_SXX, MX_SZX, xx_x, zx_x);
        Q4 rz = all4(0.f), rx = all4(0.f);
        float *fr = f + (long long)(F_VZ + p.pp_planes) * p.plane;
        if (MODE != MODE_ADJ && T.keep) {
            rz = ldg4(fr);
            rx = ldg4(fr + p.plane);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (!(mask >> j & 1)) continue;
            if constexpr (U) {
                uz.v[j] = fmaf(p.dt, vz.v[j], uz.v[j]);
                ux.v[j] = fmaf(p.dt, vx.v[j], ux.v[j]);
            }
            if (MODE == MODE_ADJ || !T.keep) {
                vz.v[j] = fmaf(crz.v[j], zx_x.v[j] + zz_z.v[j], vz.v[j]);
                vx.v[j] = fmaf(crx.v[j], xx_x.v[j] + zx_z.v[j], vx.v[j]);
            } else {
                keep_sum(vz.v[j], rz.v[j], fmaf(crz.v[j], zx_x.v[j] + zz_z.v[j], rz.v[j]));
                keep_sum(vx.v[j], rx.v[j], fmaf(crx.v[j], xx_x.v[j] + zx_z.v[j], rx.v[j]));
            }
            if constexpr (WE) we.v[j] += fmaf(vx.v[j], vx.v[j], vz.v[j] * vz.v[j]);
        }
        st4(o, vz);
        st4(o + G::OP, vx);
        if (MODE != MODE_ADJ && T.keep) {
            st4(fr, rz);
            st4(fr + p.plane, rx);
        }
        if constexpr (WE) st4(fw, we);
        if constexpr (U) {
            st4(fuz, uz);
            st4(fux, ux);
        }
    }
    if (T.slot >= 0)  // the new stresses, from the stage
        snapshot_quad<MODE>(p, T.bz, iz, ix, T.slot, lds4(azz + NS * SW), lds4(azx + NS * SW),
                            lds4(axx + NS * SW), vz, vx, uz, ux);
}

// vsrc2 + urec2 (src/cpu/n_kernel_lib_PSV.cpp:487-576) for the sources and
// receivers of a staged velocity tile by one warp, on the new velocities in
// the stage; then the snapshot fix-up of source cells (the stored velocity
// is the post-injection one).
template <int NS, int TZ, int MODE>
__device__ __forceinline__ void srcrec_warp(const StepParams<float> &p, const SrcRecParams<float> &q,
                                            float *vz, const Rec &T, int lane)
{
    float *vx = vz + Geo<NS, TZ>::OP;
    const TileSR e = T.sr;
    const int shot = p.ctl[0] + T.bz;
    auto local = [&](int pos) {
        const int iz = pos / p.pitch;
        return (iz - T.z0) * TW + pos - iz * p.pitch - T.x0;
    };
    const double sc = q.amp_scale[shot];
    const double *sz = q.stf_z + shot * q.stf_shot_stride + (long long)T.it * q.stf_ncol;
    const double *sx = q.stf_x + shot * q.stf_shot_stride + (long long)T.it * q.stf_ncol;
    auto fetch = [&](int k, int &pos, float &az, float &ax) {
        int col;
        if (q.src_kind == 0) {
            const int j = q.t_src_k[k];
            pos = q.src_pos[j];
            col = q.src_col[j];
        } else {
            const int rr = q.t_rec_r[k];
            pos = q.rec_pos[rr];
            col = rr;
        }
        if (q.stf_type == 0) {
            az = p.c_rz[pos] * (float)(sz[col] * sc * q.inv_dzdx);
            ax = p.c_rx[pos] * (float)(sx[col] * sc * q.inv_dzdx);
        } else {
            az = (float)(sz[col] * sc);
            ax = (float)(sx[col] * sc);
        }
    };
    if constexpr (MODE == MODE_ADJ) {
        for (int k = e.k0 + lane; k < e.k1; k += 32) {
            int pos;
            float az, ax;
            fetch(k, pos, az, ax);
            const int i = local(pos);
            atomicAdd(vz + i, az);
            atomicAdd(vx + i, ax);
        }
    } else {
        for (int k0 = e.k0; k0 < e.k1; k0 += 32) {
            int pos = 0, i = -1 - lane;
            float az = 0.f, ax = 0.f;
            if (k0 + lane < e.k1) {
                fetch(k0 + lane, pos, az, ax);
                i = local(pos);
            }
            if (!T.keep) {
                if (i >= 0) {
                    atomicAdd(vz + i, az);
                    atomicAdd(vx + i, ax);
                }
                continue;
            }
            // Sources that share a cell sum in their order, each in its turn.  (One
            // lane for all: 56 us a step with 480 sources on a line, 301 x 601, 8
            // shots; this 18.3; one source a shot 16.5.)
            const unsigned same = e.k1 - k0 > 1 ? __match_any_sync(ALL, i) : 0;
            const int turn = __popc(same & ((1u << lane) - 1));
            int r = 0;
            do {
                if (i >= 0 && turn == r) {
                    float *f = p.fld + (long long)T.bz * p.shot_stride + (long long)(F_VZ + p.pp_planes) * p.plane + pos;
                    float rz = __ldcg(f), rx = __ldcg(f + p.plane);
                    keep_sum(vz[i], rz, az + rz);
                    keep_sum(vx[i], rx, ax + rx);
                    f[0] = rz;
                    f[p.plane] = rx;
                }
                __syncwarp();
                r++;
            } while (__any_sync(ALL, turn >= r));
        }
    }
    __syncwarp();
    if (e.r0 < e.r1) {
        double *rz = q.rtf_z + shot * q.rtf_shot_stride;
        double *rx = q.rtf_x + shot * q.rtf_shot_stride;
        // one factor: an FP64 divide a sample holds up the tile's publication
        // (FP64 runs at a 64th of the FP32 rate)
        const double ru = q.dt_d * q.inv_dzdx * q.rec_unscale[shot];
        const long long row = (long long)T.it * q.nrec;
        for (int k = e.r0 + lane; k < e.r1; k += 32) {
            const int rr = q.t_rec_r[k];
            const int i = local(q.rec_pos[rr]);
            const double pz = T.it ? __ldcg(rz + row - q.nrec + rr) : 0.0;
            const double px = T.it ? __ldcg(rx + row - q.nrec + rr) : 0.0;
            rz[row + rr] = fma(ru, (double)vz[i], pz);
            rx[row + rr] = fma(ru, (double)vx[i], px);
        }
    }
    if (MODE != MODE_ADJ && T.slot >= 0 && q.src_kind == 0) {
        float *h = p.hist + (long long)T.bz * p.hist_shot_stride + (long long)T.slot * p.hist_slot_stride;
        for (int k = e.k0 + lane; k < e.k1; k += 32) {
            const int j = q.t_src_k[k];
            const int c = q.src_snap[j];
            if (c < 0) continue;
            const int i = local(q.src_pos[j]);
            h[H_VZ * p.snap_plane + c] = vz[i] * p.inv_dt;
            h[H_VX * p.snap_plane + c] = vx[i] * p.inv_dt;
        }
    }
}

// ------------------------------------------------------------------ kernel

// What item T will want from HBM, on its way to L2 from the moment it is
// claimed (one thread): with the wavefields out of L2 (`far`), the stress
// tile's v and sigma, We and u; on imaging steps the snapshot and the shot
// gradients, which the stages have no room for.
template <int MODE, int NS>
__device__ __forceinline__ void prefetch_item(const LoopMaps &m, const StepParams<float> &p,
                                              const LoopRun &run, const Rec &T, int pps)
{
    const int x0 = T.x0, z0 = T.z0, pb = T.bz * pps;
    if (run.far) {
        if (!T.kind) {
            tma_prefetch(&m.halo2, x0 - HX, z0 - NS, pb + F_VZ);
            tma_prefetch(&m.own3, x0, z0, pb + F_SZZ);
        } else {
            if (has_we<MODE>()) tma_prefetch(&m.own1, x0, z0, pb + (MODE == MODE_ADJ ? F_WEA : F_WE));
            if (has_u<MODE>()) tma_prefetch(&m.own2, x0, z0, pb + F_UZ);
        }
    }
    if (MODE == MODE_ADJ && T.kind && T.slot >= 0 && run.images) {
        const int x = max(x0 - (p.snap_x1 & ~3), 0), z = max(z0 - p.snap_z1, 0);
        if (x < p.snx && z < p.snz) {
            tma_prefetch(&m.hist5, x, z, (T.bz * run.images + T.slot) * NHIST);
            tma_prefetch(&m.grad3, x, z, T.bz * 3);
        }
    }
}

// Fills the stage at shared address `d` for item T (one thread).
template <int NS, int TZ, int MODE>
__device__ __forceinline__ void issue_loads(const LoopMaps &m, const Rec &T, uint32_t d, uint32_t bar, int pps)
{
    using G = Geo<NS, TZ>;
    const int x0 = T.x0, z0 = T.z0, pb = T.bz * pps;
    if (!T.kind) {
        mbar_expect_tx(bar, (uint32_t)(2 * G::HP + 3 * G::OP) * 4);
        tma_load(d, &m.halo2, x0 - HX, z0 - NS, pb + F_VZ, bar);
        tma_load(d + pad32(2 * G::HP) * 4, &m.own3, x0, z0, pb + F_SZZ, bar);
    } else {
        mbar_expect_tx(bar, (uint32_t)(3 * G::HP + 2 * G::OP) * 4);
        tma_load(d, &m.halo3, x0 - HX, z0 - NS, pb + F_SZZ, bar);
        tma_load(d + pad32(3 * G::HP) * 4, &m.own2, x0, z0, pb + F_VZ, bar);
    }
}

// Stores the stage's new values (one thread), as one bulk group.
template <int NS, int TZ>
__device__ __forceinline__ void issue_stores(const LoopMaps &m, const Rec &T, uint32_t d, int pps)
{
    using G = Geo<NS, TZ>;
    const int pb = T.bz * pps;
    if (!T.kind) tma_store(&m.own3, T.x0, T.z0, pb + F_SZZ, d + pad32(2 * G::HP) * 4);
    else tma_store(&m.own2, T.x0, T.z0, pb + F_VZ, d + pad32(3 * G::HP) * 4);
    store_commit();
}

template <int NS, int TZ, int MODE>
__global__ void __launch_bounds__((loop_threads<NS, TZ>()), ctas_per_sm<TZ>())
    k_loop(const __grid_constant__ StepParams<float> p, const __grid_constant__ SrcRecParams<float> q,
           const __grid_constant__ LoopMaps m, const LoopRun run)
{
    using G = Geo<NS, TZ>;
    constexpr int SF = stage_floats<NS, TZ>(), NST = stages<NS, TZ>(), CW = team_warps<TZ>();
    extern __shared__ __align__(128) unsigned char smraw[];
    // per stage: full (loaded), done (computed); per record: known, free
    __shared__ __align__(8) uint64_t bars[2 * NST + 4 * NST];
    __shared__ __align__(16) Rec recs[2 * NST];
    float *stg = align128(smraw);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto full = [&](int s) { return smem_u32(&bars[s]); };
    auto done = [&](int s) { return smem_u32(&bars[NST + s]); };
    auto known = [&](int r) { return smem_u32(&bars[2 * NST + r]); };
    auto spare = [&](int r) { return smem_u32(&bars[4 * NST + r]); };
    if (threadIdx.x == 0) {
        for (int s = 0; s < NST; s++) {
            mbar_init(full(s), 1);
            mbar_init(done(s), CW);
        }
        for (int r = 0; r < 2 * NST; r++) {
            mbar_init(known(r), 1);
            mbar_init(spare(r), 1);
        }
        fence_init();
    }
    __syncthreads();
    const int pps = (int)(p.shot_stride / p.plane);
    int *flags = run.sync + LOOP_SYNC_HEAD;

    if (w == CW + NST) {
        // Claimer: items k = 0, 1, ... of the CTA in list order, one for each
        // stage in turn, ahead of their use.
        List L;
        L.init(p, run.nsteps, TZ, (int)gridDim.x * 2 * NST);
        const int shot0 = p.ctl[0];
        const bool srcrec = q.src_kind >= 0 || q.rtf_z;
        int pre = 0;
        if (lane == 0) pre = atomicAdd(run.sync, 1);
        for (int k = 0, stops = 0; stops < NST; k++) {
            const int s = k % NST, j = k / NST, r = 2 * s + (j & 1);
            // near: not before the stage's current item has been loaded
            if (!run.far && j && !mbar_wait(full(s), (j - 1) & 1)) {
                if (lane == 0) atomicExch(p.err, 1);
                break;
            }
            const int n = __shfl_sync(0xffffffffu, pre, 0);
            Rec R;
            R.kind = -1;
            if (n < L.total) {
                if (lane == 0) pre = atomicAdd(run.sync, 1);  // its latency overlaps this item
                int step, half, b, c, sh;
                L.item(n, step, half, b, c, sh);
                R.sr = TileSR{0, 0, 0, 0};
                if (half && srcrec) R.sr = tile_srcrec(q, shot0, b * L.ntx + c, sh);
                R.keep = MODE != MODE_ADJ && run.keep ? run.keep[b * L.ntx + c] : 0;
                const int z0 = b * TZ, x0 = c * TW, f = (sh * L.ntz + b) * L.ntx + c;
                R.kind = half; R.bz = sh; R.z0 = z0; R.x0 = x0;
                R.plain = half ? plain_box(p, z0, z0 + TZ, x0, x0 + TW)
                               : plain_stress_box(p, z0, z0 + TZ, x0, x0 + TW);
                const int it = run.it0 + step * run.dit, rel = it / run.sdt;
                R.it = it;
                R.slot = run.snap && rel * run.sdt == it ? (rel - run.base) % run.ring : -1;
                R.need = 2 * step + half;
                R.flag[0] = f;
                R.flag[1] = b ? f - L.ntx : f;
                R.flag[2] = b + 1 < L.ntz ? f + L.ntx : f;
                R.flag[3] = c ? f - 1 : f;
                R.flag[4] = c + 1 < L.ntx ? f + 1 : f;
            } else {
                stops++;
            }
            if (j >= 2 && !mbar_wait(spare(r), (j / 2 - 1) & 1)) {
                if (lane == 0) atomicExch(p.err, 1);
                break;
            }
            if (lane == 0) {
                recs[r] = R;
                mbar_arrive(known(r));
                if (R.kind >= 0) prefetch_item<MODE, NS>(m, p, run, R, pps);
            }
            __syncwarp();
        }
    } else if (w < CW) {
        // Team: every stage in the CTA's item order.
        for (int k = 0;; k++) {
            const int s = k % NST, j = k / NST;
            if (!mbar_wait(full(s), j & 1)) {
                if (lane == 0) atomicExch(p.err, 1);
                break;
            }
            const Rec &T = recs[2 * s + (j & 1)];
            if (T.kind < 0) break;
            float *st = stg + s * SF;
            if (T.kind == 0) stress_team<NS, TZ>(p, st, T, threadIdx.x);
            else velocity_team<NS, TZ, MODE>(p, st, T, threadIdx.x);
            fence_async_smem();  // the stage's new values before the TMA store reads them
            __syncwarp();
            if (lane == 0) mbar_arrive(done(s));
        }
    } else {
        // Keeper of stage s.  While an item is loaded and computed, the next
        // one's progress words are polled and the fences paid, so that its
        // loads start as soon as the stage has been read out.
        const int s = w - CW;
        float *st = stg + s * SF;
        bool have = false, ready = false;  // the next item: record known; dependences met and fenced
        auto look = [&](int j) {  // one poll of item j's progress words
            const Rec &T = recs[2 * s + (j & 1)];
            if (T.kind < 0) return true;
            const bool ok = lane >= 5 || ld_relaxed(flags + T.flag[lane] * FLAG_STRIDE) >= T.need;
            if (!__all_sync(ALL, ok)) return false;
            acquire_fence();
            __syncwarp();
            fence_proxy_global();  // the acquires before the async-proxy reads that follow
            return true;
        };
        bool loaded = false, failed = false;
        for (int j = 0;; j++) {
            const Rec &T = recs[2 * s + (j & 1)];
            if (!loaded) {
                if (!have) failed = !__all_sync(ALL, mbar_wait(known(2 * s + (j & 1)), (j / 2) & 1));
                const unsigned long long t0 = now_ns();
                while (!failed && !ready) {
                    ready = look(j);
                    failed = !ready && __any_sync(ALL, now_ns() - t0 > WAIT_LIMIT_NS);
                }
                if (failed) break;
                if (T.kind < 0) {  // no more items: the team learns it from the record
                    if (lane == 0) mbar_arrive(full(s));
                    break;
                }
                if (lane == 0) issue_loads<NS, TZ, MODE>(m, T, smem_u32(st), full(s), pps);
            }
            loaded = have = ready = false;
            // wait for the team, looking after the next item meanwhile (every
            // decision is the warp's, not a lane's)
            const unsigned long long t0 = now_ns();
            for (;;) {
                if (!have) have = __all_sync(ALL, mbar_test(known(2 * s + ((j + 1) & 1)), ((j + 1) / 2) & 1));
                if (have && !ready) ready = look(j + 1);
                const bool d = have && ready ? mbar_try(done(s), j & 1) : mbar_test(done(s), j & 1);
                if (__all_sync(ALL, d)) break;
                failed = __any_sync(ALL, now_ns() - t0 > WAIT_LIMIT_NS);
                if (failed) break;
            }
            if (failed) break;
            if (T.kind && (T.sr.k0 != T.sr.k1 || T.sr.r0 < T.sr.r1)) {
                srcrec_warp<NS, TZ, MODE>(p, q, st + pad32(3 * G::HP), T, lane);
                fence_async_smem();
                __syncwarp();
            }
            const Rec &N = recs[2 * s + ((j + 1) & 1)];
            if (lane == 0) {
                issue_stores<NS, TZ>(m, T, smem_u32(st), pps);
                store_read_done();
            }
            __syncwarp();
            // another lane's loads: the release below waits for its own thread's
            if (lane == 1 && ready && N.kind >= 0) issue_loads<NS, TZ, MODE>(m, N, smem_u32(st), full(s), pps);
            __syncwarp();
            if (lane == 0) {
                store_done();
                st_release(flags + T.flag[0] * FLAG_STRIDE, T.need + 1);
                mbar_arrive(spare(2 * s + (j & 1)));
            }
            loaded = ready && N.kind >= 0;
            __syncwarp();
        }
        if (failed && lane == 0) atomicExch(p.err, 1);
    }
}

template <int NS, int TZ, int MODE>
cudaError_t loop_m(const StepParams<float> &p, const SrcRecParams<float> &q, const LoopMaps &m,
                   const LoopRun &run, int nbatch, cudaStream_t st)
{
    constexpr int smem = stages<NS, TZ>() * stage_floats<NS, TZ>() * 4 + 128;
    auto kernel = k_loop<NS, TZ, MODE>;
    struct Fit {
        cudaError_t e;
        int ctas;
    };
    static PerDevice<Fit> fits;  // per instantiation: CTAs the GPU holds at once
    Fit fit{cudaSuccess, 0};
    cudaError_t e = on_device(fits, [&] {
        Fit r{cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), 0};
        int per = 0, dev = 0, nsm = 0;
        if (r.e == cudaSuccess) r.e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, (loop_threads<NS, TZ>()), smem);
        if (r.e == cudaSuccess) r.e = cudaGetDevice(&dev);
        if (r.e == cudaSuccess) r.e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (r.e == cudaSuccess && per < 1) r.e = cudaErrorInvalidConfiguration;
        r.ctas = per * nsm;
        return r;
    }, &fit);
    if (e == cudaSuccess) e = fit.e;
    if (e != cudaSuccess) return e;
    const int tiles = ((p.nx + TW - 1) / TW) * ((p.nz + TZ - 1) / TZ) * nbatch;
    e = cudaMemsetAsync(run.sync, 0, (size_t)(LOOP_SYNC_HEAD + tiles * FLAG_STRIDE) * sizeof(int), st);
    if (e != cudaSuccess) return e;
    kernel<<<std::min(fit.ctas, tiles), loop_threads<NS, TZ>(), smem, st>>>(p, q, m, run);
    return cudaGetLastError();
}

template <int NS, int TZ>
cudaError_t loop_t(const StepParams<float> &p, const SrcRecParams<float> &q, const LoopMaps &m,
                   const LoopRun &run, int mode, int nbatch, cudaStream_t st)
{
    switch (mode) {
    case MODE_FWD: return loop_m<NS, TZ, MODE_FWD>(p, q, m, run, nbatch, st);
    case MODE_FWD_NOWE: return loop_m<NS, TZ, MODE_FWD_NOWE>(p, q, m, run, nbatch, st);
    case MODE_FWD_U: return loop_m<NS, TZ, MODE_FWD_U>(p, q, m, run, nbatch, st);
    case MODE_ADJ: return loop_m<NS, TZ, MODE_ADJ>(p, q, m, run, nbatch, st);
    default: return cudaErrorInvalidValue;
    }
}

template <int NS>
cudaError_t loop_n(const StepParams<float> &p, const SrcRecParams<float> &q, const LoopMaps &m,
                   const LoopRun &run, int mode, int tz, int nbatch, cudaStream_t st)
{
    switch (tz) {
    case 8: return loop_t<NS, 8>(p, q, m, run, mode, nbatch, st);
    case 16: return loop_t<NS, 16>(p, q, m, run, mode, nbatch, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

// What the listed tiles' sums kept (keep_sum), planes vz vx szz szx sxx after
// the fields' first copy: zeroed (op 0), copied to (1) or from (2) packed
// storage [batch][tile][5][tz][64] of shot stride `cstride`.
__global__ void k_loop_kept(int op, float *fld, long long shot_stride, long long plane, int pitch, int nz, int nx,
                            int ntx, int tz, const int *tiles, float *packed, long long cstride)
{
    const int tile = tiles[blockIdx.x], z0 = tile / ntx * tz, x0 = tile % ntx * TW;
    for (int e = threadIdx.x; e < 5 * tz * TW; e += blockDim.x) {
        const int k = e / (tz * TW), iz = z0 + e / TW % tz, ix = x0 + e % TW;
        if (iz >= nz || ix >= nx) continue;
        float *f = fld + blockIdx.y * shot_stride + k * plane + (long long)iz * pitch + ix;
        float *c = packed + blockIdx.y * cstride + (long long)blockIdx.x * 5 * tz * TW + e;
        if (op == 1) *c = *f;
        else *f = op == 2 ? *c : 0.f;
    }
}
cudaError_t launch_loop_kept(int op, float *fld, long long shot_stride, long long plane, int pitch, int nz, int nx,
                             int tz, const int *tiles, int ntiles, float *packed, long long cstride, int nbatch,
                             cudaStream_t st)
{
    if (ntiles <= 0) return cudaSuccess;
    k_loop_kept<<<dim3(ntiles, nbatch), 256, 0, st>>>(op, fld, shot_stride, plane, pitch, nz, nx,
                                                      (nx + TW - 1) / TW, tz, tiles, packed, cstride);
    return cudaGetLastError();
}

// The tile heights the loop is built for, and the surfaces it handles: none,
// or a top one whose mirrored rows lie in the first band of tiles.
bool loop_supported(int tz, int st, int sb, int sl, int sr, int nz1)
{
    return (tz == 8 || tz == 16) && !sb && !sl && !sr && (!st || 2 * st - nz1 < tz);
}

// Progress words of a batch: one per tile of the smallest tile height.
size_t loop_sync_bytes(int nz, int nx, int nbatch)
{
    return (size_t)(LOOP_SYNC_HEAD + (long long)((nx + TW - 1) / TW) * ((nz + 7) / 8) * nbatch * FLAG_STRIDE) * sizeof(int);
}

// Steps a launch may hold so that its items are counted in 31 bits.
int loop_max_steps(int nz, int nx, int nbatch)
{
    const long long per = 2ll * ((nx + TW - 1) / TW) * ((nz + 7) / 8) * nbatch;
    return (int)std::max(1ll, std::min(256ll, ((1ll << 31) - (1ll << 24)) / std::max(per, 1ll)));
}

int encode_loop_maps(LoopMaps *m, const float *fld, int nfplanes, int nx, int nz, int pitch,
                     long long plane, int ns, int tz, const float *hist, int nhplanes, const float *gshot,
                     int ngplanes, int snx_pitch, int snz)
{
    if (ns < 1 || ns > HX) return fail(PSV_ERR_UNSUPPORTED, "TMA tiles: stencil half-width above 4");
    if (pitch % 4 || (uintptr_t)fld % 16)
        return fail(PSV_ERR_ARG, "TMA tiles: misaligned field block");
    const int hr = tz + 2 * ns;
    PSV_TRY(encode3(&m->halo2, fld, nx, nz, pitch, plane, nfplanes, SW, hr, 2));
    PSV_TRY(encode3(&m->halo3, fld, nx, nz, pitch, plane, nfplanes, SW, hr, 3));
    PSV_TRY(encode3(&m->own1, fld, nx, nz, pitch, plane, nfplanes, TW, tz, 1));
    PSV_TRY(encode3(&m->own2, fld, nx, nz, pitch, plane, nfplanes, TW, tz, 2));
    PSV_TRY(encode3(&m->own3, fld, nx, nz, pitch, plane, nfplanes, TW, tz, 3));
    if (hist) {
        const long long sp = (long long)snz * snx_pitch;
        PSV_TRY(encode3(&m->hist5, hist, snx_pitch, snz, snx_pitch, sp, nhplanes, TW, tz, NHIST));
        PSV_TRY(encode3(&m->grad3, gshot, snx_pitch, snz, snx_pitch, sp, ngplanes, TW, tz, 3));
    }
    return PSV_OK;
}

cudaError_t launch_loop(const StepParams<float> &p, const SrcRecParams<float> &q, const LoopMaps &m,
                        const LoopRun &run, int ns, int mode, int tz, int nbatch, cudaStream_t st)
{
    switch (ns) {
    case 1: return loop_n<1>(p, q, m, run, mode, tz, nbatch, st);
    case 2: return loop_n<2>(p, q, m, run, mode, tz, nbatch, st);
    case 3: return loop_n<3>(p, q, m, run, mode, tz, nbatch, st);
    case 4: return loop_n<4>(p, q, m, run, mode, tz, nbatch, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace psv
