// psv_resident.cu -- many time steps of a small batch in one launch, with the
// wavefields on chip (FP32).
//
// A grid that gives every SM a few hundred points spends a step on the way
// between SMs, not on arithmetic: two launches cost 9 to 12 us a step however
// small the grid, the tile list of psv_loop.cu 11 to 12 (claim, load, store,
// fence and progress word of each half-step).  Here a CTA keeps one tile of
// 32 or 64 columns x tz rows of one shot for the whole launch: v, sigma and
// their halos in shared memory, u and We in registers, one or two quads of
// columns per thread; the CPML memories in registers with one quad, through L1
// with two.  Only the tiles' rims travel, once per half-step.
//
// A rim cell is sent as two 64-bit words {value, half-step number}, written by
// one 128-bit store straight into the neighbour's inbox and polled there: a
// word arrives whole, so the number says that its value is there, and neither
// side needs a fence or a separate flag.  One way is one store and one load
// through L2.  A cell of the inbox is written again only after the neighbour's
// own next rim has arrived here, which it sends after reading the cell.
//
// What bounds it: the rim's way, about 1 us of each half-step, and the chain
// of a quad's update behind it.  us a step forward / adjoint:
//   101 x 201, 1 shot, order 4    2.9 / 3.1   (tiles of 32 x 8)
//   301 x 601, 1 shot, order 4    3.6 / 4.0   (32 x 38)
//   281 x 561, 2 shots, order 4   6.9 / 8.0   (64 x 36; 13.1 / 14.6 by psv_loop.cu)
// and whole passes, two launches a step before -> here: 400 steps of modelling
// on the first grid 3591 -> 1322 us, the second's gradient (800 steps)
// 9264 -> 3992, five shots on 187 x 133, order 6, 1000 steps 10478 -> 4618.
// At 128 registers a thread (512 threads may fill an SM) every instantiation
// spills: 180 to 296 bytes stored with one quad a thread, 16 to 168 with two.
// What neither the next update nor a neighbour waits for comes after the rim
// of v is sent: snapshots, imaging, traces; source amplitudes are fetched
// before the waits.  The traces' FP64 divide, at a 64th of the FP32 rate, held
// up the next half-step of its tile: one factor for the launch instead, with
// that order, took 400 steps of modelling on 101 x 201 from 1916 to 1378 us.
//
// All CTAs must be resident: the launch is cooperative, one CTA or more per SM
// (resident_tile).  Waits are bounded: after two seconds StepParams::err is set
// and the CTA leaves; the host turns that into PSV_ERR_CUDA.
#include <algorithm>

#include "psv_plan.cuh"
#include "psv_quads.cuh"
#include "psv_tma.cuh"

namespace psv {

namespace {

constexpr int MAX_THREADS = 512;

// rw: tile columns, 32 or 64.
__host__ __device__ constexpr int staged_row(int rw) { return rw + 2 * HX; }
// Cells of a tile's rim: NS rows above and below, NS columns left and right.
__host__ __device__ constexpr int rim_cells(int ns, int rw, int tz) { return 2 * ns * (rw + tz); }
// Eight threads to a row, and at most two rim cells to a thread.
__host__ __device__ constexpr int resident_threads(int ns, int rw, int tz)
{
    const int q = 8 * tz, r = rim_cells(ns, rw, tz);
    const int n = q > r ? q : r < MAX_THREADS ? r : MAX_THREADS;
    return (n + 31) / 32 * 32;
}
// v and sigma with halo, and what the sums of five fields kept.
__host__ __device__ constexpr int resident_smem(int ns, int rw, int tz)
{
    return 4 * (5 * (tz + 2 * ns) * staged_row(rw) + 5 * tz * rw);
}

struct ResidentRun {
    LoopRun r;
    int tz, ntx, ntz;  // rows of a tile, tiles
    ulonglong2 *inbox;  // [tile][v, sigma][rim cell]
};

__device__ __forceinline__ void send(ulonglong2 *a, float x, float y, unsigned seq)
{
    const unsigned long long s = (unsigned long long)seq << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(a), "l"(s | __float_as_uint(x)),
                 "l"(s | __float_as_uint(y))
                 : "memory");
}
__device__ __forceinline__ bool poll(const ulonglong2 *a, unsigned seq, float &x, float &y)
{
    unsigned long long u, w;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(u), "=l"(w) : "l"(a) : "memory");
    x = __uint_as_float((unsigned)u);
    y = __uint_as_float((unsigned)w);
    return (unsigned)(u >> 32) == seq && (unsigned)(w >> 32) == seq;
}

// A rim cell: where it lands in the staged planes, which of the tile's own
// cells goes out in exchange, and to which cell of the inboxes.
struct Rim {
    int to, from;       // staged offsets; to < 0: no such neighbour
    int out;            // inbox index of the cell sent (v; sigma's follows at + cells)
    bool x;             // left or right face: sigma's planes szx, sxx instead of szz, szx
};

// A quad of the thread: columns ix .. ix + 3 of the tile's row.
struct Quad {
    int ix;
    bool mine, keep;  // on the grid; its sums keep their roundings
    unsigned mask;    // interior columns
    float *z, *x;     // in the z and x strips' memories, null outside
    Q4 we, uz, ux;
    Q4 mz[4], mx[4];  // CPML memories of a thread with one quad
};

// CPML of one derivative: memory `o` in registers where the thread has one
// quad, else through L1 (only this thread reads and writes it in the launch).
template <int QPT>
__device__ __forceinline__ void cpml_at(Q4 &o, float *m, const Q4 &a, const Q4 &b, const Q4 &ki, Q4 &d, unsigned mask)
{
    if constexpr (QPT > 1) o = lds4(m);
    cpml_quad(o, a, b, ki, d, mask);
    if constexpr (QPT > 1) st4(m, o);
}

template <int NS, int QPT, int MODE>
__global__ void __launch_bounds__(MAX_THREADS, 1)
    k_resident(const __grid_constant__ StepParams<float> p, const __grid_constant__ SrcRecParams<float> q,
               const __grid_constant__ ResidentRun g)
{
    constexpr bool U = has_u<MODE>(), WE = has_we<MODE>(), FWD = MODE != MODE_ADJ;
    constexpr int RW = 32 * QPT, RS = staged_row(RW);
    extern __shared__ __align__(16) float sm[];
    const LoopRun &run = g.r;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x;
    const int c = blockIdx.x % g.ntx, bc = blockIdx.x / g.ntx, b = bc % g.ntz, bz = bc / g.ntz;
    if (bz >= p.ctl[1]) return;  // the last batch may hold fewer shots
    const int tz = g.tz, HP = (tz + 2 * NS) * RS, KP = tz * RW, cells = rim_cells(NS, RW, tz);
    const int x0 = c * RW, z0 = b * tz;
    float *sv = sm, *ss = sm + 2 * HP, *kept = sm + 5 * HP;
    const int lr = tid >> 3, qc = 4 * (tid & 7);
    const int iz = z0 + lr;
    const int o0 = (lr + NS) * RS + HX + qc;  // the first quad in a staged plane; the next 32 columns on
    const int ko0 = lr * RW + qc;             // ... and in a plane of kept roundings
    float *fs = p.fld + (long long)bz * p.shot_stride;
    float *fk = fs + (long long)p.pp_planes * p.plane;  // kept roundings between launches
    Quad quad[QPT];
#pragma unroll
    for (int j = 0; j < QPT; j++) {
        Quad &t = quad[j];
        t.ix = x0 + qc + 32 * j;
        t.mine = lr < tz && iz < p.nz && t.ix < p.nx;
        t.mask = t.mine && iz >= p.nz1 && iz < p.nz2 ? inner_mask(p, t.ix) : 0;
        t.keep = FWD && t.mine && run.keep && run.keep[iz / 16 * ((p.nx + 63) / 64) + t.ix / 64];
        t.z = t.x = nullptr;
        t.we = t.uz = t.ux = all4(0.f);
    }

    // ---- what stays on chip, from the field block
    for (int e = tid; e < 5 * HP + 5 * KP; e += nthr) sm[e] = 0.f;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < QPT; j++) {
        Quad &t = quad[j];
        const int o = o0 + 32 * j, ko = ko0 + 32 * j, i = iz * p.pitch + t.ix;
        if (t.mine) {
#pragma unroll
            for (int k = 0; k < 5; k++) st4(sm + k * HP + o, ldg4(fs + i + (F_VZ + k) * p.plane));
            if (t.keep)
#pragma unroll
                for (int k = 0; k < 5; k++) st4(kept + k * KP + ko, ldg4(fk + i + (F_VZ + k) * p.plane));
            if constexpr (WE) t.we = ldg4(fs + i + (FWD ? F_WE : F_WEA) * p.plane);
            if constexpr (U) {
                t.uz = ldg4(fs + i + F_UZ * p.plane);
                t.ux = ldg4(fs + i + F_UX * p.plane);
            }
        }
        if (!t.mask) continue;
        if (iz < p.pz0 || iz >= p.pz1) {
            const int rr = iz < p.pz0 ? iz : iz - p.pz1 + p.pz0;
            t.z = p.memz + (long long)bz * p.mz_shot_stride + (long long)rr * p.pitch + t.ix;
            if constexpr (QPT == 1)
#pragma unroll
                for (int k = 0; k < 4; k++) t.mz[k] = ldg4(t.z + k * p.mz_plane);
        }
        if (t.ix < p.px0 || t.ix >= p.px1) {
            const int cc = t.ix < p.px0 ? t.ix : t.ix - p.px1 + p.px0;
            t.x = p.memx + (long long)bz * p.mx_shot_stride + (long long)iz * p.mx_pitch + cc;
            if constexpr (QPT == 1)
#pragma unroll
                for (int k = 0; k < 4; k++) t.mx[k] = ldg4(t.x + k * p.mx_plane);
        }
    }
    // ---- the rim: faces above, below, left, right
    Rim rim[2];
    const ulonglong2 *in = g.inbox + (long long)blockIdx.x * 2 * cells;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int e = tid + k * nthr;
        rim[k].to = -1;
        if (e >= cells) continue;
        const int zf = NS * RW, xf = NS * tz;  // cells of a face
        rim[k].x = e >= 2 * zf;
        int nb, back;
        bool there;
        if (!rim[k].x) {
            const int face = e / zf, w = e % zf, r = w / RW, col = HX + w % RW;
            there = face ? b + 1 < g.ntz : b > 0;
            nb = face ? g.ntx : -g.ntx;
            back = (1 - face) * zf + w;
            rim[k].to = (face ? NS + tz + r : r) * RS + col;
            rim[k].from = (face ? tz + r : NS + r) * RS + col;
        } else {
            const int w2 = e - 2 * zf, face = w2 / xf, w = w2 % xf, row = NS + w / NS, r = w % NS;
            there = face ? c + 1 < g.ntx : c > 0;
            nb = face ? 1 : -1;
            back = 2 * zf + (1 - face) * xf + w;
            rim[k].to = row * RS + (face ? HX + RW + r : HX - NS + r);
            rim[k].from = row * RS + (face ? HX + RW - NS + r : HX + r);
        }
        if (!there) {
            rim[k].to = -1;
            continue;
        }
        rim[k].out = ((int)blockIdx.x + nb) * 2 * cells + back;
        // the launch's first halo of v, where the grid has it
        const int gz = z0 + rim[k].to / RS - NS, gx = x0 + rim[k].to % RS - HX;
        if (gz >= 0 && gz < p.nz && gx >= 0 && gx < p.nx) {
            const float *h = p.fld + (long long)bz * p.shot_stride + (long long)gz * p.pitch + gx;
            sv[rim[k].to] = __ldcg(h + F_VZ * p.plane);
            sv[HP + rim[k].to] = __ldcg(h + F_VX * p.plane);
        }
    }
    auto send_rim = [&](const float *pl, bool sigma, unsigned seq) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (rim[k].to < 0) continue;
            const float *a = pl + rim[k].from + (sigma && rim[k].x ? HP : 0);
            send(g.inbox + rim[k].out + (sigma ? cells : 0), a[0], a[HP], seq);
        }
    };
    auto receive_rim = [&](float *pl, bool sigma, unsigned seq) {
        const ulonglong2 *src = in + (sigma ? cells : 0) + tid;
        bool w0 = rim[0].to >= 0, w1 = rim[1].to >= 0;
        float x[2], y[2];
        unsigned long long t0 = 0;
        for (int n = 0; w0 || w1; n++) {
            if (w0) w0 = !poll(src, seq, x[0], y[0]);
            if (w1) w1 = !poll(src + nthr, seq, x[1], y[1]);
            if ((n & 255) == 255) {
                const unsigned long long t = now_ns();
                if (!t0) t0 = t;
                else if (t - t0 > WAIT_LIMIT_NS) return true;
            }
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (rim[k].to < 0) continue;
            float *a = pl + rim[k].to + (sigma && rim[k].x ? HP : 0);
            a[0] = x[k];
            a[HP] = y[k];
        }
        return false;
    };
    // ---- the tile's sources (first warp) and receivers (last warp)
    const TileSR e = tile_srcrec(q, p.ctl[0], b * g.ntx + c, bz);
    const int shot = p.ctl[0] + bz;
    const double amp = q.src_kind >= 0 ? q.amp_scale[shot] : 0.0;
    struct Src {
        int pos, col;
        float rz, rx;  // buoyancies of a force
    };
    auto source = [&](int k) {
        Src s{0, 0, 1.f, 1.f};
        if (q.src_kind == 0) {
            const int j = q.t_src_k[k];
            s.pos = q.src_pos[j];
            s.col = q.src_col[j];
        } else {
            s.col = q.t_rec_r[k];
            s.pos = q.rec_pos[s.col];
        }
        if (q.stf_type == 0) {
            s.rz = p.c_rz[s.pos];
            s.rx = p.c_rx[s.pos];
        }
        return s;
    };
    auto scaled = [&](double x, float buoyancy) {
        return q.stf_type == 0 ? buoyancy * (float)(x * amp * q.inv_dzdx) : (float)(x * amp);
    };
    auto amplitude = [&](const double *stf, int it, int col, float buoyancy) {
        return scaled(stf[(long long)it * q.stf_ncol + col], buoyancy);
    };
    auto local = [&](int pos) {  // staged offset of a grid cell of the tile
        const int z = pos / p.pitch;
        return (z - z0 + NS) * RS + HX + pos - z * p.pitch - x0;
    };
    const bool sources = e.k0 < e.k1, shooter = warp == 0, recorder = warp == nthr / 32 - 1;
    Src s0{};
    if (shooter && e.k0 + lane < e.k1) s0 = source(e.k0 + lane);
    const double *stz = q.stf_z + shot * q.stf_shot_stride, *stx = q.stf_x + shot * q.stf_shot_stride;
    double *rtz = q.rtf_z + shot * q.rtf_shot_stride, *rtx = q.rtf_x + shot * q.rtf_shot_stride;
    // the running sums of a lane's first receiver stay in registers
    double r0z = 0.0, r0x = 0.0, ru = 0.0;
    int r0 = -1, r0o = 0;
    if (recorder && e.r0 < e.r1) {
        ru = q.dt_d / q.dzdx * q.rec_unscale[shot];  // FP64 divides are slow: once, not in every step
        if (e.r0 + lane < e.r1) {
            r0 = q.t_rec_r[e.r0 + lane];
            r0o = local(q.rec_pos[r0]);
            if (run.it0) {
                r0z = __ldcg(rtz + (long long)(run.it0 - 1) * q.nrec + r0);
                r0x = __ldcg(rtx + (long long)(run.it0 - 1) * q.nrec + r0);
            }
        }
    }
    __syncthreads();

    // A mirrored row's szz and szx are other threads' to write while its own
    // reads stresses: it reads v in their place, and writes neither.  (One
    // offset for the launch: 2.75 us a step on 101 x 201, 2.83 with loads under
    // a predicate in each step.)
    const int own0 = surface_own(iz, p.st) ? o0 : o0 - 2 * HP;
    bool failed = false;
    for (int k = 0; k < run.nsteps; k++) {
        const int it = run.it0 + k * run.dit, rel = it / run.sdt;
        const int slot = run.snap && rel * run.sdt == it ? (rel - run.base) % run.ring : -1;
        // ahead of their use: the step's amplitudes, and the snapshot it images
        double az = 0.0, ax = 0.0;
        if (shooter && e.k0 + lane < e.k1) {
            az = stz[(long long)it * q.stf_ncol + s0.col];
            ax = stx[(long long)it * q.stf_ncol + s0.col];
        }
        if constexpr (!FWD)
            if (slot >= 0 && p.snap_dx == 1) {
                const int dzr = iz - p.snap_z1;
                const float *row = p.hist + (long long)bz * p.hist_shot_stride + (long long)slot * p.hist_slot_stride +
                                   (long long)(dzr / p.snap_dz) * p.snx_pitch;
#pragma unroll
                for (int j = 0; j < QPT; j++) {
                    const int w = quad[j].ix - p.snap_x1;
                    if (quad[j].mine && dzr >= 0 && iz <= p.snap_z2 && dzr % p.snap_dz == 0 && w >= 0 && w < p.snx)
#pragma unroll
                        for (int n = 0; n < NHIST; n++)
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(row + w + n * p.snap_plane));
                }
            }
        if (k) {
            failed = receive_rim(sv, false, 2 * k);
            if (__syncthreads_or(failed)) break;
        }
        // ---- stress: vdiff2 + pml_diff2 + update_s2 + surf_mirror
        // (src/cpu/n_kernel_lib_PSV.cpp:100-205, 272-395).  A top free surface
        // and the rows it mirrors lie in the first band of tiles.
#pragma unroll
        for (int j_ = 0; j_ < QPT; j_++) {
            Quad &t = quad[j_];
            if (!t.mask) continue;
            const unsigned mask = t.mask;
            const bool keep = t.keep;
            const int ix = t.ix, o = o0 + 32 * j_, i = iz * p.pitch + ix;
            const Q4 cl = ldro4(p.c_lam + i), c2 = ldro4(p.c_l2m + i), cm = ldro4(p.c_muzx + i);
            const float *hz = sv + o - NS * RS, *hx = hz + HP;
            Q4 zz, xx, zx, xz;  // vz_z, vx_x, vz_x, vx_z
            float h[12];
            {
                Q4 w[2 * NS];
#pragma unroll
                for (int j = 0; j < 2 * NS; j++) w[j] = lds4(hz + j * RS);
                row12(hz + NS * RS, w[NS], h);
                zz = dvert<NS>(w, p.cz);
                zx = dhorz<NS, 1>(h, p.cx);
            }
            {
                Q4 w[2 * NS];
#pragma unroll
                for (int j = 0; j < 2 * NS; j++) w[j] = lds4(hx + (j + 1) * RS);
                row12(hx + NS * RS, w[NS - 1], h);
                xz = dvert<NS>(w, p.cz);
                xx = dhorz<NS, 0>(h, p.cx);
            }
            if (t.z) {
                cpml_at<QPT>(t.mz[MZ_VZ], t.z + MZ_VZ * p.mz_plane, all4(p.a_z[iz]), all4(p.b_z[iz]), all4(p.ki_z[iz]), zz, mask);
                cpml_at<QPT>(t.mz[MZ_VX], t.z + MZ_VX * p.mz_plane, all4(p.ah_z[iz]), all4(p.bh_z[iz]), all4(p.khi_z[iz]), xz, mask);
            }
            if (t.x) {
                cpml_at<QPT>(t.mx[MX_VX], t.x + MX_VX * p.mx_plane, ldro4(p.a_x + ix), ldro4(p.b_x + ix), ldro4(p.ki_x + ix), xx, mask);
                cpml_at<QPT>(t.mx[MX_VZ], t.x + MX_VZ * p.mx_plane, ldro4(p.ah_x + ix), ldro4(p.bh_x + ix), ldro4(p.khi_x + ix), zx, mask);
            }
            const bool image = surface_image(iz, p.st);
            const float *own = ss + own0 + 32 * j_;
            Q4 szz = lds4(own), szx = lds4(own + HP), sxx = lds4(ss + 2 * HP + o);
            if (FWD && keep) {
                float *r = kept + (F_SZZ - F_VZ) * KP + ko0 + 32 * j_;
                Q4 rzz = lds4(r), rzx = lds4(r + KP), rxx = lds4(r + 2 * KP);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (!(mask >> j & 1)) continue;
                    keep_sum(szz.v[j], rzz.v[j], fmaf(c2.v[j], zz.v[j], fmaf(cl.v[j], xx.v[j], rzz.v[j])));
                    keep_sum(sxx.v[j], rxx.v[j], fmaf(c2.v[j], xx.v[j], fmaf(cl.v[j], zz.v[j], rxx.v[j])));
                    keep_sum(szx.v[j], rzx.v[j], fmaf(cm.v[j], zx.v[j] + xz.v[j], rzx.v[j]));
                    if (image) rzz.v[j] = rzx.v[j] = rxx.v[j] = 0.f;
                }
                st4(r, rzz);
                st4(r + KP, rzx);
                st4(r + 2 * KP, rxx);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (!(mask >> j & 1)) continue;
                if (!FWD || !keep) {
                    szz.v[j] += fmaf(c2.v[j], zz.v[j], cl.v[j] * xx.v[j]);
                    sxx.v[j] += fmaf(c2.v[j], xx.v[j], cl.v[j] * zz.v[j]);
                    szx.v[j] = fmaf(cm.v[j], zx.v[j] + xz.v[j], szx.v[j]);
                }
                if (image) {
                    szz.v[j] = szx.v[j] = 0.f;
                    sxx.v[j] = p.fs_top[ix + j] * xx.v[j];
                }
            }
            if (surface_own(iz, p.st)) {
                st4(ss + o, szz);
                st4(ss + HP + o, szx);
            }
            st4(ss + 2 * HP + o, sxx);
            if (surface_mirrors(iz, p.st, p.nz1)) {
                float *d = ss + (2 * p.st - iz - z0 + NS) * RS + HX + ix - x0;
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (mask >> j & 1) {
                        d[j] = -szz.v[j];
                        d[HP + j] = -szx.v[j];
                    }
            }
        }
        __syncthreads();
        send_rim(ss, true, 2 * k + 1);
        float a = 0.f, d = 0.f;  // the lane's first source
        if (shooter && sources) {
            a = scaled(az, s0.rz);
            d = scaled(ax, s0.rx);
        }
        failed = receive_rim(ss, true, 2 * k + 1);
        if (__syncthreads_or(failed)) break;
        // ---- velocity: sdiff2 + pml_diff2 + update_v2
        // (src/cpu/n_kernel_lib_PSV.cpp:207-270)
#pragma unroll
        for (int j_ = 0; j_ < QPT; j_++) {
            Quad &t = quad[j_];
            if (!t.mask) continue;
            const unsigned mask = t.mask;
            const bool keep = t.keep;
            const int ix = t.ix, o = o0 + 32 * j_, i = iz * p.pitch + ix;
            const float *azz = ss + o - NS * RS, *azx = azz + HP, *axx = azx + HP;
            Q4 vz = lds4(sv + o), vx = lds4(sv + HP + o);
            const Q4 crz = ldro4(p.c_rz + i), crx = ldro4(p.c_rx + i);
            Q4 zz_z, zx_z, zx_x, xx_x;
            float h[12];
            {
                Q4 w[2 * NS];
#pragma unroll
                for (int j = 0; j < 2 * NS; j++) w[j] = lds4(azz + (j + 1) * RS);
                zz_z = dvert<NS>(w, p.cz);
            }
            {
                Q4 w[2 * NS];
#pragma unroll
                for (int j = 0; j < 2 * NS; j++) w[j] = lds4(azx + j * RS);
                row12(azx + NS * RS, w[NS], h);
                zx_z = dvert<NS>(w, p.cz);
                zx_x = dhorz<NS, 0>(h, p.cx);
            }
            row12(axx + NS * RS, lds4(axx + NS * RS), h);
            xx_x = dhorz<NS, 1>(h, p.cx);
            if (t.z) {
                cpml_at<QPT>(t.mz[MZ_SZZ], t.z + MZ_SZZ * p.mz_plane, all4(p.a_z[iz]), all4(p.b_z[iz]), all4(p.ki_z[iz]), zz_z, mask);
                cpml_at<QPT>(t.mz[MZ_SZX], t.z + MZ_SZX * p.mz_plane, all4(p.ah_z[iz]), all4(p.bh_z[iz]), all4(p.khi_z[iz]), zx_z, mask);
            }
            if (t.x) {
                cpml_at<QPT>(t.mx[MX_SXX], t.x + MX_SXX * p.mx_plane, ldro4(p.a_x + ix), ldro4(p.b_x + ix), ldro4(p.ki_x + ix), xx_x, mask);
                cpml_at<QPT>(t.mx[MX_SZX], t.x + MX_SZX * p.mx_plane, ldro4(p.ah_x + ix), ldro4(p.bh_x + ix), ldro4(p.khi_x + ix), zx_x, mask);
            }
            Q4 rz = all4(0.f), rx = all4(0.f);
            float *r = kept + ko0 + 32 * j_;
            if (FWD && keep) {
                rz = lds4(r);
                rx = lds4(r + KP);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (!(mask >> j & 1)) continue;
                if constexpr (U) {
                    t.uz.v[j] = fmaf(p.dt, vz.v[j], t.uz.v[j]);
                    t.ux.v[j] = fmaf(p.dt, vx.v[j], t.ux.v[j]);
                }
                if (!FWD || !keep) {
                    vz.v[j] = fmaf(crz.v[j], zx_x.v[j] + zz_z.v[j], vz.v[j]);
                    vx.v[j] = fmaf(crx.v[j], xx_x.v[j] + zx_z.v[j], vx.v[j]);
                } else {
                    keep_sum(vz.v[j], rz.v[j], fmaf(crz.v[j], zx_x.v[j] + zz_z.v[j], rz.v[j]));
                    keep_sum(vx.v[j], rx.v[j], fmaf(crx.v[j], xx_x.v[j] + zx_z.v[j], rx.v[j]));
                }
                if constexpr (WE) t.we.v[j] += fmaf(vx.v[j], vx.v[j], vz.v[j] * vz.v[j]);
            }
            st4(sv + o, vz);
            st4(sv + HP + o, vx);
            if (FWD && keep) {
                st4(r, rz);
                st4(r + KP, rx);
            }
        }
        __syncthreads();
        // ---- vsrc2 (src/cpu/n_kernel_lib_PSV.cpp:487-531) on the new velocities
        if (sources) {
            if (shooter)
                for (int k0 = e.k0; k0 < e.k1; k0 += 32) {
                    const int n = min(32, e.k1 - k0);
                    Src s = s0;
                    if (k0 != e.k0 && lane < n) {
                        s = source(k0 + lane);
                        a = amplitude(stz, it, s.col, s.rz);
                        d = amplitude(stx, it, s.col, s.rx);
                    }
                    const int at = lane < n ? local(s.pos) : 0;
                    if (FWD && run.keep) {  // in order: sources may share a cell
                        const int cell = (at / RS - NS) * RW + at % RS - HX;
                        // (those on one cell, each in its turn; a source at a time: 10.4 us
                        // a step with 64 on 8 x 8 cells of 301 x 601, one shot; so 5.2)
                        int turn = lane, turns = n;
                        if (n > 4) {
                            const unsigned same = __match_any_sync(0xffffffffu, lane < n ? at : -1 - lane);
                            turn = __popc(same & ((1u << lane) - 1));
                            turns = __reduce_max_sync(0xffffffffu, turn) + 1;
                        }
                        for (int j = 0; j < turns; j++) {
                            if (turn == j && lane < n) {
                                keep_sum(sv[at], kept[cell], a + kept[cell]);
                                keep_sum(sv[HP + at], kept[KP + cell], d + kept[KP + cell]);
                            }
                            __syncwarp();
                        }
                    } else if (lane < n) {
                        atomicAdd(sv + at, a);
                        atomicAdd(sv + HP + at, d);
                    }
                }
            __syncthreads();
        }
        if (k + 1 < run.nsteps) send_rim(sv, false, 2 * k + 2);
        // ---- while the rims travel: snapshot store (its velocities are the
        // injected ones) or imaging (src/cpu/n_kernel_lib_PSV.cpp:398-484)
        if (slot >= 0)
#pragma unroll
            for (int j = 0; j < QPT; j++) {
                const int o = o0 + 32 * j;
                if (quad[j].mine)
                    snapshot_quad<MODE>(p, bz, iz, quad[j].ix, slot, lds4(ss + o), lds4(ss + HP + o),
                                        lds4(ss + 2 * HP + o), lds4(sv + o), lds4(sv + HP + o), quad[j].uz, quad[j].ux);
            }
        // ---- urec2 (src/cpu/n_kernel_lib_PSV.cpp:533-576)
        if (recorder && e.r0 < e.r1) {
            const long long row = (long long)it * q.nrec;
            if (r0 >= 0) {
                r0z = fma(ru, (double)sv[r0o], r0z);
                r0x = fma(ru, (double)sv[HP + r0o], r0x);
                rtz[row + r0] = r0z;
                rtx[row + r0] = r0x;
            }
            for (int j = e.r0 + 32 + lane; j < e.r1; j += 32) {
                const int rr = q.t_rec_r[j], at = local(q.rec_pos[rr]);
                const double pz = it ? __ldcg(rtz + row - q.nrec + rr) : 0.0;
                const double px = it ? __ldcg(rtx + row - q.nrec + rr) : 0.0;
                rtz[row + rr] = fma(ru, (double)sv[at], pz);
                rtx[row + rr] = fma(ru, (double)sv[HP + at], px);
            }
        }
    }
    if (failed) atomicExch(p.err, 1);
    // ---- back to the field block
#pragma unroll
    for (int j = 0; j < QPT; j++) {
        const Quad &t = quad[j];
        const int o = o0 + 32 * j, ko = ko0 + 32 * j, i = iz * p.pitch + t.ix;
        if (t.mine) {
#pragma unroll
            for (int k = 0; k < 5; k++) st4(fs + i + (F_VZ + k) * p.plane, lds4(sm + k * HP + o));
            if (t.keep)
#pragma unroll
                for (int k = 0; k < 5; k++) st4(fk + i + (F_VZ + k) * p.plane, lds4(kept + k * KP + ko));
            if constexpr (WE) st4(fs + i + (FWD ? F_WE : F_WEA) * p.plane, t.we);
            if constexpr (U) {
                st4(fs + i + F_UZ * p.plane, t.uz);
                st4(fs + i + F_UX * p.plane, t.ux);
            }
        }
        if (QPT == 1 && t.z)
#pragma unroll
            for (int k = 0; k < 4; k++) st4(t.z + k * p.mz_plane, t.mz[k]);
        if (QPT == 1 && t.x)
#pragma unroll
            for (int k = 0; k < 4; k++) st4(t.x + k * p.mx_plane, t.mx[k]);
    }
}

// Lowers *held to the CTAs of tz rows that the current device holds at once.
template <int NS, int QPT, int MODE> cudaError_t held_m(int tz, int nsm, int *held)
{
    constexpr int RW = 32 * QPT;
    auto kernel = k_resident<NS, QPT, MODE>;
    static PerDevice<cudaError_t> opted;
    int per = 0;
    cudaError_t e = opt_in(opted, kernel, resident_smem(NS, RW, MAX_THREADS / 8));
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, resident_threads(NS, RW, tz),
                                                          resident_smem(NS, RW, tz));
    *held = e == cudaSuccess ? std::min(*held, per * nsm) : 0;
    return e;
}
template <int NS, int QPT> int held_q(int tz, int nsm)
{
    int held = 1 << 30;
    const cudaError_t e[] = {held_m<NS, QPT, MODE_FWD>(tz, nsm, &held), held_m<NS, QPT, MODE_FWD_NOWE>(tz, nsm, &held),
                             held_m<NS, QPT, MODE_FWD_U>(tz, nsm, &held), held_m<NS, QPT, MODE_ADJ>(tz, nsm, &held)};
    for (cudaError_t x : e)
        if (x != cudaSuccess) held = 0;
    if (!held) (void)cudaGetLastError();
    return held;
}

template <int NS, int QPT, int MODE>
cudaError_t resident_m(const StepParams<float> &p, const SrcRecParams<float> &q, const ResidentRun &g, int nbatch,
                       cudaStream_t st)
{
    constexpr int RW = 32 * QPT;
    auto kernel = k_resident<NS, QPT, MODE>;
    static PerDevice<cudaError_t> opted;
    cudaError_t e = opt_in(opted, kernel, resident_smem(NS, RW, MAX_THREADS / 8));
    if (e != cudaSuccess) return e;
    const int ctas = g.ntx * g.ntz * nbatch;
    e = cudaMemsetAsync(g.inbox, 0, (size_t)ctas * 2 * rim_cells(NS, RW, g.tz) * sizeof(ulonglong2), st);
    if (e != cudaSuccess) return e;
    StepParams<float> a = p;
    SrcRecParams<float> s = q;
    ResidentRun r = g;
    void *args[] = {&a, &s, &r};
    return cudaLaunchCooperativeKernel(kernel, dim3(ctas), dim3(resident_threads(NS, RW, g.tz)), args,
                                       (size_t)resident_smem(NS, RW, g.tz), st);
}

template <int NS, int QPT>
cudaError_t resident_q(const StepParams<float> &p, const SrcRecParams<float> &q, const ResidentRun &g, int mode,
                       int nbatch, cudaStream_t st)
{
    switch (mode) {
    case MODE_FWD: return resident_m<NS, QPT, MODE_FWD>(p, q, g, nbatch, st);
    case MODE_FWD_NOWE: return resident_m<NS, QPT, MODE_FWD_NOWE>(p, q, g, nbatch, st);
    case MODE_FWD_U: return resident_m<NS, QPT, MODE_FWD_U>(p, q, g, nbatch, st);
    case MODE_ADJ: return resident_m<NS, QPT, MODE_ADJ>(p, q, g, nbatch, st);
    default: return cudaErrorInvalidValue;
    }
}

template <int NS>
cudaError_t resident_n(const StepParams<float> &p, const SrcRecParams<float> &q, const ResidentRun &g, int mode, int rw,
                       int nbatch, cudaStream_t st)
{
    return rw == 32 ? resident_q<NS, 1>(p, q, g, mode, nbatch, st) : resident_q<NS, 2>(p, q, g, mode, nbatch, st);
}

}  // namespace

// Tiles that give every CTA of a batch a place on `nsm` SMs at once: 32
// columns (one quad a thread) if the batch then fits, else 64 (two); the
// fewest rows from 8 (the mirrored rows of a top surface must fit) that need
// one CTA per SM, else the fewest with which as many as fit are enough.  tz =
// 0 if nothing is, or with other surfaces, whose mirrored cells cross tiles.
// 512 threads of 128 registers fill an SM.
ResidentTile resident_tile(int nz, int nx, int nbatch, int ns, int st, int sb, int sl, int sr, int nz1, int nsm)
{
    if (ns < 1 || ns > HX || sb || sl || sr) return {0, 0};
    for (int rw : {32, 64}) {
        const int ntx = (nx + rw - 1) / rw;
        for (int most : {1, 4})
            for (int tz = 8; tz <= MAX_THREADS / 8; tz++) {
                if (st && 2 * st - nz1 >= tz) continue;
                const long long ctas = (long long)ntx * ((nz + tz - 1) / tz) * nbatch;
                const int per = std::min({most, MAX_THREADS / resident_threads(ns, rw, tz),
                                          227 * 1024 / (resident_smem(ns, rw, tz) + 1024)});
                if (ctas <= (long long)nsm * per) return {rw, tz};
            }
    }
    return {0, 0};
}

// Whether the current device holds all CTAs of a batch at once, by its own
// account: a launch that it cannot hold is refused.
bool resident_held(int nz, int nx, int nbatch, int ns, const ResidentTile &t, int nsm)
{
    const long long ctas = (long long)((nx + t.rw - 1) / t.rw) * ((nz + t.tz - 1) / t.tz) * nbatch;
    int held = 0;
    switch (ns) {
    case 1: held = t.rw == 32 ? held_q<1, 1>(t.tz, nsm) : held_q<1, 2>(t.tz, nsm); break;
    case 2: held = t.rw == 32 ? held_q<2, 1>(t.tz, nsm) : held_q<2, 2>(t.tz, nsm); break;
    case 3: held = t.rw == 32 ? held_q<3, 1>(t.tz, nsm) : held_q<3, 2>(t.tz, nsm); break;
    case 4: held = t.rw == 32 ? held_q<4, 1>(t.tz, nsm) : held_q<4, 2>(t.tz, nsm); break;
    }
    return ctas <= held;
}

size_t resident_inbox_bytes(int nz, int nx, int nbatch, int ns, const ResidentTile &t)
{
    return (size_t)((nx + t.rw - 1) / t.rw) * ((nz + t.tz - 1) / t.tz) * nbatch * 2 * rim_cells(ns, t.rw, t.tz) *
           sizeof(ulonglong2);
}

cudaError_t launch_resident(const StepParams<float> &p, const SrcRecParams<float> &q, const LoopRun &run, int ns,
                            int mode, const ResidentTile &t, int nbatch, cudaStream_t st)
{
    const ResidentRun g{run, t.tz, (p.nx + t.rw - 1) / t.rw, (p.nz + t.tz - 1) / t.tz,
                        reinterpret_cast<ulonglong2 *>(run.sync)};
    switch (ns) {
    case 1: return resident_n<1>(p, q, g, mode, t.rw, nbatch, st);
    case 2: return resident_n<2>(p, q, g, mode, t.rw, nbatch, st);
    case 3: return resident_n<3>(p, q, g, mode, t.rw, nbatch, st);
    case 4: return resident_n<4>(p, q, g, mode, t.rw, nbatch, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace psv
