// psv_quads.cuh -- four columns of one row per thread (FP32): staggered
// derivatives from a staged tile, CPML, the snapshot store / imaging sums and
// the sums that keep their roundings, shared by the kernels that run many time
// steps per launch (psv_loop.cu, psv_resident.cu).
#pragma once

#include "psv_kernels_impl.cuh"
#include "psv_surface.hpp"

namespace psv {
namespace {

constexpr int HX = 4;  // columns staged left and right of a tile

template <int MODE> __host__ __device__ constexpr bool has_u() { return MODE == MODE_ADJ || MODE == MODE_FWD_U; }
template <int MODE> __host__ __device__ constexpr bool has_we() { return MODE != MODE_FWD_NOWE; }

// ------------------------------------------------------------- quads
// Four neighbouring columns of one row.
struct Q4 {
    float v[4];
};
__device__ __forceinline__ Q4 lds4(const float *a)
{
    const float4 t = *reinterpret_cast<const float4 *>(a);
    return {{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ Q4 ldg4(const float *a)  // data other CTAs write: past L1
{
    const float4 t = __ldcg(reinterpret_cast<const float4 *>(a));
    return {{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ Q4 ldro4(const float *a)  // coefficients and profiles
{
    const float4 t = __ldg(reinterpret_cast<const float4 *>(a));
    return {{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ void st4(float *a, const Q4 &q)
{
    *reinterpret_cast<float4 *>(a) = make_float4(q.v[0], q.v[1], q.v[2], q.v[3]);
}

// s + y, with what the rounding of s dropped added into y first (r) and what
// it drops now kept in r (Knuth's two-sum).  The tiles around sources and
// receivers sum this way on forward passes: rounding the large amplitudes
// there is nine tenths of a trace's FP32 error, and a gradient multiplies it
// by traces / residual.  Traces of the 301 x 601 and 401 x 801 surveys: 1.0e-7
// and 2.0e-7 of their norm off without, 0.2e-7 and 0.4e-7 with it, for one
// band of tiles in 19 or more.
__device__ __forceinline__ void keep_sum(float &s, float &r, float y)
{
    const float t = s + y, b = t - s;
    r = (s - (t - b)) + (y - b);
    s = t;
}

// Staggered derivatives, summed from the outermost (smallest) term inwards so
// that only the leading term's rounding counts.
// Vertical, rows w[0 .. 2 NS): sum c_k (w[NS + k - 1] - w[NS - k]).
template <int NS>
__device__ __forceinline__ Q4 dvert(const Q4 *w, const float *c)
{
    Q4 o;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        float a = c[NS - 1] * (w[2 * NS - 1].v[j] - w[0].v[j]);
#pragma unroll
        for (int k = NS - 1; k >= 1; k--) a = fmaf(c[k - 1], w[NS + k - 1].v[j] - w[NS - k].v[j], a);
        o.v[j] = a;
    }
    return o;
}
// Horizontal over h[0 .. 12) = columns ix - 4 .. ix + 7: AHEAD = 1 forward
// (f[+k] - f[-k+1]), 0 backward (f[+k-1] - f[-k]).
template <int NS, int AHEAD>
__device__ __forceinline__ Q4 dhorz(const float *h, const float *c)
{
    Q4 o;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float *f = h + 4 + j + AHEAD;
        float a = c[NS - 1] * (f[NS - 1] - f[-NS]);
#pragma unroll
        for (int k = NS - 1; k >= 1; k--) a = fmaf(c[k - 1], f[k - 1] - f[-k], a);
        o.v[j] = a;
    }
    return o;
}
// Columns ix - 4 .. ix + 7 of a staged row around the quad `mid`.
__device__ __forceinline__ void row12(const float *a, const Q4 &mid, float *h)
{
    const Q4 l = lds4(a - 4), r = lds4(a + 4);
#pragma unroll
    for (int j = 0; j < 4; j++) { h[j] = l.v[j]; h[4 + j] = mid.v[j]; h[8 + j] = r.v[j]; }
}

// Which of the quad's four columns are interior (bit j: column ix + j).
__device__ __forceinline__ unsigned inner_mask(const StepParams<float> &p, int ix)
{
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (ix + j >= p.nx1 && ix + j < p.nx2) m |= 1u << j;
    return m;
}

// pml_diff2 (src/cpu/n_kernel_lib_PSV.cpp:134-178) of one derivative quad
// against its memory plane; columns outside `mask` keep their memory.
__device__ __forceinline__ void cpml_quad(Q4 &o, const Q4 &a, const Q4 &b, const Q4 &ki, Q4 &d, unsigned mask)
{
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float n = fmaf(b.v[j], o.v[j], a.v[j] * d.v[j]);
        d.v[j] = fmaf(d.v[j], ki.v[j], n);
        if (mask >> j & 1) o.v[j] = n;
    }
}
__device__ __forceinline__ void cpml_quad(float *m, const Q4 &a, const Q4 &b, const Q4 &ki, Q4 &d, unsigned mask)
{
    Q4 o = ldg4(m);
    cpml_quad(o, a, b, ki, d, mask);
    st4(m, o);
}
__device__ __forceinline__ Q4 all4(float x) { return {{x, x, x, x}}; }

// Both z-strip derivatives (planes m0, m1: on-point and half-point profiles)
// and both x-strip derivatives of a quad.  The strips' first and last columns
// are multiples of four, so a quad lies inside a strip or outside it.
__device__ __forceinline__ void cpml_quads(const StepParams<float> &p, int bz, int iz, int ix,
                                           unsigned mask, int z0, int z1, Q4 &dz0, Q4 &dz1, int x0,
                                           int x1, Q4 &dx0, Q4 &dx1)
{
    if (iz < p.pz0 || iz >= p.pz1) {
        const int rr = iz < p.pz0 ? iz : iz - p.pz1 + p.pz0;
        float *m = p.memz + (long long)bz * p.mz_shot_stride + (long long)rr * p.pitch + ix;
        cpml_quad(m + z0 * p.mz_plane, all4(p.a_z[iz]), all4(p.b_z[iz]), all4(p.ki_z[iz]), dz0, mask);
        cpml_quad(m + z1 * p.mz_plane, all4(p.ah_z[iz]), all4(p.bh_z[iz]), all4(p.khi_z[iz]), dz1, mask);
    }
    if (ix < p.px0 || ix >= p.px1) {
        const int c = ix < p.px0 ? ix : ix - p.px1 + p.px0;
        float *m = p.memx + (long long)bz * p.mx_shot_stride + (long long)iz * p.mx_pitch + c;
        cpml_quad(m + x0 * p.mx_plane, ldro4(p.a_x + ix), ldro4(p.b_x + ix), ldro4(p.ki_x + ix), dx0, mask);
        cpml_quad(m + x1 * p.mx_plane, ldro4(p.ah_x + ix), ldro4(p.bh_x + ix), ldro4(p.khi_x + ix), dx1, mask);
    }
}

// -------------------------------------------------------------- snapshots
// Elements [lo, hi) of the quad that lie in the snapshot window's columns.
__device__ __forceinline__ void st_window(float *a, const Q4 &q, int lo, int hi)
{
    if (lo == 0 && hi == 4) {
        __stcs(reinterpret_cast<float4 *>(a), make_float4(q.v[0], q.v[1], q.v[2], q.v[3]));
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (j >= lo && j < hi) __stcs(a + j, q.v[j]);
}
// Streaming loads: history and gradients are touched once per imaging step.
__device__ __forceinline__ Q4 ld_window(const float *a, int lo, int hi)
{
    if (lo == 0 && hi == 4) {
        float4 t;
        asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(t.x), "=f"(t.y), "=f"(t.z), "=f"(t.w)
                     : "l"(a));
        return {{t.x, t.y, t.z, t.w}};
    }
    Q4 q = all4(0.f);
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (j >= lo && j < hi) q.v[j] = __ldcg(a + j);
    return q;
}

// gard_fwd_storage2 / fwi_grad2 (src/cpu/n_kernel_lib_PSV.cpp:398-484) of one
// quad.  snap_dx = 1: the window's columns [lo, hi) of the quad, 16-byte
// aligned (the plan places the window's first column at its grid column
// modulo four); otherwise cell by cell.
template <int MODE>
__device__ __forceinline__ void snapshot_quad(const StepParams<float> &p, int bz, int iz, int ix,
                                              int slot, const Q4 &ozz, const Q4 &ozx, const Q4 &oxx,
                                              const Q4 &vz, const Q4 &vx, const Q4 &uz, const Q4 &ux)
{
    const int dzr = iz - p.snap_z1;
    if (dzr < 0 || iz > p.snap_z2 || dzr % p.snap_dz) return;
    const int lo = max(0, p.snap_x1 - ix), hi = min(4, p.snap_x2 + 1 - ix);
    if (lo >= hi) return;
    const long long sp = p.snap_plane;
    const long long row = (long long)(dzr / p.snap_dz) * p.snx_pitch;
    float *hb = p.hist + (long long)bz * p.hist_shot_stride + (long long)slot * p.hist_slot_stride + row;
    float *gb = p.gshot + (long long)bz * p.gshot_shot_stride + row;
    const long long i = (long long)iz * p.pitch + ix;
    if (p.snap_dx == 1) {
        float *h = hb + (ix - p.snap_x1);
        if constexpr (MODE != MODE_ADJ) {
            Q4 a, b;
#pragma unroll
            for (int j = 0; j < 4; j++) { a.v[j] = vz.v[j] * p.inv_dt; b.v[j] = vx.v[j] * p.inv_dt; }
            st_window(h + H_SZZ * sp, ozz, lo, hi);
            st_window(h + H_SZX * sp, ozx, lo, hi);
            st_window(h + H_SXX * sp, oxx, lo, hi);
            st_window(h + H_VZ * sp, a, lo, hi);
            st_window(h + H_VX * sp, b, lo, hi);
        } else {
            float *g = gb + (ix - p.snap_x1);
            const Q4 fzz = ld_window(h + H_SZZ * sp, lo, hi), fzx = ld_window(h + H_SZX * sp, lo, hi);
            const Q4 fxx = ld_window(h + H_SXX * sp, lo, hi), fvz = ld_window(h + H_VZ * sp, lo, hi);
            const Q4 fvx = ld_window(h + H_VX * sp, lo, hi);
            Q4 gl = ld_window(g, lo, hi), gm = ld_window(g + sp, lo, hi), gr = ld_window(g + 2 * sp, lo, hi);
            const Q4 g1 = ldro4(p.g1 + i), g2 = ldro4(p.g2 + i);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float s1 = g1.v[j] * ((fzz.v[j] + fxx.v[j]) * (ozz.v[j] + oxx.v[j]));
                const float s23 = g2.v[j] * fmaf(fzx.v[j], ozx.v[j],
                                                 0.25f * ((fzz.v[j] - fxx.v[j]) * (ozz.v[j] - oxx.v[j])));
                gl.v[j] -= s1;
                gm.v[j] -= s23 + s1;
                gr.v[j] = fmaf(-p.kimg, fmaf(ux.v[j], fvx.v[j], uz.v[j] * fvz.v[j]), gr.v[j]);
            }
            st_window(g, gl, lo, hi);
            st_window(g + sp, gm, lo, hi);
            st_window(g + 2 * sp, gr, lo, hi);
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int dxr = ix + j - p.snap_x1;
        if (j < lo || j >= hi || dxr % p.snap_dx) continue;
        float *h = hb + dxr / p.snap_dx;
        if constexpr (MODE != MODE_ADJ) {
            st_once(h + H_SZZ * sp, ozz.v[j]);
            st_once(h + H_SZX * sp, ozx.v[j]);
            st_once(h + H_SXX * sp, oxx.v[j]);
            st_once(h + H_VZ * sp, vz.v[j] * p.inv_dt);
            st_once(h + H_VX * sp, vx.v[j] * p.inv_dt);
        } else {
            float *g = gb + dxr / p.snap_dx;
            const float fzz = __ldcg(h + H_SZZ * sp), fzx = __ldcg(h + H_SZX * sp), fxx = __ldcg(h + H_SXX * sp);
            const float fvz = __ldcg(h + H_VZ * sp), fvx = __ldcg(h + H_VX * sp);
            const float s1 = p.g1[i + j] * ((fzz + fxx) * (ozz.v[j] + oxx.v[j]));
            const float s23 = p.g2[i + j] * fmaf(fzx, ozx.v[j], 0.25f * ((fzz - fxx) * (ozz.v[j] - oxx.v[j])));
            __stcs(g, __ldcg(g) - s1);
            __stcs(g + sp, __ldcg(g + sp) - (s23 + s1));
            __stcs(g + 2 * sp, fmaf(-p.kimg, fmaf(ux.v[j], fvx, uz.v[j] * fvz), __ldcg(g + 2 * sp)));
        }
    }
}

}  // namespace
}  // namespace psv
