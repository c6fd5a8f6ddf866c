// psv_surface.hpp -- the rows beside a top free surface (host and device).
#pragma once

#ifdef __CUDACC__
#define PSV_HD __host__ __device__ __forceinline__
#else
#define PSV_HD inline
#endif

namespace psv {

// What interior row iz has to do with a top free surface on row st (0: none)
// above which the interior starts at nz1 (surf_mirror,
// src/cpu/n_kernel_lib_PSV.cpp:272-395).  Rows [nz1, st) take szz and szx from
// the rows they mirror: their own threads leave both alone, so that every cell
// has one writer and, in a phase of the update, no other reader.
PSV_HD bool surface_own(int iz, int st) { return !st || iz >= st; }     // szz, szx are the row's own
PSV_HD bool surface_image(int iz, int st) { return st && iz == st; }    // the surface row itself
PSV_HD bool surface_mirrors(int iz, int st, int nz1)                    // mirrored into row 2 st - iz
{
    return st && iz > st && iz <= 2 * st - nz1;
}

}  // namespace psv
