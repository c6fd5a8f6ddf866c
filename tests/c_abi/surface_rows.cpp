// Rows beside a top free surface (csrc/psv_surface.hpp): who touches a row's
// szz and szx in the stress phase of a tile.
#include <cstdio>
#include <vector>

#include "psv_surface.hpp"

int main()
{
    int n = 0;
    for (int nz1 = 1; nz1 <= 4; nz1++)
        for (int nz = nz1 + 8; nz <= 40; nz++)
            for (int st = 0; st < nz / 2; st++) {
                if (st && st < nz1) continue;
                std::vector<int> own(nz, 0), written(nz, 0);
                for (int iz = nz1; iz < nz - nz1; iz++) {
                    own[iz] = psv::surface_own(iz, st);  // reads and writes its own cells
                    written[iz] += own[iz];
                    if (psv::surface_mirrors(iz, st, nz1)) written[2 * st - iz]++;
                    if (psv::surface_image(iz, st) != (st && iz == st)) return printf("image row %d, surface %d\n", iz, st), 1;
                }
                for (int iz = nz1; iz < nz - nz1; iz++, n++) {
                    const bool mirrored = st && iz < st;
                    if (own[iz] == mirrored || (written[iz] != 1 && !(mirrored && 2 * st - iz >= nz - nz1)))
                        return printf("row %d of %d, surface %d, first %d: own %d, writers %d\n", iz, nz, st, nz1,
                                      own[iz], written[iz]), 1;
                }
            }
    printf("ok %d\n", n);
    return 0;
}
