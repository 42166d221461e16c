// Host check of the tile list's packing and of the sweeps' grids (built by tests/test_tile_list.py with
// g++): every tile of a mesh that has a list comes back from its entry, the first meshes beyond the
// limits have none (their entries would not come back), and a grid never has more than 65535 rows.
#include "salec_kernels.h"

#include <cstdio>

using namespace salec;

static bool comes_back(int ti, int tj)
{
    const int e = tile_pack(ti, tj);
    return tile_column(e) == ti && tile_row(e) == tj;
}

int main()
{
    const int sizes[] = {1, 2, 3, 255, 256, 32766, 32767, 32768, 65534, 65535, 65536, 65537, 131072};
    for (int tx : sizes)
        for (int ty : sizes) {
            const bool corners = comes_back(tx - 1, ty - 1) && comes_back(0, ty - 1) && comes_back(tx - 1, 0);
            if (tiles_fit_a_list(tx, ty) && !corners) return printf("%d x %d tiles do not come back\n", tx, ty), 1;
        }
    if (!tiles_fit_a_list(65535, 32767)) return printf("the largest list\n"), 1;
    if (tiles_fit_a_list(65537, 1) || comes_back(65536, 0)) return printf("too wide a mesh\n"), 1;
    if (tiles_fit_a_list(1, 32769) || comes_back(0, 32768)) return printf("too tall a mesh\n"), 1;
    // rows of points per block; the meshes whose vertex rows just fit a grid, and what fits in front of them
    for (int rows : {1, 2, 4, 8}) {
        const int most = 65535 * rows;
        if (sweep_block_rows(most, rows) != 65535 || sweep_block_rows(most + 1, rows) != 65536) return printf("rows\n"), 1;
        if (sweep_block_rows(most - rows, rows) != 65534) return printf("rows\n"), 1;
        if (!lead_fits(sweep_block_rows(most, rows), 0) || lead_fits(sweep_block_rows(most, rows), 1)) return printf("lead\n"), 1;
        if (!lead_fits(sweep_block_rows(most - 3 * rows, rows), 3) || lead_fits(65535, 2147483647)) return printf("lead\n"), 1;
    }
    puts("OK");
    return 0;
}
