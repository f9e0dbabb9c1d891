// Prints the bounds of sphere_tables and the counts of count_sphere (8 columns per tile) for the grid and box in the arguments:
// nx ny nz lx ly lz alias_filter.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "../../gnss-1_b200/csrc/hostblock.h"

int main(int, char **argv) {
    const int nx = std::atoi(argv[1]), ny = std::atoi(argv[2]), nz = std::atoi(argv[3]);
    const double lx = std::atof(argv[4]), ly = std::atof(argv[5]), lz = std::atof(argv[6]), alias = std::atof(argv[7]);
    const volatile double kmax = alias * (nx * M_PI / lx);
    const int nkz = nz / 2 + 1;   // every column; the bounds say which have no mode
    const gnss::SphereTables t =
        gnss::sphere_tables({nx, 2 * M_PI / lx}, {ny, 2 * M_PI / ly}, {nz, 2 * M_PI / lz}, kmax * kmax, ny,
                            [](int i) { return i; }, nkz, nkz, 1);
    for (short b : t.bound) std::printf("%d ", b);
    std::printf("\n");
    for (int e : t.tiles) std::printf("%d ", e);
    std::printf("\n");
    const gnss::SphereCount n =
        gnss::count_sphere({nx, 2 * M_PI / lx}, {ny, 2 * M_PI / ly}, {nz, 2 * M_PI / lz}, kmax * kmax, ny,
                           [](int i) { return i; }, nkz, 8);
    std::printf("%.0f %.0f %.0f %.0f\n", n.modes, n.cols, n.tile_cols, n.stored);
    return 0;
}
