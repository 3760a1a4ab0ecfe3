// Prints the mixed kernel's voxel order (compact_voxel, kernels.hpp) of an nx x ny x nz
// grid, one "x y z" line per position.  tests/test_voxel_order.py checks it.
#include "kernels.hpp"

#include <cstdio>
#include <cstdlib>

int main(int argc, char** argv)
{
    if (argc != 4) return 2;
    const int nx = std::atoi(argv[1]), ny = std::atoi(argv[2]), nz = std::atoi(argv[3]);
    for (long long k = 0; k < (long long)nx * ny * nz; k++) {
        int x, y, z;
        bsar::compact_voxel(nx, ny, nz, k, x, y, z);
        std::printf("%d %d %d\n", x, y, z);
    }
    return 0;
}
