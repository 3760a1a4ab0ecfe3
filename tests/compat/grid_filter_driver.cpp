// Prints grid_filter_ok (kernels.hpp) for "nx ny uniform n1 n2 zlo zhi", one line of standard
// input per DEM.  tests/test_grid_filter_rule.py checks it.
#include "kernels.hpp"

#include <cstdio>
#include <cstdlib>

int main()
{
    char lo[64], hi[64];
    bsar::BpArgs a{};
    const float z = 0.0f;
    while (std::scanf("%d %d %d %lf %lf %63s %63s", &a.dem.nx, &a.dem.ny, &a.dem.uniform, &a.n1, &a.n2, lo, hi) == 7) {
        a.dem.z32 = &z;
        a.dem.empty = a.dem.nx == 0 || a.dem.ny == 0;
        a.zlo = (float)std::atof(lo);
        a.zhi = (float)std::atof(hi);
        std::printf("%d\n", (int)bsar::grid_filter_ok(a));
    }
    return 0;
}
