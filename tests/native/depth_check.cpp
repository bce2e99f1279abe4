// Prints, for each line "magx magy magz axes T D H W" of standard input, the tile depth
// that the library chooses for that whole series on a GPU of 152 SMs, the adjoint's, and the
// sizes of the forward's and the adjoint's uniform tables.
#include <cstdio>
#include <string>

#include "srrf_internal.h"

int main() {
    int m[3], axes, T, D, H, W;
    while (std::scanf("%d %d %d %d %d %d %d %d", m, m + 1, m + 2, &axes, &T, &D, &H, &W) == 8) {
        rfba_srrf_config c;
        rfba_srrf_config_default(&c);
        for (int a = 0; a < 3; ++a) c.mag[a] = m[a];
        c.axes_in_ring = axes;
        rfba::FwdPlan plan;
        std::string err;
        if (!rfba::build_forward_plan(c, &plan, &err)) {
            std::printf("%s\n", err.c_str());
            return 1;
        }
        const rfba::FwdRegion map = {{0, 0, 0}, {W * m[0], H * m[1], D * m[2]}};
        std::printf("%d %d %zu %zu\n", rfba::forward_depth(plan, {map}, T, 152),
                    rfba::adjoint_depth(plan, map, T, 152), plan.utab.size() / 4, plan.adj_utab.size() / 4);
    }
}
