// The shared memory that the host asks for against what the radiality kernel and its
// adjoint index, written down here from the kernels' layouts, for every tile depth over
// magnifications, ranges and rings. Prints the set-ups that do not fit, then their number.
#include <cstdio>
#include <string>

#include "srrf_internal.h"

using namespace rfba;

static bool fits(const FwdPlan& plan, const rfba_srrf_config& c, int cz, bool adjoint) {
    const int dims[4] = {96, 100, 100, 9};
    const FwdParams p = adjoint ? adjoint_params(plan, c, nullptr, dims, cz) : forward_params(plan, c, nullptr, 0, dims, 8, cz);
    const long nq = (cz + 4 + 3) / 4;  // quads that a tile's cells and their taps take
    const long gplane = nq * p.NV * p.NU, uplane = nq * p.TY * p.NU, tile = (long)p.NIX * p.NIY * p.NIZ;
    // the furthest voxel the gradient of the last cell of each axis reads
    bool ok = 4 * nq - 1 + 2 * p.R < p.NIZ && p.NV - 1 + 2 * p.R < p.NIY && p.NU - 1 + 2 * p.R < p.NIX;
    long bytes = 4L * p.lane_words + 16L * p.u_region;
    if (!adjoint) {
        bytes += 16 * 3 * gplane + (p.tma_bx > 0 ? 127 + 4L * p.tma_bx * p.NIY * p.NIZ : 0);
        ok = ok && 3 * uplane <= p.u_region && 4 * uplane + tile <= 4L * p.u_region;
        return ok && bytes <= (long)radiality_smem_bytes(p);
    }
    const long warps = p.TY * kTileX / 32, row = 4 + p.mag[0] * (15 / p.mag[0] + 6);
    bytes += 16 * (6 * gplane + 3 * uplane + warps * 2 * nq * row);
    ok = ok && 3 * uplane <= p.u_region && (tile + 3) / 4 <= p.u_region && gplane <= p.u_region;
    if (p.grad_mode == 1) ok = ok && nq * p.NIY * p.NIX <= 3 * gplane && nq * p.NIY * p.NIX <= 3 * uplane;
    return ok && bytes <= (long)radiality_adjoint_smem_bytes(p);
}

int main() {
    int bad = 0, n = 0;
    for (int axes : {2, 6, 13})
        for (int i = 0; i < 512; ++i)
            for (int range = 1; range <= 3; ++range) {
                rfba_srrf_config c;
                rfba_srrf_config_default(&c);
                for (int a = 0; a < 3; ++a) c.mag[a] = 1 + (i >> (3 * a)) % 8;
                c.axes_in_ring = axes;
                c.gradient_smooth = 1;
                c.main_range = c.x_range = c.y_range = c.z_range = range;
                FwdPlan plan;
                std::string err;
                if (!build_forward_plan(c, &plan, &err)) continue;
                for (int cz : {2, 4, 8})
                    for (bool adjoint : {false, true}) {
                        ++n;
                        if (!fits(plan, c, cz, adjoint) && ++bad <= 5)
                            std::printf("%s mag %d %d %d axes %d range %d cells %d\n", adjoint ? "adjoint" : "forward",
                                        c.mag[0], c.mag[1], c.mag[2], axes, range, cz);
                    }
            }
    std::printf("%d of %d\n", bad, n);
}
