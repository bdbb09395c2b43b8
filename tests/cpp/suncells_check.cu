// Host check of the cell counts of the grids across collimated sources (sun_cells in hrt_device.cuh):
// never more cells than the buffer holds, also where the product of the counts is no float, and the
// largest grid that fits is not refused.  Prints the failures and exits non-zero on any.
#include <cmath>
#include <cstdint>
#include <cstdio>

#include "hrt_device.cuh"

int main() {
    long bad = 0, over = 0, frames = 0;
    for (uint32_t n = 2000000; n <= 33000000u; n += 1000003u) {
        const uint32_t cap = 8u * n;
        for (uint32_t fu = 6000; fu < 30000; fu += 7) {
            const uint32_t fv = cap / fu + 1;  // one row of cells too many
            if (fv > 30000u) continue;
            // half extents of fu x fv cells of side 1
            const float hu = 0.5f * ((float)fu - 0.5f), hv = 0.5f * ((float)fv - 0.5f);
            float h = 1.f;
            int nu = 0, nv = 0;
            ++frames;
            if ((float)fu * (float)fv <= (float)cap) ++over;  // a float comparison lets it pass
            if (!hrt::sun_cells(hu, hv, cap, &h, &nu, &nv) || (uint64_t)nu * (uint64_t)nv > cap) ++bad;
            // one row less fits as it is
            h = 1.f;
            if (!hrt::sun_cells(hu, hv - 0.5f, cap, &h, &nu, &nv) || h != 1.f || nu != (int)fu || nv != (int)fv - 1) ++bad;
        }
    }
    const float none[] = {NAN, INFINITY, -INFINITY, 1e30f};
    for (float x : none) {
        float h = x == 1e30f ? 1e-8f : 1.f;
        int nu, nv;
        if (hrt::sun_cells(x, 1.f, 1000u, &h, &nu, &nv) && (uint64_t)nu * (uint64_t)nv > 1000u) ++bad;
    }
    std::printf("frames %ld, over the buffer by a float comparison %ld, failures %ld\n", frames, over, bad);
    return bad || !over ? 1 : 0;
}
