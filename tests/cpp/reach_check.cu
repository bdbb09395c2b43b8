// Host check of the bounds on ray origins that the padding of a voxel lattice starts from
// (primitives_reach and largest_coordinate in hrt_internal.h).
#include <cmath>
#include <cstdio>

#include "hrt_device.cuh"
#include "hrt_internal.h"

int main() {
    int bad = 0;
    // a 1 km ground centred at the origin under a leaf: its edges count, not its centre
    float T[32] = {1000.f, 0, 0, 0, 0, 1000.f, 0, 0, 0, 0, 1.f, 0, 0, 0, 0, 1.f,
                   0.1f, 0, 0, 0.5f, 0, 0.1f, 0, 0.5f, 0, 0, 1.f, 1.f, 0, 0, 0, 1.f};
    const float r = hrt::primitives_reach(T, 2);
    bad += !(r >= 500.f && r <= 2000.f);
    T[3] = -4000.f;  // moved away: center and half extent
    bad += !(hrt::primitives_reach(T, 2) >= 4500.f);
    T[3] = NAN;
    bad += !std::isinf(hrt::primitives_reach(T, 2));
    const float walls[6] = {-1.f, 2.f, -30000.f, 4.f, 0.f, 1.f};
    bad += hrt::largest_coordinate(walls, 6) != 30000.f;
    bad += hrt::largest_coordinate(nullptr, 0) != 0.f;
    std::printf("failures %d\n", bad);
    return bad ? 1 : 0;
}
