// hrt_voxgrid.cuh -- voxels that form a lattice, marched cell by cell.
//
// Voxels are large boxes over the leaves, so a tree that holds both has overlapping nodes and a ray
// visits most of the voxels it crosses through several of them.  Where the voxels of a scene are
// cells of one regular lattice (the host checks it, find_lattice in hrt_api.cu), a ray can step through
// the cells in order (after Amanatides and Woo, "A Fast Voxel Traversal Algorithm for Ray Tracing",
// Eurographics 1987) and stop at its first interception, which then bounds the walk through a tree
// of the other primitives alone.  Sparse lattices, few surfaces and dense leaves are faster in the one tree
// (march_pays in hrt_api.cu has both sides).  Each cell makes the test of the tree's leaves (voxel_hit: the same
// box, extinction and random number), so the closest interception is the tree's.  Measured on a section
// of the deep-scattering scene (16,001 leaves and 1,000 voxels, periodic, 285 M diffuse rays): 59.8 node
// visits and 11.6 tests per ray in one tree, 39.7 visits, 2.8 tests and 9.7 cells here; 422 -> 362 ms
// of diffuse launches.  The march's code, beside the walk's, overruns the instruction cache (4.4 cycles
// of waiting per issued instruction), which is what bounds it now.
#pragma once
#include "hrt_device.cuh"
#include "hrt_internal.h"

namespace hrt {

namespace {

// Test of lattice cell (x, y, z): the closest interception so far in *best, *code.
__device__ __forceinline__ void vox_cell(const VoxGrid &vg, int x, int y, int z, f3 o, f3 inv, const VoxKey &vk,
                                         float *best, uint32_t *code) {
    const float4 *c = vg.cells + 2 * (size_t)(((size_t)z * vg.n[1] + y) * vg.n[0] + x);
    const float4 lo = __ldg(c);
    if (!(lo.w > 0.f)) return;  // no voxel here, or one without leaves
    const float4 hi = __ldg(c + 1);
    const uint32_t id = __float_as_uint(hi.w);
    float t;
    int face;
    if (!voxel_hit(o, inv, 1e-4f, xyz(lo), xyz(hi), lo.w, *best, vk, id, &t, &face)) return;
    if (*code == kMissCode || t < *best || (t == *best && id < (*code >> 1))) {
        *best = t;
        *code = (id << 1) | (uint32_t)face;
    }
}

// Cells around (x, y, z) behind the faces in `near`: bit 2a the face of axis a that the ray leaves
// behind, bit 2a + 1 the one ahead of it.
__device__ __noinline__ void vox_neighbours(const VoxGrid &vg, int x, int y, int z, uint32_t near, f3 o, f3 inv,
                                            const VoxKey &vk, float *best, uint32_t *code) {
    const int sx = inv.x > 0.f ? 1 : -1, sy = inv.y > 0.f ? 1 : -1, sz = inv.z > 0.f ? 1 : -1;
    for (int dz = (near & 16u) ? -1 : 0; dz <= ((near & 32u) ? 1 : 0); ++dz)
        for (int dy = (near & 4u) ? -1 : 0; dy <= ((near & 8u) ? 1 : 0); ++dy)
            for (int dx = (near & 1u) ? -1 : 0; dx <= ((near & 2u) ? 1 : 0); ++dx) {
                const int cx = x + sx * dx, cy = y + sy * dy, cz = z + sz * dz;
                if ((dx | dy | dz) == 0 || cx < 0 || cy < 0 || cz < 0 || cx >= vg.n[0] || cy >= vg.n[1] || cz >= vg.n[2])
                    continue;
                vox_cell(vg, cx, cy, cz, o, inv, vk, best, code);
            }
}

// The march of one ray segment through the lattice: the cell (10 bits an axis, vg.n <= 1024), the axis
// of the face it was entered by (3: the first cell) and the distance there.
struct VoxMarch {
    uint32_t cell;
    float t0;
};
constexpr uint32_t kMarchNew = 0xFFFFFFFFu;  // VoxMarch::cell of a segment that has not begun

// Distance at which a segment leaves the lattice; *ta: where it enters.
__device__ __forceinline__ float vox_exit(const VoxGrid &vg, f3 o, f3 inv, float *ta) {
    const float ov[3] = {o.x, o.y, o.z}, iv[3] = {inv.x, inv.y, inv.z};
    float a = 1e-4f, b = 1e38f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float t0 = (vg.org[k] - vg.tol - ov[k]) * iv[k];
        const float t1 = (vg.org[k] + (float)vg.n[k] * vg.size[k] + vg.tol - ov[k]) * iv[k];
        a = fmaxf(a, fminf(t0, t1));
        b = fminf(b, fmaxf(t0, t1));
    }
    *ta = a;
    return b;
}

// One cell of the march; false: the segment is past its first interception or the lattice.  ooi: the
// origin times the inverse direction.  The march covers every voxel whose box the ray meets in FP32:
// cells are taken in order, and where the ray is within vg.tol of a cell face that it does not cross
// there, the neighbours behind that face too (the boxes may be off the lattice planes, and the march's
// crossings off the tests', by less).  Near a face means that its crossing, ahead or behind, is nearer
// than the tolerance over the slope.
__device__ __forceinline__ bool vox_step(const VoxGrid &vg, f3 o, f3 ooi, f3 inv, const VoxKey &vk, float tb,
                                         VoxMarch *m, float *best, uint32_t *code) {
    const float iv[3] = {inv.x, inv.y, inv.z}, oi[3] = {ooi.x, ooi.y, ooi.z};
    int c[3] = {(int)(m->cell & 1023u), (int)((m->cell >> 10) & 1023u), (int)((m->cell >> 20) & 1023u)};
    const uint32_t entry = m->cell >> 30;
    float tx[3];
#pragma unroll
    for (int b = 0; b < 3; ++b)
        tx[b] = __fmaf_rn(__fmaf_rn((float)(c[b] + (iv[b] > 0.f ? 1 : 0)), vg.size[b], vg.org[b]), iv[b], -oi[b]);
    const uint32_t a = tx[0] < tx[1] ? (tx[0] < tx[2] ? 0u : 2u) : (tx[1] < tx[2] ? 1u : 2u);
    const float t0 = m->t0, t1 = fmaxf(fmin3(tx[0], tx[1], tx[2]), t0);
    vox_cell(vg, c[0], c[1], c[2], o, inv, vk, best, code);
    const float te = fmin3(t1, *best, tb);
    uint32_t near = 0;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        // but for the face it came in by and the one it goes on through
        const float tol = vg.tol * fabsf(iv[b]);
        if ((uint32_t)b != entry && !(t0 - __fmaf_rn(-vg.size[b], fabsf(iv[b]), tx[b]) > tol)) near |= 1u << (2 * b);
        if (((uint32_t)b != a || te != t1) && !(tx[b] - te > tol)) near |= 2u << (2 * b);
    }
    if (__builtin_expect(near != 0u, 0)) vox_neighbours(vg, c[0], c[1], c[2], near, o, inv, vk, best, code);
    if (*best < t1 || t1 >= tb) return false;
    // into the next cell through axis a
    bool in = true;
#pragma unroll
    for (int b = 0; b < 3; ++b)
        if ((uint32_t)b == a) {
            c[b] += iv[b] > 0.f ? 1 : -1;
            in = c[b] >= 0 && c[b] < vg.n[b];
        }
    m->cell = (uint32_t)c[0] | ((uint32_t)c[1] << 10) | ((uint32_t)c[2] << 20) | (a << 30);
    m->t0 = t1;
    return in;
}

// The first cell of a segment that enters the lattice at ta.
__device__ __forceinline__ void vox_begin(const VoxGrid &vg, f3 o, f3 d, float ta, VoxMarch *m) {
    const float ov[3] = {o.x, o.y, o.z}, dv[3] = {d.x, d.y, d.z};
    uint32_t cell = 3u << 30;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        const float f = floorf((ov[b] + dv[b] * ta - vg.org[b]) * vg.inv[b]);
        cell |= (uint32_t)(int)fminf(fmaxf(f, 0.f), (float)(vg.n[b] - 1)) << (10 * b);
    }
    m->cell = cell;
    m->t0 = ta;
}

}  // namespace

}  // namespace hrt
