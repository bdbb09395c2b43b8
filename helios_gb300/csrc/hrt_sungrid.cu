// hrt_sungrid.cu -- shadow rays toward collimated sources by a grid in the plane across the source.
//
// All rays of a collimated source are parallel, so what can shadow a point is a question in two
// dimensions: the primitives whose projection along the source direction covers the point's.  Per
// source the primitives are binned into the cells of a regular grid across the direction (each
// entry a record slot and the primitive's largest depth toward the source); a ray looks up one cell
// and tests the primitives there that reach above its origin, with the primitive tests and the
// periodic wrapping of the tree traversal, so each ray's answer is the tree's.  Projected bounds
// are padded well past the rounding of the projection and of the primitive tests.
//
// Why: a shadow ray through the 4-wide tree makes 20-42 node visits of some 150 instructions and 2-4
// primitive tests; one cell lookup leaves only primitive tests, and the rays of a warp (strata of one
// primitive) read the same few cells.  The binning is bandwidth and atomics, about eight entries per
// primitive, and is repeated for every source and call: nothing is kept between calls.  Measured,
// tree -> grid, binning included: 100 M rays of the 1 M-triangle orchard 22.8 -> 3.1 ms, 20 M rays of a
// 200,004-primitive canopy 6.5 -> 1.7 ms, 6.3 M of a periodic stand 5.6 -> 1.1 ms, 2 M of the
// 20,001-patch canopy 0.69 -> 0.21 ms; 96 suns over a 100 k orchard block 344 -> 121 ms per sweep.
// A source whose grid would not pay (entries over the buffer, more than kSunLarge primitives that
// cover over kSunWide cells, a direction that is not finite, walls far beyond the scene, crowded cells) is not marked as done on the device and
// its rays go through the tree (k_direct / k_direct_sweep skip the sources done here).
#include "hrt_trace.cuh"

namespace hrt {

namespace {

constexpr int kSunThreads = 256;
constexpr int kSunTile = 2048;   // cells per block of k_sun_offsets

__device__ __forceinline__ uint32_t ordered(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unordered(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u ^ 0x80000000u) : ~u);
}

// Bounding box of record `slot` (exact for polygons and voxels, the sphere's for disks).
__device__ __forceinline__ void record_box(const float4 *__restrict__ rec, int slot, f3 *lo, f3 *hi) {
    const float4 *r = rec + 4 * (size_t)slot;
    const float4 r0 = __ldg(r), r1 = __ldg(r + 1), r2 = __ldg(r + 2), r3 = __ldg(r + 3);
    if (__float_as_uint(r0.w) == PT_DISK) {
        const float rad = r2.x;
        *lo = mk(r0.x - rad, r0.y - rad, r0.z - rad);
        *hi = mk(r0.x + rad, r0.y + rad, r0.z + rad);
        return;
    }
    // triangles repeat a corner, voxels their two corners
    *lo = mk(fminf(fminf(r0.x, r1.x), fminf(r2.x, r3.x)), fminf(fminf(r0.y, r1.y), fminf(r2.y, r3.y)),
             fminf(fminf(r0.z, r1.z), fminf(r2.z, r3.z)));
    *hi = mk(fmaxf(fmaxf(r0.x, r1.x), fmaxf(r2.x, r3.x)), fmaxf(fmaxf(r0.y, r1.y), fmaxf(r2.y, r3.y)),
             fmaxf(fmaxf(r0.z, r1.z), fmaxf(r2.z, r3.z)));
}

// Scene bounds and mean primitive extents.  out (zeroed): [0..2] ordered(-lo), [3..5] ordered(hi),
// [6..8] sums of the extents (float).
__global__ void __launch_bounds__(kSunThreads) k_scene_extent(int n, const float4 *__restrict__ rec, uint32_t *out) {
    float v[9];
    for (int k = 0; k < 6; ++k) v[k] = -INFINITY;
    for (int k = 6; k < 9; ++k) v[k] = 0.f;
    for (int i = blockIdx.x * kSunThreads + threadIdx.x; i < n; i += gridDim.x * kSunThreads) {
        f3 lo, hi;
        record_box(rec, i, &lo, &hi);
        const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (!(h[k] - l[k] >= 0.f)) continue;
            v[k] = fmaxf(v[k], -l[k]);
            v[3 + k] = fmaxf(v[3 + k], h[k]);
            v[6 + k] += h[k] - l[k];
        }
    }
    __shared__ float sh[kSunThreads / 32][9];
#pragma unroll
    for (int k = 0; k < 9; ++k)
        for (int d = 16; d > 0; d >>= 1) {
            const float o = __shfl_down_sync(0xffffffffu, v[k], d);
            v[k] = k < 6 ? fmaxf(v[k], o) : v[k] + o;
        }
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 9; ++k) sh[threadIdx.x >> 5][k] = v[k];
    __syncthreads();
    if (threadIdx.x < 9) {
        const int k = threadIdx.x;
        float a = sh[0][k];
        for (int w = 1; w < kSunThreads / 32; ++w) a = k < 6 ? fmaxf(a, sh[w][k]) : a + sh[w][k];
        if (k < 6) atomicMax(out + k, ordered(a));
        else atomicAdd((float *)out + k, a);
    }
}

// One thread per source: direction, plane axes, ray set-up and the grid's frame.
__global__ void k_sun_setup(int nb, const float *__restrict__ dirs, int dir_stride, const uint32_t *__restrict__ extent,
                            int n, uint32_t cells_cap, float wall_far, SunGrid *grids) {
    const int b = threadIdx.x;
    if (b >= nb) return;
    SunGrid g;
    const float *dp = dirs + (size_t)b * dir_stride;
    const f3 s = normalize(mk(dp[0], dp[1], dp[2]));
    f3 e1, e2;
    onb(s, &e1, &e2);
    g.s = s;
    g.e1 = e1;
    g.e2 = e2;
    const WT w = wt_setup(s);
    g.kx = w.kx;
    g.ky = w.ky;
    g.kz = w.kz;
    g.Sx = w.Sx;
    g.Sy = w.Sy;
    g.Sz = w.Sz;
    g.inv = mk(safe_inv(s.x), safe_inv(s.y), safe_inv(s.z));
    float lo[3], hi[3], mean[3], ext = 0.f, far = 0.f;
    for (int k = 0; k < 3; ++k) {
        lo[k] = -unordered(extent[k]);
        hi[k] = unordered(extent[3 + k]);
        mean[k] = __uint_as_float(extent[6 + k]) / (float)n;
        ext = fmaxf(ext, hi[k] - lo[k]);
        far = fmaxf(far, fmaxf(fabsf(lo[k]), fabsf(hi[k])));
    }
    // The projections round by about 2^-22 of the coordinates (of a wrapped ray: the walls'), the primitive
    // tests by 2^-22 of the distances; 2^-19 of both covers them.
    g.pad = (fmaxf(far, wall_far) + ext) * 1.9073486328125e-06f;
    const bool near = !(wall_far > kWallsFar * (far + ext));
    const f3 c = mk(0.5f * (lo[0] + hi[0]), 0.5f * (lo[1] + hi[1]), 0.5f * (lo[2] + hi[2]));
    const f3 half = mk(0.5f * (hi[0] - lo[0]), 0.5f * (hi[1] - lo[1]), 0.5f * (hi[2] - lo[2]));
    const float hu = fabsf(e1.x) * half.x + fabsf(e1.y) * half.y + fabsf(e1.z) * half.z + 2.f * g.pad;
    const float hv = fabsf(e2.x) * half.x + fabsf(e2.y) * half.y + fabsf(e2.z) * half.z + 2.f * g.pad;
    g.u0 = dot(c, e1) - hu;
    g.v0 = dot(c, e2) - hv;
    // Cell side: a fixed share of the mean projected extent of the primitives' boxes, which is about
    // twice the mean extent of the primitives themselves.  Smaller cells hold fewer candidates but
    // cost entries: direct pass of the 200,004-primitive canopy with half-extents times 1.5, 1, 0.7,
    // 0.5: 2.8, 2.1, 1.8, 1.65 ms; of the 1 M orchard 3.65, 3.2, 3.15, 3.15 ms.
    const float du = fabsf(e1.x) * mean[0] + fabsf(e1.y) * mean[1] + fabsf(e1.z) * mean[2];
    const float dv = fabsf(e2.x) * mean[0] + fabsf(e2.y) * mean[1] + fabsf(e2.z) * mean[2];
    float h = fmaxf(kSunCell * 0.5f * (du + dv), 4.f * g.pad);
    const float area = 4.f * hu * hv;
    h = fmaxf(h, 1.01f * sqrtf(area / (float)cells_cap));
    h = fmaxf(h, 2.f * fmaxf(hu, hv) / 30000.f);
    int nu = 1, nv = 1;
    const bool fits = sun_cells(hu, hv, cells_cap, &h, &nu, &nv);
    g.inv_h = 1.f / h;
    const bool fine = fits && near && g.inv_h > 0.f && isfinite(g.inv_h) && isfinite(g.u0) && isfinite(g.v0);
    g.nu = fine ? nu : 1;
    g.nv = fine ? nv : 1;
    g.ok = fine ? 1u : 0u;
    g.total = 0u;
    g.served = 0u;
    g.sq = 0ull;
    g.nlarge = 0u;
    grids[b] = g;
}

// Whether a binned source is traced by its grid: its entries fit, few primitives are wide and the cells
// are not crowded.  The flag of the frame is written once, by k_sun_setup, and this once, by one thread of
// the filling launch, so that the threads of a block agree on both.
__device__ __forceinline__ bool sun_served(const SunGrid &g, uint32_t entries_cap, int n) {
    return g.ok && g.nlarge <= (uint32_t)kSunLarge && g.total <= entries_cap && g.sq <= sun_crowd(n) * g.total;
}

struct CellRect {
    int u0, u1, v0, v1;
    float wmax;
    bool any;
};

// Cells under the padded projection of record `slot`, and its padded largest depth.
__device__ __forceinline__ CellRect project(const float4 *__restrict__ rec, int slot, const SunGrid &g) {
    const float4 *r = rec + 4 * (size_t)slot;
    const float4 r0 = __ldg(r), r1 = __ldg(r + 1), r2 = __ldg(r + 2);
    const uint32_t type = __float_as_uint(r0.w);
    float ulo, uhi, vlo, vhi, w;
    if (type == PT_DISK || type == PT_VOXEL) {
        f3 c, hx;
        if (type == PT_DISK) {
            c = xyz(r0);
            hx = mk(r2.x, r2.x, r2.x);
        } else {
            c = mk(0.5f * (r0.x + r1.x), 0.5f * (r0.y + r1.y), 0.5f * (r0.z + r1.z));
            hx = mk(0.5f * (r1.x - r0.x), 0.5f * (r1.y - r0.y), 0.5f * (r1.z - r0.z));
        }
        const bool disk = type == PT_DISK;
        const float hu = disk ? hx.x : fabsf(g.e1.x) * hx.x + fabsf(g.e1.y) * hx.y + fabsf(g.e1.z) * hx.z;
        const float hv = disk ? hx.x : fabsf(g.e2.x) * hx.x + fabsf(g.e2.y) * hx.y + fabsf(g.e2.z) * hx.z;
        const float hw = disk ? hx.x : fabsf(g.s.x) * hx.x + fabsf(g.s.y) * hx.y + fabsf(g.s.z) * hx.z;
        const float u = dot(c, g.e1), v = dot(c, g.e2);
        ulo = u - hu;
        uhi = u + hu;
        vlo = v - hv;
        vhi = v + hv;
        w = dot(c, g.s) + hw;
    } else {
        const float4 r3 = __ldg(r + 3);  // a triangle's repeats r2
        const f3 q[4] = {xyz(r0), xyz(r1), xyz(r2), xyz(r3)};
        ulo = uhi = dot(q[0], g.e1);
        vlo = vhi = dot(q[0], g.e2);
        w = dot(q[0], g.s);
#pragma unroll
        for (int k = 1; k < 4; ++k) {
            const float u = dot(q[k], g.e1), v = dot(q[k], g.e2);
            ulo = fminf(ulo, u);
            uhi = fmaxf(uhi, u);
            vlo = fminf(vlo, v);
            vhi = fmaxf(vhi, v);
            w = fmaxf(w, dot(q[k], g.s));
        }
    }
    CellRect c;
    const float au = floorf((ulo - g.pad - g.u0) * g.inv_h), bu = floorf((uhi + g.pad - g.u0) * g.inv_h);
    const float av = floorf((vlo - g.pad - g.v0) * g.inv_h), bv = floorf((vhi + g.pad - g.v0) * g.inv_h);
    c.any = au <= bu && av <= bv && au < (float)g.nu && av < (float)g.nv && bu >= 0.f && bv >= 0.f;
    c.u0 = c.any ? (int)fmaxf(au, 0.f) : 0;
    c.v0 = c.any ? (int)fmaxf(av, 0.f) : 0;
    c.u1 = c.any ? (int)fminf(bu, (float)(g.nu - 1)) : -1;
    c.v1 = c.any ? (int)fminf(bv, (float)(g.nv - 1)) : -1;
    c.wmax = w + g.pad;
    return c;
}

// Count the entries of every cell (cells[i].y, zeroed), or fill them (cells[i].x runs from a
// cell's first entry to its end).  Grid: x over records, y over the batch's sources.
template <bool FILL>
__global__ void __launch_bounds__(kSunThreads) k_sun_bin(int n, const float4 *__restrict__ rec, SunGrid *grids,
                                                         uint2 *cells, uint32_t cells_cap, uint2 *entries,
                                                         uint32_t entries_cap, uint32_t *done) {
    SunGrid *G = grids + blockIdx.y;
    const SunGrid &g = *G;
    const bool on = FILL ? sun_served(g, entries_cap, n) : g.ok != 0u;
    if (FILL && blockIdx.x == 0 && threadIdx.x == 0) done[blockIdx.y] = G->served = on ? 1u : 0u;
    if (!on) return;
    uint2 *cl = cells + (size_t)blockIdx.y * cells_cap;
    uint2 *en = entries + (size_t)blockIdx.y * entries_cap;
    const int i = blockIdx.x * kSunThreads + threadIdx.x;
    if (i >= n) return;
    const CellRect c = project(rec, i, g);
    if (!c.any) return;
    const int nc = (c.u1 - c.u0 + 1) * (c.v1 - c.v0 + 1);
    if (nc > kSunWide) {
        // past the limit the source is dropped, and its other wide primitives need not queue up here
        if (FILL || *(volatile const uint32_t *)&G->nlarge > (uint32_t)kSunLarge) return;
        const uint32_t k = atomicAdd(&G->nlarge, 1u);
        if (k < kSunLarge) G->large[k] = make_uint2((uint32_t)i, __float_as_uint(c.wmax));
        return;
    }
    for (int v = c.v0; v <= c.v1; ++v)
        for (int u = c.u0; u <= c.u1; ++u) {
            uint2 *q = cl + (size_t)v * g.nu + u;
            if (FILL) {
                const uint32_t at = atomicAdd(&q->x, 1u);
                if (at < entries_cap) en[at] = make_uint2((uint32_t)i, __float_as_uint(c.wmax));
            } else {
                atomicAdd(&q->y, 1u);
            }
        }
}

// First entry of every cell and the sum of squared counts: a scan within the block's cells from one range of the entries per block
// (cells of different blocks need no order).
__global__ void __launch_bounds__(kSunThreads) k_sun_offsets(SunGrid *grids, uint2 *cells, uint32_t cells_cap) {
    SunGrid *G = grids + blockIdx.y;
    if (!G->ok) return;
    const uint32_t ncell = (uint32_t)G->nu * (uint32_t)G->nv;
    const uint32_t base = blockIdx.x * kSunTile;
    if (base >= ncell) return;
    uint2 *cl = cells + (size_t)blockIdx.y * cells_cap;
    constexpr int kPer = kSunTile / kSunThreads;
    uint32_t v[kPer], sum = 0;
    unsigned long long sq = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const uint32_t i = base + threadIdx.x * kPer + j;
        v[j] = i < ncell ? cl[i].y : 0u;
        sum += v[j];
        sq += (unsigned long long)v[j] * v[j];
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, d);
    __shared__ uint32_t sh[kSunThreads / 32];
    __shared__ unsigned long long sh_sq[kSunThreads / 32];
    __shared__ uint32_t first;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) sh[warp] = x;
    if (lane == 0) sh_sq[warp] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        sq = 0;
        for (int w = 0; w < kSunThreads / 32; ++w) {
            const uint32_t s = sh[w];
            sh[w] = t;
            t += s;
            sq += sh_sq[w];
        }
        if (sq) atomicAdd(&G->sq, sq);
        first = t ? atomicAdd(&G->total, t) : 0u;  // at most kSunWide entries of 2^25 primitives: no wrap
    }
    __syncthreads();
    uint32_t at = first + sh[warp] + x - sum;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const uint32_t i = base + threadIdx.x * kPer + j;
        if (i < ncell) cl[i].x = at;
        at += v[j];
    }
}

// Does a primitive shadow the ray from o toward the source of g before tmax?
template <bool VOX>
__device__ __forceinline__ bool sun_shadowed(const TraceScene &sc, const SunGrid &g, const uint2 *cl, const uint2 *en,
                                             const WT &w, f3 o, float tmax, const VoxKey &vk) {
    const float depth = dot(o, g.s);
    float t;
    int face;
    uint32_t orig;
    const float fu = floorf((dot(o, g.e1) - g.u0) * g.inv_h), fv = floorf((dot(o, g.e2) - g.v0) * g.inv_h);
    if (fu >= 0.f && fv >= 0.f && fu < (float)g.nu && fv < (float)g.nv) {
        const uint2 c = __ldg(cl + (size_t)(int)fv * g.nu + (int)fu);
        for (uint32_t i = c.x - c.y; i < c.x; ++i) {
            const uint2 e = __ldg(en + i);
            if (__uint_as_float(e.y) < depth) continue;  // wholly behind the origin
            if (rec_hit<VOX>(sc.rec, e.x, w, o, g.s, g.inv, 1e-4f, tmax, vk, &t, &face, &orig, sc.masks)) return true;
        }
    }
    for (uint32_t i = 0; i < g.nlarge; ++i) {
        const uint2 e = g.large[i];
        if (__uint_as_float(e.y) < depth) continue;
        if (rec_hit<VOX>(sc.rec, e.x, w, o, g.s, g.inv, 1e-4f, tmax, vk, &t, &face, &orig, sc.masks)) return true;
    }
    return false;
}

// Shadow rays of a batch of sources.  SHARED: every source's rays start from the same points (the
// sweep's suns), else source k has its own random numbers.  A warp holds consecutive strata of one
// or a few primitives; all unshadowed rays of a primitive toward a source carry the same strength,
// |n . s| / R, so a ballot counts them and one FP64 product per primitive and source is added.  The
// division by R is left to the epilogue, so that the sums are exact and do not depend on the order
// in which warps add them.
template <bool SHARED, bool VOX>
__global__ void __launch_bounds__(kSunThreads, 4) k_direct_sun(const SunDirectParams P) {
    const uint32_t R = (uint32_t)(P.dimx * P.dimy);
    const uint32_t total = P.count * R;  // < 2^31: the host plans primitive chunks
    const uint32_t stride = gridDim.x * kSunThreads;
    const int lane = threadIdx.x & 31;
    const FastDiv fd_r = make_fastdiv(R ? R : 1u);
    const TraceScene &sc = P.sc;
    __shared__ SunGrid s_grid[kSunBatch];
    {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(P.grids);
        uint32_t *dst = reinterpret_cast<uint32_t *>(s_grid);
        for (uint32_t i = threadIdx.x; i < (uint32_t)P.nb * (sizeof(SunGrid) / sizeof(uint32_t)); i += kSunThreads)
            dst[i] = src[i];
        __syncthreads();
    }
    unsigned long long nrays = 0;
    for (uint32_t base = blockIdx.x * kSunThreads + (threadIdx.x & ~31u); base < total; base += stride) {
        const uint32_t id = base + (uint32_t)lane;
        const bool active = id < total;
        const uint32_t q = active ? fast_div(id, fd_r) : 0u;
        const uint32_t p = P.offset + q, r = id - q * R;
        // the lanes of each primitive: segments of the warp that start at a head lane
        const uint32_t before = __shfl_up_sync(0xffffffffu, q, 1);
        const bool head = active && (lane == 0 || before != q);
        const uint32_t heads = __ballot_sync(0xffffffffu, head) | ~__ballot_sync(0xffffffffu, active);
        const uint32_t above = lane == 31 ? 0u : heads & ~((2u << lane) - 1u);
        const uint32_t seg = (above ? (above & (0u - above)) - 1u : 0xffffffffu) & ~((1u << lane) - 1u);
        float4 g4[4];
        int ts = 3;
        uint32_t type = 0;
        if (active) {
            load_rgen(sc, p, g4);
            ts = sc.twosided[p];
            type = __float_as_uint(g4[0].w);
        }
        const f3 nrm = active ? xyz(g4[3]) : mk(0.f, 0.f, 0.f);
        const bool vox = VOX && type == PT_VOXEL;
        f3 org = mk(0.f, 0.f, 0.f);
        if (SHARED && active) {
            const u4 u = philox(r, p, 0u, 0u, P.seed, P.pass);
            org = direct_origin(g4, type, r, p, 0u, P.dimx, P.dimy, P.seed, P.pass, u, sc.masks);
        }
        for (int b = 0; b < P.nb; ++b) {
            const SunGrid &g = s_grid[b];
            if (!g.served) continue;
            const uint32_t k = (uint32_t)(P.first + b);
            const uint32_t c2 = SHARED ? 0u : (k << 1);
            const bool face = vox || dot(g.s, nrm) > 0.f;
            const bool live = active && !((!face && ts == 0) || ts == 3);
            bool clear = false;
            if (live) {
                if (!SHARED) {
                    const u4 u = philox(r, p, c2, 0u, P.seed, P.pass);
                    org = direct_origin(g4, type, r, p, c2, P.dimx, P.dimy, P.seed, P.pass, u, sc.masks);
                }
                const uint2 *cl = P.cells + (size_t)b * P.cells_cap, *en = P.entries + (size_t)b * P.entries_cap;
                const WT w{g.kx, g.ky, g.kz, g.Sx, g.Sy, g.Sz};
                f3 o = org;
                for (int wrap = 0;; ++wrap) {
                    const VoxKey vk{r, p, c2 | ((uint32_t)wrap << 16), P.seed, P.pass};
                    // a hit counts up to the periodic wall ahead; past it the ray goes on from the
                    // opposite wall, ten times at most (then it deposits nothing), as in trace_full
                    float tb = 1e38f;
                    int which = -1;
                    const bool wall = sc.nbbox > 0 && wall_closest(sc, o, w, g.inv, 1e-4f, 1e38f, &tb, &which);
                    if (sun_shadowed<VOX>(sc, g, cl, en, w, o, tb, vk)) break;
                    if (!wall) {
                        clear = true;
                        break;
                    }
                    if (wrap == 9) break;
                    o = wall_wrap(sc, add(o, scl(g.s, tb)), which);
                }
            }
            nrays += __popc(__ballot_sync(0xffffffffu, live));
            const uint32_t lit = __ballot_sync(0xffffffffu, clear) & seg;
            if (head && lit) {
                // a 24-bit factor times a small count: exact, as are the sums, in any order
                atomicAdd(P.G + ((size_t)p * P.S + k) * 2 + (face ? 1 : 0), proj(nrm, g.s, vox) * (double)__popc(lit));
            }
        }
    }
    if (lane == 0 && nrays && sc.rays) atomicAdd(sc.rays, nrays);
}

}  // namespace

cudaError_t launch_scene_extent(int n, const float4 *rec, uint32_t *out, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(out, 0, 9 * sizeof(uint32_t), s);
    if (e != cudaSuccess || n <= 0) return e;
    int nb = (n + kSunThreads - 1) / kSunThreads;
    if (nb > 608) nb = 608;
    k_scene_extent<<<nb, kSunThreads, 0, s>>>(n, rec, out);
    return cudaGetLastError();
}

SunCaps sun_caps(int n) {
    SunCaps c;
    const uint64_t nn = (uint64_t)(n > 256 ? n : 256);
    c.cells = (uint32_t)(8 * nn < (1ull << 30) ? 8 * nn : (1ull << 30));
    c.entries = 2 * c.cells;
    const uint64_t bytes = 8ull * ((uint64_t)c.cells + c.entries);
    uint64_t b = (256ull << 20) / bytes;
    c.batch = (int)(b < 1 ? 1 : (b > kSunBatch ? kSunBatch : b));
    return c;
}

size_t sun_grid_bytes(int n, int nsrc) {
    const SunCaps c = sun_caps(n);
    const int nb = nsrc < 1 ? 1 : (nsrc < c.batch ? nsrc : c.batch);
    return (size_t)nb * ((size_t)c.cells + c.entries) * sizeof(uint2);
}

cudaError_t launch_direct_sun(const SunDirectParams &p, const float *dirs, int dir_stride, const uint32_t *extent,
                              uint32_t *done, bool shared, uint32_t chunk, int max_blocks, cudaStream_t s) {
    const int n = p.sc.n;
    if (n <= 0 || p.nb <= 0 || p.nb > kSunBatch) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(p.cells, 0, (size_t)p.nb * p.cells_cap * sizeof(uint2), s);
    if (e != cudaSuccess) return e;
    k_sun_setup<<<1, kSunBatch, 0, s>>>(p.nb, dirs, dir_stride, extent, n, p.cells_cap, p.wall_far, p.grids);
    const dim3 gp((unsigned)((n + kSunThreads - 1) / kSunThreads), (unsigned)p.nb);
    k_sun_bin<false><<<gp, kSunThreads, 0, s>>>(n, p.sc.rec, p.grids, p.cells, p.cells_cap, p.entries, p.entries_cap, done);
    const dim3 gc((unsigned)((p.cells_cap + kSunTile - 1) / kSunTile), (unsigned)p.nb);
    k_sun_offsets<<<gc, kSunThreads, 0, s>>>(p.grids, p.cells, p.cells_cap);
    k_sun_bin<true><<<gp, kSunThreads, 0, s>>>(n, p.sc.rec, p.grids, p.cells, p.cells_cap, p.entries, p.entries_cap, done);
    SunDirectParams Q = p;
    for (uint32_t at = 0; at < p.count; at += Q.count) {
        Q.offset = p.offset + at;
        Q.count = p.count - at < chunk ? p.count - at : chunk;
        const unsigned long long total = (unsigned long long)Q.count * (unsigned)(Q.dimx * Q.dimy);
        unsigned long long nb = (total + kSunThreads - 1) / kSunThreads;
        if (nb > (unsigned long long)max_blocks) nb = (unsigned long long)max_blocks;
        if (nb == 0) break;
        const bool vox = p.sc.voxels != 0;
        if (shared) k_direct_sun<true, false><<<(unsigned)nb, kSunThreads, 0, s>>>(Q);
        else if (vox) k_direct_sun<false, true><<<(unsigned)nb, kSunThreads, 0, s>>>(Q);
        else k_direct_sun<false, false><<<(unsigned)nb, kSunThreads, 0, s>>>(Q);
    }
    return cudaGetLastError();
}

}  // namespace hrt
