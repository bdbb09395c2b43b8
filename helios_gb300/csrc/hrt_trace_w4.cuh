// hrt_trace_w4.cuh -- the persistent diffuse trace over compressed 4-wide nodes for scenes
// without voxels or with a lattice of them, laid out for occupancy.
//
// The trace is bound by the latency of node fetches (L1/L2 hits) and by issue slots, not by
// DRAM.  More resident warps hide more of that latency, so this kernel keeps only the state
// of the node loop in registers -- the ray origin premultiplied by the inverse direction
// (ooi), the inverse direction, best distance, current node, two postponed leaves, stack
// pointer and visit budget -- and moves the rest of each lane's state to shared memory, where
// it is touched only when a ray starts, reaches a leaf or ends: the origin, the direction and
// the watertight-test set-up (kx, ky, kz, Sx, Sy, Sz), the best hit so far, the origin
// primitive and face, the wrap count, the running-sum key and sums.
// A node visit is kept short because the kernel is issue-bound: two 256-bit node loads, each
// slab offset in one fused multiply-add from ooi (node4_offset_ooi), the nearest hit child
// found by a three-comparator tournament (node4_nearest) and entered, the other hit children
// pushed without a branch between the hit and no-hit cases, pops with no empty-stack test (a
// sentinel at the bottom of the stack), leaves postponed two per lane, and the loop left only
// when fewer than P.refill lanes remain; ray ids are split into face, primitive, ray and
// stratum by multiplication (FastDiv).
// The traversal stack keeps SD entries per lane in shared memory (indexed [entry][lane], so
// the 32 lanes of a warp always hit 32 different banks); they move to local memory all at once when
// they run out (LaneStack).  Local memory is touched only by rays whose stack is deeper than SD.
//
// Scenes with a lattice of voxels run it as the march (VG) where that is the faster form (march_pays and
// the tuner, hrt_api.cu).
//
// Hits equal those of trace_bvh / k_diffuse_ps: the same node and primitive tests, the same
// tie rule (closest, then smaller original index); only the order of work differs.
#pragma once
#include "hrt_trace.cuh"
#include "hrt_voxgrid.cuh"

namespace hrt {

namespace {

// The stack's top in shared memory ([entry][lane]) at a byte address per lane: entry 0 holds
// kSentinel, so a pop needs no empty-stack test -- popping it ends the ray's traversal.  When a visit
// could push past the SD entries, the lane's entries move to local memory and entry 0 becomes kMore;
// a lane that pops kMore leaves the node loop and takes them back.  A pop is one load and a push one
// predicated store, with no other test (before, every pop and push compared its place with SD and
// computed its address): per solve 1 M-triangle orchard 850 -> 800 ms of diffuse launches, 20,001-patch
// canopy 16.3 -> 14.7 ms, periodic stand of 63,458 primitives 36.6 -> 35.1 ms.
constexpr int32_t kMore = kSentinel + 2;
template <int SD, int BLOCK>
struct LaneStack {
    uint32_t base, top;         // shared addresses: entry 0, and the next free entry
    // Entries move in blocks, so local memory has room for the shared ones besides kStack4 more: a ray
    // whose stack fitted in both together still does.
    static constexpr int kSpill = kStack4 + SD;
    int32_t spill[kSpill + 1];  // [0] entries held (while entry 0 is kMore), then the entries
    static constexpr uint32_t kStep = 4u * BLOCK, kFull = (uint32_t)SD * kStep;
    __device__ __forceinline__ static void put(uint32_t at, int32_t v) {
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(v));
    }
    __device__ __forceinline__ static int32_t take(uint32_t at) {
        int32_t v;
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(at));
        return v;
    }
    __device__ __forceinline__ void init(const int32_t *entry0) {
        base = (uint32_t)__cvta_generic_to_shared(entry0);
        clear();
    }
    __device__ __forceinline__ void clear() {
        put(base, kSentinel);
        restart();
    }
    // For a new segment: one whose traversal ended has popped entry 0 with kSentinel in it (and nothing
    // in local memory), so the entry is still there.
    __device__ __forceinline__ void restart() { top = base + kStep; }
    __device__ __forceinline__ void push_if(float tk, int32_t v) {
        asm volatile(
            "{\n .reg .pred p;\n setp.lt.f32 p, %1, 0f7F800000;\n @p st.shared.b32 [%0], %2;\n"
            " @p add.u32 %0, %0, %3;\n}"
            : "+r"(top)
            : "f"(tk), "r"(v), "n"(kStep));
    }
    __device__ __forceinline__ int32_t pop() {
        top -= kStep;
        return take(top);
    }
    __device__ __forceinline__ bool room() const { return top + 3u * kStep <= base + kFull; }
    // Entries above entry 0 to local memory; false: no room there.
    __device__ __noinline__ bool spill_out() {
        int held = take(base) == kMore ? spill[0] : 0;
        const int n = (int)((top - base) / kStep) - 1;
        if (held + n > kSpill) return false;
        for (int i = 0; i < n; ++i) spill[1 + held + i] = take(base + kStep * (uint32_t)(1 + i));
        spill[0] = held + n;
        put(base, kMore);
        top = base + kStep;
        return true;
    }
    // The last entries held back to shared memory (kMore was popped); the top one.
    __device__ __noinline__ int32_t spill_in() {
        int held = spill[0];
        const int n = held < SD - 4 ? held : SD - 4;
        held -= n;
        for (int i = 0; i < n; ++i) put(base + kStep * (uint32_t)(1 + i), spill[1 + held + i]);
        spill[0] = held;
        put(base, held > 0 ? kMore : kSentinel);
        top = base + kStep * (uint32_t)(1 + n);
        return pop();
    }
};

// BLOCK: threads per block; MINB: resident blocks per SM the register allocation must allow.
// SD: stack entries per lane in shared memory.  KB: ray-id batch -- a warp
// takes 32 x KB consecutive ray ids from the global counter at a time and hands them to its
// idle lanes from shared memory (KB = 1: every refill takes exactly the idle lanes' count).
// MULTI (recording mode only): the launch traces several scenes -- P.slots[0..P.nslots) each
// give a scene, a primitive chunk, ray counts, seed, pass and hit buffer, with consecutive
// ranges of the launch's ray ids (id_begin) -- so one persistent launch covers the pass of
// every scene of a multi-scene sweep.  COV: translucent covers of source 0 (P.sc.cover) are passed as if they were not there.  VG: the scene's voxels form a
// lattice (P.sc.vgrid): each ray segment marches it first and then walks the tree of the surfaces
// (P.sc.nodes4s), bounded by the interception.
template <int NB, bool RECORD, bool STATS, int MINB, int SD, int BLOCK, int KB, bool MULTI = false, bool COV = false,
          bool VG = false>
__global__ void __launch_bounds__(BLOCK, MINB) k_diffuse_w4(const DiffuseParams P) {
    static_assert(!MULTI || (RECORD && !STATS), "multi-scene launches record hits only");
    __shared__ double s_sum[RECORD ? 1 : NB][BLOCK];            // running sums of the lane's origin
    __shared__ float s_ray[9][BLOCK];                            // d.xyz, Sx, Sy, Sz, o.xyz
    __shared__ uint32_t s_lane[VG ? 8 : 5][BLOCK];               // see the L_* slots below
    __shared__ int32_t s_stack[SD][BLOCK];
    __shared__ unsigned long long s_rid[RECORD ? BLOCK : 1];     // record: hit-buffer index
    __shared__ unsigned long long s_chunk[2][KB > 1 ? BLOCK / 32 : 1];  // per warp: next id, end
    __shared__ SceneSlot s_slot[MULTI ? kMaxSlots : 1];          // multi-scene: the launch's scenes
    __shared__ unsigned long long s_srays[MULTI ? kMaxSlots : 1];  // multi-scene: rays per scene
    constexpr int L_AXES = 0;  // kx | ky << 2 | kz << 4 | face << 6 | wraps << 8
    constexpr int L_P = 1;     // origin primitive
    constexpr int L_HIT = 2;   // best hit so far: prim << 1 | face, or kMissCode
    constexpr int L_KEY = 3;   // running-sum key 2p + face, or 0xFFFFFFFF
    constexpr int L_TAKEN = 4; // rays taken (lane budget)
    constexpr int L_RR = VG ? 5 : 0;    // VG: the ray's index in its primitive
    constexpr int L_CELL = VG ? 6 : 0;  // VG: the march's state (VoxMarch)
    constexpr int L_T0 = VG ? 7 : 0;
    constexpr int32_t kMarch = kSentinel + 1;  // VG: the current node of a lane whose segment is marching
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const uint32_t R = (uint32_t)(P.dimx * P.dimy);
    // count x R x faces < 2^31: the host splits larger passes into primitive chunks
    const uint32_t per_face = P.count * R;
    const int nf = ((P.faces & 1) ? 1 : 0) + ((P.faces & 2) ? 1 : 0);
    const unsigned long long total = MULTI ? P.multi_total : (unsigned long long)per_face * (unsigned long long)nf;
    int lslot = 0;  // multi-scene: the scene slot of the lane's ray
    // single-scene launches decode ray ids (< 2^31, the host plans chunks) by multiplication:
    // 165.0 against 168.0 ms per diffuse launch of the 1 M-triangle orchard
    const FastDiv fd_face = make_fastdiv(per_face ? per_face : 1u), fd_r = make_fastdiv(R ? R : 1u),
                  fd_x = make_fastdiv(P.dimx > 0 ? (uint32_t)P.dimx : 1u);
    // the scene of the lane's current ray
#define SC (MULTI ? s_slot[lslot].sc : P.sc)
    if (MULTI) {
        const int words = P.nslots * (int)(sizeof(SceneSlot) / sizeof(uint32_t));
        const uint32_t *src = reinterpret_cast<const uint32_t *>(P.slots);
        uint32_t *dst = reinterpret_cast<uint32_t *>(s_slot);
        for (int i = tid; i < words; i += BLOCK) dst[i] = src[i];
        for (int i = tid; i < P.nslots; i += BLOCK) s_srays[i] = 0ull;
        __syncthreads();
    }

    LaneStack<SD, BLOCK> stk;
    stk.init(&s_stack[0][tid]);
    uint32_t nvis = 0, ntest = 0;  // statistics builds only
    uint32_t nrays = 0;
    bool live = false, exhausted = false;
    f3 ooi = mk(0.f, 0.f, 0.f), inv = ooi;
    float best = 1e38f;
    int32_t cur = kSentinel, leaf = 0, leaf2 = 0;  // current node, up to two postponed leaves
    uint32_t budget = 0;
    if (!RECORD) {
#pragma unroll
        for (int j = 0; j < NB; ++j) s_sum[j][tid] = 0.0;
    }
    s_lane[L_KEY][tid] = 0xFFFFFFFFu;
    s_lane[L_TAKEN][tid] = 0u;
    // a lane budget retires lanes without drawing ids, so a warp could leave ids of its
    // batch untraced: batched fetch only without one
    const bool batched = KB > 1 && P.lane_budget == 0;
    // The first ray id of a lane is its thread's index, later ones come from the counter: a launch
    // of few rays per lane does not begin with every warp's atomic on one address.
    bool fresh = true;
    if (KB > 1 && lane == 0) {
        s_chunk[0][tid >> 5] = 0ull;
        s_chunk[1][tid >> 5] = 0ull;
    }
    __syncwarp();
    // ends the traversal of the lane's ray after an error, which is its own scene's (a multi-scene launch
    // leaves P.sc empty)
    auto give_up = [&](uint32_t bit) {
        raise(SC.status, bit);
        cur = kSentinel;
        leaf = 0;
        leaf2 = 0;
        stk.clear();
    };

    for (;;) {
        // ---- refill lanes without a ray (warp-vote compaction of the fetch)
        if (!live && P.lane_budget && s_lane[L_TAKEN][tid] >= P.lane_budget) exhausted = true;
        const bool need = !live && !exhausted;
        const unsigned m = __ballot_sync(0xffffffffu, need);
        if (m) {
            const int leader = __ffs(m) - 1;
            const unsigned rank = __popc(m & ((1u << lane) - 1u));
            unsigned long long id;
            if (!batched) {
                unsigned long long base;
                if (fresh) {
                    base = (unsigned long long)blockIdx.x * BLOCK + (tid & ~31);
                    fresh = false;
                } else {
                    base = 0;
                    if (lane == leader) base = atomicAdd(P.fetch, (unsigned long long)__popc(m));
                    base = __shfl_sync(0xffffffffu, base, leader) + (unsigned long long)gridDim.x * BLOCK;
                }
                id = base + rank;
            } else {
                // ids are handed out in increasing order, so every id below the end of the
                // range is drawn before any lane of the warp draws one past it
                const int w = tid >> 5;
                const unsigned nneed = __popc(m);
                const unsigned long long next = s_chunk[0][w], left = s_chunk[1][w] - next;
                unsigned long long nb = 0;
                if (left < nneed) {
                    if (lane == leader) nb = atomicAdd(P.fetch, (unsigned long long)(32 * KB));
                    nb = __shfl_sync(0xffffffffu, nb, leader);
                }
                id = rank < left ? next + rank : nb + (rank - left);
                __syncwarp();
                if (lane == leader) {
                    if (left < nneed) {
                        s_chunk[0][w] = nb + (nneed - left);
                        s_chunk[1][w] = nb + 32ull * KB;
                    } else {
                        s_chunk[0][w] = next + nneed;
                    }
                }
                __syncwarp();
            }
            if (need) {
                if (id >= total) {
                    exhausted = true;
                } else {
                    s_lane[L_TAKEN][tid] += 1u;
                    unsigned long long lid = id;
                    uint32_t Rk = R, pfk = per_face, offk = P.offset, seedk = P.seed, passk = P.pass;
                    int dxk = P.dimx, dyk = P.dimy;
                    if (MULTI) {  // the slot whose id range holds id (ranges are consecutive)
                        int k = 0;
                        while (k + 1 < P.nslots && id >= s_slot[k + 1].id_begin) ++k;
                        lslot = k;
                        const SceneSlot &S = s_slot[k];
                        lid = id - S.id_begin;
                        dxk = S.dimx;
                        dyk = S.dimy;
                        Rk = (uint32_t)(dxk * dyk);
                        pfk = S.count * Rk;
                        offk = S.offset;
                        seedk = S.seed;
                        passk = S.pass;
                    }
                    const TraceScene &sc = SC;
                    uint32_t fi, rem;
                    if (!MULTI) {
                        fi = fast_div((uint32_t)lid, fd_face);
                        rem = (uint32_t)lid - fi * pfk;
                    } else {
                        fi = (uint32_t)(lid / pfk);
                        rem = (uint32_t)(lid - (unsigned long long)fi * pfk);
                    }
                    const int face = (nf == 2) ? (fi == 0 ? 1 : 0) : ((P.faces & 1) ? 1 : 0);
                    uint32_t p, r, ti, pi;
                    if (!MULTI) {
                        const uint32_t q = fast_div(rem, fd_r);
                        p = offk + q;
                        r = rem - q * Rk;
                        pi = fast_div(r, fd_x);
                        ti = r - pi * (uint32_t)dxk;
                    } else {
                        p = offk + rem / Rk;
                        r = rem % Rk;
                        ti = r % (uint32_t)dxk;
                        pi = r / (uint32_t)dxk;
                    }
                    if (RECORD) s_rid[tid] = ((unsigned long long)fi * (unsigned long long)sc.n + p) * Rk + r;
                    const int ts = sc.twosided[p];
                    const bool skip = (face == 1 && ts == 3) || (face == 0 && ts != 1);
                    if (!skip) {
                        float4 g[4];
                        load_rgen(sc, p, g);
                        const uint32_t type = __float_as_uint(g[0].w);
                        f3 o, d;
                        diffuse_ray_cell<VG>(g, type, r, p, face, (int)ti, (int)pi, dxk, dyk, seedk, passk, &o, &d,
                                                sc.masks);
                        const WT w = wt_setup(d);
                        s_ray[0][tid] = d.x;
                        s_ray[1][tid] = d.y;
                        s_ray[2][tid] = d.z;
                        s_ray[3][tid] = w.Sx;
                        s_ray[4][tid] = w.Sy;
                        s_ray[5][tid] = w.Sz;
                        s_ray[6][tid] = o.x;
                        s_ray[7][tid] = o.y;
                        s_ray[8][tid] = o.z;
                        s_lane[L_AXES][tid] = (uint32_t)(w.kx | (w.ky << 2) | (w.kz << 4) | (face << 6));
                        s_lane[L_P][tid] = p;
                        s_lane[L_HIT][tid] = kMissCode;
                        inv = mk(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z));
                        ooi = mk(o.x * inv.x, o.y * inv.y, o.z * inv.z);
                        best = 1e38f;
                        if (VG) {
                            s_lane[L_RR][tid] = r;
                            s_lane[L_CELL][tid] = kMarchNew;
                        }
                        cur = VG ? kMarch : ((sc.n > 0) ? 0 : kSentinel);
                        leaf = 0;
                        leaf2 = 0;
                        stk.restart();
                        budget = sc.visit_budget;
                        live = true;
                        if (MULTI) atomicAdd(&s_srays[lslot], 1ull);
                        else ++nrays;
                    }
                }
            }
        }
        // A lane may be idle because its id was skipped by the face rule; only when every
        // lane has run past the end of the id range is the warp done.
        if (__all_sync(0xffffffffu, exhausted && !live)) break;
        // The lanes with a ray meet again after each phase; nothing else keeps one that leaves the node
        // loop from running ahead alone.  Per solve: 1 M-triangle orchard 863 -> 854 ms of diffuse
        // launches, a periodic stand of 63,458 primitives 40.7 -> 38.6, scenes with voxels 422 -> 377.
        const unsigned lm = __ballot_sync(0xffffffffu, live);
        if (!live) continue;

        // ---- lattice of voxels: lanes whose segment has not passed it step through its cells, together
        // until fewer than four are left at it; then the surfaces are walked (with 4, 8, 14, 20 lanes the
        // deep-scattering section took 450, 470, 535, 673 ms of diffuse launches)
        if (VG && cur == kMarch) {
            const VoxGrid &vg = *P.sc.vgrid;
            const f3 o = mk(s_ray[6][tid], s_ray[7][tid], s_ray[8][tid]);
            const f3 d = mk(s_ray[0][tid], s_ray[1][tid], s_ray[2][tid]);
            const uint32_t ax = s_lane[L_AXES][tid];
            const VoxKey vk{s_lane[L_RR][tid], s_lane[L_P][tid], ((ax >> 6) & 1u) | ((ax >> 8) << 16), P.seed, P.pass};
            uint32_t code = s_lane[L_HIT][tid];
            VoxMarch m{s_lane[L_CELL][tid], __uint_as_float(s_lane[L_T0][tid])};
            float ta;
            const float tb = vox_exit(vg, o, inv, &ta);
            bool on = true;
            if (m.cell == kMarchNew) {
                on = ta <= tb;
                if (on) vox_begin(vg, o, d, ta, &m);
            }
            // a segment steps through at most n0 + n1 + n2 cells, every round through one or more
            while (on) {
                on = vox_step(vg, o, ooi, inv, vk, tb, &m, &best, &code);
                if (__popc(__activemask()) < 4) break;
            }
            s_lane[L_HIT][tid] = code;
            if (on) {
                s_lane[L_CELL][tid] = m.cell;
                s_lane[L_T0][tid] = __float_as_uint(m.t0);
            } else {
                cur = P.sc.n4s > 0 ? 0 : kSentinel;
            }
        }

        if (VG) __syncwarp(lm);

        // ---- internal nodes; up to two leaves per lane are postponed to the primitive tests below
        const TraceScene &sc = SC;
        const uint32_t n4 = (uint32_t)(VG ? sc.n4s : sc.n4);
        if (cur >= (int32_t)n4 && cur != kSentinel && !(VG && cur == kMarch)) {
            if (cur != kMore) {
                give_up(ERR_BOUNDS);
            } else if ((cur = stk.spill_in()) < 0) {  // no leaf is postponed here
                leaf = cur;
                cur = stk.pop();
            }
        }
        // one unsigned compare says that cur is an internal node (leaves are negative, the special
        // values and any index out of range above n4: the check above handles those)
        while ((uint32_t)cur < n4) {
            if (budget == 0u) {
                give_up(ERR_BUDGET);
                break;
            }
            --budget;
            if (STATS) ++nvis;
            float4 q0, q1, q2, q3;
            load_node64(VG ? sc.nodes4s : sc.nodes4, cur, q0, q1, q2, q3);
            float tk[4];
            int32_t ck[4];  // every slot's reference: a child is hit when its tk < INFINITY
            node4_children<false>(q0, q1, q2, q3, node4_offset_ooi(q0, ooi, inv), inv, 1e-4f, best, tk, ck);
            node4_nearest(tk, ck);
            // hit children other than the nearest pushed (predicated: a visit that hits nothing pushes
            // nothing), then the nearest entered or, with no hit, the top of the stack taken
            if (__builtin_expect(!stk.room(), 0) && !stk.spill_out()) {
                give_up(ERR_STACK);
                break;
            }
            stk.push_if(tk[3], ck[3]);
            stk.push_if(tk[2], ck[2]);
            stk.push_if(tk[1], ck[1]);
            cur = ck[0];
            if (!(tk[0] < INFINITY)) cur = stk.pop();
            // a leaf is postponed while one of the two slots is free; a lane with both full stops
            // at its third leaf.  The warp leaves the loop only when fewer than P.refill lanes
            // remain in it (no vote on the leaves): 162.7 against 167.4 ms per diffuse launch of
            // the 1 M-triangle orchard with one slot and a leave-when-all-have-a-leaf vote
            if (cur < 0 && leaf2 == 0) {
                leaf2 = leaf;
                leaf = cur;
                cur = stk.pop();
            }
            if (__popc(__activemask()) < P.refill) break;
        }
        __syncwarp(lm);
        // ---- primitive tests (origin, direction and watertight set-up come back from shared memory)
        if (leaf != 0) {
            const f3 o = mk(s_ray[6][tid], s_ray[7][tid], s_ray[8][tid]);
            const f3 d = mk(s_ray[0][tid], s_ray[1][tid], s_ray[2][tid]);
            const uint32_t ax = s_lane[L_AXES][tid];
            WT w;
            w.kx = (int)(ax & 3u);
            w.ky = (int)((ax >> 2) & 3u);
            w.kz = (int)((ax >> 4) & 3u);
            w.Sx = s_ray[3][tid];
            w.Sy = s_ray[4][tid];
            w.Sz = s_ray[5][tid];
            uint32_t bcode = s_lane[L_HIT][tid];
            const VoxKey vk{0u, 0u, 0u, 0u, 0u};  // no voxels among this kernel's leaves
            while (leaf != 0) {
                const uint32_t slot = (uint32_t)(~leaf);
                if (STATS) ++ntest;
                if (slot < (uint32_t)sc.n) {
                    float t;
                    int fc;
                    uint32_t orig;
                    if (rec_hit<false>(sc.rec, slot, w, o, d, inv, 1e-4f, best, vk, &t, &fc, &orig, sc.masks) &&
                        !(COV && (__ldg(sc.cover + orig) & 1u))) {
                        if (bcode == kMissCode || t < best || (t == best && orig < (bcode >> 1))) {
                            best = t;
                            bcode = (orig << 1) | (uint32_t)fc;
                        }
                    }
                } else {
                    raise(sc.status, ERR_BOUNDS);
                }
                leaf = leaf2;
                leaf2 = 0;
                if (leaf == 0 && cur < 0) {
                    leaf = cur;
                    cur = stk.pop();
                }
            }
            s_lane[L_HIT][tid] = bcode;
        }
        __syncwarp(lm);
        if (cur != kSentinel || leaf != 0) continue;  // traversal of this ray goes on next round

        // ---- periodic walls: wrap and restart, or finish the ray
        const uint32_t bcode = s_lane[L_HIT][tid];
        bool lost = false;
        if (sc.nbbox > 0) {
            const f3 o = mk(s_ray[6][tid], s_ray[7][tid], s_ray[8][tid]);
            const f3 d = mk(s_ray[0][tid], s_ray[1][tid], s_ray[2][tid]);
            const uint32_t axw = s_lane[L_AXES][tid];
            const WT w{(int)(axw & 3u), (int)((axw >> 2) & 3u), (int)((axw >> 4) & 3u), s_ray[3][tid], s_ray[4][tid],
                       s_ray[5][tid]};
            float tb;
            int which = -1;
            if (wall_closest(sc, o, w, inv, 1e-4f, (bcode != kMissCode) ? best : 1e38f, &tb, &which) &&
                (bcode == kMissCode || tb < best)) {
                const uint32_t ax = axw;
                const uint32_t wraps = ax >> 8;
                if (wraps >= 9) {
                    lost = true;
                } else {
                    const f3 hp = wall_wrap(sc, add(o, scl(d, tb)), which);
                    s_ray[6][tid] = hp.x;
                    s_ray[7][tid] = hp.y;
                    s_ray[8][tid] = hp.z;
                    ooi = mk(hp.x * inv.x, hp.y * inv.y, hp.z * inv.z);
                    best = 1e38f;
                    s_lane[L_HIT][tid] = kMissCode;
                    s_lane[L_AXES][tid] = (ax & 0xFFu) | ((wraps + 1u) << 8);
                    if (VG) s_lane[L_CELL][tid] = kMarchNew;
                    cur = VG ? kMarch : 0;
                    stk.restart();
                    budget = sc.visit_budget;
                    continue;
                }
            }
        }
        // ---- value of the finished ray, added to the lane's running sum
        live = false;
        if (RECORD) {
            (MULTI ? s_slot[lslot].hits : P.hits)[s_rid[tid]] = lost ? kLostCode : bcode;
            continue;
        }
        if (lost) continue;
        const uint32_t face = (s_lane[L_AXES][tid] >> 6) & 1u;
        const uint32_t key = 2u * s_lane[L_P][tid] + face;
        const uint32_t akey = s_lane[L_KEY][tid];
        if (key != akey) {
            if (akey != 0xFFFFFFFFu) {
                double *dst = ((akey & 1u) ? P.Gt : P.Gb) + (size_t)(akey >> 1) * P.Bl;
#pragma unroll
                for (int j = 0; j < NB; ++j)
                    if (j < P.Bc && s_sum[j][tid] != 0.0) atomicAdd(dst + j, s_sum[j][tid]);
            }
            s_lane[L_KEY][tid] = key;
#pragma unroll
            for (int j = 0; j < NB; ++j) s_sum[j][tid] = 0.0;
        }
        if (bcode != kMissCode) {
            const float *src = ((bcode & 1u) ? P.otop : P.obot) + (size_t)(bcode >> 1) * P.Bl;
#pragma unroll
            for (int j = 0; j < NB; ++j)
                if (j < P.Bc) s_sum[j][tid] += (double)__ldg(src + j);
        } else {
            const f3 d = mk(s_ray[0][tid], s_ray[1][tid], s_ray[2][tid]);
#pragma unroll
            for (int j = 0; j < NB; ++j)
                if (j < P.Bc) {
                    const float fl = P.sky.flux[j];
                    if (fl > 0.f) s_sum[j][tid] += sky_fd(d, P.sky, j) * (double)fl;
                }
        }
    }
    if (!RECORD) {
        const uint32_t akey = s_lane[L_KEY][tid];
        if (akey != 0xFFFFFFFFu) {
            double *dst = ((akey & 1u) ? P.Gt : P.Gb) + (size_t)(akey >> 1) * P.Bl;
#pragma unroll
            for (int j = 0; j < NB; ++j)
                if (j < P.Bc && s_sum[j][tid] != 0.0) atomicAdd(dst + j, s_sum[j][tid]);
        }
    }
    if (MULTI) {  // every warp of the block is past its loop: count the rays per scene
        __syncthreads();
        for (int i = tid; i < P.nslots; i += BLOCK)
            if (s_srays[i] && s_slot[i].sc.rays) atomicAdd(s_slot[i].sc.rays, s_srays[i]);
    } else {
        add_rays(P.sc, nrays);
    }
    if (STATS) count_visits(P.sc, nvis, ntest);
#undef SC
}

}  // namespace

}  // namespace hrt
