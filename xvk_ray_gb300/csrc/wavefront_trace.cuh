// wavefront_trace.cuh -- persistent CWBVH traversal with dynamic ray fetching.
//
// Software replacement of the hardware TraceRay (opaque triangles, no culling,
// closest hit with ties to the lowest primitive id, or first hit for shadow
// rays).  Each warp keeps 32 rays in flight; once at least refill_min lanes have
// finished (or all have), the warp stores their hits and refills them from the ray
// queue with one atomic (Aila and Laine, "Understanding the Efficiency of Ray
// Traversal on GPUs", HPG 2009): the per-ray set-up (reciprocals, shear constants)
// then runs for many lanes at once instead of one or two.  The nodes are visited as
// in Ylitie, Karras and Laine, "Efficient Incoherent Ray Traversal on GPUs Through
// Compressed Wide BVHs" (HPG 2017): a lane holds one group of internal children
// still to visit (base index, hit bits in near-to-far order, internal-child
// mask) and each iteration visits at most one node.
//
// Triangle tests are decoupled from the lanes that find them: a lane appends the
// triangles of a visited node to its warp's queue and goes on with its nodes; once a
// warp's worth is queued (or too few lanes have nodes left to visit), every lane
// takes one queued test, whichever lane's ray it belongs to.
//
// What bounds it is the issue of instructions: 80-84% of the slots in the long launches, some
// 540 a round in one level and 750 in two (a frame's instructions over its rounds, with their
// share of batches, refills and entries), 23-26 of 32 lanes active (18-23), the BVH served from
// L1 and L2.  With each lane testing its own triangles, postponed below 8 lanes, tests ran at
// 12-16 lanes: 2M random rays over 1M triangles 532 -> 472 us, 1080p frames of three contexts
// 2068 -> 1657, the dynamic world 6.72 -> 5.10 ms (all steps since).
//
// The triangle test and the box test are those of traverse.cuh (same arithmetic
// as the CPU oracle); only the order of the work differs, which the closest-hit
// rule makes irrelevant for the result.
#pragma once
#include <type_traits>
#include "traverse.cuh"

namespace xr {

constexpr uint32_t kTriGroupBit = 0x80000000u;   // stack entry holds a group of instances (two-level traversal)
constexpr uint32_t kLevelBit = 0x40000000u;      // stack entry marks the return to the top-level BVH
#ifndef XR_MIN_RUNNING
#define XR_MIN_RUNNING 16
#endif
#ifndef XR_ENTER_MIN
#define XR_ENTER_MIN 4
#endif
constexpr uint32_t kMinRunning = XR_MIN_RUNNING;   // fewer lanes with nodes to visit: test what is queued
constexpr uint32_t kEnterMin = XR_ENTER_MIN;       // lanes that want an instance before they enter together
constexpr float kMinDir = 1e-20f;                 // smallest direction component seen by the box test

struct RayIn {
    float3 o, d;
    float tmin, tmax;
    uint32_t root;   // first node of the ray's scene (0 unless several scenes share the node array)
};

// Byte k of `word` placed in mantissa bits 8..15 of 1.0f by one byte permute:
// the result is exactly 1 + q / 32768.  A plane at q cells is then
// t = q s + a = fma(1 + q / 32768, 32768 s, a - 32768 s), one instruction per
// plane after the per-node constants; the extra rounding of a - 32768 s is
// below 2^-9 of a cell, inside the 1/32-cell slack of the stored boxes.
__device__ __forceinline__ float qplane(uint32_t word, uint32_t k) {
    return __uint_as_float(__byte_perm(word, 0x3F800000u, 0x7604u | (k << 4)));
}

// Three-input minimum / maximum (PTX min.f32 / max.f32 with three sources,
// sm_100 and later); like the two-input forms they return a non-NaN operand
// when there is one, so a NaN plane drops out of the slab test.
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Per-warp working set of the traversal in shared memory: the queue of triangle tests,
// and per lane its ray as the triangle test wants it and the closest hit so far.
constexpr uint32_t kTriQueue = 64;
constexpr uint32_t kStackRing = 64;
// Groups a lane's stack may hold.  A ray that enters an instance saves the next top-level node
// beside the rest of that node's group: one entry more than the group alone.
template <bool INST> constexpr uint32_t kStackMax = (uint32_t)kStackSize + (INST ? 1u : 0u);
static_assert(kStackMax<true> <= kStackRing, "the stack is a ring of this many");
template <bool INST>
struct alignas(16) TraceWarp {
    float4 ray0[32];             // the origin's components kx, ky, kz; tmin
    float4 ray1[32];             // Sx, Sy, Sz; kx | ky << 2 | kz << 4
    float2 bary[32];
    uint32_t q_slot[kTriQueue];  // triangle slot of each queued test
    float t[32];
    int32_t prim[32];
    uint8_t q_lane[kTriQueue];   // and the lane whose ray is tested
    uint8_t winner[32];
    int32_t inst[INST ? 32 : 4];
};

// LoadRay(i) -> RayIn; StoreHit(i, const HitRec&).  `sh` is the calling warp's working
// set, `next` the fetch counter (zeroed before the launch), `count` the number of rays,
// `err` the error word.  With `work` non-null (query kernels only) the node visits and
// triangle tests are summed into work[0] and work[1]; with `nonfinite` non-null, the rays
// ended early for a non-finite origin or direction are counted there.
//
// INST: two-level traversal of a scene with instances.  Rays start at the root of
// the top-level BVH (sc.tlas_nodes), whose leaf slots are instances; entering one
// saves the rest of the lane's top-level work on its stack under a level marker,
// maps the ray into the instance's object space (origin and direction by its
// world-to-object rows; t is unchanged) and continues at the root of its
// bottom-level BVH in sc.nodes.  Popping the marker, once no test of the lane is
// queued any more, restores the world-space ray (kept in the lane's registers or
// local memory since the ray's start).  Hits compare t, then instance, then primitive.
//
// RETRY (closest hit): a ray whose tmax is below retry_tmax treats its tmax
// as a guess at where it hits.  Boxes beyond it are culled from the start; a ray that
// ends without a hit inside it is traced again up to retry_tmax.  The result is the
// same either way: when a hit lies within tmax, the closest hit (and every hit tied
// with it) does too.
//
// Once the ray queue is empty, idle lanes help the warp's last rays (one-level traversal):
// a lane with groups on its stack hands the bottom one, the largest part of what it has
// left, to an idle lane with a copy of its ray.  Tests found by a helper go to the ray's
// record, and a ray is finished when neither its lane nor a helper has anything left.
template <bool ANY, bool INST = false, bool RETRY = false, typename LoadRay, typename StoreHit>
__device__ __forceinline__ void trace_persistent(TraceWarp<INST>& sh, const DeviceScene& sc, uint32_t count,
                                                 uint32_t* next, LoadRay load, StoreHit store, uint32_t* err,
                                                 unsigned long long* work = nullptr, uint32_t* nonfinite = nullptr,
                                                 float retry_tmax = 0.0f) {
    static_assert(!RETRY || !ANY, "the retry is for closest-hit traversal");
    constexpr bool HELP = !INST;
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    uint32_t n_visits = 0, n_tests = 0;
    // queue tuning of the context (0: the defaults)
    const uint32_t refill_min = sc.refill_min ? sc.refill_min : default_refill(INST, sc.n_nodes);
    const uint32_t batch = sc.postpone_below ? sc.postpone_below : default_batch(INST);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t q_head = 0, q_count = 0;   // the queue, a ring; these are the same in all lanes
    uint32_t pending = 0;               // INST: queued_rays(), kept for the pops of level markers
    bool drained = false;
    bool helping = false;                // lanes have been sent to help; the same in all lanes
    uint32_t ray_id = kInvalid;          // the lane's ray (kInvalid: none)
    uint32_t of = lane;                  // the lane whose ray it works on: its own, or the one it helps
    bool retry = false;   // RETRY: it is traced again up to retry_tmax on a miss
    float3 o = f3(0, 0, 0);
    float idx = 0, idy = 0, idz = 0, tmin_box = 0;
    float h_t = 0;        // t of the closest hit so far (sh.t of this lane)
    uint32_t flip = 0;
    uint2 stack[kStackRing];
    uint32_t sp = 0, sb = 0;             // a ring: the bottom moves up when a helper takes it
    uint32_t cur = kInvalid;             // the node to visit next (kInvalid: none)
    uint32_t tg_base = 0, tg_mask = 0;   // triangles found: first slot, hit bits; INST: instances (of that top-level node)
    bool in_blas = !INST;    // INST: the lane's ray is in an instance's object space
    int32_t cur_inst = -1;   // that instance
    // INST: the world-space ray and its box-test state, kept for instance entries
    // and for the return to the top level (no reload, no reciprocals recomputed)
    float3 wo = f3(0, 0, 0), wd = f3(0, 0, 0);
    float w_tmin = 0, widx = 0, widy = 0, widz = 0;
    uint32_t wflip = 0;
    // Box-test reciprocals of the direction with each component kept at least kMinDir in
    // magnitude (sign kept): an exactly zero component would give an infinite reciprocal,
    // and inf - inf in the per-node plane constants below is NaN, which drops that axis
    // from every slab test and walks the whole tree.  The box test then follows a ray that
    // departs from the true one by at most kMinDir * t, far inside the slack of the stored
    // boxes, so no box holding a hit is culled; the triangle test uses the true direction.
    // The sign bits select the near planes (so that -0 picks the same planes as its
    // infinite reciprocal).  The divisions are correctly rounded: rcp.approx, within an ulp,
    // would save 1.1% of the dynamic world's frame and 0.6% of one level's, but the planes'
    // constants then start from a less exact operand.
    auto set_dir = [&](float3 d) {
        idx = 1.0f / copysignf(fmaxf(fabsf(d.x), kMinDir), d.x);
        idy = 1.0f / copysignf(fmaxf(fabsf(d.y), kMinDir), d.y);
        idz = 1.0f / copysignf(fmaxf(fabsf(d.z), kMinDir), d.z);
        flip = (__float_as_uint(d.x) >> 31) | ((__float_as_uint(d.y) >> 31) << 1) | ((__float_as_uint(d.z) >> 31) << 2);
    };
    // The lane's ray as every lane's triangle test reads it.
    auto put_ray = [&](float3 ro, float3 rd, float rtmin) {
        const RayTri r = prep_ray(ro, rd);
        sh.ray0[lane] = make_float4(sel3(ro, r.kx), sel3(ro, r.ky), sel3(ro, r.kz), rtmin);
        sh.ray1[lane] = make_float4(r.Sx, r.Sy, r.Sz, __uint_as_float((uint32_t)(r.kx | (r.ky << 2) | (r.kz << 4))));
    };
    // A bound was exceeded: the ray goes on without what lies beyond it, the call fails.
    auto overflow = [&]() { atomicOr(err, (uint32_t)XR_DEVFLAG_STACK_OVERFLOW); };
    // The stack is a ring once helpers take groups from its bottom, not before.
    auto slot_of = [&](uint32_t i, auto tail) -> uint2& { return stack[decltype(tail)::value ? i & (kStackRing - 1u) : i]; };
    // Takes the first child of a group as the node to visit next; the rest goes on the stack.
    auto take_child = [&](uint2 e, auto tail) {
        const uint32_t k = __ffs(e.y) - 1u;
        e.y &= e.y - 1u;
        cur = e.x + __popc((e.y >> 8) & ((1u << (k ^ flip)) - 1u));
        if (e.y & 0xFFu) {
            if (sp - sb < kStackMax<INST>) slot_of(sp++, tail) = e;
            else overflow();
        }
    };
    // The whole ray's start: at the top-level root, or at the root of its scene.
    auto start_ray = [&](uint32_t root) {
        if (INST) {
            in_blas = false;
            cur_inst = -1;
            cur = sc.n_tlas_nodes ? 0u : kInvalid;
        } else {
            cur = root < sc.n_nodes ? root : kInvalid;   // no root: a miss
        }
    };
    // The next node: from the group `e` the last visit found, else from the stack.
    auto next_node = [&](uint2 e, auto tail) {
        if (cur != kInvalid || (INST && tg_mask && !in_blas)) return;
        while (!(e.y & 0xFFu) && sp != sb) {
            e = slot_of(sp - 1u, tail);
            if (INST && e.y == kLevelBit) {
                if (tg_mask || ((pending >> lane) & 1u)) break;   // its tests still need this object space
                // back to the top level: the world-space ray
                o = wo;
                idx = widx; idy = widy; idz = widz;
                flip = wflip;
                in_blas = false;
                cur_inst = -1;
            } else if (INST && (e.y & kTriGroupBit)) {
                tg_base = e.x;
                tg_mask = e.y & 0x00FFFFFFu;
                --sp;
                e.y = 0u;
                break;
            }
            --sp;
        }
        if (e.y & 0xFFu) take_child(e, tail);
    };
    // Rays (their lanes) with a queued test.  The entries are other lanes' writes, and a vote
    // orders no memory: without the barrier a ray could be stored before its last test.
    auto queued_rays = [&]() {
        __syncwarp();
        uint32_t m = 0u;
        for (uint32_t i = 0; i < q_count; i += 32u)
            m |= __reduce_or_sync(FULL, i + lane < q_count ? 1u << sh.q_lane[(q_head + i + lane) & (kTriQueue - 1u)] : 0u);
        return m;
    };
    // One queued test per lane, the oldest first (all lanes of the warp call this).
    auto run_tests = [&](auto tail) {
        const uint32_t ray = decltype(tail)::value ? of : lane;
        __syncwarp();
        const uint32_t k = min(q_count, 32u);
        const uint32_t at = (q_head + lane) & (kTriQueue - 1u);
        const bool on = lane < k;
        const uint32_t owner = on ? sh.q_lane[at] : lane;
        bool hit = false;
        float tt = 0.0f, b1 = 0.0f, b2 = 0.0f;
        int32_t prim = -1;
        if (on) {
            const uint32_t slot = sh.q_slot[at];
            if (slot < sc.n_tri_slots) {
                n_tests++;
                hit = hit_slot(sh.ray0[owner], sh.ray1[owner], reinterpret_cast<const float*>(sc.tri + 3u * (size_t)slot),
                               sh.t[owner], &tt, &b1, &b2, &prim);
            } else {
                overflow();
            }
        }
        const int32_t r_inst = INST ? __shfl_sync(FULL, cur_inst, owner) : -1;
        q_head = (q_head + k) & (kTriQueue - 1u);
        q_count -= k;
        // Merge: of the lanes with a hit one per ray writes it if it beats the ray's record,
        // until none is left (several hits of one ray in one batch are rare).  A record only
        // ever improves, so the order of the tests does not matter; each round settles at
        // least one lane, so at most 32 follow.
        while (__any_sync(FULL, hit)) {
            if (hit) sh.winner[owner] = (uint8_t)lane;
            __syncwarp();
            if (hit && sh.winner[owner] == lane) {
                const float ct = sh.t[owner];
                const int32_t cp = sh.prim[owner];
                bool tie_wins = prim < cp;
                if (INST) {
                    const int32_t ci = sh.inst[owner];
                    tie_wins = r_inst < ci || (r_inst == ci && prim < cp);
                }
                if (ANY ? cp < 0 : (cp < 0 ? tt <= ct : (tt < ct || (tt == ct && tie_wins)))) {
                    sh.t[owner] = tt;
                    sh.prim[owner] = prim;
                    sh.bary[owner] = make_float2(b1, b2);
                    if (INST) sh.inst[owner] = r_inst;
                }
                hit = false;
            }
            __syncwarp();
        }
        if (!ANY) h_t = sh.t[ray];
        else if (sh.prim[ray] >= 0) { cur = kInvalid; tg_mask = 0u; sp = sb = 0; }   // occluded: nothing left to visit
        // the rays, records and queue entries read above are written again from here on
        if (INST) pending = queued_rays();   // its barrier comes first
        else __syncwarp();
    };

    // One round: finished rays out and new ones in, a node per lane, the tests it gave.
    // `tail`: the ray queue is empty and lanes may help each other; what that takes stays
    // out of the rounds before (6% of their instructions).  False once no ray is left.
    auto round = [&](auto tail) -> bool {
        constexpr bool TAIL = decltype(tail)::value;
        // lanes with a node to visit (not those that wait to enter an instance)
        const uint32_t n_run = __popc(__ballot_sync(FULL, cur != kInvalid && !(INST && tg_mask)));
        if (n_run + refill_min <= 32u) {
            const bool empty = cur == kInvalid && sp == sb && !(INST && tg_mask);
            uint32_t busy = INST ? pending : queued_rays();   // rays with a queued test or a helper at work
            if (TAIL && helping) {
                busy |= __reduce_or_sync(FULL, !empty && of != lane ? 1u << of : 0u);
                if (empty) of = lane;
            }
            // finished rays are stored and idle lanes refilled, several at a time
            const bool done = empty && !((busy >> lane) & 1u);
            const uint32_t n_done = __popc(__ballot_sync(FULL, done));   // finished or idle
            if (n_done == 32u || (n_done >= refill_min && (!drained || __any_sync(FULL, done && ray_id != kInvalid)))) {
                if (done && ray_id != kInvalid) {
                    if (RETRY && retry && sh.prim[lane] < 0) {
                        // nothing within the first tmax: the same ray again from the root, up to
                        // retry_tmax.  The lane holds the world-space ray here (an emptied stack
                        // has popped every level marker), so its direction state is kept; the
                        // triangle-test set-up of a one-level ray is kept too, and a two-level
                        // ray sets it up again at each instance it enters.
                        retry = false;
                        h_t = retry_tmax;
                        sh.t[lane] = retry_tmax;
                        start_ray(INST ? 0u : load(ray_id).root);
                    } else {
                        HitRec h;
                        h.prim = sh.prim[lane];
                        h.t = sh.t[lane];
                        const float2 b = sh.bary[lane];
                        h.b1 = b.x; h.b2 = b.y;
                        h.inst = INST ? sh.inst[lane] : -1;
                        store(ray_id, h);
                        ray_id = kInvalid;
                    }
                }
                const uint32_t idle = __ballot_sync(FULL, ray_id == kInvalid);
                if (!TAIL && idle && !drained) {
                    const uint32_t n_idle = __popc(idle);
                    uint32_t base = 0;
                    if (lane == 0) base = atomicAdd(next, n_idle);
                    base = __shfl_sync(FULL, base, 0);
                    if (base + n_idle >= count) drained = true;
                    const uint32_t my = base + __popc(idle & lt_mask);
                    if (ray_id == kInvalid && my < count) {
                        const RayIn r = load(my);
                        ray_id = my;
                        o = r.o;
                        tmin_box = r.tmin * (1.0f - 1e-6f) - 1e-30f;
                        set_dir(r.d);
                        if (INST) { wo = r.o; wd = r.d; w_tmin = r.tmin; widx = idx; widy = idy; widz = idz; wflip = flip; }
                        else put_ray(r.o, r.d, r.tmin);
                        if (RETRY) retry = r.tmax < retry_tmax;
                        h_t = r.tmax;
                        sh.t[lane] = r.tmax;
                        sh.prim[lane] = -1;
                        sh.bary[lane] = make_float2(0.0f, 0.0f);
                        if (INST) sh.inst[lane] = -1;
                        sp = sb = 0u;
                        start_ray(r.root);
                        // A non-finite origin or direction (or a zero direction) can hit
                        // nothing -- every triangle test fails -- but would make every box
                        // test pass through NaN slabs and walk the whole tree: end it as a miss.
                        const float chk = r.o.x + r.o.y + r.o.z + r.d.x + r.d.y + r.d.z;
                        if (!isfinite(chk) || (r.d.x == 0.0f && r.d.y == 0.0f && r.d.z == 0.0f)) {
                            cur = kInvalid;
                            if (nonfinite) atomicAdd(nonfinite, 1u);
                            if (RETRY) retry = false;
                        }
                    }
                }
                if (!__any_sync(FULL, ray_id != kInvalid)) return false;
            }
            if (TAIL) {
                const bool idle = ray_id == kInvalid && of == lane;
                const uint32_t m_idle = __ballot_sync(FULL, idle), m_give = __ballot_sync(FULL, sp != sb);
                const uint32_t n = min(__popc(m_idle), __popc(m_give));
                if (n) {   // the r-th idle lane takes from the r-th lane with a stack
                    helping = true;
                    const uint32_t r_give = __popc(m_give & lt_mask), r_take = __popc(m_idle & lt_mask);
                    uint2 e = make_uint2(0u, 0u);
                    if (sp != sb && r_give < n) {
                        e = slot_of(sb++, tail);
                        sh.winner[r_give] = (uint8_t)lane;
                    }
                    __syncwarp();
                    const bool take = idle && r_take < n;
                    const uint32_t from = take ? sh.winner[r_take] : lane;
                    e.x = __shfl_sync(FULL, e.x, from);
                    e.y = __shfl_sync(FULL, e.y, from);
                    o.x = __shfl_sync(FULL, o.x, from);
                    o.y = __shfl_sync(FULL, o.y, from);
                    o.z = __shfl_sync(FULL, o.z, from);
                    idx = __shfl_sync(FULL, idx, from);
                    idy = __shfl_sync(FULL, idy, from);
                    idz = __shfl_sync(FULL, idz, from);
                    flip = __shfl_sync(FULL, flip, from);
                    tmin_box = __shfl_sync(FULL, tmin_box, from);
                    h_t = __shfl_sync(FULL, h_t, from);
                    of = __shfl_sync(FULL, of, from);
                    if (take) {
                        sp = sb = 0u;
                        take_child(e, tail);
                    }
                }
            }
        }

        // ---- visit a node ----
        uint2 found = make_uint2(0u, 0u);   // the internal children hit
        uint32_t tg_valid = 0u;             // the child mask tg_mask's bits are of (triangles)
        if (cur != kInvalid && !(INST && tg_mask)) {
            const uint32_t node = cur;
            cur = kInvalid;
            const WideNode* level_nodes = (INST && !in_blas) ? sc.tlas_nodes : sc.nodes;
            const uint32_t level_count = (INST && !in_blas) ? sc.n_tlas_nodes : sc.n_nodes;
            if (node >= level_count) {
                overflow();
            } else {
                n_visits++;
                const uint4* np = reinterpret_cast<const uint4*>(level_nodes + node);
                const uint4 w0 = __ldg(np + 0), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3),
                            w4 = __ldg(np + 4);
                // per axis: S = 32768 * 2^e / d and A = (p - o) / d - S (see qplane)
                const float sx = __uint_as_float(w0.w & 0xFFFF0000u) * idx;
                const float sy = __uint_as_float(w0.w << 16) * idy;
                const float sz = __uint_as_float(w1.w) * idz;
                const float ax = __fmaf_rn(__uint_as_float(w0.x) - o.x, idx, -sx);
                const float ay = __fmaf_rn(__uint_as_float(w0.y) - o.y, idy, -sy);
                const float az = __fmaf_rn(__uint_as_float(w0.z) - o.z, idz, -sz);
                const float tlimit = h_t * (1.0f + 1e-6f) + 1e-30f;
                // near and far quantised planes per axis, chosen once per node from the
                // sign bits of the direction (a negative axis enters through the high plane)
                const bool nx = (flip & 1u) != 0u, ny = (flip & 2u) != 0u, nz = (flip & 4u) != 0u;
                const uint32_t xn0 = nx ? w3.z : w2.x, xn1 = nx ? w3.w : w2.y;
                const uint32_t xf0 = nx ? w2.x : w3.z, xf1 = nx ? w2.y : w3.w;
                const uint32_t yn0 = ny ? w4.x : w2.z, yn1 = ny ? w4.y : w2.w;
                const uint32_t yf0 = ny ? w2.z : w4.x, yf1 = ny ? w2.w : w4.y;
                const uint32_t zn0 = nz ? w4.z : w3.x, zn1 = nz ? w4.w : w3.y;
                const uint32_t zf0 = nz ? w3.x : w4.z, zf1 = nz ? w3.y : w4.w;
                uint32_t hm = 0;   // the hit slots' bits of the child mask
#pragma unroll
                for (uint32_t i = 0; i < 8; i++) {
                    const float txn = __fmaf_rn(qplane(i < 4 ? xn0 : xn1, i & 3u), sx, ax);
                    const float txf = __fmaf_rn(qplane(i < 4 ? xf0 : xf1, i & 3u), sx, ax);
                    const float tyn = __fmaf_rn(qplane(i < 4 ? yn0 : yn1, i & 3u), sy, ay);
                    const float tyf = __fmaf_rn(qplane(i < 4 ? yf0 : yf1, i & 3u), sy, ay);
                    const float tzn = __fmaf_rn(qplane(i < 4 ? zn0 : zn1, i & 3u), sz, az);
                    const float tzf = __fmaf_rn(qplane(i < 4 ? zf0 : zf1, i & 3u), sz, az);
                    const float tn = fmaxf(max3f(txn, tyn, tzn), tmin_box);
                    const float tf = fminf(min3f(txf, tyf, tzf), tlimit);
                    if (tn <= __fmaf_rn(tf, 1.0f + 2e-6f, 1e-30f)) hm |= (7u << (3u * i)) | (1u << (24u + i));
                }
                // internal hits from slot order to near-to-far order (bit k = slot k ^ flip)
                hm &= w1.z;
                uint32_t ih = hm >> 24;
                if (flip & 1u) ih = ((ih & 0x55u) << 1) | ((ih >> 1) & 0x55u);
                if (flip & 2u) ih = ((ih & 0x33u) << 2) | ((ih >> 2) & 0x33u);
                if (flip & 4u) ih = ((ih & 0x0Fu) << 4) | ((ih >> 4) & 0x0Fu);
                found = make_uint2(w1.x, ih | ((w1.z >> 16) & 0xFF00u));
                // children come after their parent, so every descent ends
                if (ih && w1.x <= node) { overflow(); found.y = 0u; }
                tg_base = INST && !in_blas ? node : w1.y;
                tg_valid = w1.z;
                tg_mask = hm & 0x00FFFFFFu;
            }
        }

        if (!INST || !tg_mask || in_blas) next_node(found, tail);
        else if (found.y & 0xFFu) take_child(found, tail);   // top level: instances found go first

        // ---- instances found in a top-level node: enter one in object space ----
        // (the set-up is long: a lane waits until several want it or few can go on)
        const bool enter = INST && !in_blas && tg_mask != 0u;
        if (INST && (n_run < kMinRunning || __popc(__ballot_sync(FULL, enter)) >= (int)kEnterMin) && enter) {
            const uint4 w1 = __ldg(reinterpret_cast<const uint4*>(sc.tlas_nodes + tg_base) + 1);
            // the instances of the node in the order its children are visited, nearest octant first
            uint32_t m = tg_mask, part;
            if ((part = m & ((flip & 4u) ? 0xFFF000u : 0x000FFFu))) m = part;
            if ((part = m & ((flip & 2u) ? 0xFC0FC0u : 0x03F03Fu))) m = part;
            if ((part = m & ((flip & 1u) ? 0xE38E38u : 0x1C71C7u))) m = part;
            m &= 0u - m;
            const uint32_t slot = w1.y + __popc(w1.z & (m - 1u));
            tg_mask ^= m;
            if (slot >= sc.n_inst_slots || sp + 3u > kStackMax<INST>) {
                overflow();
                tg_mask = 0u;
            } else {
                const float4* ip = sc.inst_slots + 4u * slot;
                const float4 m0 = __ldg(ip), m1 = __ldg(ip + 1), m2 = __ldg(ip + 2), m3 = __ldg(ip + 3);
                // the rest of the top-level work (the next node as a group of one), then the level marker
                if (cur != kInvalid) slot_of(sp++, tail) = make_uint2(cur, 1u << flip);
                if (tg_mask) slot_of(sp++, tail) = make_uint2(tg_base, tg_mask | kTriGroupBit);
                slot_of(sp++, tail) = make_uint2(0u, kLevelBit);
                tg_mask = 0u;
                o = xform_point(m0, m1, m2, wo);
                const float3 od = xform_dir(m0, m1, m2, wd);
                set_dir(od);
                put_ray(o, od, w_tmin);
                cur_inst = (int32_t)__float_as_uint(m3.x);
                in_blas = true;
                const uint32_t root = __float_as_uint(m3.y);
                const float chk = o.x + o.y + o.z + od.x + od.y + od.z;
                const bool ok = root < sc.n_nodes && isfinite(chk) && !(od.x == 0.0f && od.y == 0.0f && od.z == 0.0f);
                cur = ok ? root : kInvalid;
            }
        }

        // ---- queue the triangles found ----
        auto put_test = [&](uint32_t at) {
            sh.q_slot[at & (kTriQueue - 1u)] = tg_base + __popc(tg_valid & (tg_mask - 1u) & ~tg_mask);
            sh.q_lane[at & (kTriQueue - 1u)] = (uint8_t)(TAIL ? of : lane);
            tg_mask &= tg_mask - 1u;
        };
        while (true) {
            const uint32_t n_tri = (!INST || in_blas) ? __popc(tg_mask) : 0u;
            const uint32_t m = __ballot_sync(FULL, n_tri != 0u);
            bool more = false;
            if (m) {
                const uint32_t tail = q_head + q_count;
                if (q_count + 3u * __popc(m) <= kTriQueue) {
                    // up to three per lane, where few lanes have any (few nodes give a lane more)
                    const uint32_t n = n_tri < 3u ? n_tri : 3u;
                    const uint32_t p0 = __ballot_sync(FULL, n & 1u), p1 = __ballot_sync(FULL, n & 2u);
                    const uint32_t at = tail + __popc(p0 & lt_mask) + 2u * __popc(p1 & lt_mask);
                    if (n > 0u) put_test(at);
                    if (n > 1u) put_test(at + 1u);
                    if (n > 2u) put_test(at + 2u);
                    q_count += __popc(p0) + 2u * __popc(p1);
                } else {
                    if (n_tri) put_test(tail + __popc(m & lt_mask));
                    q_count += __popc(m);
                }
                if (INST) pending |= m;
                more = __any_sync(FULL, tg_mask != 0u && (!INST || in_blas));
            }
            // a whole batch, or what there is when too few lanes have nodes to visit
            while (q_count >= batch || (!more && q_count && n_run < kMinRunning)) run_tests(tail);
            if (!more) break;
        }
        return true;
    };
    bool going = true;
    while (going && !(HELP && drained)) going = round(std::false_type{});
    if (HELP)
        while (going) going = round(std::true_type{});
    if (work) {
        atomicAdd(&work[0], (unsigned long long)n_visits);
        atomicAdd(&work[1], (unsigned long long)n_tests);
    }
}

}  // namespace xr
