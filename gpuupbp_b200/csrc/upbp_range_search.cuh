// Packet search of the range queries: a warp takes up to 32 queries that are
// neighbours in the processing order and finds their (query, neighbour) pairs
// together.  Included by upbp_camera_pass.cuh, which states the modes and the
// rounds.
//
// A walk with one query per lane (22 of 32 lanes active, about 180 warp
// instructions a step) read the same nodes again for every query.  Here the
// lanes hold nodes and leaves instead of queries:
//
//   * the queries of a group (2^k neighbours whose ends lie close together)
//     share one bound, the hull swept by the box of their start points moving
//     to the box of their end points; 32 (node, group) entries of the warp's
//     stack are tested at once, one per lane, whatever groups they belong to,
//     so the lanes stay busy (30.6 of 32 on the media field) down to groups
//     of one query;
//   * 32 (leaf, group) entries reached are tested against their group's
//     queries in turn, one leaf per lane, from shared memory;
//   * pairs that pass that cheap conservative test are gathered by 32 for the
//     exact predicate, and accepted ones by 32 for the hit list.
//
// The bound is conservative (its boxes are padded by the rounding of the
// test), and a pair's acceptance depends on the predicate and the chunk's
// reporting rule alone, so the accepted pairs are those of any other walk.
//
// Measured, BB1D search and evaluation, before -> now: media field at
// 1280x720 24.2 -> 16.0 ms (search 11.1: 456M four-wide node tests instead of
// 1393M two-wide ones), box 256x256 25.1 -> 11.1, dense beams 480x270 55.3 ->
// 42.3, 64x64 preview 1.32 -> 0.13 ms.  What bounds it now: issue (71%) and
// the L1 data pipe (85%) together; on the dense beams the L2, whose 126 MB
// the map and the query records share.
#pragma once

#include "upbp_queries.cuh"

namespace upbp {

constexpr int kPacketStack = 384;   // stack of a warp: node | group << kLeafShift
constexpr int kPacketLeaves = 160;  // < 32 waiting + 128 of a step

struct SearchWarp {
    float4 qa[32];              // origin, tmin (point queries: position)
    float4 qb[32];              // direction, tmax
    float4 qc[32];              // BB1D: origin x direction, origin . direction
    float4 bound[3][32];        // per group (named by its first query): sweep_axis of x, y, z (points: the box)
    uint2 qk[32];               // query record, BB1D: medium
    uint2 group[32];            // per group: its queries; segments: axes moving down (bits 0..2)
    unsigned stack[kPacketStack + 4];
    unsigned leaves[kPacketLeaves];  // leaf | group << kLeafShift
    unsigned pairs[64];         // BB1D pairs for the exact predicate: leaf | query << kLeafShift
    uint2 hit_qb[64];
};
static_assert(kLeafShift + 5 <= 32, "group and query bits of an entry");
constexpr unsigned kNoHit = 0xffffffffu;  // query of an empty slot of the hit list
constexpr unsigned kEntryMask = (1u << kLeafShift) - 1u;

// Bounds of a group of queries: boxes of the start and of the end points.
struct PacketBox {
    float3 alo, ahi, blo, bhi;
};

UPBP_D float3 shfl3_xor(float3 a, int m)
{
    return make_float3(__shfl_xor_sync(~0u, a.x, m), __shfl_xor_sync(~0u, a.y, m), __shfl_xor_sync(~0u, a.z, m));
}

// One axis of the swept box against a node's box, as the interval of s (0
// at the start box, 1 at the end box) in which they overlap: entered at
// plane * x + y and left at plane * z + w.  Moving up the axis, the high side
// passes the lower plane first and the low side the upper plane last;
// moving down (`down`) the planes swap.  Where the two sides do not move the
// same way the axis is bounded by its whole range instead (a slope of
// 1e-20: every s inside it, none outside).
UPBP_D float4 sweep_axis(float alo, float ahi, float blo, float bhi, float pad, bool& down)
{
    alo -= pad;
    blo -= pad;
    ahi += pad;
    bhi += pad;
    float el = blo - alo, eh = bhi - ahi;
    down = el < -1e-12f && eh < -1e-12f;
    if (!down && !(el > 1e-12f && eh > 1e-12f)) {
        alo = fminf(alo, blo);
        ahi = fmaxf(ahi, bhi);
        el = eh = 1e-20f;
    }
    const float il = 1.f / el, ih = 1.f / eh;
    const float ol = -alo * il, oh = -ahi * ih;
    return down ? make_float4(il, ol, ih, oh) : make_float4(ih, oh, il, ol);
}

// Three-input minimum and maximum (one instruction on sm_100).
UPBP_D float fmin3(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
UPBP_D float fmax3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// State of a warp's search; the scalars have the same value in every lane.
struct PacketState {
    int sp;                     // nodes on the stack
    int nleaf, npair, nhit;     // waiting leaves, pairs and hits
    unsigned long long seen;    // hit total after the last reservation
    unsigned long long at;      // next slot of the warp's reserved part of the hit list
    unsigned room, grab;        // slots left of it, slots to reserve next
    unsigned visits;            // of the warp
    unsigned cand, hits;        // of the lane
    bool overflow;
    bool exact;                 // the round has one query
};

// Reserves the warp's next part of the hit list.  One atomic on the list's
// total per 32 hits held the whole search to about two nanoseconds for each
// (they all meet at one address): a warp that finds many pairs reserves ever
// larger parts, up to hit_reserve slots, and marks at the end what it did not
// use.  A round of one query (`exact`) reserves by 32 only, whatever the list,
// so that a list its pairs just fit is enough.
UPBP_D void packet_reserve(PacketState& s, unsigned lane)
{
    const DeviceParams& p = c_params;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&p.hit_state->total, (unsigned long long)s.grab);
    s.at = __shfl_sync(~0u, base, 0);
    s.room = s.grab;
    s.seen = s.at + s.grab;
    s.grab = s.exact ? 32u : min(2u * s.grab, p.hit_reserve);
}

// Accepted pairs of up to 32 lanes, gathered by 32 for the hit list.
UPBP_D void packet_hits(SearchWarp& w, PacketState& s, unsigned lane, bool hit, uint2 qb)
{
    const DeviceParams& p = c_params;
    const unsigned m = __ballot_sync(~0u, hit);
    if (!m) return;
    if (hit) {
        w.hit_qb[s.nhit + __popc(m & ((1u << lane) - 1u))] = qb;
        s.hits++;
    }
    s.nhit += __popc(m);
    if (s.nhit >= 32) {
        __syncwarp();
        if (s.room == 0) packet_reserve(s, lane);
        // streamed: the list is larger than the L2, which the map needs
        if (s.at + lane < p.hit_capacity) __stcs(p.hit_qb + s.at + lane, w.hit_qb[lane]);
        s.at += 32;
        s.room -= 32;
        __syncwarp();
        if ((int)lane + 32 < s.nhit) w.hit_qb[lane] = w.hit_qb[lane + 32];
        s.nhit -= 32;
    }
    __syncwarp();
}

// The exact BB1D test of the `count` (at most 32) oldest waiting pairs.
UPBP_D void packet_pairs(SearchWarp& w, PacketState& s, unsigned lane, int count)
{
    const DeviceParams& p = c_params;
    __syncwarp();
    bool hit = false;
    uint2 qb = make_uint2(0u, 0u);
    if ((int)lane < count) {
        const unsigned pr = w.pairs[lane];
        const unsigned leaf = pr & ((1u << kLeafShift) - 1u), j = pr >> kLeafShift;
        const float4 q0 = w.qa[j], q1 = w.qb[j];
        const uint2 qk = w.qk[j];
        qb.x = qk.x;
        BeamSegHit h;
        hit = beam_chunk_vs_segment(p.beam_map, (int)leaf, xyz(q0), xyz(q1), q0.w, q1.w, p.radius_bb1d_2,
                                    p.do_bp2d != 0, (int)qk.y, s.cand, h);
        qb.y = h.beam;
    }
    __syncwarp();
    if ((int)lane + count < s.npair) w.pairs[lane] = w.pairs[lane + count];
    s.npair -= count;
    packet_hits(w, s, lane, hit, qb);
}

// Up to 32 waiting leaves, one per lane, against the queries of their group.
template <int kMode>
UPBP_D void packet_leaves(SearchWarp& w, PacketState& s, unsigned lane)
{
    const DeviceParams& p = c_params;
    __syncwarp();
    const int n = min(s.nleaf, 32);
    const bool mine = (int)lane < n;
    const unsigned entry = mine ? w.leaves[s.nleaf - n + lane] : 0u;
    const unsigned leaf = entry & kEntryMask;
    unsigned m = mine ? w.group[entry >> kLeafShift].x : 0u;  // this lane's queries
    s.nleaf -= n;
    if constexpr (kMode == kModePb2d) {
        const float4 pp = __ldg(&p.med_map.pos[leaf]);
        s.cand += __popc(m);
        while (__any_sync(~0u, m != 0u)) {
            const int j = m ? __ffs(m) - 1 : 0;
            const float4 q0 = w.qa[j], q1 = w.qb[j];
            float dist, rad2;
            const bool hit = m && pred_ray_disc(xyz(q0), xyz(q1), q0.w, q1.w, xyz(pp), p.radius_pb2d_2, dist, rad2);
            m &= m - 1;
            packet_hits(w, s, lane, hit, make_uint2(w.qk[j].x, fbits(pp.w)));
        }
    } else if constexpr (kMode == kModeBp2d) {
        // the chunk holding the beam's closest point reports it
        const uint2 ch = __ldg(&p.beam_map.chunk[leaf]);
        const unsigned beam = ch.x & 0x7fffffffu, ck = ch.y & 0xffffu, cn = ch.y >> 16;
        const float4 s0 = __ldg(&p.beam_map.beams[beam].q[0]), s1 = __ldg(&p.beam_map.beams[beam].q[1]);
        const float t0 = chunk_t(s0.w, ck, cn), t1 = chunk_t(s0.w, ck + 1, cn);
        s.cand += __popc(m);
        while (__any_sync(~0u, m != 0u)) {
            const int j = m ? __ffs(m) - 1 : 0;
            const float4 q0 = w.qa[j];
            float dist, rad2;
            const bool hit = m && pred_ray_disc(xyz(s0), xyz(s1), 0.f, s0.w, xyz(q0), p.radius_bp2d_2, dist, rad2) &&
                             dist >= t0 && dist < t1;
            m &= m - 1;
            packet_hits(w, s, lane, hit, make_uint2(w.qk[j].x, beam));
        }
    } else {
        // A conservative form of pred_beam_beam on the chunk's part of the
        // beam: with the moments o x d of both lines, their distance times
        // sin theta is |d1 . m2 + d2 . m1|, and t1, t2 follow from the dot
        // products.  The margins cover the rounding of both forms: eps =
        // 4e-6 of the coordinates' magnitude for the distance (both forms
        // stay below 1.5e-6), and 1e-4 of it for t1 and t2 (each off by a few
        // 1e-7 of it over |d1.d2| sin^2 theta, so they are only looked at
        // where that product is above a tenth; the predicate's closest points
        // then lie well within the dilation, where the chunk that holds t2
        // reports).
        const uint2 ch = __ldg(&p.beam_map.chunk[leaf]);
        const BeamRec* beam = p.beam_map.beams + (ch.x & 0x7fffffffu);
        const float4 s0 = __ldg(&beam->q[0]), s1 = __ldg(&beam->q[1]);
        const float3 o2 = xyz(s0), d2 = xyz(s1), m2 = cross(o2, d2);
        const float o2d2 = dot(o2, d2);
        const float margin = p.beam_cull_eps, eps = 4.f * p.cull_eps;
        // the chunk's range, by a reciprocal (chunk_t divides) with its error in the margin
        const float per = s0.w * __frcp_rn((float)(ch.y >> 16)), from = (float)(ch.y & 0xffffu);
        const float slack = fmaf(1e-6f, s0.w, margin);
        const float t0 = fmaf(per, from, -slack), t1 = fmaf(per, from + 1.f, slack);
        const float r2 = 1.02f * p.radius_bb1d_2, add = fmaf(r2, 1e-6f, 51.f * eps * eps);
        if (p.do_bp2d && !(ch.x >> 31)) m = 0u;
        while (__any_sync(~0u, m != 0u)) {
            const int j = m ? __ffs(m) - 1 : 0;
            const float4 q0 = w.qa[j], q1 = w.qb[j], q2 = w.qc[j];
            const float3 o1 = xyz(q0), d1 = xyz(q1);
            const float dd = dot(d1, d2), ss = fmaf(-dd, dd, 1.f);
            const float ad = dot(d1, m2) + dot(d2, xyz(q2));
            const float wd1 = dot(o2, d1) - q2.w, wd2 = o2d2 - dot(o1, d2);
            const float n1 = fmaf(-dd, wd2, wd1), n2 = fmaf(dd, wd1, -wd2);
            const bool out = n2 < t0 * ss || n2 > t1 * ss || n1 < (q0.w - margin) * ss || n1 > (q1.w + margin) * ss;
            const bool pass = m && ad * ad < fmaf(r2, ss, add) && !(out && fabsf(dd) * ss > 0.1f);
            m &= m - 1;
            const unsigned pm = __ballot_sync(~0u, pass);
            if (pass) w.pairs[s.npair + __popc(pm & ((1u << lane) - 1u))] = leaf | (unsigned)j << kLeafShift;
            s.npair += __popc(pm);
            if (s.npair >= 32) packet_pairs(w, s, lane, 32);
        }
    }
    __syncwarp();
}

// The pairs of a packet's groups: the map's nodes against the bounds of the
// groups, 32 (node, group) entries at a time, and the leaves reached against
// the groups' queries.  The stack holds the first entries on entry.
template <int kMode>
UPBP_D void packet_walk(SearchWarp& w, PacketState& s, unsigned lane, const QNode4* nodes)
{
    for (;;) {
        if (s.nleaf >= 32 || s.sp == 0) {
            if (s.nleaf == 0) break;
            packet_leaves<kMode>(w, s, lane);
            continue;
        }
        __syncwarp();
        // as many entries as leave room for a depth-first walk of the rest (a
        // step adds at most three to the stack for each entry it takes)
        const int n = max(1, min(min(s.sp, 32), (kPacketStack - 2 * kStackDepth - s.sp) / 3));
        const bool mine = (int)lane < n;
        const unsigned entry = mine ? w.stack[s.sp - 1 - lane] : 0u;
        s.sp -= n;
        __syncwarp();
        unsigned hit = 0;   // children reached: bit c
        unsigned k0 = 0, k1 = 0;
        s.visits += n;
        if (mine) {
            const QNode4* nd = nodes + (entry & kEntryMask);
            const unsigned g = entry >> kLeafShift;
            const float4 a = __ldg(&nd->a);
            const uint4 b = __ldg(&nd->b), c = __ldg(&nd->c);
            const float4 gx = w.bound[0][g], gy = w.bound[1][g], gz = w.bound[2][g];
            const unsigned e = __float_as_uint(a.w);
            const float sx = qnode_step(e & 0xffu), sy = qnode_step((e >> 8) & 0xffu), sz = qnode_step((e >> 16) & 0xffu);
            auto q = [](unsigned word, int byte) { return (float)((word >> (8 * byte)) & 0xffu); };
            if constexpr (RangeMode<kMode>::seg) {
                // the planes entered first to the even bytes
                const unsigned down = w.group[g].y;
                const unsigned px = down & 1u ? 0x2301u : 0x3210u, py = down & 2u ? 0x2301u : 0x3210u,
                               pz = down & 4u ? 0x2301u : 0x3210u;
                const unsigned x0 = __byte_perm(b.x, 0u, px), x1 = __byte_perm(b.y, 0u, px);
                const unsigned y0 = __byte_perm(b.z, 0u, py), y1 = __byte_perm(b.w, 0u, py);
                const unsigned z0 = __byte_perm(c.x, 0u, pz), z1 = __byte_perm(c.y, 0u, pz);
                const float ex = sx * gx.x, ey = sy * gy.x, ez = sz * gz.x;
                const float lx = sx * gx.z, ly = sy * gy.z, lz = sz * gz.z;
                const float oex = fmaf(a.x, gx.x, gx.y), oey = fmaf(a.y, gy.x, gy.y), oez = fmaf(a.z, gz.x, gz.y);
                const float olx = fmaf(a.x, gx.z, gx.w), oly = fmaf(a.y, gy.z, gy.w), olz = fmaf(a.z, gz.z, gz.w);
                auto test = [&](unsigned wx, unsigned wy, unsigned wz, int k) {
                    const float tn = fmax3(fmaf(q(wx, k), ex, oex), fmaf(q(wy, k), ey, oey), fmaf(q(wz, k), ez, oez));
                    const float tf =
                        fmin3(fmaf(q(wx, k + 1), lx, olx), fmaf(q(wy, k + 1), ly, oly), fmaf(q(wz, k + 1), lz, olz));
                    return fmaxf(tn, 0.f) <= fminf(tf, 1.f);
                };
                hit = (test(x0, y0, z0, 0) ? 1u : 0u) | (test(x0, y0, z0, 2) ? 2u : 0u) |
                      (test(x1, y1, z1, 0) ? 4u : 0u) | (test(x1, y1, z1, 2) ? 8u : 0u);
            } else {
                auto test = [&](unsigned wx, unsigned wy, unsigned wz, int k) {
                    return fmaf(q(wx, k), sx, a.x) <= gx.y && fmaf(q(wx, k + 1), sx, a.x) >= gx.x &&
                           fmaf(q(wy, k), sy, a.y) <= gy.y && fmaf(q(wy, k + 1), sy, a.y) >= gy.x &&
                           fmaf(q(wz, k), sz, a.z) <= gz.y && fmaf(q(wz, k + 1), sz, a.z) >= gz.x;
                };
                hit = (test(b.x, b.z, c.x, 0) ? 1u : 0u) | (test(b.x, b.z, c.x, 2) ? 2u : 0u) |
                      (test(b.y, b.w, c.y, 0) ? 4u : 0u) | (test(b.y, b.w, c.y, 2) ? 8u : 0u);
            }
            k0 = c.z;
            k1 = c.w;
            hit &= ~((k0 & kQnodeSingle ? 2u : 0u) | (k1 & kQnodeSingle ? 8u : 0u));
        }
        // children reached: leaves wait for their test, inner nodes go onto
        // the stack (one scan of both counts over the lanes)
        const unsigned leafbits = (k0 & kQnodeLeaf0 ? 1u : 0u) | (k0 & kQnodeLeaf1 ? 2u : 0u) |
                                  (k1 & kQnodeLeaf0 ? 4u : 0u) | (k1 & kQnodeLeaf1 ? 8u : 0u);
        const unsigned leaf = hit & leafbits, inner = hit & ~leafbits;
        const unsigned own = __popc(inner) | __popc(leaf) << 16;
        unsigned sum = own;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const unsigned v = __shfl_up_sync(~0u, sum, d);
            if ((int)lane >= d) sum += v;
        }
        const unsigned total = __shfl_sync(~0u, sum, 31);
        const unsigned tag = entry & ~kEntryMask;
        const unsigned i0 = k0 & kEntryMask, i1 = k1 & kEntryMask;
        unsigned at = (unsigned)s.sp + ((sum - own) & 0xffffu), la = (unsigned)s.nleaf + ((sum - own) >> 16);
        if (inner) {
            if (inner & 1u) w.stack[at++] = i0 | tag;
            if (inner & 2u) w.stack[at++] = (i0 + 1u) | tag;
            if (inner & 4u) w.stack[at++] = i1 | tag;
            if (inner & 8u) w.stack[at++] = (i1 + 1u) | tag;
        }
        if (leaf) {
            if (leaf & 1u) w.leaves[la++] = i0 | tag;
            if (leaf & 2u) w.leaves[la++] = (i0 + 1u) | tag;
            if (leaf & 4u) w.leaves[la++] = i1 | tag;
            if (leaf & 8u) w.leaves[la++] = (i1 + 1u) | tag;
        }
        s.sp += total & 0xffffu;
        s.nleaf += total >> 16;
        if (s.sp > kPacketStack) {
            s.overflow = true;
            s.sp = kPacketStack;
        }
    }
}

template <int kMode>
__global__ void __launch_bounds__(kPassThreads, 7) range_search_kernel(int slot)
{
    using M = RangeMode<kMode>;
    begin_kernel(M::kern, slot);
    const DeviceParams& p = c_params;
    __shared__ SearchWarp s_warp[kPassWarps];
    SearchWarp& w = s_warp[threadIdx.x >> 5];
    const unsigned lane = threadIdx.x & 31;
    // this round's range of the processing order, within the queue
    const unsigned nq = M::seg ? min(p.queue_count[0], p.seg_capacity) : min(p.queue_count[1], p.pt_capacity);
    const unsigned n = min(p.query_end, nq) - min(p.query_begin, min(p.query_end, nq));
    // Queries a warp takes at once, a power of two: an even share of the
    // queries left, split units_per_warp ways so that the warps finish
    // together, and no more than unit_max (range_search_split).
    const unsigned share = gridDim.x * kPassWarps * p.units_per_warp;
    auto next_unit = [&](unsigned left) {
        const unsigned u = left / share;
        return u >= p.unit_max ? p.unit_max : u <= 1u ? 1u : 1u << (31 - __clz(u));
    };
    unsigned unit = next_unit(n);
    const BvhView bvh = range_map_bvh<kMode>();
    float3 rlo = v3(-kInfinity), rhi = v3(kInfinity);  // box of the whole map
    if (M::seg && bvh.count > 1) {
        const float4 a = __ldg(&bvh.qnodes[0].a);
        const unsigned e = __float_as_uint(a.w);
        const float3 step = make_float3(qnode_step(e & 0xffu), qnode_step((e >> 8) & 0xffu), qnode_step((e >> 16) & 0xffu));
        const float3 pad = v3(4.f * p.cull_eps);
        rlo = xyz(a) - pad;
        rhi = xyz(a) + 255.f * step + pad;
    }
    PacketState s;
    s.sp = s.nleaf = s.npair = s.nhit = 0;
    s.seen = s.at = 0;
    s.room = 0;
    s.grab = 32;
    s.visits = s.cand = s.hits = 0;
    s.overflow = false;
    s.exact = n <= 1u;
    for (;;) {
        // no new queries once the hit list is 3/4 full, as far as this warp
        // saw at its last flush of hits
        unsigned base = ~0u;
        if (lane == 0 && s.seen < p.hit_soft_limit) base = atomicAdd(&p.hit_state->fetched, unit);
        base = __shfl_sync(~0u, base, 0);
        if (base >= n) break;
        const unsigned take = unit;
        unit = next_unit(n - base);
        bool active = lane < take && base + lane < n;
        PacketBox box;
        box.alo = box.blo = v3(kInfinity);
        box.ahi = box.bhi = v3(-kInfinity);
        if (active) {
            const unsigned j = p.query_begin + base + lane;
            if constexpr (M::seg) {
                const unsigned qk = p.seg_order ? __ldg(&p.seg_order[j]) : j;
                const float4* r = p.seg_queue[qk].q;
                const float4 q0 = __ldg(&r[0]), q1 = __ldg(&r[1]);
                const float3 o = xyz(q0), d = xyz(q1);
                w.qk[lane] = make_uint2(qk, kMode == kModeBb1d ? fbits(__ldg(&r[2]).w) : 0u);
                w.qa[lane] = q0;
                w.qb[lane] = q1;
                if (kMode == kModeBb1d) {
                    const float3 m1 = cross(o, d);
                    w.qc[lane] = make_float4(m1.x, m1.y, m1.z, dot(o, d));
                }
                // the part of the segment inside the map's box
                auto away = [](float x) { return fabsf(x) > 1e-20f ? x : 1e-20f; };
                const float3 inv = safe_inv(make_float3(away(d.x), away(d.y), away(d.z))), oi = oinv_of(o, inv);
                const float x0 = fmaf(rlo.x, inv.x, -oi.x), x1 = fmaf(rhi.x, inv.x, -oi.x);
                const float y0 = fmaf(rlo.y, inv.y, -oi.y), y1 = fmaf(rhi.y, inv.y, -oi.y);
                const float z0 = fmaf(rlo.z, inv.z, -oi.z), z1 = fmaf(rhi.z, inv.z, -oi.z);
                const float ta = fmaxf(fmaxf(fminf(x0, x1), fminf(y0, y1)), fmaxf(fminf(z0, z1), q0.w));
                const float tb = fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fminf(fmaxf(z0, z1), q1.w));
                active = ta <= tb;
                if (active) {
                    const float3 a = o + d * ta, b = o + d * tb;
                    box.alo = box.ahi = a;
                    box.blo = box.bhi = b;
                }
            } else {
                // point queries of other estimators, or of camera paths that
                // failed earlier, are skipped
                const unsigned qk = p.pt_order ? __ldg(&p.pt_order[j]) : j;
                const float4 q8 = __ldg(&p.pt_queue[qk].q8);
                active = (fbits(q8.y) & kQueryBp2d) && event_kept(fbits(q8.z), fbits(q8.w));
                if (active) {
                    const float4 q0 = __ldg(&p.pt_queue[qk].v.q[0]);
                    w.qk[lane] = make_uint2(qk, 0u);
                    w.qa[lane] = q0;
                    box.alo = box.ahi = box.blo = box.bhi = xyz(q0);
                }
            }
        }
        const unsigned live = __ballot_sync(~0u, active);
        if (!live) continue;
        __syncwarp();
        // groups: the largest aligned runs of 2^k queries whose boxes stay
        // within the spread limit
        const float limit = p.group_spread;
        int level = 0;
        {
            PacketBox b = box;
            for (int k = 0; (1u << k) < take; k++) {
                const int x = 1 << k;
                b.alo = min3f(b.alo, shfl3_xor(b.alo, x));
                b.ahi = max3f(b.ahi, shfl3_xor(b.ahi, x));
                if constexpr (M::seg) {
                    b.blo = min3f(b.blo, shfl3_xor(b.blo, x));
                    b.bhi = max3f(b.bhi, shfl3_xor(b.bhi, x));
                }
                float spread = max_component(b.ahi - b.alo);
                if constexpr (M::seg) spread = fmaxf(spread, max_component(b.bhi - b.blo));
                const bool both = __shfl_xor_sync(~0u, level, x) == k && level == k;
                if (both && spread <= limit) {
                    level = k + 1;
                    box = b;
                }
            }
        }
        {
            // a group is named by its first query, whose lane writes its bound
            const unsigned first = lane & ~((1u << level) - 1u);
            const unsigned group = live & (level == 5 ? ~0u : ((1u << (1 << level)) - 1u) << first);
            const bool leads = lane == first && group != 0u;
            if (leads) {
                unsigned down = 0;
                if constexpr (M::seg) {
                    const float pad = 4.f * p.cull_eps;
                    bool dx, dy, dz;
                    w.bound[0][lane] = sweep_axis(box.alo.x, box.ahi.x, box.blo.x, box.bhi.x, pad, dx);
                    w.bound[1][lane] = sweep_axis(box.alo.y, box.ahi.y, box.blo.y, box.bhi.y, pad, dy);
                    w.bound[2][lane] = sweep_axis(box.alo.z, box.ahi.z, box.blo.z, box.bhi.z, pad, dz);
                    down = (dx ? 1u : 0u) | (dy ? 2u : 0u) | (dz ? 4u : 0u);
                } else {
                    w.bound[0][lane] = make_float4(box.alo.x, box.ahi.x, 0.f, 0.f);
                    w.bound[1][lane] = make_float4(box.alo.y, box.ahi.y, 0.f, 0.f);
                    w.bound[2][lane] = make_float4(box.alo.z, box.ahi.z, 0.f, 0.f);
                }
                w.group[lane] = make_uint2(group, down);
            }
            const unsigned lead = __ballot_sync(~0u, leads);
            const int at = __popc(lead & ((1u << lane) - 1u));
            // every group starts at the root (a one-leaf map: at its leaf)
            s.sp = bvh.count > 1 ? __popc(lead) : 0;
            s.nleaf = bvh.count == 1 ? __popc(lead) : 0;
            if (leads) (bvh.count > 1 ? w.stack : w.leaves)[at] = lane << kLeafShift;
        }
        packet_walk<kMode>(w, s, lane, bvh.qnodes);
        // the waiting pairs name this packet's queries
        if (s.npair) packet_pairs(w, s, lane, s.npair);
        __syncwarp();
    }
    __syncwarp();
    // the last hits, and the unused slots of the warp's part marked empty
    if (s.nhit && s.room == 0) {
        s.grab = (unsigned)s.nhit;
        packet_reserve(s, lane);
    }
    for (unsigned k = lane; k < s.room; k += 32)
        if (s.at + k < p.hit_capacity) __stcs(p.hit_qb + s.at + k, k < (unsigned)s.nhit ? w.hit_qb[k] : make_uint2(kNoHit, 0u));
    count_work(kCtrNodes, lane == 0 ? s.visits : 0u);
    count_work(M::beams ? kCtrBeamCand : kCtrPointCand, s.cand);
    count_work(M::beams ? kCtrBeamHit : kCtrPointHit, s.hits);
    if (s.overflow) flag_status(kErrTraversalStack);
}

}  // namespace upbp
