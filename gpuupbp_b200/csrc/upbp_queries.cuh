// Range queries over the per-iteration photon maps.  Each walker visits the
// BVH leaves whose box (built dilated by the map's largest query radius) the
// query touches, and
// calls f for every photon or beam that passes the estimator's exact
// predicate; the neighbour set is therefore defined by the predicate alone
// (the reference's OptiX intersection programs apply the same predicates,
// gpuupbp/kernel/pde/program_*.cu).  Rendering uses points_in_radius_warp
// (SURF, PP3D) and the packet searches of upbp_range_search.cuh, which share
// the leaf tests here; the walkers of one query per lane (points_in_radius,
// points_near_segment, beams_near_segment, beams_near_point) serve the
// diagnostic neighbour-set query (upbp_debug_query), another route to the
// same sets.
#pragma once

#include "upbp_paths.cuh"

namespace upbp {

// Photons within radius r of x (SURF, PP3D): f(vertex slot).
template <class F>
UPBP_D void points_in_radius(const PointMap& map, float3 x, float r2, F&& f)
{
    unsigned cand = 0, hits = 0;
    const bool ok = bvh_walk(
        map.bvh, [&](float3 lo, float3 hi) { return inside(lo, hi, x); },
        [&](int i) {
            const float4 pp = __ldg(&map.pos[i]);
            cand++;
            if (pred_point_point(x, xyz(pp), r2)) {
                hits++;
                f(fbits(pp.w));
            }
            return true;
        });
    count_work(kCtrPointCand, cand);
    count_work(kCtrPointHit, hits);
    if (!ok) flag_status(kErrTraversalStack);
}

// The same by a whole warp, one query per lane (`on` tells which lanes have
// one): f as above, at most once a step, and step() by every lane after each
// step of the walks.  The caller counts what it merges.
template <class F, class S>
UPBP_D void points_in_radius_warp(bool on, const PointMap& map, float3 x, float r2, F&& f, S&& step)
{
    unsigned visits = 0, cand = 0;
    bool ok = true;
    int stack[kStackDepth];
    int sp = 0;
    int node = on && map.bvh.count > 0 ? (map.bvh.count > 1 ? 0 : ~0) : kWalkDone;
    while (__any_sync(~0u, node != kWalkDone)) {
        bool pop = false;
        if (node >= 0) {
            visits++;
            const NodeBoxes nb = load_node(map.bvh.nodes, node);
            const bool hl = inside(nb.llo, nb.lhi, x), hr = inside(nb.rlo, nb.rhi, x);
            if (hl && hr) {
                if (sp < kStackDepth)
                    stack[sp++] = nb.r;
                else
                    ok = false;
            }
            if (hl || hr)
                node = hl ? nb.l : nb.r;
            else
                pop = true;
        }
        if (!pop && node < 0 && node != kWalkDone) {
            const int first = leaf_first(node), cnt = leaf_count(node);
            const float4 pp = __ldg(&map.pos[first]);
            cand++;
            if (pred_point_point(x, xyz(pp), r2)) f(fbits(pp.w));
            if (cnt > 1)
                node = leaf_link(first + 1, cnt - 1);
            else
                pop = true;
        }
        if (pop) node = sp > 0 ? stack[--sp] : kWalkDone;
        step();
    }
    if (!on) return;
    count_work(kCtrNodes, visits);
    count_work(kCtrPointCand, cand);
    if (!ok) flag_status(kErrTraversalStack);
}

// Photons whose disc of radius r the query segment (o, d, (tmin, tmax))
// crosses (PB2D): f(vertex slot, distance along the query, squared radius).
template <class F>
UPBP_D void points_near_segment(const PointMap& map, float3 o, float3 d, float tmin, float tmax, float r2, F&& f)
{
    const float3 inv = safe_inv(d), oinv = oinv_of(o, inv);
    unsigned cand = 0, hits = 0;
    const bool ok = bvh_walk(
        map.bvh, [&](float3 lo, float3 hi) { return slab(lo, hi, inv, oinv, tmin, tmax); },
        [&](int i) {
            const float4 pp = __ldg(&map.pos[i]);
            float dist, rad2;
            cand++;
            if (pred_ray_disc(o, d, tmin, tmax, xyz(pp), r2, dist, rad2)) {
                hits++;
                f(fbits(pp.w), dist, rad2);
            }
            return true;
        });
    count_work(kCtrPointCand, cand);
    count_work(kCtrPointHit, hits);
    if (!ok) flag_status(kErrTraversalStack);
}

// Photon beams passing within sqrt(r2) of the query segment (BB1D); with
// need_mask only beams of the first bb1d_used_light_subpath_count light
// paths.  f(beam index, distance, sin theta, t along query, t along beam).
// Beams are stored as chunks; a beam is reported only through the chunk that
// holds its closest point, so each beam appears at most once.  med >= 0
// skips beams of other media before the predicate (the estimator only merges
// beams in the query segment's medium, functs_bb1d.cuh:66).
struct BeamSegHit {
    unsigned beam;
    float dist, sin_theta, t1, t2;
};

// Segment [tmin, tmax] of (o, d) vs chunk k of n of a beam, with the box
// test of the beam-map walk (same box, same dilation, same arithmetic).
UPBP_D bool chunk_reached(float3 bo, float3 bd, float len, unsigned k, unsigned n, float dilate, float3 o, float3 d,
                          float tmin, float tmax)
{
    float3 lo, hi;
    chunk_box(bo, bd, len, k, n, lo, hi);
    dilate_box(lo, hi, dilate);
    const float3 inv = safe_inv(d);
    return slab(lo, hi, inv, oinv_of(o, inv), tmin, tmax);
}

// The BB1D test of one beam-map leaf against a query segment: the path mask,
// the exact beam-beam predicate, which looks at the whole beam, so every
// chunk of an accepted beam passes it, and the medium filter; one of the
// chunks reports the beam.  That is the chunk holding the beam's closest
// point t2 when the query reaches its box.  The predicate's t2 can be far
// from the true closest point (it divides by d1.d2, which is tiny for nearly
// perpendicular lines), and then the chunk holding it can lie outside the
// query's reach: in that case the first chunk of the beam whose box the query
// reaches reports instead (a check that is only needed when the computed
// closest points are far apart).  A walk tests at least the chunks whose
// boxes the query reaches, so exactly one chunk reports each accepted beam,
// and the set equals a test of every beam, however many further chunks the
// walk tests.  cand counts the leaves that reach the predicate.
UPBP_D bool beam_chunk_vs_segment(const BeamMap& map, int i, float3 o, float3 d, float tmin, float tmax, float r2,
                                  bool need_mask, int med, unsigned& cand, BeamSegHit& h)
{
    const uint2 ch = __ldg(&map.chunk[i]);
    const unsigned bits = ch.x;
    if (need_mask && !(bits >> 31)) return false;
    const BeamRec* beam = map.beams + (bits & 0x7fffffffu);
    const float4 s0 = __ldg(&beam->q[0]), s1 = __ldg(&beam->q[1]);
    cand++;
    if (!pred_beam_beam(o, d, tmin, tmax, xyz(s0), xyz(s1), s0.w, r2, h.dist, h.sin_theta, h.t1, h.t2)) return false;
    if (med >= 0 && (int)fbits(s1.w) != med) return false;
    h.beam = bits & 0x7fffffffu;
    const unsigned k = ch.y & 0xffffu, n = ch.y >> 16;
    const bool mine = h.t2 >= chunk_t(s0.w, k, n) && h.t2 < chunk_t(s0.w, k + 1, n);
    const float3 bo = xyz(s0), bd = xyz(s1);
    // Usual case: the computed closest points lie within the dilation of each
    // other (less a rounding margin), so the query passes through the dilated
    // own box of the chunk holding t2 at t1, and the walk reached that chunk.
    const float3 gap = (o + d * h.t1) - (bo + bd * h.t2);
    const float inner = map.dilate - 2.f * c_params.cull_eps;
    if (inner > 0.f && dot(gap, gap) <= inner * inner) return mine;
    // a walk may test a chunk out of the query's reach, so its own box
    // decides, as for every other chunk
    if (!chunk_reached(bo, bd, s0.w, k, n, map.dilate, o, d, tmin, tmax)) return false;
    if (mine) return true;
    if (chunk_reached(bo, bd, s0.w, chunk_of(h.t2, s0.w, n), n, map.dilate, o, d, tmin, tmax)) return false;
    for (unsigned j = 0; j < k; j++)
        if (chunk_reached(bo, bd, s0.w, j, n, map.dilate, o, d, tmin, tmax)) return false;
    return true;
}

template <class F>
UPBP_D void beams_near_segment(const BeamMap& map, float3 o, float3 d, float tmin, float tmax, float r2,
                               bool need_mask, int med, F&& f)
{
    const float3 inv = safe_inv(d), oinv = oinv_of(o, inv);
    unsigned cand = 0, hits = 0, visits = 0;
    bool overflow = false;
    WalkState s;
    walk_begin(s, map.bvh);
    while (s.node != kWalkDone) {
        const int leaf = walk_step(
            s, map.bvh, [&](float3 lo, float3 hi) { return slab(lo, hi, inv, oinv, tmin, tmax); }, overflow, visits);
        BeamSegHit h;
        if (leaf >= 0 &&
            beam_chunk_vs_segment(map, leaf, o, d, tmin, tmax, r2, need_mask, med, cand, h)) {
            hits++;
            f(h.beam, h.dist, h.sin_theta, h.t1, h.t2);
        }
    }
    count_work(kCtrNodes, visits);
    count_work(kCtrBeamCand, cand);
    count_work(kCtrBeamHit, hits);
    if (overflow) flag_status(kErrTraversalStack);
}

// The BP2D test of one beam-map leaf against a point: the exact ray-disc
// predicate on the whole beam; the chunk holding its closest point reports it.
UPBP_D bool beam_chunk_vs_point(const BeamMap& map, int i, float3 x, float r2, unsigned& beam, float& dist, float& rad2)
{
    const uint2 ch = __ldg(&map.chunk[i]);
    beam = ch.x & 0x7fffffffu;
    const float4 s0 = __ldg(&map.beams[beam].q[0]), s1 = __ldg(&map.beams[beam].q[1]);
    if (!pred_ray_disc(xyz(s0), xyz(s1), 0.f, s0.w, x, r2, dist, rad2)) return false;
    const unsigned k = ch.y & 0xffffu, n = ch.y >> 16;
    return dist >= chunk_t(s0.w, k, n) && dist < chunk_t(s0.w, k + 1, n);
}

// Photon beams whose disc of radius sqrt(r2) contains x (BP2D):
// f(beam index, distance along the beam, squared radius).
template <class F>
UPBP_D void beams_near_point(const BeamMap& map, float3 x, float r2, F&& f)
{
    unsigned cand = 0, hits = 0;
    const bool ok = bvh_walk(
        map.bvh, [&](float3 lo, float3 hi) { return inside(lo, hi, x); },
        [&](int i) {
            float dist, rad2;
            unsigned beam;
            cand++;
            if (beam_chunk_vs_point(map, i, x, r2, beam, dist, rad2)) {
                hits++;
                f(beam, dist, rad2);
            }
            return true;
        });
    count_work(kCtrBeamCand, cand);
    count_work(kCtrBeamHit, hits);
    if (!ok) flag_status(kErrTraversalStack);
}

}  // namespace upbp
