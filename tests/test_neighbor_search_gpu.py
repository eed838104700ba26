"""The searches that render find the neighbour sets of a brute-force search
with the same exact predicates (oracle/neighbors.py): the packet searches of
PB2D, BB1D and BP2D -- shared bounds, the clip to the map's box, the
conservative BB1D test before the exact one, hit slots, rounds -- and the
merging walk of SURF and PP3D with its pending photons (upbp_debug_search).

How queries share a walk depends on how many a warp takes and how close their
ends lie; here both are set, so that the same queries are searched alone, in
the groups of an iteration, and in groups far wider than an iteration's."""
import os

import numpy as np
import pytest

import neighbors
from gpuupbp_b200 import scenes
from test_neighbors_gpu import _beam_frames, _beam_pair_ill_posed, _media_renderer, _renderer

pytestmark = pytest.mark.gpu

ALL6 = "upbp_bpt+surf+pp3d+pb2d+bb1d+bp2d"
# (grid limit, queries a warp takes, spread of a group in query radii; 0: the renderer's)
SPLITS = [(0, 0, 0), (0, 1, 0), (1, 8, 4), (1, 32, 1000)]


def _check(r, kind, queries, brute, radius, splits=SPLITS, ignore=None):
    """Sets equal brute force under every split; ignore(query, id) leaves a
    pair out on both sides.  Returns the sizes of the sets."""
    want = [np.sort(brute(q)) for q in queries]
    if ignore is not None:
        want = [np.array([i for i in w if not ignore(q, i)], np.int64) for q, w in zip(queries, want)]
    for limit, unit, spread in splits:
        assert r._L.upbp_set_grid_limit(r._ctx, limit) == 0
        sets, counts = r.search(kind, queries, unit, spread * radius)
        assert counts.max() <= 4096
        for k, (q, got, w) in enumerate(zip(queries, sets, want)):
            assert len(got) == counts[k] == len(np.unique(got)), "duplicate neighbour"
            if ignore is not None:
                got = np.array([i for i in got if not ignore(q, i)], np.int64)
            assert np.array_equal(np.sort(got), w), (kind, limit, unit, spread, k, q.tolist(), np.setxor1d(got, w))
    assert r._L.upbp_set_grid_limit(r._ctx, 0) == 0
    return np.array([len(w) for w in want])


def _points(x):
    q = np.zeros((len(x), 8), np.float32)
    q[:, :3] = x
    return q


def _unit(d):
    return (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def _segments(rng, centres, size, fan=32):
    """Segments through `centres`: the first third each of its own direction,
    the second in fans of `fan` from one start, the rest along the axes (two
    components of the direction are zero), some unbounded, some short, some
    that start or end far outside the map."""
    n = len(centres)
    q = np.zeros((n, 8), np.float32)
    d = rng.normal(size=(n, 3))
    a, b = n // 3, 2 * n // 3
    start = centres - _unit(d) * size
    for k in range(a, b):
        if (k - a) % fan == 0:
            s = centres[k] - _unit(rng.normal(size=(1, 3)))[0] * size
        start[k] = s
        # neighbours in a fan pass close to one another
        d[k] = centres[k - (k - a) % fan] + rng.normal(size=3) * 0.02 * size - s
    axis = rng.integers(0, 3, n)
    for k in range(b, n):
        d[k] = 0.0
        d[k, axis[k]] = rng.choice([-1.0, 1.0])
        start[k] = centres[k] - d[k] * size
    q[:, :3] = start
    q[:, 3:6] = _unit(d)
    q[:, 6] = np.where(rng.random(n) < 0.5, 0.0, rng.uniform(0.0, 0.5 * size, n))
    q[:, 7] = rng.uniform(size, 2 * size, n)
    odd = rng.random(n)
    q[odd < 0.1, 7] = np.inf
    q[(odd >= 0.1) & (odd < 0.15), 7] = 1e-3 * size
    far = (odd >= 0.15) & (odd < 0.25)
    q[far, :3] -= q[far, 3:6] * np.float32(50 * size)
    q[far, 6] = 0.0
    q[far, 7] = np.float32(60 * size)
    return q


def _path_limit(r):
    """Beams of the first so many light paths are BB1D's, with BP2D on."""
    used = r.config.bb1d_used_light_subpath_count
    return int(used) if used > 0 else int(np.floor(-used * r.config.path_count_per_iter))


@pytest.mark.parametrize("workload,tiny,args", [
    ("box_medium", False, ["-l", "8", "-r", "64x64", "-r_initial", "-0.02"]),
    ("dense_beams", True, ["-l", "16", "-r", "48x48", "-r_initial_bb1d", "-0.004", "-r_initial_bp2d", "-0.004",
                           "-pbc", "-0.5"]),
    ("media_field", True, ["-l", "12", "-r", "64x64"]),
])
def test_searches_equal_brute_force(scene_dir, workload, tiny, args):
    r = _renderer(scene_dir, workload, tiny, ["-a", ALL6] + args)
    rb1, rb2, rpb, rpp, rsu, _ = r.stats()["radius"]
    surf, med, beams = r.photons(0), r.photons(1), r.photons(2)
    assert len(surf) and len(med) and len(beams)
    rng = np.random.default_rng(17)
    slots_s, slots_m = surf[:, 3].view(np.uint32), med[:, 3].view(np.uint32)
    n = 801  # not a multiple of a warp; with one block, units of 32

    def near(pts, scale):
        p = pts[np.sort(rng.integers(0, len(pts), n)), :3]  # neighbours in the map are neighbours here
        return (p + rng.normal(size=p.shape) * scale).astype(np.float32)

    got = _check(r, 0, _points(near(surf, rsu)), lambda q: slots_s[neighbors.points_in_radius(surf, q[:3], np.float32(rsu) ** 2)],
                 rsu)
    assert (got > 0).sum() > 100
    got = _check(r, 1, _points(near(med, rpp)), lambda q: slots_m[neighbors.points_in_radius(med, q[:3], np.float32(rpp) ** 2)],
                 rpp)
    assert (got > 0).sum() > 100
    size = float(np.median(beams[:, 3]))
    got = _check(r, 2, _segments(rng, near(med, rpb), size),
                 lambda q: slots_m[neighbors.points_near_segment(med, q, np.float32(rpb) ** 2)], rpb)
    assert (got > 0).sum() > 100
    pick = beams[np.sort(rng.integers(0, len(beams), n))]
    on_beam = pick[:, :3] + pick[:, 4:7] * (rng.uniform(0, 1, n).astype(np.float32) * pick[:, 3])[:, None]
    centres = (on_beam + rng.normal(size=(n, 3)) * rb1).astype(np.float32)
    limit = _path_limit(r)
    # pairs on which the predicate itself hangs on rounding are left out
    # (_beam_pair_ill_posed tells which and why)
    got = _check(r, 3, _segments(rng, centres, size),
                 lambda q: neighbors.beams_near_segment(beams, q, np.float32(rb1) ** 2, limit), rb1,
                 ignore=lambda q, i: _beam_pair_ill_posed(q, beams[i], rb1))
    assert (got > 0).sum() > 50
    x = (on_beam + rng.normal(size=(n, 3)) * rb2).astype(np.float32)
    got = _check(r, 4, _points(x), lambda q: neighbors.beams_near_point(beams, q[:3], np.float32(rb2) ** 2), rb2)
    assert (got > 0).sum() > 100
    r.close()


@pytest.mark.parametrize("sort", [True, False])
def test_near_parallel_bb1d(scene_dir, sort):
    """Queries almost parallel to a beam, where both forms of the test -- the
    conservative one and the exact -- carry their largest errors in t; half of
    them end just short of the closest approach."""
    r = _media_renderer(scene_dir)
    rb1 = np.float32(r.stats()["radius"][0])
    beams = r.photons(2)
    rng = np.random.default_rng(31)
    n = 1501
    d2, u, v, mid = _beam_frames(beams, rb1, rng, n)
    sin2 = 10.0 ** rng.uniform(np.log10(1.5e-5), -3.0, n)
    d1 = np.sqrt(1.0 - sin2)[:, None] * d2 + np.sqrt(sin2)[:, None] * u
    centre = mid + v * (float(rb1) * rng.uniform(0.5, 0.999, n))[:, None]
    half = 20.0 * float(rb1)
    q = np.zeros((n, 8), np.float32)
    q[:, :3] = centre - d1 * half
    q[:, 3:6] = _unit(d1)
    q[:, 7] = 2 * half
    short = np.arange(n) % 2 == 1
    extent = float(np.abs(beams[:, :3]).max())
    q[short, 7] = half - rng.uniform(0.0, 0.02 * extent, short.sum())
    q = q[q[:, 7] > 0.0]
    if sort:
        q = q[np.lexsort(q[:, :3].T)]
    got = _check(r, 3, q, lambda qq: neighbors.beams_near_segment(beams, qq, rb1 ** 2), rb1,
                 ignore=lambda qq, i: _beam_pair_ill_posed(qq, beams[i], rb1))
    assert (got > 0).sum() > n // 4
    r.close()


def test_near_perpendicular_bb1d(scene_dir):
    """Queries almost perpendicular to a beam, where the exact predicate's t2
    divides by a tiny d1.d2 and lands far from the true closest point."""
    r = _media_renderer(scene_dir)
    rb1 = np.float32(r.stats()["radius"][0])
    beams = r.photons(2)
    rng = np.random.default_rng(37)
    n = 1501
    d2, u, v, mid = _beam_frames(beams, rb1, rng, n)
    eps = 10.0 ** rng.uniform(-7.0, -2.0, n) * rng.choice([-1.0, 1.0], n)
    d1 = u + eps[:, None] * d2
    d1 /= np.linalg.norm(d1, axis=1, keepdims=True)
    w = np.cross(d1, d2)
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    centre = mid + w * (float(rb1) * rng.uniform(0.0, 0.999, n))[:, None]
    half = float(rb1) * rng.uniform(2.0, 10.0, n)
    q = np.zeros((n, 8), np.float32)
    q[:, :3] = centre - d1 * half[:, None]
    q[:, 3:6] = _unit(d1)
    q[:, 7] = 2 * half
    got = _check(r, 3, q, lambda qq: neighbors.beams_near_segment(beams, qq, rb1 ** 2), rb1)
    assert (got > 0).sum() > n // 4
    r.close()


@pytest.mark.parametrize("iteration,leaves", [(0, (1, 0)), (1, (2, 1)), (4, (0, 0))])
def test_smallest_maps(scene_dir, iteration, leaves):
    """A beam map of one chunk and of two, a medium photon map of one, empty
    maps: one light path at a radius of a fifth of the scene's."""
    from gpuupbp_b200 import upbp
    path = scenes.write_workload("box_medium", scene_dir, tiny=True)
    r = upbp.Renderer(["-s", "-1", path, "-a", ALL6, "-l", "8", "-r", "33x29", "-pcpi", "1", "-r_initial", "-0.2"])
    r.run_iteration(iteration)
    rb1, rb2, rpb, rpp, rsu, _ = r.stats()["radius"]
    med, beams = r.photons(1), r.photons(2)
    assert (len(beams), len(med)) == leaves and r.beam_map()["chunks"] == leaves[0]
    slots = med[:, 3].view(np.uint32)
    rng = np.random.default_rng(47)
    n = 77
    centres = rng.uniform(-0.5, 0.5, (n, 3))
    if len(beams):
        centres = beams[rng.integers(0, len(beams), n), :3] + rng.normal(size=(n, 3)) * 0.1
    q, x = _segments(rng, centres, 0.5), _points(centres)
    sizes = [_check(r, 2, q, lambda qq: slots[neighbors.points_near_segment(med, qq, np.float32(rpb) ** 2)], rpb),
             _check(r, 3, q, lambda qq: neighbors.beams_near_segment(beams, qq, np.float32(rb1) ** 2), rb1,
                    ignore=lambda qq, i: _beam_pair_ill_posed(qq, beams[i], rb1)),
             _check(r, 4, x, lambda qq: neighbors.beams_near_point(beams, qq[:3], np.float32(rb2) ** 2), rb2),
             _check(r, 1, x, lambda qq: slots[neighbors.points_in_radius(med, qq[:3], np.float32(rpp) ** 2)], rpp)]
    assert [bool(s.sum()) for s in sizes[:3]] == [leaves[1] > 0, leaves[0] > 0, leaves[0] > 0]
    r.close()


def test_short_hit_list(scene_dir):
    """A list that holds a few queries' pairs: rounds, repeated rounds, empty
    slots between the hits of a round."""
    os.environ["UPBP_MAX_HITS"] = "3000"
    try:
        r = _renderer(scene_dir, "box_medium", True, ["-a", ALL6, "-l", "8", "-r", "24x24", "-pcpi", "4000",
                                                      "-r_initial", "-0.02"])
    finally:
        os.environ.pop("UPBP_MAX_HITS", None)
    rb1 = r.stats()["radius"][0]
    beams = r.photons(2)
    rng = np.random.default_rng(41)
    pick = beams[rng.integers(0, len(beams), 1200)]
    q = _segments(rng, pick[:, :3] + pick[:, 4:7] * (0.5 * pick[:, 3])[:, None], 0.3)
    got = _check(r, 3, q, lambda qq: neighbors.beams_near_segment(beams, qq, np.float32(rb1) ** 2, _path_limit(r)), rb1,
                 ignore=lambda qq, i: _beam_pair_ill_posed(qq, beams[i], rb1))
    assert got.sum() > 5 * 3000 and got.max() < 3000
    r.close()


@pytest.mark.parametrize("radius", [-0.002, -0.05, -0.2])
def test_merges_equal_brute_force(scene_dir, radius):
    """SURF and PP3D at radii that give a query no photon, exactly the eight
    it keeps waiting, and many times that; in an order that puts them with other
    queries in a warp, and in numbers that leave a warp part empty."""
    r = _renderer(scene_dir, "fog_box", True, ["-a", "upbp_bpt+surf+pp3d", "-l", "8", "-r", "41x37", "-r_initial", str(radius)])
    rad = r.stats()["radius"]
    rng = np.random.default_rng(43)
    sizes = []
    for kind, rr in ((0, rad[4]), (1, rad[3])):
        pts = r.photons(kind)
        slots = pts[:, 3].view(np.uint32)
        x = pts[rng.integers(0, len(pts), 500), :3] + rng.normal(size=(500, 3)) * rng.choice([0.2, 1.0, 20.0], 500)[:, None] * rr
        q = _points(x.astype(np.float32))
        for order in (np.arange(500), rng.permutation(500), np.arange(33), np.arange(1)):
            sizes.append(_check(r, kind, q[order], lambda qq: slots[neighbors.points_in_radius(pts, qq[:3], np.float32(rr) ** 2)],
                                rr, splits=[(0, 0, 0)]))
    sizes = np.concatenate(sizes)
    assert (sizes == 0).any() and (sizes > 0).any()
    if radius == -0.2:
        assert (sizes > 64).sum() > 100
    if radius == -0.05:
        assert (sizes == 8).any() and (sizes == 9).any() and ((sizes > 0) & (sizes < 8)).any()
    r.close()


def test_what_the_search_refuses(scene_dir):
    from gpuupbp_b200 import upbp
    r = _renderer(scene_dir, "box_medium", True, ["-a", ALL6, "-l", "6", "-r", "16x16", "-r_initial", "-0.02"])
    before = r.stats()["work"]
    q = np.zeros((3, 8), np.float32)
    q[:, 3] = 1.0
    q[:, 7] = 1.0
    r.search(3, q)
    assert r.stats()["work"] == before  # an iteration's counters are its own
    for bad in (dict(unit_max=3), dict(unit_max=64)):
        with pytest.raises(upbp.UpbpError):
            r.search(3, q, **bad)
    q[1, 3] = 0.5
    with pytest.raises(upbp.UpbpError):
        r.search(2, q)
    r.close()
