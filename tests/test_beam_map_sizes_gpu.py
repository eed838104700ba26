"""The clustered beam map at the sizes where its kernels change shape: one
chunk (no tree), two and three, around a tile of 512 clusters, around the
1024 clusters one block finishes, several tiles.  Every size finds the pairs
of the Morton-split LBVH (UPBP_BEAM_MAP=lbvh), and renders the same image up to
the order of the float additions: 1e-4 as in tests/test_range_search_gpu.py."""
import os

import numpy as np
import pytest

from gpuupbp_b200 import scenes

pytestmark = pytest.mark.gpu


def _render(args, lbvh):
    from gpuupbp_b200 import upbp
    if lbvh:
        os.environ["UPBP_BEAM_MAP"] = "lbvh"
    try:
        r = upbp.Renderer(args)
    finally:
        os.environ.pop("UPBP_BEAM_MAP", None)
    status = r.run_iteration(1)
    st, img = r.stats(), r.iteration_image()
    r.close()
    return status, st, img


def _compare(args):
    s0, a, img0 = _render(args, False)
    s1, b, img1 = _render(args, True)
    assert s0 == s1 and a["beam_chunks"] == b["beam_chunks"] and b["beam_map_passes"] == 0
    assert (a["beam_map_passes"] > 0) == (a["beam_chunks"] > 1)
    for k in ("bb1d_query", "bp2d_query"):
        assert a["work"][k]["beam_hit"] == b["work"][k]["beam_hit"] > 0, k
    assert np.allclose(img0, img1, rtol=1e-4, atol=1e-7)
    return a["beam_chunks"]


# light paths and radii
@pytest.mark.parametrize("paths,radius", [(5, -0.02), (60, -0.05), (420, -0.02), (900, -0.02), (4000, -0.02)])
def test_clustered_map_equals_lbvh(scene_dir, paths, radius):
    path = scenes.write_workload("box_medium", scene_dir, tiny=True)
    chunks = _compare(["-s", "-1", path, "-a", "upbp_bb1d+bp2d", "-l", "8", "-r", "33x29", "-pcpi", str(paths),
                       "-r_initial", str(radius)])
    assert chunks > 4096 or paths < 4000


def _chunks(lengths, radius):
    """Chunks of beams of these lengths: one for every six radii, at most 64."""
    step = np.float32(6.0) * np.float32(radius)
    return int(np.maximum(1, np.minimum(np.ceil(lengths / step), 64)).sum())


@pytest.mark.parametrize("paths,chunks", [(1, 2), (1, 3), (200, 511), (200, 512), (200, 513), (300, 1023), (300, 1024),
                                          (300, 1025)])
def test_exact_sizes(scene_dir, paths, chunks):
    """The radius that gives exactly this many chunks: their number falls with
    the radius, a beam at a time."""
    from gpuupbp_b200 import upbp
    path = scenes.write_workload("box_medium", scene_dir, tiny=True)
    args = ["-s", "-1", path, "-a", "upbp_bb1d+bp2d", "-l", "8", "-r", "33x29", "-pcpi", str(paths), "-r_initial"]
    r = upbp.Renderer(args + ["-0.02"])
    r.run_iteration(1)  # the light paths depend on the iteration alone, not on the radius
    lengths = r.photons(2)[:, 3].copy()
    r.close()
    assert 0 < len(lengths) <= chunks
    lo, hi = np.float32(1e-6).view(np.int32), np.float32(10.0).view(np.int32)  # the order of floats is that of their bits
    while hi - lo > 1:
        mid = (int(lo) + int(hi)) // 2
        lo, hi = (mid, hi) if _chunks(lengths, np.int32(mid).view(np.float32)) >= chunks else (lo, mid)
    radius = np.int32(lo).view(np.float32)
    assert _chunks(lengths, radius) == chunks
    assert _compare(args + ["%.9g" % radius]) == chunks
    r = upbp.Renderer(args + ["%.9g" % radius])
    r.run_iteration(1)
    info = r.beam_map()
    r.close()
    # many-cluster passes from 1025 clusters on, one block of 512 clusters a tile
    assert info["chunks"] == chunks and (info["passes"] > 0) == (chunks > 1024)
    assert info["blocks"] == -(-chunks // 512) and info["tail_iterations"] > 0


def _blocks(scene_dir, env, limit):
    from gpuupbp_b200 import upbp
    path = scenes.write_workload("box_medium", scene_dir, tiny=True)
    os.environ.update(env)  # read when the renderer is created
    try:
        r = upbp.Renderer(["-s", "-1", path, "-a", "upbp_bb1d+bp2d", "-l", "8", "-r", "33x29", "-pcpi", "4000",
                           "-r_initial", "-0.02"])
    finally:
        for k in env:
            os.environ.pop(k, None)
    assert r._L.upbp_set_grid_limit(r._ctx, limit) == 0
    status = r.run_iteration(1)
    st, img, info = r.stats(), r.iteration_image().copy(), r.beam_map()
    r.close()
    return status, {k: st["work"][k]["beam_hit"] for k in ("bb1d_query", "bp2d_query")}, img, info


@pytest.mark.parametrize("limit", [1, 3])
def test_clustering_keeps_to_the_grid_limit(scene_dir, limit):
    """The clustering's blocks, which have to be on the device all at once, are
    capped like the other launches, and the map finds the same pairs."""
    s0, hits0, img0, a = _blocks(scene_dir, {}, 0)
    s1, hits1, img1, b = _blocks(scene_dir, {}, limit)
    assert a["chunks"] == b["chunks"] > 4096 and a["blocks"] == -(-a["chunks"] // 512)  # one block a tile
    assert b["blocks"] == limit and b["passes"] == a["passes"] > 0
    assert s0 == s1 and hits0 == hits1 and np.allclose(img0, img1, rtol=1e-4, atol=1e-7)


def test_refused_clustering_falls_back(scene_dir):
    """More blocks than the device holds at once: the runtime refuses the
    launch, and the iteration renders with the LBVH."""
    s0, hits0, img0, a = _blocks(scene_dir, {}, 0)
    s1, hits1, img1, b = _blocks(scene_dir, {"UPBP_PLOC_BLOCKS": "65536"}, 0)
    assert a["blocks"] > 0 and b == {"chunks": a["chunks"], "passes": 0, "tail_iterations": 0, "blocks": 0}
    assert s0 == s1 and hits0 == hits1 and np.allclose(img0, img1, rtol=1e-4, atol=1e-7)
