"""The clustered beam map at the sizes where its kernels change shape: two
chunks, less and more than a tile of 512 clusters, around the 1024 clusters
one block finishes, several tiles.  Every size finds the pairs of the
Morton-split LBVH (UPBP_BEAM_MAP=lbvh), and renders the same image up to the
order of the float additions: 1e-4 as in tests/test_range_search_gpu.py."""
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


# light paths; the chunks they give are asserted below to span the sizes
@pytest.mark.parametrize("paths,radius", [(3, -0.2), (5, -0.02), (60, -0.05), (120, -0.02), (330, -0.02), (420, -0.02),
                                          (900, -0.02), (4000, -0.02)])
def test_clustered_map_equals_lbvh(scene_dir, paths, radius):
    path = scenes.write_workload("box_medium", scene_dir, tiny=True)
    args = ["-s", "-1", path, "-a", "upbp_bb1d+bp2d", "-l", "8", "-r", "33x29", "-pcpi", str(paths),
            "-r_initial", str(radius)]
    s0, a, img0 = _render(args, False)
    s1, b, img1 = _render(args, True)
    assert s0 == s1 and a["beam_chunks"] == b["beam_chunks"] and b["beam_map_passes"] == 0
    assert (a["beam_map_passes"] > 0) == (a["beam_chunks"] > 1)
    for k in ("bb1d_query", "bp2d_query"):
        assert a["work"][k]["beam_hit"] == b["work"][k]["beam_hit"], k
    assert np.allclose(img0, img1, rtol=1e-4, atol=1e-7)


def test_sizes_span_the_tiles(scene_dir):
    """The light paths above give fewer than 512, about 1024 and several
    thousand chunks."""
    path = scenes.write_workload("box_medium", scene_dir, tiny=True)
    got = []
    for paths in (60, 330, 4000):
        _, st, _ = _render(["-s", "-1", path, "-a", "upbp_bb1d+bp2d", "-l", "8", "-r", "33x29", "-pcpi", str(paths),
                            "-r_initial", "-0.02"], False)
        got.append(st["beam_chunks"])
    assert 0 < got[0] < 512 and 512 < got[1] < 2048 and got[2] > 4096


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
