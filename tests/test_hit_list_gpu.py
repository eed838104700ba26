"""Range searches whose hit list is held down (UPBP_MAX_HITS, or a device
short of memory): the rounds they take, and the pairs they find.

A warp reserves slots of the list ahead of the pairs it finds.  What the
warps hold in reserve has to fit the quarter of the list that a round keeps
free, or rounds overflow on empty slots alone and are thrown away.
"""
import math
import os

import numpy as np
import pytest

from gpuupbp_b200 import scenes

pytestmark = pytest.mark.gpu


def _render(args, max_hits=None, iteration=0):
    from gpuupbp_b200 import upbp
    if max_hits is not None:
        os.environ["UPBP_MAX_HITS"] = str(max_hits)  # read when the renderer is created
    try:
        r = upbp.Renderer(args)
    finally:
        os.environ.pop("UPBP_MAX_HITS", None)
    for _ in range(2):  # the first iteration sizes the lists
        status = r.run_iteration(iteration)
    st, img = r.stats(), r.iteration_image().copy()
    r.close()
    return status, st, img


@pytest.mark.parametrize("max_hits", [1 << 21, 1 << 22])
def test_rounds_of_a_limited_list(scene_dir, max_hits):
    """Queries of a few pairs each and a list several times too short: a round
    fills at least 5/8 of the list (it ends at 3/4, of which an eighth may be
    slots not used), and no search is repeated."""
    path = scenes.write_workload("box_medium", scene_dir)
    args = ["-s", "-1", path, "-a", "upbp_bb1d", "-l", "6", "-r", "1024x1024", "-pcpi", "16384", "-r_initial", "-0.0004"]
    s0, a, img0 = _render(args)
    s1, b, img1 = _render(args, max_hits)
    pairs = a["work"]["bb1d_query"]["beam_hit"]
    assert 2 * max_hits < pairs < 16 * max_hits, pairs
    # the queries in flight (8 in each of 4 warps of 7 blocks on 148 SMs) fit the
    # quarter of the list a round keeps free, also where pairs are twice as dense
    assert 148 * 7 * 4 * 8 * 2 * pairs / a["segment_queries"] < max_hits / 4
    assert s0 == s1 and b["work"]["bb1d_query"]["beam_hit"] == pairs
    rounds = math.ceil(pairs / (0.625 * max_hits))
    # a round: one search and one evaluation
    assert b["kernel_launches"] - a["kernel_launches"] <= 2 * (rounds - 1), (pairs, a["kernel_launches"], b["kernel_launches"])
    # sums in another order, as in tests/test_range_search_gpu.py
    assert np.allclose(img0, img1, rtol=1e-4, atol=1e-7)


def test_list_that_the_pairs_just_fit(scene_dir):
    """A round of one query reserves exactly what it finds: a list of that
    size is enough."""
    from gpuupbp_b200 import upbp
    path = scenes.write_workload("box_medium", scene_dir, tiny=True)
    args = ["-s", "-1", path, "-a", "upbp_bb1d", "-l", "6", "-r", "1x1", "-pcpi", "4000", "-r_initial", "-0.02"]
    r = upbp.Renderer(args)
    it = 0
    for it in range(200):
        r.run_iteration(it)
        st = r.stats()
        if st["segment_queries"] == 1 and st["work"]["bb1d_query"]["beam_hit"] > 64:
            break
    r.close()
    pairs = st["work"]["bb1d_query"]["beam_hit"]
    assert st["segment_queries"] == 1 and pairs > 64 and pairs % 32
    status, b, _ = _render(args, pairs, it)
    assert b["work"]["bb1d_query"]["beam_hit"] == pairs and status == 0
    assert b["kernel_launches"] == st["kernel_launches"]
