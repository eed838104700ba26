"""The packet range searches find the same pairs however their queries are
split over warps and groups.

A warp of the PB2D, BB1D and BP2D searches takes 1 to 32 neighbouring queries
at a time, by the queries' number and the launch's blocks, and walks the map
once per group of queries close together.  upbp_set_grid_limit changes the
split (a few queries on many warps: one query a unit and groups of one; one
block: units of the largest size), the accepted pairs depend on the exact
predicates alone: their numbers are equal, and the images equal up to the
order of the float additions.  Each estimate is summed in float32 over the
pairs of a pixel, so two orders of n additions of terms of one sign differ by
at most 2 n 2^-24 of the pixel, and typically by its square root: 1e-4 holds
for the largest n here (a few thousand pairs).
"""
import numpy as np
import pytest

from gpuupbp_b200 import scenes

pytestmark = pytest.mark.gpu

TECH = "upbp_bpt+surf+pp3d+pb2d+bb1d+bp2d"


# one query and a remainder of a unit; one warp's worth and one more; a few
# hundred queries; a beam map of one chunk, which has no inner node (ONE_LEAF)
ONE_LEAF = ["-pcpi", "1", "-r_initial", "-0.2"]


@pytest.mark.parametrize("workload,res,extra", [
    ("box_medium", "2x1", []),
    ("box_medium", "8x4", []),
    ("box_medium", "11x3", ["-pcpi", "40"]),
    ("box_medium", "61x47", []),
    ("fog_box", "37x29", ["-qbt", "S"]),
    ("dense_beams", "41x23", ["-r_initial_bb1d", "-0.004", "-r_initial_bp2d", "-0.004", "-pbc", "300"]),
    ("media_field", "53x31", ["-pbt", "S"]),
    ("box_medium", "33x31", ["-pcpi", "3"]),
    ("box_medium", "33x31", ONE_LEAF),
])
def test_pairs_do_not_depend_on_the_split(scene_dir, workload, res, extra):
    from gpuupbp_b200 import upbp
    path = scenes.write_workload(workload, scene_dir, tiny=True)
    radius = [] if workload in ("dense_beams", "media_field") or "-r_initial" in extra else ["-r_initial", "-0.02"]
    r = upbp.Renderer(["-s", "-1", path, "-a", TECH, "-l", "9", "-r", res] + radius + extra)
    got = []
    for limit in (0, 1, 3):
        assert r._L.upbp_set_grid_limit(r._ctx, limit) == 0
        status = r.run_iteration(2)
        st = r.stats()
        got.append((status, r.iteration_image(), {k: (w["beam_hit"], w["point_hit"]) for k, w in st["work"].items()},
                    st["light_beams"]))
    r.close()
    if extra == ONE_LEAF:
        assert st["beam_chunks"] == 1 and st["work"]["bb1d_query"]["beam_hit"] > 0
    for status, img, hits, beams in got[1:]:
        assert status == got[0][0] and beams == got[0][3]
        assert hits == got[0][2]
        assert np.isfinite(img).all()
        assert np.allclose(img, got[0][1], rtol=1e-4, atol=1e-7)


def test_split_case_has_pairs(scene_dir):
    """The comparison above is of searches that find something."""
    from gpuupbp_b200 import upbp
    path = scenes.write_workload("box_medium", scene_dir, tiny=True)
    r = upbp.Renderer(["-s", "-1", path, "-a", TECH, "-l", "9", "-r", "61x47", "-r_initial", "-0.02"])
    r.run_iteration(2)
    w = r.stats()["work"]
    r.close()
    assert w["bb1d_query"]["beam_hit"] > 10000 and w["pb2d_query"]["point_hit"] > 1000
    assert w["bp2d_query"]["beam_hit"] > 1000
