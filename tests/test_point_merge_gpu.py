"""SURF and PP3D keep the photons a query finds, up to eight, until the warp
merges them together.  Radii that give queries hardly a photon, a few, and many
times eight, with partial warps: rendered by all blocks and by one (each warp
then merges for many warps' worth of queries in turn), the numbers of photons
merged -- counted where they are merged -- and the image are the same (1e-4: sums
in another order, as in tests/test_range_search_gpu.py).  Which photons are
merged is compared with brute force in tests/test_neighbor_search_gpu.py, both
estimators' images with the reference's in the parity cases."""
import numpy as np
import pytest

from gpuupbp_b200 import scenes

pytestmark = pytest.mark.gpu


# photons merged by a point query, on average: bounds of SURF's and PP3D's
# (278107 and 33682 for 5141 queries at the largest radius)
@pytest.mark.parametrize("radius,res,surf,pp3d", [(-0.0005, "9x5", (0.0, 0.1), (0.0, 0.1)),
                                                  (-0.01, "33x31", (0.05, 1.0), (0.0, 0.1)),
                                                  (-0.2, "41x37", (16.0, 128.0), (4.0, 64.0))])
def test_merges_do_not_depend_on_the_blocks(scene_dir, radius, res, surf, pp3d):
    from gpuupbp_b200 import upbp
    path = scenes.write_workload("fog_box", scene_dir, tiny=True)
    r = upbp.Renderer(["-s", "-1", path, "-a", "upbp_bpt+surf+pp3d", "-l", "8", "-r", res, "-r_initial", str(radius)])
    got = []
    for limit in (0, 1):
        assert r._L.upbp_set_grid_limit(r._ctx, limit) == 0
        status = r.run_iteration(0)
        st = r.stats()
        got.append((status, r.iteration_image(), st["work"]["surf_query"]["point_hit"],
                    st["work"]["pp3d_query"]["point_hit"], st["point_queries"]))
    a, b = got
    assert a[0] == b[0] and a[2:] == b[2:]
    assert surf[0] * a[4] <= a[2] <= surf[1] * a[4]
    assert pp3d[0] * a[4] <= a[3] <= pp3d[1] * a[4]
    assert np.allclose(a[1], b[1], rtol=1e-4, atol=1e-7)
    r.close()
