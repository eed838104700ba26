"""SURF and PP3D keep the photons a query finds, up to eight, until the warp
merges them together.  Radii that give queries hardly a photon, a few, and many
times eight, with partial warps: the grid limit changes which queries share a
warp, and neither the numbers of merged photons nor the image may depend on it
(1e-4: sums in another order, as in tests/test_range_search_gpu.py; against
the reference's images the parity cases compare both estimators)."""
import numpy as np
import pytest

from gpuupbp_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,res,most", [(-0.0005, "9x5", 8), (-0.01, "33x31", 64), (-0.2, "41x37", 10 ** 6)])
def test_merges_do_not_depend_on_the_warp(scene_dir, radius, res, most):
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
    assert a[2] <= most * a[4]
    if most > 64:
        # many queries merge more than twice eight photons: their number grows
        # with the radius squared, 8.3 a query at 0.08 of the scene, so about 50 here
        assert a[2] > 16 * a[4]
    assert np.allclose(a[1], b[1], rtol=1e-4, atol=1e-7)
    r.close()
