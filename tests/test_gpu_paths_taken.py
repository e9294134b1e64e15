"""GPU test that the calls of the tests beside it run where those tests say they do: subcell lists that are not
written out (by the launches of the insert) and builds under the plan of the first."""
import numpy as np
import pytest

from test_gpu_build_ranks import LOGDIM, _points

pytestmark = pytest.mark.gpu


def _insert_launches(gvx, pos, radius, topo, fp16, colours=False, trans=None, move=None):
    import torch

    g = gvx.Grid(0)
    g.configure((3, 3, 3, 3, 5))
    g.add_channel(0, gvx.T_FLOAT, 1)
    n = len(pos)
    p = torch.from_numpy(pos).cuda()
    g.set_points(n, p, clr=torch.zeros((n, 4), dtype=torch.uint8, device="cuda") if colours else None)
    g.rebuild_topology(n, topo, mode=gvx.TOPO_FULL)
    g.update_atlas()
    g.sync()
    if move is not None:
        p.copy_(torch.from_numpy(move))
        torch.cuda.synchronize()
    before = g.kernel_launches()
    (g.insert_points_subcell_fp16 if fp16 else g.insert_points_subcell)(4, n, radius, trans)
    count = g.kernel_launches() - before
    g.close()
    return count


@pytest.mark.parametrize("n,side,radius,topo", [(50, 20, 1.0, 2.0), (3000, 60, 0.0, 0.0), (3000, 60, 2.0, 3.0),
                                                 (40_000, 50, 1.0, 2.0), (40_000, 200, 1.5, 0.0)])
@pytest.mark.parametrize("fp16", [True, False])
def test_lists_are_not_written(gvx_mod, n, side, radius, topo, fp16):
    rng = np.random.default_rng(n + side)
    pos = (rng.random((n, 3)) * side + 20.0).astype(np.float32)
    pos[3] = (-1.0, 30.0, 30.0)
    moved = (pos + rng.normal(0.0, 1.0, pos.shape)).astype(np.float32)
    args = (gvx_mod, pos, radius, topo, fp16)
    direct = _insert_launches(*args)
    assert direct == 3  # the error word, the points, the runs
    # written: the error word, count, scan, emission, histograms, passes, copy
    written = _insert_launches(*args, colours=True)
    assert written >= 7
    assert _insert_launches(*args, trans=(1.0, -2.0, 0.5)) == written
    assert _insert_launches(*args, move=moved) >= direct + written - 2  # tried, then written


@pytest.mark.parametrize("box,n", [((240, 500, 500), 3000), ((1000, 1000, 500), 3000), ((1000, 1000, 1000), 3000),
                                   ((2000, 1000, 1000), 60_000), ((4000, 4000, 2000), 3000)])
def test_builds_run_under_the_plan(gvx_mod, box, n):
    g = gvx_mod.Grid(0)
    g.configure(LOGDIM)
    g.add_channel(0, gvx_mod.T_FLOAT, 1)
    for k, seed in enumerate((1, 2, 3)):
        g.commit_points_host(_points(n, box, seed))
        g.rebuild_topology(n, 2.0, mode=gvx_mod.TOPO_FULL)
        assert g.info()["planned_builds"] == k
    g.close()
