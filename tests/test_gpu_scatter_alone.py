"""GPU test of ScatterDensity where it is one launch or two: bricks of which there is a block each, or of many points
in few turns, or points for a few turns of the warps; against the oracle."""
import numpy as np
import pytest

from test_gpu_scatter_split import _most

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_brick,n,side,cluster", [(3, 300, 60, 0), (3, 1000, 300, 0), (3, 1023, 300, 0), (3, 1024, 300, 0),
                                                      (3, 1024, 300, 700), (3, 3000, 300, 700), (3, 40_000, 100, 0),
                                                      (3, 80_000, 100, 0), (2, 80_000, 60, 0), (3, 200_000, 180, 0),
                                                      (4, 3000, 300, 700)])
@pytest.mark.parametrize("colours", [None, "avg", "one"])
def test_scatter(gvx_mod, orc, log_brick, n, side, cluster, colours):
    import torch

    rng = np.random.default_rng(n + cluster)
    pos = (rng.random((n, 3)) * side).astype(np.float32)
    pos[:cluster] = 40.0 + rng.random((cluster, 3)) * 3.9
    pos = pos[rng.permutation(n)]
    clr = rng.integers(0, 256, (n, 4)).astype(np.uint8)
    logdim = (log_brick, 3, 3, 3, 5)
    g, o = gvx_mod.Grid(0), orc.Oracle(logdim)
    g.configure(logdim)
    for c, t in ((0, gvx_mod.T_FLOAT), (1, gvx_mod.T_UCHAR4), (2, gvx_mod.T_FLOAT), (3, gvx_mod.T_UCHAR4)):
        g.add_channel(c, t)
        o.add_channel(c, t)
    pd, cd = torch.from_numpy(pos).cuda(), torch.from_numpy(clr.view(np.int32)).cuda()
    g.set_points(n, pd, clr=cd if colours else None)
    g.rebuild_topology(n, 0.0, mode=gvx_mod.TOPO_FULL)
    g.update_atlas()
    o.rebuild_topology(pos, 0.0)
    o.update_atlas()
    g.scatter_density(n, 2.5, avg_color=colours == "avg")
    o.scatter_density(pos, 2.5, clr=clr if colours else None, avg_color=colours == "avg")
    used = o.used_leaves()
    got, ref = g.read_channel(0)[:used].astype(np.float64), o.read_channel(0)[:used]
    # a term 1 + c (-3 + c (3 - c)), 0 <= c <= 1: its rounding, and c's, within 24 units; one more a sum
    assert np.abs(got - ref).max() <= _most(pos) * 2.0 ** -24 * (24 + np.abs(ref).max())
    if colours:
        chan = 1 if colours == "avg" else 3
        assert np.array_equal(g.read_channel(chan)[:used], o.read_channel(chan)[:used].astype(np.uint8))
    g.close()
