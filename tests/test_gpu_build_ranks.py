"""GPU test of the ranks and key lists of a build on both sides of the sizes (2^20, 2^25 leaf cells) from which their
sums take a launch of their own, and larger blocks: a first build, a planned one, and appended frames, against the oracle."""
import numpy as np
import pytest

from parity_util import compare_topology

pytestmark = pytest.mark.gpu

LOGDIM = (3, 3, 3, 3, 5)


def _points(n, box, seed):
    rng = np.random.default_rng(seed)
    p = (rng.random((n, 3)) * (np.array(box) - 40.0) + 20.0).astype(np.float32)
    p[0], p[1] = 20.0, np.array(box) - 20.0  # the corners: the key space spans the box
    return p


@pytest.mark.parametrize("radius", [0.0, 2.0])
@pytest.mark.parametrize("box,n", [((100, 100, 100), 40), ((240, 500, 500), 3000), ((1000, 1000, 500), 3000),
                                   ((1000, 1000, 1000), 3000), ((2000, 1000, 1000), 60_000),
                                   ((4000, 4000, 2000), 3000)])
def test_builds_against_the_oracle(gvx_mod, orc, box, n, radius):
    g = gvx_mod.Grid(0)
    g.configure(LOGDIM)
    g.add_channel(0, gvx_mod.T_FLOAT, 1)
    for seed in (1, 2, 3):  # the second and third under the first one's plan
        pos = _points(n, box, seed)
        g.commit_points_host(pos)
        g.rebuild_topology(n, radius, mode=gvx_mod.TOPO_FULL)
        g.update_atlas()
        o = orc.Oracle(LOGDIM, apron=1)
        o.add_channel(0, orc.T_FLOAT)
        o.rebuild_topology(pos, radius)
        o.update_atlas()
        compare_topology(g, o, check_childlists=True)
    for seed in (4, 5):
        pos = _points(n, [b - 100 for b in box], seed) if box[0] > 200 else _points(n, box, seed)
        g.commit_points_host(pos)
        g.rebuild_topology(n, radius, mode=gvx_mod.TOPO_ACCUMULATE)
        g.update_atlas()
        o.rebuild_topology(pos, radius, mode=orc.TOPO_ACCUMULATE)
        o.update_atlas()
        compare_topology(g, o, check_childlists=True)
