"""GPU test of the trilinear density splat of compact clouds around the size that makes a dense unit, in full builds
and in builds under a plan (which know whether there are dense leaves)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1400, 1500, 1501, 1502, 4000, 20_000])
@pytest.mark.parametrize("spread", [0.0, 6.0, 60.0])
def test_compact_clouds(gvx_mod, orc, n, spread):
    rng = np.random.default_rng(n)
    pos = (96.0 + rng.random((n, 3)) * (6.0 + spread)).astype(np.float32)
    pos[0], pos[1] = 60.0, 180.0  # (points of one brick make no tree)
    w = rng.uniform(0.5, 1.5, n).astype(np.float32)
    logdim = (3, 3, 3, 3, 5)
    o = orc.Oracle(logdim)
    o.add_channel(0, orc.T_FLOAT)
    o.rebuild_topology(pos, 1.0)
    o.update_atlas()
    o.splat(orc.SPLAT_TRILINEAR, pos, 1.0, weight=w)
    g = gvx_mod.Grid(0)
    g.configure(logdim)
    g.add_channel(0, gvx_mod.T_FLOAT, 1)
    # one rounding a term (they are positive), six of a weight; the terms are the points of eight cells
    _, c = np.unique(pos.astype(np.int64) @ [1 << 20, 1 << 10, 1], return_counts=True)
    tol = (8 * int(c.max()) + 6) * 2.0 ** -24
    first = None
    for k in range(3):
        g.commit_points_host(pos, weight=w)
        g.rebuild_topology(n, 1.0, mode=gvx_mod.TOPO_FULL)
        assert g.info()["planned_builds"] == k
        g.update_atlas()
        used = g.info()["used_leaves"]
        g.splat(gvx_mod.SPLAT_TRILINEAR, n, 1.0)
        got, ref = g.read_channel(0)[:used], o.read_channel(0)[:used]
        assert np.all(np.abs(got - ref) <= tol * np.abs(ref) + 2.0 ** -60)
        first = got.tobytes() if first is None else first
        assert got.tobytes() == first
    g.close()
