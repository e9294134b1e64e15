"""GPU test of the cubic splats' work units against the oracle: brick sizes and slab heights, hits that
fill the batches dealt at once, whole bricks pushed by table and bricks with missing neighbours."""
import numpy as np
import pytest

from parity_util import DENSITY_TOL, rel_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_brick,n,side,radius,vel,ppr,accum", [
    (1, 400, 40, 0.9, False, False, False), (2, 3000, 60, 1.5, True, False, False), (2, 3000, 60, 1.0, False, True, False),
    (3, 40, 30, 2.0, True, False, False), (3, 60_000, 100, 2.0, True, False, False), (3, 60_000, 100, 2.0, True, False, True),
    (3, 60_000, 100, 3.4, True, False, False), (3, 60_000, 100, 2.0, False, True, False), (3, 2000, 16, 2.0, True, False, False),
    (3, 20_000, 90, 3.0, True, True, False), (3, 3000, 200, 2.0, False, False, True), (4, 20_000, 90, 3.5, False, False, False),
    (4, 40_000, 60, 2.0, True, False, False), (5, 20_000, 90, 2.0, True, False, False), (5, 20_000, 90, 6.0, False, True, False)])
def test_cubic_units(gvx_mod, orc, log_brick, n, side, radius, vel, ppr, accum):
    rng = np.random.default_rng(n + side)
    brick = 1 << log_brick
    # across a corner of the level-1 nodes: the root is a higher one, and holds every dilated brick
    pos = (max(2.0 * brick, 8.0 * brick - 0.5 * side) + rng.random((n, 3)) * side).astype(np.float32)
    w = rng.uniform(0.5, 1.5, n).astype(np.float32)
    u = rng.normal(0.0, 1.0, (n, 3)).astype(np.float32) if vel else None
    r = rng.uniform(0.5 * radius, radius, n).astype(np.float32) if ppr else None
    logdim = (log_brick, 3, 3, 3, 4)
    topo = min(float(np.ceil(radius)), 0.5 * (brick - 1))
    topo = topo if topo >= 1.0 else 0.0
    g, o = gvx_mod.Grid(0), orc.Oracle(logdim)
    g.configure(logdim)
    for grid, mod in ((g, gvx_mod), (o, orc)):
        args = ((0, mod.T_FLOAT),) + (((1, mod.T_FLOAT3),) if vel else ())
        for c, t in args:
            grid.add_channel(c, t)
    g.commit_points_host(pos, vel=u, weight=w, radius=r)
    g.rebuild_topology(n, topo, mode=gvx_mod.TOPO_FULL)
    g.update_atlas()
    o.rebuild_topology(pos, topo)
    o.update_atlas()
    kw = dict(weight=w, radius_pp=r, vel=u, chan_vel=1 if vel else -1)
    for k in range(2 if accum else 1):
        g.splat(gvx_mod.SPLAT_CUBIC, n, radius, chan_density=0, chan_vel=1 if vel else -1, accum=k > 0)
        o.splat(orc.SPLAT_CUBIC, pos, radius, accum=k > 0, **kw)
    used = g.info()["used_leaves"]
    if accum:  # an accumulating splat leaves apron voxels of missing neighbours to UpdateApron
        for c in (0, 1)[:1 + vel]:
            g.update_apron(c, 0.0)
            o.update_apron(c)
    assert rel_error(g.read_channel(0)[:used], o.read_channel(0)[:used]) <= DENSITY_TOL
    if vel:
        got, ref = g.read_channel(1)[:used, ..., :3], o.read_channel(1)[:used, ..., :3]
        assert np.abs(got - ref).max() <= DENSITY_TOL * np.abs(ref).max()
    g.close()
