"""GPU test of the cubic splats over bricks that no point reaches -- a unit without candidates -- beside ones
that points do reach: the topology's dilation is wider than the splat's support."""
import numpy as np
import pytest

from parity_util import DENSITY_TOL, rel_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_brick,n,side,radius,vel,ppr,accum", [
    (3, 30, 90.0, 1.0, False, False, False), (3, 30, 90.0, 1.0, True, False, False), (3, 30, 90.0, 1.0, True, False, True),
    (3, 9000, 1.9, 1.0, True, False, False), (3, 30, 90.0, 2.5, False, True, False), (2, 30, 50.0, 0.8, False, False, False),
    (4, 30, 90.0, 1.0, True, True, False)])
@pytest.mark.parametrize("batch", [False, True])
def test_bricks_out_of_reach(gvx_mod, orc, log_brick, n, side, radius, vel, ppr, accum, batch):
    rng = np.random.default_rng(n + log_brick)
    brick = 1 << log_brick
    # (the root holds every dilated brick)
    pos = (3.25 * brick + rng.random((n, 3)) * side).astype(np.float32)
    if side < brick:
        pos[0] = 6.25 * brick  # (points of one brick make no tree)
    w = rng.uniform(0.5, 1.5, n).astype(np.float32)
    u = rng.normal(0.0, 1.0, (n, 3)).astype(np.float32) if vel else None
    r = rng.uniform(0.5 * radius, radius, n).astype(np.float32) if ppr else None
    logdim = (log_brick, 3, 3, 3, 4)
    topo = 0.5 * (brick - 1)
    g, o = gvx_mod.Grid(0), orc.Oracle(logdim)
    g.configure(logdim)
    for grid, mod in ((g, gvx_mod), (o, orc)):
        for c, t in ((0, mod.T_FLOAT),) + (((1, mod.T_FLOAT3),) if vel else ()):
            grid.add_channel(c, t)
    g.commit_points_host(pos, vel=u, weight=w, radius=r)
    g.rebuild_topology(n, topo, mode=gvx_mod.TOPO_FULL)
    g.update_atlas()
    g.insert_points(n)
    o.rebuild_topology(pos, topo)
    o.update_atlas()
    for c in (0, 1)[:1 + vel]:
        g.fill_channel(c, [0.0, 0.0, 0.0, 0.0] if accum else [9.0, 9.0, 9.0, 9.0])
    chan_vel = 1 if vel else -1
    if batch:
        b = gvx_mod.Batch(0)
        b.set_grids([g])
        b.splat(gvx_mod.SPLAT_CUBIC, radius, chan_vel=chan_vel, accum=accum)
        g.sync()
        b.close()
    else:
        g.splat(gvx_mod.SPLAT_CUBIC, n, radius, chan_vel=chan_vel, accum=accum)
    o.splat(orc.SPLAT_CUBIC, pos, radius, weight=w, radius_pp=r, vel=u, chan_vel=chan_vel)
    used = g.info()["used_leaves"]
    for c in (0, 1)[:1 + vel]:
        g.update_apron(c, 0.0)
        o.update_apron(c)
    ref = o.read_channel(0)[:used]
    empty = ~ref.reshape(used, -1).any(axis=1)
    assert empty.sum() > 4  # (the case is what it says)
    got = g.read_channel(0)[:used]
    assert rel_error(got, ref) <= DENSITY_TOL and not got[empty].any()
    if vel:
        got, ref = g.read_channel(1)[:used, ..., :3], o.read_channel(1)[:used, ..., :3]
        assert np.abs(got - ref).max() <= DENSITY_TOL * np.abs(ref).max() and not got[empty].any()
    g.close()
