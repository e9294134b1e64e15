"""GPU test of the gather of written lists of 4^3 subcells: lists of none, one, 31 to 33 and many entries, other
brick sizes, accumulation, colours."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_brick,n,cluster,levelset,accum", [
    (3, 60, 1, False, False), (3, 60, 31, True, False), (3, 60, 32, False, True), (3, 60, 33, True, True),
    (2, 400, 64, False, True), (4, 400, 65, True, False), (4, 20_000, 500, False, True), (5, 3000, 5000, True, True)])
def test_lists_against_the_oracle(gvx_mod, orc, log_brick, n, cluster, levelset, accum):
    import torch

    rng = np.random.default_rng(n + cluster)
    # background points in 150^3, and the cluster in the middle of one subcell (radius 0.5 stays inside it)
    pos = np.concatenate([rng.random((n, 3)) * 150.0 + 4.0, 97.0 + rng.random((cluster, 3)) * 1.4]).astype(np.float32)
    n = len(pos)
    clr = rng.integers(0, 256, (n, 4), dtype=np.uint8)
    clr[:, 3] = rng.integers(0, 100, n)
    logdim = (log_brick, 3, 3, 3, 5)
    g, o = gvx_mod.Grid(0), orc.Oracle(logdim)
    g.configure(logdim)
    for c, t in ((0, gvx_mod.T_FLOAT), (1, gvx_mod.T_UCHAR4)):
        g.add_channel(c, t, 1)
        o.add_channel(c, t)
    pd, cd = torch.from_numpy(pos).cuda(), torch.from_numpy(clr.view(np.int32)).cuda()
    g.set_points(n, pd, clr=cd)
    g.rebuild_topology(n, 1.0, mode=gvx_mod.TOPO_FULL)
    g.update_atlas()
    o.rebuild_topology(pos, 1.0)
    o.update_atlas()
    used = o.used_leaves()
    m = g.insert_points_subcell(4, n, 0.5)
    f = g.gather_levelset if levelset else g.gather_density
    for k in range(2 if accum else 1):
        f(4, n, 1.5, m, chan=0, chan_clr=1, accum=k == 1)
        assert m == o.gather(levelset, pos, 1.5, 0.5, subcell=4, chan=0, chan_clr=1, clr=clr, accum=k == 1)
    inner = (slice(None),) + (slice(1, -1),) * 3
    got, ref = g.read_channel(0)[:used][inner].astype(np.float64), o.read_channel(0)[:used][inner]
    # distances up to 8 of coordinates up to 155 (exact differences): four roundings, and the radius taken off
    assert np.abs(got - ref).max() <= 8.0 * 8 * 2.0 ** -24
    a, b = g.read_channel(1)[:used][inner].astype(np.int64), o.read_channel(1)[:used][inner].astype(np.int64)
    assert np.abs(a - b).max() <= (2 if accum else 1)  # truncated FP32 sums against FP64, once a gather
