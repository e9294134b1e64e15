"""GPU test of ScatterDensity where its two kernels meet: bricks of a few points (a warp each) and bricks
from 256 points (a block each), other brick sizes, with and without apron, expansion and colours; and of
channel smoothing over few and many bricks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(background, cluster, seed):
    rng = np.random.default_rng(seed)
    p = rng.random((background, 3)) * 160.0
    c = 96.0 + rng.random((cluster, 3)) * 7.99  # one brick of 8
    p = np.concatenate([p, c]).astype(np.float32)
    return p[rng.permutation(len(p))], rng.integers(0, 256, (len(p), 4)).astype(np.uint8)


def _most(pos):
    """the most points that seven neighbouring cells hold, at most"""
    c = pos.astype(np.int64)
    _, n = np.unique((c[:, 0] * 1024 + c[:, 1]) * 1024 + c[:, 2], return_counts=True)
    return 7 * int(n.max())


@pytest.mark.parametrize("log_brick,background,cluster,apron,expand,colours", [
    (3, 60, 1, 1, True, "avg"), (3, 60, 255, 1, True, "avg"), (3, 60, 256, 1, True, "avg"), (3, 60, 257, 1, True, "one"),
    (3, 3000, 255, 0, True, "one"), (3, 3000, 5000, 0, True, "avg"), (3, 3000, 70_000, 1, False, "avg"),
    (3, 90_000, 5000, 1, True, None), (2, 3000, 4000, 1, True, "avg"), (4, 3000, 4000, 1, True, "one")])
def test_scatter_against_the_oracle(gvx_mod, orc, log_brick, background, cluster, apron, expand, colours):
    import torch

    pos, clr = _points(background, cluster, background + cluster)
    logdim = (log_brick, 3, 3, 3, 5)
    g = gvx_mod.Grid(0)
    g.configure(logdim)
    o = orc.Oracle(logdim, apron=apron)
    for c, t in ((0, gvx_mod.T_FLOAT), (1, gvx_mod.T_UCHAR4), (2, gvx_mod.T_FLOAT), (3, gvx_mod.T_UCHAR4)):
        g.add_channel(c, t, apron)
        o.add_channel(c, t)
    pd, cd = torch.from_numpy(pos).cuda(), torch.from_numpy(clr.view(np.int32)).cuda()
    g.set_points(len(pos), pd, clr=cd if colours else None)
    g.rebuild_topology(len(pos), 0.0, mode=gvx_mod.TOPO_FULL)
    g.update_atlas()
    o.rebuild_topology(pos, 0.0)
    o.update_atlas()
    used = o.used_leaves()
    for _ in range(2):  # onto a cleared channel, then onto what is there
        g.scatter_density(len(pos), 2.5, expand=expand, avg_color=colours == "avg")
        o.scatter_density(pos, 2.5, clr=clr if colours else None, expand=expand, avg_color=colours == "avg")
    got, ref = g.read_channel(0)[:used].astype(np.float64), o.read_channel(0)[:used]
    # a term 1 + c (-3 + c (3 - c)), 0 <= c <= 1: its rounding, and c's, within 24 units; one more a sum
    n = 2 * _most(pos)
    assert np.abs(got - ref).max() <= n * 2.0 ** -24 * (24 + np.abs(ref).max())
    if colours:
        chan = 1 if colours == "avg" else 3
        assert np.array_equal(g.read_channel(chan)[:used], o.read_channel(chan)[:used].astype(np.uint8))


@pytest.mark.parametrize("n", [1, 5, 700, 30_000, 400_000])
def test_smooth_few_and_many_bricks(gvx_mod, n):
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 3)) * 260.0).astype(np.float32)
    g = gvx_mod.Grid(0)
    g.configure((3, 3, 3, 3, 5))
    g.add_channel(0, gvx_mod.T_FLOAT, 1)
    g.commit_points_host(pos)
    g.rebuild_topology(n, 0.0, mode=gvx_mod.TOPO_FULL)
    g.update_atlas()
    data = (rng.integers(-64, 64, g.read_channel(0).shape) / 8.0).astype(np.float32)
    g.write_channel(0, data)
    p1 = 2.0
    g.compute(gvx_mod.FUNC_SMOOTH, 0, 1, (p1, 0.25, 0.0), update_apron=False, skip_over_aprons=True)
    d = data.astype(np.float64).reshape(-1, 10, 10, 10)
    ref = d.copy()
    c = slice(1, 9)
    s = p1 * d[:, c, c, c]
    for axis in (1, 2, 3):
        for sh in (slice(0, 8), slice(2, 10)):
            ix = [slice(None), c, c, c]
            ix[axis] = sh
            s = s + d[tuple(ix)]
    ref[:, c, c, c] = s / (p1 + 6.0) + 0.25
    got = g.read_channel(0).reshape(ref.shape)
    # eight roundings of values up to 64 in the sum, an eighth of it, and two more
    assert np.abs(got - ref).max() <= (8 * 64 / 8.0 + 2 * 9) * 2.0 ** -24
    edge = np.ones((10, 10, 10), bool)
    edge[c, c, c] = False
    assert np.array_equal(got[:, edge], data.reshape(ref.shape)[:, edge])
