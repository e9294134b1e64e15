"""GPU test of the trilinear density splat where its paths meet: leaves at the size from which their
points are put in cell order, bricks dense enough to be summed voxel by voxel (where they are met, or
listed for a launch of their own), other brick sizes, aprons at missing neighbours, accumulation."""
import numpy as np
import pytest

from parity_util import compare_topology

pytestmark = pytest.mark.gpu


def _cloud(n, cluster, sigma, seed):
    """n background points in 200^3 and a cluster around a brick's corner"""
    rng = np.random.default_rng(seed)
    p = rng.random((n, 3)) * 200.0
    if sigma == 0:  # all in one brick: its leaf holds exactly the cluster
        c = 96.0 + rng.random((cluster, 3)) * 7.99
    else:
        c = 96.0 + rng.normal(0.0, sigma, (cluster, 3))
    p = np.concatenate([p, c]).astype(np.float32)
    return p[rng.permutation(len(p))], rng.uniform(0.5, 1.5, len(p)).astype(np.float32)


def _bound(pos):
    """relative rounding bound of a voxel's sum: one rounding a term (the terms are positive), and six of
    a weight; the terms are the points of the eight cells around the voxel"""
    c = pos.astype(np.int64)
    key = (c[:, 0] * 1024 + c[:, 1]) * 1024 + c[:, 2]
    _, n = np.unique(key, return_counts=True)
    return (8 * int(n.max()) + 6) * 2.0 ** -24


@pytest.mark.parametrize("log_brick,n,cluster,sigma,apron", [
    (3, 40, 127, 0, 1), (3, 60, 128, 0, 1), (3, 50, 129, 0, 1), (3, 3000, 12_000, 3.0, 1), (3, 3000, 12_000, 3.0, 0),
    (3, 2000, 30_760, 5.0, 1), (3, 30_000, 20_000, 2.0, 1), (3, 200_000, 3000, 1.0, 1), (2, 2000, 9000, 3.0, 1),
    (1, 500, 1000, 2.0, 1), (4, 2000, 9000, 3.0, 1), (5, 2000, 9000, 3.0, 1)])
def test_dense_clouds_against_the_oracle(gvx_mod, orc, log_brick, n, cluster, sigma, apron):
    pos, w = _cloud(n, cluster, sigma, n + cluster)
    logdim = (log_brick, 3, 3, 3, 5)
    g = gvx_mod.Grid(0)
    g.configure(logdim)
    g.add_channel(0, gvx_mod.T_FLOAT, apron)
    g.commit_points_host(pos, weight=w)
    topo = 1.0 if log_brick > 1 else 0.0
    g.rebuild_topology(len(pos), topo, mode=gvx_mod.TOPO_FULL)
    g.update_atlas()
    g.splat(gvx_mod.SPLAT_TRILINEAR, len(pos), 1.0)
    o = orc.Oracle(logdim, apron=apron)
    o.add_channel(0, orc.T_FLOAT)
    o.rebuild_topology(pos, topo)
    o.update_atlas()
    compare_topology(g, o, check_childlists=False)
    o.splat(orc.SPLAT_TRILINEAR, pos, 1.0, weight=w)
    used = g.info()["used_leaves"]
    once = g.read_channel(0)[:used]
    ref = o.read_channel(0)[:used]
    tol = _bound(pos)
    assert np.all(np.abs(once - ref) <= tol * np.abs(ref) + 2.0 ** -60)
    # the same again gives the same bytes, and the aprons are the neighbours' values
    g.splat(gvx_mod.SPLAT_TRILINEAR, len(pos), 1.0)
    assert g.read_channel(0)[:used].tobytes() == once.tobytes()
    g.channel_device_ptr(0)
    g.update_apron(0, 0.0)
    assert g.read_channel(0)[:used].tobytes() == once.tobytes()
    # accumulation: the interiors twice the sum, one rounding a term again
    g.splat(gvx_mod.SPLAT_TRILINEAR, len(pos), 1.0, accum=True)
    i = slice(apron, apron + (1 << log_brick))
    twice = g.read_channel(0)[:used][:, i, i, i]
    assert np.all(np.abs(twice - 2.0 * ref[:, i, i, i]) <= 2.0 * tol * 2.0 * ref[:, i, i, i] + 2.0 ** -60)
    g.close()


def test_listed_and_met_units_give_the_same_bits(gvx_mod):
    """a batch lists its dense units whatever the point count, a single splat of few points does not"""
    pos, w = _cloud(3000, 12_000, 3.0, 1)
    g = gvx_mod.Grid(0)
    g.configure((3, 3, 3, 3, 5))
    g.add_channel(0, gvx_mod.T_FLOAT, 1)
    g.commit_points_host(pos, weight=w)
    g.rebuild_topology(len(pos), 1.0, mode=gvx_mod.TOPO_FULL)
    g.update_atlas()
    g.splat(gvx_mod.SPLAT_TRILINEAR, len(pos), 1.0)
    used = g.info()["used_leaves"]
    ref = g.read_channel(0)[:used].tobytes()
    b = gvx_mod.Batch(0)
    b.set_grids([g])
    for graph in (False, True, True):
        g.fill_channel(0, [9.0])
        b.splat(gvx_mod.SPLAT_TRILINEAR, 1.0, graph=graph)
        g.sync()
        assert g.read_channel(0)[:used].tobytes() == ref
    g.close()
