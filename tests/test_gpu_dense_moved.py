"""GPU test of the trilinear density splat of dense leaves whose points were written in place after the build
grouped them: before the insert that orders their cells, or after it, with the attributes set again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("when", ["before the insert", "after a splat"])
@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("share", [1.0, 0.001])
@pytest.mark.parametrize("far", [False, True])
def test_moved_points(gvx_mod, orc, when, batch, share, far):
    import torch

    rng = np.random.default_rng(11)
    n = 12_000
    pos = np.concatenate([96.0 + rng.normal(0.0, 3.0, (n, 3)), rng.random((300, 3)) * 200.0 + 8.0]).astype(np.float32)
    n = len(pos)
    w = rng.uniform(0.5, 1.5, n).astype(np.float32)
    # inside their octants of bricks, where the splat finds them, or by up to 1.5 voxels (inside the dilated
    # bricks): the points that change their octant may be found or not
    moved = pos.copy()
    pick = rng.random(n) < share
    m = pick.sum()
    if far:
        moved[pick] += rng.uniform(-1.5, 1.5, (m, 3)).astype(np.float32)
    else:
        moved[pick] = 4.0 * np.floor(pos[pick] / 4.0) + rng.integers(0, 256, (m, 3)) / 64.0
    stay = (np.floor(pos / 4.0) == np.floor(moved / 4.0)).all(axis=1)
    assert stay.all() != far
    logdim = (3, 3, 3, 3, 5)
    g = gvx_mod.Grid(0)
    g.configure(logdim)
    g.add_channel(0, gvx_mod.T_FLOAT, 1)
    p, wd = torch.from_numpy(pos).cuda(), torch.from_numpy(w).cuda()
    g.set_points(n, p)
    g.set_point_attribs(weight=wd)
    g.rebuild_topology(n, 2.0, mode=gvx_mod.TOPO_FULL)
    g.update_atlas()
    if when == "after a splat":
        g.splat(gvx_mod.SPLAT_TRILINEAR, n, 1.0)
    g.sync()
    p.copy_(torch.from_numpy(moved))
    torch.cuda.synchronize()
    if when == "after a splat":
        g.set_point_attribs(weight=wd)
    if batch:
        b = gvx_mod.Batch(0)
        b.set_grids([g])
        b.splat(gvx_mod.SPLAT_TRILINEAR, 1.0)
        g.sync()
        b.close()
    else:
        g.splat(gvx_mod.SPLAT_TRILINEAR, n, 1.0)
    used = g.info()["used_leaves"]
    got = g.read_channel(0)[:used]
    # one rounding a term (they are positive), six of a weight; the terms are the points of eight cells
    _, c = np.unique(moved.astype(np.int64) @ [1 << 20, 1 << 10, 1], return_counts=True)
    tol = (8 * int(c.max()) + 6) * 2.0 ** -24
    o = orc.Oracle(logdim)
    o.add_channel(0, orc.T_FLOAT)
    o.rebuild_topology(pos, 2.0)
    o.update_atlas()
    o.splat(orc.SPLAT_TRILINEAR, moved, 1.0, weight=w)
    assert np.all(got <= (1.0 + tol) * o.read_channel(0)[:used] + 2.0 ** -60)
    o.splat(orc.SPLAT_TRILINEAR, moved, 1.0, weight=np.where(stay, w, np.float32(0.0)))
    assert np.all(got >= (1.0 - tol) * o.read_channel(0)[:used] - 2.0 ** -60)
    g.close()
