"""GPU test of the subcell lists that are not written out (bricks of 8, subcells of 4, no colours, the
points of the last full build) against the written ones, which point colours call for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lists(gvx, pos, radius, fp16, op, accum, colours, topo, trans=None, move=None):
    """(entries, channel bricks) of one build, insert and gather; move: positions written over the bound
    ones after the build"""
    import torch

    g = gvx.Grid(0)
    g.configure((3, 3, 3, 3, 5))
    g.add_channel(0, gvx.T_FLOAT, 1)
    n = len(pos)
    p = torch.from_numpy(pos).cuda()
    c = torch.zeros((n, 4), dtype=torch.uint8, device="cuda") if colours else None
    g.set_points(n, p, clr=c)
    g.rebuild_topology(n, topo, mode=gvx.TOPO_FULL)
    g.update_atlas()
    g.fill_channel(0, [0.5])
    if move is not None:
        p.copy_(torch.from_numpy(move))
        torch.cuda.synchronize()
    if fp16:
        m = g.insert_points_subcell_fp16(4, n, radius, trans)
        # the lists are the insert's: what is bound or grouped afterwards changes nothing
        g.set_points(n, torch.zeros_like(p))
        g.gather_levelset_fp16(4, n, radius, m, trans, chan=0)
    else:
        m = g.insert_points_subcell(4, n, radius, trans)
        f = g.gather_levelset if op == "levelset" else g.gather_density
        f(4, n, radius, m, trans, chan=0, accum=accum)
    out = g.read_channel(0)[:g.info()["used_leaves"]].copy()
    g.close()
    return m, out


@pytest.mark.parametrize("n,side,radius,topo", [(2, 12, 1.0, 2.0), (50, 20, 1.0, 2.0), (3000, 60, 0.0, 0.0),
                                                 (3000, 60, 2.0, 3.0), (40_000, 50, 1.0, 2.0), (40_000, 200, 1.5, 0.0)])
@pytest.mark.parametrize("fp16,op,accum", [(True, "levelset", False), (False, "levelset", False),
                                           (False, "levelset", True), (False, "density", False), (False, "density", True)])
def test_direct_lists_equal_the_written_ones(gvx_mod, n, side, radius, topo, fp16, op, accum):
    rng = np.random.default_rng(n + side)
    pos = (rng.random((n, 3)) * side + 20.0).astype(np.float32)
    pos[::7] = np.round(pos[::7])  # on the faces of voxels, subcells and bricks
    if n > 10:
        pos[3] = (-1.0, 30.0, 30.0)  # dropped by the build
        pos[5] = (61.0, 62.0, 63.0)
    args = (gvx_mod, pos, radius, fp16, op, accum)
    m, got = _lists(*args, False, topo)
    k, ref = _lists(*args, True, topo)
    assert m == k
    if fp16:
        assert got.tobytes() == ref.tobytes()
    else:  # distances of at most 12 voxels, four roundings either way
        assert np.abs(got - ref).max() <= 8 * 12 * 2.0 ** -24


@pytest.mark.parametrize("fp16", [True, False])
def test_points_moved_in_place_and_translations(gvx_mod, fp16):
    """points that are no longer where the build found them, or are inserted with a translation, are
    listed where they are"""
    rng = np.random.default_rng(4)
    pos = (rng.random((5000, 3)) * 60 + 20.0).astype(np.float32)
    moved = (pos + rng.normal(0.0, 1.0, pos.shape)).astype(np.float32)
    for kw in (dict(move=moved), dict(trans=(1.0, -2.0, 0.5))):
        m, got = _lists(gvx_mod, pos, 1.0, fp16, "levelset", False, False, 2.0, **kw)
        k, ref = _lists(gvx_mod, pos, 1.0, fp16, "levelset", False, True, 2.0, **kw)
        assert m == k and got.tobytes() == ref.tobytes()
