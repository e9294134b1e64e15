"""GPU test of batch frames whose grids are grouped again between them -- by an insert with a translation, which
lays the tables of the leaves out for fewer of them than a frame's plan has room for: what the frames, and the
single and batched splats after them, use of those tables is the frame's own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOGDIM = (3, 3, 3, 3, 5)
N_CLUSTER, N_SPREAD = 12_000, 300


def _cloud(seed, leaves):
    """points of a few dense bricks, and N_SPREAD over `leaves` bricks of their own inside the same box"""
    rng = np.random.default_rng(seed)
    dense = 96.0 + rng.normal(0.0, 3.0, (N_CLUSTER, 3))
    cells = np.stack(np.meshgrid(*[np.arange(16)] * 3, indexing="ij"), -1).reshape(-1, 3)
    cells = cells[(np.abs(cells - 12) > 3).any(axis=1)]
    pick = cells[rng.permutation(len(cells))[:leaves]]
    pick[0], pick[1] = 0, 15  # the box stays
    spread = (pick[np.arange(N_SPREAD) % leaves] + 0.25 + 0.5 * rng.random((N_SPREAD, 3))) * 8.0 + 32.0
    p = np.concatenate([dense + 32.0, spread]).astype(np.float32)
    order = np.random.default_rng(1).permutation(len(p))
    return p[order]


def _reference(gvx, pos, w):
    g = gvx.Grid(0)
    g.configure(LOGDIM)
    g.add_channel(0, gvx.T_FLOAT, 1)
    g.commit_points_host(pos, weight=w)
    g.rebuild_topology(len(pos), 0.0, mode=gvx.TOPO_FULL)
    g.update_atlas()
    g.splat(gvx.SPLAT_TRILINEAR, len(pos), 1.0)
    used = g.info()["used_leaves"]
    out = g.read_channel(0)[:used].copy()
    g.close()
    return used, out


@pytest.mark.parametrize("after", ["single", "batch", "recaptured"])
def test_frames_after_another_grouping(gvx_mod, after):
    import torch

    clouds = [_cloud(2, 150), _cloud(3, 150), _cloud(4, 200), _cloud(5, 120)]
    n = len(clouds[0])
    w = np.random.default_rng(7).uniform(0.5, 1.5, n).astype(np.float32)
    refs = [_reference(gvx_mod, c, w) for c in clouds]
    g = gvx_mod.Grid(0)
    g.configure(LOGDIM)
    g.add_channel(0, gvx_mod.T_FLOAT, 1)
    p, wd = torch.from_numpy(clouds[0]).cuda(), torch.from_numpy(w).cuda()
    g.set_points(n, p)
    g.set_point_attribs(weight=wd)
    b = gvx_mod.Batch(0)
    b.set_grids([g])

    def frame(k):
        p.copy_(torch.from_numpy(clouds[k]))
        torch.cuda.synchronize()
        g.fill_channel(0, [9.0])
        b.frame(0.0, gvx_mod.SPLAT_TRILINEAR, 1.0)
        check(k)

    def check(k):
        used, den = refs[k]
        g.sync()
        assert g.info()["used_leaves"] == used
        assert g.read_channel(0)[:used].tobytes() == den.tobytes()

    def splat(k):
        g.fill_channel(0, [9.0])
        g.splat(gvx_mod.SPLAT_TRILINEAR, n, 1.0)
        check(k)

    frame(0)
    frame(1)
    assert b.frame_path() == (1, 0)
    g.insert_points(n, (0.25, 0.0, 0.0))  # before the capture
    frame(2)
    assert b.frame_path() == (2, 0)
    frame(1)
    splat(1)
    g.insert_points(n, (0.25, 0.0, 0.0))
    if after == "recaptured":
        # other attributes: a capture of its own
        wd2 = wd.clone()
        g.set_point_attribs(weight=wd2)
    frame(2)  # more bricks than the grouping in between had
    assert b.frame_path() == (2, 0)
    if after == "batch":
        g.fill_channel(0, [9.0])
        b.splat(gvx_mod.SPLAT_TRILINEAR, 1.0)
        check(2)
    else:
        splat(2)
    frame(3)
    assert b.frame_path() == (2, 0)
    splat(3)
    b.close()
    g.close()
