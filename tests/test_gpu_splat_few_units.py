"""GPU test of the cubic splats on both sides of the unit counts from which warps look ahead: the same sums, bit for
bit, where a brick's neighbourhood is the same, in grids of few and of many bricks, single and batched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(gvx, pos, w, vel, logdim):
    g = gvx.Grid(0)
    g.configure(logdim)
    g.add_channel(0, gvx.T_FLOAT, 1)
    g.add_channel(1, gvx.T_FLOAT3, 1)
    g.commit_points_host(pos, vel=vel, weight=w)
    g.rebuild_topology(len(pos), 2.0, mode=gvx.TOPO_FULL)
    g.update_atlas()
    g.insert_points(len(pos))
    return g


@pytest.mark.parametrize("log_brick,extra", [(3, 2), (3, 2000), (3, 8000), (3, 30_000), (3, 100_000), (4, 20_000)])
@pytest.mark.parametrize("chan_vel", [-1, 1])
@pytest.mark.parametrize("batch", [False, True])
def test_same_bits(gvx_mod, log_brick, extra, chan_vel, batch):
    rng = np.random.default_rng(3)
    brick = 1 << log_brick
    logdim = (log_brick, 3, 3, 3, 4)
    # a dense cloud, and points far from it that only add bricks
    core = 200.0 + rng.normal(0.0, 12.0, (20_000, 3))
    far = rng.random((extra, 3)) * 500.0 + 330.0
    far[:2] = [[330.0] * 3, [830.0] * 3]
    ends = np.array([[100.0] * 3, [300.0] * 3])  # (the root is the same)
    pos = np.concatenate([core, ends, far]).astype(np.float32)
    w = rng.uniform(0.5, 1.5, len(pos)).astype(np.float32)
    vel = rng.normal(0.0, 1.0, pos.shape).astype(np.float32)
    m = len(core) + 2

    def bricks(n):
        g = _grid(gvx_mod, pos[:n], w[:n], vel[:n], logdim)
        for c in (0, 1):
            g.fill_channel(c, [9.0] * 4)
        if batch and n > m:
            b = gvx_mod.Batch(0)
            b.set_grids([g])
            b.splat(gvx_mod.SPLAT_CUBIC, 2.5, chan_vel=chan_vel, graph=False)
            g.sync()
            b.close()
        else:
            g.splat(gvx_mod.SPLAT_CUBIC, n, 2.5, chan_vel=chan_vel)
        used = g.info()["used_leaves"]
        amap = g.read_atlas_map()[:used, :3]
        out = {}
        chans = [g.read_channel(c) for c in ((0, 1) if chan_vel > 0 else (0,))]
        i = slice(1, 1 + brick)
        for s in np.nonzero((amap < 312).all(axis=1))[0]:
            out[tuple(amap[s])] = tuple(c[s][i, i, i].tobytes() for c in chans)
        g.close()
        return out

    ref, got = bricks(m), bricks(len(pos))
    assert len(ref) > 50 and got == ref
