"""GPU test of the adjoint splat of points written in place after the splat grouped them: their gradients are
those of where they are now, also beyond the neighbours of the brick they were grouped in."""
import numpy as np
import pytest

from test_gpu_backward_edges import _adjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_brick,n,step,mode", [(3, 200, 2.0, 1), (3, 200, 20.0, 1), (2, 100, 9.0, 1), (3, 200, 20.0, 0),
                                                   (4, 60, 30.0, 1)])
def test_moved_points(gvx_mod, log_brick, n, step, mode):
    import torch

    rng = np.random.default_rng(n + int(step))
    brick = 1 << log_brick
    pos = (rng.random((n, 3)) * 5 * brick + 0.1).astype(np.float32)
    pos[-1] = 9.5 * brick  # the root holds all neighbours of the cluster
    moved = np.abs(pos + rng.uniform(-step, step, (n, 3))).astype(np.float32)
    moved[::4] = pos[::4]
    w = rng.uniform(0.5, 1.5, n).astype(np.float32)
    r = rng.uniform(0.6, min(3.5, brick - 1.1), n).astype(np.float32)
    g = gvx_mod.Grid(0)
    g.configure((log_brick, 3, 3, 3))
    g.add_channel(0, gvx_mod.T_FLOAT, 1)
    p, wd, rd = [torch.from_numpy(x).cuda() for x in (pos, w, r)]
    g.set_points(n, p)
    g.set_point_attribs(weight=wd, radius=rd if mode else None)
    g.rebuild_topology(n, 1.0, mode=gvx_mod.TOPO_FULL)
    g.update_atlas()
    kind = gvx_mod.SPLAT_CUBIC if mode else gvx_mod.SPLAT_TRILINEAR
    g.splat(kind, n, 1.0)
    g.sync()
    p.copy_(torch.from_numpy(moved))
    torch.cuda.synchronize()
    g.set_point_attribs(weight=wd, radius=rd if mode else None)
    used, P = g.info()["used_leaves"], brick + 2
    G = np.zeros(g.channel_bytes(0) // 4, np.float32).reshape(-1, P, P, P)
    G[:] = rng.normal(0.0, 1.0, G.shape)
    slot = {tuple(q[:3] // brick): i for i, q in enumerate(g.read_atlas_map()[:used])}

    def owner(v):
        s = slot.get(tuple(x // brick for x in v), -1)
        return float(G[s, v[2] % brick + 1, v[1] % brick + 1, v[0] % brick + 1]) if s >= 0 else 0.0

    out = [torch.full(s, 7.0, device="cuda") for s in ((n, 3), (n,), (n,))]
    g.splat_backward(kind, n, 1.0, torch.from_numpy(G).cuda(), out[0], out[1], out[2] if mode else None)
    g.sync()
    for got, want in zip(out[:3 if mode else 2], _adjoint(moved, w, r, G, owner, mode)):
        # the adjoint's stated bound: 1e-4 of the largest gradient of its kind
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-4 * np.abs(want).max()
    g.close()
