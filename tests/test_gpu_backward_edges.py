"""GPU test of the adjoint splat where its loops end: point counts around the claims of a warp, supports
of a few voxels and of almost a brick's width, points beside the zero planes, missing bricks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _adjoint(pos, w, r, G, owner, mode):
    """dL/dp, dL/dw, dL/dR in FP64: sums over the voxels that `owner` has"""
    gp, gw, gr = np.zeros((len(pos), 3)), np.zeros(len(pos)), np.zeros(len(pos))
    for i, (p, wi, R) in enumerate(zip(pos.astype(np.float64), w.astype(np.float64), r.astype(np.float64))):
        lo = np.maximum(np.floor(p - R).astype(int), 0) if mode else np.floor(p).astype(int)
        hi = np.ceil(p + R).astype(int) if mode else lo + 1
        v = np.stack(np.meshgrid(*[np.arange(a, b + 1) for a, b in zip(lo, hi)], indexing="ij"), -1).reshape(-1, 3)
        g = np.array([owner(tuple(x)) for x in v])
        d = v - p
        if mode:
            h = 0.5 * R
            dist = np.sqrt((d * d).sum(1))
            q = dist / h
            m4 = np.where(q < 1, 1 - 1.5 * q ** 2 + 0.75 * q ** 3, np.where(q < 2, 0.25 * (2 - q) ** 3, 0.0))
            dm = np.where(q < 1, -3 * q + 2.25 * q ** 2, np.where(q < 2, -0.75 * (2 - q) ** 2, 0.0))
            norm = 1.0 / (np.pi * h ** 3)
            gw[i] = (g * norm * m4).sum()
            gr[i] = -(g * wi * norm * (3 * m4 + q * dm)).sum() / (2 * h)
            s = np.where(dist > 0, g * wi * norm * dm / (h * np.maximum(dist, 1e-300)), 0.0)
            gp[i] = (s[:, None] * -d).sum(0)
        else:
            u = np.maximum(1 - np.abs(d), 0.0)
            sg = np.where(d <= 0, -1.0, 1.0)
            gw[i] = (g * u.prod(1)).sum()
            for k in range(3):
                o = [j for j in range(3) if j != k]
                gp[i, k] = (g * wi * sg[:, k] * u[:, o[0]] * u[:, o[1]]).sum()
    return gp, gw, gr


@pytest.mark.parametrize("log_brick,n,rmin,rmax,mode", [(3, 1, 2.0, 2.0, 1), (3, 7, 1.0, 3.0, 1), (3, 9, 0.6, 6.9, 1),
                                                        (3, 300, 0.6, 3.5, 1), (4, 33, 1.0, 14.5, 1), (2, 65, 0.6, 2.9, 1),
                                                        (3, 17, 1.0, 1.0, 0), (4, 300, 1.0, 1.0, 0)])
def test_adjoint_against_sums(gvx_mod, log_brick, n, rmin, rmax, mode):
    import torch

    rng = np.random.default_rng(n)
    brick = 1 << log_brick
    pos = (rng.random((n, 3)) * 4 * brick + 0.1).astype(np.float32)
    far = np.array([[9.5 * brick] * 3], np.float32)  # the root holds all neighbours of the cluster
    pos = np.concatenate([pos, far])
    n += 1
    w = rng.uniform(0.5, 1.5, n).astype(np.float32)
    r = rng.uniform(rmin, rmax, n).astype(np.float32)
    g = gvx_mod.Grid(0)
    g.configure((log_brick, 3, 3, 3))
    g.add_channel(0, gvx_mod.T_FLOAT, 1)
    dev = [torch.from_numpy(x).cuda() for x in (pos, w, r)]
    g.set_points(n, dev[0])
    g.set_point_attribs(weight=dev[1], radius=dev[2] if mode else None)
    g.rebuild_topology(n, 1.0 if log_brick > 1 else 0.0, mode=gvx_mod.TOPO_FULL)
    g.update_atlas()
    g.splat(gvx_mod.SPLAT_CUBIC if mode else gvx_mod.SPLAT_TRILINEAR, n, 1.0)
    used, P = g.info()["used_leaves"], brick + 2
    G = np.zeros(g.channel_bytes(0) // 4, np.float32).reshape(-1, P, P, P)
    G[:] = rng.normal(0.0, 1.0, G.shape)
    amap = g.read_atlas_map()[:used]
    slot = {tuple(p[:3] // brick): i for i, p in enumerate(amap)}

    def owner(v):
        s = slot.get(tuple(x // brick for x in v), -1)
        return float(G[s, v[2] % brick + 1, v[1] % brick + 1, v[0] % brick + 1]) if s >= 0 else 0.0

    out = [torch.full(s, 7.0, device="cuda") for s in ((n, 3), (n,), (n,))]
    g.splat_backward(gvx_mod.SPLAT_CUBIC if mode else gvx_mod.SPLAT_TRILINEAR, n, 1.0, torch.from_numpy(G).cuda(), out[0],
                     out[1], out[2] if mode else None)
    g.sync()
    ref = _adjoint(pos, w, r, G, owner, mode)
    for got, want in zip(out[:3 if mode else 2], ref):
        # the adjoint's stated bound: 1e-4 of the largest gradient of its kind
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-4 * np.abs(want).max()
    g.close()
