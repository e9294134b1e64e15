"""GPU test of splats and scatters from several threads, a grid each: launches of one kernel whose shared memory
differs with the grid (the slab height follows the brick count, the colour table the colour mode) do not disturb
each other."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["trilinear", "cubic", "cubic16", "scatter"])
def test_grids_of_different_sizes(gvx_mod, what):
    import torch

    rng = np.random.default_rng(5)
    logdim = (4 if what == "cubic16" else 3, 3, 3, 3, 5)
    grids = []
    for k, (n, side) in enumerate([(60, 40.0), (40_000, 700.0)] * 2):
        p = torch.from_numpy((rng.random((n, 3)) * side + 40.0).astype(np.float32)).cuda()
        c = torch.zeros((n, 4), dtype=torch.uint8, device="cuda") if what == "scatter" and k % 2 else None
        g = gvx_mod.Grid(0)
        g.configure(logdim)
        g.add_channel(0, gvx_mod.T_FLOAT, 1)
        g.add_channel(1, gvx_mod.T_UCHAR4, 1)
        g.set_points(n, p, clr=c)
        g.rebuild_topology(n, 1.0, mode=gvx_mod.TOPO_FULL)
        g.update_atlas()
        grids.append((g, n, p, c))
    torch.cuda.synchronize()

    def call(g, n):
        if what == "scatter":
            g.scatter_density(n, 1.0, avg_color=True)
        elif what == "trilinear":
            g.splat(gvx_mod.SPLAT_TRILINEAR, n, 1.0)
        else:
            g.splat(gvx_mod.SPLAT_CUBIC, n, 3.0)

    ref = []
    if what != "scatter":
        for g, n, _, _ in grids:
            call(g, n)
            g.sync()
            ref.append(g.read_channel(0)[:g.info()["used_leaves"]].tobytes())
    failed = []

    def loop(g, n):
        try:
            for _ in range(1500):
                call(g, n)
            g.sync()
        except gvx_mod.GvxError as e:
            failed.append(str(e))

    threads = [threading.Thread(target=loop, args=(g, n)) for g, n, _, _ in grids]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for (g, _, _, _), r in zip(grids, ref):
        assert g.read_channel(0)[:g.info()["used_leaves"]].tobytes() == r
    for g, _, _, _ in grids:
        g.close()
