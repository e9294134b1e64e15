"""GPU test of the launch count of a batch's splats: the same with a captured graph as without, capture and replay
alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["trilinear", "cubic"])
def test_counts(gvx_mod, mode):
    rng = np.random.default_rng(2)
    kind = gvx_mod.SPLAT_TRILINEAR if mode == "trilinear" else gvx_mod.SPLAT_CUBIC
    grids = []
    for n in (2000, 5000):
        g = gvx_mod.Grid(0)
        g.configure((3, 3, 3, 3, 5))
        g.add_channel(0, gvx_mod.T_FLOAT, 1)
        g.commit_points_host((rng.random((n, 3)) * 60.0 + 20.0).astype(np.float32))
        g.rebuild_topology(n, 1.0, mode=gvx_mod.TOPO_FULL)
        g.update_atlas()
        grids.append(g)
    b = gvx_mod.Batch(0)
    b.set_grids(grids)

    def splat(graph):
        before = b.kernel_launches()
        b.splat(kind, 1.5, graph=graph)
        return b.kernel_launches() - before

    plain = splat(False)
    # the splat, and for trilinear density the launch that sums the listed dense units
    assert plain == (2 if mode == "trilinear" else 1)
    assert [splat(True) for _ in range(4)] == [plain] * 4
    b.close()
    for g in grids:
        g.close()
