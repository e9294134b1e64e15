"""GPU test of a wait that ran out (a smoothing with a withheld slot) with another call before the next check: the
calls that start a device error record of their own leave the timeout in it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["sort", "subcell lists", "adjoint", "import"])
def test_timeout_is_reported(gvx_mod, call, tmp_path):
    import torch

    rng = np.random.default_rng(1)
    n = 3000
    pos = torch.from_numpy((rng.random((n, 3)) * 60.0 + 20.0).astype(np.float32)).cuda()
    g = gvx_mod.Grid(0)
    g.configure((3, 3, 3, 3, 5))
    g.add_channel(0, gvx_mod.T_FLOAT, 1)
    g.set_points(n, pos)
    g.rebuild_topology(n, 1.0, mode=gvx_mod.TOPO_FULL)
    g.finish_topology()
    g.update_atlas()
    g.splat(gvx_mod.SPLAT_TRILINEAR, n, 1.0)
    if call == "import":
        g.save_vbx(str(tmp_path / "a.vbx"))
    g.sync()
    assert g.lib.gvx_test_smooth_withheld_slot(g.h, 0, 3) == 0
    with pytest.raises(gvx_mod.GvxError) as e:
        if call == "sort":
            keys = torch.from_numpy(rng.integers(0, 1 << 16, n).astype(np.int32)).cuda()
            out = torch.empty_like(keys), torch.empty_like(keys)
            gvx_mod.radix_sort(g, keys, keys, out[0], out[1], n, 16)
        elif call == "subcell lists":
            g.insert_points_subcell(4, n, 1.0)
        elif call == "import":
            g.load_vbx(str(tmp_path / "a.vbx"))
        else:
            dl = torch.ones(g.channel_bytes(0) // 4, device="cuda")
            grads = torch.empty((n, 3), device="cuda"), torch.empty(n, device="cuda")
            g.splat_backward(gvx_mod.SPLAT_TRILINEAR, n, 1.0, dl, grads[0], grads[1])
        g.sync()
    assert e.value.status == gvx_mod.ERR_TIMEOUT
    # reported once: the grid goes on
    g.set_points(n, pos)
    g.rebuild_topology(n, 1.0, mode=gvx_mod.TOPO_FULL)
    g.update_atlas()
    g.splat(gvx_mod.SPLAT_TRILINEAR, n, 1.0)
    g.sync()
    g.close()
