"""GPU test of a smoothing whose wait for a slot runs out (the slot is withheld by a test hook; no GPU fault): no
slot is written that was not read, the error is reported, and the grid goes on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(gvx, rng):
    g = gvx.Grid(0)
    g.configure((3, 3, 3, 3, 5))
    g.set_channel_default(20, 20, 15)  # 6000 slots, several for every block
    g.add_channel(0, gvx.T_FLOAT, 1)
    a = rng.normal(0.0, 1.0, g.channel_bytes(0) // 4).astype(np.float32).reshape(-1, 10, 10, 10)
    g.write_channel(0, a)
    return g, a


@pytest.mark.parametrize("slot", [0, 1234, 3000, 5999])
def test_withheld_slot_stays_as_it_is(gvx_mod, slot):
    g, a = _grid(gvx_mod, np.random.default_rng(slot))
    assert g.lib.gvx_test_smooth_withheld_slot(g.h, 0, slot) == 0
    with pytest.raises(gvx_mod.GvxError) as e:
        g.sync()
    assert e.value.status == gvx_mod.ERR_TIMEOUT
    g.sync()  # reported once
    got = g.read_channel(0)
    g.write_channel(0, a)
    g.compute(gvx_mod.FUNC_SMOOTH, 0, 1, (4.0, 0.1, 0.0), update_apron=False, skip_over_aprons=True)
    g.sync()
    ref = g.read_channel(0)
    assert got[slot].tobytes() == a[slot].tobytes()
    kept = np.array([got[s].tobytes() == a[s].tobytes() for s in range(len(a))])
    done = np.array([got[s].tobytes() == ref[s].tobytes() for s in range(len(a))])
    assert np.all(kept | done) and 1 <= kept.sum() <= 4  # (the block's later slots)
    g.close()
