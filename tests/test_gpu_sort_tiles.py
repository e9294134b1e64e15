"""GPU test of the radix sort at the edges of its tiles and of the sizes that choose them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 1023, 1024, 1025, 4097, 299_999, 300_000, 300_001, 1_999_999, 2_000_001,
                               2_007_041])
@pytest.mark.parametrize("bits", [1, 8, 13, 24, 32])
@pytest.mark.parametrize("spread", ["full", "few"])
def test_sorted_as_numpy_sorts(gvx_mod, n, bits, spread):
    import torch

    rng = np.random.default_rng(n + bits)
    top = (1 << bits) if spread == "full" else min(1 << bits, 3)  # few: long runs of equal digits
    keys = rng.integers(0, top, n, dtype=np.uint64).astype(np.uint32)
    if spread == "few":
        keys[rng.random(n) < 0.01] = (1 << bits) - 1  # the digits that pairs past the end would have
    vals = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    g = gvx_mod.Grid(0)
    kd, vd = torch.from_numpy(keys.view(np.int32)).cuda(), torch.from_numpy(vals.view(np.int32)).cuda()
    ko, vo = torch.empty_like(kd), torch.empty_like(vd)
    gvx_mod.radix_sort(g, kd, vd, ko, vo, n, bits)
    g.sync()
    order = np.argsort(keys, kind="stable")
    rk, rv = keys[order], vals[order]
    assert np.array_equal(ko.cpu().numpy().view(np.uint32), rk)
    assert np.array_equal(vo.cpu().numpy().view(np.uint32), rv)
    assert np.array_equal(kd.cpu().numpy().view(np.uint32), keys)  # the input is left as it was
    assert np.array_equal(vd.cpu().numpy().view(np.uint32), vals)
    # the same with outputs that are the inputs, and with an input beside the output in one buffer
    both = torch.cat([kd, kd])
    gvx_mod.radix_sort(g, both[:n], vd, both[n:], vo, n, bits)
    gvx_mod.radix_sort(g, kd, vd, kd, vd, n, bits)
    g.sync()
    assert np.array_equal(both[n:].cpu().numpy().view(np.uint32), rk)
    assert np.array_equal(kd.cpu().numpy().view(np.uint32), rk)
    assert np.array_equal(vd.cpu().numpy().view(np.uint32), rv)
    g.close()
