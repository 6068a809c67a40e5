"""Neighbour lists exported into memory that is not plain host memory: device and
pinned arrays take them too."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coded", [False, True])
@pytest.mark.parametrize("place", ["device", "pinned"])
@pytest.mark.parametrize("n", [130, 100003])
def test_lists_into(n, place, coded):
    import sphg as S
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    sim = S.Sim(S.params(order="morton", h=1.5 / np.sqrt(n), lo=(0, 0), hi=(1, 1)), n)
    sim.upload(*rng.uniform(0, 1, (4, n)))
    sim.preloop()
    offs, idx = sim.neighbor_lists_encoded() if coded else sim.neighbor_lists()
    where = dict(device="cuda") if place == "device" else dict(pin_memory=True)
    o, i = torch.zeros(n + 1, dtype=torch.int64, **where), torch.zeros(len(idx), dtype=torch.int32, **where)
    torch.cuda.synchronize()
    total = ctypes.c_int64()
    f = S.lib().sphg_neighbor_lists_encoded if coded else S.lib().sphg_neighbor_lists
    S.check(f(sim._h, ctypes.cast(o.data_ptr(), ctypes.POINTER(ctypes.c_int64)),
              ctypes.cast(i.data_ptr(), ctypes.POINTER(ctypes.c_int32)), ctypes.byref(total), None))
    torch.cuda.synchronize()
    assert total.value == len(idx)
    assert np.array_equal(o.cpu().numpy(), offs) and np.array_equal(i.cpu().numpy(), idx)
    sim.close()
