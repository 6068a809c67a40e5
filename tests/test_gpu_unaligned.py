"""Caller's arrays at addresses that are no multiple of their entries' size (fields
of a packed record): the device leaves them to the host, the values are those of
aligned arrays."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("x", "y", "vx", "vy", "rho", "fx", "fy")


def _unaligned(n, dtype, by):
    """n entries that start `by` bytes past an aligned address."""
    size = np.dtype(dtype).itemsize
    raw = np.zeros(n * size + 64, np.uint8)
    at = -raw.ctypes.data % 16 + by
    a = np.frombuffer(raw, dtype, n, offset=at)
    assert a.ctypes.data % size
    return a


def _sim(S, n, prec):
    rng = np.random.default_rng(n)
    sim = S.Sim(S.params(order="morton", h=0.07, lo=(0, 0), hi=(1, 1)), n,
                S.options(precision=S.SPLIT if prec == "split" else S.PLAIN))
    state = rng.uniform(0, 1, (4, n))
    sim.upload(*state)
    sim.preloop()
    return sim, state


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("prec", ["plain", "split"])
@pytest.mark.parametrize("by", [1, 4, 6])
def test_download(by, prec, mode):
    import sphg as S
    n = 1001
    sim, _ = _sim(S, n, prec)
    want = sim.download()
    sim.set_host_access(mode)
    for odd in NAMES + ("ids",):
        if odd == "ids" and by == 4:
            continue  # aligned
        out = {k: np.zeros(n) for k in NAMES}
        out["ids"] = np.zeros(n, np.int32)
        out[odd] = _unaligned(n, out[odd].dtype, by)
        sim.download(out=out)
        for k in out:
            assert np.array_equal(out[k], want[k]), (odd, k)
    sim.close()


@pytest.mark.parametrize("by", [1, 2, 3])
def test_neighbour_lists(by):
    import sphg as S
    n = 1001
    sim, _ = _sim(S, n, "plain")
    offs, idx = sim.neighbor_lists()
    total = ctypes.c_int64()
    o, i = _unaligned(n + 1, np.int64, by), _unaligned(len(idx), np.int32, by)
    S.check(S.lib().sphg_neighbor_lists(sim._h, o.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)),
                                        i.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), ctypes.byref(total), None))
    assert total.value == len(idx) and np.array_equal(o, offs) and np.array_equal(i, idx)
    sim.close()


@pytest.mark.parametrize("prec", ["plain", "split"])
@pytest.mark.parametrize("by", [1, 4])
def test_upload(by, prec):
    import sphg as S
    n = 1001
    sim, state = _sim(S, n, prec)
    sim.set_host_access(0)
    sim.upload(*state)
    sim.preloop()
    want = sim.download()
    sim.set_host_access(1)
    for odd in range(4):
        arrays = list(state)
        arrays[odd] = _unaligned(n, np.float64, by)
        arrays[odd][:] = state[odd]
        sim.upload(*arrays)
        sim.preloop()
        got = sim.download()
        for k in want:
            assert np.array_equal(got[k], want[k]), (odd, k)
    sim.close()


@pytest.mark.parametrize("by", [1, 4])
def test_headers(by):
    import sphg as S
    n = 1001
    sim, state = _sim(S, n, "split")
    want = sim.step_headers(5)
    sim.upload(*state)
    sim.preloop()
    got = _unaligned(5 * 6, np.float64, by)
    sim.step_headers(5, out=got)
    one = _unaligned(6, np.float64, by)
    sim.diagnostics_async(one.ctypes.data)
    sim.diagnostics()  # waits
    assert np.array_equal(got, want.ravel()) and np.array_equal(one, want.ravel()[-6:])
    sim.close()
