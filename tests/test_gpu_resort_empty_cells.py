"""Movers of one warp into empty cells, whose insertion points are searched once for
every cell: the order of the full sort, and the time of a search or two instead of
one for every mover."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["morton", "rowmajor"])
@pytest.mark.parametrize("cells", [1, 2, 5, 31])
@pytest.mark.parametrize("block", [0, 128])
def test_one_warp_to_several_empty_cells(cells, order, block):
    """31 particles of one cell go to 1, 2, 5 or 31 empty cells at once, in turn."""
    import sphg as S
    rng = np.random.default_rng(cells)
    h, n = 1.0 / 64, 700
    x, y = rng.uniform(0.3, 0.7, n), rng.uniform(0.7, 0.95, n)
    x[:31], y[:31] = 5.5 * h, 20.5 * h
    to = np.arange(31) % cells
    vx, vy = np.zeros(n), np.zeros(n)
    vx[:31], vy[:31] = (3 + 2 * (to % 6)) * h / 1e-3, (to // 6 + 1) * h / 1e-3
    mix = rng.permutation(n)
    state = [v[mix] for v in (x, y, vx, vy)]
    prm = S.params(order=order, h=h, dt=1e-3, k=0.0, mu=0.0, gx=0.0, gy=0.0, lo=(0, 0), hi=(1, 1))
    out = []
    for resort in (1, 0):
        sim = S.Sim(prm, n, S.options(precision=S.SPLIT, resort=resort, block_threads=block))
        sim.upload(*state)
        sim.preloop()
        sim.step(1)
        if resort:
            assert sim.debug(S.DBG_RESORT)[:2].tolist() == [1, 31]
        o = sim.download()
        o["keys"], o["perm"] = sim.debug(S.DBG_KEYS), sim.debug(S.DBG_PERM)
        o["offs"], o["idx"] = sim.neighbor_lists()  # walks the cell ranges
        out.append(o)
        sim.close()
    for f in out[0]:
        assert np.array_equal(out[0][f], out[1][f], equal_nan=True), f


def test_a_clump_into_an_empty_cell_costs_little():
    """32 particles of one cell that move to the next, empty one every iteration,
    against the same at rest: 6 us an iteration more, 20 with a search each."""
    import sphg as S
    rng = np.random.default_rng(1)
    n, many, h = 30000, 32, 1.0 / 256
    x, y = rng.uniform(0, 1, n), rng.uniform(0.5, 1, n)
    x[:many], y[:many] = ((10 + rng.uniform(0.3, 0.7, many)) * h for _ in range(2))
    prm = S.params(order="morton", h=h, dt=1e-3, k=0.0, mu=0.0, gx=0.0, gy=0.0, lo=(0, 0), hi=(1, 1))
    sim = S.Sim(prm, n, S.options(precision=S.SPLIT))
    best = []
    for speed in (h / 1e-3, 0.0):
        vx = np.zeros(n)
        vx[:many] = speed
        t = []
        for _ in range(7):
            sim.upload(x, y, vx, np.zeros(n))
            sim.preloop()
            sim.diagnostics()  # waits
            a = time.perf_counter()
            sim.step(100)
            sim.diagnostics()
            t.append((time.perf_counter() - a) / 100)
        assert sim.debug(S.DBG_RESORT)[:2].tolist() == [1, many if speed else 0]
        best.append(min(t))
    sim.close()
    assert best[0] - best[1] <= 13e-6, best
