"""The most movers that an iteration merges: 64 into one gap of the order, 512 into
one run of 512 slots -- merged up to them, sorted fully beyond, the same bits either
way; in the kernels of a graph and in the cluster of a small instance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "vx", "vy", "rho", "fx", "fy", "ids")


def _one_iteration(S, order, h, state, resort, block):
    prm = S.params(order=order, h=h, dt=1e-3, k=0.0, mu=0.0, gx=0.0, gy=0.0, lo=(0, 0), hi=(1, 1))
    sim = S.Sim(prm, len(state[0]), S.options(precision=S.SPLIT, resort=resort, block_threads=block))
    sim.upload(*state)
    sim.preloop()
    sim.step(1)
    rs = sim.debug(S.DBG_RESORT)
    o = sim.download()
    o["keys"], o["perm"] = sim.debug(S.DBG_KEYS), sim.debug(S.DBG_PERM)
    o["offs"], o["idx"] = sim.neighbor_lists()  # walks the cell ranges
    sim.close()
    return rs, o


def _check(S, order, h, state, movers, merged):
    for block in (0, 128):
        rs, a = _one_iteration(S, order, h, state, 1, block)
        _, b = _one_iteration(S, order, h, state, 0, block)
        assert rs[1] == movers and rs[0] == int(merged)
        for f in a:
            assert np.array_equal(a[f], b[f], equal_nan=True), f


@pytest.mark.parametrize("many", [63, 64, 65])
def test_movers_into_one_gap(many):
    import sphg as S
    rng = np.random.default_rng(many)
    h = 0.125
    x, y = (np.concatenate([rng.uniform(0.26, 0.37, many), rng.uniform(0.8, 0.99, 20)]) for _ in range(2))
    vx = np.concatenate([np.full(many, h / 1e-3), np.zeros(20)])  # one cell an iteration, an empty one
    _check(S, "morton", h, (x, y, vx, np.zeros(len(x))), many, many <= 64)


@pytest.mark.parametrize("many", [511, 512, 513])
def test_movers_into_one_run_of_slots(many):
    """Slots 0 to 511 are sixteen particles in each of the 32 cells of the first row;
    the movers come from the third row, 16 or 17 to each of the first 31 cells."""
    import sphg as S
    rng = np.random.default_rng(many)
    h = 1.0 / 32
    cx = np.concatenate([np.repeat(np.arange(32), 16), np.arange(many) % 31])
    x = (cx + rng.uniform(0.1, 0.9, len(cx))) * h
    y = rng.uniform(0.1, 0.9, len(cx)) * h
    vy = np.zeros(len(cx))
    y[512:] += 2 * h
    vy[512:] = -2 * h / 1e-3
    _check(S, "rowmajor", h, (x, y, np.zeros(len(cx)), vy), many, many <= 512)
