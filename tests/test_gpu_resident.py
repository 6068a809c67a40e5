"""Many iterations of a small instance in one cluster (the default up to 16,384
particles) against the graph of kernels (chosen by naming a block size): the
same bits, states and step headers alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(S, prm, n, state, prec, steps):
    out = []
    for block in (0, 128):
        sim = S.Sim(prm, n, S.options(precision=prec, block_threads=block))
        sim.upload(*state)
        sim.preloop()
        h = [sim.step_headers(steps)]
        sim.step(1)
        h.append(sim.step_headers(2))
        o = sim.download()
        o["headers"] = np.concatenate(h)
        o["keys"], o["perm"], o["resort"] = (sim.debug(k) for k in (S.DBG_KEYS, S.DBG_PERM, S.DBG_RESORT))
        o["diag"] = sim.diagnostics()
        out.append(o)
        sim.close()
    for f in out[0]:
        assert np.array_equal(out[0][f], out[1][f], equal_nan=True), f
    return out[0]


@pytest.mark.parametrize("prec", ["plain", "split"])
@pytest.mark.parametrize("nx,ny", [(1, 1), (8, 5), (31, 33), (128, 32), (129, 127), (128, 128)])
def test_resident_equals_kernels(nx, ny, prec):
    import sphg as S
    import workloads as W
    dx = 0.4 / nx
    p, x, y, _, _ = W.dam_break(nx, ny, dx, seed=nx, order="rowmajor" if nx % 2 else "morton",
                                box=(2.5 * nx * dx, 1.25 * ny * dx))
    rng = np.random.default_rng(ny)
    vx, vy = rng.uniform(-20, 20, (2, len(x))) * dx / 0.005  # a few percent change cell every iteration
    _both(S, S.params(**p), len(x), (x, y, vx, vy), S.SPLIT if prec == "split" else S.PLAIN,
          130 if nx * ny < 2000 else 20)  # 130: more than one launch holds


@pytest.mark.parametrize("prec", ["plain", "split"])
def test_resident_full_sort(prec):
    """More than 8,192 of 12,000 free particles change cell every iteration: the
    cluster sorts by counting."""
    import sphg as S
    rng = np.random.default_rng(3)
    n, h = 12000, 1.0 / 90
    x, y = rng.uniform(0, 1, (2, n)).astype(np.float32).astype(np.float64)
    vx, vy = rng.uniform(0.6, 1.0, (2, n)) * rng.choice([-1, 1], (2, n)) * h / 1e-3
    prm = S.params(order="morton", h=h, dt=1e-3, k=0.0, mu=0.0, gx=0.0, gy=0.0, lo=(0, 0), hi=(1, 1))
    o = _both(S, prm, n, (x, y, vx, vy), S.SPLIT if prec == "split" else S.PLAIN, 5)
    assert o["resort"][0] == 0 and o["resort"][1] > 8192


def test_resident_periodic_many_neighbours():
    """A periodic vortex of wide kernels: more neighbours than the density pass records."""
    import sphg as S
    import workloads as W
    p, x, y, vx, vy, _ = W.taylor_green(60, seed=2)
    p["h"] = 3.2 / 60
    _both(S, S.params(**p), len(x), (x, y, vx, vy), S.PLAIN, 30)


@pytest.mark.parametrize("order", ["morton", "rowmajor"])
@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("cells", [3, 4, 5, 9])
def test_split_update_in_a_few_cells(cells, periodic, order):
    """Split positions in grids of a few cells: the kernels update a particle that
    stays in a cell clear of the walls without the walls' and the key's arithmetic,
    the resident iteration never does -- the same bits at every wall and edge."""
    import sphg as S
    rng = np.random.default_rng(cells + periodic)
    n, h = 60 * cells, 1.0
    lo, hi = (-0.25, 0.5), (-0.25 + cells * h - 0.3 * (1 - periodic), 0.5 + cells * h - 0.01 * (1 - periodic))
    x, y = rng.uniform(lo[0], hi[0], n), rng.uniform(lo[1], hi[1], n)
    vx, vy = rng.normal(0, 30, (2, n))
    prm = S.params(order=order, h=h, dt=1e-3, k=1.0, mu=0.01, lo=lo, hi=hi, periodic=periodic)
    _both(S, prm, n, (x, y, vx, vy), S.SPLIT, 60)
