"""The incremental re-sort (merge of the particles that changed cell, which also
writes the cell ranges) against the full radix sort: the same order and
therefore the same bits, at the sizes where its blocks end (512 slots, 32,768
slots), with many particles moving, into empty cells and past both ends of the
order, and with more particles moving into one gap than it merges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "vx", "vy", "rho", "fx", "fy", "ids")


def _run(S, prms, counts, state, prec, resort, steps):
    sim = S.Sim(prms, counts, S.options(precision=prec, resort=resort))
    sim.upload(*state)
    sim.preloop()
    merged, out = [], []
    for _ in range(steps):
        sim.step(1)
        merged.append(sim.debug(S.DBG_RESORT)[:2].tolist())
        o = sim.download()
        o["keys"], o["perm"] = sim.debug(S.DBG_KEYS), sim.debug(S.DBG_PERM)
        o["offs"], o["idx"] = sim.neighbor_lists()  # walks the cell ranges
        out.append(o)
    sim.close()
    return merged, out


def _same(a, b):
    for f in FIELDS + ("keys", "perm", "offs", "idx"):
        assert np.array_equal(a[f], b[f], equal_nan=True), f


def _free(n, rng, order, periodic=0, speed=0.25):
    """n free particles (no forces), about a third of the cells occupied, moving
    up to `speed` cells an iteration."""
    side = max(4, int(np.ceil(np.sqrt(3.0 * n))))
    h = 1.0 / side
    p = dict(order=order, h=h, dt=1e-3, k=0.0, mu=0.0, gx=0.0, gy=0.0, alpha=0.0, lo=(0, 0), hi=(1, 1),
             periodic=periodic)
    x, y = rng.uniform(0, 1, (2, n)).astype(np.float32).astype(np.float64)
    vx, vy = rng.uniform(-1, 1, (2, n)) * speed * h / 1e-3
    return p, x, y, vx, vy


@pytest.mark.parametrize("prec", ["plain", "split"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 511, 512, 513, 1024, 4095, 32767, 32768, 32769, 66000])
def test_merge_equals_full_sort_at_block_edges(n, prec):
    import sphg as S
    P = S.SPLIT if prec == "split" else S.PLAIN
    rng = np.random.default_rng(n)
    # at most an eighth of the large states moves, so the merge handles them
    p, *state = _free(n, rng, "morton" if n % 2 else "rowmajor", periodic=int(n % 3 == 0 and prec == "plain"),
                      speed=0.25 if n < 8192 else 0.08)
    prm = S.params(**p)
    merged, a = _run(S, prm, n, state, P, 1, 4)
    _, b = _run(S, prm, n, state, P, 0, 4)
    assert all(m == 1 for m, _ in merged), merged
    if n >= 511:
        assert max(c for _, c in merged) > n // 40
    for u, v in zip(a, b):
        _same(u, v)


@pytest.mark.parametrize("many", [40, 63, 64, 65, 300])
def test_many_movers_into_one_gap(many):
    """`many` particles of one cell move into one empty cell at once: merged up to
    64, sorted fully beyond, the same order either way."""
    import sphg as S
    rng = np.random.default_rng(many)
    h = 0.125
    x = np.concatenate([rng.uniform(0.26, 0.37, many), rng.uniform(0.8, 0.99, 20)])
    y = np.concatenate([rng.uniform(0.26, 0.37, many), rng.uniform(0.8, 0.99, 20)])
    x, y = (v.astype(np.float32).astype(np.float64) for v in (x, y))
    vx = np.concatenate([np.full(many, h / 1e-3), np.zeros(20)])  # one cell an iteration
    z = np.zeros(len(x))
    prm = S.params(order="morton", h=h, dt=1e-3, k=0.0, mu=0.0, gx=0.0, gy=0.0, lo=(0, 0), hi=(1, 1))
    merged, a = _run(S, prm, len(x), (x, y, vx, z), S.SPLIT, 1, 3)
    _, b = _run(S, prm, len(x), (x, y, vx, z), S.SPLIT, 0, 3)
    assert [m for m, _ in merged] == [1 if many <= 63 else 0] * 3 or many == 64, merged
    for u, v in zip(a, b):
        _same(u, v)


def test_batched_merge_equals_full_sort():
    """Instances of odd sizes, one of a single particle, one that moves as a whole."""
    import sphg as S
    rng = np.random.default_rng(5)
    inst = [_free(n, rng, o, speed=s) for n, o, s in ((700, "morton", 0.3), (1, "rowmajor", 0.0), (513, "rowmajor", 0.3),
                                                      (2048, "morton", 0.0), (333, "morton", 1.0))]
    prms, counts = [S.params(**i[0]) for i in inst], [len(i[1]) for i in inst]
    state = [np.concatenate([i[k] for i in inst]) for k in (1, 2, 3, 4)]
    merged, a = _run(S, prms, counts, state, S.SPLIT, 1, 4)
    _, b = _run(S, prms, counts, state, S.SPLIT, 0, 4)
    assert all(m == 1 for m, _ in merged), merged
    for u, v in zip(a, b):
        _same(u, v)
