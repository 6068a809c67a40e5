"""Neighbour lists assembled in one launch, at the ends of its 128-particle
blocks and with lists longer than it keeps in shared memory (32), against the
oracle: offsets, entries in stencil order, and their ascending delta code; twice
and across sizes of a handle's life, since counters and buffers are kept."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["plain", "split"])
@pytest.mark.parametrize("wide", [1.3, 4.2])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 4127])
def test_lists_at_block_edges(n, wide, prec):
    import oracle as O
    import sphg as S
    rng = np.random.default_rng(n)
    side = int(np.ceil(np.sqrt(n)))
    k = rng.permutation(side * side)[:n]
    x, y = (((k % side) + 0.5) / side, ((k // side) + 0.5) / side)
    x, y = (v + rng.uniform(-0.2, 0.2, n) / side for v in (x, y))
    x, y = (v.astype(np.float32).astype(np.float64) for v in (x, y))
    kw = dict(order="morton", h=wide / side, lo=(0, 0), hi=(1, 1))
    sim = S.Sim(S.params(**kw), n, S.options(precision=S.SPLIT if prec == "split" else S.PLAIN))
    z = np.zeros(n)
    for turn in range(2):
        sim.upload(x, y, z, z)
        sim.preloop()
        g = sim.download()
        keys = sim.debug(S.DBG_KEYS)
        p = O.params(**kw)
        _, _, sk, s, e = O.find_neighbors(p, g["x"], g["y"])
        assert (sk == keys).all()
        want_offs, want_idx = O.neighbor_lists(p, g["x"], g["y"], sk, s, e)
        offs, idx = sim.neighbor_lists()
        assert np.array_equal(offs, want_offs) and np.array_equal(idx, want_idx)
        if wide > 2 and n > 4000:
            assert np.diff(offs).max() > 32
        offs2, enc = sim.neighbor_lists_encoded()
        assert np.array_equal(offs2, offs)
        code = np.concatenate([np.concatenate([l[:1], np.diff(l) - 1]) for l in
                               (np.sort(idx[a:b]) for a, b in zip(offs[:-1], offs[1:]))])
        assert np.array_equal(enc, code)
        x, y = x[::-1].copy(), y[::-1].copy()
    sim.close()
