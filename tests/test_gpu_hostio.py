"""Downloads written by the device straight into the caller's arrays: every
alignment of the arrays inside a 128-byte line, sizes around a warp and a block,
pages the host has never touched, nothing written beside the arrays -- the values
of the staging path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("x", "y", "vx", "vy", "rho", "fx", "fy")


@pytest.mark.parametrize("prec", ["plain", "split"])
@pytest.mark.parametrize("n", [1, 31, 33, 225, 4097])
def test_download_alignments(n, prec):
    import sphg as S
    rng = np.random.default_rng(n)
    x, y, vx, vy = rng.uniform(0, 1, (4, n))
    sim = S.Sim(S.params(order="rowmajor", h=0.1, lo=(0, 0), hi=(1, 1)), n,
                S.options(precision=S.SPLIT if prec == "split" else S.PLAIN))
    sim.upload(x, y, vx, vy)
    sim.preloop()
    sim.set_host_access(0)
    want = sim.download()
    sim.set_host_access(1)
    for shift in range(0, 17, 3):
        raw = {k: np.full(n + 64, -7.0) for k in NAMES}
        raw["ids"] = np.full(n + 64, -7, np.int32)
        at = {k: (shift + 5 * q) % 33 for q, k in enumerate(raw)}  # each array its own offset
        sim.download(out={k: raw[k][at[k]:at[k] + n] for k in raw})
        for k in raw:
            assert np.array_equal(raw[k][at[k]:at[k] + n], want[k]), (k, shift)
            assert (raw[k][:at[k]] == -7).all() and (raw[k][at[k] + n:] == -7).all(), (k, shift)
    sim.close()


def test_download_into_untouched_pages():
    import sphg as S
    n = 300007
    rng = np.random.default_rng(1)
    x, y, vx, vy = rng.uniform(0, 1, (4, n))
    sim = S.Sim(S.params(order="morton", h=0.003, lo=(0, 0), hi=(1, 1)), n)
    sim.upload(x, y, vx, vy)
    sim.preloop()
    sim.step(3)
    fresh = sim.download()  # np.empty: pages never written
    again = sim.download(out={k: v.copy() for k, v in fresh.items()})
    sim.set_host_access(0)
    want = sim.download()
    for k in want:
        assert np.array_equal(fresh[k], want[k]) and np.array_equal(again[k], want[k]), k
    sim.close()


@pytest.mark.parametrize("bad", [0, 1, 4096])
def test_upload_reports_the_first_bad_particle_and_recovers(bad):
    import sphg as S
    n = 4097
    rng = np.random.default_rng(2)
    x, y, vx, vy = rng.uniform(0, 1, (4, n))
    sim = S.Sim(S.params(order="morton", h=0.05, lo=(0, 0), hi=(1, 1)), n)
    for arrays in ((x, y, vx, vy), (x, y, vx, vy)):  # twice: the report is armed again
        broken = [a.copy() for a in arrays]
        broken[1][bad] = np.nan
        broken[2][n - 1] = np.inf
        with pytest.raises(S.SphgError) as e:
            sim.upload(*broken)
        assert e.value.status == S.NONFINITE and "particle %d" % bad in str(e.value)
        sim.upload(*arrays)
    sim.preloop()
    assert sim.diagnostics()[0, 5] == 0
    sim.close()


def test_served_positions_round_once():
    """A served position near a tie of its FP32 offset: c cs is taken off x - lo in
    one rounding, and added back to lo in one."""
    from fractions import Fraction
    import sphg as S
    lo, cs, m = (-0.3, 0.7), 0.01, 40
    rng = np.random.default_rng(5)
    c = 3 * np.arange(m) + 1  # particles three cells apart: no pair, no force, nothing moves
    xs, want = [], []
    for axis in (0, 1):
        o = rng.uniform(0.2 * cs, 0.8 * cs, m).astype(np.float32)
        tie = (o.astype(np.float64) + np.nextafter(o, np.float32(1)).astype(np.float64)) / 2
        x = np.array([float(Fraction(lo[axis]) + int(k) * Fraction(cs) + Fraction(t)) for k, t in zip(c, tie)])
        xs.append(x)
        off = [np.float32(float(Fraction(v - lo[axis]) - int(k) * Fraction(cs))) for v, k in zip(x, c)]
        want.append(np.array([float(Fraction(lo[axis]) + int(k) * Fraction(cs)) + float(f) for k, f in zip(c, off)]))
    x, y = (a.ravel() for a in np.meshgrid(xs[0], xs[1], indexing="ij"))
    wx, wy = (a.ravel() for a in np.meshgrid(want[0], want[1], indexing="ij"))
    prm = S.params(order="morton", h=cs, lo=lo, hi=(lo[0] + 1.27, lo[1] + 1.27), gx=0.0, gy=0.0, dt=1e-6)
    srv = S.Server(2e8, max_instances=4, opts=S.options(precision=S.SPLIT))
    rid = srv.submit(prm, x, y, np.zeros_like(x), np.zeros_like(x), 1)
    while srv.tick()[0]:
        pass
    r = srv.result(rid)
    assert np.array_equal(r["x"], wx[r["ids"]]) and np.array_equal(r["y"], wy[r["ids"]])
    srv.close()
