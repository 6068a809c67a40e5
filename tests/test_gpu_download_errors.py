"""A download that reports a state that is not valid writes nothing into the
caller's arrays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("x", "y", "vx", "vy", "rho", "fx", "fy")


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_failed_download_leaves_the_arrays(mode):
    """Isolated particles driven together until their lists outgrow the buffer that
    the pre-loop sized (SPHG_CAPACITY)."""
    import sphg as S
    h = 0.005
    g = (np.arange(64) - 31.5) * 2 * h + 0.5
    x, y = [a.ravel().astype(np.float32).astype(np.float64) for a in np.meshgrid(g, g, indexing="xy")]
    sim = S.Sim(S.params(order="morton", h=h, dt=1e-4, lo=(0, 0), hi=(1, 1), gy=0.0), len(x),
                S.options(compute="lists"))
    sim.set_host_access(mode)
    sim.upload(x, y, -300.0 * (x - 0.5), -300.0 * (y - 0.5))
    sim.preloop()
    good = sim.download()
    sim.step(35)
    out = {k: v.copy() for k, v in good.items()}
    for forces in (True, False):
        with pytest.raises(S.SphgError) as e:
            sim.download(forces=forces, out=out)
        assert e.value.status == S.CAPACITY
        for k in NAMES + (("ids",) if mode else ()):
            assert np.array_equal(out[k], good[k]), k
    sim.close()
