"""Time steps from the device maxima, and a changed time step taken into a graph
that is there already: the same bits as in one captured with it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [[1], [255], [257], [20503], [1, 700, 5000]])
def test_cfl_maxima(counts):
    import sphg as S
    rng = np.random.default_rng(len(counts) + counts[0])
    n = sum(counts)
    x, y = rng.uniform(0, 1, (2, n))
    vx, vy = rng.normal(0, 2, (2, n))
    kw = dict(order="morton", h=0.05, dt=1e-4, lo=(0, 0), hi=(1, 1))
    sim = S.Sim([S.params(**kw)] * len(counts) if len(counts) > 1 else S.params(**kw),
                counts if len(counts) > 1 else n)
    sim.upload(x, y, vx, vy)
    sim.preloop()
    for _ in range(2):  # the counters are left at zero
        got = sim.cfl_dt(0.3, 0.2)
        o = sim.download()
        at = 0
        for c, dt in zip(counts, got):
            v = np.sqrt(np.max(o["vx"][at:at + c] ** 2 + o["vy"][at:at + c] ** 2))
            a = np.sqrt(np.max(o["fx"][at:at + c] ** 2 + o["fy"][at:at + c] ** 2))
            assert dt == min(0.3 * 0.05 / (S.params().c0 + v), 0.2 * np.sqrt(0.05 / a))
            at += c
        sim.step(1)
    sim.close()


@pytest.mark.parametrize("opts", [dict(), dict(block_threads=128), dict(compute="lists"), dict(tile_bits=3),
                                  dict(fused=1), dict(use_graph=0), dict(resort=0)])
@pytest.mark.parametrize("headers", [False, True])
def test_changed_time_step(opts, headers):
    import sphg as S
    import workloads as W
    p, x, y, vx, vy = W.dam_break(60, 70, 0.005, seed=4, dt=1e-5)
    out = []
    for first in (1e-5, 2e-5):  # the graphs exist with the old time step / are made with the new one
        sim = S.Sim(S.params(**dict(p, dt=first)), len(x), S.options(precision=S.SPLIT, **opts))
        sim.upload(x, y, vx, vy)
        sim.preloop()
        if first == 1e-5:
            sim.step(2)
            sim.step_headers(2)
        sim.set_dt(2e-5)
        sim.upload(x, y, vx, vy)
        sim.preloop()
        for dt in (2e-5, 3e-5):
            sim.set_dt(dt)
            h = sim.step_headers(3) if headers else sim.step(3)
            sim.step(1)
        o = sim.download()
        if headers:
            o["headers"] = h
        out.append(o)
        sim.close()
    for f in out[0]:
        assert np.array_equal(out[0][f], out[1][f]), f


def test_time_step_of_a_captured_iteration():
    """An iteration in a caller's graph keeps the time step it was captured with
    and leaves the handle's own as it is."""
    import sphg as S
    import torch
    import workloads as W
    p, x, y, vx, vy = W.dam_break(60, 70, 0.005, seed=4, dt=1e-5)
    out = []
    for captured in (True, False):
        sim = S.Sim(S.params(**p), len(x), S.options(precision=S.SPLIT, use_graph=0))
        st = torch.cuda.Stream()
        ptr = st.cuda_stream
        sim.upload(x, y, vx, vy, stream=ptr)
        sim.preloop(stream=ptr)
        sim.set_dt(2e-5)
        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st):
                sim.step(1, stream=ptr)
        for dt in (1e-5, 3e-5):
            sim.set_dt(dt)
            sim.step(1, stream=ptr)
            if captured:
                with torch.cuda.stream(st):
                    g.replay()
            else:
                sim.set_dt(2e-5)
                sim.step(1, stream=ptr)
                sim.set_dt(dt)
            sim.step(2, stream=ptr)
        out.append(sim.download(stream=ptr))
        sim.close()
    for f in out[0]:
        assert np.array_equal(out[0][f], out[1][f]), f
