"""Many handles stepped in turn on the legacy default stream, where a graph's launch
waits on the streams inside every other handle's: the same bits, and the time, of
handles whose kernels are launched without graphs."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MANY = 64


def _handles(S, prm, state, graph):
    sims = []
    for _ in range(MANY):
        s = S.Sim(prm, len(state[0]), S.options(precision=S.SPLIT, use_graph=graph))
        s.upload(*state)
        s.preloop()
        sims.append(s)
    return sims


@pytest.mark.parametrize("k", [1, 10])
def test_many_handles_in_turn(k):
    """At most one and a half times the time without graphs (measured: the same)."""
    import sphg as S
    import workloads as W
    nx = 130  # above the sizes whose iterations need no graph
    dx = 0.4 / nx
    p, *state = W.dam_break(nx, nx, dx, seed=1, box=(2.5 * nx * dx, 1.25 * nx * dx))
    prm = S.params(**p)
    best, out = [], []
    for graph in (1, 0):
        sims = _handles(S, prm, state, graph)
        t = []
        for _ in range(4):
            a = time.perf_counter()
            for _ in range(max(1, 4 // k)):
                for s in sims:
                    s.step(k)
            sims[-1].diagnostics()  # waits
            t.append(time.perf_counter() - a)
        best.append(min(t))
        out.append([sims[q].download() for q in (0, MANY - 1)])
        for s in sims:
            s.close()
    for a, b in zip(*out):
        for f in a:
            assert np.array_equal(a[f], b[f]), f
    assert best[0] <= 1.5 * best[1], best
