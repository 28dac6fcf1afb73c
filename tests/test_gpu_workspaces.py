"""Calls that share a kept workspace give each caller its own answer: states of
instances of unequal meshes one after another, in both directions, and several
threads on streams of their own."""
import threading

import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.batch import EulerBatch
from graphite_b200.euler import EulerCase

pytestmark = pytest.mark.gpu
P, T = 1.0, 1.0 / 1.4


def bcs(m):
    return [("farfield", "farfield", m, 0.0, 0.02, P, T), ("slip", "sides"), ("slip", "wing")]


@pytest.fixture(scope="module")
def cases(tmp_path_factory):
    d = tmp_path_factory.mktemp("ws")
    out = []
    for k, (na, nr) in enumerate(((16, 5), (40, 21), (24, 9))):
        p = str(d / f"{k}.su2")
        meshgen.airfoil_2d_prisms(na, nr).write_su2(p)
        out.append(EulerCase(p))
    return out


def test_states_and_forces_of_unequal_instances(cases):
    """Small after large and large after small; a second run replays the kept
    graph, one with another CFL does not."""
    mach = [0.4, 0.5, 0.6, 0.7]
    with EulerBatch(cases, [(0, bcs(0.4)), (1, bcs(0.5)), (2, bcs(0.6)), (0, bcs(0.7))]) as b:
        def solve(cfl, n):
            for i in range(4):
                b.init_uniform(i, (mach[i], 0.0, 0.02), P, T)
            hist = b.run(cfl, n, history=True)[4]
            return hist, [b.get_state(i) for i in (1, 0, 2, 3)], [b.wall_force(i, "wing") for i in (3, 1, 0, 2)]

        first, other, again = solve(0.5, 12), solve(0.3, 12), solve(0.5, 12)
        assert np.array_equal(first[0], again[0]) and not np.array_equal(first[0], other[0])
        for x, y in zip(first[1], again[1]):
            assert all(np.array_equal(p, q) for p, q in zip(x, y))
        assert all(np.array_equal(p, q) for p, q in zip(first[2], again[2]))
        longer = solve(0.5, 20)[0]               # a longer history than the one kept
        assert np.array_equal(longer[:, :12], first[0])
        for k, i in enumerate((1, 0, 2, 3)):     # states go back in and come out as they were
            b.set_state(i, *first[1][k])
        for k, i in enumerate((1, 0, 2, 3)):
            assert all(np.array_equal(p, q) for p, q in zip(first[1][k], b.get_state(i)))
        # and each instance is a plain solve of it
        for k, (c, m, order) in enumerate(((0, 0.4, 1), (1, 0.5, 0), (2, 0.6, 2))):
            cases[c].init((m, 0.0, 0.02), P, T)
            cases[c].run(bcs(m), 0.5, 12)
            for x, y in zip(cases[c].fields(), first[1][order]):
                assert np.array_equal(x, y)
            assert np.array_equal(cases[c].wall_force("wing"), first[2][(2, 1, 3)[k]])


def test_threads_take_turns(cases):
    import torch
    want = {}
    for c in range(3):
        cases[c].init((0.5, 0.0, 0.02), P, T)
        cases[c].run(bcs(0.5), 0.5, 8)
        want[c] = [cases[c].wall_force(r) for r in ("wing", "farfield")]
    wrong = []

    def worker(c, region, k):
        s = torch.cuda.Stream()
        capi.load().gbSetStream(s.cuda_stream)
        for _ in range(50):
            if not np.array_equal(cases[c].wall_force(region), want[c][k]):
                wrong.append((c, region))

    torch.cuda.synchronize()
    threads = [threading.Thread(target=worker, args=(c, r, k)) for c in range(3) for k, r in
               enumerate(("wing", "farfield"))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong
