"""A persistent launch that is refused (as the driver refuses a cooperative launch
whose blocks do not fit on the GPU together) is no error: the run replays its
graphs with the same results, and the next run is persistent again.  The
refusal is made on the host: the launch is not made and its error code returned."""
import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.batch import EulerBatch
from graphite_b200.euler import EulerCase
from graphite_b200.nsi import NSICase

pytestmark = pytest.mark.gpu
P, T = 1.0, 1.0 / 1.4
WING = [("farfield", "farfield", 0.6, 0.0, 0.05, P, T), ("slip", "sides"), ("slip", "wing")]
DUCT = [("farfield", "inlet", 0.5, 0.0, 0.0, P, T), ("slip", "lower"), ("farfield", "outlet", 0.5, 0.0, 0.0, P, T),
        ("slip", "sides"), ("slip", "upper")]
CYLINDER = [("wall", "cylinder"), ("inletoutlet", "farfield", 1.0, 0.0, 0.05, 0.0), ("slip", "sides")]


def same(a, b):
    return [k for k, (x, y) in enumerate(zip(a, b)) if not np.array_equal(np.asarray(x), np.asarray(y))]


def three_runs(inject, run):
    """Persistent, refused, persistent: outputs, and the launches of each."""
    lib = capi.load()
    outs, launches = [], []
    for k in range(3):
        if k == 1:
            inject()
        n0 = lib.gbKernelLaunchCount()
        outs.append(run())
        launches.append(lib.gbKernelLaunchCount() - n0)
    assert launches[2] <= launches[0] < 20 < 100 < launches[1]       # the first makes what the loop keeps
    assert same(outs[0], outs[1]) == [] and same(outs[0], outs[2]) == []


# conditions inside the gradient pass, and by a ghost kernel
@pytest.mark.parametrize("make,bcs", [(lambda: meshgen.airfoil_2d_prisms(66, 69), WING),
                                      (lambda: meshgen.channel_bump(24, 15, 6, cells="tet"), DUCT)])
def test_euler_refused_launch(tmp_path, make, bcs):
    p = str(tmp_path / "m.su2")
    make().write_su2(p)
    lib = capi.load()
    with EulerCase(p) as c:
        def run():
            c.init(bcs[0][2:5], P, T)
            h = c.run_density(bcs, 0.5, 60, check_every=20)
            out = [*h, *c.fields(), c.error_values(), np.float64(c.residual())]
            c.step(0.5)
            return out + list(c.fields())

        three_runs(lambda: capi.check(lib.gbMeshInjectLoopRefusal(c.mesh), "inject"), run)


def test_nsi_refused_launch(tmp_path):
    p = str(tmp_path / "m.su2")
    meshgen.cylinder_ogrid(48, 23, ratio=1.1, r_far=10.0).write_su2(p)
    lib = capi.load()
    c = NSICase(p)

    def run():
        c.init((1.0, 0.0, 0.05), 0.0)
        out = [c.run(CYLINDER, 0.5, 60, check_every=20), *c.fields(), np.float64(c.residual())]
        c.step(0.5)
        return out + list(c.fields())

    three_runs(lambda: capi.check(lib.gbMeshInjectLoopRefusal(c.mesh), "inject"), run)
    c.close()


def test_batch_refused_launch(tmp_path):
    p = str(tmp_path / "m.su2")
    meshgen.airfoil_2d_prisms(64, 31).write_su2(p)
    lib = capi.load()
    case = EulerCase(p)
    with EulerBatch([case], [(0, WING)] * 3) as b:
        def run():
            for i in range(3):
                b.init_uniform(i, (0.4 + 0.1 * i, 0.0, 0.02), P, T)
            return list(b.run(0.5, 60, check_every=20, history=True)) + [x for i in range(3) for x in b.get_state(i)]

        run()                                     # what is made once
        three_runs(lambda: capi.check(lib.gbBatchInjectLoopRefusal(b.h), "inject"), run)
    case.close()


def test_autotune_with_a_refused_launch(tmp_path):
    """The trial that would have run as the loop is timed as kernels; states stay as they were."""
    p = str(tmp_path / "m.su2")
    meshgen.airfoil_2d_prisms(62, 29).write_su2(p)
    lib = capi.load()
    case = EulerCase(p)
    with EulerBatch([case], [(0, WING)] * 2) as b:
        for i in range(2):
            b.init_uniform(i, (0.4 + 0.1 * i, 0.0, 0.02), P, T)
        before = [x for i in range(2) for x in b.get_state(i)]
        capi.check(lib.gbBatchInjectLoopRefusal(b.h), "inject")
        b.autotune(0.5, 5)
        assert same(before, [x for i in range(2) for x in b.get_state(i)]) == []
        done, its, rat, st = b.run(0.5, 20)
        assert done == 20 and its.tolist() == [20, 20]
    case.close()
