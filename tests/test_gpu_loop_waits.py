"""The bounded waits of the persistent loops, made to run out without a fault:
with a limit of one poll a wait whose data is not there yet gives up, the
kernel ends, the call returns an error, and the next call (default limit) gives
bit for bit what a mesh or batch that never failed gives.  Each launch shape of
each loop: workers, the block that sums the residual, its density part."""
import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.batch import EulerBatch
from graphite_b200.euler import EulerCase
from graphite_b200.nsi import NSICase

pytestmark = pytest.mark.gpu
P, T = 1.0, 1.0 / 1.4
WING = [("farfield", "farfield", 0.6, 0.0, 0.05, P, T), ("slip", "sides"), ("slip", "wing")]
CYLINDER = [("wall", "cylinder"), ("inletoutlet", "farfield", 1.0, 0.0, 0.05, 0.0), ("slip", "sides")]


def write(tmp_path, mesh):
    p = str(tmp_path / "m.su2")
    mesh.write_su2(p)
    return p


def same(a, b):
    return all(np.array_equal(np.asarray(x), np.asarray(y)) for x, y in zip(a, b))


# cells per block up to 256; one face at a time; face normals in global memory
@pytest.mark.parametrize("shape", [(66, 69), (300, 140), (440, 168)])
@pytest.mark.parametrize("density", [False, True])
def test_euler_loop_gives_up_and_recovers(tmp_path, shape, density):
    path = write(tmp_path, meshgen.airfoil_2d_prisms(*shape))
    lib = capi.load()

    def run(c):
        c.init((0.6, 0.0, 0.05), P, T)
        return c.run_density(WING, 0.5, 40) if density else [c.run(WING, 0.5, 40)]

    with EulerCase(path) as c:
        want = [*run(c), *c.fields()]
    with EulerCase(path) as c:
        for _ in range(2):
            capi.check(lib.gbMeshSetLoopWaitLimit(c.mesh, 1), "gbMeshSetLoopWaitLimit")
            with pytest.raises(capi.GraphiteError, match="gave up"):
                run(c)
            capi.check(lib.gbMeshSetLoopWaitLimit(c.mesh, 0), "gbMeshSetLoopWaitLimit")
            assert same(want, [*run(c), *c.fields()])


@pytest.mark.parametrize("shape", [(48, 23), (396, 250)])
@pytest.mark.parametrize("limited", [False, True])
def test_nsi_loop_gives_up_and_recovers(tmp_path, shape, limited):
    path = write(tmp_path, meshgen.cylinder_ogrid(*shape, ratio=1.1 if shape[0] < 100 else 1.02, r_far=10.0))
    lib = capi.load()

    def run(c):
        c.init((1.0, 0.0, 0.05), 0.0)
        return [c.run(CYLINDER, 0.5, 40)]

    NSICase.set_constants(1.0, 0.03, 2.0, True, limited)
    try:
        c = NSICase(path)
        want = [*run(c), *c.fields()]
        c.close()
        c = NSICase(path)
        for _ in range(2):
            capi.check(lib.gbMeshSetLoopWaitLimit(c.mesh, 1), "gbMeshSetLoopWaitLimit")
            with pytest.raises(capi.GraphiteError, match="gave up"):
                run(c)
            capi.check(lib.gbMeshSetLoopWaitLimit(c.mesh, 0), "gbMeshSetLoopWaitLimit")
            assert same(want, [*run(c), *c.fields()])
        c.close()
    finally:
        NSICase.set_constants()


@pytest.mark.parametrize("shape,n", [((64, 31), 3), ((244, 100), 2)])
def test_batch_loop_gives_up_and_recovers(tmp_path, shape, n):
    lib = capi.load()
    case = EulerCase(write(tmp_path, meshgen.airfoil_2d_prisms(*shape)))

    def run(b):
        for i in range(n):
            b.init_uniform(i, (0.4 + 0.1 * i, 0.0, 0.02), P, T)
        out = list(b.run(0.5, 40, history=True))
        return out + [x for i in range(n) for x in b.get_state(i)]

    spec = [(0, WING) for _ in range(n)]
    with EulerBatch([case], spec) as b:
        want = run(b)
    with EulerBatch([case], spec) as b:
        for _ in range(2):
            capi.check(lib.gbBatchSetLoopWaitLimit(b.h, 1), "gbBatchSetLoopWaitLimit")
            with pytest.raises(capi.GraphiteError, match="gave up"):
                run(b)
            capi.check(lib.gbBatchSetLoopWaitLimit(b.h, 0), "gbBatchSetLoopWaitLimit")
            assert same(want, run(b))
    case.close()


def test_limits_refuse_null():
    lib = capi.load()
    assert lib.gbMeshSetLoopWaitLimit(None, 1) == 1 and "null mesh" in capi.last_error()
    assert lib.gbBatchSetLoopWaitLimit(None, 1) == 1 and "null batch" in capi.last_error()
