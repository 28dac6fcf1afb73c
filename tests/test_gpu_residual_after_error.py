"""FvmFieldReduceSum after a run that ended in an error: the sum of the error
field as it is, not the partial sums that an earlier run left (or memory that
no run has written)."""
import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.euler import EulerCase
from graphite_b200.nsi import NSICase

pytestmark = pytest.mark.gpu
P, T = 1.0, 1.0 / 1.4
WING = [("farfield", "farfield", 0.6, 0.0, 0.05, P, T), ("slip", "sides"), ("slip", "wing")]
CYLINDER = [("wall", "cylinder"), ("inletoutlet", "farfield", 1.0, 0.0, 0.05, 0.0), ("slip", "sides")]


def check_residual(c, run):
    """An error field of known values, a run whose first wait gives up, then the residual."""
    lib = capi.load()
    run()
    n = int(lib.cuMeshGetnCells(c.mesh))
    size = int(lib.cuMeshGetVarSize(c.mesh))
    capi.set_field_values(c.error, np.random.default_rng(3).uniform(1e3, 2e3, size))
    capi.check(lib.gbVarCpuToGpu(c.mesh, c.error), "gbVarCpuToGpu")
    capi.check(lib.gbMeshSetLoopWaitLimit(c.mesh, 1), "gbMeshSetLoopWaitLimit")
    with pytest.raises(capi.GraphiteError, match="gave up"):
        run()
    got = c.residual()
    lib.VarGpuToCpu(c.error)
    want = float(np.sum(capi.field_values(c.error)[:n].astype(np.float64)))
    assert want > 0 and abs(got - want) <= 2e-7 * want       # a float32 of the float64 sum


@pytest.mark.parametrize("density", [False, True])
def test_euler_residual_after_a_wait_that_gave_up(tmp_path, density):
    p = str(tmp_path / "m.su2")
    meshgen.airfoil_2d_prisms(66, 69).write_su2(p)
    with EulerCase(p) as c:
        c.init((0.6, 0.0, 0.05), P, T)
        c.run(WING, 0.5, 20)          # the partial sums of a plain run; the density run needs twice their number
        check_residual(c, lambda: c.run_density(WING, 0.5, 20) if density else c.run(WING, 0.5, 20))


def test_nsi_residual_after_a_wait_that_gave_up(tmp_path):
    p = str(tmp_path / "m.su2")
    meshgen.cylinder_ogrid(48, 23, ratio=1.1, r_far=10.0).write_su2(p)
    c = NSICase(p)
    c.init((1.0, 0.0, 0.05), 0.0)
    check_residual(c, lambda: c.run(CYLINDER, 0.5, 20))
    c.close()
