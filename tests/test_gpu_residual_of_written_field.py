"""FvmFieldReduceSum of an error field that a step has written (with its block sums
beside it) and a generic call has overwritten since: the sum of what the field
holds now."""
import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.euler import EulerCase

pytestmark = pytest.mark.gpu
P, T = 1.0, 1.0 / 1.4
DUCT = [("farfield", "inlet", 0.5, 0.0, 0.0, P, T), ("slip", "lower"), ("farfield", "outlet", 0.5, 0.0, 0.0, P, T),
        ("slip", "sides"), ("slip", "upper")]


@pytest.mark.parametrize("how", ["init", "axpy", "terms"])
def test_sum_of_an_overwritten_error_field(tmp_path, how):
    p = str(tmp_path / "m.su2")
    meshgen.channel_bump(12, 7, 4, cells="mixed").write_su2(p)
    lib = capi.load()
    with EulerCase(p) as c:
        c.init(DUCT[0][2:5], P, T)
        for _ in range(3):
            c.iterate(DUCT, 0.5)
        size = int(lib.cuMeshGetVarSize(c.mesh))
        x = lib.FvmFieldNew(4, size, b"x", 1)
        capi.set_field_values(x, np.random.default_rng(2).uniform(1, 2, size))
        capi.check(lib.gbVarCpuToGpu(c.mesh, x), "gbVarCpuToGpu")
        if how == "init":
            capi.check(lib.gbFieldInit(c.mesh, c.error, capi.vec(2.5, 0, 0)), "gbFieldInit")
        elif how == "axpy":
            capi.check(lib.gbFieldAxpy(c.mesh, c.error, 100.0, x), "gbFieldAxpy")
        else:
            capi.check(lib.gbFvmGradient(c.mesh, x), "gbFvmGradient")
            t = (capi.gbFvmTerm * 1)(capi.gbFvmTerm(0, 1.0, x, None, capi.vec(1, 0.5, 0)))
            for op in range(9):                  # the first operator that makes a scalar of x and a constant velocity
                t[0].op = op
                if lib.gbFvmApplyTerms(c.mesh, 1, t, c.error) == 0:
                    break
            else:
                raise AssertionError("no operator applied")
        got = c.residual()
        v = c.error_values()[: c.n_cells].astype(np.float64)
        assert abs(got - v.sum()) <= 2e-7 * np.abs(v).sum()
        lib.FvmFieldFree(x)
