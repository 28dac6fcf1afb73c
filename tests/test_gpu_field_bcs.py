"""Field conditions are recorded and applied by the next call that uses the
field: whichever call that is, it sees what applying each at once would give."""
import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.euler import EulerCase

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case(tmp_path_factory):
    p = str(tmp_path_factory.mktemp("bc") / "m.su2")
    meshgen.channel_bump(7, 5, 3, cells="mixed").write_su2(p)
    with EulerCase(p) as c:
        yield c


def field(c, comps, values):
    f = c.lib.FvmFieldNew(4 * comps, c.n_cells + c.n_ghosts, b"f", 1)
    capi.set_field_values(f, values)
    capi.check(c.lib.gbVarCpuToGpu(c.mesh, f), "gbVarCpuToGpu")
    return f


@pytest.mark.parametrize("comps", [1, 3])
@pytest.mark.parametrize("reader", ["download", "gradient", "operand", "velocity", "axpy", "upload", "init"])
def test_pending_conditions_reach_every_reader(case, comps, reader):
    c, lib, mesh = case, case.lib, case.mesh
    n, N = c.n_cells + c.n_ghosts, c.n_cells
    rng = np.random.default_rng(3)
    shape = (n,) if comps == 1 else (n, 3)
    vals = rng.standard_normal(shape).astype(np.float32)
    cfs, cc = capi.mesh_array(mesh, "cell_faces_starts"), capi.mesh_array(mesh, "cell_connects")
    gid, gs = capi.mesh_array(mesh, "ghost_cell_ids"), capi.mesh_array(mesh, "ghost_cell_starts")

    def ghosts(region):
        r = lib.cuMeshGetRegionId(mesh, region.encode())
        return r, gid[gs[r]:gs[r + 1]]

    want = vals.copy()
    f = field(c, comps, vals)
    for region, kind in (("lower", "fixed"), ("inlet", "zero"), ("lower", "zero"), ("sides", "fixed")):
        r, g = ghosts(region)
        if kind == "fixed":
            capi.check(lib.gbFieldBcFixed(mesh, f, capi.vec((7.0, -1.0, 2.0)), r), "gbFieldBcFixed")
            want[g] = 7.0 if comps == 1 else np.float32([7.0, -1.0, 2.0])
        else:
            capi.check(lib.gbFieldBcZeroGrad(mesh, f, r), "gbFieldBcZeroGrad")
            want[g] = vals[cc[cfs[g]]]

    ref = field(c, comps, want)                   # the same values without conditions
    others = [f, ref]

    def new(k):
        o = field(c, k, np.zeros((n,) if k == 1 else (n, 3), np.float32))
        others.append(o)
        return o

    def values(x):
        lib.VarAllGpuToCpu(x)
        return [capi.field_values(x)] + list(capi.field_gradients(x))

    def terms(x):
        out = new(comps)
        arr = (capi.gbFvmTerm * 1)()
        if reader == "velocity":
            u = field(c, comps, vals)
            others.append(u)
            arr[0] = capi.gbFvmTerm(9 if comps == 1 else 10, 1.0, u, x if comps == 3 else new(3), capi.vec((1, 0, 0)))
        else:
            arr[0] = capi.gbFvmTerm(7 if comps == 1 else 10, 1.0, x, None if comps == 1 else new(3), capi.vec((1, 2, 3)))
        capi.check(lib.gbFvmApplyTerms(mesh, 1, arr, out), "gbFvmApplyTerms")
        return values(out)

    if reader == "download":
        got, exp = values(f), values(ref)
    elif reader == "gradient":
        for x in (f, ref):
            capi.check(lib.gbFvmGradient(mesh, x), "gbFvmGradient")
        got, exp = values(f), values(ref)
    elif reader in ("operand", "velocity"):
        got, exp = terms(f), terms(ref)
    elif reader == "axpy":
        y = new(comps)
        capi.check(lib.gbFieldAxpy(mesh, f, 0.5, y), "gbFieldAxpy")
        got, exp = values(f), values(ref)
    elif reader == "upload":                      # an upload after the conditions wins
        capi.set_field_values(f, vals)
        capi.check(lib.gbVarCpuToGpu(mesh, f), "gbVarCpuToGpu")
        got, exp = values(f)[:1], [vals]
    else:
        capi.check(lib.gbFieldInit(mesh, f, capi.vec((2.0, 2.0, 2.0))), "gbFieldInit")
        got, exp = values(f)[:1], [np.full(shape, 2.0, np.float32)]
    for a, b in zip(got, exp):
        assert np.array_equal(a, b)
    if reader == "download":
        assert np.array_equal(got[0], want)
    assert N < n
    for x in others:
        lib.FvmFieldFree(x)
