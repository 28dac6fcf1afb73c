"""What a run that ends in a residual that is not finite leaves behind -- states,
ghosts, error field, face states or gradients -- is what the per-call loop
leaves when it stops at that iteration: persistent launches and replayed
graphs (check_every below 4), conditions applied inside the gradient pass or by
a ghost kernel, a bad first state and one that overflows later."""
import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.euler import EulerCase
from graphite_b200.nsi import NSICase

pytestmark = pytest.mark.gpu
P, T = 1.0, 1.0 / 1.4
DUCT = [("farfield", "inlet", 0.5, 0.0, 0.0, P, T), ("slip", "lower"), ("farfield", "outlet", 0.5, 0.0, 0.0, P, T),
        ("slip", "sides"), ("slip", "upper")]
AIRFOIL = [("farfield", "farfield", 0.6, 0.0, 0.05, P, T), ("slip", "sides"), ("slip", "wing")]
NSI_DUCT = [("wall", "lower"), ("slip", "upper"), ("slip", "sides"), ("inletoutlet", "inlet", 1.0, 0.0, 0.05, 0.0),
            ("inletoutlet", "outlet", 1.0, 0.0, 0.05, 0.0)]
CYLINDER = [("wall", "cylinder"), ("inletoutlet", "farfield", 1.0, 0.0, 0.05, 0.0), ("slip", "sides")]


def loop(c, bcs, cfl, form):
    """Iterates until the residual is not finite: call by call, or as one run."""
    if form == "percall":
        for it in range(200):
            c.apply_bcs(bcs)
            c.prepare()
            c.step(cfl)
            c.lib.VarGpuToCpu(c.error)           # (FvmFieldReduceSum's float32 overflows before the sum does)
            if not np.all(np.isfinite(capi.field_values(c.error)[:c.n_cells])):
                return it + 1
        raise AssertionError("did not diverge")
    with pytest.raises(capi.GraphiteError, match="not finite"):
        c.run(bcs, cfl, 200, check_every=100 if form == "persistent" else 2)
    return None


def same(a, b):
    return [k for k, (x, y) in enumerate(zip(a, b)) if not np.array_equal(x, y, equal_nan=True)]


EULER = {
    "airfoil_9108": (lambda: meshgen.airfoil_2d_prisms(66, 69), AIRFOIL),
    "airfoil_84000": (lambda: meshgen.airfoil_2d_prisms(300, 140), AIRFOIL),
    "tet_12960": (lambda: meshgen.channel_bump(24, 15, 6, cells="tet"), DUCT),
}


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("name", list(EULER))
def test_euler_diverged_run(tmp_path, name, bad):
    make, bcs = EULER[name]
    p = str(tmp_path / "m.su2")
    make().write_su2(p)
    out = {}
    for form in ("percall", "graphs", "persistent"):
        with EulerCase(p) as c:
            c.init(bcs[0][2:5], P, T)
            c.run(bcs, 0.5, 9)
            q = [x.copy() for x in c.fields()]
            q[0][c.n_cells // 2] = bad
            c.set_state(*q)
            loop(c, bcs, 0.5, form)
            got = [*c.fields(), c.error_values()]
            c.step(0.5)                          # from the face states of the last gradient pass
            out[form] = got + list(c.fields())
    assert np.isfinite(out["percall"][0]).mean() > 0.9
    assert same(out["percall"], out["graphs"]) == []
    assert same(out["percall"], out["persistent"]) == []


NSI = {
    "cylinder_1104": (lambda: meshgen.cylinder_ogrid(48, 23, ratio=1.1, r_far=10.0), CYLINDER),
    "cylinder_99000": (lambda: meshgen.cylinder_ogrid(396, 250), CYLINDER),
    "tet_6210": (lambda: meshgen.channel_bump(23, 9, 5, cells="tet"), NSI_DUCT),
}


@pytest.mark.parametrize("limited", [False, True])
@pytest.mark.parametrize("name", list(NSI))
def test_nsi_diverged_run(tmp_path, name, limited):
    make, bcs = NSI[name]
    p = str(tmp_path / "m.su2")
    make().write_su2(p)
    out = {}
    NSICase.set_constants(1.0, 0.03, 2.0, True, limited)
    try:
        for form in ("percall", "graphs", "persistent"):
            c = NSICase(p)
            c.init((1.0, 0.0, 0.05), 0.0)
            c.run(bcs, 0.5, 9)
            u, q = (x.copy() for x in c.fields())
            q[c.n_cells // 3] = np.nan         # an interior cell
            c.set_state(u, q)
            loop(c, bcs, 0.5, form)
            got = list(c.fields())
            for f in (c.pressure, c.velocity, c.error):
                c.lib.VarAllGpuToCpu(f)
                got += [capi.field_values(f), *capi.field_gradients(f)]
            c.step(0.5)                          # from the gradients of the last pass
            out[form] = got + list(c.fields())
            c.close()
    finally:
        NSICase.set_constants()
    assert np.isfinite(out["percall"][0]).mean() > 0.8
    assert same(out["percall"], out["graphs"]) == []
    assert same(out["percall"], out["persistent"]) == []


def test_euler_run_that_diverges_later(tmp_path):
    """A step far too large: the state overflows after some iterations, inside a launch."""
    p = str(tmp_path / "m.su2")
    meshgen.airfoil_2d_prisms(66, 69).write_su2(p)
    out, ran = {}, None
    for form in ("percall", "graphs", "persistent"):
        with EulerCase(p) as c:
            c.init(AIRFOIL[0][2:5], P, T)
            ran = loop(c, AIRFOIL, 40.0, form) or ran
            got = [*c.fields(), c.error_values()]
            c.step(0.5)
            out[form] = got + list(c.fields())
    assert ran > 4
    assert same(out["graphs"], out["persistent"]) == []
    assert same(out["percall"], out["graphs"]) == []
