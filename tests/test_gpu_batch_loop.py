"""The batched persistent loop against the replayed kernels of an iteration,
bit for bit (launches of fewer than four iterations always run the kernels):
several meshes and element kinds at once, both launch shapes, instances that
stop in the middle of a launch, one that is not finite, one without a
condition on a region, one with a given residual scale."""
import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.batch import EulerBatch
from graphite_b200.euler import EulerCase

pytestmark = pytest.mark.gpu
P, T = 1.0, 1.0 / 1.4

WING = ["farfield", "sides", "wing"]
DUCT = ["inlet", "outlet", "lower", "upper", "sides"]
MESHES = {
    "airfoil_640": (lambda: meshgen.airfoil_2d_prisms(32, 10), WING),
    "airfoil_3968": (lambda: meshgen.airfoil_2d_prisms(64, 31), WING),
    "airfoil_48800": (lambda: meshgen.airfoil_2d_prisms(244, 100), WING),
    "tet": (lambda: meshgen.channel_bump(13, 7, 4, cells="tet"), DUCT),
    "mixed": (lambda: meshgen.channel_bump(11, 5, 3, cells="mixed"), DUCT),
    "hex_1": (lambda: meshgen.channel_bump(1, 1, 1, cells="hex"), DUCT),
}


def bcs(regions, m):
    far = ("farfield", "inlet", "outlet")
    return [("farfield", r, m, 0.0, 0.02, P, T) if r in far else ("slip", r) for r in regions]


@pytest.fixture(scope="module")
def case_of(tmp_path_factory):
    made = {}
    d = tmp_path_factory.mktemp("batch_loop")

    def get(name):
        if name not in made:
            p = str(d / f"{name}.su2")
            MESHES[name][0]().write_su2(p)
            made[name] = EulerCase(p)
        return made[name]

    return get


def solve(cases, names, inst, check_every, n, cfl=0.5, tolerance=0.0, bad=None, scale=None, skip=None):
    lib = capi.load()
    spec = []
    for k, (c, m) in enumerate(inst):
        b = bcs(MESHES[names[c]][1], m)
        spec.append((c, b[:1] + b[2:] if k == skip else b))
    with EulerBatch(cases, spec) as b:
        for i, (c, m) in enumerate(inst):
            b.init_uniform(i, (m, 0.0, 0.02), P, T)
        if bad is not None:
            q = [x.copy() for x in b.get_state(bad)]
            q[0][3] = np.nan
            b.set_state(bad, *q)
        if scale is not None:
            b.set_residual_scale(scale, 0.123)
        launches = lib.gbKernelLaunchCount()
        out = list(b.run(cfl, n, tolerance=tolerance, check_every=check_every, history=True))
        launches = lib.gbKernelLaunchCount() - launches
        out += list(b.run(cfl, 8, check_every=check_every))[1:]      # goes on from there
        for i in range(len(inst)):
            out += list(b.get_state(i))
        return out, launches


def same(a, b):
    return [k for k, (x, y) in enumerate(zip(a, b)) if not np.array_equal(np.asarray(x), np.asarray(y), equal_nan=True)]


SMALL = (["airfoil_640", "airfoil_3968", "tet", "mixed", "hex_1"],
         [(0, 0.4), (1, 0.5), (2, 0.3), (1, 0.7), (3, 0.35), (4, 0.3), (0, 0.6)])
LARGE = (["airfoil_48800", "airfoil_640"], [(0, 0.4), (1, 0.5), (0, 0.6)])


@pytest.mark.parametrize("transposed", [0, 1])
@pytest.mark.parametrize("which", ["small", "large"])
def test_batch_loop_is_bitwise_the_kernels(case_of, which, transposed):
    names, inst = SMALL if which == "small" else LARGE
    cases = [case_of(n) for n in names]
    lib = capi.load()
    lib.gbSetReferenceMomentumReconstruction(transposed)
    try:
        kernels, many = solve(cases, names, inst, 2, 40)
        loop, few = solve(cases, names, inst, 16, 40)
    finally:
        lib.gbSetReferenceMomentumReconstruction(1)
    assert few == 3 + 1 + len(names) and many == 40 * 3 + 1      # launches, last ghosts, one preparation per mesh
    assert same(kernels, loop) == []


@pytest.mark.parametrize("kw", [dict(tolerance=0.2), dict(bad=3), dict(scale=1, tolerance=0.1), dict(skip=2),
                                dict(tolerance=0.2, skip=0, bad=1)])
def test_batch_loop_stops_and_options(case_of, kw):
    names, inst = SMALL
    cases = [case_of(n) for n in names]
    kernels, _ = solve(cases, names, inst, 1, 60, **kw)
    loop, few = solve(cases, names, inst, 60, 60, **kw)
    assert few < 8
    kernels[0] = loop[0]         # iterations of the whole call: whole launches
    assert same(kernels, loop) == []
    if "bad" in kw:
        assert loop[3][kw["bad"]] == 3


@pytest.mark.parametrize("make,regions,n", [
    (lambda: meshgen.airfoil_2d_prisms(500, 148), WING, 2),           # 296,000 cells: below the line
    (lambda: meshgen.airfoil_2d_prisms(500, 151), WING, 2),           # 302,000: staged, five slots
    (lambda: meshgen.channel_bump(62, 41, 61, cells="hex"), DUCT, 2),  # staged, six slots
])
def test_default_form_of_large_batches_is_bitwise_the_unstaged_one(tmp_path, make, regions, n):
    p = str(tmp_path / "m.su2")
    make().write_su2(p)
    c = EulerCase(p)
    out = []
    for tuning in ((256, 1), (256, 3), (512, 4)):
        with EulerBatch([c], [(0, bcs(regions, 0.4 + 0.1 * i)) for i in range(n)]) as b:
            b.set_tuning(*tuning)
            for i in range(n):
                b.init_uniform(i, (0.4 + 0.1 * i, 0.0, 0.02), P, T)
            b.run(0.5, 12)
            out.append([x for i in range(n) for x in b.get_state(i)])
    c.close()
    assert same(out[0], out[1]) == [] and same(out[0], out[2]) == []
