"""The persistent incompressible loop against the graph-replayed one, bit for
bit (``check_every`` picks the form: launches of fewer than four iterations
always replay the graphs): each launch shape, element kind, Laplacian and
limiter, meshes smaller than a warp, a stop inside a launch, a region without a
condition."""
import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.nsi import NSICase

pytestmark = pytest.mark.gpu

CHANNEL = [("wall", "lower"), ("slip", "upper"), ("slip", "sides"), ("inletoutlet", "inlet", 1.0, 0.0, 0.05, 0.0),
           ("inletoutlet", "outlet", 1.0, 0.0, 0.05, 0.0)]
CYLINDER = [("wall", "cylinder"), ("inletoutlet", "farfield", 1.0, 0.0, 0.05, 0.0), ("slip", "sides")]
MESHES = {
    "hex_1": (lambda: meshgen.channel_bump(1, 1, 1, cells="hex"), CHANNEL),
    "tet_6": (lambda: meshgen.channel_bump(1, 1, 1, cells="tet"), CHANNEL),
    "tet_6210": (lambda: meshgen.channel_bump(23, 9, 5, cells="tet"), CHANNEL),
    "prism": (lambda: meshgen.channel_bump(17, 9, 4, cells="prism"), CHANNEL),
    "pyramid": (lambda: meshgen.channel_bump(11, 5, 3, cells="pyramid"), CHANNEL),
    "mixed": (lambda: meshgen.channel_bump(19, 7, 3, cells="mixed"), CHANNEL),
    "cylinder_1104": (lambda: meshgen.cylinder_ogrid(48, 23, ratio=1.1, r_far=10.0), CYLINDER),
    "cylinder_99000": (lambda: meshgen.cylinder_ogrid(396, 250), CYLINDER),
    "cylinder_118000": (lambda: meshgen.cylinder_ogrid(472, 250), CYLINDER),
    "tet_147840": (lambda: meshgen.channel_bump(88, 40, 7, cells="tet"), CHANNEL),
}


@pytest.fixture(scope="module")
def mesh_paths(tmp_path_factory):
    made = {}
    d = tmp_path_factory.mktemp("nsi_loop")

    def get(name):
        if name not in made:
            made[name] = str(d / f"{name}.su2")
            MESHES[name][0]().write_su2(made[name])
        return made[name]

    return get


def solve(path, bcs, check_every, n, corrected, limited, tolerance=0.0):
    lib = capi.load()
    NSICase.set_constants(1.0, 0.03, 2.0, corrected, limited)
    try:
        c = NSICase(path)
        c.init((1.0, 0.0, 0.05), 0.0)
        launches = lib.gbKernelLaunchCount()
        out = [c.run(bcs, 0.5, n, tolerance=tolerance, check_every=check_every)]
        launches = lib.gbKernelLaunchCount() - launches
        out += list(c.fields()) + [np.float64(c.residual())]
        for f in (c.pressure, c.velocity, c.error):
            lib.VarAllGpuToCpu(f)
            out += [capi.field_values(f), *capi.field_gradients(f)]
        out.append(c.wall_force(bcs[0][1]))
        c.step(0.5)                              # with the gradients that the loop left
        out += list(c.fields())
        c.close()
        return out, launches
    finally:
        NSICase.set_constants()


def same(a, b):
    return all(np.array_equal(np.asarray(x), np.asarray(y), equal_nan=True) for x, y in zip(a, b))


@pytest.mark.parametrize("limited,corrected", [(False, True), (True, True), (False, False)])
@pytest.mark.parametrize("name", list(MESHES))
def test_persistent_loop_is_bitwise_the_graph_loop(mesh_paths, name, limited, corrected):
    bcs = MESHES[name][1]
    graphs, many = solve(mesh_paths(name), bcs, 3, 50, corrected, limited)
    loop, few = solve(mesh_paths(name), bcs, 25, 50, corrected, limited)
    assert few < 12 < many
    assert same(graphs, loop)


@pytest.mark.parametrize("kw", [dict(tolerance=0.3), dict(bcs="missing")])
def test_persistent_loop_options(mesh_paths, kw):
    name = "cylinder_1104" if "tolerance" in kw else "mixed"
    bcs = MESHES[name][1]
    if kw.pop("bcs", None):
        bcs = bcs[:2] + bcs[3:]
    graphs, _ = solve(mesh_paths(name), bcs, 3, 80, True, False, **kw)
    loop, few = solve(mesh_paths(name), bcs, 100, 80, True, False, **kw)
    assert few < 12
    assert same(graphs, loop)
    if "tolerance" in kw:
        assert 1 < len(loop[0]) < 80
