"""The persistent Euler loop against the graph-replayed one, bit for bit.

``check_every`` picks the form: launches of fewer than four iterations always
replay the graphs.  The meshes cover each launch shape of the persistent form
(cells per block up to 256, 320, 416 and 512, the last with the face normals
left in global memory), every element kind, blocks with idle threads, and a
mesh smaller than a warp.
"""
import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.euler import EulerCase

pytestmark = pytest.mark.gpu

P, T = 1.0, 1.0 / 1.4
CHANNEL = [("farfield", "inlet", 0.5, 0.0, 0.0, P, T), ("slip", "lower"), ("farfield", "outlet", 0.5, 0.0, 0.0, P, T),
           ("slip", "sides"), ("slip", "upper")]
AIRFOIL = [("farfield", "farfield", 0.6, 0.0, 0.05, P, T), ("slip", "sides"), ("slip", "wing")]
WING = [("farfield", "farfield", 0.8, 0.0, 0.04, P, T), ("slip", "symmetry"), ("slip", "wing")]

MESHES = {
    "hex_1": (lambda: meshgen.channel_bump(1, 1, 1, cells="hex"), CHANNEL),
    "tet_6": (lambda: meshgen.channel_bump(1, 1, 1, cells="tet"), CHANNEL),
    "tet_12960": (lambda: meshgen.channel_bump(24, 15, 6, cells="tet"), CHANNEL),
    "hex_1155": (lambda: meshgen.channel_bump(21, 11, 5, cells="hex"), CHANNEL),
    "mixed": (lambda: meshgen.channel_bump(19, 7, 3, cells="mixed"), CHANNEL),
    "layered": (lambda: meshgen.channel_bump(13, 6, 4, cells="layered"), CHANNEL),
    "wing_18376": (lambda: meshgen.swept_wing(40, 14, 10, 6), WING),
    "airfoil_9108": (lambda: meshgen.airfoil_2d_prisms(66, 69), AIRFOIL),
    "airfoil_84000": (lambda: meshgen.airfoil_2d_prisms(300, 140), AIRFOIL),
    "airfoil_121680": (lambda: meshgen.airfoil_2d_prisms(390, 156), AIRFOIL),
    "airfoil_147840": (lambda: meshgen.airfoil_2d_prisms(440, 168), AIRFOIL),
    "hex_102400": (lambda: meshgen.channel_bump(160, 80, 8, cells="hex"), CHANNEL),
}


@pytest.fixture(scope="module")
def mesh_paths(tmp_path_factory):
    made = {}
    d = tmp_path_factory.mktemp("loop")

    def get(name):
        if name not in made:
            made[name] = str(d / f"{name}.su2")
            MESHES[name][0]().write_su2(made[name])
        return made[name]

    return get


def solve(path, bcs, check_every, n, transposed=True, tolerance=0.0, density=False):
    lib = capi.load()
    lib.gbSetReferenceMomentumReconstruction(1 if transposed else 0)
    try:
        with EulerCase(path) as c:
            far = [b for b in bcs if b[0] == "farfield"][0]
            c.init(far[2:5], P, T)
            launches = lib.gbKernelLaunchCount()
            if density:
                hist = np.concatenate(c.run_density(bcs, 0.5, n, tolerance=tolerance, check_every=check_every))
            else:
                hist = c.run(bcs, 0.5, n, tolerance=tolerance, check_every=check_every)
            launches = lib.gbKernelLaunchCount() - launches
            out = [hist, *c.fields(), c.error_values(), np.float64(c.residual())]
            # the step that follows finds the face states of the last gradient pass
            c.step(0.5)
            out += list(c.fields())
            return out, launches
    finally:
        lib.gbSetReferenceMomentumReconstruction(1)


def same(a, b):
    return all(np.array_equal(np.asarray(x), np.asarray(y), equal_nan=True) for x, y in zip(a, b))


@pytest.mark.parametrize("name", list(MESHES))
def test_persistent_loop_is_bitwise_the_graph_loop(mesh_paths, name):
    bcs = MESHES[name][1]
    n = 70
    graphs, many = solve(mesh_paths(name), bcs, 2, n)
    loop, few = solve(mesh_paths(name), bcs, 35, n)
    assert few < 10 < many                       # the two forms did run
    assert same(graphs, loop)


@pytest.mark.parametrize("kw", [dict(transposed=False), dict(density=True), dict(tolerance=0.5), dict(bcs="missing")])
def test_persistent_loop_options(mesh_paths, kw):
    """Consistent momentum gradient; density history; a stop inside a launch;
    regions without a condition keep their ghosts."""
    name = "airfoil_9108" if kw.get("bcs") is None else "tet_12960"
    bcs = MESHES[name][1]
    if kw.pop("bcs", None):
        bcs = bcs[:2]
    graphs, _ = solve(mesh_paths(name), bcs, 2, 90, **kw)
    loop, few = solve(mesh_paths(name), bcs, 100, 90, **kw)
    assert few < 10
    assert same(graphs, loop)
    if "tolerance" in kw:
        assert 1 < len(loop[0]) < 90 and loop[0][-1] / loop[0][0] < 0.5
