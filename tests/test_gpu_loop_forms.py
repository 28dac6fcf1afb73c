"""Which form a run takes.  Meshes whose block size (224 and 256 threads on a GPU
of 148 SMs) is too large for the wide form's shared memory: the persistent loop
against the replayed kernels, bit for bit, for one mesh and for a batch, which
takes the loop there as it does for smaller and larger meshes.  Meshes at which
the loop is the slower form: the kernels."""
import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.batch import EulerBatch
from graphite_b200.euler import EulerCase

pytestmark = pytest.mark.gpu
P, T = 1.0, 1.0 / 1.4
AIRFOIL = [("farfield", "farfield", 0.6, 0.0, 0.05, P, T), ("slip", "sides"), ("slip", "wing")]
DUCT = [("farfield", "inlet", 0.5, 0.0, 0.0, P, T), ("slip", "lower"), ("farfield", "outlet", 0.5, 0.0, 0.0, P, T),
        ("slip", "sides"), ("slip", "upper")]
CYLINDER = [("farfield", "farfield", 0.3, 0.0, 0.0, P, T), ("slip", "sides"), ("slip", "cylinder")]
# faces per cell and threads per block (148 SMs); whether a batch takes the loop too
MESHES = {
    "prism_70000": (lambda: meshgen.airfoil_2d_prisms(350, 100), AIRFOIL, True),           # 5, 256
    "cylinder_62000": (lambda: meshgen.cylinder_ogrid(310, 200), CYLINDER, True),          # 6, 224
    "cylinder_72000": (lambda: meshgen.cylinder_ogrid(360, 200), CYLINDER, True),          # 6, 256
    "hex_72000": (lambda: meshgen.channel_bump(100, 90, 8, cells="hex"), DUCT, False),    # 6, 256: short runs only
}
# sizes between two that take the loop at which it was slower than the kernels
SLOWER = {
    "mixed_67000": (lambda: meshgen.channel_bump(60, 46, 8, cells="mixed"), DUCT),
    "pyramid_99000": (lambda: meshgen.channel_bump(55, 30, 10, cells="pyramid"), DUCT),
    "tet_136000": (lambda: meshgen.channel_bump(81, 40, 7, cells="tet"), DUCT),
}


def same(a, b):
    return [k for k, (x, y) in enumerate(zip(a, b)) if not np.array_equal(np.asarray(x), np.asarray(y))]


@pytest.mark.parametrize("name", list(MESHES))
def test_loop_where_the_wide_form_does_not_fit(tmp_path, name):
    make, bcs, batch_loop = MESHES[name]
    p = str(tmp_path / "m.su2")
    make().write_su2(p)
    lib = capi.load()
    with EulerCase(p) as c:
        out = []
        for check_every in (2, 32):
            c.init(bcs[0][2:5], P, T)
            n0 = lib.gbKernelLaunchCount()
            h = c.run(bcs, 0.5, 64, check_every=check_every)
            launches = lib.gbKernelLaunchCount() - n0
            assert launches > 180 if check_every == 2 else launches < 10
            got = [h, *c.fields(), c.error_values()]
            c.step(0.5)
            out.append(got + list(c.fields()))
        assert same(out[0], out[1]) == []
        out = []
        for check_every in (2, 32):
            with EulerBatch([c], [(0, bcs)]) as b:
                b.init_uniform(0, bcs[0][2:5], P, T)
                n0 = lib.gbKernelLaunchCount()
                r = b.run(0.5, 64, check_every=check_every, history=True)
                launches = lib.gbKernelLaunchCount() - n0
                assert launches < 10 if check_every == 32 and batch_loop else launches > 180
                out.append([*r, *b.get_state(0)])
        assert same(out[0], out[1]) == []


@pytest.mark.parametrize("name", list(SLOWER))
def test_kernels_where_the_loop_is_slower(tmp_path, name):
    """A run of the usual launch length replays the graphs, alone and in a batch."""
    make, bcs = SLOWER[name]
    p = str(tmp_path / "m.su2")
    make().write_su2(p)
    lib = capi.load()
    with EulerCase(p) as c:
        c.init(bcs[0][2:5], P, T)
        n0 = lib.gbKernelLaunchCount()
        c.run(bcs, 0.5, 100)
        assert lib.gbKernelLaunchCount() - n0 >= 300
        with EulerBatch([c], [(0, bcs)]) as b:
            b.init_uniform(0, bcs[0][2:5], P, T)
            n0 = lib.gbKernelLaunchCount()
            b.run(0.5, 100)
            assert lib.gbKernelLaunchCount() - n0 >= 300
