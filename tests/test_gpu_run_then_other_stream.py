"""A run returns its residuals, so its caller may go on with the fields on another
stream without ordering the two: the step after it finds the face states or
gradients of the run's last iteration.  Another stream's products keep the GPU
full when the run ends, so that its last kernels are still queued while the step's
stream, of a higher priority, gets through."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.euler import EulerCase
from graphite_b200.nsi import NSICase

pytestmark = pytest.mark.gpu
P, T = 1.0, 1.0 / 1.4
AIRFOIL = [("farfield", "farfield", 0.6, 0.0, 0.05, P, T), ("slip", "sides"), ("slip", "wing")]
DUCT = [("farfield", "inlet", 0.5, 0.0, 0.0, P, T), ("slip", "lower"), ("farfield", "outlet", 0.5, 0.0, 0.0, P, T),
        ("slip", "sides"), ("slip", "upper")]
CYLINDER = [("wall", "cylinder"), ("inletoutlet", "farfield", 1.0, 0.0, 0.05, 0.0), ("slip", "sides")]


def run_then_step(torch, case, run, crowded):
    """The states of a run on one stream and a step on another."""
    lib = case.lib
    a, b, busy = torch.cuda.Stream(), torch.cuda.Stream(priority=-1), torch.cuda.Stream()
    m = torch.ones((8192, 8192), device="cuda", dtype=torch.bfloat16)
    torch.matmul(m, m)
    torch.cuda.synchronize()
    done = threading.Event()

    def crowd():
        torch.cuda.set_device(0)
        time.sleep(0.005)                        # the run's launch is under way
        with torch.cuda.stream(busy):
            for _ in range(60):
                torch.matmul(m, m)
        done.set()

    helper = threading.Thread(target=crowd)
    try:
        lib.gbSetStream(C.c_void_p(a.cuda_stream))
        if crowded:
            helper.start()
        run()
        if crowded:
            done.wait(20)
        lib.gbSetStream(C.c_void_p(b.cuda_stream if crowded else a.cuda_stream))
        case.step(0.5)
        return [x.copy() for x in case.fields()]
    finally:
        if crowded:
            helper.join()
        torch.cuda.synchronize()
        lib.gbSetStream(None)


@pytest.mark.parametrize("make,bcs", [(lambda: meshgen.airfoil_2d_prisms(300, 140), AIRFOIL),
                                      (lambda: meshgen.channel_bump(60, 20, 6, cells="tet"), DUCT)])
def test_euler_run_then_a_step_on_another_stream(tmp_path, make, bcs):
    import torch

    p = str(tmp_path / "m.su2")
    make().write_su2(p)
    with EulerCase(p) as c:
        def run():
            c.init(bcs[0][2:5], P, T)
            c.run(bcs, 0.5, 2000, check_every=2000)

        want = run_then_step(torch, c, run, False)
        for _ in range(6):
            got = run_then_step(torch, c, run, True)
            assert all(np.array_equal(x, y) for x, y in zip(want, got))


def test_nsi_run_then_a_step_on_another_stream(tmp_path):
    import torch

    p = str(tmp_path / "m.su2")
    meshgen.cylinder_ogrid(240, 150).write_su2(p)
    c = NSICase(p)

    def run():
        c.init((1.0, 0.0, 0.05), 0.0)
        c.run(CYLINDER, 0.5, 3000, check_every=3000)

    want = run_then_step(torch, c, run, False)
    for _ in range(6):
        got = run_then_step(torch, c, run, True)
        assert all(np.array_equal(x, y) for x, y in zip(want, got))
    c.close()
