"""Where the device has no memory for what the persistent loop keeps, a run replays
its graphs with the same results, and nothing of a half-made loop stays allocated."""
import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.batch import EulerBatch
from graphite_b200.euler import EulerCase

pytestmark = pytest.mark.gpu
P, T = 1.0, 1.0 / 1.4
WING = [("farfield", "farfield", 0.6, 0.0, 0.05, P, T), ("slip", "sides"), ("slip", "wing")]


def fill(torch):
    """Takes all device memory but the size of torch's small segments (about 20 MB)."""
    taken, size = [], 1 << 34
    while size >= 1 << 21:
        try:
            taken.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size //= 2
    return taken


def test_batch_without_memory_for_the_loop(tmp_path):
    import torch

    p = str(tmp_path / "m.su2")
    meshgen.airfoil_2d_prisms(360, 150).write_su2(p)             # 108,000 cells: 26 MB of records
    lib = capi.load()
    with EulerCase(p) as c:
        def run(b, check_every):
            b.init_uniform(0, (0.5, 0.0, 0.02), P, T)
            n0 = lib.gbKernelLaunchCount()
            b.run(0.5, 40, check_every=check_every)
            return list(b.get_state(0)), lib.gbKernelLaunchCount() - n0

        with EulerBatch([c], [(0, WING)]) as b:
            run(b, 20)                       # every kernel of the loop is loaded
        with EulerBatch([c], [(0, WING)]) as b:
            want, many = run(b, 2)           # the graph, its items and the copy of the state are made
            taken = fill(torch)
            try:
                free = torch.cuda.mem_get_info()[0]
                got, launches = run(b, 20)
                left = torch.cuda.mem_get_info()[0]
            finally:
                taken.clear()
                torch.cuda.empty_cache()
            assert launches > 100 and many > 100
            assert left == free
            assert all(np.array_equal(x, y) for x, y in zip(want, got))


def test_mesh_without_memory_for_the_loop(tmp_path):
    import torch

    p = str(tmp_path / "m.su2")
    meshgen.airfoil_2d_prisms(360, 150).write_su2(p)
    lib = capi.load()
    with EulerCase(p) as c:
        def run(case, check_every):
            case.init((0.5, 0.0, 0.02), P, T)
            n0 = lib.gbKernelLaunchCount()
            h = case.run(WING, 0.5, 40, check_every=check_every)
            return [h, *case.fields()], lib.gbKernelLaunchCount() - n0

        run(c, 20)
        with EulerCase(p) as d:
            want, many = run(d, 2)
            taken = fill(torch)
            try:
                free = torch.cuda.mem_get_info()[0]
                got, launches = run(d, 20)
                left = torch.cuda.mem_get_info()[0]
            finally:
                taken.clear()
                torch.cuda.empty_cache()
            assert launches > 100 and many > 100
            assert left == free
            assert all(np.array_equal(x, y) for x, y in zip(want, got))
