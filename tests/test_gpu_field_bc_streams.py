"""gbFieldBcFixed / gbFieldBcZeroGrad are recorded and launched by the next call that
uses the field; what a caller ordered against the calls themselves holds all the
same: a condition asked for while the caller captures the stream is part of the
graph, one asked for before the capture is not, and a stream that waits for an
event recorded after the call sees the ghosts, whichever stream used the field
first."""
import ctypes as C

import numpy as np
import pytest

from graphite_b200 import capi, meshgen
from graphite_b200.euler import EulerCase

pytestmark = pytest.mark.gpu


class Fields:
    def __init__(self, path):
        self.lib = capi.load()
        self.c = EulerCase(path)
        self.mesh, self.n = self.c.mesh, self.c.n_cells
        size = int(self.lib.cuMeshGetVarSize(self.mesh))
        self.u = self.lib.FvmFieldNew(4, size, b"u", 1)
        self.x = self.lib.FvmFieldNew(4, size, b"x", 1)
        starts = capi.mesh_array(self.mesh, "cell_faces_starts")
        inner = capi.mesh_array(self.mesh, "cell_connects")[starts[self.n:-1]]
        ids, first = capi.mesh_array(self.mesh, "ghost_cell_ids"), capi.mesh_array(self.mesh, "ghost_cell_starts")
        self.ghosts = ids[first[0]:first[1]].astype(int)          # of region 0
        self.inner = inner[self.ghosts - self.n]
        rng = np.random.default_rng(4)
        self.u0, self.dx = (rng.integers(0, 100, size).astype(np.float32) for _ in range(2))
        for f, v in ((self.u, self.u0), (self.x, self.dx)):
            capi.set_field_values(f, v)
            capi.check(self.lib.gbVarCpuToGpu(self.mesh, f), "gbVarCpuToGpu")
        self.gradient()                                            # allocates what it needs

    def on(self, stream):
        self.lib.gbSetStream(C.c_void_p(stream.cuda_stream if stream else None))

    def gradient(self):
        capi.check(self.lib.gbFvmGradient(self.mesh, self.u), "gbFvmGradient")

    def axpy(self):
        capi.check(self.lib.gbFieldAxpy(self.mesh, self.u, 1.0, self.x), "gbFieldAxpy")

    def fixed(self, v):
        capi.check(self.lib.gbFieldBcFixed(self.mesh, self.u, capi.vec(v, 0, 0), 0), "gbFieldBcFixed")

    def zero_grad(self):
        capi.check(self.lib.gbFieldBcZeroGrad(self.mesh, self.u, 0), "gbFieldBcZeroGrad")

    def values(self):
        self.lib.VarGpuToCpu(self.u)
        assert capi.last_error() == ""
        return capi.field_values(self.u)


@pytest.fixture
def fields(tmp_path):
    import torch

    p = str(tmp_path / "m.su2")
    meshgen.channel_bump(12, 7, 4, cells="mixed").write_su2(p)
    f = Fields(p)
    torch.cuda.synchronize()
    yield f
    torch.cuda.synchronize()
    f.on(None)
    f.lib.FvmFieldFree(f.u)
    f.lib.FvmFieldFree(f.x)
    f.c.close()


def test_condition_inside_a_capture_is_part_of_the_graph(fields):
    import torch

    f, s = fields, torch.cuda.Stream()
    f.on(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        f.axpy()
        f.zero_grad()                    # the last call of the capture
    v = f.values()
    assert np.array_equal(v, f.u0)       # nothing has run
    for k in (1, 2):
        with torch.cuda.stream(s):
            g.replay()
        v = f.values()
        want = f.u0[: f.n] + k * f.dx[: f.n]
        assert np.array_equal(v[: f.n], want) and np.array_equal(v[f.ghosts], want[f.inner])


@pytest.mark.parametrize("asked_on", ["same stream", "default stream"])
def test_condition_before_a_capture_is_applied_outside_the_graph(fields, asked_on):
    import torch

    f, s = fields, torch.cuda.Stream()
    f.on(s if asked_on == "same stream" else None)
    f.axpy()
    f.zero_grad()
    s.wait_event(torch.cuda.default_stream().record_event())
    f.on(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        f.gradient()                     # the first use of the field since
        f.axpy()
    v = f.values()
    once = f.u0[: f.n] + f.dx[: f.n]
    assert np.array_equal(v[: f.n], once) and np.array_equal(v[f.ghosts], once[f.inner])
    f.fixed(1000.0)
    assert np.all(f.values()[f.ghosts] == 1000.0)
    with torch.cuda.stream(s):
        g.replay()
    v = f.values()
    assert np.array_equal(v[: f.n], once + f.dx[: f.n])
    assert np.all(v[f.ghosts] == 1000.0)      # the replay does not repeat the condition


@pytest.mark.parametrize("asked_on", ["stream", "default stream"])
@pytest.mark.parametrize("first_use", ["asking stream", "other stream"])
def test_streams_ordered_behind_the_call_see_the_condition(fields, first_use, asked_on):
    import torch

    f = fields
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    if asked_on == "default stream":
        a = torch.cuda.default_stream()
    f.on(a)
    f.fixed(500.0)
    after = a.record_event()
    b.wait_event(after)
    early, late = (a, b) if first_use == "asking stream" else (b, a)
    with torch.cuda.stream(early):
        torch.cuda._sleep(200_000_000)   # the launch that the next call makes waits behind it
    f.on(early)
    f.gradient()
    f.on(late)
    assert np.all(f.values()[f.ghosts] == 500.0)


@pytest.mark.parametrize("asked_on", ["stream", "default stream"])
def test_both_streams_in_turn_and_a_capture_of_the_second(fields, asked_on):
    """An application on another stream is waited for by a captured use of the field too."""
    import torch

    f = fields
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    if asked_on == "default stream":
        a = torch.cuda.default_stream()
    f.on(a)
    f.fixed(500.0)
    b.wait_event(a.record_event())
    with torch.cuda.stream(a):
        torch.cuda._sleep(200_000_000)
    f.gradient()
    f.on(b)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=b):
        f.gradient()
    with torch.cuda.stream(b):
        g.replay()
    got = f.values()
    assert np.all(got[f.ghosts] == 500.0)


def test_field_with_a_pending_condition_can_be_freed(fields):
    size = int(fields.lib.cuMeshGetVarSize(fields.mesh))
    u = fields.lib.FvmFieldNew(12, size, b"v", 1)
    capi.check(fields.lib.gbFieldBcZeroGrad(fields.mesh, u, 1), "gbFieldBcZeroGrad")
    fields.lib.FvmFieldFree(u)
    fields.gradient()
    assert np.array_equal(fields.values(), fields.u0)
