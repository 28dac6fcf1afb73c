"""gbReduceSumNoAlloc after calls that overlapped on one arrival counter: an overlap
may spoil the results of the calls that overlap, but every later call, in order,
writes its sum.  Captured calls keep their counter, so two graphs whose calls were
captured 64 calls apart share one."""
import ctypes

import pytest

from graphite_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(5_000_017, 5_000_017), (5_000_017, 100_003), (300_001, 1_300_000)])
def test_later_calls_are_right_after_an_overlap(sizes):
    import torch

    lib = capi.load()

    def call(x, out):
        rc = lib.gbReduceSumNoAlloc(ctypes.c_void_p(x.data_ptr()), x.numel(), ctypes.c_void_p(out.data_ptr()),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0, capi.last_error()

    xs = [(torch.arange(n, device="cuda", dtype=torch.float32) % 1021) - 300.5 for n in sizes]
    want = [float(x.double().sum()) for x in xs]           # halves below 2^53: exact in every order
    outs = [torch.zeros(1, dtype=torch.float64, device="cuda") for _ in xs]
    small = torch.ones(3000, device="cuda")
    one = torch.zeros(1, dtype=torch.float64, device="cuda")
    call(xs[0], one)                                       # looks the scratch's address up before the captures
    torch.cuda.synchronize()
    graphs = []
    for k, x in enumerate(xs):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            call(x, outs[k])
        graphs.append(g)
        if k == 0:
            for _ in range(63):                            # the next capture takes the same counter
                call(small, one)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(40):
        torch.cuda._sleep(4_000_000)                       # both streams' replays queue up behind it
        go = torch.cuda.current_stream().record_event()
        for s in streams:
            s.wait_event(go)
        for _ in range(20):
            for g, s in zip(graphs, streams):
                with torch.cuda.stream(s):
                    g.replay()
        torch.cuda.synchronize()
    for _ in range(3):
        for k, g in enumerate(graphs):                     # in order from here on
            outs[k].fill_(-1.0)
            g.replay()
            torch.cuda.synchronize()
            assert outs[k].item() == want[k]
        for _ in range(64):                                # every counter
            one.fill_(-1.0)
            call(xs[0], one)
            torch.cuda.synchronize()
            assert one.item() == want[0]
