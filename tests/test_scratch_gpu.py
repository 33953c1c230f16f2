"""Scratch memory of calls with several launches: one call never sees what another one writes there."""
import threading

import pytest
import torch
import torch.nn as nn

from daceml_b200 import lib as L
from daceml_b200.torch import DaceModule

pytestmark = pytest.mark.gpu


def _conv(seed, size=40):
    """A small fp32 convolution whose channels-last copy of X lives in scratch memory, an input and its result."""
    torch.manual_seed(seed)
    net = nn.Conv2d(24, 32, 3, padding=1).cuda()
    x = torch.randn(2, 24, size, size, device="cuda")
    module = DaceModule(net, dummy_inputs=(x, ))
    return module, x, module(x).clone()


def _run_threads(cases, streams, rounds=150):
    bad = []

    def work(case, stream):
        module, x, want = case
        with torch.cuda.stream(stream):
            for _ in range(rounds):
                outs = [module(x) for _ in range(4)]
                if not all(torch.equal(o, want) for o in outs):
                    bad.append(case)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=a) for a in zip(cases, streams)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    torch.cuda.synchronize()
    assert not bad and L.get_context(0).device_status() == 0


@pytest.mark.parametrize("shared", [True, False], ids=["one stream", "own streams"])
def test_threads_with_modules_of_their_own(shared):
    cases = [_conv(i) for i in range(3)]
    stream = torch.cuda.Stream()
    _run_threads(cases, [stream if shared else torch.cuda.Stream() for _ in cases])


def test_graphs_of_one_capture_stream_run_side_by_side():
    cases = [_conv(i, 64) for i in range(2)]
    side, graphs, outs = torch.cuda.Stream(), [], []
    torch.cuda.synchronize()
    for module, x, _ in cases:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(side):
            graph.capture_begin(capture_error_mode="thread_local")
            outs.append(module(x))
            graph.capture_end()
        graphs.append(graph)
    streams = [torch.cuda.Stream() for _ in cases]
    for _ in range(200):
        for graph, stream in zip(graphs, streams):
            with torch.cuda.stream(stream):
                graph.replay()
    torch.cuda.synchronize()
    for out, (_, _, want) in zip(outs, cases):
        assert torch.equal(out, want)


def test_blocks_of_dropped_graphs_and_many_streams_are_used_again():
    module, x, want = _conv(0)

    def graph_once():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = module(x)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)

    graph_once()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(40):
        graph_once()
    assert free - torch.cuda.mem_get_info()[0] < 32 << 20  # one block is 2 MB: 40 of them would be 80 MB
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1) for _ in range(40)]
    for stream in streams:
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            y = module(x)
        stream.synchronize()
        assert torch.equal(y, want)
