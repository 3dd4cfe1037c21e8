"""Launches of small graphs (graphgolf_b200/csrc/apsp_slice.cuh) on several
streams, and captured ones: whatever becomes of launches that overlap, later
calls answer for their own graph."""
import ctypes

import numpy as np
import pytest
import torch

import graphgolf_b200 as gg
import oracle
from graphgolf_b200 import graphs
from graphgolf_b200._native import ggb_result, last_error

pytestmark = pytest.mark.gpu


def _launch(lib, adj, stream):
    n, d = adj.shape
    assert lib.ggb_launch_general_device(n, n, 1, d, adj.data_ptr(), 0, stream) == 0, last_error()


def test_later_calls_after_overlapping_launches(gpu):
    host = [graphs.random_regular(n, d, n).adj for n, d in [(256, 4), (1024, 8), (3000, 6), (4600, 8), (96, 5)]]
    want = [oracle.general(a) for a in host]
    dev = [torch.from_numpy(a).cuda() for a in host]
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    r = ggb_result()
    for rounds in range(20):
        for i in range(12):
            _launch(gpu, dev[(rounds + i) % 5], streams[i % 3].cuda_stream)
        gpu.ggb_collect(streams[11 % 3].cuda_stream, ctypes.byref(r))   # overlapped: no claim on its result
        torch.cuda.synchronize()
        for a, w in zip(host, want):
            got = gg.evaluate(a)
            assert (got.connected, got.diameter, got.aspl, got.total) == w


def test_captured_launch(gpu):
    """The captured launch follows its adjacency, replay after replay, with
    other evaluations between (of as many vertices: ggb_collect completes the
    answer by the last call's number)."""
    a, b = (graphs.random_regular(1024, 8, s).adj for s in (1, 2))
    dev = torch.from_numpy(a).cuda()
    r = ggb_result()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        _launch(gpu, dev, stream.cuda_stream)
        assert gpu.ggb_collect(stream.cuda_stream, ctypes.byref(r)) == 0, last_error()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            _launch(gpu, dev, stream.cuda_stream)
        for adj in (a, b, a):
            dev.copy_(torch.from_numpy(adj))
            graph.replay()
            assert gpu.ggb_collect(stream.cuda_stream, ctypes.byref(r)) == 0, last_error()
            assert (r.diameter, r.total) == oracle.general(adj)[1::2]
            small = graphs.random_regular(1024, 6, 3).adj
            got = gg.evaluate(small)
            assert (got.diameter, got.total) == oracle.general(small)[1::2]
