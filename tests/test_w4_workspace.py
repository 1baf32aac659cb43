"""The scratch that ``ops.w4a16_g128`` brings itself: one per device and stream, its own for a captured call."""

import pytest
import torch

from jax_metallib_b200 import ops


def test_one_per_stream(monkeypatch):
    monkeypatch.setattr(ops, "_w4_workspaces", {})
    cpu = torch.device("cpu")
    a, b = ops._w4_workspace(cpu, 1, 4096), ops._w4_workspace(cpu, 2, 4096)
    assert a.data_ptr() != b.data_ptr() and not a.any()
    assert ops._w4_workspace(cpu, 1, 4096) is a
    grown = ops._w4_workspace(cpu, 1, 2 << 20)
    assert grown.numel() >= 2 << 20 and not grown.any() and ops._w4_workspace(cpu, 2, 4096) is b
    for stream in range(3, 200):
        ops._w4_workspace(cpu, stream, 16)
    assert len(ops._w4_workspaces) <= ops._MAX_W4_WORKSPACES


def _layer(m, k, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    byte = lambda *shape: torch.randint(0, 256, shape, dtype=torch.uint8, device="cuda", generator=g)   # noqa: E731
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    s = torch.rand(k // 128, n, device="cuda", generator=g).bfloat16()
    return x, byte(k // 2, n), s, byte(k // 128, n // 2)


def _run(layer):
    x, w, s, z = layer
    return ops.w4a16_g128(x, w, s, z, zeros_packed=True, static_weights=True)


# widths that the kernel with partial sums in the workspace takes
@pytest.mark.gpu
def test_two_streams(cuda):
    layers = [_layer(8, 2048, 16512, 1), _layer(4, 4096, 20480, 2)]
    expected = [_run(layer) for layer in layers]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    results = ([], [])
    for _ in range(20):
        for stream, layer, out in zip(streams, layers, results):
            with torch.cuda.stream(stream):
                out.append(_run(layer))
    torch.cuda.synchronize()
    for want, got in zip(expected, results):
        assert all(torch.equal(y, want) for y in got)


@pytest.mark.gpu
@pytest.mark.parametrize("m,k,n", [(8, 2048, 16512), (8, 1024, 512)])   # with and without use of the workspace
def test_captured(cuda, m, k, n):
    """A graph's calls neither need a call before the capture nor share scratch with one another's graphs."""
    layer = _layer(m, k, n, 3)
    stream = torch.cuda.Stream()
    graphs, results = [], []
    for _ in range(2):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            results.append((_run(layer), _run(layer)))
        graphs.append(graph)
    with torch.cuda.stream(stream):
        expected = _run(layer)
    torch.cuda.synchronize()
    for _ in range(3):
        for graph, pair in zip(reversed(graphs), reversed(results)):
            for y in pair:
                y.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert all(torch.equal(y, expected) for y in pair)
    del graphs
