"""Scratch of the split-K products: one per stream, and one per CUDA graph and stream of its capture."""
import types

import pytest
import torch

from dart_pytorch_b200.ops import kernels as K


def test_every_capture_has_its_own(monkeypatch):
    state = types.SimpleNamespace(stream=7, capture=0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: types.SimpleNamespace(cuda_stream=state.stream))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state.capture != 0)
    monkeypatch.setattr(K.N, "load", lambda *a: types.SimpleNamespace(dptb_capture_id=lambda s: state.capture))
    for name in ("_SPLITK_WS", "_SPLITK_GRAPH_WS"):
        monkeypatch.setattr(K, name, {}, raising=False)
    monkeypatch.setattr(K, "SPLITK_WS_BYTES", 64)
    dev = torch.device("cpu", 0)

    def at(stream, capture):
        state.stream, state.capture = stream, capture
        return K.splitk_workspace(dev)
    kept = {(s, c): at(s, c) for s, c in ((7, 0), (7, 1), (8, 1), (7, 2), (8, 0))}
    assert len({t.data_ptr() for pair in kept.values() for t in pair}) == 10
    for s, c in ((7, 0), (8, 0), (7, 2)):               # one after the other on a stream, or within a graph: the same
        assert at(s, c)[1] is kept[s, c][1]
    assert all(not t.any() for _, t in kept.values())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_graphs_of_one_capture_stream_run_at_once(dtype):
    """Two graphs, the later one first, then both at once on two streams: the bits of the eager products."""
    Kd = 4096
    a = [torch.randn(40, Kd, device="cuda").to(dtype) for _ in range(2)]
    w = [torch.randn(64, Kd, device="cuda").to(dtype) for _ in range(2)]
    out = [torch.zeros(40, 64, device="cuda", dtype=dtype) for _ in range(2)]
    want, graphs, scratch = [], [], []
    for i in range(2):
        want.append(K.gemm(a[i], w[i], torch.empty_like(out[i]), trans_b=True, splits=4))
    torch.cuda.synchronize()
    for i in range(2):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            scratch.append(K.splitk_workspace(a[i].device)[0].data_ptr())
            for _ in range(20):
                K.gemm(a[i], w[i], out[i], trans_b=True, splits=4)
        graphs.append(g)
    assert len({*scratch, K.splitk_workspace(a[0].device)[0].data_ptr()}) == 3
    graphs[1].replay()
    torch.cuda.synchronize()
    assert torch.equal(out[1], want[1])
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(20):
        for i in range(2):
            with torch.cuda.stream(streams[i]):
                out[i].zero_()
                graphs[i].replay()
        torch.cuda.synchronize()
        assert torch.equal(out[0], want[0]) and torch.equal(out[1], want[1])
