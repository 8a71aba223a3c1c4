"""A layer call without a stream goes to torch's current one, whichever way its handle is found.  Shown by capture: under a capture of that
stream a call is recorded and does not run, and anything put on another stream would not be in the graph."""
import numpy as np
import pytest
import torch

from smallframework_b200 import interface as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("raw", [True, False], ids=["raw_handle", "stream_object"])
def test_layer_runs_on_the_current_stream(monkeypatch, raw):
    if raw:
        assert S._raw_stream is not None  # the short way is there in this torch
    else:
        monkeypatch.setattr(S, "_raw_stream", None)
    x = np.random.default_rng(3).uniform(-1, 1, 2 * 16 * 9 * 7).astype(np.float32)
    I, O = S.FloatBuffer(data=x), S.FloatBuffer(data=np.full(x.size, 7, np.float32))
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        assert S._stream(None) == stream.cuda_stream
    assert S._stream(None) == torch.cuda.current_stream().cuda_stream != stream.cuda_stream
    with torch.cuda.graph(graph, stream=stream):
        S.ReLUActivation(16, 9, 7, I, O, batch=2)
    torch.cuda.synchronize()
    assert (O.numpy() == 7).all()
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(O.numpy(), np.maximum(x, 0))


def test_an_explicit_stream_wins():
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        assert S._stream(b) == S._stream(b.cuda_stream) == b.cuda_stream
