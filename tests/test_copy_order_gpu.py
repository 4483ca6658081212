"""Copies of a state (copy, assign) are of the state as it was at the call: each
handle has a stream of its own, and what the source is given next waits for
the copy, which takes milliseconds at this size, to have read it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["copy", "assign"])
@pytest.mark.parametrize("change", ["gates", "reset", "measure", "delete"])
def test_the_source_may_change_at_once(qsl, kind, change):
    import torch
    n = 27
    src, dst = qsl.Qubits(n), qsl.Qubits(n)
    view = src.device_view()
    view.normal_(generator=torch.Generator(device="cuda").manual_seed(7))
    view.mul_(2.0 ** -14)
    want = view.clone()
    torch.cuda.synchronize()
    if kind == "copy":
        dst = src.copy()
    else:
        dst.assign(src)
    if change == "gates":
        for t in (0, 26, 13):
            src.gate("rotateX", t, None, 1.0)
            src.gate("rotateY", (t + 5) % n, None, 0.5)
        src.flush()
    elif change == "reset":
        src.reset()
    elif change == "measure":
        src.measure(26, 0.5)
    else:
        del view, src
    dst.synchronize()
    assert torch.equal(dst.device_view(), want)


def test_assign_may_be_captured(qsl):
    """Captured from the destination's stream, the copy is one of the source as
    it is at each replay; the source's stream stays out of the capture."""
    import torch
    n = 12
    src, dst = qsl.Qubits(n), qsl.Qubits(n)
    stream = torch.cuda.Stream()
    dst.set_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        dst.assign(src)
        src.gate("hadamard", 0, None, 0.0)      # runs at once
        src.flush()
    for t in range(n):
        src.gate("rotateX", t, None, 0.3 + t)
        src.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        want = src.getState()
        assert t or np.count_nonzero(want) == 2     # the Hadamard, and rotateX on its qubit
        assert np.array_equal(dst.getState().view(np.uint64), want.view(np.uint64))
