"""The persistent decode step wants a CTA on every multiprocessor of the device: where the current context or the stream has fewer, steps stay with the separate launches."""
import pytest
import torch

pytestmark = pytest.mark.gpu
WIDTHS = [(2048, 2048, 1024, 6144), (1024, 2048, 1024, 3072)]


def test_green_contexts():
    import nano_qwen3tts_vllm_b200._native as nat
    green = pytest.importorskip("torch.cuda.green_contexts")
    if not green.SUPPORTED:
        pytest.skip("torch without green contexts")
    torch.zeros(1, device="cuda")
    both = lambda: {(nat.decode_rows_supported(2, *w), nat.decode_rows_taken(2, 256, *w)) for w in WIDTHS}
    assert both() == {(True, True)}
    small = green.GreenContext.create(num_sms=64, device_id=0)
    small.set_context()
    try:
        assert both() == {(False, False)}
    finally:
        small.pop_context()
    assert both() == {(True, True)}
    with torch.cuda.stream(torch.cuda.Stream()):
        assert both() == {(True, True)}


def test_asked_under_capture():
    import nano_qwen3tts_vllm_b200._native as nat
    x, graph = torch.zeros(4, device="cuda"), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x += 1
        assert all(nat.decode_rows_taken(1, 4096, *w) for w in WIDTHS)
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1.0] * 4
