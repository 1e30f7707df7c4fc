"""The Python binding's own host code, without a GPU."""
from types import SimpleNamespace


def test_stream_handle_without_the_private_names_of_torch(engine):
    public = SimpleNamespace(current_stream=lambda: SimpleNamespace(cuda_stream=77))
    assert engine.engine._stream_ptr(SimpleNamespace(_C=SimpleNamespace(), cuda=public)) == 77
    private = SimpleNamespace(_cuda_getDevice=lambda: 1, _cuda_getCurrentRawStream=lambda device: 40 + device)
    assert engine.engine._stream_ptr(SimpleNamespace(_C=private, cuda=public)) == 41
