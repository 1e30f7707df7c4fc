"""The binding's native calls take the plain form of a call only; every other form goes the general way with the results and
errors it always had.  Both ways on the same inputs have to give the same bits."""
import ctypes

import numpy as np
import pytest

from helpers import make_activations, make_weight, to_torch_bf16

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def weight(engine):
    _, codes, scales, s2 = make_weight(384, 512, seed=3)
    return engine.Nvfp4Weight.from_host(codes, scales, s2)


def _general(engine, monkeypatch, call):
    """The call with every native function declining."""
    class Declines:
        def __getattr__(self, name):
            return lambda *a: NotImplemented

    with monkeypatch.context() as mp:
        mp.setattr(engine.engine if hasattr(engine, "engine") else engine, "_native_module", Declines())
        return call()


@pytest.mark.parametrize("m", [1, 8])
def test_same_bits_either_way(engine, weight, monkeypatch, m):
    import torch

    x = to_torch_bf16(make_activations(m, 512, seed=m))
    res = torch.randn((m, 384), device="cuda").to(torch.bfloat16)
    scratch = engine.act_scratch(m, 512, x.device)
    calls = [lambda: engine.gemv_w4a16(weight, x), lambda: engine.gemv_w4a16(weight, x, kernel=engine.GEMV_SIMT),
             lambda: engine.gemv_w4a16_f32(weight, x[0].float(), 0.5), lambda: engine.project_prefill(weight, x),
             lambda: engine.project_prefill(weight, x, scratch=scratch, global_scale=0.01, residual=res),
             lambda: engine.project_prefill(weight, x.float(), scratch=scratch),
             lambda: engine.gemm_w4a4(weight, *engine.quantize_activations(x), m)]
    for call in calls:
        a, b = call().clone(), _general(engine, monkeypatch, call)
        assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)


def test_other_forms(engine, weight):
    import torch

    x = to_torch_bf16(make_activations(2, 512, seed=9))
    want = engine.gemv_w4a16(weight, x)
    assert torch.equal(engine.gemv_w4a16(weight, x[0]), want[:1])          # a vector: one row comes back
    out = torch.zeros(2 * 384, dtype=torch.bfloat16, device="cuda")
    assert engine.gemv_w4a16(weight, x, out=out) is out and torch.equal(out.view(2, 384), want)
    assert torch.equal(engine.gemv_w4a16(weight, torch.nn.Parameter(x, requires_grad=False)), want)
    wide = torch.zeros((2, 400), dtype=torch.bfloat16, device="cuda")
    got = engine.project_prefill(weight, x, out=wide[:, :384])
    assert got.data_ptr() == wide.data_ptr() and torch.equal(wide[:, :384], engine.project_prefill(weight, x))
    for bad in (x.float(), x[:, :256], x.t()):
        with pytest.raises(AssertionError):
            engine.gemv_w4a16(weight, bad)
    with pytest.raises(engine.Q35bError):
        engine.gemv_w4a16(weight, x.repeat(5, 1))                            # ten tokens
    with pytest.raises(RuntimeError):
        engine.quantize_activations(x, scratch=engine.act_scratch(4, 512, x.device))
    with torch.cuda.stream(torch.cuda.Stream()):
        other = engine.gemv_w4a16(weight, x)
        torch.cuda.current_stream().synchronize()
    assert torch.equal(other, want)
    w2 = engine.Nvfp4Weight.from_host(np.zeros((128, 128), dtype=np.uint8), np.zeros((128, 16), dtype=np.uint8), 1.0)
    w2.close()
    with pytest.raises(Exception):
        engine.gemv_w4a16(w2, x[:, :256].contiguous())


@pytest.mark.parametrize("bad", [None, "1", 1.5])
def test_kernel_numbers_and_scales_of_other_types_stay_refused(engine, weight, bad):
    """What ctypes refuses on the general path is not converted by the native one."""
    import torch

    x = to_torch_bf16(make_activations(1, 512, seed=2))
    scratch = engine.act_scratch(1, 512, x.device)
    with pytest.raises(ctypes.ArgumentError):
        engine.gemv_w4a16(weight, x, kernel=bad)
    if bad is None or bad == "1":  # a scale may be anything that has a float
        with pytest.raises(ctypes.ArgumentError):
            engine.gemv_w4a16_f32(weight, x[0].float(), bad)
        with pytest.raises(ctypes.ArgumentError):
            engine.quantize_activations(x, bad, scratch)
    else:
        assert torch.equal(engine.gemv_w4a16_f32(weight, x[0].float(), bad), engine.gemv_w4a16_f32(weight, x[0].float(), float(bad)))


def _events(torch, call):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        call()
    return {e.key for e in prof.key_averages()}


def _nodes(torch, call, tmp_path):
    """Kernels of a captured call."""
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    graph.enable_debug_mode()
    with torch.cuda.graph(graph):
        call()
    path = tmp_path / f"{len(list(tmp_path.iterdir()))}.dot"
    graph.debug_dump(str(path))
    return path.read_text()


def test_new_outputs_are_seen_by_a_profiler_and_filled_where_that_is_asked_for(engine, weight, tmp_path):
    """Outputs are made without the dispatcher, but not where someone would miss it."""
    import torch

    x = to_torch_bf16(make_activations(2, 512, seed=4))
    calls = [lambda: engine.gemv_w4a16(weight, x), lambda: engine.gemv_w4a16_f32(weight, x[0].float()), lambda: engine.project_prefill(weight, x)]
    for call in calls:
        call()
        assert "aten::empty" in _events(torch, call)
    plain = _nodes(torch, calls[0], tmp_path)
    assert torch.utils.deterministic.fill_uninitialized_memory
    torch.use_deterministic_algorithms(True)
    try:
        filled = _nodes(torch, calls[0], tmp_path)
    finally:
        torch.use_deterministic_algorithms(False)
    assert "FillFunctor" not in plain and "FillFunctor" in filled
