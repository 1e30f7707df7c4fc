"""The activation quantiser where some of its CTAs are not there when the others meet: those that wait deal the whole tensor
out among themselves, or take the maximum alone, with the same bytes.  Also beside kernels that hold most of the GPU."""
import ctypes as C

import numpy as np
import pytest

from helpers import make_activations, to_torch_bf16

pytestmark = pytest.mark.gpu


def _quantize(engine, torch, x, scratch, workspace, polls, help_polls, absent):
    m, k = x.shape
    fn = engine.lib().q35b_debug_quantize_wait
    fn.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_uint, C.c_void_p]
    codes, scales, g = scratch
    assert fn(x.data_ptr(), m, k, codes.data_ptr(), scales.data_ptr(), g.data_ptr(), workspace.data_ptr(), polls, help_polls, absent,
              torch.cuda.current_stream().cuda_stream) == 0


# one CTA, a few, a grid of several turns per thread, rows with padding; the largest value in the first, a middle or the last place
@pytest.mark.parametrize("m,k", [(1, 48), (4, 1024), (5, 1040), (130, 1040), (1300, 4112), (3000, 3072)])
@pytest.mark.parametrize("polls,help_polls,absent", [(0, 1 << 12, 1), (3, 1 << 12, 7), (0, 0, 1), (0, 1 << 12, 0), (2, 1, 0)])
def test_bytes_without_the_absent(engine, oracle, m, k, polls, help_polls, absent):
    import torch

    xb = make_activations(m, k, seed=m + k)
    workspace = torch.zeros(int(engine.lib().q35b_quant_workspace_bytes()), dtype=torch.uint8, device="cuda")
    for at in (0, m * k // 2 + 3, m * k - 1):
        x = xb.copy()
        x.reshape(-1)[at] = 0x4490  # 1152
        xt = to_torch_bf16(x)
        scratch = engine.act_scratch(m, k, "cuda")
        for _ in range(2):
            for t in scratch:
                t.zero_()
            _quantize(engine, torch, xt, scratch, workspace, polls, help_polls, absent)
            e_codes, e_scales, e_g = oracle.quantize_nvfp4(oracle.bf16_to_f32(x), 0.0)
            assert np.float32(scratch[2].item()) == np.float32(e_g)
            assert np.array_equal(scratch[0].cpu().numpy().reshape(m, k // 2), e_codes)
            assert np.array_equal(scratch[1].cpu().numpy(), oracle.swizzle_scales(e_scales).reshape(-1))
            assert not bool(workspace.any())  # zero between calls


def test_beside_kernels_of_another_stream(engine):
    """Decode steps that hold every SM run on one stream, quantisations on another: same bytes, call after call."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(1)
    n, k, m = 28672, 9216, 1
    w = engine.Nvfp4Weight.from_device(torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen),
                                       torch.full((n, k // 16), 0x30, dtype=torch.uint8, device="cuda"), 1e-3)
    batch = engine.GemvBatch([(w, torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16),
                               torch.empty((m, n), dtype=torch.bfloat16, device="cuda"))], m)
    x = torch.randn((4096, 2560), device="cuda", generator=gen).to(torch.bfloat16)
    want = [t.clone() for t in engine.quantize_activations(x)]
    torch.cuda.synchronize()
    side, got = torch.cuda.Stream(), []
    with torch.cuda.stream(side):
        for _ in range(200):
            batch.run()
    for _ in range(50):
        got.append(engine.quantize_activations(x))
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for out in got for a, b in zip(out, want))


def test_built_in_scratch_has_room_for_the_counts(engine):
    """The words the quantiser counts in stand in front of the scale word and the status word of the built-in scratch: the same
    outputs as with a scratch of the caller's, twice in a row and with a scale whose bits are a large count."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(2)
    n, k, m = 256, 1024, 700
    w = engine.Nvfp4Weight.from_device(torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen),
                                       torch.full((n, k // 16), 0x30, dtype=torch.uint8, device="cuda"), 1e-3)
    for factor in (1.0, 1e6, 1e-6, 1.0):
        x = (torch.randn((m, k), device="cuda", generator=gen) * factor).to(torch.bfloat16)
        assert torch.equal(engine.project_prefill_static(w, x), engine.project_prefill(w, x))
    assert engine.static_prefill_status() == 0
