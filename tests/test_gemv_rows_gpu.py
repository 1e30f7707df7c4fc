"""The single decode projection on the SIMT kernel where it can go wrong: K of one block, of a partial piece and of several
rounds of pieces (multiples of 16 that are none of 32 or 256), row counts on both sides of one and two rows per warp and
of four warps per row, every token count, fp32 activations, and BF16 activations that are not 16-byte aligned.  Against
the CPU oracle: fp32 sums in another order, so one BF16 rounding (relative L2 2^-9) or, in fp32, K rounding errors of 2^-24
that add up like a random walk (below 1e-5 for K up to 10^4)."""
import numpy as np
import pytest

from helpers import from_torch_bf16, make_activations, make_weight, to_torch_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", range(1, 9))
@pytest.mark.parametrize("n,k", [(1, 16), (3, 48), (155, 1792), (100, 4144), (1183, 1040), (1185, 2064), (2367, 272), (2369, 528)])
def test_bf16(engine, oracle, n, k, m):
    _, codes, scales, s2 = make_weight(n, k, seed=n + k)
    xb = make_activations(m, k, seed=m, outlier_frac=0.001)
    w = engine.Nvfp4Weight.from_host(codes, scales, s2)
    y = engine.gemv_w4a16(w, to_torch_bf16(xb))
    eb, _ = oracle.gemv_bf16(codes, scales, s2, xb, threads=8)
    assert oracle.rel_l2(oracle.bf16_to_f32(from_torch_bf16(y)), oracle.bf16_to_f32(eb)) <= 1e-3


@pytest.mark.parametrize("n,k", [(1, 16), (155, 1792), (100, 4144), (1185, 2064), (2369, 528), (300, 9200)])
def test_f32(engine, oracle, n, k):
    import torch

    _, codes, scales, s2 = make_weight(n, k, seed=n + k)
    x = torch.randn(k, generator=torch.Generator().manual_seed(k))
    w = engine.Nvfp4Weight.from_host(codes, scales, s2)
    y = engine.gemv_w4a16_f32(w, x.cuda(), 0.75).cpu().double()
    c = torch.from_numpy(np.stack([codes & 15, codes >> 4], axis=-1).reshape(n, k).astype(np.int64))
    level = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64)
    b = torch.from_numpy(scales.astype(np.int64))
    e, f = (b >> 3) & 15, (b & 7).double()
    scale = torch.where(e == 0, f * 2.0 ** -9, (8 + f) * 2.0 ** (e.double() - 10))
    wide = level[c & 7] * torch.where(c >= 8, -1.0, 1.0).double() * scale.repeat_interleave(16, dim=1) * float(s2)
    want = wide @ (x * 0.75).double()
    assert float((y - want).norm() / want.norm()) <= 1e-5


def test_unaligned_activations_where_k_is_no_multiple_of_32(engine):
    import torch

    _, codes, scales, s2 = make_weight(77, 1040, seed=3)
    w = engine.Nvfp4Weight.from_host(codes, scales, s2)
    wide = torch.randn(2 * 1040 + 1, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").to(torch.bfloat16)
    x = wide[1:].view(2, 1040)
    y, z = engine.gemv_w4a16(w, x).float(), engine.gemv_w4a16(w, x.clone()).float()
    assert float((y - z).norm() / z.norm()) <= 1e-3
