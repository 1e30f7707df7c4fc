"""The K-split prefill GEMM (weight rows on the 128-row side, a cluster of CTAs sharing a tile's K steps) where it can go
wrong: token counts around the tile widths, weight rows that are no multiple of 4, 16 or 128 (narrow stores), a K of one
short step, and row blocks few enough for every split.  Against the CPU oracle on the GPU quantiser's bytes; the result
is one BF16 rounding of an fp32 sum, so it may differ from the oracle's by flipped roundings only: the relative L2 error
of outputs that all flipped would be 2^-8 / sqrt(12) = 1.1e-3."""
import numpy as np
import pytest

from helpers import from_torch_bf16, make_activations, make_weight, to_torch_bf16

pytestmark = pytest.mark.gpu

REL_L2_TOL = 1e-3

SHAPES = [  # m, n, k and the split that the plan picks
    (1, 1, 64, 1), (1, 3, 4096, 8), (15, 127, 192, 1), (16, 129, 512, 1), (17, 108, 5760, 8), (7, 5001, 2048, 2),  # one short K step
    (63, 512, 2304, 1), (64, 512, 2304, 1), (65, 512, 4672, 4), (127, 250, 9216, 8), (128, 256, 9216, 8),  # 64- and 128-token tiles
    (129, 2560, 320, 1), (255, 1022, 1024, 1), (300, 1001, 704, 1),  # several token tiles, the last one partial
    (1000, 3584, 256, 1),  # more tiles than SMs
]


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("m,n,k,split", SHAPES)
def test_against_oracle(engine, oracle, m, n, k, split, residual):
    import torch

    plan = engine.gemm_plan(m, n, k)
    assert plan["split"] == split and not plan["pairs"]
    _, codes, scales, s2 = make_weight(n, k, seed=m + n + k)
    xb = make_activations(m, k, m + 1, outlier_frac=0.001)
    w = engine.Nvfp4Weight.from_host(codes, scales, s2)
    a_codes, a_scales, g = engine.quantize_activations(to_torch_bf16(xb))
    # a residual whose rows start at an odd address: the narrow path on an output that is aligned
    wide = torch.randn((m, n + 1), generator=torch.Generator(device="cuda").manual_seed(m), device="cuda").to(torch.bfloat16)
    res = wide[:, 1:] if residual else None
    c = engine.gemm_w4a4(w, a_codes, a_scales, g, m, residual=res)
    assert engine.gemm_default_status() == 0
    e_codes, e_scales, e_g = oracle.quantize_nvfp4(xb)
    eb, ef = oracle.gemm_w4a4(codes, scales, s2, e_codes, e_scales, e_g, threads=8)
    want = oracle.bf16_to_f32(eb)
    if residual:
        want = torch.from_numpy(np.asarray(ef) + res.float().cpu().numpy()).to(torch.bfloat16).float().numpy()
    err = oracle.rel_l2(oracle.bf16_to_f32(from_torch_bf16(c)), want)
    assert err <= REL_L2_TOL, (m, n, k, err)


@pytest.mark.parametrize("m", [1, 33, 100, 200, 513])
@pytest.mark.parametrize("inter,k", [(64, 64), (192, 4096), (1000, 512), (2504, 2048)])  # split in 1, 2, 4 and 8
def test_gate_up_matches_its_halves(engine, oracle, m, inter, k):
    """silu(gate) * up of the fused epilogue against the two halves projected on their own (BF16 outputs): two roundings of
    2^-9 on its inputs and one on the result, and silu's slope is at most 1.1."""
    import torch

    _, gc, gs, g2 = make_weight(inter, k, seed=inter + k)
    _, uc, us, u2 = make_weight(inter, k, seed=inter + k + 1)
    a = engine.quantize_activations(to_torch_bf16(make_activations(m, k, m)))
    fused = engine.gemm_w4a4(engine.Nvfp4Weight.gate_up_from_host(gc, gs, g2, uc, us, u2), *a, m)
    gate = engine.gemm_w4a4(engine.Nvfp4Weight.from_host(gc, gs, g2), *a, m).double()
    up = engine.gemm_w4a4(engine.Nvfp4Weight.from_host(uc, us, u2), *a, m).double()
    want = gate / (1 + torch.exp(-gate)) * up
    assert engine.gemm_default_status() == 0
    assert float((fused.double() - want).norm() / want.norm()) <= 3 * 2.0 ** -9


@pytest.mark.parametrize("n,k", [(256, 256), (9216, 4096), (4608, 2560), (256, 4096)])  # split in 1, 2, 4 and 8
def test_own_status_word_is_read_after_the_stream_has_set_it(engine, n, k):
    """A status word that a kernel right in front of the GEMM sets to zero, one that lets its successor start early (the
    single projection, whose outputs are zero for a zero input): the GEMM runs, every time.  With a code on record it
    stores nothing and leaves the code."""
    import torch

    m, wide, iters = 8, 32768, 30
    rnd = torch.Generator(device="cuda").manual_seed(1)
    codes = torch.randint(0, 256, (wide, 3360), dtype=torch.uint8, device="cuda", generator=rnd)
    scales = torch.randint(1, 0x7f, (wide, 420), dtype=torch.uint8, device="cuda", generator=rnd)
    front = engine.Nvfp4Weight.from_device(codes, scales, 1e-3)
    zero, words = torch.zeros(6720, device="cuda"), torch.empty(wide, device="cuda")
    w = engine.Nvfp4Weight.from_device(codes[:n, :k // 2], scales[:n, :k // 16], 1e-3)
    a = engine.quantize_activations(torch.randn((m, k), device="cuda", generator=rnd).to(torch.bfloat16))
    want = engine.gemm_w4a4(w, *a, m)
    status = words.view(torch.int32)[-1:]
    c = torch.empty_like(want)
    for i in range(iters):
        c.fill_(float(i))
        words.view(torch.int32).fill_(9)
        engine.gemv_w4a16_f32(front, zero, out=words, kernel=engine.GEMV_SIMT)
        engine.gemm_w4a4(w, *a, m, out=c, status=status)
        assert int(status.item()) == 0 and torch.equal(c, want), i
    c.fill_(3.0)
    status.fill_(9)
    engine.gemm_w4a4(w, *a, m, out=c, status=status)
    assert int(status.item()) == 9 and bool((c == 3.0).all())
