"""The prefill GEMM of CTA pairs (256 x 256 tiles), values of its epilogues on ragged problems: token and row counts that are
no multiple of a tile, rows narrower than the row stride, a K that ends inside a step, residual, gate/up.  Weight rows
sampled from both ends against the CPU oracle on the GPU quantiser's bytes (one BF16 rounding of an fp32 sum: relative L2
within 1e-3), and every element against the K-split kernel, which an output that is not 32-byte aligned takes: the sums
are the same fp32 additions, so BF16 results are at most one rounding step, 2^-7 of the value, apart."""
import numpy as np
import pytest

from helpers import from_torch_bf16, make_activations, to_torch_bf16

pytestmark = pytest.mark.gpu

REL_L2_TOL = 1e-3


def _weight(engine, n, k, seed):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(seed)
    return engine.quantize_weight(torch.randn((n, k), device="cuda", generator=gen) * 0.02)


def _sample(n):
    return np.unique(np.concatenate([np.arange(8), np.arange(n - 24, n), np.random.default_rng(n).choice(n, 24, replace=False)]))


def _outputs(engine, w, a, m, n, residual):
    """The kernel of CTA pairs on aligned rows, the K-split kernel on unaligned ones."""
    import torch

    ldc = (n + 15) // 16 * 16
    pairs = torch.full((m, ldc + 16), 7.0, dtype=torch.bfloat16, device="cuda")
    other = torch.zeros((m, n + 1 + n % 2), dtype=torch.bfloat16, device="cuda")
    assert engine.gemm_plan(m, w.rows, w.k)["pairs"] and not engine.gemm_plan(m, w.rows, w.k, rows_aligned=False)["pairs"]
    engine.gemm_w4a4(w, *a, m, out=pairs[:, :n], residual=residual)
    engine.gemm_w4a4(w, *a, m, out=other[:, :n], residual=residual)
    assert engine.gemm_default_status() == 0 and bool((pairs[:, n:] == 7.0).all())  # nothing past the last column
    got, ref = pairs[:, :n].float(), other[:, :n].float()
    assert bool(((got - ref).abs() <= 2.0 ** -7 * torch.maximum(got.abs(), ref.abs())).all())
    return from_torch_bf16(pairs[:, :n])


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("m,n,k", [(1100, 9216, 512), (1111, 9203, 320), (2049, 2570, 4672)])
def test_plain_and_residual(engine, oracle, m, n, k, residual):
    codes, scales, s2 = _weight(engine, n, k, seed=n + k)
    w = engine.Nvfp4Weight.from_device(codes, scales, s2)
    xb = make_activations(m, k, seed=m, outlier_frac=0.001)
    res = None
    if residual:
        import torch

        gen = torch.Generator(device="cuda").manual_seed(m)
        res = torch.randn((m, (n + 15) // 8 * 8), device="cuda", generator=gen).to(torch.bfloat16)[:, :n]
    got = _outputs(engine, w, engine.quantize_activations(to_torch_bf16(xb)), m, n, res)
    rows = _sample(n)
    e = oracle.quantize_nvfp4(xb)
    _, want = oracle.gemm_w4a4(codes.cpu().numpy()[rows], scales.cpu().numpy()[rows], s2, *e, threads=8)
    if residual:
        want = want + res.float().cpu().numpy()[:, rows]
    want = oracle.bf16_to_f32(oracle.bf16_round(want.astype(np.float32)))
    assert oracle.rel_l2(oracle.bf16_to_f32(got)[:, rows], want) <= REL_L2_TOL


@pytest.mark.parametrize("m,inter,k", [(1100, 4608, 512), (1111, 4600, 1024)])
def test_gate_up(engine, oracle, m, inter, k):
    gate, up = _weight(engine, inter, k, 1), _weight(engine, inter, k, 2)
    halves = [v.cpu().numpy() if hasattr(v, "cpu") else v for v in (*gate, *up)]
    w = engine.Nvfp4Weight.gate_up_from_host(*halves)
    xb = make_activations(m, k, seed=m, outlier_frac=0.001)
    got = _outputs(engine, w, engine.quantize_activations(to_torch_bf16(xb)), m, inter, None)
    rows = _sample(inter)
    e = oracle.quantize_nvfp4(xb)
    _, g = oracle.gemm_w4a4(halves[0][rows], halves[1][rows], halves[2], *e, threads=8)
    _, u = oracle.gemm_w4a4(halves[3][rows], halves[4][rows], halves[5], *e, threads=8)
    want = oracle.bf16_to_f32(oracle.bf16_round((g / (1 + np.exp(-g)) * u).astype(np.float32)))
    assert oracle.rel_l2(oracle.bf16_to_f32(got)[:, rows], want) <= REL_L2_TOL


@pytest.mark.parametrize("m,n,k", [(1100, 9216, 512), (1111, 9203, 320), (4096, 2560, 1024)])
def test_residual_in_place(engine, m, n, k):
    """The output over its residual, several tiles per CTA pair and a ragged last chunk: every box is read before it is written."""
    import torch

    codes, scales, s2 = _weight(engine, n, k, seed=n)
    w = engine.Nvfp4Weight.from_device(codes, scales, s2)
    assert engine.gemm_plan(m, n, k)["pairs"]
    a = engine.quantize_activations(to_torch_bf16(make_activations(m, k, seed=m)))
    res = torch.randn((m, (n + 15) // 8 * 8), device="cuda", generator=torch.Generator(device="cuda").manual_seed(m)).to(torch.bfloat16)
    want = torch.empty_like(res)
    engine.gemm_w4a4(w, *a, m, out=want[:, :n], residual=res[:, :n])
    for _ in range(5):
        both = res.clone()
        engine.gemm_w4a4(w, *a, m, out=both[:, :n], residual=both[:, :n])
        assert torch.equal(both[:, :n], want[:, :n]) and torch.equal(both[:, n:], res[:, n:])
    assert engine.gemm_default_status() == 0
