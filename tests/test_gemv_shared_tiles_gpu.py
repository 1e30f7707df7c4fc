"""Decode work lists whose tiles are shared by several CTAs (fewer tiles than CTAs, or five to eight tokens): parts of two
K steps and of many, tiles of odd row counts, residuals, a gate/up weight, dependent items, both shapes of CTA, and runs
repeated on the same list (the parts' counters have to be back at zero).  Against the CPU oracle; the sums are fp32 in
another order, so a result differs by flipped BF16 roundings at most: relative L2 far below 2^-8 / sqrt(12) = 1.1e-3."""
import numpy as np
import pytest

from helpers import from_torch_bf16, make_activations, make_weight, to_torch_bf16

pytestmark = pytest.mark.gpu

REL_L2_TOL = 1e-3


def _rel_l2_rounded(oracle, got, want):
    return oracle.rel_l2(oracle.bf16_to_f32(from_torch_bf16(got)), oracle.bf16_to_f32(oracle.bf16_round(want.astype(np.float32))))


@pytest.mark.parametrize("m", [1, 2, 4, 5, 8])
@pytest.mark.parametrize("shapes", [[(1, 256)], [(130, 768)], [(257, 9216)], [(2560, 9216), (100, 512)], [(5000, 1280)] * 12])
def test_independent_items(engine, oracle, m, shapes):
    import torch

    items, host = [], []
    for j, (n, k) in enumerate(shapes):
        _, codes, scales, s2 = make_weight(n, k, seed=n + k + j)
        xb = make_activations(m, k, seed=j + 1, outlier_frac=0.001)
        res = torch.randn((m, n), generator=torch.Generator(device="cuda").manual_seed(j), device="cuda").to(torch.bfloat16) if j % 2 else None
        y = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
        items.append((engine.Nvfp4Weight.from_host(codes, scales, s2), to_torch_bf16(xb), y, res))
        host.append((codes, scales, s2, xb))
    batch = engine.GemvBatch(items, m)
    first = None
    for _ in range(3):
        for it in items:
            it[2].zero_()
        batch.run()
        assert batch.status() == 0
        bits = [from_torch_bf16(it[2]) for it in items]
        assert first is None or all(np.array_equal(a, b) for a, b in zip(first, bits))
        first = bits
    for (w, x, y, res), (codes, scales, s2, xb) in zip(items, host):
        _, ef = oracle.gemv_bf16(codes, scales, s2, xb, threads=8)
        want = np.asarray(ef) + (res.float().cpu().numpy() if res is not None else 0.0)
        assert _rel_l2_rounded(oracle, y, want) <= REL_L2_TOL


@pytest.mark.parametrize("m", [1, 3, 8])
@pytest.mark.parametrize("hidden,inter", [(256, 256), (512, 8192), (2560, 1280)])
def test_mlp_block(engine, oracle, m, hidden, inter):
    """gate/up with the SiLU epilogue, then down + residual reading its output, both shared; replayed from a graph too."""
    import torch

    _, gc, gs, g2 = make_weight(inter, hidden, seed=1)
    _, uc, us, u2 = make_weight(inter, hidden, seed=2)
    _, dc, ds, d2 = make_weight(hidden, inter, seed=3)
    xb = make_activations(m, hidden, seed=4)
    x, res = to_torch_bf16(xb), to_torch_bf16(make_activations(m, hidden, seed=5))
    h = torch.zeros((m, inter), dtype=torch.bfloat16, device="cuda")
    y = torch.zeros((m, hidden), dtype=torch.bfloat16, device="cuda")
    batch = engine.GemvBatch([(engine.Nvfp4Weight.gate_up_from_host(gc, gs, g2, uc, us, u2), x, h),
                              (engine.Nvfp4Weight.from_host(dc, ds, d2), h, y, res, 0)], m)
    batch.run()
    torch.cuda.synchronize()
    _, gate = oracle.gemv_bf16(gc, gs, g2, xb, threads=8)
    _, up = oracle.gemv_bf16(uc, us, u2, xb, threads=8)
    want_h = gate / (1.0 + np.exp(-gate.astype(np.float64))) * up
    assert _rel_l2_rounded(oracle, h, want_h) <= REL_L2_TOL
    _, ef = oracle.gemv_bf16(dc, ds, d2, from_torch_bf16(h), threads=8)
    want = np.asarray(ef) + res.float().cpu().numpy()
    assert _rel_l2_rounded(oracle, y, want) <= REL_L2_TOL
    kept = y.clone()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(3):
                batch.run()
        y.zero_()
        graph.replay()
        graph.replay()
        stream.synchronize()
    assert batch.status() == 0 and torch.equal(y, kept)


@pytest.mark.parametrize("m,hidden,inter", [(1, 512, 8192), (8, 512, 8192), (3, 512, 4096)])
@pytest.mark.parametrize("back_to_back", [False, True])
def test_list_recovers_from_an_expired_wait(engine, m, hidden, inter, back_to_back):
    """Every other CTA of a run gives up waiting for the gate/up item, so some parts of each of the down projection's tiles
    arrive and others do not.  Such a run reports it and stores none of these tiles, however many of them follow one
    another or start under one another's tail, and the next good ones, nothing reset but the limit, are right."""
    import torch

    _, gc, gs, g2 = make_weight(inter, hidden, seed=1)
    _, uc, us, u2 = make_weight(inter, hidden, seed=2)
    _, dc, ds, d2 = make_weight(hidden, inter, seed=3)
    x = to_torch_bf16(make_activations(m, hidden, seed=4))
    h = torch.zeros((m, inter), dtype=torch.bfloat16, device="cuda")
    y = torch.zeros((m, hidden), dtype=torch.bfloat16, device="cuda")
    batch = engine.GemvBatch([(engine.Nvfp4Weight.gate_up_from_host(gc, gs, g2, uc, us, u2), x, h),
                              (engine.Nvfp4Weight.from_host(dc, ds, d2), h, y, None, 0)], m)
    batch.run()
    assert batch.status() == 0
    good = y.clone()
    for _ in range(4):
        batch.debug_wait(4096, 1)
        y.zero_()
        for _ in range(4 if back_to_back else 1):
            batch.run()
        assert batch.status() == 15 and not bool(y.any())
    batch.debug_wait(1 << 22, 0)
    for _ in range(3):
        y.zero_()
        batch.run()
        assert batch.status() == 0 and torch.equal(y, good)
