"""Inputs replaced in place between calls that follow one another on a stream: every kernel is launched under the tail of the
one before it, and the words handed from kernel to kernel (a token's or tensor's scale, digits, codes) have the same
addresses in every call, so anything kept from the call before shows as an output that is wrong by a power of two or a NaN."""
import pytest

pytestmark = pytest.mark.gpu

FACTORS = [1.0, 2.0 ** 40, float("nan"), 2.0 ** -40, float("inf"), 1.0, 2.0 ** -100, 2.0 ** 90]


def _versions(torch, m, k, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for f in FACTORS:
        x = torch.randn((m, k), device="cuda", generator=gen)
        if f == f and f != float("inf"):
            x *= f
        else:
            x[m - 1, 3] = f
        out.append(x.to(torch.bfloat16))
    return out


def _same(torch, a, b):
    return bool(((a == b) | (torch.isnan(a) & torch.isnan(b))).all())


def _weight(engine, torch, n, k, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return engine.Nvfp4Weight.from_device(torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen),
                                          torch.randint(0x20, 0x40, (n, k // 16), dtype=torch.uint8, device="cuda", generator=gen), 1e-3)


@pytest.mark.parametrize("m,rows", [(1, 28672), (8, 28672), (2, 512)])
def test_decode_list(engine, m, rows):
    """A list on the tensor cores, and one on the other kernel."""
    import torch

    k = 9216
    w = _weight(engine, torch, rows, k, m)
    x, y = torch.empty((m, k), dtype=torch.bfloat16, device="cuda"), torch.empty((m, rows), dtype=torch.bfloat16, device="cuda")
    batch = engine.GemvBatch([(w, x, y)], m)
    versions = _versions(torch, m, k, m)
    want = []
    for v in versions:
        x.copy_(v)
        torch.cuda.synchronize()
        batch.run()
        torch.cuda.synchronize()
        want.append(y.clone())
    assert bool(torch.isnan(want[2][m - 1]).all()) and bool(torch.isfinite(want[3]).all()) and bool(want[0].any())
    for _ in range(10):
        got = []
        torch.cuda.synchronize()
        for v in versions:
            x.copy_(v)
            batch.run()
            got.append(y.clone())
        assert all(_same(torch, a, b) for a, b in zip(got, want))
    assert batch.status() == 0


@pytest.mark.parametrize("m", [16, 700])
def test_prefill(engine, m):
    import torch

    n, k = 2048, 1024
    w = _weight(engine, torch, n, k, 3)
    x, scratch = torch.empty((m, k), dtype=torch.bfloat16, device="cuda"), engine.act_scratch(m, k, "cuda")
    res = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    versions, residuals = _versions(torch, m, k, m), _versions(torch, m, n, m + 1)
    want = []
    for v, r in zip(versions, residuals):
        torch.cuda.synchronize()
        want.append(engine.project_prefill(w, v, residual=r).clone())
    for _ in range(10):
        got = []
        torch.cuda.synchronize()
        for v, r in zip(versions, residuals):
            x.copy_(v)
            res.copy_(r)
            got.append(engine.project_prefill(w, x, scratch=scratch, residual=res))
        assert all(_same(torch, a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("m", [1, 8])
def test_single_projection(engine, m):
    import torch

    n, k = 3584, 1024
    w = _weight(engine, torch, n, k, 5)
    x = torch.empty((m, k), dtype=torch.bfloat16, device="cuda")
    versions = _versions(torch, m, k, m)
    want = []
    for v in versions:
        torch.cuda.synchronize()
        want.append(engine.gemv_w4a16(w, v).clone())
    got = []
    for v in versions * 5:
        x.copy_(v)
        got.append(engine.gemv_w4a16(w, x))
    assert all(_same(torch, a, b) for a, b in zip(got, want * 5))


@pytest.mark.parametrize("m", [16, 300])
def test_prefill_reading_what_the_call_before_wrote(engine, m):
    """Two projections in a row, the second quantising the first one's output: nothing of it may be read before the first one's
    kernel, which lets its successor start early, is complete."""
    import torch

    k, n = 2560, 2048
    w1, w2 = _weight(engine, torch, n, k, 8), _weight(engine, torch, 512, n, 9)
    gen = torch.Generator(device="cuda").manual_seed(m)
    xs = [(torch.randn((m, k), device="cuda", generator=gen) * 4.0 ** i).to(torch.bfloat16) for i in range(8)]
    s1, s2 = engine.act_scratch(m, k, "cuda"), engine.act_scratch(m, n, "cuda")
    between = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    want = []
    for x in xs:
        torch.cuda.synchronize()
        engine.project_prefill(w1, x, out=between, scratch=s1)
        torch.cuda.synchronize()
        want.append(engine.project_prefill(w2, between, scratch=s2).clone())
    for _ in range(20):
        torch.cuda.synchronize()
        got = []
        for x in xs:
            engine.project_prefill(w1, x, out=between, scratch=s1)
            got.append(engine.project_prefill(w2, between, scratch=s2))
        assert all(_same(torch, a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("m,hidden,inter", [(1, 1024, 3584), (2, 2560, 9216), (4, 512, 4096)])
def test_decode_chain(engine, m, hidden, inter):
    """One launch per item, each started under the one before it: what the second one reads has the same address in every run, and
    none of it may be left from the run before."""
    import torch

    up, down = _weight(engine, torch, inter, hidden, 1), _weight(engine, torch, hidden, inter, 2)
    x, h, y = (torch.empty((m, n), dtype=torch.bfloat16, device="cuda") for n in (hidden, inter, hidden))
    res = torch.zeros((m, hidden), dtype=torch.bfloat16, device="cuda")
    batch = engine.GemvBatch([(up, x, h), (down, h, y, res, 0)], m)
    before = engine.launch_count()
    batch.run()
    assert engine.launch_count() - before == 2
    versions, residuals = _versions(torch, m, hidden, m), _versions(torch, m, hidden, m + 10)
    want = []
    for v, r in zip(versions, residuals):
        x.copy_(v)
        res.copy_(r)
        torch.cuda.synchronize()
        batch.run()
        torch.cuda.synchronize()
        want.append((h.clone(), y.clone()))
        plain = engine.gemv_w4a16(up, v, kernel=engine.GEMV_SIMT)
        assert _same(torch, want[-1][0].isfinite(), plain.isfinite())
        kept, ref = want[-1][0].nan_to_num(0.0, 0.0, 0.0).double(), plain.nan_to_num(0.0, 0.0, 0.0).double()
        assert float((kept - ref).norm()) <= 1e-3 * float(ref.norm())  # both fp32 sums: flipped roundings, a few in 10^4
    for _ in range(10):
        got = []
        torch.cuda.synchronize()
        for v, r in zip(versions, residuals):
            x.copy_(v)
            res.copy_(r)
            batch.run()
            got.append((h.clone(), y.clone()))
        assert all(_same(torch, a, b) for g, w in zip(got, want) for a, b in zip(g, w))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):  # run behind run, with nothing but the copies between
        got = []
        for v, r in zip(versions, residuals):
            x.copy_(v)
            res.copy_(r)
            batch.run()
            got.append((h.clone(), y.clone()))
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(_same(torch, a, b) for g, w in zip(got, want) for a, b in zip(g, w)) and batch.status() == 0
