"""Large decode lists run on the tensor cores with every BF16 activation split into octal NVFP4 digits (gemm_wstream.cu): eight
of them, and six deep ones in the K steps where a value needs them.  No value loses anything down to 2^-38 of its token's
largest, so the outputs are those of 64-bit sums of the same products to fp32 accuracy: after the BF16 rounding they differ
in flipped roundings only, relative L2 below 2e-4 (a result flips where the fp32 error, some 2^-22 of the terms' size, spans
a rounding boundary 2^-9 wide: a few in 10^4 values by one step of 2^-8)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E2M1 = [0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0]


def _random_weight(engine, torch, gen, n, k, nan_scale=False):
    codes = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen)
    scales = torch.randint(0, 0x7f, (n, k // 16), dtype=torch.uint8, device="cuda", generator=gen)
    if nan_scale:
        scales[n // 2, 1] = 0x7f
    table = torch.tensor(E2M1 + [-v for v in E2M1], dtype=torch.float64, device="cuda")
    sb = scales.to(torch.int64)
    decoded = torch.where(sb < 8, (sb & 7) * 2.0 ** -9, (8 + (sb & 7)) * torch.pow(2.0, ((sb >> 3) - 10).double()))
    w = torch.stack([table[(codes & 15).long()], table[(codes >> 4).long()]], dim=2).view(n, k) * decoded.repeat_interleave(16, dim=1)
    return engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -12), w * 2.0 ** -12


def _filler(engine, torch, gen, m):
    """What makes a list large enough for the tensor cores: 142 MiB of weights nobody looks at."""
    n, k = 28672, 9216
    w = engine.Nvfp4Weight.from_device(torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen),
                                       torch.full((n, k // 16), 0x30, dtype=torch.uint8, device="cuda"), 1e-3)
    return w, torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16), torch.empty((m, n), dtype=torch.bfloat16, device="cuda")


def _run(engine, torch, items, m, launches=2):
    batch = engine.GemvBatch(items, m)
    before = engine.launch_count()
    batch.run()
    assert engine.launch_count() - before == launches
    batch.run()
    torch.cuda.synchronize()
    assert batch.status() == 0


def _rel(y, want):
    import torch

    want = want.to(torch.bfloat16).double()
    return ((y.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("m", [1, 2, 3, 5, 8])
def test_outputs(engine, m):
    """Rows around a tile, one and many K steps, a residual, activations over the whole range of a token, zeros."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(m)
    items, want = [_filler(engine, torch, gen, m)], [None]
    for j, (n, k) in enumerate([(1, 256), (127, 512), (129, 2560), (640, 9216), (256, 1024), (300, 768)]):
        w, wd = _random_weight(engine, torch, gen, n, k)
        x = torch.randn((m, k), device="cuda", generator=gen)
        if j == 2:
            x *= torch.exp2(torch.randint(-30, 30, (m, k), device="cuda", generator=gen).float())
        if j == 4:
            x[0] *= 0.0 if m > 1 else 1.0
            x[:, 16:32] *= 2.0 ** -100
        if j == 5:
            x *= 2.0 ** -110
        x = x.to(torch.bfloat16)
        res = torch.randn((m, n), device="cuda", generator=gen).to(torch.bfloat16) if j == 3 else None
        y = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
        items.append((w, x, y, res))
        want.append(x.double() @ wd.T + (res.double() if res is not None else 0.0))
    _run(engine, torch, items, m)
    for item, e in list(zip(items, want))[1:]:
        assert _rel(item[2], e) <= 2e-4, item[0].rows


def _below(torch, gen, m, k, where, depth):
    """Activations N(0, 1) whose columns `where` are 2^-depth of the token's largest value, which is a power of two."""
    x = torch.randn((m, k), device="cuda", generator=gen).clamp_(-3.9, 3.9)
    x[:, 0] = 4.0
    x[:, where] = torch.sign(x[:, where]) * (1.0 + torch.rand((m, len(where)), device="cuda", generator=gen)) * 2.0 ** (2 - depth)
    return x.to(torch.bfloat16)


# depth: of the values that decide the outputs, in powers of two below the token's largest; two K steps, and so many that the
# words that name the deep ones are more than one and more than a producer's 128 steps
@pytest.mark.parametrize("m", range(1, 9))
@pytest.mark.parametrize("k", [512, 9216, 33280])
def test_small_values_beside_large_ones_keep_their_bits(engine, m, k):
    """Weight rows that are zero except at small activations, which stand in the blocks of the large ones or in blocks of
    their own: every output for itself, against 64 bits.  An output is exact up to fp32 sums of a few terms, 2^-20 of their
    magnitudes, and its own BF16 rounding, half of a step of 2^-7 of its binade and so 2^-8 of it at most.  Some tokens of a list have such values and others have not, in this run and the one before."""
    import torch

    if m * (k + 32) * 2 > 150_000:
        k = 9216 - 256
    gen = torch.Generator(device="cuda").manual_seed(100 * m + k)
    blocks = k // 16
    inside = torch.arange(5, k, 16, device="cuda")[torch.randperm(blocks, device="cuda", generator=gen)[: blocks // 2]]
    alone = torch.arange(32, 48, device="cuda")
    rows = 130
    items, checks = [_filler(engine, torch, gen, m)] * (3 if k > 9216 else 1), []  # a share of the GPU has room for the long tiles
    for depth in (9, 15, 16, 17, 20, 24, 28, 31):
        for where in (inside, alone):
            codes = torch.zeros((rows, k), dtype=torch.uint8, device="cuda")
            # one to three of the small columns per row, in places that no other row shares
            pick = torch.randint(0, len(where), (rows, 3), device="cuda", generator=gen)
            codes.scatter_(1, where[pick], torch.randint(1, 8, (rows, 3), dtype=torch.uint8, device="cuda", generator=gen))
            packed = codes[:, 0::2] | codes[:, 1::2] << 4
            scales = torch.full((rows, k // 16), 0x38, dtype=torch.uint8, device="cuda")
            w = engine.Nvfp4Weight.from_device(packed.contiguous(), scales, 1.0)
            x = _below(torch, gen, m, k, where, depth)
            if m > 1:
                x[1::2] = torch.randint(-3, 4, (len(range(1, m, 2)), k), device="cuda", generator=gen).to(torch.bfloat16)
            y = torch.zeros((m, rows), dtype=torch.bfloat16, device="cuda")
            items.append((w, x, y))
            table = torch.tensor(E2M1, dtype=torch.float64, device="cuda")
            checks.append((x, y, table[codes.long()]))
    batch = engine.GemvBatch(items, m)
    before = engine.launch_count()
    for turn in range(3):
        batch.run()
        torch.cuda.synchronize()
        assert engine.launch_count() - before == 2 * (turn + 1) and batch.status() == 0
        for x, y, wd in checks:
            want = x.double() @ wd.T
            # the few terms of an output have the same size, so it is not far below their sum of magnitudes
            bound = 2.0 ** -8 * want.abs() + 2.0 ** -20 * (x.double().abs() @ wd.T)
            assert bool(((y.double() - want).abs() <= bound).all()), (turn, (y.double() - want).abs().max().item())
            if m > 1:
                x.copy_(x.roll(1, 0))  # other tokens have the small values in the next run


@pytest.mark.parametrize("m", [1, 4])
def test_infinities_and_nans(engine, m):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(7)
    w, wd = _random_weight(engine, torch, gen, 200, 512)
    for value in (float("inf"), float("-inf"), float("nan")):
        x = torch.randn((m, 512), device="cuda", generator=gen).to(torch.bfloat16)
        x[m - 1, 37] = value
        y = torch.zeros((m, 200), dtype=torch.bfloat16, device="cuda")
        _run(engine, torch, [_filler(engine, torch, gen, m), (w, x, y)], m)
        want = (x.double() @ wd.T).to(torch.bfloat16)
        same = (y == want) | (torch.isnan(y) & torch.isnan(want))
        assert bool(same[m - 1].all())
        if m > 1:
            assert _rel(y[: m - 1], want[: m - 1].double()) <= 2e-4


def test_gate_up(engine):
    import torch

    m, k, half = 3, 1024, 200
    gen = torch.Generator(device="cuda").manual_seed(11)
    gu, parts = [], []
    for _ in range(2):
        c = torch.randint(0, 256, (half, k // 2), dtype=torch.uint8, device="cuda", generator=gen)
        s = torch.full((half, k // 16), 0x38, dtype=torch.uint8, device="cuda")
        table = torch.tensor(E2M1 + [-v for v in E2M1], dtype=torch.float64, device="cuda")
        parts.append(torch.stack([table[(c & 15).long()], table[(c >> 4).long()]], dim=2).view(half, k) * 2.0 ** -6)
        gu += [c.cpu().numpy(), s.cpu().numpy(), 2.0 ** -6]
    x = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)
    y = torch.zeros((m, half), dtype=torch.bfloat16, device="cuda")
    _run(engine, torch, [_filler(engine, torch, gen, m), (engine.Nvfp4Weight.gate_up_from_host(*gu), x, y)], m)
    gate, up = x.double() @ parts[0].T, x.double() @ parts[1].T
    assert _rel(y, gate / (1 + torch.exp(-gate)) * up) <= 3e-4


@pytest.mark.parametrize("what", ["0x7f", "after", "small"])
def test_lists_that_stay_on_the_other_kernel(engine, what):
    """A scale byte that is NaN to the tensor cores (480 here), an item that waits for another one, few weights."""
    import torch

    m, gen = 2, torch.Generator(device="cuda").manual_seed(5)
    w, wd = _random_weight(engine, torch, gen, 256, 512, nan_scale=what == "0x7f")
    x = torch.randn((m, 512), device="cuda", generator=gen).to(torch.bfloat16)
    y = torch.zeros((m, 256), dtype=torch.bfloat16, device="cuda")
    items = [(w, x, y)] if what == "small" else [_filler(engine, torch, gen, m), (w, x, y)]
    if what == "after":
        w2, _ = _random_weight(engine, torch, gen, 128, 256)
        items.append((w2, y, torch.zeros((m, 128), dtype=torch.bfloat16, device="cuda"), None, 1))
    _run(engine, torch, items, m, launches=1)
    assert _rel(y, x.double() @ wd.T) <= 1e-3


def test_activations_too_large_for_the_other_kernel_stay_refused(engine):
    import torch

    n, k, m = 8192, 32768, 8
    w = engine.Nvfp4Weight.from_device(torch.zeros((n, k // 2), dtype=torch.uint8, device="cuda"),
                                       torch.full((n, k // 16), 0x30, dtype=torch.uint8, device="cuda"), 1.0)
    x, y = torch.zeros((m, k), dtype=torch.bfloat16, device="cuda"), torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
    items = [(w, x, y)] * 5  # 320 tiles of 128 steps: whole ones
    with pytest.raises(engine.Q35bError) as e:
        engine.GemvBatch(items, m)
    assert e.value.status == 2


@pytest.mark.parametrize("m", [1, 3, 8])
def test_outputs_of_infinities(engine, m):
    """An infinity times a weight is one of that sign, or a NaN where the weight or its block's scale is zero; two of opposite
    signs are a NaN.  Rows around a warp's 32, the first and last columns, infinities in every column, one and two K steps."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(17 + m)
    inf = float("inf")
    items, want = [_filler(engine, torch, gen, m)], []
    for j, (n, k) in enumerate([(33, 256), (127, 512), (160, 2560), (65, 512)]):
        codes = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen)
        scales = torch.randint(0, 0x7f, (n, k // 16), dtype=torch.uint8, device="cuda", generator=gen)
        x = torch.randn((m, k), device="cuda", generator=gen)
        if j == 0:
            x[0, 0], x[m - 1, k - 1] = inf, -inf
        elif j == 1:
            codes = codes % 7 * 16 + codes % 5 + 0x11 & 0x77  # no weight is zero or negative
            scales.clamp_(min=1)
            x[m - 1] = inf
            x[0, 300:] = -inf
        elif j == 2:
            scales[:, ::3] = 0
            x[m // 2, torch.randint(0, k, (3,), device="cuda", generator=gen)] = inf
            x[m // 2, 16 * 3] = -inf                           # under a scale of zero
        else:
            x[m - 1, 5], x[m - 1, 6], x[0, 7] = inf, float("nan"), -inf
        if j == 1 and m == 1:
            x[0] = inf
        table = torch.tensor(E2M1 + [-v for v in E2M1], dtype=torch.float64, device="cuda")
        sb = scales.to(torch.int64)
        decoded = torch.where(sb < 8, (sb & 7) * 2.0 ** -9, (8 + (sb & 7)) * torch.pow(2.0, ((sb >> 3) - 10).double()))
        w = torch.stack([table[(codes & 15).long()], table[(codes >> 4).long()]], dim=2).view(n, k)
        x = x.to(torch.bfloat16)
        y = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
        items.append((engine.Nvfp4Weight.from_device(codes.contiguous(), scales, 1.0), x, y))
        # products one by one: a matrix product may skip what it multiplies by zero
        want.append(((x.double()[:, None] * w[None]) * decoded.repeat_interleave(16, dim=1)[None]).sum(2))
    _run(engine, torch, items, m)
    for (_, x, y), e in zip(items[1:], want):
        bad = ~torch.isfinite(e)
        assert bool(bad.any()) and bool(torch.equal(torch.isnan(e), torch.isnan(y)))
        assert bool((y.double()[bad & ~torch.isnan(e)] == e[bad & ~torch.isnan(e)]).all())
        for t in range(m):
            if not bool(bad[t].any()):
                assert _rel(y[t], e[t]) <= 2e-4


def test_infinities_and_nans_cost_little(engine):
    """A list with such tokens takes about as long as one without; a serial sum over all columns per output took 10 times that."""
    import torch

    m, gen = 8, torch.Generator(device="cuda").manual_seed(3)
    w, x, y = _filler(engine, torch, gen, m)
    batch = engine.GemvBatch([(w, x, y)], m)

    def run():
        a, b = torch.cuda.Event(True), torch.cuda.Event(True)
        batch.run()
        a.record()
        for _ in range(20):
            batch.run()
        b.record()
        b.synchronize()
        return a.elapsed_time(b)

    finite = min(run() for _ in range(3))
    x[:, 1000] = float("inf")
    x[0, 1000] = float("nan")
    assert min(run() for _ in range(3)) <= 4 * finite and batch.status() == 0


# few long tiles, of which whole ones come out uneven over the SMs, and many; 128 MiB of weights and less
@pytest.mark.parametrize("shapes,launches", [([(20480, 16384)], 1), ([(8192, 16384)], 1), ([(2560, 9216)] * 16, 2),
                                             ([(32768, 2560)] * 4, 2), ([(32768, 2560)] * 2, 1), ([(1000, 4096)] * 64, 2)])
def test_lists_whose_whole_tiles_come_out_uneven_stay_on_the_other_kernel(engine, shapes, launches):
    import torch

    m, gen = 4, torch.Generator(device="cuda").manual_seed(4)
    items = []
    for n, k in shapes:
        w = engine.Nvfp4Weight.from_device(torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen),
                                           torch.full((n, k // 16), 0x30, dtype=torch.uint8, device="cuda"), 1e-3)
        items.append((w, torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16),
                      torch.empty((m, n), dtype=torch.bfloat16, device="cuda")))
    _run(engine, torch, items, m, launches=launches)


@pytest.mark.parametrize("m", [6, 7, 8])
def test_lists_of_short_tiles(engine, m):
    """Tiles of four K steps on average, from seven tokens on with another number of warps that take turns at the tokens: rows
    around a tile, a residual, one to four K steps, an infinity and a NaN in the last tokens."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(m)
    n, k = 28672, 1024
    w = engine.Nvfp4Weight.from_device(torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen),
                                       torch.full((n, k // 16), 0x30, dtype=torch.uint8, device="cuda"), 1e-3)
    items = [(w, torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16), torch.empty((m, n), dtype=torch.bfloat16, device="cuda")) for _ in range(10)]
    first = len(items)
    want = []
    for j, (n, k) in enumerate([(1, 256), (129, 1024), (300, 768), (640, 512), (256, 1024)]):
        w, wd = _random_weight(engine, torch, gen, n, k)
        x = torch.randn((m, k), device="cuda", generator=gen)
        if j == 2:
            x *= torch.exp2(torch.randint(-30, 30, (m, k), device="cuda", generator=gen).float())
        if j == 4:
            x[m - 1, 700], x[m - 2, 3] = float("inf"), float("nan")
        x = x.to(torch.bfloat16)
        res = torch.randn((m, n), device="cuda", generator=gen).to(torch.bfloat16) if j == 3 else None
        y = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
        items.append((w, x, y, res))
        want.append(x.double() @ wd.T + (res.double() if res is not None else 0.0))
    _run(engine, torch, items, m)
    for item, e in zip(items[first:], want):
        rows = m - 2 if item is items[-1] else m
        assert _rel(item[2][:rows], e[:rows]) <= 2e-4, item[0].rows
    last, e = items[-1][2].double(), want[-1]
    assert bool(torch.isnan(last[m - 2]).all()) and torch.equal(last[m - 1].nan_to_num(0.5), e[m - 1].nan_to_num(0.5))
