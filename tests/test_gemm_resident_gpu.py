"""Projections whose operand is made in shared memory (gemm_resident.cu): chains of a decode work list and single decode
projections, activations as octal digits.  Against 64-bit sums of the same products: the sums are fp32, so after the BF16
rounding an output differs by a flipped rounding at most, relative L2 below 2e-4 over many outputs (a few in 10^4 values by one
step of 2^-8) and below 2^-8 for one."""
import pytest

pytestmark = pytest.mark.gpu

E2M1 = [0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0]


def _weight(engine, torch, gen, n, k, gate_up=False):
    codes = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen)
    scales = torch.randint(0, 0x7f, (n, k // 16), dtype=torch.uint8, device="cuda", generator=gen)
    table = torch.tensor(E2M1 + [-v for v in E2M1], dtype=torch.float64, device="cuda")
    sb = scales.to(torch.int64)
    decoded = torch.where(sb < 8, (sb & 7) * 2.0 ** -9, (8 + (sb & 7)) * torch.pow(2.0, ((sb >> 3) - 10).double()))
    w = torch.stack([table[(codes & 15).long()], table[(codes >> 4).long()]], dim=2).view(n, k) * decoded.repeat_interleave(16, dim=1)
    return (codes, scales), w * 2.0 ** -12


def _rel(y, want):
    import torch

    want = want.to(torch.bfloat16).double()
    return ((y.double() - want).norm() / want.norm().clamp_min(1e-300)).item()


def _limit(count):
    return 2e-4 if count >= 1000 else 2.0 ** -8


def _run(engine, torch, items, m, launches):
    batch = engine.GemvBatch(items, m)
    engine.lib().q35b_debug_gemv_batch_chain(batch._h)  # sizes at which one launch of the other kernel is the faster one, too
    before = engine.launch_count()
    batch.run()
    assert engine.launch_count() - before == launches
    first = [it[2].clone() for it in items]
    batch.run()
    torch.cuda.synchronize()
    assert batch.status() == 0 and all(torch.equal(a.view(torch.int16), it[2].view(torch.int16)) for a, it in zip(first, items))
    return batch


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("n,k", [(1, 256), (127, 512), (130, 1280), (640, 9216), (2600, 2560)])
def test_one_item(engine, m, n, k):
    """Rows around a tile, splits from one to eight CTAs (also uneven ones), a residual, activations over the range of a token."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(m + n)
    (codes, scales), wd = _weight(engine, torch, gen, n, k)
    w = engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -12)
    for kind in range(4):
        x = torch.randn((m, k), device="cuda", generator=gen)
        if kind == 1:
            x *= torch.exp2(torch.randint(-30, 30, (m, k), device="cuda", generator=gen).float())
        if kind == 2:
            x *= 2.0 ** -110
            x[0] *= 0.0 if m > 1 else 1.0
        if kind == 3:
            x[:, k // 2:] *= 2.0 ** -60  # CTAs of a cluster that count in units far apart
        x = x.to(torch.bfloat16)
        res = torch.randn((m, n), device="cuda", generator=gen).to(torch.bfloat16) if kind == 0 else None
        y = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
        _run(engine, torch, [(w, x, y, res)], m, 1)
        assert _rel(y, x.double() @ wd.T + (res.double() if res is not None else 0.0)) <= _limit(m * n), kind


@pytest.mark.parametrize("m", [1, 2, 4, 6])
@pytest.mark.parametrize("hidden,inter", [(256, 256), (768, 2304), (2560, 3584)])
def test_chain(engine, m, hidden, inter):
    """Gate/up, then down reading its output: one launch each, replayed from a graph too."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(m)
    (gc, gs), gd = _weight(engine, torch, gen, inter, hidden)
    (uc, us), ud = _weight(engine, torch, gen, inter, hidden)
    (dc, ds), dd = _weight(engine, torch, gen, hidden, inter)
    gate_up = engine.Nvfp4Weight.gate_up_from_host(*(t.cpu().numpy() for t in (gc, gs)), 2.0 ** -12, *(t.cpu().numpy() for t in (uc, us)), 2.0 ** -13)
    x = (torch.randn((m, hidden), device="cuda", generator=gen) * 2.0 ** -4).to(torch.bfloat16)
    res = torch.randn((m, hidden), device="cuda", generator=gen).to(torch.bfloat16)
    h = torch.zeros((m, inter), dtype=torch.bfloat16, device="cuda")
    y = torch.zeros((m, hidden), dtype=torch.bfloat16, device="cuda")
    batch = _run(engine, torch, [(gate_up, x, h), (engine.Nvfp4Weight.from_device(dc, ds, 2.0 ** -12), h, y, res, 0)], m, 2)
    gate, up = x.double() @ gd.T, x.double() @ ud.T / 2
    assert _rel(h, gate / (1 + torch.exp(-gate)) * up) <= 1e-3  # the sigmoid in fp32 before the product is rounded
    assert _rel(y, h.double() @ dd.T + res.double()) <= _limit(m * hidden)
    kept = y.clone()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(3):
                batch.run()
        y.zero_()
        graph.replay()
        stream.synchronize()
    assert batch.status() == 0 and torch.equal(y, kept)


@pytest.mark.parametrize("m", [1, 2, 4, 8])
@pytest.mark.parametrize("n,k", [(2500, 4160), (1300, 7232), (9000, 2624), (2560, 9216)])
def test_single_projections(engine, m, n, k):
    """What AUTO chooses, K ending anywhere in a K step."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(m)
    (codes, scales), wd = _weight(engine, torch, gen, n, k)
    w = engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -12)
    x = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)
    want = x.double() @ wd.T
    assert _rel(engine.gemv_w4a16(w, x), want) <= 2e-4
    assert _rel(engine.gemv_w4a16(w, x, kernel=engine.GEMV_SIMT), want) <= 2e-4


@pytest.mark.parametrize("depth", [18, 24, 37])
@pytest.mark.parametrize("m", [1, 3, 6])
def test_small_values_beside_large_ones(engine, m, depth):
    """Where the weights of a row are zero at the large values of every block, the small ones are all it has."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(depth)
    n, k = 300, 2560
    (codes, scales), wd = _weight(engine, torch, gen, n, k)
    codes[:, ::8] &= 0xf0  # the first element of every block
    wd[:, ::16] = 0.0
    w = engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -12)
    x = torch.randn((m, k), device="cuda", generator=gen) * 2.0 ** -depth
    x[:, ::16] = 1.0
    x = x.to(torch.bfloat16)
    y = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
    _run(engine, torch, [(w, x, y)], m, 1)
    # multiples of 2^-40 of the block's largest binade: half of one per value, against values of 2^-depth
    assert _rel(y, x.double() @ wd.T) <= max(4e-3, 2.0 ** (depth - 39))


@pytest.mark.parametrize("large,small", [(0, -33), (0, -41), (3, -60), (100, -100), (127, -133), (17, -133)])
@pytest.mark.parametrize("m,n,k", [(1, 2500, 4160), (2, 2560, 9216), (4, 9000, 2624), (5, 1300, 7232), (8, 2500, 4160)])
def test_nothing_of_an_activation_is_lost(engine, m, n, k, large, small):
    """Values far below what fourteen digits beside the largest of their block hold, down to the smallest there is, in rows whose
    weights are zero at the large ones: the outputs are the sums of the small ones alone.  Also some small values in one token
    only, and one block of nothing else."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(m)
    (codes, scales), wd = _weight(engine, torch, gen, n, k)
    codes[:, ::8] &= 0xf0  # the first element of every block
    wd[:, ::16] = 0.0
    s2 = 2.0 ** min(-small, 30)
    w = engine.Nvfp4Weight.from_device(codes, scales, s2)
    for kind in range(3):
        x = torch.randn((m, k), device="cuda", generator=gen, dtype=torch.float64) * 2.0 ** small
        if kind == 1:
            x[: m - 1] *= 2.0 ** (min(large, 30) - small - 4)  # one token only
        if kind == 2:
            x[:, torch.rand(k, device="cuda", generator=gen) < 0.99] = 0.0
        x[:, ::16] = 2.0 ** large
        x[:, 32:48] = 2.0 ** small
        x = x.to(torch.bfloat16)
        want = x.double() @ (wd * 2.0 ** 12 * s2).T
        assert _rel(engine.gemv_w4a16(w, x), want) <= 1e-3, kind
        if k % 256 == 0 and m <= 6:
            y = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
            _run(engine, torch, [(w, x, y)], m, 1)
            assert _rel(y, want) <= 1e-3, kind


@pytest.mark.parametrize("m", [1, 4])
def test_infinities_and_nans(engine, m):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(m)
    n, k = 400, 2560
    (codes, scales), wd = _weight(engine, torch, gen, n, k)
    codes[:200, 350] &= 0xf0  # zero weights at column 700
    w = engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -12)
    for places in ([(700, float("inf"))], [(5, float("-inf")), (2500, float("inf"))], [(1000, float("nan"))]):
        x = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)
        for at, v in places:
            x[m - 1, at] = v
        y = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
        _run(engine, torch, [(w, x, y)], m, 1)
        want = engine.gemv_w4a16(w, x, kernel=engine.GEMV_SIMT)
        assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y[want.isinf()], want[want.isinf()])
        assert _rel(y[want.isfinite()], want[want.isfinite()].double()) <= 4e-3 if bool(want.isfinite().any()) else True


@pytest.mark.parametrize("m,hidden,inter", [(1, 256, 256), (2, 2560, 9216), (5, 512, 4096)])
def test_a_run_that_gives_up_leaves_a_list_that_works(engine, m, hidden, inter):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(m)
    (uc, us), _ = _weight(engine, torch, gen, inter, hidden)
    (dc, ds), _ = _weight(engine, torch, gen, hidden, inter)
    x = torch.randn((m, hidden), device="cuda", generator=gen).to(torch.bfloat16)
    h = torch.zeros((m, inter), dtype=torch.bfloat16, device="cuda")
    y = torch.zeros((m, hidden), dtype=torch.bfloat16, device="cuda")
    batch = _run(engine, torch, [(engine.Nvfp4Weight.from_device(uc, us, 2.0 ** -16), x, h), (engine.Nvfp4Weight.from_device(dc, ds, 2.0 ** -16), h, y, None, 0)], m, 2)
    good = y.clone()
    for limit in (1, 2, 5, 20, 100):
        batch.debug_wait(limit, 0)
        for _ in range(3):
            batch.run()
        torch.cuda.synchronize()
        assert batch.status() == 0 or 51 <= batch.status() <= 56
        batch.debug_wait(1 << 22, 0)
        y.zero_()
        batch.run()
        torch.cuda.synchronize()
        assert batch.status() == 0 and torch.equal(y, good)


@pytest.mark.parametrize("m,sizes", [(1, (300, 512, 700)), (2, (2560, 9216, 2560)), (4, (1024, 300 * 8, 512, 256))])
def test_what_runs_after_an_item_that_gave_up_stores_nothing(engine, m, sizes):
    """Every other row block of one item of a chain gives up: its other rows are stored, none of the later items' are (what they
    read would be an earlier run's), and the next run is right with nothing reset but the hook."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(m)
    sizes = [-(-n // 256) * 256 for n in sizes[:-1]] + [sizes[-1]]
    xs = [torch.randn((m, sizes[0]), device="cuda", generator=gen).to(torch.bfloat16)]
    items = []
    for i, (k, n) in enumerate(zip(sizes, sizes[1:])):
        (codes, scales), _ = _weight(engine, torch, gen, n, k)
        xs.append(torch.zeros((m, n), dtype=torch.bfloat16, device="cuda"))
        items.append((engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -18), xs[i], xs[i + 1], None) + ((i - 1,) if i else ()))
    batch = _run(engine, torch, items, m, len(items))
    good = [x.clone() for x in xs[1:]]
    for item in range(len(items)):
        batch.debug_wait(4096, 0)
        batch.debug_absent(item)
        for x in xs[1:]:
            x.fill_(7.0)
        for _ in range(2):
            batch.run()
        torch.cuda.synchronize()
        assert batch.status() == 53
        for i, (x, want) in enumerate(zip(xs[1:], good)):
            gave = (torch.arange(x.shape[1], device="cuda") // 128 % 2 == 0) if i == item else torch.full((x.shape[1],), i > item, device="cuda")
            assert bool((x[:, gave] == 7.0).all()) and torch.equal(x[:, ~gave], want[:, ~gave]), (item, i)
        batch.debug_wait(1 << 22, 0)
        batch.debug_absent(-1)
        batch.run()
        torch.cuda.synchronize()
        assert batch.status() == 0 and all(torch.equal(x, want) for x, want in zip(xs[1:], good))


def _resident(engine, torch, w, x, y, limit=1 << 20):
    stream = torch.cuda.current_stream().cuda_stream
    assert engine.lib().q35b_debug_gemv_resident(w.handle, x.data_ptr(), x.shape[0], y.data_ptr(), limit, stream) == 0


@pytest.mark.parametrize("m,n,k,resident", [(1, 2500, 4160, True), (4, 1300, 7232, True), (8, 9000, 2624, True), (2, 2560, 9216, True), (8, 2560, 9216, True), (1, 3584, 1024, False),
                                            (8, 300, 8192, False), (4, 1183, 6912, False), (4, 1300, 6912, True), (8, 4720, 4096, False), (2, 6072, 4352, False),
                                            (2, 15992, 6400, False), (1, 27760, 2816, False), (1, 16000, 4096, True), (5, 7048, 1280, False), (7, 7048, 1280, True)])
def test_which_kernel_a_single_projection_takes(engine, m, n, k, resident):
    """Both sides of each line of the rule, and the same sums."""
    import ctypes

    import torch

    gen = torch.Generator(device="cuda").manual_seed(m)
    (codes, scales), wd = _weight(engine, torch, gen, n, k)
    w = engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -12)
    taken = ctypes.c_int(-1)
    assert engine.lib().q35b_debug_gemv_auto(w.handle, m, ctypes.byref(taken)) == 0 and taken.value == resident
    x = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)
    assert _rel(engine.gemv_w4a16(w, x), x.double() @ wd.T) <= 2e-4


@pytest.mark.parametrize("m", [1, 7, 8])
@pytest.mark.parametrize("n,k", [(130, 192), (300, 4160), (1300, 7232), (257, 2624)])
def test_single_projections_over_the_range_of_activations(engine, m, n, k):
    """The resident kernel whatever AUTO says, at its most operand rows and with K ending inside a K step: tokens of wide range and of
    zeros; infinities and NaNs, among them in the last columns, as fp32 arithmetic has them; residues that differ from CTA to CTA."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(n)
    (codes, scales), wd = _weight(engine, torch, gen, n, k)
    codes[: n // 2, k // 2 - 1] &= 0x0f  # zero weights in the last column
    wd[: n // 2, k - 1] = 0.0
    w = engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -12)
    y = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
    for kind in range(3):
        x = torch.randn((m, k), device="cuda", generator=gen)
        if kind == 1:
            x *= torch.exp2(torch.randint(-60, 60, (m, k), device="cuda", generator=gen).float())
        if kind == 2:
            x[:, k // 2:] *= 2.0 ** -90
            x[0] *= 0.0 if m > 1 else 1.0
        x = x.to(torch.bfloat16)
        _resident(engine, torch, w, x, y)
        assert _rel(y, x.double() @ wd.T) <= _limit(m * n), kind
    for places in ([(k - 1, float("inf"))], [(k - 70 if k > 70 else 3, float("-inf")), (k - 1, float("inf"))], [(k - 1, float("nan"))], [(5, float("inf")), (k - 3, 2.0 ** 100)]):
        x = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)
        for at, v in places:
            x[m - 1, at] = v
        _resident(engine, torch, w, x, y)
        want = engine.gemv_w4a16(w, x, kernel=engine.GEMV_SIMT)
        assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y[want.isinf()], want[want.isinf()])
        finite = want.isfinite()
        assert not bool(finite.any()) or _rel(y[finite], want[finite].double()) <= 4e-3
    assert engine.gemm_default_status() == 0


def test_a_single_projection_that_gave_up_is_reported_and_stops_no_other_call(engine):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(1)
    m, n, k = 2, 700, 4160
    (codes, scales), wd = _weight(engine, torch, gen, n, k)
    w = engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -12)
    x = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)
    many = torch.randn((16, k), device="cuda", generator=gen).to(torch.bfloat16)
    good, prefill = engine.gemv_w4a16(w, x), [engine.project_prefill(w, v).clone() for v in (x, many)]
    y = torch.full((m, n), 7.0, dtype=torch.bfloat16, device="cuda")
    assert engine.gemm_default_status() == 0
    _resident(engine, torch, w, x, y, 1)
    torch.cuda.synchronize()
    assert bool((y == 7.0).all())
    # the code is not read yet
    assert all(torch.equal(engine.project_prefill(w, v), p) for v, p in zip((x, many), prefill))
    _resident(engine, torch, w, x, y)
    assert _rel(y, x.double() @ wd.T) <= 2e-4 and _rel(y, good.double()) <= 2e-4
    assert 51 <= engine.gemm_default_status() <= 56 and engine.gemm_default_status() == 0


@pytest.mark.parametrize("m,sizes,launches", [(2, (2560, 9216, 2560), 2), (4, (1024, 3584, 1024), 2), (6, (1024, 3584, 1024), 2), (4, (512, 1024, 512), 2),
                                             (4, (512, 768, 512), 1), (2, (5120, 5120, 5120), 2), (4, (5120, 5120, 5120), 1), (5, (1024, 1024, 1024), 1), (6, (2048, 12288, 2048), 1), (7, (1024, 3584, 1024), 1)])
def test_where_a_chain_is_one_launch_per_item(engine, m, sizes, launches):
    """Both sides of each line of the rule, with the same results."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(m)
    xs, items = [torch.randn((m, sizes[0]), device="cuda", generator=gen).to(torch.bfloat16)], []
    want = xs[0]
    for i, (k, n) in enumerate(zip(sizes, sizes[1:])):
        (codes, scales), wd = _weight(engine, torch, gen, n, k)
        xs.append(torch.zeros((m, n), dtype=torch.bfloat16, device="cuda"))
        items.append((engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -18), xs[i], xs[i + 1], None) + ((i - 1,) if i else ()))
        want = (want.double() @ wd.T * 2.0 ** -6).to(torch.bfloat16)
    batch = engine.GemvBatch(items, m)
    before = engine.launch_count()
    batch.run()
    assert engine.launch_count() - before == launches
    torch.cuda.synchronize()
    # an input of the second item that was rounded the other way, a few in 10^4, moves its outputs by 2^-9 of its share
    assert batch.status() == 0 and _rel(xs[-1], want.double()) <= 1e-3


@pytest.mark.parametrize("m,n,k,chain", [(1, 300, 4096, True), (2, 2560, 9216, True), (1, 9328, 8448, False), (4, 2560, 4096, True), (4, 9432, 2816, False), (6, 1024, 3584, True),
                                         (6, 9432, 2816, False), (4, 2048, 2048, True), (4, 2049, 2048, False), (1, 3584, 1024, False), (1, 1024, 1536, False)])
def test_which_kernel_a_list_of_one_item_takes(engine, m, n, k, chain):
    """Both sides of each line of the rule: only a chain takes the hook of one."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(m)
    (codes, scales), wd = _weight(engine, torch, gen, n, k)
    x = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)
    y = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
    batch = engine.GemvBatch([(engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -12), x, y)], m)
    batch.run()
    torch.cuda.synchronize()
    assert batch.status() == 0 and _rel(y, x.double() @ wd.T) <= _limit(m * n)
    assert (engine.lib().q35b_debug_gemv_batch_absent(batch._h, -1) == 0) == chain


@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("m,n,k", [(1, 64, 64), (3, 129, 5184), (4, 2100, 1344), (9, 471, 2432), (14, 1500, 320), (28, 300, 256), (2, 12500, 2816)])
def test_prefill_in_one_launch(engine, m, n, k, dtype):
    """Quantisation and projection of a small activation: outputs, codes, scales and scale word of the two launches, bit for
    bit; K ending anywhere in a K step, residuals on unaligned rows, zeros, infinities and NaNs among the activations."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(m + n)
    (codes, scales), _ = _weight(engine, torch, gen, n, k)
    w = engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -12)
    for kind in range(4):
        x = torch.randn((m, k), device="cuda", generator=gen)
        if kind == 1:
            x[:, ::100] *= 50.0
        if kind == 2:
            x *= 0.0
        if kind == 3:
            x[0, 3], x[-1, k - 1] = float("nan"), float("inf")
        x = x.to(torch.bfloat16 if dtype == "bf16" else torch.float32)
        res = torch.randn((m, n + 3), device="cuda", generator=gen).to(torch.bfloat16)[:, :n] if kind == 1 else None
        one, two = engine.act_scratch(m, k, x.device), engine.act_scratch(m, k, x.device)
        for t in one:
            t.fill_(3)
        a = engine.quantize_activations(x, scratch=two)
        before = engine.launch_count()
        got = engine.project_prefill(w, x, scratch=one, residual=res)
        assert engine.launch_count() - before == 1
        want = engine.gemm_w4a4(w, *a, m, residual=res)
        assert torch.equal(got.view(torch.int16), want.view(torch.int16)) or (kind == 3 and torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0)))
        assert all(torch.equal(p.view(torch.uint8), q.view(torch.uint8)) for p, q in zip(one, two))
    assert engine.gemm_default_status() == 0


def test_prefill_of_a_gate_up_weight_in_one_launch(engine):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(1)
    parts = [_weight(engine, torch, gen, 200, 576)[0] for _ in range(2)]
    host = [t.cpu().numpy() for p in parts for t in p]
    w = engine.Nvfp4Weight.gate_up_from_host(host[0], host[1], 2.0 ** -12, host[2], host[3], 2.0 ** -13)
    x = torch.randn((7, 576), device="cuda", generator=gen).to(torch.bfloat16)
    want = engine.gemm_w4a4(w, *engine.quantize_activations(x), 7)
    before = engine.launch_count()
    got = engine.project_prefill(w, x)
    assert engine.launch_count() - before == 1 and torch.equal(got, want)


@pytest.mark.parametrize("m,n,k,at", [(4, 1344, 1344, 0), (9, 2432, 2432, 0), (3, 129, 5184, 3 * 5184 - 8), (7, 640, 576, -3 * 640)])
def test_prefill_whose_output_lies_over_its_activations(engine, m, n, k, at):
    """All of x is read before anything is stored over it, so two launches; in place, over the last eight values, over the first
    rows."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(n)
    (codes, scales), _ = _weight(engine, torch, gen, n, k)
    w = engine.Nvfp4Weight.from_device(codes, scales, 2.0 ** -12)
    scratch = engine.act_scratch(m, k, "cuda")
    memory = torch.zeros(3 * m * (n + k), dtype=torch.bfloat16, device="cuda")
    begin = (m * n + 7) // 8 * 8
    x, out = memory[begin: begin + m * k].view(m, k), memory[begin + at: begin + at + m * n].view(m, n)
    for _ in range(5):
        value = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)
        engine.project_prefill(w, value, scratch=scratch)  # the stream's workspace
        before = engine.launch_count()
        want = engine.project_prefill(w, value, scratch=scratch)
        assert engine.launch_count() - before == 1
        x.copy_(value)
        before = engine.launch_count()
        got = engine.project_prefill(w, x, out=out, scratch=scratch)
        assert engine.launch_count() - before == 2
        assert torch.equal(got, want)
    assert engine.gemm_default_status() == 0


CAPTURED = """
import torch
import qwen35x_b200 as q
torch.manual_seed(0)
w = q.Nvfp4Weight.from_device(*q.quantize_weight(torch.randn((2560, 4160), device="cuda")))
xs = [torch.randn((m, 4160), device="cuda").to(torch.bfloat16) for m in (1, 4, 8)]
outs = [torch.empty((x.shape[0], 2560), dtype=torch.bfloat16, device="cuda") for x in xs]
torch.cuda.synchronize()
stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
with torch.cuda.stream(stream):
    with torch.cuda.graph(graph, stream=stream):
        for x, out in zip(xs, outs):
            q.gemv_w4a16(w, x, out=out)
    graph.replay()
    stream.synchronize()
    for x, out in zip(xs, outs):
        assert torch.equal(out, q.gemv_w4a16(w, x))
        assert float((out.double() - q.gemv_w4a16(w, x, kernel=q.GEMV_SIMT).double()).norm()) <= 1e-3 * float(out.double().norm())
assert q.gemm_default_status() == 0
"""


def test_the_first_single_projection_of_a_process_inside_a_capture():
    """The rule asks the runtime how many clusters fit, once per shape: also under capture."""
    import subprocess
    import sys
    from pathlib import Path

    r = subprocess.run([sys.executable, "-c", CAPTURED], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
