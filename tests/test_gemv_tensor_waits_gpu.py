"""Expired waits of decode lists on the tensor cores: a run whose waits are cut short records the code of one of them (41..45),
waits for its own copies and MMAs, and leaves everything so that the next run, with the usual limit, is right."""
import pytest

pytestmark = pytest.mark.gpu


def _list(engine, torch, kind, m):
    gen = torch.Generator(device="cuda").manual_seed(m)
    shapes = {"large": [(28672, 9216)], "few_tiles": [(384, 512), (130, 1280)], "one_step": [(128, 256)]}[kind]
    items = []
    for n, k in shapes:
        w = engine.Nvfp4Weight.from_device(torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen),
                                           torch.randint(0x20, 0x40, (n, k // 16), dtype=torch.uint8, device="cuda", generator=gen), 1e-3)
        x = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)
        items.append((w, x, torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")))
    return engine.GemvBatch(items, m, digits=0 if kind == "large" else 5), [y for _, _, y in items]


@pytest.mark.parametrize("kind", ["large", "few_tiles", "one_step"])
@pytest.mark.parametrize("m", [1, 8])
def test_a_run_that_gives_up_leaves_a_list_that_works(engine, kind, m):
    import torch

    batch, outputs = _list(engine, torch, kind, m)
    batch.run()
    torch.cuda.synchronize()
    want = [y.clone() for y in outputs]
    for limit in (1, 2, 5, 20, 100, 1000):
        batch.debug_wait(limit, 0)
        for _ in range(3):
            batch.run()
        torch.cuda.synchronize()
        code = batch.status()
        assert code == 0 or 41 <= code <= 45
        if limit == 1:
            assert code != 0
        batch.debug_wait(1 << 22, 0)
        for y in outputs:
            y.zero_()
        batch.run()
        torch.cuda.synchronize()
        assert batch.status() == 0
        assert all(torch.equal(y, e) for y, e in zip(outputs, want))
