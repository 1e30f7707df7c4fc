"""Prefill projections whose sums do round: block scales over the whole E4M3 range on both sides, so that fp32 sums in
another order differ in their last bits and, here and there, in the BF16 rounding.  What must not change the order: the
row shard, the row stride of the output, the gather, the NVFP4 epilogue, and from 129 tokens on how many tokens there
are.  Bit for bit, against the unsharded projection of all tokens."""
import pytest

pytestmark = pytest.mark.gpu


def _operands(engine, m, n, k):
    import torch

    rnd = torch.Generator(device="cuda").manual_seed(m + n + k)
    codes = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=rnd)
    scales = torch.randint(8, 0x7f, (n, k // 16), dtype=torch.uint8, device="cuda", generator=rnd)
    x = torch.randn((m, k // 16, 16), device="cuda", generator=rnd)
    x = (x * torch.exp2(8 * torch.rand((m, k // 16, 1), device="cuda", generator=rnd) - 8)).view(m, k).to(torch.bfloat16)
    return codes, scales, x


@pytest.mark.parametrize("m,n,k,fewer", [(1024, 9216, 2560, (513, 300, 200, 129)), (512, 2560, 9216, (384, 200, 129)),
                                         (300, 512, 4096, (129,)), (128, 2560, 9216, ()), (40, 1024, 4096, ()), (7, 9216, 2560, ())])
def test_same_bits_however_it_is_dealt_out(engine, m, n, k, fewer):
    import torch

    codes, scales, x = _operands(engine, m, n, k)
    w = engine.Nvfp4Weight.from_device(codes, scales, 1e-4)
    a = engine.quantize_activations(x, 0.01)
    whole = engine.gemm_w4a4(w, *a, m)
    unaligned = torch.empty((m, n + 1), dtype=torch.bfloat16, device="cuda")[:, :n]
    engine.gemm_w4a4(w, *a, m, out=unaligned)
    assert torch.equal(unaligned, whole)
    for tokens in fewer:
        assert torch.equal(engine.gemm_w4a4(w, *engine.quantize_activations(x[:tokens], 0.01), tokens), whole[:tokens]), tokens
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for world in (2, 4):
        shards = [engine.Nvfp4Weight.from_device(codes, scales, 1e-4, shard_index=r, shard_count=world) for r in range(world)]
        assert torch.equal(torch.cat([engine.gemm_w4a4(s, *a, m) for s in shards], 1), whole), world
        buffers = [engine.PeerBuffer.create(m, n) for _ in range(world)]
        for r in range(world):
            engine.gemm_w4a4_allgather(shards[r], *a, m, buffers, r, 1, status, wait=False)
        for r in range(world):
            engine.peer_gather_wait(buffers, r, 1, status)
        assert int(status.item()) == 0 and all(torch.equal(b.tensor(), whole) for b in buffers), world
    assert engine.gemm_default_status() == 0


@pytest.mark.parametrize("m,inter,k", [(7, 4608, 4096), (40, 512, 4096), (100, 128, 4096), (7, 128, 4096), (100, 4608, 1024), (257, 192, 4096), (1100, 4608, 512)])
def test_nvfp4_epilogue_and_its_shards(engine, oracle, m, inter, k):
    """The gate/up projection that writes NVFP4 (splits 1 to 8 and the kernel of CTA pairs): the bytes of the quantiser
    applied to its own BF16 output, also when two shards fill them."""
    import torch

    codes, scales, x = _operands(engine, m, 2 * inter, k)
    halves = [t.cpu().numpy() for t in (codes[:inter], scales[:inter], codes[inter:], scales[inter:])]

    def weight(**shard):
        return engine.Nvfp4Weight.gate_up_from_host(halves[0], halves[1], 3e-6, halves[2], halves[3], 2e-6, **shard)

    a = engine.quantize_activations(x, 0.01)
    h = engine.gemm_w4a4(weight(), *a, m)
    scale = (h.float().abs().max() / 2688.0).reshape(1)
    want_codes, want_scales, _ = engine.quantize_activations(h, float(scale.item()))
    for world in (1, 2):
        scratch = engine.act_scratch(m, inter, x.device)
        for t in scratch[:2]:
            t.zero_()
        for r in range(world):
            w = weight(shard_index=r, shard_count=world)
            got_codes, got_scales, _ = engine.gemm_w4a4_gate_up_quant(w, *a, m, scale, scratch)
        assert torch.equal(got_codes, want_codes), world
        rows, cols = torch.arange(m, device="cuda")[:, None], torch.arange(inter // 16, device="cuda")[None, :]
        at = (((rows // 128) * (inter // 64) + cols // 4) * 32 + rows % 32) * 16 + (rows % 128) // 32 * 4 + cols % 4
        assert torch.equal(got_scales.reshape(-1)[at], want_scales.reshape(-1)[at]), world
    assert engine.gemm_default_status() == 0
