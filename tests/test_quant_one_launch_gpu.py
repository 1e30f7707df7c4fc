"""The activation quantiser (amax, per-tensor scale and codes in one launch) where it can go wrong: BF16 values next to a
rounding boundary under every scale byte, scales at the ends of the multipliers' range, sizes around a CTA's share."""
import numpy as np
import pytest

from helpers import make_activations, to_torch_bf16
from test_quant_gpu import _run

pytestmark = pytest.mark.gpu

BOUNDARIES = np.array([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0])


def _beside_boundaries(g):
    """One row per scale byte 1..0x7e, its blocks holding the BF16 values around boundary * divisor, and as the last element
    the amax that makes the encoder choose the byte."""
    sb = np.arange(1, 0x7f)
    dec = np.where(sb < 8, (sb & 7) * 2.0 ** -9, (8 + (sb & 7)) * 2.0 ** ((sb >> 3) - 10.0)).astype(np.float32)
    d = dec * np.float32(g)
    x = np.zeros((len(sb), 64), dtype=np.uint16)
    at = (BOUNDARIES[None, :] * d[:, None].astype(np.float64)).astype(np.float32).view(np.uint32) >> 16  # rounded down to BF16
    for j, step in enumerate((0, 1, -1, 2)):
        v = (at.astype(np.int64) + step).clip(0, 0x7f7f).astype(np.uint16)
        v[:, j & 1:: 2] |= 0x8000
        x[:, 16 * j: 16 * j + 7] = v
        x[:, 16 * j + 8: 16 * j + 15] = v ^ 0x8000
        x[:, 16 * j + 15] = ((np.float32(6.0) * d).view(np.uint32) + 0x8000) >> 16
    return x


@pytest.mark.parametrize("exponent", [-62, -60, -20, -8, 0, 6, 7, 30, 60])
def test_values_next_to_every_boundary(engine, oracle, exponent):
    rng = np.random.default_rng(exponent + 100)
    # mantissas: a power of two and three quarters of one (every tie exact), then arbitrary ones
    for mant in [1.0, 1.5, 1.25 + 2.0 ** -20] + list(rng.uniform(1.0, 2.0, 12)):
        g = float(np.float32(mant) * np.float32(2.0) ** exponent)
        if abs(exponent) < 60 or mant == 1.0:
            _run(engine, oracle, _beside_boundaries(g), global_scale=g)


def test_boundary_values_where_a_bf16_value_is_closest(engine, oracle):
    """Per-tensor scales chosen so that a BF16 value lies within a few fp32 steps above boundary * divisor."""
    for n, off in [(4, 1), (5, 1), (6, 2), (7, 3), (4, -1), (5, -2), (6, 1), (7, -1)]:
        for top in (0x8100, 0x9300, 0xc700, 0xff00):
            mant = ((top << 8 << 2) - off) // n  # in units of 2^-23 (quarters divided out)
            while mant < (1 << 23):
                mant *= 2
            while mant >= (1 << 24):
                mant //= 2
            g = float(np.float32(mant) * np.float32(2.0 ** -30))
            _run(engine, oracle, _beside_boundaries(g), global_scale=g)


# 16-element blocks per row in multiples of four, rows padded to 128, 256 block slots per CTA and turn: one CTA's worth and a
# little more, rows that end inside a quad, a grid of several turns per thread (more than 148 * 4 * 256 slots per turn)
@pytest.mark.parametrize("m,k", [(4, 1024), (5, 1024), (129, 16), (1, 48), (130, 1040), (2000, 1552), (1300, 4112), (3000, 3072), (2400, 4096)])
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
def test_sizes_around_the_grid(engine, oracle, m, k, dtype):
    import torch

    xb = make_activations(m, k, seed=m * 7 + k)
    for scale in (0.0, 0.004):
        if dtype == "bf16":
            _run(engine, oracle, xb, global_scale=scale)
        else:
            xf = oracle.bf16_to_f32(xb) * np.float32(1.0009765)
            codes, scales, g = engine.quantize_activations(torch.from_numpy(xf).cuda(), scale)
            e_codes, e_scales, e_g = oracle.quantize_nvfp4(xf, scale)
            assert np.float32(g.item()) == np.float32(e_g)
            assert np.array_equal(codes.cpu().numpy(), e_codes) and np.array_equal(scales.cpu().numpy(), oracle.swizzle_scales(e_scales))


@pytest.mark.parametrize("bits", [0x7fc0, 0xffc0, 0x7f80, 0xff80, 0x0001, 0x8001, 0x7f7f])
def test_special_words_in_any_place(engine, oracle, bits):
    """NaN (skipped by the amax), infinities, the smallest and the largest value, at the first, a middle and the last element."""
    for at in (0, 1, 517, 2 * 1040 - 1):
        xb = make_activations(2, 1040, seed=at)
        xb.reshape(-1)[at] = bits
        for scale in (0.0, 0.01):
            _run(engine, oracle, xb, global_scale=scale)
