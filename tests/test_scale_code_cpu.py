"""The group scale code formed from max * float(1/6) equals the one from max / 6.

The prepare and the scaled weight quantisation use the product. It may differ from the quotient in the last bit, so the claim is
that no value which can be a group's maximum lies that close to a boundary of the UE4M3 codes: bf16 values, and residuals
x - q * s of at most 13 significant bits. Both are enumerated.
"""
import numpy as np
import torch

EPS, MAX = np.float32(2.0 ** -9), np.float32(448.0)


def _code(v):
    """UE4M3 bits of float32 values after the clamp of the kernels (round to nearest even)."""
    return torch.from_numpy(np.clip(v.astype(np.float32), EPS, MAX)).to(torch.float8_e4m3fn).view(torch.uint8).numpy()


def test_code_of_the_product_equals_code_of_the_quotient():
    significands = np.arange(2 ** 12, 2 ** 13, dtype=np.float32)  # every 13-bit significand
    for e in range(-30, 4):  # from below the smallest scale to above the largest (448 * 6 < 2^12)
        v = significands * np.float32(2.0 ** e)
        assert np.array_equal(_code(v * np.float32(1.0 / 6.0)), _code(v / np.float32(6.0))), e


def test_full_significands_can_differ():
    """The enumeration above can fail: some float32 values of 24 significant bits get another code."""
    v = np.arange(2 ** 23, 2 ** 24, dtype=np.float32)
    differ = [int((_code(v * np.float32(2.0 ** e) * np.float32(1.0 / 6.0)) != _code(v * np.float32(2.0 ** e) / np.float32(6.0))).sum())
              for e in range(-33, -10)]
    assert sum(differ) > 0


def _significant_bits(v):
    """Significant bits of non-zero float64 values that are exact."""
    m, _ = np.frexp(v)
    m = np.abs(m * 2.0 ** 53).astype(np.int64)
    return 53 - np.log2((m & -m).astype(np.float64))


def test_residuals_have_few_significant_bits():
    """x - q * s for every scale code and every bf16 x: at most 13 bits, or so large that the code saturates."""
    scales = torch.arange(1, 127, dtype=torch.uint8).view(torch.float8_e4m3fn).double().numpy()
    scales = scales[scales >= 2.0 ** -9]
    levels = np.array([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0])
    significands = np.arange(128, 256, dtype=np.float64)
    for s in scales:
        for e in range(int(np.floor(np.log2(s))) - 12, int(np.floor(np.log2(s))) + 8):
            x = significands * 2.0 ** (e - 7)
            at = np.clip(np.searchsorted(levels, x / s), 1, len(levels) - 1)
            low, high = levels[at - 1], levels[at]
            below, above = x / s - low, high - x / s
            # q is the nearest level; the kernel rounds x * (1 / s), so next to a tie it may be either
            for q, mine, other in ((low, below, above), (high, above, below)):
                r = (x - q * s)[mine <= other * (1 + 1e-5)]
                r = r[r != 0]
                ok = (_significant_bits(r) <= 13) | (np.abs(r) / 6 >= 448)
                assert ok.all(), (s, e, r[~ok][:4])
