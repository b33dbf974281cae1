"""The NVFP4 quantizer's codes by a rounded quotient against the reference's chain of compares, on the CPU."""
import numpy as np
import pytest

BOUNDS = ((0.25, False), (0.75, True), (1.25, False), (1.75, True), (2.5, False), (3.5, True), (5.0, False))  # True: the bound itself counts
VALUES = np.array([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=np.float64)


def f32_fma(a, b, c):
    """a * b + c rounded once: a * b is exact in 64 bits, the sum of such a product and a near number too (residuals)."""
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(np.float32)


def nearest_even_code(q):
    """Nearest E2M1 value, ties to the even code, saturating: what the conversion instruction does."""
    q = q.astype(np.float64)
    mid = (VALUES[:-1] + VALUES[1:]) / 2
    code = (q[..., None] > mid).sum(-1)
    tie = (q[..., None] == mid).any(-1)
    return np.where(tie & (code % 2 == 1), code + 1, code)


@pytest.mark.parametrize("ex", range(16))
def test_rounded_quotient_gives_the_chains_codes(ex):
    man = np.arange(8 if ex < 15 else 7, dtype=np.float64)  # 448 is the largest scale
    scales = man / 512.0 if ex == 0 else (8.0 + man) / 8.0 * 2.0 ** (ex - 7)
    scales = scales[scales > 0].astype(np.float32)[:, None]
    # every float within 64 units of a bound, floats between the bounds, and the ends
    rng = np.random.default_rng(ex)
    bounds = np.array([b for b, _ in BOUNDS], dtype=np.float32)
    at = (scales * bounds)[..., None].view(np.int32) + np.arange(-64, 65, dtype=np.int32)
    m = [at.view(np.float32).reshape(len(scales), -1), scales * rng.uniform(0, 8, (len(scales), 20000)).astype(np.float32),
         np.broadcast_to(np.array([0, 1e-45, 1e-38, 1e-20, 1e20, 1e30], dtype=np.float32), (len(scales), 6))]
    m = np.concatenate(m, 1)
    want = sum(((m >= scales * np.float32(b)) if inclusive else (m > scales * np.float32(b))).astype(int) for b, inclusive in BOUNDS)
    inv = (np.float32(1.0) / scales).astype(np.float32)
    q0 = m * inv
    q1 = f32_fma(f32_fma(-q0, np.broadcast_to(scales, m.shape), m), np.broadcast_to(inv, m.shape), q0)
    assert np.array_equal(nearest_even_code(q1), want)
