"""Affine-Q4 projections of several tokens (q4_batch_kernel) at the edges of its tiles: row tails, chunk and group
remainders, every pass size, and groups whose bias rules the exact one-rounding dequantisation out."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from gpu_util import gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,C", [(1, 64), (63, 192), (64, 256), (65, 320), (130, 704), (33, 8192)])
@pytest.mark.parametrize("B", [2, 3, 4, 5, 9])
def test_batch_projection_vs_oracle(orc, synth, R, C, B):
    rng = np.random.default_rng(R * 1000 + C + B)
    v, s, b = synth.make_q4(rng, R, C)
    if B == 3:                                     # zero points close to zero, zero biases, negative scales
        b = b.copy()
        b[::3] = synth.bf16_round(np.float32(1e-5) * synth.bf16_to_f32(s[::3]))
        b[1::5] = 0
        s = s.copy()
        s[::7] ^= 0x8000
    xs = rng.standard_normal((B, C)).astype(np.float32)
    ys = np.zeros((B, R), np.float32)
    g = gpu()
    g.set_mapped_only(0)
    assert g.proj_batch(v, s, b, R, C, xs, ys, 0x51000000 + R * 100000 + C * 10 + B) == 0
    for t in range(B):
        assert_bits_equal(ys[t], orc.q4_matvec(v, s, b, R, C, xs[t]), f"{R}x{C} token {t} of {B}")


def test_single_token_of_a_wide_row(orc, synth):
    """More columns than the one-token kernel holds in shared memory."""
    rng = np.random.default_rng(17)
    R, C = 70, 12288
    v, s, b = synth.make_q4(rng, R, C)
    x, y = rng.standard_normal(C).astype(np.float32), np.zeros(R, np.float32)
    g = gpu()
    g.set_mapped_only(0)
    assert g.q4_matvec(v, s, b, R, C, x, y) == 0
    assert_bits_equal(y, orc.q4_matvec(v, s, b, R, C, x), "70 x 12288")
