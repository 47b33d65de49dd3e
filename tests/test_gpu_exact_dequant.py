"""Affine-Q4 groups whose bias is far larger than the scale (groups of almost equal weights; a quantiser's least scale): the
weight fl(fl(q s) + b) keeps its two roundings.  A tile takes the one-rounding form only if all of its groups allow it, so
every group of a tensor is of the same kind."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from gpu_util import gpu

pytestmark = pytest.mark.gpu

_CASES = [(1.8046875, float.fromhex("0x1.74p-29")), (-1.71875, -float.fromhex("0x1.6ap-29")),
          (1.0, -float.fromhex("0x1.26p-24")), (1.0, -float.fromhex("0x1.2ap-28")), (-1.546875, float.fromhex("0x1.fcp-26")),
          (0.5, 1e-7), (1.0, 1e-7), (0.0078125, -1e-7), (1.0, 1e-30), (1e30, 1.0), (3.0, 0.0),
          # the lines of the rule: ratios around 2^22 and 2^-4, zeros, scales around 2^103
          (1.9921875, 2.0 ** -22), (1.0, 1.9921875 * 2.0 ** -23), (2.0 ** -10, 2.0 ** -6), (1.9921875 * 2.0 ** -11, -2.0 ** -6),
          (0.0, 0.013), (0.0, 0.0), (-7e30, 1e30), (-7e31, 1e31)]


@pytest.mark.parametrize("case", range(len(_CASES) + 4))
@pytest.mark.parametrize("B", [1, 2, 5])
def test_weights_near_a_large_bias(orc, synth, case, B):
    R, C = 65, 320
    rng = np.random.default_rng(case * 10 + B)
    groups = R * C // 64
    if case < len(_CASES):
        bias, scale = (np.full(groups, v, np.float32) for v in _CASES[case])
    else:                                          # random, a decade of ratios each
        bias = rng.uniform(1, 2, groups) * rng.choice((-1, 1), groups)
        scale = rng.uniform(1, 2, groups) * rng.choice((-1, 1), groups) * 2.0 ** -rng.integers(6 * (case - len(_CASES)) + 10,
                                                                                              6 * (case - len(_CASES)) + 16, groups)
    s, b = synth.bf16_round(scale.astype(np.float32)), synth.bf16_round(bias.astype(np.float32))
    v = rng.integers(0, 1 << 32, R * C // 8, dtype=np.uint32)
    xs, ys = rng.standard_normal((B, C)).astype(np.float32), np.zeros((B, R), np.float32)
    xs[:, 1:] = 0.0                                # the product with the first column shows its weight as it is
    xs[1:] = rng.standard_normal((B - 1, C)).astype(np.float32)
    g = gpu()
    g.set_mapped_only(0)
    assert g.proj_batch(v, s, b, R, C, xs, ys, 0x52000000 + case * 10 + B) == 0
    for t in range(B):
        assert_bits_equal(ys[t], orc.q4_matvec(v, s, b, R, C, xs[t]), f"case {case}, token {t} of {B}")
