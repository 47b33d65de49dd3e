"""Results of host-pointer calls around the sizes where they stop being written straight into host memory and are copied
instead, for the kernels that store single floats (affine 8-bit, any-shape Q4 and NVFP4, bf16) and those that store whole
lines; and that a large result of single floats does take the copy, which is about twice as fast."""
import time

import numpy as np
import pytest

from conftest import assert_bits_equal
from gpu_util import backend_mod, gpu

pytestmark = pytest.mark.gpu

_next = [0]


def _key():
    _next[0] += 1
    return 0x53000000 + _next[0]


def _q8(rng, synth, R, C):
    groups = (R * C + 63) // 64
    v = rng.integers(0, 256, (R * C + 3) // 4 * 4, dtype=np.uint8).view(np.uint32)
    return v, synth.bf16_round(rng.uniform(0.001, 0.002, groups).astype(np.float32)), \
        synth.bf16_round(rng.uniform(-0.2, -0.1, groups).astype(np.float32))


def _any_q4(rng, synth, R, C):
    """Q4 tensor of any shape: groups run on over the rows."""
    groups = (R * C + 63) // 64
    v = rng.integers(0, 1 << 32, (R * C + 7) // 8, dtype=np.uint32)
    return v, synth.bf16_round(rng.uniform(0.005, 0.02, groups).astype(np.float32)), \
        synth.bf16_round(rng.uniform(-0.1, -0.05, groups).astype(np.float32))


@pytest.mark.parametrize("R", [4096, 8191, 8192, 8193])
def test_single_floats(orc, synth, R):
    g, rng = gpu(), np.random.default_rng(R)
    g.set_mapped_only(0)
    x, y = rng.standard_normal(72).astype(np.float32), np.zeros(R, np.float32)
    t = _any_q4(rng, synth, R, 72)
    xs, ys = rng.standard_normal((2, 72)).astype(np.float32), np.zeros((2, R), np.float32)
    assert g.proj_batch(*t, R, 72, xs, ys, _key()) == 0
    for k in range(2):
        assert_bits_equal(ys[k], orc.q4_matvec(*t, R, 72, xs[k]), f"q4 {R} x 72")
    t = _q8(rng, synth, R, 72)
    assert g.q8_batch([t[0]], [t[1]], [t[2]], [x], [y], [_key()], [R], 72) == 0
    assert_bits_equal(y, orc.q8_matvec(*t, R, 72, x), f"q8 {R} x 72")
    W = (rng.standard_normal((R, 72)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    bm, key = backend_mod(), _key()
    assert g.weight_resource_bind(bm.RESOURCE_TRUNK, 5300 + R, W) == 0
    assert g.bf16_resource_slot(bm.RESOURCE_TRUNK, 5300 + R, key, W, R, 72) == 0
    assert g.bf16_matvec(key, R, 72, x, y) == 0
    assert_bits_equal(y, orc.bf16_matvec(W, R, 72, x), f"bf16 {R} x 72")
    assert g.bf16_matvec_batch(key, R, 72, 2, xs, ys) == 0
    assert_bits_equal(ys, orc.bf16_matvec_serial(W, R, 72, xs), f"bf16 batch {R} x 72")
    assert g.weight_resource_unbind(bm.RESOURCE_TRUNK, 5300 + R) == 0


@pytest.mark.parametrize("R,B,C", [(4095, 2, 48), (4096, 2, 48), (4097, 2, 48), (4097, 2, 256), (32768, 4, 256), (32769, 4, 256)])
def test_nvfp4(orc, synth, R, B, C):
    g, bm = gpu(), backend_mod()
    rng = np.random.default_rng(R + C)
    packed, scales, divisor = synth.make_nvfp4(rng, R, C)
    buf = np.concatenate([packed.reshape(-1), scales.reshape(-1), np.zeros(-(R * C // 16) % 4, np.uint8),
                          np.array([divisor, 64.0], np.float32).view(np.uint8)])
    p, s, key = buf[:R * C // 2], buf[R * C // 2:R * C // 2 + R * C // 16], _key()
    assert g.weight_resource_bind(bm.RESOURCE_EXPERT_LAYER, 5299, buf) == 0
    assert g.nvfp4_resource_slot(bm.RESOURCE_EXPERT_LAYER, 5299, key, p, s, buf[-8:-4], buf[-4:], R, C) == 0
    xs, ys = rng.standard_normal((B, C)).astype(np.float32), np.zeros((B, R), np.float32)
    assert g.nvfp4_matvec_batch(key, R, C, xs, ys) == 0
    for t in range(B):
        rc, want = orc.nvfp4_matvec(p.reshape(R, C // 2), s.reshape(R, C // 16), float(divisor), 64.0, R, C, xs[t], threads=4)
        assert rc == 0
        assert_bits_equal(ys[t], want, f"nvfp4 {R}x{C} token {t} of {B}")
    assert g.weight_resource_unbind(bm.RESOURCE_EXPERT_LAYER, 5299) == 0


@pytest.mark.parametrize("group,routed", [(1, 96), (2, 64), (24, 72), (24, 128)])
def test_chain(orc, synth, group, routed):
    """Both store forms behind one chain, below and above the line of single floats."""
    g, bm, H = gpu(), backend_mod(), 192
    rng = np.random.default_rng(group * 100 + routed)
    t = [_any_q4(rng, synth, r, c) for r, c in ((routed, H), (routed, H), (H, routed))]
    x, y = rng.standard_normal((2 * group, H)).astype(np.float32), np.zeros((2 * group, H), np.float32)
    fields = []
    for v, s, b in t:
        fields += [v.ctypes.data, s.ctypes.data, b.ctypes.data, _key()]
    g.set_mapped_only(0)
    assert g.q4_moe_chain([bm.MoeExpert(*fields, group, -1, 0)] * 2, H, routed, x, y) == 0
    for i in range(2 * group):
        gate, up = (orc.q4_matvec(*t[k], routed, H, x[i]) for k in range(2))
        mid = np.array([orc.gelu_tanh(v) for v in gate], np.float32) * up
        assert_bits_equal(y[i], orc.q4_matvec(*t[2], H, routed, mid), f"row {i}")


def _best_us(call):
    assert call() == 0
    best = 1e9
    for _ in range(40):
        t0 = time.perf_counter()
        call()
        best = min(best, time.perf_counter() - t0)
    return best * 1e6


def test_large_results_of_single_floats_are_copied(synth):
    """131072 results: 207 to 229 us written one by one over the bus, 80 to 130 copied; the same results as whole lines take
    40 to 50, which is the measure of the host at hand."""
    g, rng, R = gpu(), np.random.default_rng(1), 131072
    g.set_mapped_only(0)
    y = np.zeros(R, np.float32)
    keep = _any_q4(rng, synth, R, 64), _any_q4(rng, synth, R, 72), _q8(rng, synth, R, 64)
    x = rng.standard_normal(72).astype(np.float32)
    lines = _best_us(lambda: g.q4_matvec(*keep[0], R, 64, x[:64], y))
    single = _best_us(lambda: g.q4_matvec(*keep[1], R, 72, x, y)), _best_us(lambda: g.q8_matvec(*keep[2], R, 64, x[:64], y))
    print(f"whole lines {lines:.1f} us, any-shape q4 {single[0]:.1f} us, q8 {single[1]:.1f} us")
    assert single[0] < 3.0 * lines and single[1] < 4.0 * lines
