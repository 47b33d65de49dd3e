"""Rows at and beyond the widest that the tiled Q4 kernel holds in shared memory (25728 columns): the same bits from the
any-shape kernels, one matrix and gate with up, several tokens per job."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from gpu_util import backend_mod, gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [25728, 25792])
def test_wide_rows(orc, synth, C):
    g, bm, M, tokens = gpu(), backend_mod(), 64, 6
    rng = np.random.default_rng(C)
    g.set_mapped_only(0)
    key = 0x54000000 + C * 8
    gate, up, down = synth.make_q4(rng, M, C), synth.make_q4(rng, M, C), synth.make_q4(rng, C, M)
    x, y = rng.standard_normal((tokens, C)).astype(np.float32), np.zeros((tokens, M), np.float32)
    assert g.proj_batch(*gate, M, C, x, y, key) == 0
    gates = np.stack([orc.q4_matvec(*gate, M, C, x[t]) for t in range(tokens)])
    assert_bits_equal(y, gates, f"{M} x {C}")
    fields = []
    for i, (v, s, b) in enumerate((gate, up, down)):
        fields += [v.ctypes.data, s.ctypes.data, b.ctypes.data, key + 1 + i]
    out = np.zeros_like(x)
    assert g.q4_moe_chain([bm.MoeExpert(*fields, tokens, -1, 0)], C, M, x, out) == 0
    for t in range(tokens):
        mid = np.array([orc.gelu_tanh(v) for v in gates[t]], np.float32) * orc.q4_matvec(*up, M, C, x[t])
        assert_bits_equal(out[t], orc.q4_matvec(*down, C, M, mid), f"chain over {C} columns, token {t}")
