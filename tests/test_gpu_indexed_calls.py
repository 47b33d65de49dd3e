"""Asynchronous indexed projections back to back: the rows of a call whose columns are no multiple of four leave the staging
cursor off a 16-byte boundary, from which the next call's rows were read in 16-byte pieces."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from gpu_util import gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [1, 66, 199])
def test_rows_after_a_ragged_call(orc, synth, first):
    g, rng = gpu(), np.random.default_rng(first)
    g.set_mapped_only(0)
    R, shapes = 33, (first, 64, first, 320)
    rc, out = g.shared_buffer_alloc(4 * 3 * R * len(shapes))
    assert rc == 0
    got, kept = out.array(), []
    got[:] = 0
    for i, C in enumerate(shapes):
        groups = (R * C + 63) // 64
        t = (rng.integers(0, 1 << 32, (R * C + 7) // 8, dtype=np.uint32),
             synth.bf16_round(rng.uniform(0.005, 0.02, groups).astype(np.float32)),
             synth.bf16_round(rng.uniform(-0.1, -0.05, groups).astype(np.float32)))
        x = rng.standard_normal((3, C)).astype(np.float32)
        assert g.proj_batch_indexed(*t, R, C, 3, 1, 1, x, out, i * 3 * R, 0x55000000 + first * 8 + i) == 0
        kept.append((t, x))
    assert g.sync() == 0
    for i, C in enumerate(shapes):
        t, x = kept[i]
        assert_bits_equal(got[(i * 3 + 1) * R:(i * 3 + 2) * R].copy(), orc.q4_matvec(*t, R, C, x[1]), f"call {i}: {C} columns")
    assert g.shared_buffer_free(out) == 0
