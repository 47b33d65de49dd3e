"""A refused call leaves nothing behind: the next valid call of the thread does not report its error."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from gpu_util import backend_mod, gpu, stack_mod

pytestmark = pytest.mark.gpu


def test_valid_call_after_a_refused_allocation(orc):
    g, bm, n = gpu(), backend_mod(), 256
    rc, buf = g.shared_buffer_alloc(4 * 3 * n)
    assert rc == 0
    f = buf.array(np.float32)
    x = np.random.default_rng(5).standard_normal(n).astype(np.float32)
    f[:n], f[n:2 * n] = x, 1.0
    with pytest.raises(RuntimeError):                        # 550 GB of activations: the allocator's own refusal
        stack_mod().MoeStack(1 << 24, 8192, 64, 4, 2)
    assert g.exact_cells([bm.exact_cell(bm.EXACT_RMSNORM, [buf] * 3, [0, n, 2 * n], n, aux=1, eps=1e-6)]) == 0
    rc, want = orc.rmsnorm(x, np.ones(n, np.float32), 1e-6)
    assert_bits_equal(f[2 * n:].copy(), want, "norm after a refused call")
    assert g.shared_buffer_free(buf) == 0
