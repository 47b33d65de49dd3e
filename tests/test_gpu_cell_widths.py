"""Exact cells at widths around the shared memory that a launch has without asking for more (rows and the in-order sum's scratch
together) and at the widest rows the cells take."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from gpu_util import backend_mod, gpu

pytestmark = pytest.mark.gpu

# (2 n + 8) floats of the norms, 2 n (padded to 4) + 8 of the post-norm and n + 8 of the combine, beside 5.2 KB
NORM = (5370, 5371, 5486, 5487, 5622, 5623, 6140, 8192, 25596)
POSTNORM = (5368, 5372, 5484, 5485, 5620, 6136, 6140, 6141, 25596)
COMBINE = (10744, 10745, 10972, 10973, 11244, 12280, 12281, 51192)


def _rows(n, count, seed):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal(n).astype(np.float32) for _ in range(count)]


@pytest.mark.parametrize("n", NORM)
def test_norms(orc, n):
    g, bm = gpu(), backend_mod()
    rc, buf = g.shared_buffer_alloc(4 * 3 * n)
    assert rc == 0
    f = buf.array(np.float32)
    x, w = _rows(n, 2, n)
    f[:n], f[n:2 * n] = x, w
    for kind, want in ((bm.EXACT_RMSNORM, orc.rmsnorm(x, w, 1e-6)), (bm.EXACT_ROUTER_INPUT, orc.router_input(x, w, 1e-6))):
        assert want[0] == 0
        assert g.exact_cells([bm.exact_cell(kind, [buf] * 3, [0, n, 2 * n], n, aux=1, eps=1e-6)]) == 0
        assert_bits_equal(f[2 * n:3 * n].copy(), want[1], f"cell {kind} of {n} columns")
    assert g.shared_buffer_free(buf) == 0


@pytest.mark.parametrize("n", POSTNORM)
def test_residual_postnorm(orc, n):
    g, bm = gpu(), backend_mod()
    rc, buf = g.shared_buffer_alloc(4 * 4 * n)
    assert rc == 0
    f = buf.array(np.float32)
    a = _rows(n, 3, n)
    for k in range(3):
        f[k * n:(k + 1) * n] = a[k]
    rc, want = orc.residual_postnorm(*a, 1e-6)
    assert rc == 0
    assert g.exact_cells([bm.exact_cell(bm.EXACT_RESIDUAL_POSTNORM, [buf] * 4, [0, n, 2 * n, 3 * n], n, eps=1e-6)]) == 0
    assert_bits_equal(f[3 * n:4 * n].copy(), want, f"residual cell of {n} columns")
    assert g.shared_buffer_free(buf) == 0


@pytest.mark.parametrize("n", COMBINE)
def test_parallel_combine(orc, n):
    g, bm = gpu(), backend_mod()
    rc, buf = g.shared_buffer_alloc(4 * 9 * n)
    assert rc == 0
    f = buf.array(np.float32)
    a = _rows(n, 6, n)
    for k in range(6):
        f[k * n:(k + 1) * n] = a[k]
    rc, want, _ = orc.parallel_ffn_combine(*a, 0.75, 1e-6)
    assert rc == 0
    cell = bm.exact_cell(bm.EXACT_PARALLEL_COMBINE, [buf] * 8, [k * n for k in range(7)] + [8 * n], n, eps=1e-6, scalar=0.75)
    assert g.exact_cells([cell]) == 0
    assert_bits_equal(f[8 * n:9 * n].copy(), want, f"combine cell of {n} columns")
    assert g.shared_buffer_free(buf) == 0


@pytest.mark.parametrize("n", [3, 64, 127, 128, 319, 575, 576, 577, 580, 640])
def test_sums_of_few_squares(orc, n):
    """One warp adds up to 576 squares in a row, with a tail of less than 64; above that the block adds them in pieces."""
    test_norms(orc, n)
    test_residual_postnorm(orc, n)
    test_parallel_combine(orc, n)


def test_wider_rows_are_refused():
    g, bm = gpu(), backend_mod()
    n = 51200
    rc, buf = g.shared_buffer_alloc(4 * 9 * n)
    assert rc == 0
    buf.array(np.float32)[:] = 1.0
    assert g.exact_cells([bm.exact_cell(bm.EXACT_RMSNORM, [buf] * 3, [0, n, 2 * n], 25600, aux=1, eps=1e-6)]) == -1
    assert g.exact_cells([bm.exact_cell(bm.EXACT_ROUTER_INPUT, [buf] * 3, [0, n, 2 * n], 25600, eps=1e-6)]) == -1
    assert g.exact_cells([bm.exact_cell(bm.EXACT_RESIDUAL_POSTNORM, [buf] * 4, [0, n, 2 * n, 3 * n], 25600, eps=1e-6)]) == -1
    cell = bm.exact_cell(bm.EXACT_PARALLEL_COMBINE, [buf] * 8, [k * n for k in range(7)] + [8 * n], n, eps=1e-6, scalar=0.75)
    assert g.exact_cells([cell]) == -1
    assert g.shared_buffer_free(buf) == 0


def test_counts_beyond_int_are_refused_on_the_host():
    """Cells whose element counts wrap around in 32 bits, over views that claim to be large enough: no launch, no access."""
    g, bm = gpu(), backend_mod()
    rc, buf = g.shared_buffer_alloc(4096)
    assert rc == 0
    claim = bm.SharedBuffer(buf.contents, 1 << 40, buf.backend)
    for kind in (bm.EXACT_RMSNORM, bm.EXACT_ROUTER_INPUT, bm.EXACT_RESIDUAL_POSTNORM, bm.EXACT_PARALLEL_COMBINE, bm.EXACT_SOFTCAP, bm.EXACT_TOPK):
        for n in (0x80000000, 0x80000004, 0xfffffffc, 0xffffffff):
            assert g.exact_cells([bm.exact_cell(kind, [claim] * 8, [0] * 8, n, aux=1, eps=1e-6, scalar=1.0)]) == -1, (kind, n)
    for kind in (bm.EXACT_RMSNORM, bm.EXACT_ROUTER_INPUT, bm.EXACT_RESIDUAL_POSTNORM, bm.EXACT_PARALLEL_COMBINE):
        for n in (0x40000000, 0x7ffffffd, 0x7fffffff):
            assert g.exact_cells([bm.exact_cell(kind, [claim] * 8, [0] * 8, n, aux=1, eps=1e-6, scalar=1.0)]) == -1, (kind, n)
    assert g.exact_cells([bm.exact_cell(bm.EXACT_TOPK, [claim] * 4, [0] * 4, (1 << 30) + 8, aux=1 << 30)]) == -1
    assert g.shared_buffer_free(buf) == 0
