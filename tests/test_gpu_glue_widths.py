"""The row-wise glue (reduce, RMSNorm, router input) at batches of several hundred rows: which form a batch takes follows from
its size and the row's width alone, and both forms give the oracle's bits at widths that end anywhere in a warp's share."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from gpu_util import d2h, stack_mod
from graph_util import captured_kernels

pytestmark = pytest.mark.gpu

SMS = 148


def _line(n):
    """Most rows that the block form takes with two in-order sums."""
    return (4 if n <= 1024 else 1 if n <= 1664 else 2 if n <= 5120 else 3) * SMS


def _stack(synth, n, rows, norm=True, topk=2):
    experts = max(4, topk)
    st = stack_mod().MoeStack(rows, n, 64, experts, topk)
    layers = [synth.make_q4_moe_layer(800 + n + i, hidden=n, inter=64, n_experts=experts, topk=topk) for i in range(2)]
    for layer in layers:
        layer.router_scale[:] = 1.0 + 0.01 * np.arange(n) / n
        st.add_layer(layer, with_norm=norm)
    return st, layers


@pytest.mark.parametrize("n", [64, 192, 256, 320, 1024, 1088, 2048, 2816, 2880, 3072, 3328, 4096, 5056, 6144])
@pytest.mark.parametrize("extra", [0, 1, 6])
def test_rows_vs_oracle(orc, synth, n, extra):
    rows = _line(n) + extra                                  # the line, and row remainders above it
    st, layers = _stack(synth, n, rows)
    import torch
    x = synth.make_tokens(801 + n, rows, n)
    d_x, d_y = torch.from_numpy(x).cuda(), torch.zeros(rows, n, device="cuda")
    assert st.layer_experts(0, d_x.data_ptr(), rows) == 0
    assert st.layer_combine(0, rows, d_y.data_ptr(), prepare_next=True) == 0
    assert st.layer_experts(1, d_y.data_ptr(), rows, router_input_ready=True) == 0        # logits of the prepared input
    assert st.status() == 0
    ws, y = st.workspace(), d_y.cpu().numpy()
    logits = d2h(ws.logits, rows * 4, np.float32).reshape(rows, 4)
    for t in sorted({0, 1, 2, 3, rows // 2, rows - 2, rows - 1}):
        want, _, _ = orc.moe_layer_q4(layers[0], x[t:t + 1], threads=4)
        rc, normed = orc.rmsnorm(want[0], layers[0].norm_weight, layers[0].eps, True)
        assert rc == 0
        assert_bits_equal(y[t], normed, f"row {t} of {rows} x {n}")
        rc, r = orc.router_input(normed, layers[1].router_scale, layers[1].eps)
        assert rc == 0
        assert_bits_equal(logits[t], orc.router_scores(layers[1].router_w, None, r), f"logits of row {t} of {rows} x {n}")
    st.close()


@pytest.mark.parametrize("n", [64, 1024, 1088, 1664, 1728, 2048, 2816, 3072, 4096, 4160, 5120, 5184, 6080])
def test_form_follows_from_sizes(synth, n):
    import torch
    line = _line(n)
    assert torch.cuda.get_device_properties(0).multi_processor_count == SMS
    st, _ = _stack(synth, n, line + 1)
    for rows, blocks in ((line, line), (line + 1, (line + 4) // 4)):
        x = torch.randn(rows, n, device="cuda")
        y = torch.zeros_like(x)
        assert st.layer_experts(0, x.data_ptr(), rows) == 0
        torch.cuda.synchronize()

        def call(stream):
            assert st.layer_combine(0, rows, y.data_ptr(), prepare_next=True, stream=stream) == 0
        (name, grid), = captured_kernels(call)
        assert grid == (blocks, 1, 1), (name, n, rows)
    st.close()


def test_flagged_rows(synth):
    """A non-finite row sets the status word in the warp form too, and leaves the other rows as they are."""
    import torch
    n, rows = 2048, 2 * SMS + 5
    st, _ = _stack(synth, n, rows)
    x = torch.randn(rows, n, device="cuda")
    y = [torch.zeros_like(x) for _ in range(2)]
    assert st.layer_experts(0, x.data_ptr(), rows) == 0 and st.layer_combine(0, rows, y[0].data_ptr()) == 0
    assert st.status() == 0
    c2g = d2h(st.workspace().canonical_to_grouped, rows * 2, np.int32)
    grouped = st.workspace().grouped_out
    bad = int(c2g[2 * 7])                                   # a grouped row of token 7
    inf = np.full(1, np.inf, np.float32)
    import ctypes as C
    assert C.CDLL("libcuda.so.1").cuMemcpyHtoD_v2(C.c_uint64(grouped + (bad * n + 5) * 4), C.c_void_p(inf.ctypes.data), C.c_size_t(4)) == 0
    assert st.layer_combine(0, rows, y[1].data_ptr()) == 0
    assert st.status() != 0
    keep = [t for t in range(rows) if t != 7]
    assert torch.equal(y[0][keep], y[1][keep])
    st.close()


@pytest.mark.parametrize("n,rounds", [(1024, 4), (1088, 1), (2048, 1), (2112, 2), (5120, 2), (5184, 3), (6144, 3)])
def test_form_of_one_sum(orc, synth, n, rounds):
    """With one in-order sum (a prompt's router input, a last layer's norm) the line lies elsewhere; both sides of it."""
    import torch
    line = rounds * SMS
    st, layers = _stack(synth, n, line + 1)
    for rows, blocks in ((line, line), (line + 1, (line + 4) // 4)):
        x = synth.make_tokens(830 + n, rows, n)
        d_x, y = torch.from_numpy(x).cuda(), torch.zeros(rows, n, device="cuda")
        assert st.layer_experts(0, d_x.data_ptr(), rows) == 0
        torch.cuda.synchronize()

        def call(stream):
            assert st.layer_combine(0, rows, y.data_ptr(), apply_norm=True, stream=stream) == 0
        (name, grid), = captured_kernels(call)
        assert grid == (blocks, 1, 1), (name, n, rows)
        call(torch.cuda.current_stream().cuda_stream)
        assert st.status() == 0
        for t in (0, rows // 2, rows - 1):
            want, _, _ = orc.moe_layer_q4(layers[0], x[t:t + 1], threads=4)
            assert_bits_equal(y[t].cpu().numpy(), orc.rmsnorm(want[0], layers[0].norm_weight, layers[0].eps, True)[1], f"row {t} of {rows} x {n}")
    st.close()


@pytest.mark.parametrize("n,topk,rounds", [(64, 2, 4), (1024, 2, 4), (1088, 2, 1), (2048, 2, 1), (2112, 2, 2), (4096, 2, 2), (4160, 2, 1), (5120, 2, 1),
                                           (5184, 2, 2), (6144, 2, 2), (1024, 5, 6), (1088, 5, 1), (2048, 5, 2), (2112, 5, 3), (2816, 5, 3),
                                           (2880, 5, 2), (5120, 5, 1)])
def test_form_without_a_sum(orc, synth, n, topk, rounds):
    """The reduce alone: both sides of its line."""
    import torch
    line = rounds * SMS
    st, layers = _stack(synth, n, line + 1, topk=topk)
    for rows, blocks in ((line, line), (line + 1, (line + 4) // 4)):
        x = synth.make_tokens(840 + n, rows, n)
        d_x, y = torch.from_numpy(x).cuda(), torch.zeros(rows, n, device="cuda")
        assert st.layer_experts(0, d_x.data_ptr(), rows) == 0
        torch.cuda.synchronize()

        def call(stream):
            assert st.layer_combine(0, rows, y.data_ptr(), apply_norm=False, stream=stream) == 0
        (name, grid), = captured_kernels(call)
        assert grid == (blocks, 1, 1), (name, n, rows)
        call(torch.cuda.current_stream().cuda_stream)
        assert st.status() == 0
        for t in (0, rows // 2, rows - 1):
            want, _, _ = orc.moe_layer_q4(layers[0], x[t:t + 1], threads=4)
            assert_bits_equal(y[t].cpu().numpy(), want[0], f"row {t} of {rows} x {n}")
    st.close()
