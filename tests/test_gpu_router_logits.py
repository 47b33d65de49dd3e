"""Router logits at the edges of the kernels' tiles: expert and row remainders, a half slab of columns, each number of
chains per lane, against the CPU oracle bit for bit."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from gpu_util import d2h, stack_mod
from graph_util import captured_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,E,B", [(64, 8, 5), (320, 24, 9), (192, 40, 300), (128, 130, 33), (192, 70, 430), (64, 129, 700),
                                   (320, 65, 1500)])
def test_router_logits_ragged_vs_oracle(orc, synth, H, E, B):
    import torch
    K = 2
    layer = synth.make_q4_moe_layer(600 + E, hidden=H, inter=64, n_experts=E, topk=K)
    st = stack_mod().MoeStack(B, H, 64, E, K)
    st.add_layer(layer)
    x = synth.make_tokens(601 + B, B, H)
    d_x = torch.from_numpy(x).cuda()
    assert st.layer_experts(0, d_x.data_ptr(), B) == 0
    assert st.status() == 0
    got = d2h(st.workspace().logits, B * E, np.float32).reshape(B, E)
    want = np.empty_like(got)
    for t in range(B):
        rc, rin = orc.router_input(x[t], layer.router_scale, layer.eps)
        assert rc == 0
        want[t] = orc.router_scores(layer.router_w, None, rin)
    assert_bits_equal(got, want, f"logits of {B} rows x {E} experts over {H} columns")
    st.close()


# The block-per-chain form (both piece counts, a column remainder) and the top-k behind it: experts that
# share a router row tie (the lower one wins), one, several and more than four keys per lane, top-k up to all experts.
@pytest.mark.parametrize("H,E,K,B", [(64, 2, 2, 1), (2816, 33, 8, 2), (3136, 128, 8, 4), (192, 129, 6, 3), (256, 128, 32, 1),
                                     (128, 64, 4, 20)])
def test_router_topk_ties_vs_oracle(orc, synth, H, E, K, B):
    import torch
    layer = synth.make_q4_moe_layer(650 + E, hidden=H, inter=64, n_experts=E, topk=K)
    layer.router_w[1::2] = layer.router_w[0:E - E % 2:2]
    st = stack_mod().MoeStack(B, H, 64, E, K)
    st.add_layer(layer)
    x = synth.make_tokens(651 + B, B, H)
    x[0] = 0.0                                             # logits of either sign of zero: all tie
    d_x = torch.from_numpy(x).cuda()
    assert st.layer_experts(0, d_x.data_ptr(), B) == 0
    assert st.status() == 0
    ws = st.workspace()
    got = d2h(ws.logits, B * E, np.float32).reshape(B, E)
    sel, wts = d2h(ws.selected, B * K, np.int32).reshape(B, K), d2h(ws.weights, B * K, np.float32).reshape(B, K)
    for t in range(B):
        rc, rin = orc.router_input(x[t], layer.router_scale, layer.eps)
        assert rc == 0
        logits = orc.router_scores(layer.router_w, None, rin)
        assert_bits_equal(got[t], logits, f"logits of row {t}")
        rc, want_sel, want_w = orc.router_topk(logits, layer.per_expert_scale, K, True)
        assert rc == 0
        assert_bits_equal(sel[t], want_sel, f"selected of row {t}")
        assert_bits_equal(wts[t], want_w, f"weights of row {t}")
    st.close()


def _hard_rows(rng, E, H):
    """Router rows whose running sums do what a block that adds a chain in pieces has to survive."""
    w = np.empty((E, H), np.float32)
    for e in range(E):
        g = rng.standard_normal(H)
        kind = e % 12
        if kind == 1:
            g *= 10.0 ** rng.uniform(-16, 16, H)                   # most terms vanish, a few decide
        elif kind == 2:
            g = rng.integers(-8, 9, H) * 0.25                      # half-way cases, exact zeros on the way
        elif kind == 3:
            g[1::2] = -g[0::2]                                     # pairs that nearly cancel
        elif kind == 4:
            g[H // 2:] = -g[:H - H // 2]
        elif kind == 5:
            g = np.sin(np.arange(H) * 0.01) * 3.0                  # passes zero and comes back
        elif kind == 6:
            g *= 1e-38                                             # subnormal terms and sums
        elif kind == 7:
            g = np.sign(g) * 2.0 ** rng.integers(-12, 12, H)
        elif kind == 8:
            g = np.where(np.arange(H) < H - 3, 0.0, g)             # zeros, then the only terms
        elif kind == 9:
            g[0], g[-1] = 1e30, -1e30                              # everything between is lost
        elif kind == 10:
            g = np.abs(g)
        elif kind == 11:
            g[H // 3] = -np.abs(g).sum()                           # from far below zero back up
        w[e] = g
    return w


# One launch per layer (one token) and a block per chain: widths that one warp adds, of odd and even numbers of pieces, and the
# widest of each kernel.
@pytest.mark.parametrize("H,B,fused", [(64, 1, True), (192, 1, True), (2816, 1, True), (3200, 1, True), (64, 4, False), (704, 3, False),
                                       (2816, 2, False), (5120, 1, False), (5120, 4, False)])
def test_router_chains_with_hard_rows_vs_oracle(orc, synth, H, B, fused):
    import torch
    E, K = 48, 4
    layer = synth.make_q4_moe_layer(670 + H, hidden=H, inter=64, n_experts=E, topk=K)
    layer.router_w[:] = _hard_rows(np.random.default_rng(671 + H + B), E, H)
    st = stack_mod().MoeStack(B, H, 64, E, K)
    st.add_layer(layer)
    x = synth.make_tokens(672 + B, B, H)
    d_x = torch.from_numpy(x).cuda()
    d_y = torch.zeros_like(d_x)
    if fused:
        assert st.forward_device(d_x.data_ptr(), B, d_y.data_ptr()) == 0
    else:
        assert st.layer_experts(0, d_x.data_ptr(), B) == 0
    st.status()                                                    # a selection among huge logits may be refused: not the point here
    got = d2h(st.workspace().logits, B * E, np.float32).reshape(B, E)
    for t in range(B):
        rc, rin = orc.router_input(x[t], layer.router_scale, layer.eps)
        assert rc == 0
        assert_bits_equal(got[t], orc.router_scores(layer.router_w, None, rin), f"logits of row {t} over {H} columns")
    st.close()


# Every pair of products nearly cancels (from the first, from the middle or but for the last columns): segments without an answer up to their limit and past it.
@pytest.mark.parametrize("H,B,fused", [(896, 1, True), (2816, 1, True), (960, 2, False), (2816, 3, False), (5120, 2, False)])
def test_router_chains_of_cancelling_pairs_vs_oracle(orc, synth, H, B, fused):
    import torch
    E, K = 12, 4
    layer = synth.make_q4_moe_layer(700 + H, hidden=H, inter=64, n_experts=E, topk=K)
    rng = np.random.default_rng(701 + H)
    w = rng.standard_normal((E, H))
    for e in range(E):
        lo, hi = [(0, H), (H // 2 + 2 * (e // 3), H), (0, H - 64 * (e // 3 + 1))][e % 3]
        w[e, lo + 1:hi:2] = -w[e, lo:hi - 1:2] * (1.0 + 1e-6 * rng.standard_normal((hi - lo) // 2))
    layer.router_w[:] = w.astype(np.float32)
    layer.router_scale[:] = 1.0
    st = stack_mod().MoeStack(B, H, 64, E, K)
    st.add_layer(layer)
    d_x = torch.ones(B, H, device="cuda")
    d_y = torch.zeros_like(d_x)
    if fused:
        assert st.forward_device(d_x.data_ptr(), B, d_y.data_ptr()) == 0
    else:
        assert st.layer_experts(0, d_x.data_ptr(), B) == 0
    assert st.status() == 0
    got = d2h(st.workspace().logits, B * E, np.float32).reshape(B, E)
    rc, rin = orc.router_input(np.ones(H, np.float32), layer.router_scale, layer.eps)
    assert rc == 0
    want = orc.router_scores(layer.router_w, None, rin)
    for t in range(B):
        assert_bits_equal(got[t], want, f"logits of row {t} over {H} columns")
    st.close()


# Both sides of the lines (148 SMs): one warp adds a chain of up to 832 columns (squares: 576), of more where more chains share an SM;
# a block per chain up to so many chains, the kernel of a chain per lane above.
@pytest.mark.parametrize("H,B", [(512, 15), (512, 16), (576, 1), (640, 1), (832, 2), (896, 2), (1024, 3), (1024, 4), (1024, 16), (1536, 7), (1536, 8),
                                 (2048, 12), (2048, 13), (2048, 17), (2048, 18), (2816, 21), (2816, 22), (5120, 33), (5120, 34)])
def test_router_chains_at_the_lines(orc, synth, H, B):
    test_router_chains_with_hard_rows_vs_oracle(orc, synth, H, B, False)


@pytest.mark.parametrize("H,most", [(64, 15), (512, 15), (1600, 15), (2048, 17), (2816, 21), (5120, 33), (5184, 0)])
def test_form_follows_from_chains_and_length(synth, H, most):
    import torch
    assert torch.cuda.get_device_properties(0).multi_processor_count == 148
    E, K, B = 48, 4, most + 1
    st = stack_mod().MoeStack(B, H, 64, E, K)
    st.add_layer(synth.make_q4_moe_layer(690 + H, hidden=H, inter=64, n_experts=E, topk=K))
    x = torch.randn(B, H, device="cuda")
    sel, w = torch.zeros(B * K, dtype=torch.int32, device="cuda"), torch.zeros(B * K, device="cuda")
    assert st.layer_route(0, x.data_ptr(), B, sel.data_ptr(), w.data_ptr()) == 0
    for rows in range(max(1, most), B + 1):
        def call(stream):
            assert st.layer_route(0, x.data_ptr(), rows, sel.data_ptr(), w.data_ptr(), router_input_ready=True, stream=stream) == 0
        grids = [grid for _, grid in captured_kernels(call)]
        assert ((E, rows, 1) in grids) == (rows <= most), (H, rows, grids)
    st.close()


# The tiles of many rows with seven and with eight adding warps, of two and of four rows each, and their last, partial rows.
@pytest.mark.parametrize("H,E,B", [(192, 128, 900), (128, 130, 1190), (64, 128, 2073), (192, 64, 2400), (64, 128, 2100)])
def test_router_logits_adding_warps_vs_oracle(orc, synth, H, E, B):
    test_router_logits_ragged_vs_oracle(orc, synth, H, E, B)
