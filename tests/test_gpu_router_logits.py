"""Router logits at the edges of the kernels' tiles: expert and row remainders, a half slab of columns, each number of
chains per lane, against the CPU oracle bit for bit."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from gpu_util import d2h, stack_mod

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


# The chain-per-block form (one to four rows, both piece counts, a column remainder) and the top-k behind it: experts that
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
