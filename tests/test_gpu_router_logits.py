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
