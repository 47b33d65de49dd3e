"""Buffers of a stack that later calls outgrow: what was set up with them before keeps working on memory that is still its own."""
import pytest

from conftest import assert_bits_equal
from gpu_util import stack_mod
from test_gpu_moe import _oracle_ffn_block

pytestmark = pytest.mark.gpu


def test_wider_dense_branch_attached_later(orc, synth):
    import torch
    H, M, E, K, B = 256, 128, 16, 4, 5
    st, layers, blocks = stack_mod().MoeStack(8, H, M, E, K), [], []
    for i, dense in enumerate((192, 1024, 320)):
        layers.append(synth.make_q4_moe_layer(880 + i, hidden=H, inter=M, n_experts=E, topk=K))
        blocks.append(synth.make_ffn_block(883 + i, hidden=H, dense_inter=dense))
        st.add_layer(layers[i])
        assert st.attach_ffn_block(i, blocks[i]) == 0
    x = synth.make_tokens(886, B, H)
    d_x, d_y = torch.from_numpy(x).cuda(), torch.zeros(B, H, device="cuda")
    for i in (0, 1, 2, 0):
        assert st.ffn_block_forward(i, d_x.data_ptr(), B, d_y.data_ptr()) == 0
        assert st.status() == 0
        assert_bits_equal(d_y.cpu().numpy(), _oracle_ffn_block(orc, layers[i], blocks[i], x), f"layer {i}")
    st.close()
