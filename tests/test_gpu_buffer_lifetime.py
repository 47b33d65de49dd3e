"""Buffers of a stack that later calls outgrow: what was set up with them before keeps working on memory that is still its own."""
import pytest

from conftest import assert_bits_equal
from gpu_util import oracle_stack, stack_mod
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


@pytest.mark.parametrize("level", [1, 2])
def test_captured_pass_after_layers_were_added(orc, synth, level):
    """A captured one-token pass replayed after a longer pass has run: the longer one needs more counters and arguments."""
    import torch
    H, M, E, K = 512, 128, 16, 4
    layers = [synth.make_q4_moe_layer(890 + i, hidden=H, inter=M, n_experts=E, topk=K) for i in range(5)]
    st, stream = stack_mod().MoeStack(4, H, M, E, K), torch.cuda.Stream()
    st.set_fused_decode(level)
    st.add_layer(layers[0])
    st.add_layer(layers[1])
    x, other = (torch.from_numpy(synth.make_tokens(s, 1, H)).cuda() for s in (895, 896))
    y, z = torch.zeros(1, H, device="cuda"), torch.zeros(1, H, device="cuda")
    assert st.graph_capture(x.data_ptr(), 1, y.data_ptr(), stream.cuda_stream) == 0
    want, _ = oracle_stack(orc, layers[:2], x.cpu().numpy(), threads=4)
    for layer in layers[2:]:
        st.add_layer(layer)
    assert st.forward_device(other.data_ptr(), 1, z.data_ptr(), stream=stream.cuda_stream) == 0
    stream.synchronize()
    full, _ = oracle_stack(orc, layers, other.cpu().numpy(), threads=4)
    assert_bits_equal(z.cpu().numpy(), full, "all layers")
    held = [torch.full((1 << 18,), 7, dtype=torch.int32, device="cuda") for _ in range(16)]     # where freed memory would go
    y.zero_()
    torch.cuda.synchronize()
    assert st.graph_launch(stream.cuda_stream) == 0
    assert st.status(stream.cuda_stream) == 0
    assert_bits_equal(y.cpu().numpy(), want, "replayed pass over the first two layers")
    assert all(int(h.min()) == 7 and int(h.max()) == 7 for h in held)
    st.close()


def test_captured_whole_pass_keeps_its_arguments(orc, synth):
    """All layers in one launch: the arguments of a captured pass are its own, whatever passes run between its replays."""
    import torch
    H, M, E, K = 512, 128, 16, 4
    layers = [synth.make_q4_moe_layer(900 + i, hidden=H, inter=M, n_experts=E, topk=K) for i in range(4)]
    st, stream = stack_mod().MoeStack(4, H, M, E, K), torch.cuda.Stream()
    for layer in layers:
        st.add_layer(layer)
    st.set_fused_decode(2)
    x, other = (torch.from_numpy(synth.make_tokens(s, 1, H)).cuda() for s in (905, 906))
    y, z = torch.zeros(1, H, device="cuda"), torch.zeros(1, H, device="cuda")
    assert st.graph_capture(x.data_ptr(), 1, y.data_ptr(), stream.cuda_stream, first=0, count=2) == 0
    want, _ = oracle_stack(orc, layers[:2], x.cpu().numpy(), threads=4)
    between, _ = oracle_stack(orc, layers[1:], other.cpu().numpy(), threads=4)
    for _ in range(2):
        assert st.forward_device(other.data_ptr(), 1, z.data_ptr(), first=1, count=3, stream=stream.cuda_stream) == 0
        y.zero_()
        torch.cuda.synchronize()
        assert st.graph_launch(stream.cuda_stream) == 0
        assert st.status(stream.cuda_stream) == 0
        assert_bits_equal(y.cpu().numpy(), want, "replayed pass")
        assert_bits_equal(z.cpu().numpy(), between, "pass between")
    st.close()


def test_captured_pass_is_dropped_with_the_grouped_buffer(orc, synth):
    import torch
    H, M, E, K, B = 512, 128, 16, 4, 3
    layer = synth.make_q4_moe_layer(910, hidden=H, inter=M, n_experts=E, topk=K)
    st, stream = stack_mod().MoeStack(4, H, M, E, K), torch.cuda.Stream()
    st.add_layer(layer)
    x = torch.from_numpy(synth.make_tokens(911, B, H)).cuda()
    y, grouped = torch.zeros(B, H, device="cuda"), torch.zeros(4 * K * H, device="cuda")
    assert st.graph_capture(x.data_ptr(), B, y.data_ptr(), stream.cuda_stream) == 0
    torch.cuda.synchronize()
    assert st.set_grouped_out(grouped.data_ptr(), grouped.numel() * 4) == 0
    assert st.graph_launch(stream.cuda_stream) == -1
    assert st.graph_capture(x.data_ptr(), B, y.data_ptr(), stream.cuda_stream) == 0
    y.zero_()
    torch.cuda.synchronize()
    assert st.graph_launch(stream.cuda_stream) == 0 and st.status(stream.cuda_stream) == 0
    assert_bits_equal(y.cpu().numpy(), orc.moe_layer_q4(layer, x.cpu().numpy(), threads=4)[0], "captured anew")
    st.close()
