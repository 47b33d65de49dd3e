"""Activation rows that do not start on a 16-byte boundary: refused where a kernel moves them in 16-byte pieces (it would
fault), taken as before where it does not."""
import pytest

from gpu_util import stack_mod

pytestmark = pytest.mark.gpu

H, M, E, K, T = 512, 256, 8, 2, 8


@pytest.mark.parametrize("fmt", ["q4", "fp4"])
def test_misaligned_rows(synth, fmt):
    import torch
    st = stack_mod().MoeStack(T, H, M, E, K)
    if fmt == "q4":
        st.add_layer(synth.make_q4_moe_layer(870, hidden=H, inter=M, n_experts=E, topk=K))
        assert st.attach_ffn_block(0, synth.make_ffn_block(871, hidden=H, dense_inter=192)) == 0
    else:
        st.add_nvfp4_layer(synth.make_nvfp4_moe_layer(872, hidden=H, inter=M, n_experts=E, topk=K))
    room, x = torch.zeros(T * H + 4, device="cuda"), torch.randn(T, H, device="cuda")
    y, z = torch.zeros(T, H, device="cuda"), torch.zeros(T, H, device="cuda")
    ids = torch.zeros(T, dtype=torch.int32, device="cuda")
    for off in (1, 2, 3):
        room[off:off + T * H] = x.reshape(-1)
        bad = room.data_ptr() + 4 * off
        n0 = st.launch_count()
        for B in (1, 2, T):
            for mode in (False, "split", "single"):
                assert st.layer_experts(0, bad, B, tensor_core=mode) == -1
                assert st.layer_experts_routed(0, bad, ids.data_ptr(), B, y.data_ptr(), tensor_core=mode) == -1
        assert st.forward_device(bad, 2, y.data_ptr()) == -1
        assert st.launch_count() == n0
        if fmt == "q4":
            assert st.forward_device(x.data_ptr(), 1, y.data_ptr()) == 0 and st.forward_device(bad, 1, z.data_ptr()) == 0
            assert torch.equal(y[0], z[0])
            assert st.ffn_block_forward(0, x.data_ptr(), T, y.data_ptr()) == 0
            assert st.ffn_block_forward(0, bad, T, z.data_ptr()) == 0
            assert torch.equal(y, z)
    assert st.layer_experts(0, x.data_ptr(), T) == 0 and st.status() == 0
    st.close()
