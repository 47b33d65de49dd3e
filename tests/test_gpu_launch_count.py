"""salt_b200_launch_count against the kernels that a captured call holds, for every form of a layer."""
import pytest

from gpu_util import stack_mod
from graph_util import captured_kernels

pytestmark = pytest.mark.gpu

H, M, E, K, T = 512, 256, 8, 2, 40


@pytest.fixture(scope="module")
def stacks(synth):
    q4, fp4 = stack_mod().MoeStack(T, H, M, E, K), stack_mod().MoeStack(T, H, M, E, K)
    for i in range(2):
        q4.add_layer(synth.make_q4_moe_layer(700 + i, hidden=H, inter=M, n_experts=E, topk=K))
        fp4.add_nvfp4_layer(synth.make_nvfp4_moe_layer(710 + i, hidden=H, inter=M, n_experts=E, topk=K))
    assert q4.attach_ffn_block(0, synth.make_ffn_block(720, hidden=H, dense_inter=192)) == 0
    yield {"q4": q4, "fp4": fp4}
    q4.close()
    fp4.close()


def _counted(st, call):
    seen = []

    def once(stream):
        n0 = st.launch_count()
        assert call(stream) == 0
        seen.append(st.launch_count() - n0)
    kernels = captured_kernels(once)
    assert seen == [len(kernels)] * 2, [k for k, _ in kernels]
    assert st.status() == 0


@pytest.mark.parametrize("fmt", ["q4", "fp4"])
@pytest.mark.parametrize("level", [1, 2, 0])
@pytest.mark.parametrize("B", [1, 3, 8, 9, 33])
def test_forward(stacks, fmt, level, B):
    import torch
    st = stacks[fmt]
    x = torch.randn(B, H, device="cuda")
    y = torch.zeros_like(x)
    st.set_fused_decode(level)
    _counted(st, lambda s: st.forward_device(x.data_ptr(), B, y.data_ptr(), stream=s))
    st.set_fused_decode(1)


@pytest.mark.parametrize("fmt,mode", [("q4", False), ("q4", "split"), ("q4", "single"), ("fp4", False), ("fp4", "split")])
@pytest.mark.parametrize("B", [5, 40])
def test_layer_calls(stacks, fmt, mode, B):
    import torch
    st = stacks[fmt]
    x = torch.randn(B, H, device="cuda")
    y = torch.zeros_like(x)
    _counted(st, lambda s: st.layer_experts(0, x.data_ptr(), B, tensor_core=mode, stream=s))
    _counted(st, lambda s: st.layer_combine(0, B, y.data_ptr(), prepare_next=True, stream=s))
    sel, wts = torch.zeros(B, K, dtype=torch.int32, device="cuda"), torch.zeros(B, K, device="cuda")
    _counted(st, lambda s: st.layer_route(0, x.data_ptr(), B, sel.data_ptr(), wts.data_ptr(), stream=s))
    _counted(st, lambda s: st.layer_experts_routed(0, x.data_ptr(), sel.data_ptr(), B, y.data_ptr(), tensor_core=mode, stream=s))


@pytest.mark.parametrize("B", [2, 17])
def test_ffn_block(stacks, B):
    import torch
    st = stacks["q4"]
    x = torch.randn(B, H, device="cuda")
    y = torch.zeros_like(x)
    _counted(st, lambda s: st.ffn_block_forward(0, x.data_ptr(), B, y.data_ptr(), stream=s))
