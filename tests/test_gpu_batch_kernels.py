"""The projection kernel for jobs of several tokens (batch_kernels.cu) at the edges of its tiles: row tails, chunk and
group remainders, every pass size, and affine-Q4 groups whose bias rules the exact one-rounding dequantisation out."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from gpu_util import backend_mod, gpu, stack_mod
from graph_util import captured_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,C", [(1, 64), (63, 192), (64, 256), (65, 320), (130, 704), (33, 8192)])
@pytest.mark.parametrize("B", [2, 3, 4, 5, 9])
def test_batch_projection_vs_oracle(orc, synth, R, C, B):
    rng = np.random.default_rng(R * 1000 + C + B)
    v, s, b = synth.make_q4(rng, R, C)
    if B == 3:                                     # zero points close to zero, zero biases, negative scales
        b = b.copy()
        b[::3] = synth.bf16_round(np.float32(1e-5) * synth.bf16_to_f32(s[::3]))
        b[1::5] = 0
        s = s.copy()
        s[::7] ^= 0x8000
    xs = rng.standard_normal((B, C)).astype(np.float32)
    ys = np.zeros((B, R), np.float32)
    g = gpu()
    g.set_mapped_only(0)
    assert g.proj_batch(v, s, b, R, C, xs, ys, 0x51000000 + R * 100000 + C * 10 + B) == 0
    for t in range(B):
        assert_bits_equal(ys[t], orc.q4_matvec(v, s, b, R, C, xs[t]), f"{R}x{C} token {t} of {B}")


def test_single_token_of_a_wide_row(orc, synth):
    """12288 columns: scale tables of 192 words per row."""
    rng = np.random.default_rng(17)
    R, C = 70, 12288
    v, s, b = synth.make_q4(rng, R, C)
    x, y = rng.standard_normal(C).astype(np.float32), np.zeros(R, np.float32)
    g = gpu()
    g.set_mapped_only(0)
    assert g.q4_matvec(v, s, b, R, C, x, y) == 0
    assert_bits_equal(y, orc.q4_matvec(v, s, b, R, C, x), "70 x 12288")


@pytest.mark.parametrize("R,C", [(1, 256), (33, 768), (65, 512)])
def test_nvfp4_batch_projection_vs_oracle(orc, synth, R, C):
    g, bm = gpu(), backend_mod()
    rng = np.random.default_rng(R + C)
    packed, scales, divisor = synth.make_nvfp4(rng, R, C)
    buf = np.concatenate([packed.reshape(-1), scales.reshape(-1), np.zeros(-(R * C // 16) % 4, np.uint8),
                          np.array([divisor, 64.0], np.float32).view(np.uint8)])
    p, s = buf[:R * C // 2], buf[R * C // 2:R * C // 2 + R * C // 16]
    assert g.weight_resource_bind(bm.RESOURCE_EXPERT_LAYER, 97, buf) == 0
    assert g.nvfp4_resource_slot(bm.RESOURCE_EXPERT_LAYER, 97, 0xF9700, p, s, buf[-8:-4], buf[-4:], R, C) == 0
    for B in (1, 2, 3, 4, 6):
        xs = rng.standard_normal((B, C)).astype(np.float32)
        ys = np.zeros((B, R), np.float32)
        assert g.nvfp4_matvec_batch(0xF9700, R, C, xs, ys) == 0
        for t in range(B):
            rc, want = orc.nvfp4_matvec(p.reshape(R, C // 2), s.reshape(R, C // 16), float(divisor), 64.0, R, C, xs[t],
                                        threads=4)
            assert rc == 0
            assert_bits_equal(ys[t], want, f"nvfp4 {R}x{C} token {t} of {B}")
    assert g.weight_resource_unbind(bm.RESOURCE_EXPERT_LAYER, 97) == 0


def test_down_of_a_whole_block_shares_the_layers_kernel(synth):
    """The dense down product of a block runs the kernel of the routed one, not the one for a projection by itself (the last template
    argument: groups per iteration)."""
    import torch
    H, M, E, K, B = 256, 64, 8, 2, 2
    st = stack_mod().MoeStack(B, H, M, E, K)
    st.add_layer(synth.make_q4_moe_layer(91, hidden=H, inter=M, n_experts=E, topk=K))
    assert st.attach_ffn_block(0, synth.make_ffn_block(92, hidden=H, dense_inter=128)) == 0
    x = torch.randn(B, H, device="cuda")
    y = torch.zeros_like(x)

    def call(stream):
        assert st.ffn_block_forward(0, x.data_ptr(), B, y.data_ptr(), stream=stream) == 0
    names = [name for name, _ in captured_kernels(call) if "batch_kernel" in name]
    assert len(names) == 4 and names[1] == names[3] and "ILi0ELi1ELi2ELi1E" in names[1], names
    st.close()
