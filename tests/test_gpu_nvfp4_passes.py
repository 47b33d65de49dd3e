"""Exact NVFP4 layers whose expert groups are cut into passes of four tokens: every remainder, expert ranges, the batch from
which whole groups are jobs again, and grids that hold no more blocks than the passes a batch can have."""
import numpy as np
import pytest

import oracle
from conftest import assert_bits_equal
from gpu_util import d2h, stack_mod
from graph_util import captured_kernels

pytestmark = pytest.mark.gpu


def _check(orc, layer, x, y, tokens, what):
    want, _, _ = oracle.moe_layer_nvfp4(orc, layer, np.ascontiguousarray(x[tokens]), threads=8)
    assert_bits_equal(y[tokens], want, what)


@pytest.mark.parametrize("H,M,E,K,B", [(512, 256, 8, 2, 2), (512, 256, 8, 2, 9), (256, 512, 8, 8, 7), (256, 256, 8, 8, 4),
                                       (512, 256, 130, 3, 33), (256, 256, 5, 2, 70), (256, 256, 3, 1, 21)])
def test_group_sizes_vs_oracle(orc, synth, H, M, E, K, B):
    import torch
    layer = synth.make_nvfp4_moe_layer(830 + B, hidden=H, inter=M, n_experts=E, topk=K)
    x = synth.make_tokens(831 + B, B, H)
    d_x, d_y = torch.from_numpy(x).cuda(), torch.zeros(B, H, device="cuda")
    whole = stack_mod().MoeStack(B, H, M, E, K)
    whole.add_nvfp4_layer(layer)
    assert whole.layer_experts(0, d_x.data_ptr(), B) == 0
    assert whole.layer_combine(0, B, d_y.data_ptr(), apply_norm=False) == 0
    assert whole.status() == 0
    sizes = np.diff(d2h(whole.workspace().group_offsets, E + 1, np.int32))
    assert sizes.sum() == B * K
    y = d_y.cpu().numpy()
    _check(orc, layer, x, y, np.unique(np.linspace(0, B - 1, 9).astype(int)), f"groups {sorted(set(sizes.tolist()))}")
    # the same rows from two expert ranges
    shared = torch.zeros(B * K * H, device="cuda")
    for lo, hi in ((0, E // 2), (E // 2, E)):
        part = stack_mod().MoeStack(B, H, M, E, K, expert_begin=lo, expert_end=hi)
        part.add_nvfp4_layer(layer)
        assert part.set_grouped_out(shared.data_ptr(), shared.numel() * 4) == 0
        assert part.layer_experts(0, d_x.data_ptr(), B) == 0 and part.status() == 0
        part.close()
    assert_bits_equal(shared.cpu().numpy(), d2h(whole.workspace().grouped_out, B * K * H, np.float32), "expert ranges")
    whole.close()


def test_more_passes_than_a_grid_holds(orc, synth):
    import torch
    H, M, E, K, B = 256, 256, 8, 2, 65600                 # 2 (8 + 131200 / 4) jobs do not fit the y extent
    layer = synth.make_nvfp4_moe_layer(850, hidden=H, inter=M, n_experts=E, topk=K)
    x = synth.make_tokens(851, B, H)
    d_x, d_y = torch.from_numpy(x).cuda(), torch.zeros(B, H, device="cuda")
    st = stack_mod().MoeStack(B, H, M, E, K)
    st.add_nvfp4_layer(layer)
    assert st.layer_experts(0, d_x.data_ptr(), B) == 0
    assert st.layer_combine(0, B, d_y.data_ptr(), apply_norm=False) == 0
    assert st.status() == 0
    _check(orc, layer, x, d_y.cpu().numpy(), np.array([0, 1, 777, B // 2, B - 2, B - 1]), "whole groups as jobs")
    st.close()


@pytest.mark.parametrize("B", [4, 16, 70, 256])
def test_grid_spans_passes_only(synth, B):
    import torch
    H, M, E, K = 512, 256, 8, 2
    st = stack_mod().MoeStack(B, H, M, E, K)
    st.add_nvfp4_layer(synth.make_nvfp4_moe_layer(860, hidden=H, inter=M, n_experts=E, topk=K))
    x = torch.randn(B, H, device="cuda")

    def call(stream):
        assert st.layer_experts(0, x.data_ptr(), B, stream=stream) == 0
    grids = [g for name, g in captured_kernels(call) if "batch_kernel" in name]
    assert len(grids) == 2
    most = min(B * K, E + B * K // 4)                     # passes of four tokens that B K selections can make
    for (tiles, jobs, deep), matrices in zip(grids, (2, 1)):
        assert jobs * deep <= matrices * most, grids
    st.close()
