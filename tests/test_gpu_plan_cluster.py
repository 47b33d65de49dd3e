"""Grouping of 2048 selections and more, by a cluster of eight blocks: the stable counting sort at parts that are ragged, end in the
middle of a warp's segment or hold few experts, against numpy."""
import numpy as np
import pytest

from gpu_util import d2h, stack_mod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,K,E,lo,hi", [(256, 8, 16, 0, 16), (255, 8, 16, 0, 16), (300, 7, 40, 0, 40), (1027, 2, 3, 0, 3), (2049, 1, 5, 0, 5),
                                         (700, 3, 130, 20, 90)])
def test_grouping_is_the_stable_sort(synth, B, K, E, lo, hi):
    import torch
    st = stack_mod().MoeStack(B, 64, 64, E, K, expert_begin=lo, expert_end=hi)
    st.add_layer(synth.make_q4_moe_layer(880 + B, hidden=64, inter=64, n_experts=E, topk=K))
    x = torch.from_numpy(synth.make_tokens(881 + B, B, 64)).cuda()
    assert st.layer_experts(0, x.data_ptr(), B) == 0
    assert st.status() == 0
    ws, n = st.workspace(), B * K
    sel = d2h(ws.selected, n, np.int32)
    order = np.argsort(sel, kind="stable")
    assert np.array_equal(d2h(ws.grouped_to_canonical, n, np.int32), order)
    place = np.empty(n, np.int32)
    place[order] = np.arange(n)
    assert np.array_equal(d2h(ws.canonical_to_grouped, n, np.int32), place)
    assert np.array_equal(d2h(ws.group_offsets, E + 1, np.int32), np.concatenate(([0], np.bincount(sel, minlength=E).cumsum())))
    st.close()
