"""Grouping with expert counts whose histograms end just below and above 48 KB of shared memory, with the top-k in the same launch (a
few rows) and without."""
import numpy as np
import pytest

from gpu_util import d2h, stack_mod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,E", [(12, e) for e in (316, 317, 356, 358, 361, 362, 700)] + [(6, e) for e in (212, 215, 241, 243, 245, 300)])
def test_grouping(synth, B, E):
    import torch
    K = 2
    st = stack_mod().MoeStack(B, 64, 64, E, K)
    st.add_layer(synth.make_q4_moe_layer(890, hidden=64, inter=64, n_experts=E, topk=K))
    x = torch.from_numpy(synth.make_tokens(891, B, 64)).cuda()
    assert st.layer_experts(0, x.data_ptr(), B) == 0
    assert st.status() == 0
    ws, n = st.workspace(), B * K
    sel = d2h(ws.selected, n, np.int32)
    assert np.array_equal(d2h(ws.grouped_to_canonical, n, np.int32), np.argsort(sel, kind="stable"))
    assert np.array_equal(d2h(ws.group_offsets, E + 1, np.int32), np.concatenate(([0], np.bincount(sel, minlength=E).cumsum())))
    st.close()
