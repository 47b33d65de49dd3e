"""Rows sent with an expert id that does not exist are reported, come back as zeros, and change no other row, whatever an earlier
and larger batch left in the tables."""
import pytest

from gpu_util import stack_mod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,mode", [("q4", False), ("q4", "split"), ("q4", "single"), ("fp4", False), ("fp4", "split")])
def test_other_rows_stay(synth, fmt, mode):
    import torch
    H, M, E, K, T = 512, 256, 8, 2, 64
    st = stack_mod().MoeStack(T, H, M, E, K)
    if fmt == "q4":
        st.add_layer(synth.make_q4_moe_layer(920, hidden=H, inter=M, n_experts=E, topk=K))
    else:
        st.add_nvfp4_layer(synth.make_nvfp4_moe_layer(921, hidden=H, inter=M, n_experts=E, topk=K))
    many = torch.randn(T * K, H, device="cuda")
    ids = torch.arange(T * K, dtype=torch.int32, device="cuda") % E
    out = torch.zeros_like(many)
    assert st.layer_experts_routed(0, many.data_ptr(), ids.data_ptr(), T * K, out.data_ptr(), tensor_core=mode) == 0
    assert st.status() == 0
    for n in (1, 5, 33):
        rows = torch.randn(n, H, device="cuda")
        good = torch.arange(n, dtype=torch.int32, device="cuda") % E
        want, got = torch.zeros_like(rows), torch.full_like(rows, 7.0)
        assert st.layer_experts_routed(0, rows.data_ptr(), good.data_ptr(), n, want.data_ptr(), tensor_core=mode) == 0
        assert st.status() == 0
        # a larger batch again, so that the tables hold its rows
        assert st.layer_experts_routed(0, many.data_ptr(), ids.data_ptr(), T * K, out.data_ptr(), tensor_core=mode) == 0
        bad = good.clone()
        lost = list(range(0, n, 3))
        bad[lost] = torch.tensor([-1, E, 99, -2 ** 31, 2 ** 31 - 1], dtype=torch.int32, device="cuda").repeat(n)[:len(lost)]
        assert st.layer_experts_routed(0, rows.data_ptr(), bad.data_ptr(), n, got.data_ptr(), tensor_core=mode) == 0
        assert st.status() & 2
        kept = [i for i in range(n) if i not in lost]
        assert torch.equal(got[kept], want[kept]) and not got[lost].any()
    st.close()
