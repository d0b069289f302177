"""The outer layer on few tokens (decode steps, short prompts: `ttt_layer_small_*`) and on lengths that leave a remainder
(pitched inner loop and tail), against the CPU restatement."""

import pytest
import torch

from conftest import assert_close
from oracle import ttt_layer_oracle as LO
from test_layer_gpu import _layer_from_params, _random_case


@pytest.mark.gpu
@pytest.mark.parametrize("B,T,H,F,use_gate,start", (
    (1, 1, 1, 64, False, 0), (8, 1, 12, 64, True, 21), (17, 1, 12, 64, False, 3), (1, 1, 4, 32, True, 0),
    (2, 16, 4, 32, False, 0), (1, 31, 3, 64, True, 0), (4, 7, 24, 32, False, 5), (32, 1, 32, 64, True, 9),
    (33, 1, 12, 64, True, 9), (1, 41, 3, 64, True, 0), (2, 145, 4, 32, False, 0)))
def test_short_and_ragged_calls_match_the_restatement(B, T, H, F, use_gate, start):
    import ttt_rs_b200 as tb
    dev = torch.device("cuda:0")
    x, p = _random_case(B, T, H, 41 + B, False, use_gate, torch.bfloat16, F)
    m, inner = _layer_from_params(tb, p, False, use_gate, torch.bfloat16, dev, H)
    inner.allow_partial = True
    with torch.no_grad():
        state = inner.init_state(B)
        y = m(x.to(torch.bfloat16).to(dev), inner, state, start)
    tb.TttTileMultiKernel.check_status()
    want, st = LO.ttt_layer_forward(x, p, num_heads=H, use_gate=use_gate, start_idx=start)
    assert_close(y, want, 3e-2, "layer output", max_bad_frac=1e-3)
    assert_close(state.weight, st["weight"], 2e-2, "state weight", max_bad_frac=1e-3)
    assert_close(state.bias, st["bias"], 2e-2, "state bias", max_bad_frac=5e-3)


@pytest.mark.gpu
def test_one_token_of_sequences_in_a_buffer_beyond_32_bit_offsets():
    """A decode step on a slice of a [2, T, C] buffer with T C = 2^31: the rows' pitch does not fit 32 bits."""
    import ttt_rs_b200 as tb
    H, C, far = 2, 128, 1 << 31
    cfg = tb.TTTLayerConfig(hidden_size=C, num_heads=H)
    torch.manual_seed(5)
    m = tb.TTT(cfg, device="cuda", dtype=torch.bfloat16)
    inner = tb.new_inner(cfg, device="cuda", dtype=torch.bfloat16, allow_partial=True)
    rows = (torch.randn(2, 1, C, device="cuda") * 0.5).bfloat16()
    x = torch.empty(far + C, dtype=torch.bfloat16, device="cuda").as_strided((2, 1, C), (far, C, 1))
    x.copy_(rows)
    with torch.no_grad():
        assert torch.equal(m(x, inner, inner.init_state(2)), m(rows, inner, inner.init_state(2)))


@pytest.mark.gpu
def test_a_call_that_goes_another_way_advances_the_state_once(monkeypatch):
    """Post-norm parameters off the 16-byte grid: the native layer call declines them, and has touched nothing by then."""
    import ttt_rs_b200 as tb
    H, C = 2, 128
    cfg = tb.TTTLayerConfig(hidden_size=C, num_heads=H)
    torch.manual_seed(6)
    m = tb.TTT(cfg, device="cuda", dtype=torch.bfloat16)
    inner = tb.new_inner(cfg, device="cuda", dtype=torch.bfloat16, allow_partial=True, partial_in_place=True)
    x = (torch.randn(3, 1, C, device="cuda") * 0.5).bfloat16()

    def step():
        with torch.no_grad():
            state = inner.init_state(3)
            return m(x, inner, state), state.weight, state.bias

    step()
    m.post_norm_weight = torch.nn.Parameter(torch.ones(C + 1, device="cuda", dtype=torch.bfloat16)[1:])
    got = step()
    monkeypatch.setattr(m, "_infer_native", lambda *a: None)
    for a, b in zip(got, step()):
        assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("T", (1, 40, 128))  # few-token form; general form with a remainder; one-launch projections
def test_token_eta_follows_its_parameters_at_every_call(T):
    """Also through `.data`, which leaves the parameter's version as it was; the kernels form the values that tensor
    operations give (negative sums clamped, sums rounded to bf16)."""
    import ttt_rs_b200 as tb
    H, C = 2, 128
    cfg = tb.TTTLayerConfig(hidden_size=C, num_heads=H)
    torch.manual_seed(8)
    m = tb.TTT(cfg, device="cuda", dtype=torch.bfloat16)
    inner = tb.new_inner(cfg, device="cuda", dtype=torch.bfloat16, allow_partial=True)
    x = (torch.randn(3, T, C, device="cuda") * 0.5).bfloat16()

    def run():
        with torch.no_grad():
            state = inner.init_state(3)
            return [m(x, inner, state), state.weight, state.bias]

    run()
    seen = []
    for shift in (0.37, -0.4):
        m.learnable_token_idx.data.add_(shift)
        seen.append(run())
        te = torch.clamp_min(m.token_idx + m.learnable_token_idx, 0.0)
        idx, learnable = m.token_idx, m.learnable_token_idx
        m.token_idx, m.learnable_token_idx = te.detach(), torch.nn.Parameter(torch.zeros_like(te))
        for a, b in zip(seen[-1], run()):
            assert torch.equal(a, b)
        m.token_idx, m.learnable_token_idx = idx, learnable
    assert not torch.equal(seen[0][1], seen[1][1])


@pytest.mark.gpu
@pytest.mark.parametrize("B,H,use_gate", ((16, 32, True), (17, 32, False), (32, 32, True), (17, 12, True), (24, 16, False),
                                          (25, 16, False), (32, 12, False), (17, 22, False)))
def test_either_side_of_where_the_general_form_takes_over(B, H, use_gate):
    import ttt_rs_b200 as tb
    x, p = _random_case(B, 1, H, 7 + H, False, use_gate, torch.bfloat16)
    m, inner = _layer_from_params(tb, p, False, use_gate, torch.bfloat16, torch.device("cuda:0"), H)
    inner.allow_partial = True
    with torch.no_grad():
        state = inner.init_state(B)
        y = m(x.bfloat16().cuda(), inner, state, 3)
    want, st = LO.ttt_layer_forward(x, p, num_heads=H, use_gate=use_gate, start_idx=3)
    assert_close(y, want, 3e-2, "layer output", max_bad_frac=1e-3)
    assert_close(state.weight, st["weight"], 2e-2, "state weight", max_bad_frac=1e-3)
