"""Training through the one-launch projections (bf16, sequences of a multiple of 128 tokens) against training through the
separate product and prologue: same output and gradients to bf16 rounding, with and without the gate whose gradient shares
the projections' gradient buffer, also when that gradient does not come straight from the epilogue."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,mb,pos,gate", [(1, 128, 1, 16, "rope", False), (2, 384, 3, 16, "none", True),
                                               (3, 128, 5, 8, "rope", True), (1, 640, 12, 16, "rope", False)])
def test_training_step_matches_the_unfused_projections(monkeypatch, B, T, H, mb, pos, gate):
    import ttt_rs_b200 as tb
    from ttt_rs_b200 import layer as L
    torch.manual_seed(T + H)
    cfg = tb.TTTLayerConfig(hidden_size=64 * H, num_heads=H, mini_batch_size=mb, pos_encoding=pos, use_gate=gate)
    m = tb.TTT(cfg, device="cuda", dtype=torch.bfloat16)
    inner = tb.new_inner(cfg, checkpoint_interval=4, device="cuda", dtype=torch.bfloat16)
    x = (torch.randn(B, T, 64 * H, device="cuda") * 0.5).bfloat16().requires_grad_()
    gy = (torch.randn(B, T, 64 * H, device="cuda") * 0.1).bfloat16()
    leaves = [x] + list(m.parameters()) + list(inner.inner.parameters())

    def step():
        y = m(x, inner, inner.init_state(B))
        return [y.detach()] + list(torch.autograd.grad(y, leaves, gy))

    used = []
    plain = L.layer_projections
    monkeypatch.setattr(L, "layer_projections", lambda *a, **k: used.append(1) or plain(*a, **k))
    fused = step()
    assert used, "the one-launch projections did not run"
    epilogue = L._EpilogueFn.apply
    monkeypatch.setattr(L, "_EpilogueFn", type("E", (), {"apply": staticmethod(lambda *a: epilogue(*a[:5]))}))
    apart = step()  # the gate's gradient in a buffer of its own
    monkeypatch.setattr(tb.TTT, "_can_fuse_projections", lambda *a: False)
    want = step()
    tb.check_status()
    for got in (fused, apart):
        for a, r in zip(got, want):
            assert (a.float() - r.float()).norm() <= 2e-2 * r.float().norm() + 1e-5


def test_frozen_projections_cost_no_weight_product(monkeypatch):
    import ttt_rs_b200 as tb
    H, T, C = 3, 128, 192
    cfg = tb.TTTLayerConfig(hidden_size=C, num_heads=H, use_gate=True)
    torch.manual_seed(2)
    m = tb.TTT(cfg, device="cuda", dtype=torch.bfloat16)
    inner = tb.new_inner(cfg, device="cuda", dtype=torch.bfloat16)
    x = (torch.randn(2, T, C, device="cuda") * 0.5).bfloat16().requires_grad_()
    gy = (torch.randn(2, T, C, device="cuda") * 0.1).bfloat16()
    shapes, matmul = [], torch.matmul

    def counted(a, b):
        shapes.append((a.shape[0], b.shape[-1]))
        return matmul(a, b)

    def step():
        shapes.clear()
        m(x, inner, inner.init_state(2)).backward(gy)
        g, x.grad = x.grad, None
        return g

    monkeypatch.setattr(torch, "matmul", counted)
    N = m._stack_weights()[0].shape[0]
    want = step()
    assert (N, C) in shapes
    for p in (m.q_proj, m.k_proj, m.v_proj, m.g_proj, m.learnable_ttt_lr_weight):
        p.requires_grad_(False)
    assert torch.equal(step(), want)
    assert (N, C) not in shapes


def test_lengths_without_the_one_launch_form_stack_no_weights(monkeypatch):
    import ttt_rs_b200 as tb
    H, C = 2, 128
    cfg = tb.TTTLayerConfig(hidden_size=C, num_heads=H)
    m = tb.TTT(cfg, device="cuda", dtype=torch.bfloat16)
    inner = tb.new_inner(cfg, device="cuda", dtype=torch.bfloat16)
    calls, stack = [], m._stack_weights
    monkeypatch.setattr(m, "_stack_weights", lambda: calls.append(1) or stack())
    for T, n in ((144, 0), (256, 1)):
        m(torch.randn(1, T, C, device="cuda").bfloat16(), inner, inner.init_state(1)).sum().backward()
        assert len(calls) == n
