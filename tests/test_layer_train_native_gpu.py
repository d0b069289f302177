"""The training step of the layer as one native node against the composition of its steps: same output, state and gradients."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _step(m, inner, x, gy, leaves):
    state = inner.init_state(x.shape[0])
    y = m(x, inner, state)
    grads = torch.autograd.grad(y, leaves, gy, allow_unused=True)
    return [y.detach(), state.weight, state.bias] + list(grads)


def _setup(dtype, B, T, H, F, mb, pos, gate, taps=0, K=4):
    import ttt_rs_b200 as tb
    torch.manual_seed(T + H)
    cfg = tb.TTTLayerConfig(hidden_size=F * H, num_heads=H, mini_batch_size=mb, pos_encoding=pos, use_gate=gate,
                            **(dict(share_qk=True, conv_kernel_size=taps) if taps else {}))
    m = tb.TTT(cfg, device="cuda", dtype=dtype)
    inner = tb.new_inner(cfg, checkpoint_interval=K, device="cuda", dtype=dtype)
    with torch.no_grad():
        for p in list(m.parameters()) + list(inner.inner.parameters()):
            p.add_(torch.randn_like(p) * 0.01)
    x = (torch.randn(B, T, F * H, device="cuda") * 0.5).to(dtype)
    gy = (torch.randn(B, T, F * H, device="cuda") * 0.1).to(dtype)
    return m, inner, x, gy


@pytest.mark.parametrize("dtype,B,T,H,F,mb,pos,gate,taps", [
    (torch.bfloat16, 1, 16, 1, 64, 16, "rope", False, 0), (torch.bfloat16, 2, 144, 3, 64, 16, "rope", True, 0),
    (torch.bfloat16, 3, 200, 5, 64, 8, "none", True, 0), (torch.bfloat16, 2, 128, 4, 32, 16, "rope", True, 0),
    (torch.bfloat16, 1, 256, 2, 64, 16, "rope_global", False, 0), (torch.float32, 2, 48, 3, 64, 16, "rope", True, 0),
    (torch.float32, 1, 128, 2, 64, 16, "rope", False, 0), (torch.float32, 2, 24, 2, 32, 8, "rope", True, 0),
    (torch.bfloat16, 2, 144, 3, 64, 16, "rope", True, 4), (torch.bfloat16, 1, 128, 2, 64, 16, "none", False, 2),
    (torch.float32, 2, 48, 2, 32, 16, "rope", True, 3)])
def test_one_node_equals_the_composition(monkeypatch, dtype, B, T, H, F, mb, pos, gate, taps):
    from ttt_rs_b200 import layer as L
    m, inner, x, gy = _setup(dtype, B, T, H, F, mb, pos, gate, taps)
    x.requires_grad_()
    leaves = [x] + list(m.parameters()) + list(inner.inner.parameters())
    used, native = [], L._train_native

    def counted(*a):
        r = native(*a)
        used.append(r is not None)
        return r

    monkeypatch.setattr(L, "_train_native", counted)
    got = _step(m, inner, x, gy, leaves)
    assert used == [True]
    # a strided view of the input, and a second backward over the same graph
    wide = torch.stack((x.detach(), x.detach()), dim=-1)[..., 0].requires_grad_()
    again = _step(m, inner, wide, gy, [wide] + leaves[1:])
    monkeypatch.setattr(L, "_train_native", lambda *a: None)
    want = _step(m, inner, x, gy, leaves)
    # bf16: two orders of the same sums, 2-norm; float32 sums over tokens likewise
    tol = 2e-2 if dtype == torch.bfloat16 else 1e-4
    for a, b, c in zip(got, again, want):
        assert a.shape == c.shape and a.dtype == c.dtype
        assert (a.float() - c.float()).norm() <= tol * c.float().norm() + 1e-6
        assert torch.equal(a, b)


def test_frozen_parameters_and_a_second_backward():
    m, inner, x, gy = _setup(torch.bfloat16, 2, 48, 2, 64, 16, "rope", True)
    state = inner.init_state(2)
    y = m(x, inner, state)  # the input itself needs no gradient
    params = list(m.parameters()) + list(inner.inner.parameters())
    a = torch.autograd.grad(y, params, gy, retain_graph=True)
    b = torch.autograd.grad(y, params, gy)
    assert all(torch.equal(p, q) for p, q in zip(a, b))
    for p in (m.q_proj, m.k_proj, m.v_proj, m.g_proj, m.learnable_ttt_lr_weight, m.o_proj):
        p.requires_grad_(False)
    rest = [p for p in params if p.requires_grad]
    c = torch.autograd.grad(m(x, inner, inner.init_state(2)), rest, gy)
    want = {id(p): g for p, g in zip(params, a)}
    assert all(torch.equal(g, want[id(p)]) for p, g in zip(rest, c))


def test_saved_tensors_go_through_hooks():
    m, inner, x, gy = _setup(torch.bfloat16, 1, 32, 2, 64, 16, "rope", False)
    params = list(m.parameters())
    want = torch.autograd.grad(m(x, inner, inner.init_state(1)), params, gy)
    with torch.autograd.graph.save_on_cpu():
        y = m(x, inner, inner.init_state(1))
    got = torch.autograd.grad(y, params, gy)
    assert all(torch.equal(p, q) for p, q in zip(got, want))
