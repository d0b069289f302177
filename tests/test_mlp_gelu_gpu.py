"""TTT-MLP where GELU saturates: pre-activations of tens to a thousand beside ordinary ones, against float64, and that no
token's result depends on a later token of its mini-batch (needs a B200)."""

import pytest
import torch

from oracle import ttt_oracle as O

pytestmark = pytest.mark.gpu
MLP_IN = ("xq", "xk", "xv", "w1", "b1", "w2", "b2", "token_eta", "ttt_lr_eta", "ln_weight", "ln_bias")
STATE = ("w1", "b1", "w2", "b2")


def _case(B, H, NS, seed):
    t = O.make_inputs(B, H, NS * 16, 64, 16, seed=seed, dtype=torch.bfloat16, inner="mlp")
    g = torch.Generator().manual_seed(seed + 1)
    for k, at, scale in (("ln_weight", 1.0, 0.1), ("ln_bias", 0.0, 0.1), ("b1", 0.0, 0.05), ("b2", 0.0, 0.05)):
        t[k] = (at + scale * torch.randn(t[k].shape, generator=g)).to(torch.bfloat16)
    return t


def _forward(t, ws=False):
    import ttt_rs_b200 as tb
    cfg = tb.FusedTttConfig.new(16, 64, 1e-6, 256, 1)
    d = {k: v.cuda() for k, v in t.items()}
    st = tb.TTTMLPState(*[d[k] for k in STATE])
    args = (d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"], d["ln_bias"])
    space = tb.mlp_backward_workspace(d["xq"], cfg) if ws else None
    out, new = tb.fused_ttt_mlp_forward(*args, cfg, backward_workspace=space)
    grads = tb.fused_ttt_mlp_backward(*args, d["grad_output"], cfg, workspace_from_forward=space) if ws else None
    torch.cuda.synchronize()
    tb.TttTileMultiKernel.check_status()
    return out, new, grads


def _err(got, want):
    return ((got.double().cpu() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("z", (-10.0, -30.0, -100.0, -300.0, -1000.0, 30.0))
def test_features_far_out(z):
    """b1 of every fourth hidden feature at z.  Below zero such a feature is dead: its columns of W1 and b1 stay what they were,
    bit for bit, and their gradients are those of the final state (none here).  1e-2 is the bf16 tolerance of L2 errors (measured
    at most 3.6e-3)."""
    t = _case(1, 3, 4, 70)
    t["b1"][..., ::4] = z
    out, new, grads = _forward(t, ws=True)
    a = [t[k].double() for k in MLP_IN]
    ref = O.ttt_mlp_forward(*a, mini_batch=16, eps=1e-6)
    want = O.ttt_mlp_backward_autograd(*a, t["grad_output"].double())
    errs = {"output": _err(out, ref["output"]), **{k: _err(getattr(new, k), ref[k]) for k in STATE},
            **{k: _err(grads[k], want[k]) for k in want if k in grads}}
    print(z, " ".join(f"{k} {e:.2e}" for k, e in errs.items()))
    if z < 0:
        assert torch.equal(new.w1[..., ::4].cpu(), t["w1"][..., ::4]) and torch.equal(new.b1[..., ::4].cpu(), t["b1"][..., ::4])
        for k in ("grad_w1", "grad_b1"):
            dead, live = grads[k][..., ::4].float().abs().max().item(), grads[k].float().pow(2).mean().sqrt().item()
            assert dead < 1e-12 * live, f"{k}: {dead} beside {live}"
    assert max(errs.values()) < 1e-2, errs


def test_one_token_far_out():
    """A single token with pre-activations of both signs in the hundreds: where they are negative it leaves W1 and b1 alone.
    (The biases start from 0: their rounding is then relative to what the mini-batch changed.)"""
    t = _case(2, 2, 1, 80)
    for k in ("b1", "b2"):
        t[k].zero_()
    t["xk"][:, :, 6] *= 20000
    z = torch.einsum("bhk,bhke->bhe", t["xk"][:, :, 6].double(), t["w1"].double())
    assert 200 < z.abs().mean() < 2000
    out, new, _ = _forward(t)
    ref = O.ttt_mlp_forward(*[t[k].double() for k in MLP_IN], mini_batch=16, eps=1e-6)
    errs = {"output": _err(out, ref["output"])}
    for k in STATE:  # what the mini-batch changed
        errs[k] = _err(getattr(new, k).double().cpu() - t[k].double(), ref[k] - t[k].double())
    print(" ".join(f"{k} {e:.2e}" for k, e in errs.items()))
    assert max(errs.values()) < 1e-2, errs


@pytest.mark.parametrize("scale", (1.0, 2000.0))
@pytest.mark.parametrize("last", (7, 14, 15))
def test_no_token_sees_a_later_one(last, scale):
    """Another token `last` in a sequence's last mini-batch: the outputs before it are the same bits."""
    t = _case(2, 3, 2, 90)
    out, _, _ = _forward(t)
    at = 16 + last
    g = torch.Generator().manual_seed(last)
    for k in ("xq", "xk", "xv"):
        t[k] = t[k].clone()
        t[k][:, :, at] = (scale * torch.randn(2, 3, 64, generator=g)).to(torch.bfloat16)
    other, _, _ = _forward(t)
    assert torch.equal(out[:, :, :at], other[:, :, :at])
    assert not torch.equal(out[:, :, at], other[:, :, at])
